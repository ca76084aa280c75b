// lbm_fast.cu -- f32-arithmetic step kernels for f32, binary16-shift and
// bfloat16-shift storage (ModeFast).  Built with multiply-add contraction on.
#include "lbm_batch.cuh"
#include "lbm_compact.cuh"
#include "lbm_kernels.cuh"
#include "lbm_launch.h"

namespace lbm {

// The list of k_step4's leading blocks that quad q belongs to (QuadKind), or
// -1 for the quads that the plain path steps.
struct RuleQuadKind {
    Params P;
    __device__ int operator()(int q) const
    {
        const int idx0 = 4 * q;
        int x, y, z0;
        decode_xyz(P, idx0, x, y, z0);
        const uint32_t fl4 = P.has_flags ? *reinterpret_cast<const uint32_t*>(P.flags + idx0) : 0u;
        if (quad_on_walled_face(P, x, y, z0)) return QUAD_KIND_OTHER;
        if (fl4 == 0u || fl4 == QUAD_SOLID || fl4 == QUAD_INFLOW) return -1;  // k_step4 steps it
        // bytes of four cells, each fluid or solid (near-solid bits allowed)
        if ((fl4 & 0x02020202u) == 0u) return QUAD_KIND_NEAR;
        if (fl4 == QUAD_OUTFLOW) {
            const int gx = x == 0 ? P.nx - 1 : x - 1;
            const uint32_t g4 = *reinterpret_cast<const uint32_t*>(P.flags + idx0 + (gx - x) * P.nynz);
            if (g4 == 0u && !quad_on_walled_face(P, gx, y, z0)) return QUAD_KIND_OUTFLOW;
        }
        return QUAD_KIND_OTHER;
    }
};

// Items (of vec cells) on the walled faces are kind 0; the others have their
// place in the visit order by their rank in the interior box.
struct FaceItem {
    Params P;
    int vec;
    __host__ __device__ long long inner_items() const
    {
        const long long bx = P.nx - 2 * (int)P.walled[0], by = P.ny - 2 * (int)P.walled[1],
                        bz = P.nz / vec - 2 * (int)P.walled[2];
        return bx > 0 && by > 0 && bz > 0 ? bx * by * bz : 0;
    }
    // rank in the interior box, or -1 for an item on a walled face
    __device__ int inner_rank(int p) const
    {
        const int nzi = P.nz / vec;  // items per row
        int x, y, z0;
        decode_xyz(P, p * vec, x, y, z0);
        const int zi = z0 / vec;
        const int xo = (int)P.walled[0], yo = (int)P.walled[1], zo = (int)P.walled[2];
        const int bx = P.nx - 2 * xo, by = P.ny - 2 * yo, bz = nzi - 2 * zo;
        const bool inner = bx > 0 && by > 0 && bz > 0 && x >= xo && x < P.nx - xo && y >= yo && y < P.ny - yo &&
                           zi >= zo && zi < nzi - zo;
        return inner ? ((x - xo) * by + (y - yo)) * bz + (zi - zo) : -1;
    }
    __device__ int operator()(int p) const { return inner_rank(p) < 0 ? 0 : -1; }
};

__global__ void k_inner_order(FaceItem F, int items, int* __restrict__ order)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= items) return;
    const int r = F.inner_rank(p);
    if (r >= 0) order[items - (int)F.inner_items() + r] = p;
}

cudaError_t launch_face_order(const Params& P, int vec, int* order, cudaStream_t s)
{
    const FaceItem F{P, vec};
    const int items = P.n / vec;
    int* faces = order + items;
    k_inner_order<<<grid_for(items, 256), 256, 0, s>>>(F, items, order);
    return compact<1>(F, items, order, 0, faces, faces + 1, s);
}

size_t face_order_ints(int items) { return (size_t)items + 1 + compact_scratch(items, 1); }

cudaError_t launch_list_rule_quads(const Params& P, int* lists, cudaStream_t s)
{
    const size_t cap = (size_t)P.n / 4;
    int* counts = lists + QUAD_KINDS * cap;
    return compact<QUAD_KINDS>(RuleQuadKind{P}, (int)cap, lists, cap, counts, counts + QUAD_KINDS, s);
}

size_t rule_quad_ints(int quads)
{
    return (size_t)QUAD_KINDS * quads + QUAD_KINDS + compact_scratch(quads, QUAD_KINDS);
}

// Kind 0: the flat quads that k_step4_flat leaves to its leading blocks.
struct FlatRuleQuad {
    Params P;
    __device__ int operator()(int q) const
    {
        const int idx0 = 4 * q;
        int x, y, z0;
        decode_xyz(P, idx0, x, y, z0);
        if (flat_quad_split(P, idx0, x, y, z0)) return 0;
        const uint32_t fl4 = P.has_flags ? *reinterpret_cast<const uint32_t*>(P.flags + idx0) : 0u;
        return fl4 == 0u || fl4 == QUAD_SOLID || fl4 == QUAD_INFLOW ? -1 : 0;
    }
};

cudaError_t launch_list_flat_rules(const Params& P, int* list, cudaStream_t s)
{
    const int quads = (P.n + 3) / 4;
    int* count = list + quads;
    return compact<1>(FlatRuleQuad{P}, quads, list, 0, count, count + 1, s);
}

size_t flat_rule_ints(int quads) { return (size_t)quads + 1 + compact_scratch(quads, 1); }

// k_step4 over the window's quads, led by the blocks that step the rule quads
// (a.rules_grid of them, at most one task per thread).
template <class M, int FM>
static cudaError_t launch_step4(const LaunchArgs& a, const Streams<typename M::T>& S)
{
    const int total = a.rule_counts[0] + a.rule_counts[1] + a.rule_counts[2];
    const size_t cap = (size_t)a.P.n / 4;
    const int* L = a.rule_quads;
    RuleQuads rq{L + QUAD_KIND_NEAR * cap, L + QUAD_KIND_OUTFLOW * cap, L + QUAD_KIND_OTHER * cap,
                 a.rule_counts[QUAD_KIND_NEAR], a.rule_counts[QUAD_KIND_OUTFLOW], a.rule_counts[QUAD_KIND_OTHER], 0};
    const int block = a.block < 128 ? a.block : 128;  // the kernel's bound
    if (total > 0) {
        const int one_each = grid_for(2LL * total, block);
        rq.blocks = a.rules_grid > 0 && a.rules_grid < one_each ? a.rules_grid : one_each;
    }
    k_step4<M, FM><<<rq.blocks + grid_for(window_cells(a.P) / 4, block), block, 0, a.stream>>>(a.P, S, rq);
    return cudaGetLastError();
}

// k_step4_flat over the window's quads, led by the blocks that step the cells
// of the rule quads (a.rules_grid of them, at most one cell per thread).
template <class M, int FM>
static cudaError_t launch_step4_flat(const LaunchArgs& a, const Streams<typename M::T>& S)
{
    const int block = a.block < 128 ? a.block : 128;  // the kernel's bound
    const int first = a.P.cell0 / 4, end = a.P.cell_end < a.P.n ? a.P.cell_end : a.P.n;
    const int rules = a.rule_counts[0];
    int rblocks = 0;
    if (rules > 0) {
        const int one_each = grid_for(4LL * rules, block);
        rblocks = a.rules_grid > 0 && a.rules_grid < one_each ? a.rules_grid : one_each;
    }
    const int grid = rblocks + grid_for((end + 3) / 4 - first, block);
    k_step4_flat<M, FM><<<grid, block, 0, a.stream>>>(a.P, S, a.rule_quads, rules, rblocks);
    return cudaGetLastError();
}

template <class M, int FM, int OUT>
static cudaError_t launch_step_out(int kernel, const LaunchArgs& a, int grid)
{
    using T = typename M::T;
    Outputs<float> out{(float*)a.rho, (float*)a.u, a.partials, a.prev_partials, a.prev_count, a.prev_sums};
    const Streams<T> S = make_streams<T>(a.src, a.dst, a.P.stride);
    if constexpr (sizeof(T) == 2 && OUT == OUT_NONE) {
        if (kernel == KERNEL_STEP && a.vec == 2 && a.pipe_grid > 0) {
            k_step2_pipe<M, FM><<<a.pipe_grid, a.block, 0, a.stream>>>(a.P, S);
            if (a.grid_used) *a.grid_used = a.pipe_grid;
            return cudaGetLastError();
        }
        if (kernel == KERNEL_STEP && a.vec == 4) return launch_step4<M, FM>(a, S);
        if (kernel == KERNEL_STEP && a.flat) return launch_step4_flat<M, FM>(a, S);
    }
    // Steps with readback or sums of a four-cell lattice run the two-cell kernels.
    if constexpr (OUT == OUT_SUMS) {
        if (kernel == KERNEL_STEP && a.vec >= 2 && a.sums_grid > 0) {
            k_step2_sums<M, FM><<<a.sums_grid, a.block, 0, a.stream>>>(a.P, S, out);
            if (a.grid_used) *a.grid_used = a.sums_grid;
            return cudaGetLastError();
        }
    }
    if (kernel == KERNEL_STEP && a.vec >= 2) {
        // at most the kernel's bound (128 threads for 16-bit storage)
        const int block = a.block < Step2Bounds<T>::threads ? a.block : Step2Bounds<T>::threads;
        const int grid2 = grid_for(window_cells(a.P) / 2, block);
        if (OUT == OUT_NONE && a.P.first.on)
            k_step2<M, FM, OUT, OUT == OUT_NONE><<<grid2, block, 0, a.stream>>>(a.P, S, out);
        else
            k_step2<M, FM, OUT><<<grid2, block, 0, a.stream>>>(a.P, S, out);
        if (a.grid_used) *a.grid_used = grid2;
        return cudaGetLastError();
    }
    if (kernel == KERNEL_STEP)
        k_step<M, FM, OUT><<<grid, a.block, 0, a.stream>>>(a.P, S, out);
    else
        k_collide_local<M, FM, OUT><<<grid, a.block, 0, a.stream>>>(a.P, S, out);
    if (a.grid_used) *a.grid_used = grid;
    return cudaGetLastError();
}

template <class T, int FM>
static cudaError_t launch_fast_t(int kernel, const LaunchArgs& a)
{
    using M = ModeFast<T>;
    const int grid = grid_for(kernel == KERNEL_OBSERVE ? a.P.n : window_cells(a.P), a.block);
    if (kernel == KERNEL_OBSERVE) {
        Outputs<float> out{(float*)a.rho, (float*)a.u, a.partials, a.prev_partials, a.prev_count, a.prev_sums,
                          a.first, a.count};
        const int ogrid = a.count < 0 ? grid : grid_for(a.count, a.block);
        k_observe<M, FM><<<ogrid, a.block, 0, a.stream>>>(a.P, make_streams<T>(a.src, nullptr, a.P.stride), a.post,
                                                          a.f_out, out);
        return cudaGetLastError();
    }
    if (kernel != KERNEL_STEP && kernel != KERNEL_COLLIDE_LOCAL) return cudaErrorInvalidValue;
    if ((a.vec == 2 && (a.P.nz % 2) != 0) || (a.vec == 4 && (a.P.nz % 4 != 0 || sizeof(T) != 2)))
        return cudaErrorInvalidValue;
    switch (out_bits(a)) {
    case OUT_NONE: return launch_step_out<M, FM, OUT_NONE>(kernel, a, grid);
    case OUT_RHO_U: return launch_step_out<M, FM, OUT_RHO_U>(kernel, a, grid);
    case OUT_SUMS: return launch_step_out<M, FM, OUT_SUMS>(kernel, a, grid);
    default: return cudaErrorInvalidValue;
    }
}

template <class T>
static cudaError_t launch_fast_fm(int kernel, int force_mode, const LaunchArgs& a)
{
    switch (force_mode) {
    case FORCE_NONE: return launch_fast_t<T, FORCE_NONE>(kernel, a);
    case FORCE_UNIFORM: return launch_fast_t<T, FORCE_UNIFORM>(kernel, a);
    case FORCE_FIELD: return launch_fast_t<T, FORCE_FIELD>(kernel, a);
    case FORCE_DRAG: return launch_fast_t<T, FORCE_DRAG>(kernel, a);
    default: return cudaErrorInvalidValue;
    }
}

template <class T, int FM>
static cudaError_t batch_fm(int sched, bool collide, const void* records, const void* items, int nitems, int span,
                            int phase, int grid, int block, cudaStream_t s)
{
    using M = ModeFast<T>;
    const auto* L = (const BatchLattice<T>*)records;
    const auto* I = (const BatchItem*)items;
    if (collide) {
        k_collide_batch<M, FM><<<grid, block, 0, s>>>(L, I, nitems, span, phase);
        return cudaGetLastError();
    }
    if constexpr (FM == FORCE_NONE || FM == FORCE_UNIFORM) {
        if (sched == SCHED_PAIR_SCALAR) {
            k_step_batch<M, FM, SCHED_PAIR_SCALAR><<<grid, block, 0, s>>>(L, I, nitems, phase);
            return cudaGetLastError();
        }
        if (sched == SCHED_PAIR_MIXED) {
            k_step_batch<M, FM, SCHED_PAIR_MIXED><<<grid, block, 0, s>>>(L, I, nitems, phase);
            return cudaGetLastError();
        }
    }
    if (sched != SCHED_SINGLE) return cudaErrorInvalidValue;
    k_step_batch<M, FM, SCHED_SINGLE><<<grid, block, 0, s>>>(L, I, nitems, phase);
    return cudaGetLastError();
}

template <class T>
static cudaError_t batch_t(int force_mode, int sched, bool collide, const void* records, const void* items,
                           int nitems, int span, int phase, int grid, int block, cudaStream_t s)
{
    switch (force_mode) {
    case FORCE_NONE: return batch_fm<T, FORCE_NONE>(sched, collide, records, items, nitems, span, phase, grid, block, s);
    case FORCE_UNIFORM:
        return batch_fm<T, FORCE_UNIFORM>(sched, collide, records, items, nitems, span, phase, grid, block, s);
    case FORCE_FIELD:
        return batch_fm<T, FORCE_FIELD>(sched, collide, records, items, nitems, span, phase, grid, block, s);
    case FORCE_DRAG: return batch_fm<T, FORCE_DRAG>(sched, collide, records, items, nitems, span, phase, grid, block, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_batch_exact(int force_mode, bool collide, const void* records, const void* items, int nitems,
                               int span, int phase, int grid, int block, cudaStream_t s);

cudaError_t launch_batch_step(int storage, int force_mode, int sched, bool collide, const void* records,
                              const void* items, int nitems, int span, int phase, int grid, int block,
                              cudaStream_t s)
{
    switch (storage) {
    case STORAGE_F64:
        if (sched != SCHED_SINGLE && !collide) return cudaErrorInvalidValue;
        return launch_batch_exact(force_mode, collide, records, items, nitems, span, phase, grid, block, s);
    case STORAGE_F32:
        return batch_t<float>(force_mode, sched, collide, records, items, nitems, span, phase, grid, block, s);
    case STORAGE_F16:
        return batch_t<__half>(force_mode, sched, collide, records, items, nitems, span, phase, grid, block, s);
    case STORAGE_BF16:
        return batch_t<__nv_bfloat16>(force_mode, sched, collide, records, items, nitems, span, phase, grid, block,
                                      s);
    default: return cudaErrorInvalidValue;
    }
}

size_t batch_record_bytes(int storage)
{
    switch (storage) {
    case STORAGE_F64: return sizeof(BatchLattice<double>);
    case STORAGE_F32: return sizeof(BatchLattice<float>);
    case STORAGE_F16: return sizeof(BatchLattice<__half>);
    case STORAGE_BF16: return sizeof(BatchLattice<__nv_bfloat16>);
    default: return 0;
    }
}

// Resident blocks per SM x SMs of the current device for a kernel.
template <class K>
static int resident_grid(K kernel, int block)
{
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0) != cudaSuccess) return 0;
    return sms * per_sm;
}

template <class T, int FM>
static int loop_grid_t(bool sums, int block)
{
    if (sums) return resident_grid(k_step2_sums<ModeFast<T>, FM>, block);
    if constexpr (sizeof(T) == 2) return resident_grid(k_step2_pipe<ModeFast<T>, FM>, block);
    return 0;
}

template <class T>
static int loop_grid_fm(bool sums, int force_mode, int block)
{
    switch (force_mode) {
    case FORCE_NONE: return loop_grid_t<T, FORCE_NONE>(sums, block);
    case FORCE_UNIFORM: return loop_grid_t<T, FORCE_UNIFORM>(sums, block);
    case FORCE_FIELD: return loop_grid_t<T, FORCE_FIELD>(sums, block);
    case FORCE_DRAG: return loop_grid_t<T, FORCE_DRAG>(sums, block);
    default: return 0;
    }
}

static int loop_grid(bool sums, int storage, int force_mode, int block)
{
    switch (storage) {
    case STORAGE_F32: return loop_grid_fm<float>(sums, force_mode, block);
    case STORAGE_F16: return loop_grid_fm<__half>(sums, force_mode, block);
    case STORAGE_BF16: return loop_grid_fm<__nv_bfloat16>(sums, force_mode, block);
    default: return 0;
    }
}

int pipe_grid_fast(int storage, int force_mode, int block) { return loop_grid(false, storage, force_mode, block); }

int sums_grid_fast(int storage, int force_mode, int block) { return loop_grid(true, storage, force_mode, block); }

template <class T, int FM>
static cudaError_t persistent_fm_t(const LaunchArgs& a, int steps, GridBarrier* bar, unsigned missing,
                                   unsigned long long timeout_ns, int* grid_out)
{
    if (a.vec >= 2) return persistent_t<ModeFast<T, true>, FM, 2>(a, steps, bar, missing, timeout_ns, grid_out);
    return persistent_t<ModeFast<T, true>, FM, 1>(a, steps, bar, missing, timeout_ns, grid_out);
}

template <class T>
static cudaError_t persistent_fast_t(int force_mode, const LaunchArgs& a, int steps, GridBarrier* bar,
                                     unsigned missing, unsigned long long timeout_ns, int* grid_out)
{
    switch (force_mode) {
    case FORCE_NONE: return persistent_fm_t<T, FORCE_NONE>(a, steps, bar, missing, timeout_ns, grid_out);
    case FORCE_UNIFORM: return persistent_fm_t<T, FORCE_UNIFORM>(a, steps, bar, missing, timeout_ns, grid_out);
    case FORCE_FIELD: return persistent_fm_t<T, FORCE_FIELD>(a, steps, bar, missing, timeout_ns, grid_out);
    case FORCE_DRAG: return persistent_fm_t<T, FORCE_DRAG>(a, steps, bar, missing, timeout_ns, grid_out);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_persistent_exact(int force_mode, const LaunchArgs& a, int steps, GridBarrier* bar,
                                    unsigned missing, unsigned long long timeout_ns, int* grid_out);

cudaError_t launch_persistent(int storage, int force_mode, const LaunchArgs& a, int steps, GridBarrier* bar,
                              unsigned missing, unsigned long long timeout_ns, int* grid_out)
{
    switch (storage) {
    case STORAGE_F64: return launch_persistent_exact(force_mode, a, steps, bar, missing, timeout_ns, grid_out);
    case STORAGE_F32: return persistent_fast_t<float>(force_mode, a, steps, bar, missing, timeout_ns, grid_out);
    case STORAGE_F16: return persistent_fast_t<__half>(force_mode, a, steps, bar, missing, timeout_ns, grid_out);
    case STORAGE_BF16:
        return persistent_fast_t<__nv_bfloat16>(force_mode, a, steps, bar, missing, timeout_ns, grid_out);
    default: return cudaErrorInvalidValue;
    }
}

template <class T, int FM>
static cudaError_t read_t(const Params& P, const void* src, bool post, double* rho, double* u, cudaStream_t s)
{
    using M = ModeFast<T>;
    const Streams<T> S = make_streams<T>(src, nullptr, P.stride);
    const int block = 128;
    // two doubles at a time where the arrays allow it (n is even for even nz)
    const bool wide = post && P.nz % 2 == 0 && (uintptr_t)rho % 16 == 0 && (uintptr_t)u % 16 == 0;
    if constexpr (sizeof(T) == 2) {
        if (wide && P.nz % 4 == 0) {
            k_read<M, FM, 4><<<grid_for(P.n / 4, block), block, 0, s>>>(P, S, post, rho, u);
            return cudaGetLastError();
        }
    }
    if (wide) k_read<M, FM, 2><<<grid_for(P.n / 2, block), block, 0, s>>>(P, S, post, rho, u);
    else k_read<M, FM, 1><<<grid_for(P.n, block), block, 0, s>>>(P, S, post, rho, u);
    return cudaGetLastError();
}

template <class T>
static cudaError_t read_fm(int force_mode, const Params& P, const void* src, bool post, double* rho, double* u,
                           cudaStream_t s)
{
    switch (force_mode) {
    case FORCE_NONE: return read_t<T, FORCE_NONE>(P, src, post, rho, u, s);
    case FORCE_UNIFORM: return read_t<T, FORCE_UNIFORM>(P, src, post, rho, u, s);
    case FORCE_FIELD: return read_t<T, FORCE_FIELD>(P, src, post, rho, u, s);
    case FORCE_DRAG: return read_t<T, FORCE_DRAG>(P, src, post, rho, u, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_read(int storage, int force_mode, const Params& P, const void* src, bool post, double* rho,
                        double* u, cudaStream_t s)
{
    switch (storage) {
    case STORAGE_F32: return read_fm<float>(force_mode, P, src, post, rho, u, s);
    case STORAGE_F16: return read_fm<__half>(force_mode, P, src, post, rho, u, s);
    case STORAGE_BF16: return read_fm<__nv_bfloat16>(force_mode, P, src, post, rho, u, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_fast(int storage, int kernel, int force_mode, const LaunchArgs& a)
{
    switch (storage) {
    case STORAGE_F32: return launch_fast_fm<float>(kernel, force_mode, a);
    case STORAGE_F16: return launch_fast_fm<__half>(kernel, force_mode, a);
    case STORAGE_BF16: return launch_fast_fm<__nv_bfloat16>(kernel, force_mode, a);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace lbm
