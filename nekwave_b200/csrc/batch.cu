// batch.cu -- kernels of the multi-cavity pool.
//
// One launch per order and LSRK stage advances that order's resident cavities:
// a block takes the tile (EPB consecutive elements of one cavity) that the work
// list has at its index and runs the single-mesh default's tile of that order
// (stage_bulk.cuh, stage_quad.cuh, stage_dmma.cuh) on the slot's arrays.  The other
// mode is one persistent launch per stage whatever the orders: blocks of
// kBatchThreads threads take tiles through a per-stage atomic counter, largest
// first, and run the tile of its order that fits such a block.
// A cavity's arithmetic does not depend on which other cavities share the
// launch, so each result is bit-identical alone and in any mix.
#include "batch.cuh"
#include "stage_kernel.cuh"
#include "stage_pipe.cuh"
#include "stage_dmma.cuh"
#include "stage_bulk.cuh"
#include "stage_quad.cuh"
#include "stage_variants.h"

namespace nwb {
namespace {

using stage::SmemLayout;
using stage::stage_tile;

// Shape per N for the batch kernel's blocks (kBatchThreads = 128): KS threads
// per column, EPB elements, ALG the kernel family -- the single-mesh default's
// arithmetic for each N, in a shape that
// fits, so a cavity in the pool evolves bit for bit as it does alone.  N = 8 in
// FP64 runs the field-split tensor-core tile (stage_dmma.cuh, 128 threads) as the
// single-mesh default does; ALG below is its FP32-bulk shape.
template <int N> struct BShape;
template <> struct BShape<2> { static constexpr int KS = 2, EPB = 16, ALG = 4; };
template <> struct BShape<3> { static constexpr int KS = 1, EPB = 14, ALG = 4; };
template <> struct BShape<4> { static constexpr int KS = 2, EPB = 4, ALG = 4; };
template <> struct BShape<5> { static constexpr int KS = 2, EPB = 2, ALG = 4; };
template <> struct BShape<6> { static constexpr int KS = 2, EPB = 1, ALG = 4; };
template <> struct BShape<7> { static constexpr int KS = 2, EPB = 1, ALG = 4; };
template <> struct BShape<8> { static constexpr int KS = 2, EPB = 1, ALG = 4; };
template <> struct BShape<9> { static constexpr int KS = 1, EPB = 1, ALG = 4; };
template <> struct BShape<10> { static constexpr int KS = 1, EPB = 1, ALG = 4; };

// N = 8 in FP64: the single-mesh default is the field-split tensor-core tile
template <int N, bool F32>
__host__ __device__ constexpr bool dmma_tile() { return N == 8 && !F32; }

// the family of an N in the mixed launch: FP32-bulk keeps the first at 2, 3 and 10 points
template <int N, bool F32>
__host__ __device__ constexpr int balg() { return F32 && (N == 2 || N == 3 || N == 10) ? 0 : BShape<N>::ALG; }

template <int N, bool F32>
constexpr int bsmem() {
    using B = BShape<N>;
    constexpr int ALG = balg<N, F32>();
    if constexpr (dmma_tile<N, F32>()) return stage::DmmaLayout8::total;
    else if constexpr (ALG == 0) return SmemLayout<N, F32, B::EPB, false>::total;
    else return stage::Layout2<N, F32, B::EPB, false, (((ALG - 2) & 4) != 0),
                               stage::flux_planes<GEO_BOX, (((ALG - 2) & 2) != 0)>()>::total;
}

// One tile of the second family without the persistent loop: stage u_in (and D,
// geometry, connections), wait, compute.  Threads beyond the shape's count take
// part in the barriers only.
template <int N, bool F32, int KS, int EPB, int ALG>
__device__ __forceinline__ void tile2(const StageParams& P, int e0, unsigned char* smem, int tid,
                                      const double* Dc = nullptr) {
    constexpr bool SPLIT = ((ALG - 2) & 2) != 0, PAD = ((ALG - 2) & 4) != 0;
    constexpr bool CONSTD = ((ALG - 2) & 8) != 0;
    static_assert(((ALG - 2) & 1) == 0 && ((ALG - 2) & 16) == 0, "one tile per call, tile resident");
    using L2 = stage::Layout2<N, F32, EPB, false, PAD, stage::flux_planes<GEO_BOX, SPLIT>()>;
    constexpr int NT = EPB * KS * N * N;
    double* sD = reinterpret_cast<double*>(smem + L2::D);
    double* su = reinterpret_cast<double*>(smem + L2::u0);
    ElemGeo* sg = reinterpret_cast<ElemGeo*>(smem + L2::geo0);
    int* sc = reinterpret_cast<int*>(smem + L2::conn0);
    if (tid < NT) {
        for (int x = tid; x < N * N; x += NT) stage::cp_async8(sD + x, P.D + x);
        stage::issue2<N, GEO_BOX, EPB, NT, PAD>(P, e0, su, sg, sc, tid);
    }
    stage::cp_async_commit();
    stage::cp_async_wait<0>();
    __syncthreads();
    stage::FaceRegs<N, GEO_BOX, KS, SPLIT> G;
    stage::compute2<N, GEO_BOX, F32, KS, EPB, SPLIT, PAD, CONSTD>(P, e0, su, sg, sc, sD,
                                                                  reinterpret_cast<double*>(smem + L2::flux),
                                                                  smem + L2::uc, tid, G, Dc);
}

template <int N, bool F32>
__device__ __forceinline__ void run_tile(const StageParams& P, int e0, unsigned char* smem, int tid) {
    using B = BShape<N>;
    static_assert(B::KS * B::EPB * N * N <= kBatchThreads, "shape too large");
    if constexpr (dmma_tile<N, F32>())
        stage::dmma8_tile(P, e0, smem, tid,
                             reinterpret_cast<const double*>(smem + stage::DmmaLayout8::D));
    else if constexpr (balg<N, F32>() == 0)
        stage_tile<N, GEO_BOX, F32, B::KS, B::EPB, false, false>(P, e0, smem, tid);
    else
        tile2<N, F32, B::KS, B::EPB, balg<N, F32>()>(P, e0, smem, tid);
}

// Carpenter-Kennedy LSRK45 (src/dg_solver.cpp:58-69), for the host and the device.
#define NWB_RK4A {0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0, \
                  -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0}
#define NWB_RK4B {1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0, \
                  1720146321549.0 / 2090206949498.0, 3134564353537.0 / 4481467310338.0, \
                  2277821191437.0 / 14882151754819.0}
__constant__ double c_rk4a[5] = NWB_RK4A;
__constant__ double c_rk4b[5] = NWB_RK4B;
const double kRk4a[5] = NWB_RK4A;
const double kRk4b[5] = NWB_RK4B;

template <bool F32>
__global__ void __launch_bounds__(kBatchThreads, 3)
batch_stage_kernel(const SlotDev* __restrict__ slots, const WorkItem* __restrict__ work,
                   const int* __restrict__ ntiles_p, int* __restrict__ counters, int stage, int dry) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_tile;
    const int tid = threadIdx.x;
    const int ntiles = *ntiles_p;
    for (;;) {
        __syncthreads();  // the previous tile is done with shared memory
        if (tid == 0) s_tile = atomicAdd(&counters[stage], 1);
        __syncthreads();
        const int t = s_tile;
        if (t >= ntiles) break;
        const WorkItem w = work[t];
        const SlotDev& S = slots[w.slot];
        if (!S.active || S.oblique) continue;
        const int par = S.par ^ (stage & 1);
        StageParams P;
        P.u_in = S.u[par];
        P.u_out = S.u[par ^ 1];
        P.k = S.k;
        P.stride = S.stride;
        P.nelt = S.nelt;
        P.kio = stage_kio(stage);
        P.D = S.D;
        P.geo = S.geo;
        P.conn = S.conn;
        P.met_n = nullptr;
        P.fnrm = nullptr;
        P.flift = nullptr;
        P.fplus = nullptr;
        P.nfp = 0;
        P.err = nullptr;  // no bounded waits in this launch's tiles
        P.snel[0] = P.snel[1] = P.snel[2] = 0;  // connections from the slot's table
        P.spmask = 0;
        for (int x = 0; x < 10; ++x) P.zl[x] = S.zl[x];
        P.c0 = S.c0;
        P.a = dry ? 0.0 : c_rk4a[stage];
        P.b = dry ? 0.0 : c_rk4b[stage];
        P.dt = dry ? 0.0 : S.dt;
        switch (w.N) {
            case 2: run_tile<2, F32>(P, w.e0, smem, tid); break;
            case 3: run_tile<3, F32>(P, w.e0, smem, tid); break;
            case 4: run_tile<4, F32>(P, w.e0, smem, tid); break;
            case 5: run_tile<5, F32>(P, w.e0, smem, tid); break;
            case 6: run_tile<6, F32>(P, w.e0, smem, tid); break;
            case 7: run_tile<7, F32>(P, w.e0, smem, tid); break;
            case 8: run_tile<8, F32>(P, w.e0, smem, tid); break;
            case 9: run_tile<9, F32>(P, w.e0, smem, tid); break;
            case 10: run_tile<10, F32>(P, w.e0, smem, tid); break;
            default: break;
        }
    }
}

// What a per-N launch knows of its stage: the LSRK coefficients are kernel parameters
// (constant-bank operands, no registers); dry: a = b = dt = 0 (timing only).
// The stages of one N follow each other on one stream: all but the first may start
// early (launch_overlapped; the slot table does not change within a step).
struct BatchStage {
    double a, b;
    int stage, dry;
    int* err;  // the pool's status word: a bulk tile whose bounded wait expires records it there
    bool overlap() const { return stage > 0; }
};

// Stage parameters of one tile's slot.
__device__ __forceinline__ StageParams slot_params(const SlotDev& S, const BatchStage& bs) {
    const int par = S.par ^ (bs.stage & 1);
    StageParams P;
    P.u_in = S.u[par];
    P.u_out = S.u[par ^ 1];
    P.k = S.k;
    P.stride = S.stride;
    P.nelt = S.nelt;
    P.kio = stage_kio(bs.stage);
    P.D = S.D;
    P.geo = S.geo;
    P.conn = S.conn;
    P.met_n = nullptr;
    P.fnrm = nullptr;
    P.flift = nullptr;
    P.fplus = nullptr;
    P.nfp = 0;
    P.err = bs.err;
    for (int x = 0; x < 3; ++x) P.snel[x] = S.snel[x];
    for (int x = 0; x < 2; ++x) {
        P.sdiv[x] = S.sdiv[x];
        P.sshift[x] = S.sshift[x];
    }
    P.spmask = S.spmask;
    for (int x = 0; x < 10; ++x) P.zl[x] = S.zl[x];
    P.c0 = S.c0;
    P.a = bs.a;
    P.b = bs.b;
    P.dt = bs.dry ? 0.0 : S.dt;
    return P;
}

// D of one N by value, for the constant-bank form of the per-N kernels.
struct DParam {
    double d[100];
    float f[100];  // rounded to FP32 (FP32-bulk)
};

// D of one N by value (null: zeros, for kernels that take it from shared memory).
DParam d_param(int N, const double* Dh) {
    DParam dp{};
    for (int x = 0; Dh && x < N * N; ++x) {
        dp.d[x] = Dh[x];
        dp.f[x] = static_cast<float>(Dh[x]);
    }
    return dp;
}

// N = 8 in FP64, per-N mode: the single-mesh default's field-split tensor-core tile
// (128 threads, one element per block), D from dp (CD) or from shared memory.
template <int MINB, bool CD>
__global__ void __launch_bounds__(128, MINB)
batch_dmma8_kernel(const SlotDev* __restrict__ slots, const WorkItem* __restrict__ work,
                   const __grid_constant__ BatchStage bs, const __grid_constant__ DParam dp) {
    extern __shared__ __align__(16) unsigned char smem[];
    const WorkItem w = work[blockIdx.x];
    const SlotDev& S = slots[w.slot];
    if (!S.active) {
        stage::grid_wait();
        return;
    }
    const StageParams P = slot_params(S, bs);
    stage::dmma8_tile(P, w.e0, smem, threadIdx.x,
                         CD ? dp.d : reinterpret_cast<const double*>(smem + stage::DmmaLayout8::D));
}

template <bool CD>
cudaError_t launch_dmma8_n(const BatchStage& bs, const SlotDev* slots, const WorkItem* work, int ntiles,
                           const DParam& dp, cudaStream_t st) {
    constexpr int smem = stage::DmmaLayout8::total;
    auto kern = batch_dmma8_kernel<4, CD>;
    static std::atomic<int> attr_set[kMaxDeviceSlots];  // per kernel and device
    if (cudaError_t e = set_smem_once(kern, smem, attr_set); e != cudaSuccess) return e;
    if (ntiles <= 0) return cudaSuccess;
    return launch_overlapped(kern, ntiles, 128, smem, st, bs.overlap(), slots, work, bs, dp);
}

// FP32-bulk per-N shapes at 2, 3 and 10 points: the first family's tile, the single-mesh
// default there.
template <int N> struct NShape;
template <> struct NShape<2> { static constexpr int KS = 2, EPB = 16, KSM = 1, MINB = 1; };
template <> struct NShape<3> { static constexpr int KS = 1, EPB = 16, KSM = 0, MINB = 4; };
template <> struct NShape<10> { static constexpr int KS = 2, EPB = 1, KSM = 0, MINB = 2; };

template <int N>
__global__ void __launch_bounds__(NShape<N>::EPB * NShape<N>::KS * N * N, NShape<N>::MINB)
batch_first_n_kernel(const SlotDev* __restrict__ slots, const WorkItem* __restrict__ work,
                     const __grid_constant__ BatchStage bs) {
    extern __shared__ __align__(16) unsigned char smem[];
    using Sh = NShape<N>;
    const WorkItem w = work[blockIdx.x];
    const SlotDev& S = slots[w.slot];
    stage::grid_launch_dependents();
    stage::grid_wait();
    if (!S.active) return;
    const StageParams P = slot_params(S, bs);
    stage_tile<N, GEO_BOX, true, Sh::KS, Sh::EPB, (Sh::KSM != 0), true>(P, w.e0, smem, threadIdx.x);
}

// FP64 per-N shapes: the single-mesh default at every N but 8, the bulk-copy one-tile form
// with the t-derivative's D from the parameters (CD of the kernels below) and neighbour
// traces requested while the tile's copies fly.  KSM: k staged in shared memory.  AHEAD = 1:
// each block pulls into L2 the tile of the block half a wave of resident blocks after it
// (PoolPull).  4 points: the four-thread form (NQuad) at every size.
template <int N> struct NBulk;
template <> struct NBulk<2> { static constexpr int EPB = 16, MINB = 4, KSM = 1, AHEAD = 0; };
template <> struct NBulk<3> { static constexpr int EPB = 8, MINB = 4, KSM = 1, AHEAD = 0; };
template <> struct NBulk<5> { static constexpr int EPB = 1, MINB = 8, KSM = 1, AHEAD = 0; };
template <> struct NBulk<6> { static constexpr int EPB = 2, MINB = 3, KSM = 1, AHEAD = 1; };
template <> struct NBulk<7> { static constexpr int EPB = 1, MINB = 4, KSM = 1, AHEAD = 0; };
template <> struct NBulk<9> { static constexpr int EPB = 1, MINB = 2, KSM = 1, AHEAD = 0; };
template <> struct NBulk<10> { static constexpr int EPB = 1, MINB = 2, KSM = 0, AHEAD = 0; };

// The four-threads-per-column form, for launches over few elements (NWB_SMALL): form 1.  Not at
// 8 points.
template <int N> struct NQuad { static constexpr int EPB = 1, MINB = 2, KSM = 1; };
template <> struct NQuad<2> { static constexpr int EPB = 8, MINB = 4, KSM = 1; };
template <> struct NQuad<3> { static constexpr int EPB = 2, MINB = 8, KSM = 1; };
template <> struct NQuad<4> { static constexpr int EPB = 2, MINB = 8, KSM = 1; };
template <> struct NQuad<5> { static constexpr int EPB = 1, MINB = 6, KSM = 1; };
template <> struct NQuad<9> { static constexpr int EPB = 1, MINB = 1, KSM = 1; };
template <> struct NQuad<10> { static constexpr int EPB = 1, MINB = 1, KSM = 0; };

// Thread 0's L2 pull in a per-N bulk kernel: the tile of the work item about AHEAD/2
// waves of resident blocks after this block's (that N's tiles are the grid, one per
// block, in work-list order), in whichever cavity it lies.
template <int N>
struct PoolPull {
    const SlotDev* slots;
    const WorkItem* work;
    int stage;
    __device__ __forceinline__ void operator()() const {
        const int b = stage::tile_ahead<NBulk<N>::AHEAD, NBulk<N>::MINB>(blockIdx.x);
        if (b < 0) return;
        const WorkItem w = work[b];
        const SlotDev& S = slots[w.slot];
        if (!S.active) return;
        constexpr long long N3 = N * N * N;
        stage::prefetch_nodes_l2(S.u[S.par ^ (stage & 1)], S.k, S.stride, w.e0 * N3,
                                 min(NBulk<N>::EPB, S.nelt - w.e0) * N3, stage_kio(stage));
    }
};

template <int N, int EPB, int MINB, bool KSM, bool PULL, bool CD, int KIO>
__global__ void __launch_bounds__(EPB * 2 * N * N, MINB)
batch_bulk_n_kernel(const SlotDev* __restrict__ slots, const WorkItem* __restrict__ work,
                    const __grid_constant__ BatchStage bs, const __grid_constant__ DParam dp) {
    extern __shared__ __align__(16) unsigned char smem[];
    const WorkItem w = work[blockIdx.x];
    const SlotDev& S = slots[w.slot];
    if (!S.active) {
        stage::grid_wait();
        return;
    }
    const StageParams P = slot_params(S, bs);
    if constexpr (PULL)
        stage::bulk_tile<N, GEO_BOX, 2, EPB, CD, false, KSM, true, false, false, false, KIO>(
            P, w.e0, smem, threadIdx.x, dp.d, PoolPull<N>{slots, work, bs.stage});
    else
        stage::bulk_tile<N, GEO_BOX, 2, EPB, CD, false, KSM, true, false, false, false, KIO>(P, w.e0, smem, threadIdx.x,
                                                                                             dp.d);
}

template <int N, int EPB, int MINB, bool KSM, bool CD>
__global__ void __launch_bounds__(stage::Quad<N, EPB>::threads, MINB)
batch_quad_n_kernel(const SlotDev* __restrict__ slots, const WorkItem* __restrict__ work,
                    const __grid_constant__ BatchStage bs, const __grid_constant__ DParam dp) {
    extern __shared__ __align__(16) unsigned char smem[];
    const WorkItem w = work[blockIdx.x];
    const SlotDev& S = slots[w.slot];
    if (!S.active) {
        stage::grid_wait();
        return;
    }
    const StageParams P = slot_params(S, bs);
    stage::quad_tile<N, EPB, KSM, CD>(P, w.e0, smem, threadIdx.x, dp.d);
}

template <int N, int EPB, bool KSM, class K>
cudaError_t launch_tiles(K kern, int threads, std::atomic<int>* attr_set, const BatchStage& bs, const SlotDev* slots,
                         const WorkItem* work, int ntiles, const DParam& dp, cudaStream_t st) {
    constexpr int smem = stage::BulkLayout<N, EPB, KSM>::total;
    if (cudaError_t e = set_smem_once(kern, smem, attr_set); e != cudaSuccess) return e;
    if (ntiles <= 0) return cudaSuccess;
    return launch_overlapped(kern, ntiles, threads, smem, st, bs.overlap(), slots, work, bs, dp);
}

template <int N, int EPB, int MINB, bool KSM, bool PULL, bool CD, int KIO>
cudaError_t launch_bulk_kio(const BatchStage& bs, const SlotDev* slots, const WorkItem* work, int ntiles,
                            const DParam& dp, cudaStream_t st) {
    static std::atomic<int> attr_set[kMaxDeviceSlots];  // per kernel and device
    return launch_tiles<N, EPB, KSM>(batch_bulk_n_kernel<N, EPB, MINB, KSM, PULL, CD, KIO>, EPB * 2 * N * N, attr_set,
                                     bs, slots, work, ntiles, dp, st);
}

// A kernel of its own for the first, the inner and the last stage, as in launch_bulk; without
// the parameters' D (CD), a rare pool, one that tests at run time.
template <int N, int EPB, int MINB, bool KSM, bool PULL, bool CD>
cudaError_t launch_bulk_n(const BatchStage& bs, const SlotDev* slots, const WorkItem* work, int ntiles,
                          const DParam& dp, cudaStream_t st) {
#define NWB_KIO(x) launch_bulk_kio<N, EPB, MINB, KSM, PULL, CD, x>(bs, slots, work, ntiles, dp, st)
    if constexpr (!CD) return NWB_KIO(0);
    else {
        if (ntiles > 0) {
            switch (stage_kio(bs.stage)) {
                case kKWrite: return NWB_KIO(kKWrite);
                case kKRead: return NWB_KIO(kKRead);
                default: return NWB_KIO(kKRead | kKWrite);
            }
        }
        cudaError_t e = NWB_KIO(kKWrite);
        if (e == cudaSuccess) e = NWB_KIO(kKRead);
        if (e == cudaSuccess) e = NWB_KIO(kKRead | kKWrite);
        return e;
    }
#undef NWB_KIO
}

template <int N, bool CD>
cudaError_t launch_quad_n(const BatchStage& bs, const SlotDev* slots, const WorkItem* work, int ntiles,
                          const DParam& dp, cudaStream_t st) {
    using Q = NQuad<N>;
    static std::atomic<int> attr_set[kMaxDeviceSlots];  // per kernel and device
    return launch_tiles<N, Q::EPB, Q::KSM != 0>(batch_quad_n_kernel<N, Q::EPB, Q::MINB, Q::KSM != 0, CD>,
                                                stage::Quad<N, Q::EPB>::threads, attr_set, bs, slots, work, ntiles,
                                                dp, st);
}

// The form of a per-N launch (batch_form_n): 0 large, 1 four threads per column, 2 (6 points)
// one element per block.  4 and 8 points have one form.
template <int N, bool CD>
cudaError_t launch_form_n(int form, const BatchStage& bs, const SlotDev* slots, const WorkItem* work, int ntiles,
                          const DParam& dp, cudaStream_t st) {
    if constexpr (N == 4) return launch_quad_n<N, CD>(bs, slots, work, ntiles, dp, st);
    else if constexpr (N == 8) return launch_dmma8_n<CD>(bs, slots, work, ntiles, dp, st);
    else {
        if (form == 1) return launch_quad_n<N, CD>(bs, slots, work, ntiles, dp, st);
        if constexpr (N == 6)
            if (form == 2) return launch_bulk_n<N, 1, 5, true, false, CD>(bs, slots, work, ntiles, dp, st);
        using B = NBulk<N>;
        return launch_bulk_n<N, B::EPB, B::MINB, B::KSM != 0, (B::AHEAD > 0), CD>(bs, slots, work, ntiles, dp, st);
    }
}

// FP32-bulk, per-N mode: the single-mesh form (stage::F32Shape), D from dp (CD) or from
// shared memory.
template <int N, bool CD>
__global__ void __launch_bounds__(stage::F32Shape<N>::EPB * 2 * N * N, stage::F32Shape<N>::MINB)
batch_f32_n_kernel(const SlotDev* __restrict__ slots, const WorkItem* __restrict__ work,
                   const __grid_constant__ BatchStage bs, const __grid_constant__ DParam dp) {
    extern __shared__ __align__(16) unsigned char smem[];
    using Sh = stage::F32Shape<N>;
    const WorkItem w = work[blockIdx.x];
    const SlotDev& S = slots[w.slot];
    if (!S.active) {
        stage::grid_wait();
        return;
    }
    const StageParams P = slot_params(S, bs);
    stage::bulk_tile<N, GEO_BOX, 2, Sh::EPB, CD && Sh::CD != 0, false, Sh::KSM != 0, true, false, false, true>(
        P, w.e0, smem, threadIdx.x, dp.d, stage::NoPull(), dp.f);
}

template <int N, bool CD>
cudaError_t launch_f32_n(const BatchStage& bs, const SlotDev* slots, const WorkItem* work, int ntiles,
                         const DParam& dp, cudaStream_t st) {
    using Sh = stage::F32Shape<N>;
    constexpr int smem = stage::BulkLayout<N, Sh::EPB, Sh::KSM != 0, GEO_BOX, true>::total;
    auto kern = batch_f32_n_kernel<N, CD>;
    static std::atomic<int> attr_set[kMaxDeviceSlots];  // per kernel and device
    if (cudaError_t e = set_smem_once(kern, smem, attr_set); e != cudaSuccess) return e;
    if (ntiles <= 0) return cudaSuccess;
    return launch_overlapped(kern, ntiles, Sh::EPB * 2 * N * N, smem, st, bs.overlap(), slots, work, bs, dp);
}

template <int N>
cudaError_t launch_n_first(const BatchStage& bs, const SlotDev* slots, const WorkItem* work, int ntiles,
                           cudaStream_t st) {
    using Sh = NShape<N>;
    constexpr int threads = Sh::EPB * Sh::KS * N * N;
    constexpr int smem = SmemLayout<N, true, Sh::EPB, (Sh::KSM != 0)>::total;
    auto kern = batch_first_n_kernel<N>;
    static std::atomic<int> attr_set[kMaxDeviceSlots];  // per kernel and device
    if (cudaError_t e = set_smem_once(kern, smem, attr_set); e != cudaSuccess) return e;
    if (ntiles <= 0) return cudaSuccess;
    return launch_overlapped(kern, ntiles, threads, smem, st, bs.overlap(), slots, work, bs);
}

// Dh: this N's D on the host when every resident cavity of this N uses it (the
// constant-bank form then applies), else null.
template <int N, bool F32>
cudaError_t launch_n(int form, const BatchStage& bs, const SlotDev* slots, const WorkItem* work, int ntiles,
                     const double* Dh, cudaStream_t st) {
    if constexpr (stage::F32Shape<N>::on && F32) {
        const DParam dp = d_param(N, Dh);
        if (Dh) return launch_f32_n<N, true>(bs, slots, work, ntiles, dp, st);
        if (ntiles <= 0) {  // set-up call: prepare both forms
            cudaError_t e = launch_f32_n<N, true>(bs, slots, work, 0, dp, st);
            if (e != cudaSuccess) return e;
        }
        return launch_f32_n<N, false>(bs, slots, work, ntiles, dp, st);
    } else if constexpr (F32) {
        return launch_n_first<N>(bs, slots, work, ntiles, st);
    } else {
        const DParam dp = d_param(N, Dh);
        if (ntiles <= 0) {  // set-up call: prepare every form
            for (int f = 0; f < kBatchForms; ++f) {
                cudaError_t e = launch_form_n<N, true>(f, bs, slots, work, 0, dp, st);
                if (e == cudaSuccess) e = launch_form_n<N, false>(f, bs, slots, work, 0, dp, st);
                if (e != cudaSuccess) return e;
            }
            return cudaSuccess;
        }
        return Dh ? launch_form_n<N, true>(form, bs, slots, work, ntiles, dp, st)
                  : launch_form_n<N, false>(form, bs, slots, work, ntiles, dp, st);
    }
}

// The stage of the slots whose metrics are diagonal and whose normals are not along the axes
// (arrays of a user's own: no mesher makes them).  The axis-aligned class's tiles take the
// normals for granted, so these slots have the first family's general tile, in FP64 in both
// precisions.  Launched only where an order has such a slot.
template <int N>
__global__ void __launch_bounds__(kBatchThreads)
batch_oblique_kernel(const SlotDev* __restrict__ slots, const WorkItem* __restrict__ work,
                     const __grid_constant__ BatchStage bs) {
    extern __shared__ __align__(16) unsigned char smem[];
    using B = BShape<N>;
    const WorkItem w = work[blockIdx.x];
    const SlotDev& S = slots[w.slot];
    if (!S.active || !S.oblique) return;
    const StageParams P = slot_params(S, bs);
    stage_tile<N, GEO_AFFINE, false, B::KS, B::EPB, false, false>(P, w.e0, smem, threadIdx.x);
}

template <int N>
cudaError_t launch_oblique_n(const BatchStage& bs, const SlotDev* slots, const WorkItem* work, int ntiles,
                             cudaStream_t st) {
    constexpr int smem = SmemLayout<N, false, BShape<N>::EPB, false>::total;
    auto kern = batch_oblique_kernel<N>;
    static std::atomic<int> attr_set[kMaxDeviceSlots];  // per kernel and device
    if (cudaError_t e = set_smem_once(kern, smem, attr_set); e != cudaSuccess) return e;
    if (ntiles <= 0) return cudaSuccess;
    return launch_overlapped(kern, ntiles, kBatchThreads, smem, st, false, slots, work, bs);
}

// Does this slot record energy after the step it is taking now (post = 1), or
// is this the initial-state record (post = 0)?
__device__ __forceinline__ bool wants_energy(const SlotDev& S, int post) {
    if (!post) return true;
    const int next = S.done + 1;
    return (next % S.energy_every) == 0 || next == S.nsteps;
}

// Energy partial of each tile, fixed order within the tile.
__global__ void __launch_bounds__(256)
batch_diag_kernel(const SlotDev* __restrict__ slots, const WorkItem* __restrict__ work, int ntiles_v,
                  const int* __restrict__ ntiles_p, int post) {
    stage::grid_launch_dependents();
    stage::grid_wait();
    const int ntiles = ntiles_p ? *ntiles_p : ntiles_v;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int t = blockIdx.x * 8 + warp; t < ntiles; t += gridDim.x * 8) {
        const WorkItem w = work[t];
        const SlotDev& S = slots[w.slot];
        if (!(S.active || !post) || !wants_energy(S, post)) continue;
        const double* u = S.u[post ? (S.par ^ 1) : S.par];
        const int N3 = S.N * S.N * S.N;
        const int e1 = min(S.nelt, w.e0 + S.epb);
        double acc = 0.0;
        for (int e = w.e0; e < e1; ++e) {
            const double J = S.geo[e].jdet;
            const long long base = static_cast<long long>(e) * N3;
            for (int m = lane; m < N3; m += 32) {
                const long long p = base + m;
                const long long st = S.stride;
                const double ex = u[p], ey = u[st + p], ez = u[2 * st + p];
                const double hx = u[3 * st + p], hy = u[4 * st + p], hz = u[5 * st + p];
                acc += 0.5 * ((ex * ex + ey * ey + ez * ez) + (hx * hx + hy * hy + hz * hz)) *
                       (J * S.w3[m]);
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
        if (lane == 0) S.partial[w.tile] = acc;
    }
}

// One block per slot: warp 0 sums the energy partials in a fixed order, warps
// 1..kMaxProbes evaluate the probes (tensor-product Lagrange interpolation of
// the element's nodes, as ProbeManager::record does on the host,
// src/probe.cpp:192-216), then thread 0 advances the slot's step bookkeeping.
__global__ void __launch_bounds__(32 * (kMaxProbes + 1))
batch_epilogue_kernel(SlotDev* __restrict__ slots, const int* __restrict__ slot_list, int first_slot, int post,
                      int* __restrict__ counters) {
    stage::grid_wait();
    if (blockIdx.x == 0 && threadIdx.x < 8 && counters) counters[threadIdx.x] = 0;
    SlotDev& S = slots[slot_list ? slot_list[blockIdx.x] : first_slot + static_cast<int>(blockIdx.x)];
    if (post && !S.active) return;
    if (!post && !S.u[0]) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int idx = post ? S.done + 1 : 0;  // history index written by this call
    const double* u = S.u[post ? (S.par ^ 1) : S.par];
    if (warp == 0 && wants_energy(S, post)) {
        double acc = 0.0;
        for (int t = lane; t < S.ntiles; t += 32) acc += S.partial[t];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
        if (lane == 0) S.energy[idx] = acc;
    } else if (warp == 0 && lane == 0) {
        S.energy[idx] = __longlong_as_double(0x7ff8000000000000LL);  // not recorded this step
    }
    if (warp >= 1 && warp - 1 < S.nprobes) {
        const int pr = warp - 1;
        const int N = S.N, N2 = N * N, N3 = N2 * N;
        const double* wr = S.probe_w + pr * 3 * N;
        const double* ws = wr + N;
        const double* wt = ws + N;
        const long long base = static_cast<long long>(S.probe_elem[pr]) * N3;
        double acc[6] = {0, 0, 0, 0, 0, 0};
        // four nodes of a lane in flight (one at a time the loop waited for L2 at each)
        const double* up = u + base;
        const long long st = S.stride;
        for (int m0 = lane; m0 < N3; m0 += 128) {
            double w[4], v[4][6];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int m = min(m0 + 32 * q, N3 - 1);
                const int i = m % N, j = (m / N) % N, k = m / N2;
                w[q] = wr[i] * ws[j] * wt[k];
#pragma unroll
                for (int c = 0; c < 6; ++c) v[q][c] = stage::ld_state(up + c * st + m);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (m0 + 32 * q < N3) {
#pragma unroll
                    for (int c = 0; c < 6; ++c) acc[c] += w[q] * v[q][c];
                }
        }
#pragma unroll
        for (int c = 0; c < 6; ++c) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) acc[c] += __shfl_down_sync(0xffffffffu, acc[c], off);
        }
        if (lane == 0) {
            double* out = S.probes + (static_cast<long long>(idx) * S.nprobes + pr) * 6;
#pragma unroll
            for (int c = 0; c < 6; ++c) out[c] = acc[c];
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && post) {
        S.par ^= 1;
        S.done += 1;
        if (S.done >= S.nsteps) S.active = 0;
    }
}

template <bool F32>
int max_batch_smem() {
    int m = 0;
    m = max(m, bsmem<2, F32>()); m = max(m, bsmem<3, F32>()); m = max(m, bsmem<4, F32>());
    m = max(m, bsmem<5, F32>()); m = max(m, bsmem<6, F32>()); m = max(m, bsmem<7, F32>());
    m = max(m, bsmem<8, F32>()); m = max(m, bsmem<9, F32>()); m = max(m, bsmem<10, F32>());
    return m;
}

}  // namespace

cudaError_t launch_batch_stage_n(int N, int f32, int form, int stage, const SlotDev* slots,
                                 const WorkItem* work, int ntiles, int dry, const double* Dh, int* err,
                                 cudaStream_t st) {
    const BatchStage bs{dry ? 0.0 : kRk4a[stage], dry ? 0.0 : kRk4b[stage], stage, dry, err};
    switch (N) {
#define NWB_CASE(n) \
        case n: return f32 ? launch_n<n, true>(form, bs, slots, work, ntiles, Dh, st) \
                           : launch_n<n, false>(form, bs, slots, work, ntiles, Dh, st);
        NWB_CASE(2) NWB_CASE(3) NWB_CASE(4) NWB_CASE(5) NWB_CASE(6) NWB_CASE(7) NWB_CASE(8)
        NWB_CASE(9) NWB_CASE(10)
#undef NWB_CASE
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_batch_oblique(int N, int stage, const SlotDev* slots, const WorkItem* work, int ntiles, int dry,
                                 cudaStream_t st) {
    const BatchStage bs{dry ? 0.0 : kRk4a[stage], dry ? 0.0 : kRk4b[stage], stage, dry, nullptr};
    switch (N) {
#define NWB_CASE(n) case n: return launch_oblique_n<n>(bs, slots, work, ntiles, st);
        NWB_CASE(2) NWB_CASE(3) NWB_CASE(4) NWB_CASE(5) NWB_CASE(6) NWB_CASE(7) NWB_CASE(8)
        NWB_CASE(9) NWB_CASE(10)
#undef NWB_CASE
        default: return cudaErrorInvalidValue;
    }
}

namespace {
template <int N>
int epb_n(int f32, int form) {
    if (f32) {
        if constexpr (stage::F32Shape<N>::on) return stage::F32Shape<N>::EPB;
        else return NShape<N>::EPB;
    }
    if constexpr (N == 4) return NQuad<N>::EPB;
    else if constexpr (N == 8) return 1;
    else return form == 1 ? NQuad<N>::EPB : form == 2 ? 1 : NBulk<N>::EPB;
}
}  // namespace

int batch_form_n(int N, int f32, long long nelt) {
    if (f32) return 0;
#define NWB_X(n, i) if (nelt <= (n)) return form; ++form;
    int form = 1;
    switch (N) {
#define NWB_CASE(k) case k: { NWB_SMALL_##k(NWB_X) break; }
        NWB_CASE(2) NWB_CASE(3) NWB_CASE(4) NWB_CASE(5) NWB_CASE(6) NWB_CASE(7) NWB_CASE(8) NWB_CASE(9) NWB_CASE(10)
#undef NWB_CASE
        default: break;
    }
#undef NWB_X
    return 0;
}

int batch_epb_n(int N, int f32, int form) {
    switch (N) {
        case 2: return epb_n<2>(f32, form); case 3: return epb_n<3>(f32, form); case 4: return epb_n<4>(f32, form);
        case 5: return epb_n<5>(f32, form); case 6: return epb_n<6>(f32, form); case 7: return epb_n<7>(f32, form);
        case 8: return epb_n<8>(f32, form); case 9: return epb_n<9>(f32, form); case 10: return epb_n<10>(f32, form);
        default: return 1;
    }
}

BatchShape batch_shape(int N, int f32) {
    (void)f32;
    switch (N) {
        case 2: return {BShape<2>::KS, BShape<2>::EPB};
        case 3: return {BShape<3>::KS, BShape<3>::EPB};
        case 4: return {BShape<4>::KS, BShape<4>::EPB};
        case 5: return {BShape<5>::KS, BShape<5>::EPB};
        case 6: return {BShape<6>::KS, BShape<6>::EPB};
        case 7: return {BShape<7>::KS, BShape<7>::EPB};
        case 8: return {BShape<8>::KS, BShape<8>::EPB};
        case 9: return {BShape<9>::KS, BShape<9>::EPB};
        case 10: return {BShape<10>::KS, BShape<10>::EPB};
        default: return {0, 0};
    }
}

int batch_smem(int N, int f32) {
    switch (N) {
        case 2: return f32 ? bsmem<2, true>() : bsmem<2, false>();
        case 3: return f32 ? bsmem<3, true>() : bsmem<3, false>();
        case 4: return f32 ? bsmem<4, true>() : bsmem<4, false>();
        case 5: return f32 ? bsmem<5, true>() : bsmem<5, false>();
        case 6: return f32 ? bsmem<6, true>() : bsmem<6, false>();
        case 7: return f32 ? bsmem<7, true>() : bsmem<7, false>();
        case 8: return f32 ? bsmem<8, true>() : bsmem<8, false>();
        case 9: return f32 ? bsmem<9, true>() : bsmem<9, false>();
        case 10: return f32 ? bsmem<10, true>() : bsmem<10, false>();
        default: return 0;
    }
}

cudaError_t batch_prepare(int f32, int smem) {
    const int cap = f32 ? max_batch_smem<true>() : max_batch_smem<false>();
    if (smem > cap) smem = cap;
    return f32 ? cudaFuncSetAttribute(batch_stage_kernel<true>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, cap)
               : cudaFuncSetAttribute(batch_stage_kernel<false>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
}

cudaError_t launch_batch_stage(int f32, int stage, const SlotDev* slots, const WorkItem* work,
                               const int* ntiles, int* counters, int grid, int smem, int dry,
                               cudaStream_t st) {
    if (f32)
        batch_stage_kernel<true><<<grid, kBatchThreads, smem, st>>>(slots, work, ntiles, counters, stage, dry);
    else
        batch_stage_kernel<false><<<grid, kBatchThreads, smem, st>>>(slots, work, ntiles, counters, stage, dry);
    return cudaGetLastError();
}

cudaError_t launch_batch_diag(SlotDev* slots, const WorkItem* work, int ntiles, const int* ntiles_p, int post,
                              int grid, bool overlap, cudaStream_t st) {
    return launch_overlapped(batch_diag_kernel, grid, 256, 0, st, overlap, slots, work, ntiles, ntiles_p, post);
}

cudaError_t launch_batch_epilogue(SlotDev* slots, const int* slot_list, int first_slot, int nslots, int post,
                                  int* counters, bool overlap, cudaStream_t st) {
    if (nslots < 1) return cudaSuccess;
    return launch_overlapped(batch_epilogue_kernel, nslots, 32 * (kMaxProbes + 1), 0, st, overlap, slots, slot_list,
                             first_slot, post, counters);
}

}  // namespace nwb
