// stage_bulk.cuh -- the second-family stage kernel with its tile loaded by the
// bulk-copy engine (FP64; axis-aligned and affine classes).
//
// One block per tile.  Thread 0 issues the tile's u_in, its LSRK register k,
// the per-element geometry and the connections as a dozen cp.async.bulk copies
// (plain copies from this GPU's own memory, no multicast) that complete on one
// mbarrier by byte count; every thread waits for them, then compute2 runs the
// face and column phases as in the other one-tile forms, with k read from
// shared memory.  Against the per-thread cp.async loads of those forms this
// takes a few hundred load instructions per block off the issue slots, and the
// column phase no longer waits on L2 for each plane's k.  It is the FP64 default of
// the axis-aligned class but at 4 points (four threads per column) and 8 (tensor-core
// tile), and carries the general classes and FP32-bulk from 4 points up
// (stage_variants.h, GeneralShape and F32Shape have the figures).
//
// Bulk copies start and end on 16-byte boundaries.  A tile whose first node or
// length is odd (odd N) is copied from the boundary at or below its first value
// to the one at or above its last (at most one double more at either end, inside
// the state arrays: components are 512-byte aligned and rounded up to 64
// doubles) into a component slot with two doubles of slack, and read from
// offset (first node & 1).  Connections are copied the same way (the solver pads
// its connection table to a multiple of four entries; a pool cavity's table
// lies in a 256-byte-rounded range of its arena), and D (N^2 doubles, rounded up to 16
// bytes) likewise.
//
// The wait is bounded (kWaitNs of the global timer, about a thousand times a
// normal stage).  When it expires the block records a code in *P.err (when the
// caller keeps one), waits once more, bounded, for its copies, and returns.
#pragma once
#include "stage_pipe.cuh"

#include <cstdint>

namespace nwb {
namespace stage {

constexpr unsigned long long kWaitNs = 1000000000ull;  // 1 s
constexpr int kErrTileWait = 1;  // a block's wait for its tile expired

__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for the phase of the given parity to complete; false when kWaitNs pass first.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
    if (mbar_test(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (;;) {
        for (int k = 0; k < 32; ++k)
            if (mbar_test(bar, parity)) return true;
        if (global_ns() - t0 > kWaitNs) return false;
    }
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void bulk_prefetch_l2(const void* src, unsigned bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void report(const StageParams& P, int code) {
    if (P.err) *reinterpret_cast<volatile int*>(P.err) = code;
}

// Shared-memory layout of one tile: u_in (and with KSM k) [6][CSR] doubles with
// slack, geometry, connections, D, the lifted fluxes, the mbarrier and a flag.
template <int N, int EPB, bool KSM, int GEO = GEO_BOX, bool F32 = false>
struct BulkLayout {
    static constexpr int N2 = N * N, N3 = N2 * N;
    static constexpr int CSR = (EPB * N3 + 2 + 1) / 2 * 2;
    static constexpr int tile_u = 6 * CSR * 8;
    static constexpr int u0 = 0;
    static constexpr int k0 = u0 + tile_u;
    static constexpr int geo0 = k0 + (KSM ? tile_u : 0);
    static constexpr int geo_b = GEO == GEO_NODAL ? 0 : EPB * static_cast<int>(sizeof(ElemGeo));
    static constexpr int conn0 = geo0 + geo_b;
    static constexpr int conn_b = align16((EPB * 6 + 6) * 4);
    static constexpr int D = conn0 + conn_b;
    static constexpr int flux0 = D + align16(N2 * 8);
    // FP32-bulk: the deviations, the fit and the maxima (as Layout2::uc)
    static constexpr int uc = flux0 + EPB * flux_planes<GEO, true>() * N2 * 8;
    static constexpr int bar = uc + (F32 ? align16(6 * CSR * 4) + align16((EPB * 30 + 10) * 8) + align16(EPB * 8) : 0);
    static constexpr int flag = bar + 8;
    static constexpr int total = flag + 16;
};

// Thread 0's part of a tile load: the tile's u_in (and with KSM its k; otherwise k's
// lines are prefetched into L2), geometry and connections as bulk copies that
// complete on the mbarrier at smem + L::bar, which must be initialised.  Waits for the
// launches before this one (grid_wait) ahead of the first access to u and k.
template <int N, int EPB, bool KSM, int GEO, bool F32>
__device__ __forceinline__ void bulk_issue(const StageParams& P, const int e0, unsigned char* smem) {
    using L = BulkLayout<N, EPB, KSM, GEO, F32>;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::bar);
    const long long S = P.stride;
    const long long g0 = static_cast<long long>(e0) * L::N3;
    const int nvalid = min(EPB, P.nelt - e0);
    const long long a0 = g0 & ~1ll, a1 = (g0 + static_cast<long long>(nvalid) * L::N3 + 1) & ~1ll;
    const unsigned ub = static_cast<unsigned>((a1 - a0) * 8);
    const long long c0 = static_cast<long long>(e0) * 6, c1 = c0 + 6 * nvalid;
    const long long ca0 = c0 & ~3ll, ca1 = (c1 + 3) & ~3ll;
    const unsigned cb = static_cast<unsigned>((ca1 - ca0) * 4);
    const unsigned gb = static_cast<unsigned>(nvalid * sizeof(ElemGeo));
    const bool kread = (P.kio & kKRead) != 0;
    constexpr unsigned db = (L::N2 * 8 + 15) / 16 * 16;  // D, to the 16-byte boundary (its array is padded)
    mbar_arrive_expect_tx(bar, (KSM && kread ? 12 : 6) * ub + db + (GEO == GEO_NODAL ? 0 : gb + cb));
    // constant data before grid_wait()
    bulk_g2s(smem + L::D, P.D, db, bar);
    if constexpr (GEO == GEO_NODAL) {
        // the column phase reads the metrics plane by plane: into L2 meanwhile
#pragma unroll
        for (int c = 0; c < 9; ++c) bulk_prefetch_l2(P.met_n + c * S + a0, ub);
    } else {
        bulk_g2s(smem + L::geo0, P.geo + e0, gb, bar);
        bulk_g2s(smem + L::conn0, P.conn + ca0, cb, bar);
    }
    grid_wait();
    double* su = reinterpret_cast<double*>(smem + L::u0);
#pragma unroll
    for (int c = 0; c < 6; ++c) bulk_g2s(su + c * L::CSR, P.u_in + c * S + a0, ub, bar);
    if (!kread) {
        // the first stage of a step: no k
    } else if constexpr (KSM) {
        double* sk = reinterpret_cast<double*>(smem + L::k0);
#pragma unroll
        for (int c = 0; c < 6; ++c) bulk_g2s(sk + c * L::CSR, P.k + c * S + a0, ub, bar);
    } else {
#pragma unroll
        for (int c = 0; c < 6; ++c) bulk_prefetch_l2(P.k + c * S + a0, ub);
    }
}

// Every thread's wait for the tile issued by bulk_issue: true when it is resident.
// On expiry thread 0 records the code, waits once more (bounded) for the copies so
// that none lands in a finished block, and every thread gets false.
template <int N, int EPB, bool KSM, int GEO, bool F32>
__device__ __forceinline__ bool bulk_wait_tile(const StageParams& P, unsigned char* smem, const int tid) {
    using L = BulkLayout<N, EPB, KSM, GEO, F32>;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::bar);
    int* flag = reinterpret_cast<int*>(smem + L::flag);
    if (tid == 0) *flag = mbar_wait(bar, 0) ? 1 : 0;
    __syncthreads();
    if (!*flag) {
        if (tid == 0) {
            report(P, kErrTileWait);
            mbar_wait(bar, 0);
        }
        return false;
    }
    mbar_test(bar, 0);  // the phase is complete: acquire the tile for this thread
    return true;
}

// One tile of the bulk-copy one-tile form, for the single-mesh kernel below and
// the pool's per-N kernels.  All NT = EPB*KS*N*N threads of the block call it.
// EARLY: the neighbour traces of the face phase are requested from global memory
// (through the box structure when there is one) while the tile's copies are in
// flight.  VROW: the r-derivative's node rows read with 16-byte loads.  Dc: D where
// the t contraction of CONSTD reads it (a parameter copy).  pull: called by thread 0
// right after it has issued the tile's copies (NoPull, or a functor that pulls a
// later block's tile into L2).
template <int N, int GEO, int KS, int EPB, bool CONSTD, bool DSMEM, bool KSM, bool EARLY,
          bool VROW = false, bool ILP2 = false, bool F32 = false, int KIO = 0, class Pull = NoPull>
__device__ __forceinline__ void bulk_tile(const StageParams& P, const int e0, unsigned char* smem,
                                          const int tid, const double* Dc, const Pull& pull = Pull(),
                                          const float* Dcf = nullptr) {
    using L = BulkLayout<N, EPB, KSM, GEO, F32>;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::bar);
    double* sD = reinterpret_cast<double*>(smem + L::D);
    grid_launch_dependents();
    // the copies first (a block of a large grid waits for nothing before them): only
    // thread 0 touches the mbarrier before the block's next barrier
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
        bulk_issue<N, EPB, KSM, GEO, F32>(P, e0, smem);
        pull();
    }
    const long long g0 = static_cast<long long>(e0) * L::N3;
    FaceRegs<N, GEO, KS, true> G;
    if constexpr (EARLY && GEO == GEO_BOX) gather_box_nodes<N, KS, EPB, false>(P, e0, nullptr, tid, G);
    if constexpr (EARLY && GEO != GEO_BOX) gather2<N, GEO, KS, EPB, false, false>(P, e0, nullptr, nullptr, tid, G);
    grid_wait();
    if constexpr (EARLY && GEO == GEO_BOX) gather_box_values<N, KS, EPB, false, false>(P, e0, nullptr, tid, G);
    if (!bulk_wait_tile<N, EPB, KSM, GEO, F32>(P, smem, tid)) return;
    const int off = static_cast<int>(g0 & 1);
    const double* su = reinterpret_cast<const double*>(smem + L::u0) + off;
    const double* sk = KSM ? reinterpret_cast<const double*>(smem + L::k0) + off : nullptr;
    const ElemGeo* sg = reinterpret_cast<const ElemGeo*>(smem + L::geo0);
    const int* sc = reinterpret_cast<const int*>(smem + L::conn0) + ((e0 * 6) & 3);
    double* sflux = reinterpret_cast<double*>(smem + L::flux0);
    compute2<N, GEO, F32, KS, EPB, true, false, CONSTD, EARLY, false, DSMEM, CtaBar, L::CSR, KSM, VROW, ILP2, KIO>(
        P, e0, su, sg, sc, sD, sflux, smem + L::uc, tid, G, Dc, CtaBar(), sk, Dcf);
}

// Tile taken by block b.  ZCOL on a structured box whose rows hold whole tiles:
// blocks walk the tiles of one (x-tile, y) column through every z before the next
// column, so an element's z-neighbours (nx*ny elements away in memory) are
// loaded by blocks that run at about the same time and their shared face planes
// come from L2 instead of a second DRAM read.  Otherwise tiles in memory order.
template <int EPB, bool ZCOL>
__device__ __forceinline__ int bulk_tile_index(const StageParams& P, int b) {
    if constexpr (ZCOL) {
        const int nx = P.snel[0], ny = P.snel[1], nz = P.snel[2];
        if (nx > 0 && nx % EPB == 0) {
            const int col = b / nz, ez = b - col * nz;
            const int ntx = nx / EPB;
            const int ey = col / ntx, xt = col - ey * ntx;
            return xt + ntx * (ey + ny * ez);
        }
    }
    return b;
}

// Thread 0's L2 pull of the single-mesh kernel: the tile of the block that starts
// about AHEAD/2 waves of resident blocks after this one (tile_ahead), in the same
// tile order.
template <int N3, int EPB, int MINB, int AHEAD, bool ZCOL>
struct MeshPull {
    const StageParams& P;
    __device__ __forceinline__ void operator()() const {
        const int b = tile_ahead<AHEAD, MINB>(blockIdx.x);
        if (b < 0) return;
        const int e = bulk_tile_index<EPB, ZCOL>(P, b) * EPB;
        prefetch_tile_l2<N3>(P, e, min(EPB, P.nelt - e));
    }
};

// AHEAD (0, 1, 2): block b also pulls into L2 the tile of the block that starts
// about AHEAD/2 waves of resident blocks later, so that block's bulk copies read L2
// instead of DRAM; 0: no pull.  On B200 this pays at 6 points (3 resident blocks
// per SM, whose tile waits the other blocks hide least); at 9 points, with 2, it paid only
// while the faces kept the L1 pipe busy.
template <int N, int GEO, int KS, int EPB, int MINB, bool CONSTD, bool DSMEM, bool KSM, bool EARLY,
          bool ZCOL, bool VROW, bool ILP2, int AHEAD, bool F32, int KIO>
__global__ void __launch_bounds__(EPB * KS * N * N, MINB)
    stage_bulk_kernel(const __grid_constant__ StageParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int t = bulk_tile_index<EPB, ZCOL>(P, blockIdx.x);
    if constexpr (AHEAD > 0)
        bulk_tile<N, GEO, KS, EPB, CONSTD, DSMEM, KSM, EARLY, VROW, ILP2, F32, KIO>(
            P, t * EPB, smem, threadIdx.x, P.Dc, MeshPull<N * N * N, EPB, MINB, AHEAD, ZCOL>{P}, P.Dcf);
    else
        bulk_tile<N, GEO, KS, EPB, CONSTD, DSMEM, KSM, EARLY, VROW, ILP2, F32, KIO>(P, t * EPB, smem, threadIdx.x,
                                                                                   P.Dc, NoPull(), P.Dcf);
}

template <int N, int GEO, int KS, int EPB, int MINB, bool CONSTD, bool DSMEM, bool KSM, bool EARLY,
          bool ZCOL, bool VROW, bool ILP2, int AHEAD, bool F32, int KIO>
cudaError_t launch_bulk_kio(const StageParams* p, cudaStream_t st) {
    using L = BulkLayout<N, EPB, KSM, GEO, F32>;
    auto kern = stage_bulk_kernel<N, GEO, KS, EPB, MINB, CONSTD, DSMEM, KSM, EARLY, ZCOL, VROW, ILP2, AHEAD, F32, KIO>;
    static std::atomic<int> attr_set[kMaxDeviceSlots];  // per kernel and device
    if (cudaError_t e = set_smem_once(kern, L::total, attr_set); e != cudaSuccess) return e;
    if (!p) return cudaSuccess;
    return launch_overlapped(kern, (p->nelt + EPB - 1) / EPB, EPB * KS * N * N, L::total, st,
                             (p->kio & kOverlap) != 0, *p);
}

// SPEC: a kernel of its own for the first, the inner and the last stage of a step, without
// the tests on the register's accesses in the plane loop (the defaults; the other
// shapes test at run time).  B200, per step: 64x64x32 elements of 6 points 5393 -> 5260 us,
// 20^3 of 10 points 1806 -> 1782 us.
template <int N, int GEO, int KS, int EPB, int MINB, bool CONSTD, bool DSMEM, bool KSM, bool EARLY,
          bool ZCOL, bool VROW, bool ILP2, int AHEAD = 0, bool F32 = false, bool SPEC = false>
cudaError_t launch_bulk(const StageParams* p, cudaStream_t st, StageConfig* cfg) {
    using L = BulkLayout<N, EPB, KSM, GEO, F32>;
    if (cfg) *cfg = StageConfig{KS, EPB, EPB * KS * N * N, L::total, KSM ? 1 : 0, MINB};
#define NWB_KIO(x) launch_bulk_kio<N, GEO, KS, EPB, MINB, CONSTD, DSMEM, KSM, EARLY, ZCOL, VROW, ILP2, AHEAD, F32, x>(p, st)
    if constexpr (!SPEC) return NWB_KIO(0);
    else {
        if (p) {
            switch (p->kio & (kKRead | kKWrite)) {
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

// Shapes of the general classes (affine and per-node geometry) in FP64: the bulk-copy
// tile with the field split, k in shared memory and the face data requested while the
// copies fly.  Bound by latency and the shared pipe: three derivatives of three
// components per field (18 sums a node instead of 12) and, per node, nine metrics
// (72 B on top of the 192), which thread 0 pulls into L2 and the column phase requests
// one plane ahead.  MINB leaves the registers that takes; CD: t-derivative coefficients from
// the parameter bank with the plane loop unrolled (at 7 and 8 points only where the
// metrics do not need the registers, CDN / CDA).  From a sweep of four shapes per N
// on 1.5 to 1.7 M nodes.  B200, per step, before (per-thread copies, k and metrics
// read from L2 in the plane loop) -> now, per-node class: 17x15x19 elements of 6 points
// 572 -> 375 us, 26x26x24 of 4 points 504 -> 323 us, 12x13x12 of 8 points 452 -> 366 us;
// affine class, 16x16x12 of 8 points 449 -> 378 us.
template <int N> struct GeneralShape;
template <> struct GeneralShape<2> { static constexpr int EPB = 8, MINB = 6, CDN = 1, CDA = 1; };
template <> struct GeneralShape<3> { static constexpr int EPB = 8, MINB = 3, CDN = 1, CDA = 1; };
template <> struct GeneralShape<4> { static constexpr int EPB = 4, MINB = 3, CDN = 1, CDA = 1; };
template <> struct GeneralShape<5> { static constexpr int EPB = 1, MINB = 8, CDN = 1, CDA = 1; };
template <> struct GeneralShape<6> { static constexpr int EPB = 1, MINB = 4, CDN = 1, CDA = 1; };
template <> struct GeneralShape<7> { static constexpr int EPB = 1, MINB = 3, CDN = 0, CDA = 1; };
template <> struct GeneralShape<8> { static constexpr int EPB = 1, MINB = 3, CDN = 0, CDA = 1; };
template <> struct GeneralShape<9> { static constexpr int EPB = 1, MINB = 2, CDN = 1, CDA = 1; };
template <> struct GeneralShape<10> { static constexpr int EPB = 1, MINB = 1, CDN = 1, CDA = 1; };

template <int N, int GEO>
cudaError_t launch_general(const StageParams* p, cudaStream_t st, StageConfig* cfg) {
    using Sh = GeneralShape<N>;
    constexpr bool cd = (GEO == GEO_NODAL ? Sh::CDN : Sh::CDA) != 0;
    return launch_bulk<N, GEO, 2, Sh::EPB, Sh::MINB, cd, false, true, true, false, false, false, 0, false, true>(p, st,
                                                                                                               cfg);
}

// Shapes of the axis-aligned class in FP32-bulk at 4 to 9 points (on): the bulk-copy tile
// with the same arithmetic as before.  Beside u_in the tile holds its FP32 copy; the column
// phase's FP64 loop serves the elements that fall back, most of them in the benchmark's
// fields, so it takes its D rows in registers and (CD) the unrolled loop of the FP64 class
// (with its D rows read from shared memory at each use it did more than twice the shared
// loads of the FP64 class); at 8 points it is the tensor-core column phase of the FP64
// class.  k in shared memory (KSM) only at 5 points: elsewhere it costs a resident block.
// From a sweep of four shapes per N.  B200, per step, before -> now: 25^3 elements of 8 points
// 1917 -> 1406 us, 34^3 of 6 points 2452 -> 2019 us, 22^3 of 9 points 2631 -> 1750 us, 40^3 of 5
// points 2569 -> 2122 us.
template <int N> struct F32Shape { static constexpr bool on = false; static constexpr int EPB = 1, MINB = 1, KSM = 0, CD = 0; };
template <> struct F32Shape<4> { static constexpr bool on = true; static constexpr int EPB = 2, MINB = 8, KSM = 0, CD = 1; };
template <> struct F32Shape<5> { static constexpr bool on = true; static constexpr int EPB = 1, MINB = 8, KSM = 1, CD = 1; };
template <> struct F32Shape<6> { static constexpr bool on = true; static constexpr int EPB = 1, MINB = 5, KSM = 0, CD = 1; };
template <> struct F32Shape<7> { static constexpr bool on = true; static constexpr int EPB = 1, MINB = 4, KSM = 0, CD = 1; };
template <> struct F32Shape<8> { static constexpr bool on = true; static constexpr int EPB = 1, MINB = 4, KSM = 0, CD = 1; };
template <> struct F32Shape<9> { static constexpr bool on = true; static constexpr int EPB = 1, MINB = 2, KSM = 0, CD = 1; };

template <int N>
cudaError_t launch_f32(const StageParams* p, cudaStream_t st, StageConfig* cfg) {
    using Sh = F32Shape<N>;
    return launch_bulk<N, GEO_BOX, 2, Sh::EPB, Sh::MINB, Sh::CD != 0, false, Sh::KSM != 0, true, false, false, false, 0,
                       true, true>(p, st, cfg);
}

}  // namespace stage
}  // namespace nwb
