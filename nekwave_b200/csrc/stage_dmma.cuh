// stage_dmma.cuh -- fused LSRK45 stage for 8 points per direction, axis-aligned
// elements, FP64, with the r and s contractions on the FP64 tensor cores
// (mma.sync m8n8k4 f64) and the residual split by field between two warps.
//
// Why: in the SIMT forms every lane reads, for each r and s derivative it forms,
// the N values of a row or column from shared memory, and a 64-bit warp load costs
// two wavefronts however many lanes share an address; ncu shows those loads
// keeping the L1/shared pipe at 80-90 % at N = 8.  As an 8x8x8 product per plane
// and component, a warp reads each node value once per direction (one 64-bit
// fragment load per lane per k-step) and keeps D in two registers.  tcgen05 has no
// FP64 kind; mma.sync .f64 is sm_100a's FP64 tensor-core instruction.
//
// Block = one element, 128 threads = 2 warps per field:
//   1. cp.async of u_in (16-byte copies), D, geometry, connections; k lines of the
//      element into L2;
//   2. neighbour traces requested while the copies fly; face phase (face_phase_box:
//      faces 0..3 through shared memory); the faces across t belong to the lanes of the
//      column phase;
//   3. warps 0, 1 form the E residual from V = H (+curl H), warps 2, 3 the H residual
//      from V = E (-curl E), split by component: the first warp of a field forms its x
//      component on all planes and its z component on planes 0..3, the second its y
//      component and the z component on planes 4..7.  A warp then differentiates one
//      component along t (x needs Vy, y needs Vx, z none) and holds one pair of node
//      columns in registers instead of two: with planes split between the warps instead,
//      the tile sat at its limit of 128 registers and spilled, 4 blocks to an SM.
//      Lane 4g + t owns nodes (i = 2t, 2t+1; j = g) of every plane k.  The r derivatives
//      come in the original form (A = rows of the plane, B = D^T) and the s derivatives in
//      the swapped form (A = D, B = columns of the plane), which land on the same two
//      nodes; the t derivatives are SIMT sums over the lane's two node columns with
//      D(k,l) from the kernel's parameter bank.  Then the lifted face terms in face order
//      0..5 and the LSRK update in FP64, two adjacent nodes per 16-byte access; the
//      next plane's k is requested before this plane's stores.
//      B200, per step: 32^3 elements 2820 -> 2597 us (86 % of the measured copy rate), 512
//      elements 49.7 -> 47.1 us; 5 blocks to an SM are 2 % slower than 4, 3 the same.
#pragma once

#include "stage_pipe.cuh"

namespace nwb {
namespace stage {

struct DmmaLayout8 {
    static constexpr int u = 0;                                   // [6][512] doubles
    static constexpr int geo = u + 6 * 512 * 8;
    static constexpr int conn = geo + static_cast<int>(sizeof(ElemGeo));
    static constexpr int D = conn + 32;
    static constexpr int flux = D + 64 * 8;                       // [4 faces][4][64]
    // the faces across t: two lifted fluxes (one component at the lane's two nodes) per thread
    // and face
    static constexpr int zflux = flux + flux_planes<GEO_BOX, true>() * 64 * 8;
    static constexpr int total = zflux + 4 * 128 * 8;
};

// Values of components ca and cb across face f (4, 5) at the nodes (i, j) and (i+1, j) of
// element e, i even: 16-byte loads where the two are adjacent in memory.  zv: wall code
// where negative.
__device__ __forceinline__ void dmma8_z_gather(const StageParams& P, int e, int f, int i, int j, int ca, int cb,
                                               int& zv, double2 (&z)[2]) {
    const long long S = P.stride;
    int v0, v1;
    if (P.snel[0] > 0) {
        int ex, ey, ez;
        struct_coords(P, e, ex, ey, ez);
        const int eB = struct_neighbour(P, ex, ey, ez, e, f);
        v0 = eB < 0 ? kConnPEC : eB * 512 + face_local<8>(f == 4 ? 5 : 4, i, j);
        v1 = v0 + 1;
    } else {
        const int cd = __ldg(P.conn + e * 6 + f);
        v0 = conn_node<8>(cd, i, j);
        v1 = conn_node<8>(cd, i + 1, j);
    }
    zv = v0;
    if (v0 < 0) return;
    const bool pair = v1 == v0 + 1 && (v0 & 1) == 0;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const double* u = P.u_in + (c == 0 ? ca : cb) * S;
        z[c] = pair ? ld_state(reinterpret_cast<const double2*>(u + v0))
                    : make_double2(ld_state(u + v0), ld_state(u + v1));
    }
}

// One element.  Dc: D (column-major) where the t contraction reads it -- the
// kernel's parameter copy when the caller has one (constant-bank operands), else
// the tile's shared copy at smem + DmmaLayout8::D (the same values either way).
// All threads of the block call it.  e_ahead >= 0: thread 0 also pulls the u_in and k of
// that element into L2, for the block that loads it later.
__device__ __forceinline__ void dmma8_tile(const StageParams& P, const int e, unsigned char* smem,
                                           const int tid, const double* Dc, const int e_ahead = -1) {
    constexpr int N = 8, N3 = 512, NT = 128;
    using L = DmmaLayout8;
    double* su = reinterpret_cast<double*>(smem + L::u);
    ElemGeo* sg = reinterpret_cast<ElemGeo*>(smem + L::geo);
    int* sc = reinterpret_cast<int*>(smem + L::conn);
    double* sD = reinterpret_cast<double*>(smem + L::D);
    double* sflux = reinterpret_cast<double*>(smem + L::flux);

    grid_launch_dependents();
    if (tid < 64) cp_async8(sD + tid, P.D + tid);
    grid_wait();
    issue2<N, GEO_BOX, 1, NT, false>(P, e, su, sg, sc, tid);
    if (tid == 0 && e_ahead >= 0) prefetch_tile_l2<N3>(P, e_ahead, 1);
    cp_async_commit();

    const int warp = tid >> 5, lane = tid & 31;
    const int field = warp >> 1, role = warp & 1;
    const int g = lane >> 2, t = lane & 3;
    const int src = field == 0 ? 3 : 0;  // differentiated field
    const int dst = 3 - src;             // residual components formed
    // neighbour traces while the tile's copies fly: the thread's points of faces 0..3, and
    // of its two node columns across t.  The flux component x (role 0) takes the jumps of
    // D_x and S_y of the residual's own field D and the other S, y those of D_y and S_x.
    BoxFaces<box_points<2>()> G;
    gather_box_nodes<N, 2, 1, false, false>(P, e, nullptr, tid, G);
    gather_box_values<N, 2, 1, false, false, 0, false>(P, e, nullptr, tid, G);
    const int cd = dst + role, cs = src + 1 - role;
    double2 zn[2][2];
    int zv[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) dmma8_z_gather(P, e, 4 + s, 2 * t, g, cd, cs, zv[s], zn[s]);
    cp_async_wait<0>();
    __syncthreads();
    face_phase_box<N, false, 2, 1, false, true>(P, e, su, sg, sc, sflux, tid, G);
    // lifted fluxes of the lane's nodes on the faces across t (box_flux, one component), kept
    // in shared memory: the registers of the plane loop are all taken
    double2* zf = reinterpret_cast<double2*>(smem + L::zflux) + tid;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const int m = (s == 0 ? 0 : 448) + 8 * g + 2 * t;
        const double2 od = *reinterpret_cast<const double2*>(su + cd * N3 + m);
        const double2 os = *reinterpret_cast<const double2*>(su + cs * N3 + m);
        double2 jd, js;
        if (zv[s] >= 0) {
            jd = make_double2(zn[s][0].x - od.x, zn[s][0].y - od.y);
            js = make_double2(zn[s][1].x - os.x, zn[s][1].y - os.y);
        } else {
            // the mirror turns E at a PEC wall, H at a PMC wall
            const bool turns_d = (zv[s] == kConnPMC) == (field == 1);
            jd = turns_d ? make_double2(-2.0 * od.x, -2.0 * od.y) : make_double2(0.0, 0.0);
            js = turns_d ? make_double2(0.0, 0.0) : make_double2(-2.0 * os.x, -2.0 * os.y);
        }
        const double nd = sg->nrm[4 + s][2], lift = sg->lift[4 + s];
        const double hc = 0.5 * P.c0 * (nd * nd), hs = field == role ? -0.5 * nd : 0.5 * nd;
        zf[s * 128] = make_double2(lift * (hc * jd.x + hs * js.x), lift * (hc * jd.y + hs * js.y));
    }
    __syncthreads();

    const double sgn = field == 0 ? 1.0 : -1.0;
    const double* V = su + src * N3;
    const double d0 = sD[g + 8 * t];        // D(q = g, l = t)
    const double d1 = sD[g + 8 * (4 + t)];  // D(q = g, l = 4 + t)
    const double rx = sgn * sg->met[0], sy = sgn * sg->met[4], tz = sgn * sg->met[8];
    const long long ebase = static_cast<long long>(e) * N3;
    if (role == 0) dmma8_columns<0, N3>(P, su, V, sflux, g, t, dst, d0, d1, rx, sy, tz, ebase, Dc, zf, zf + 128);
    else dmma8_columns<1, N3>(P, su, V, sflux, g, t, dst, d0, d1, rx, sy, tz, ebase, Dc, zf, zf + 128);
}

// AHEAD (0, 1, 2): block e also pulls into L2 the element of the block that starts
// about AHEAD/2 waves of resident blocks later (tile_ahead); 0: no prefetch.
template <int MINB, int AHEAD>
__global__ void __launch_bounds__(128, MINB) stage_dmma8_kernel(const __grid_constant__ StageParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int e_ahead = AHEAD > 0 ? tile_ahead<(AHEAD > 0 ? AHEAD : 1), MINB>(blockIdx.x) : -1;
    dmma8_tile(P, blockIdx.x, smem, threadIdx.x, P.Dc, e_ahead);
}

template <int MINB, int AHEAD = 0>
cudaError_t launch_dmma8(const StageParams* p, cudaStream_t st, StageConfig* cfg) {
    constexpr int smem = DmmaLayout8::total;
    auto kern = stage_dmma8_kernel<MINB, AHEAD>;
    if (cfg) *cfg = StageConfig{2, 1, 128, smem, 0, MINB};
    static std::atomic<int> attr_set[kMaxDeviceSlots];  // per kernel and device
    if (cudaError_t e = set_smem_once(kern, smem, attr_set); e != cudaSuccess) return e;
    if (!p) return cudaSuccess;
    return launch_overlapped(kern, p->nelt, 128, smem, st, (p->kio & kOverlap) != 0, *p);
}

}  // namespace stage
}  // namespace nwb
