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
// Fragment layout (m8n8k4, A row-major 8x4, B column-major 4x8, C 8x8): lane
// L = 4g + t holds A[g][t], B[t][g], C[g][2t] and C[g][2t+1].
#pragma once

#include "stage_mma.cuh"
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
        const int nx = P.snel[0], r = e / nx;
        const int eB = struct_neighbour(P, e - r * nx, r % P.snel[1], r / P.snel[1], e, f);
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
        z[c] = pair ? __ldg(reinterpret_cast<const double2*>(u + v0)) : make_double2(__ldg(u + v0), __ldg(u + v1));
    }
}

// Column phase of one warp: field src -> dst, residual components ROLE (0: x, 1: y) on all
// planes and z on planes 4 ROLE .. 4 ROLE + 3.
template <int ROLE>
__device__ __forceinline__ void dmma8_columns(const StageParams& P, const double* su, const double* V,
                                              const double* Fl, int g, int t, int dst, double d0, double d1,
                                              double rx, double sy, double tz, long long ebase,
                                              const double* __restrict__ Dc, const double2* zf) {
    constexpr int N3 = 512;
    const double A = P.a, B = P.b, DT = P.dt;
    const bool kread = (P.kio & kKRead) != 0, kwrite = (P.kio & kKWrite) != 0;
    const int hf = dst == 0 ? 0 : 1;
    const long long S = P.stride;
    const int m0 = 8 * g + 2 * t;  // the lane's first node in a plane
    // its two node columns of the component differentiated along t
    double2 col[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) col[l] = *reinterpret_cast<const double2*>(V + (1 - ROLE) * N3 + 64 * l + m0);
    double* const k1 = P.k + (dst + ROLE) * S + ebase + m0;
    double* const k2 = P.k + (dst + 2) * S + ebase + m0;
    double* const o1 = P.u_out + (dst + ROLE) * S + ebase + m0;
    double* const o2 = P.u_out + (dst + 2) * S + ebase + m0;
    auto load_k = [&](const double* p) {
        return kread ? __ldcg(reinterpret_cast<const double2*>(p)) : make_double2(0.0, 0.0);
    };
    auto update = [&](double* kp, double* op, const double* up, double2 kold, double r0, double r1) {
        const double kn0 = A * kold.x + DT * r0, kn1 = A * kold.y + DT * r1;
        const double2 uo = *reinterpret_cast<const double2*>(up);
        if (kwrite) __stcs(reinterpret_cast<double2*>(kp), make_double2(kn0, kn1));
        __stcs(reinterpret_cast<double2*>(op), make_double2(uo.x + B * kn0, uo.y + B * kn1));
    };
    const bool onx = t == 0 || t == 3, ony = g == 0 || g == 7;
    const double* Fx = Fl + ((t == 0 ? 3 : 1) * 4 + 2 * hf) * 64 + g;      // x faces: y, z components
    const double* Fy = Fl + ((g == 0 ? 0 : 2) * 4 + 2 * hf) * 64 + 2 * t;  // y faces: z, x components
    double2 n1 = load_k(k1), n2 = make_double2(0.0, 0.0);
    if (ROLE == 0) n2 = load_k(k2);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const bool z_now = (k >= 4) == (ROLE == 1), z_next = (k + 1 >= 4) == (ROLE == 1);
        const double2 c1 = n1, c2 = n2;
        if (k < 7) {
            n1 = load_k(k1 + 64 * (k + 1));
            if (z_next) n2 = load_k(k2 + 64 * (k + 1));
        }
        const double* Vz = V + 2 * N3 + 64 * k;
        double a0 = 0.0, a1 = 0.0;
        if constexpr (ROLE == 0) {  // s (swapped form): B[t][g] = V(i = g, l = t, k)
            dmma_f64(a0, a1, d0, Vz[8 * t + g]);
            dmma_f64(a0, a1, d1, Vz[8 * (4 + t) + g]);
        } else {  // r (original form): A[g][t] = V(l = t, j = g, k)
            dmma_f64(a0, a1, Vz[8 * g + t], d0);
            dmma_f64(a0, a1, Vz[8 * g + 4 + t], d1);
        }
        // t: sums over the cached columns, D(k, l) from Dc (the parameter bank when the
        // caller has it there, else shared memory: the same values either way)
        double b0 = 0.0, b1 = 0.0;
#pragma unroll
        for (int l = 0; l < 8; ++l) {
            const double dk = Dc[k + 8 * l];
            b0 += dk * col[l].x;
            b1 += dk * col[l].y;
        }
        double r0, r1;
        if constexpr (ROLE == 0) {
            r0 = sy * a0 - tz * b0;
            r1 = sy * a1 - tz * b1;
            if (ony) {
                const double2 y = *reinterpret_cast<const double2*>(Fy + 64 + 8 * k);
                r0 += y.x;
                r1 += y.y;
            }
        } else {
            r0 = tz * b0 - rx * a0;
            r1 = tz * b1 - rx * a1;
            if (onx) {
                const double x = Fx[8 * k];
                if (t == 0) r0 += x;
                else r1 += x;
            }
        }
        if (k == 0 || k == 7) {
            const double2 z = zf[k == 0 ? 0 : 128];
            r0 += z.x;
            r1 += z.y;
        }
        if (z_now) {
            const double* Vy = V + N3 + 64 * k;
            const double* Vx = V + 64 * k;
            double yr0 = 0.0, yr1 = 0.0, xs0 = 0.0, xs1 = 0.0;
            dmma_f64(yr0, yr1, Vy[8 * g + t], d0);
            dmma_f64(yr0, yr1, Vy[8 * g + 4 + t], d1);
            dmma_f64(xs0, xs1, d0, Vx[8 * t + g]);
            dmma_f64(xs0, xs1, d1, Vx[8 * (4 + t) + g]);
            double q0 = rx * yr0 - sy * xs0, q1 = rx * yr1 - sy * xs1;
            // face order: y-, x+, y+, x- (add_lifts_xy)
            double x = 0.0;
            double2 y = make_double2(0.0, 0.0);
            if (onx) x = Fx[64 + 8 * k];
            if (ony) y = *reinterpret_cast<const double2*>(Fy + 8 * k);
            const bool xfirst = t == 3 && g == 7;
            q0 = (q0 + y.x) + (t == 0 ? x : 0.0);
            const double xb = t == 3 ? x : 0.0;
            q1 = (q1 + (xfirst ? xb : y.y)) + (xfirst ? y.y : xb);
            update(k2 + 64 * k, o2 + 64 * k, su + (dst + 2) * N3 + 64 * k + m0, c2, q0, q1);
        }
        // LSRK45 (src/device/dg_kernels.cu:404-406), FP64
        update(k1 + 64 * k, o1 + 64 * k, su + (dst + ROLE) * N3 + 64 * k + m0, c1, r0, r1);
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
    if (role == 0) dmma8_columns<0>(P, su, V, sflux, g, t, dst, d0, d1, rx, sy, tz, ebase, Dc, zf);
    else dmma8_columns<1>(P, su, V, sflux, g, t, dst, d0, d1, rx, sy, tz, ebase, Dc, zf);
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
