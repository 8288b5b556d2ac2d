// stage_quad.cuh -- bulk-copy tile with four threads per node column (FP64, axis-aligned
// class): the residual split by field and, within a field, by component.
//
// The two-thread form (stage_bulk.cuh with the field split) holds two node columns and
// both of its D rows, 8N registers, and forms three components a plane: 128 to 168
// registers a thread, 12 to 16 warps to an SM, which wait for the latency of their shared
// loads and FMAs with no unit of the SM above 70-80 %.  Here the first thread of a field
// forms its x component on all planes and z on the lower half of them, the second y and
// the upper half of z, as the warps of the tensor-core tile do.  A thread then
// differentiates one component along t and holds one column and its D rows, 6N registers,
// and half the work: more warps fit, and an element's critical path is half as long.
//
// The four roles of a column run different code, so each role's threads are whole warps:
// GW = EPB N^2 rounded up to 32 threads (at 5, 7 and 9 points 78, 77 and 84 % of the lanes,
// no fewer than in the two-thread form).  Role group f also has face f (0..3): one face
// point a thread.  Arithmetic and order of every sum are those of compute2's FP64 field
// split, so the results are the same bits.
//
// On B200 this is the shape for few elements (NWB_SMALL in stage_variants.h, with the times
// where the lines lie), and at 4 points for all: 50^3 elements 1450 -> 1405 us a step.  On
// large meshes of 5 and more points it is slower, 5 points 1580 -> 1596 us, 7 points 1639 ->
// 1870, 9 points 1499 -> 1936: unrolled over all planes it needs more registers than 6N
// suggests, spills at the residency that would pay and gains no warps without.
#pragma once
#include "stage_bulk.cuh"

namespace nwb {
namespace stage {

template <int N, int EPB>
struct Quad {
    static constexpr int N2 = N * N;
    static constexpr int GW = (EPB * N2 + 31) / 32 * 32;  // threads per role
    static constexpr int threads = 4 * GW;
};

// Column phase of role ROLE (0: x and the lower half of z, 1: y and the upper half of z) of
// the field src -> dst, at node column (i, j) of one element.
template <int N, int CS, bool KSM, bool CD, int ROLE>
__device__ __forceinline__ void quad_columns(const StageParams& P, const double* su, const double* sk,
                                             const double* sD, const ElemGeo& geo, const double* Fl, int i, int j,
                                             int src, int dst, const double (&zf)[2], long long ebase,
                                             const double* __restrict__ Dc) {
    constexpr int N2 = N * N;
    constexpr int HZ = (N + 1) / 2;  // planes of z that role 0 takes
    const long long S = P.stride;
    const double A = P.a, B = P.b, DT = P.dt;
    const bool kread = (P.kio & kKRead) != 0, kwrite = (P.kio & kKWrite) != 0;
    const int hf = dst == 0 ? 0 : 1;
    const double sgn = hf == 0 ? 1.0 : -1.0;
    const double* V = su + src * CS;
    double col[N], Dr[N], Ds[N];
#pragma unroll
    for (int l = 0; l < N; ++l) {
        col[l] = V[(1 - ROLE) * CS + i + N * j + N2 * l];
        Dr[l] = sD[i + l * N];
        Ds[l] = sD[j + l * N];
    }
    const double rx = geo.met[0], sy = geo.met[4], tz = geo.met[8];
    const bool onx = i == 0 || i == N - 1, ony = j == 0 || j == N - 1;
    const bool xfirst = i == N - 1 && j == N - 1;
    const double* Fx = Fl + ((i == 0 ? 3 : 1) * 4 + 2 * hf) * N2 + j;  // x faces: y, z components
    const double* Fy = Fl + ((j == 0 ? 0 : 2) * 4 + 2 * hf) * N2 + i;  // y faces: z, x components
    const int m0 = i + N * j;
    const double* k1s = sk + (dst + ROLE) * CS + m0;
    const double* k2s = sk + (dst + 2) * CS + m0;
    double* const k1 = P.k + (dst + ROLE) * S + ebase + m0;
    double* const k2 = P.k + (dst + 2) * S + ebase + m0;
    double* const o1 = P.u_out + (dst + ROLE) * S + ebase + m0;
    double* const o2 = P.u_out + (dst + 2) * S + ebase + m0;
    auto load_k1 = [&](int k) { return !kread ? 0.0 : (KSM ? k1s[N2 * k] : ld_state(k1 + N2 * k)); };
    auto load_k2 = [&](int k) { return !kread ? 0.0 : (KSM ? k2s[N2 * k] : ld_state(k2 + N2 * k)); };
    auto update = [&](double* kp, double* op, double u, double kold, double r) {
        const double kn = A * kold + DT * r;
        if (kwrite) __stcs(kp, kn);
        __stcs(op, u + B * kn);
    };
    // the next plane's k is requested before this plane's stores
    double n1 = load_k1(0), n2 = ROLE == 0 ? load_k2(0) : 0.0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const bool z_now = (k >= HZ) == (ROLE == 1), z_next = k + 1 < N && (k + 1 >= HZ) == (ROLE == 1);
        const double c1 = n1, c2 = n2;
        if (k + 1 < N) n1 = load_k1(k + 1);
        if (z_next) n2 = load_k2(k + 1);
        const double* Vz = V + 2 * CS + N2 * k;
        double a = 0.0, b = 0.0;
#pragma unroll
        for (int l = 0; l < N; ++l) {
            const double dt = CD ? Dc[k + l * N] : sD[k + l * N];
            if constexpr (ROLE == 0) a += Ds[l] * Vz[N * l + i];
            else a += Dr[l] * Vz[N * j + l];
            b += dt * col[l];
        }
        double r = sgn * (ROLE == 0 ? sy * a - tz * b : tz * b - rx * a);
        if constexpr (ROLE == 0) {
            if (ony) r += Fy[N2 + N * k];
        } else {
            if (onx) r += Fx[N * k];
        }
        if (k == 0) r += zf[0];
        if (k == N - 1) r += zf[1];
        if (z_now) {
            const double* Vy = V + CS + N2 * k;
            const double* Vx = V + N2 * k;
            double yr = 0.0, xs = 0.0;
#pragma unroll
            for (int l = 0; l < N; ++l) {
                yr += Dr[l] * Vy[N * j + l];
                xs += Ds[l] * Vx[N * l + i];
            }
            double q = sgn * (rx * yr - sy * xs);
            // face order: y-, x+, y+, x- (add_lifts_xy)
            double x = 0.0, y = 0.0;
            if (onx) x = Fx[N2 + N * k];
            if (ony) y = Fy[N * k];
            q = (q + (xfirst ? x : y)) + (xfirst ? y : x);
            update(k2 + N2 * k, o2 + N2 * k, su[(dst + 2) * CS + m0 + N2 * k], c2, q);
        }
        // LSRK45 (src/device/dg_kernels.cu:404-406), FP64
        update(k1 + N2 * k, o1 + N2 * k, su[(dst + ROLE) * CS + m0 + N2 * k], c1, r);
    }
}

// One tile of EPB elements.  All threads of the block call it.  CD: D of the t-derivative
// from Dc (a parameter copy), else from shared memory.  pull: see bulk_tile.
template <int N, int EPB, bool KSM, bool CD, class Pull = NoPull>
__device__ __forceinline__ void quad_tile(const StageParams& P, const int e0, unsigned char* smem, const int tid,
                                          const double* Dc, const Pull& pull = Pull()) {
    using L = BulkLayout<N, EPB, KSM>;
    constexpr int N2 = N * N, N3 = N2 * N, CS = L::CSR;
    constexpr int GW = Quad<N, EPB>::GW;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::bar);
    grid_launch_dependents();
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
        bulk_issue<N, EPB, KSM, GEO_BOX, false>(P, e0, smem);
        pull();
    }
    const int h = tid / GW, c = tid - h * GW;
    const int team = c / N2, loc = c - team * N2;
    const int i = loc % N, j = loc / N;
    const int field = h >> 1, role = h & 1;
    const int src = field == 0 ? 3 : 0, dst = 3 - src;
    const bool active = team < min(EPB, P.nelt - e0);  // lanes past EPB N^2: team >= EPB
    const int e = e0 + team;
    const long long S = P.stride;
    // neighbour traces while the copies fly: the thread's point of face h, and of its column
    // on the two faces across t the jumps its component takes (D_x and S_y for x, D_y and S_x
    // for y)
    const int ca = (h & 1) ? 1 : 2, cb = (h & 1) ? 2 : 0;
    const int zd = dst + role, zs = src + 1 - role;
    int vB = kConnPEC, zv[2] = {kConnPEC, kConnPEC};
    double nb[4], zn[2][2];
    if (active) {
        if (P.snel[0] > 0) {
            int ex, ey, ez;
            struct_coords(P, e, ex, ey, ez);
            auto node = [&](int f) {
                const int eB = struct_neighbour(P, ex, ey, ez, e, f);
                return eB < 0 ? kConnPEC : eB * N3 + face_local<N>(opposite_face(f), i, j);
            };
            vB = node(h);
            zv[0] = node(4);
            zv[1] = node(5);
        } else {
            vB = conn_node<N>(__ldg(P.conn + e * 6 + h), i, j);
            zv[0] = conn_node<N>(__ldg(P.conn + e * 6 + 4), i, j);
            zv[1] = conn_node<N>(__ldg(P.conn + e * 6 + 5), i, j);
        }
    }
    grid_wait();
    if (vB >= 0) {
        const double* u = P.u_in + vB;
        nb[0] = ld_state(u + ca * S);
        nb[1] = ld_state(u + cb * S);
        nb[2] = ld_state(u + (3 + ca) * S);
        nb[3] = ld_state(u + (3 + cb) * S);
    }
#pragma unroll
    for (int s = 0; s < 2; ++s)
        if (zv[s] >= 0) {
            zn[s][0] = ld_state(P.u_in + zd * S + zv[s]);
            zn[s][1] = ld_state(P.u_in + zs * S + zv[s]);
        }
    if (!bulk_wait_tile<N, EPB, KSM, GEO_BOX, false>(P, smem, tid)) return;
    const int off = static_cast<int>((static_cast<long long>(e0) * N3) & 1) + team * N3;
    const double* su = reinterpret_cast<const double*>(smem + L::u0) + off;
    const double* sk = KSM ? reinterpret_cast<const double*>(smem + L::k0) + off : nullptr;
    const double* sD = reinterpret_cast<const double*>(smem + L::D);
    const ElemGeo* sg = reinterpret_cast<const ElemGeo*>(smem + L::geo0) + team;
    double* sflux = reinterpret_cast<double*>(smem + L::flux0) + team * 16 * N2;
    // lifted fluxes: face h into shared memory, the faces across t into registers (box_flux)
    double zf[2] = {0.0, 0.0};
    if (active) {
        const double* own = su + face_local<N>(h, i, j);
        double jmp[4], F[4];
        box_jumps(vB, nb, own[ca * CS], own[cb * CS], own[(3 + ca) * CS], own[(3 + cb) * CS], jmp);
        box_flux<double>(sg->nrm[h][(h & 1) ? 0 : 1], P.c0, sg->lift[h], jmp, F);
        double* out = sflux + h * 4 * N2 + loc;
#pragma unroll
        for (int x = 0; x < 4; ++x) out[x * N2] = F[x];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int m = i + N * j + (s ? N2 * (N - 1) : 0);
            const double od = su[zd * CS + m], os = su[zs * CS + m];
            double jd, js;
            if (zv[s] >= 0) {
                jd = zn[s][0] - od;
                js = zn[s][1] - os;
            } else {
                // the mirror turns E at a PEC wall, H at a PMC wall
                const bool turns_d = (zv[s] == kConnPMC) == (field == 1);
                jd = turns_d ? -2.0 * od : 0.0;
                js = turns_d ? 0.0 : -2.0 * os;
            }
            const double nd = sg->nrm[4 + s][2];
            const double hc = 0.5 * P.c0 * (nd * nd), hs = 0.5 * nd;
            zf[s] = sg->lift[4 + s] * (field == role ? hc * jd - hs * js : hs * js + hc * jd);
        }
    }
    __syncthreads();
    if (!active) return;
    const long long ebase = static_cast<long long>(e) * N3;
    if (role == 0)
        quad_columns<N, CS, KSM, CD, 0>(P, su, sk, sD, *sg, sflux, i, j, src, dst, zf, ebase, Dc);
    else
        quad_columns<N, CS, KSM, CD, 1>(P, su, sk, sD, *sg, sflux, i, j, src, dst, zf, ebase, Dc);
}

template <int N, int EPB, int MINB, bool KSM>
__global__ void __launch_bounds__(Quad<N, EPB>::threads, MINB)
    stage_quad_kernel(const __grid_constant__ StageParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    quad_tile<N, EPB, KSM, true>(P, blockIdx.x * EPB, smem, threadIdx.x, P.Dc);
}

template <int N, int EPB, int MINB, bool KSM>
cudaError_t launch_quad(const StageParams* p, cudaStream_t st, StageConfig* cfg) {
    using L = BulkLayout<N, EPB, KSM>;
    constexpr int threads = Quad<N, EPB>::threads;
    auto kern = stage_quad_kernel<N, EPB, MINB, KSM>;
    if (cfg) *cfg = StageConfig{4, EPB, threads, L::total, KSM ? 1 : 0, MINB};
    static std::atomic<int> attr_set[kMaxDeviceSlots];  // per kernel and device
    if (cudaError_t e = set_smem_once(kern, L::total, attr_set); e != cudaSuccess) return e;
    if (!p) return cudaSuccess;
    return launch_overlapped(kern, (p->nelt + EPB - 1) / EPB, threads, L::total, st, (p->kio & kOverlap) != 0, *p);
}

}  // namespace stage
}  // namespace nwb
