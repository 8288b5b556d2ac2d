// diag_kernels.cu -- device diagnostics: the FP64 discrete energy of
// Case::computeTotalEnergy (src/case.cpp:733-766) and the largest |E| and |H| of
// Case::getMaxE / getMaxH (src/case.cpp:768-794) as deterministic two-pass reductions,
// the probe values of ProbeManager::record (src/probe.cpp:192-216), and an L2-evicting
// buffer write used between timed iterations.
//
// The reductions are bound by HBM on large states (48 bytes a node, read two nodes
// per 16-byte load) and by latency on small ones, so the second pass sums its at most
// 1184 partials with a block, and results go to mapped host memory (no copy).
// B200, 792 elements of 7 points: ten steps with a probe read after each, then the energy
// and the norms, 1275 -> 901 us.
#include "nwb_internal.h"

namespace nwb {
namespace {

constexpr int kEnergyThreads = 256;

// Contiguous range of nodes of this block, starting at an even node (the states'
// component rows are 512-byte aligned, so node pairs are 16-byte aligned).
__device__ __forceinline__ void node_range(int npts, int* lo, int* hi) {
    const int pairs = (npts + 1) / 2;
    const int per = (pairs + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
    *lo = min(pairs, per * static_cast<int>(blockIdx.x));
    *hi = min(pairs, *lo + per);
}

// Block b sums 1/2 (|E|^2 + |H|^2) J w3 over a contiguous range of node pairs with a
// fixed per-thread order and a fixed shuffle tree, so repeated calls agree bit
// for bit.  jac_e (per element) or jac_n (per node) supplies J.  Node indices fit an
// int (at most 2^31 - 1 nodes); a row's padding holds the odd last pair's partner.
__global__ void __launch_bounds__(kEnergyThreads)
energy_partials_kernel(const double* __restrict__ u, long long stride, int N3, int npts,
                       const double* __restrict__ jac_e, const double* __restrict__ jac_n,
                       const double* __restrict__ w3, double* __restrict__ partial) {
    int lo, hi;
    node_range(npts, &lo, &hi);
    double acc = 0.0;
    for (int x = lo + static_cast<int>(threadIdx.x); x < hi; x += kEnergyThreads) {
        const int p = 2 * x;
        double2 v[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) v[c] = __ldg(reinterpret_cast<const double2*>(u + c * stride + p));
        const unsigned e = static_cast<unsigned>(p) / static_cast<unsigned>(N3);
        const int m = p - static_cast<int>(e) * N3;
        const double dV = (jac_n ? jac_n[p] : jac_e[e]) * w3[m];
        acc += 0.5 *
               ((v[0].x * v[0].x + v[1].x * v[1].x + v[2].x * v[2].x) +
                (v[3].x * v[3].x + v[4].x * v[4].x + v[5].x * v[5].x)) *
               dV;
        if (p + 1 < npts) {
            const bool next = m + 1 == N3;
            const double dW = (jac_n ? jac_n[p + 1] : jac_e[next ? e + 1 : e]) * w3[next ? 0 : m + 1];
            acc += 0.5 *
                   ((v[0].y * v[0].y + v[1].y * v[1].y + v[2].y * v[2].y) +
                    (v[3].y * v[3].y + v[4].y * v[4].y + v[5].y * v[5].y)) *
                   dW;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    __shared__ double warp_sums[kEnergyThreads / 32];
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < kEnergyThreads / 32; ++w) s += warp_sums[w];
        partial[blockIdx.x] = s;
    }
}

// One block: strided sums in a fixed order, then a fixed tree.  (One thread summing them
// one after the other waited for L2 at every fourth: about 100 us for 1184.)
__global__ void __launch_bounds__(kEnergyThreads)
energy_final_kernel(const double* __restrict__ partial, int n, double* __restrict__ out) {
    __shared__ double s[kEnergyThreads];
    double acc = 0.0;
    for (int b = threadIdx.x; b < n; b += kEnergyThreads) acc += partial[b];
    s[threadIdx.x] = acc;
    __syncthreads();
#pragma unroll
    for (int w = kEnergyThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = s[0];
}

// Largest |E|^2 and |H|^2 over the nodes of a contiguous range per block, the squares
// formed as Case::getMaxE / getMaxH (src/case.cpp:768-794) form them on the host:
// (x*x + y*y) + z*z with separate multiply and add roundings (no contraction), kept when
// larger than the running maximum (a NaN node never is).  The correctly rounded
// square root is monotone, so the root of the largest square, taken once at the end, is
// the host's largest root bit for bit, in any order.
// partial[2b] = max |E|^2, partial[2b+1] = max |H|^2 of block b.
__device__ __forceinline__ double square3_rn(double x, double y, double z) {
    return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

__global__ void __launch_bounds__(kEnergyThreads)
maxnorm_partials_kernel(const double* __restrict__ u, long long stride, int npts,
                        double* __restrict__ partial) {
    int lo, hi;
    node_range(npts, &lo, &hi);
    double me = 0.0, mh = 0.0;
    for (int x = lo + static_cast<int>(threadIdx.x); x < hi; x += kEnergyThreads) {
        const int p = 2 * x;
        double2 v[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) v[c] = __ldg(reinterpret_cast<const double2*>(u + c * stride + p));
        double e = square3_rn(v[0].x, v[1].x, v[2].x), h = square3_rn(v[3].x, v[4].x, v[5].x);
        if (e > me) me = e;
        if (h > mh) mh = h;
        if (p + 1 < npts) {
            e = square3_rn(v[0].y, v[1].y, v[2].y);
            h = square3_rn(v[3].y, v[4].y, v[5].y);
            if (e > me) me = e;
            if (h > mh) mh = h;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double oe = __shfl_down_sync(0xffffffffu, me, off);
        const double oh = __shfl_down_sync(0xffffffffu, mh, off);
        if (oe > me) me = oe;
        if (oh > mh) mh = oh;
    }
    __shared__ double warp_max[2][kEnergyThreads / 32];
    if ((threadIdx.x & 31) == 0) {
        warp_max[0][threadIdx.x >> 5] = me;
        warp_max[1][threadIdx.x >> 5] = mh;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double m = 0.0;
        for (int w = 0; w < kEnergyThreads / 32; ++w)
            if (warp_max[threadIdx.x][w] > m) m = warp_max[threadIdx.x][w];
        partial[2 * blockIdx.x + threadIdx.x] = m;
    }
}

// One warp per field over the blocks' maxima.
__global__ void __launch_bounds__(64)
maxnorm_final_kernel(const double* __restrict__ partial, int n, double* __restrict__ out) {
    const int field = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double m = 0.0;
#pragma unroll 4
    for (int b = lane; b < n; b += 32) {
        const double v = partial[2 * b + field];
        if (v > m) m = v;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double o = __shfl_down_sync(0xffffffffu, m, off);
        if (o > m) m = o;
    }
    if (lane == 0) out[field] = __dsqrt_rn(m);
}

// ProbeManager::record (src/probe.cpp:192-216): warp c of block pr forms the N^3 products
// w[p] * u[offset + p] of component c with coalesced loads, then its first lane adds
// them in node order, with separate multiply and add roundings as on the host, so the
// values equal the reference's bit for bit on the same state and weights.  (One thread
// per component loading as it adds waited for L2 at every fourth node.)  The weights are
// loaded before the wait: the launch may overlap the stage before it.  So the state is
// not (launch_overlapped): coherent loads behind the wait.
constexpr int kProbeThreads = 192;
__global__ void __launch_bounds__(kProbeThreads)
probe_kernel(const double* u, long long stride, int N3,
             const long long* __restrict__ offset, const double* __restrict__ w, int nprobes,
             double* __restrict__ out) {
    __shared__ double prod[6][1000];
    const int pr = blockIdx.x;
    const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double* wp = w + static_cast<long long>(pr) * N3;
    const double* up = u + c * stride + offset[pr];
    for (int p = lane; p < N3; p += 32) prod[c][p] = wp[p];
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
#pragma unroll 4
    for (int p = lane; p < N3; p += 32) prod[c][p] = __dmul_rn(prod[c][p], __ldcg(up + p));
    __syncwarp();
    if (lane != 0) return;
    double acc = 0.0;
#pragma unroll 16
    for (int p = 0; p < N3; ++p) acc = __dadd_rn(acc, prod[c][p]);
    out[pr * 6 + c] = acc;
}

__global__ void l2_flush_kernel(int4* __restrict__ buf, size_t n16) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t x = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; x < n16; x += stride)
        buf[x] = make_int4(static_cast<int>(x), 0, 0, 0);
}

// Gaussian pulses on the nodes of a box (launch_box_pulse).  Here, in a small module, and not
// beside the pool's kernels: the first launch from a module loads the whole of it.
__global__ void box_pulse_kernel(const BoxPulse b, double* __restrict__ u, long long stride) {
    const int N = b.N, N3 = N * N * N;
    const long long npts = static_cast<long long>(b.nel[0]) * b.nel[1] * b.nel[2] * N3;
    for (long long p = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; p < npts;
         p += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long e = p / N3;
        const int m = static_cast<int>(p - e * N3);
        const int i = m % N, j = (m / N) % N, k = m / (N * N);
        const int ex = static_cast<int>(e % b.nel[0]);
        const int ey = static_cast<int>((e / b.nel[0]) % b.nel[1]);
        const int ez = static_cast<int>(e / (static_cast<long long>(b.nel[0]) * b.nel[1]));
        const double x = b.lo[0] + (ex + 0.5 * (b.z[i] + 1.0)) * b.h[0];
        const double y = b.lo[1] + (ey + 0.5 * (b.z[j] + 1.0)) * b.h[1];
        const double z = b.lo[2] + (ez + 0.5 * (b.z[k] + 1.0)) * b.h[2];
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            const double* q = b.pulse + 5 * c;
            double v = 0.0;
            if (q[4] > 0.0) {
                const double dx = x - q[1], dy = y - q[2], dz = z - q[3];
                v = q[0] * exp(-(dx * dx + dy * dy + dz * dz) / (q[4] * q[4]));
            }
            u[c * stride + p] = v;
        }
    }
}

}  // namespace

int energy_blocks(int nelt) {
    const int b = (nelt + 3) / 4;
    return b < 1 ? 1 : (b > 1184 ? 1184 : b);
}

cudaError_t launch_energy(const double* u, long long stride, int N, int nelt,
                          const double* jac_e, const double* jac_n, const double* w3,
                          double* partial, int nblocks, double* out, cudaStream_t st) {
    const int N3 = N * N * N;
    const int npts = nelt * N3;
    energy_partials_kernel<<<nblocks, kEnergyThreads, 0, st>>>(u, stride, N3, npts, jac_e, jac_n,
                                                               w3, partial);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    energy_final_kernel<<<1, kEnergyThreads, 0, st>>>(partial, nblocks, out);
    return cudaGetLastError();
}

cudaError_t launch_max_norms(const double* u, long long stride, long long npts, double* partial,
                             int nblocks, double* out, cudaStream_t st) {
    maxnorm_partials_kernel<<<nblocks, kEnergyThreads, 0, st>>>(u, stride, static_cast<int>(npts), partial);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    maxnorm_final_kernel<<<1, 64, 0, st>>>(partial, nblocks, out);
    return cudaGetLastError();
}

cudaError_t launch_probes(const double* u, long long stride, int N3, const long long* offset,
                          const double* w, int nprobes, double* out, cudaStream_t st) {
    if (nprobes <= 0) return cudaSuccess;
    return launch_overlapped(probe_kernel, nprobes, kProbeThreads, 0, st, true, u, stride, N3, offset, w, nprobes,
                             out);
}

cudaError_t launch_box_pulse(const BoxPulse& b, double* u, long long stride, cudaStream_t st) {
    box_pulse_kernel<<<148 * 8, 256, 0, st>>>(b, u, stride);
    return cudaGetLastError();
}

cudaError_t launch_l2_flush(void* buf, size_t bytes, cudaStream_t st) {
    const size_t n16 = bytes / 16;
    l2_flush_kernel<<<148 * 4, 256, 0, st>>>(static_cast<int4*>(buf), n16);
    return cudaGetLastError();
}

}  // namespace nwb
