// Tree transfers of the batched form (64 fields per block).
//
// The proxies of a panel are its N x N Chebyshev nodes (N = d + 1), proxy
// p = i + l N at (xi_i, eta_l).  A parent's degree-d barycentric Lagrange
// basis (bli_module.f90:50-113) restricted to a child is a degree-d
// polynomial in each coordinate, so the child's nodes reproduce it exactly:
//     L^p_j(x) = sum_i L^p_j(xc_i) L^c_i(x).
// Children halve their parent's interval in each coordinate, and the bases
// are invariant under affine maps of the interval, so the matrices
// H_h[j][i] = L^p_j(xc_i) are the same two (lower half h = 0, upper h = 1) for
// every panel.  With A = H of the child's xi half and B = H of its eta half:
//   child-to-parent (upward):  W_p(j, k) += sum_i A[j][i] sum_l B[k][l] W_c(i, l)
//     -- the parent's proxy weights sum_s L^p_j(xi_s) L^p_k(eta_s) w_s from
//     its children's, without revisiting the points;
//   parent-to-child (downward): Phi_c(i, l) (+)= sum_j A[j][i] sum_k B[k][l] Phi_p(j, k)
//     -- the parent's potential interpolant evaluated at the child's nodes,
//     so the child's interpolant reproduces it.
// Both are exact in exact arithmetic.  Each is two 1-D transfers (2 N^3
// multiply-adds per field instead of N^4), in FP32 like the rows they read
// and write (a transfer rounds at the 1e-7 level; FP64 sums made the solve
// 0.35 ms slower at 2.3M cells x 64 fields and were no more accurate against
// the direct sum).  Both are bound by memory at the deepest level and by the
// latency of one CTA at the others (a tree has 4 to 7 levels, a launch each, of
// 6 to a few thousand tasks).  So one CTA of 16 N threads per task (l2l: and
// component), whose thread (q = t % 16, r = t / 16) reads row r of the tile for
// fields 4q .. 4q + 3 straight into registers (m2m: a child ahead); only the
// first transfer's result goes through shared memory.  A matrix entry is one
// shared-memory broadcast, and those bound the arithmetic, so each feeds four
// fields.  The loops are unrolled over the compile-time N.  Deepest level at
// 655,362 cells x 64 fields: l2l (4,336 tasks, 0.6 GB) 224 -> 101 us, m2m
// (1,087) 81 -> 39 us; smallest l2l level (20 tasks) 25 -> 5.5 us, m2m 17 -> 11
// us; against one thread a field, tiles through shared memory, a CTA for all
// three components.  (Registers without the wider threads: 197 and 69 us.)
#include <cuda_runtime.h>

#include "kernels.cuh"
#include "mixed.cuh"

namespace sal {
namespace mix {

namespace {
constexpr int kF = 64;
constexpr int kQ = kF / 4;   // a row's float4s

// both matrices and `tiles` float tiles
template <int N>
constexpr size_t transfer_smem(int tiles) {
    return (2 * N * N + tiles * (size_t)N * N * kF) * sizeof(float);
}

__device__ __forceinline__ float4 fma4(float a, float4 x, float4 c) {
    const float2 lo = __ffma2_rn(make_float2(a, a), make_float2(x.x, x.y), make_float2(c.x, c.y));
    const float2 hi = __ffma2_rn(make_float2(a, a), make_float2(x.z, x.w), make_float2(c.z, c.w));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
}  // namespace

// Child-to-parent transfer of one tree level.  tasks: 6 per parent (parent
// slot, 4 child slots or -1, the children's halves: bits 2c (xi) and 2c + 1
// (eta) for child c).  H: the two N x N transfer matrices.  w: the weight
// rows of the slots, N^2 rows of 64 fields per slot.
template <int N>
__global__ void __launch_bounds__(kQ * N) m2m_kernel(const int32_t *__restrict__ tasks, const double *__restrict__ H,
                                                     float4 *__restrict__ w) {
    dev::after_previous();
    constexpr int P = N * N;
    extern __shared__ __align__(16) float smf[];
    float4 *T = reinterpret_cast<float4 *>(smf);   // two tiles, children in turn
    float *Hs = smf + 2 * P * kF;
    const int32_t *tk = tasks + 6 * (size_t)blockIdx.x;
    const int tid = threadIdx.x, q = tid & (kQ - 1), r = tid / kQ;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 wv[N], nx[N];   // a child's W_c(r, l), the next one's
    auto load = [&](int c, float4 (&v)[N]) {
        const int child = tk[1 + c];
        const float4 *src = w + (size_t)(child < 0 ? 0 : child) * P * kQ + q;
#pragma unroll
        for (int l = 0; l < N; ++l) v[l] = child < 0 ? zero : src[(r + l * N) * kQ];
    };
    load(0, nx);
    for (int e = tid; e < 2 * P; e += kQ * N) Hs[e] = (float)H[e];
    float4 acc[N];   // W_p(j, r), j = 0 .. N-1
#pragma unroll
    for (int j = 0; j < N; ++j) acc[j] = zero;
    const int code = tk[5];
    int turn = 0;   // of the children that are there
    __syncthreads();
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int l = 0; l < N; ++l) wv[l] = nx[l];
        if (c < 3) load(c + 1, nx);
        if (tk[1 + c] < 0) continue;
        const float *A = Hs + ((code >> (2 * c)) & 1) * P, *B = Hs + ((code >> (2 * c + 1)) & 1) * P;
        float4 *Tc = T + turn * P * kQ;
        turn ^= 1;
        // T(r, k) = sum_l B[k][l] W_c(r, l)
#pragma unroll
        for (int k = 0; k < N; ++k) {
            float4 s = zero;
#pragma unroll
            for (int l = 0; l < N; ++l) s = fma4(B[k * N + l], wv[l], s);
            Tc[(r + k * N) * kQ + q] = s;
        }
        __syncthreads();   // (the tile of two children ago was read before the last one)
        // W_p(j, r) += sum_i A[j][i] T(i, r)
#pragma unroll
        for (int i = 0; i < N; ++i) wv[i] = Tc[(i + r * N) * kQ + q];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            float4 s = zero;
#pragma unroll
            for (int i = 0; i < N; ++i) s = fma4(A[j * N + i], wv[i], s);
            acc[j] = add4(acc[j], s);
        }
    }
    float4 *dst = w + (size_t)tk[0] * P * kQ + q;
#pragma unroll
    for (int j = 0; j < N; ++j) dst[(j + r * N) * kQ] = acc[j];
}

// Parent-to-child transfer of one tree level.  tasks: 4 per child (child
// slot, parent slot, own: 1 adds to the child's own potentials, 0 replaces
// them, the child's halves: bit 0 xi, bit 1 eta).  phi: per slot 3 N^2 rows
// (proxy p, Cartesian component c at row 3p + c) of 64 fields.
template <int N>
__global__ void __launch_bounds__(kQ * N) l2l_kernel(const int32_t *__restrict__ tasks, const double *__restrict__ H,
                                                     float4 *__restrict__ phi) {
    dev::after_previous();
    constexpr int P = N * N;
    extern __shared__ __align__(16) float smf[];
    float4 *T = reinterpret_cast<float4 *>(smf);
    float *Hs = smf + P * kF;
    const int32_t *tk = tasks + 4 * (size_t)(blockIdx.x / 3);
    const int child = tk[0], parent = tk[1], own = tk[2], code = tk[3];
    const int tid = threadIdx.x, q = tid & (kQ - 1), r = tid / kQ, c = blockIdx.x % 3;
    const float4 *src = phi + ((size_t)parent * 3 * P + c) * kQ + q;
    float4 *dst = phi + ((size_t)child * 3 * P + c) * kQ + q;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 pv[N], ov[N];   // Phi_p(r, k), the child's own Phi_c(i, r)
#pragma unroll
    for (int k = 0; k < N; ++k) pv[k] = src[3 * (r + k * N) * kQ];
    if (own) {
#pragma unroll
        for (int i = 0; i < N; ++i) ov[i] = dst[3 * (i + r * N) * kQ];
    }
    for (int e = tid; e < 2 * P; e += kQ * N) Hs[e] = (float)H[e];
    const float *A = Hs + (code & 1) * P, *B = Hs + ((code >> 1) & 1) * P;
    __syncthreads();
    // T(r, l) = sum_k B[k][l] Phi_p(r, k)
#pragma unroll
    for (int l = 0; l < N; ++l) {
        float4 s = zero;
#pragma unroll
        for (int k = 0; k < N; ++k) s = fma4(B[k * N + l], pv[k], s);
        T[(r + l * N) * kQ + q] = s;
    }
    __syncthreads();
    // Phi_c(i, r) (+)= sum_j A[j][i] T(j, r)
#pragma unroll
    for (int j = 0; j < N; ++j) pv[j] = T[(j + r * N) * kQ + q];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float4 s = zero;
#pragma unroll
        for (int j = 0; j < N; ++j) s = fma4(A[j * N + i], pv[j], s);
        dst[3 * (i + r * N) * kQ] = own ? add4(ov[i], s) : s;
    }
}

template <int N>
static void launch_m2m_n(const int32_t *tasks, int ntasks, const double *H, float *w, cudaStream_t st) {
    static std::atomic<unsigned long long> done{0};
    smem_attr_once((const void *)m2m_kernel<N>, (int)transfer_smem<N>(2), done);
    dev::launch_next(m2m_kernel<N>, ntasks, kQ * N, transfer_smem<N>(2), st, tasks, H, reinterpret_cast<float4 *>(w));
}

template <int N>
static void launch_l2l_n(const int32_t *tasks, int ntasks, const double *H, float *phi, cudaStream_t st) {
    static std::atomic<unsigned long long> done{0};
    smem_attr_once((const void *)l2l_kernel<N>, (int)transfer_smem<N>(1), done);
    dev::launch_next(l2l_kernel<N>, 3 * ntasks, kQ * N, transfer_smem<N>(1), st, tasks, H, reinterpret_cast<float4 *>(phi));
}

// N = d + 1 from 2 to kMaxTreeDegree + 1 (the plan turns the tree passes off
// above that)
#define SAL_TRANSFER_DISPATCH(fn, n, ...)                       \
    switch (n) {                                                \
        case 2: fn<2>(__VA_ARGS__); break;                      \
        case 3: fn<3>(__VA_ARGS__); break;                      \
        case 4: fn<4>(__VA_ARGS__); break;                      \
        case 5: fn<5>(__VA_ARGS__); break;                      \
        case 6: fn<6>(__VA_ARGS__); break;                      \
        case 7: fn<7>(__VA_ARGS__); break;                      \
        case 8: fn<8>(__VA_ARGS__); break;                      \
        case 9: fn<9>(__VA_ARGS__); break;                      \
        case 10: fn<10>(__VA_ARGS__); break;                    \
        case 11: fn<11>(__VA_ARGS__); break;                    \
        default: break;                                         \
    }
static_assert(kMaxTreeDegree + 1 == 11, "the dispatch covers N = 2 .. kMaxTreeDegree + 1");

void launch_m2m(const int32_t *tasks, int ntasks, const double *H, int n, float *w, cudaStream_t st) {
    if (ntasks <= 0) return;
    SAL_TRANSFER_DISPATCH(launch_m2m_n, n, tasks, ntasks, H, w, st)
}

void launch_l2l(const int32_t *tasks, int ntasks, const double *H, int n, float *phi, cudaStream_t st) {
    if (ntasks <= 0) return;
    SAL_TRANSFER_DISPATCH(launch_l2l_n, n, tasks, ntasks, H, phi, st)
}

}  // namespace mix
}  // namespace sal
