// Device kernels of the FP64 SAL-gradient treecode (sm_100a).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "sal_internal.hpp"

namespace sal {
namespace dev {

// A solve is a chain of launches, most of them short on a small grid: 6 in the
// FP64 forms, 18 to 22 a batched block.  Each is launched to come up while the
// one before it in the stream ends (launch_next), and every thread of it begins
// with after_previous(): that waits until the kernels before it are complete and
// their writes visible, so nothing is read early, and lets the next one come up
// in its turn.  3,000 points (FP64): 70.0 -> 61.5 us; 40,962 cells x 1
// field batched: 872 -> 850; 163,842 x 13: 2,736 -> 2,710.  A chain's first
// kernel, a kernel behind a memset or another stream's event, and the mma.sync
// passes (where it cost 2 %) are launched the plain way; after_previous() is
// then no wait.
__device__ __forceinline__ void after_previous() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}
template <class... P, class... A>
inline void launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

// fast_sum_module.f90:14,23-25: literal constants folded in double precision,
// exactly as gfortran folds (1.0_8-6.21196_8) and (2.7_8+6.0_8).
constexpr double kCons = -2.343256857908601e-9;
constexpr double kC1 = 1.0 - 6.21196;
constexpr double kC2 = 2.7 + 6.0;
constexpr int kErrTimeout = 1;

// ----------------------------------------------------------------- PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// Bulk (non-tensor) TMA copy global -> this CTA's shared memory, completing
// on an mbarrier.  No multicast.  Both addresses 16-byte aligned, bytes a
// multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
// The same with an L2 cache policy (createpolicy): a stream read once can
// leave L2 to data that is read again.
__device__ __forceinline__ void bulk_g2s_hint(void *dst, const void *src, uint32_t bytes, uint64_t *bar,
                                              uint64_t policy) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
        : "memory");
}
__device__ __forceinline__ uint64_t l2_evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_evict_last() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// A poll that suspends the thread until the phase completes, or at most about
// `ns` nanoseconds.
__device__ __forceinline__ bool mbar_try_wait_ns(uint64_t *bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(ns)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait: gives up after `polls` polls and raises the grid's error
// flag, so a copy that never lands cannot hang the GPU.
constexpr uint32_t kDefaultPolls = 1u << 24;
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, int *err,
                                                  uint32_t polls = kDefaultPolls) {
    for (uint32_t it = 0; it < polls; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    atomicExch(err, kErrTimeout);
    return false;
}

// ----------------------------------------------------------------- kernels of the SAL gradient
// Target-only terms of sal_grad_gfunc (fast_sum_module.f90:19,26-27), hoisted.
struct Tgt {
    double x, y, z, omx32, inv_mp2;
    bool live;  // outside the pole guard
};

__device__ __forceinline__ double tgt_omx32(double z) { return __dsub_rn(1.0, __dmul_rn(z, z)); }
__device__ __forceinline__ bool tgt_live(double z) {
    return (fabs(__dsub_rn(z, 1.0)) > 1e-15) && (fabs(__dadd_rn(z, 1.0)) > 1e-15);
}
__device__ __forceinline__ void tgt_init(Tgt &t, double x, double y, double z) {
    t.x = x; t.y = y; t.z = z;
    t.omx32 = tgt_omx32(z);
    t.inv_mp2 = __ddiv_rn(1.0, __dsqrt_rn(t.omx32));
    t.live = tgt_live(z);
}

// sal_grad_gfunc (fast_sum_module.f90:9-31) for a live target, operation for
// operation with IEEE division and square root and without contraction, so the
// singular self pair s == t rounds exactly as the reference's does.  The
// division by sqrt(1-tz^2) is a multiply by its hoisted reciprocal.  Used for
// the batched form's self pairs.
__device__ __forceinline__ void gref_exact(const Tgt &t, double sx, double sy, double sz, double &gx, double &gy) {
    double gxy = __dadd_rn(__dmul_rn(t.x, sx), __dmul_rn(t.y, sy));
    double g = __dadd_rn(gxy, __dmul_rn(t.z, sz));
    g = fmax(fmin(g, 1.0), -1.0);
    double mp = __dsub_rn(2.0, __dmul_rn(2.0, g));
    double sqp = __dsqrt_rn(mp);
    double p1 = __ddiv_rn(kC1, __dadd_rn(__dmul_rn(sqp, mp), 1e-16));
    double p2 = __ddiv_rn(__dmul_rn(kC2, __dadd_rn(__dmul_rn(2.0, g), sqp)),
                          __dadd_rn(__dmul_rn(2.0, __dsub_rn(__dmul_rn(g, g), 1.0)), 1e-16));
    double val = __dmul_rn(__dadd_rn(p1, p2), kCons);
    double ny = __dsub_rn(__dmul_rn(sz, t.omx32), __dmul_rn(t.z, gxy));
    double nx = __dsub_rn(__dmul_rn(t.x, sy), __dmul_rn(t.y, sx));
    gy = __dmul_rn(__dmul_rn(ny, t.inv_mp2), val);
    gx = __dmul_rn(__dmul_rn(nx, t.inv_mp2), val);
}

// Reciprocal and square root for the treecode's inner loops: the hardware's
// FP64 approximation (about 20 good bits, no conversion to FP32 and back, which
// costs four conversions a pair on the SFU's pipe), refined by one step of
// Householder's third-order iteration, whose error is the cube of the seed's:
// for 1/x, r (1 + e + e^2) with e = 1 - x r; for sqrt(x) = x y with
// y ~ 1/sqrt(x), g (1 + e/2 + 3 e^2/8) with g = x y and e = 1 - g y.  Accurate
// to about one ulp for normal x whose reciprocal (inverse square root) is
// normal; 0, infinities and NaN do not give IEEE results, and callers keep
// them away.
__device__ __forceinline__ double rcp_seed(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}
__device__ __forceinline__ double fast_rcp(double x) {
    const double r = rcp_seed(x), e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ double fast_sqrt(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double g = x * y, e = fma(-g, y, 1.0);
    return fma(g * e, fma(e, 0.375, 0.5), g);
}

// The kernel's scalar val w / kCons as a function of mp = 2 - 2g alone.  With
// q = sqrt(mp): 2g + q = (2 - q)(1 + q) and 2(g^2 - 1) = -mp (2 - q)(2 + q)/2,
// so p1 + p2 = N / D with
//   N = kC1 (2 + q) - 2 kC2 (q + mp),  D = q^3 (2 + q) = mp (2 q + mp):
// one square root, one reciprocal, no cancellation.  kReg: p1's + 1e-16,
// folded into D: c (2 + b q) there takes c kC1/q^6 off N / D up to 4 c/q of it
// (c = 1e-16, b = 1 + 2 kC2/kC1); p2's is below 2e-13 of the value for
// q > 1e-3.  Without kReg (far pairs, q > 0.0122, where c is 5e-11 of q^3) b q
// is a constant, its value at q = 0.01225: 1e-13 of the value left, at q = 0.02,
// and no instruction more than with no c at all.  14 FP64 instructions (15 with
// kReg) against 31 of the two denominators' form with its FP32 seeds.
template <bool kReg>
__device__ __forceinline__ double val_chord(double mp, double w) {
    const double q = fast_sqrt(mp);
    const double n = fma(-2.0 * kC2, mp, fma(kC1 - 2.0 * kC2, q, 2.0 * kC1));
    const double t = fma(2.0, q, mp);
    constexpr double b = 1e-16 * (1.0 + 2.0 * kC2 / kC1);
    const double d = fma(mp, t, kReg ? fma(b, q, 2e-16) : 2e-16 + 0.01225 * b);
    const double r = rcp_seed(d), e = fma(-d, r, 1.0), u = n * r;
    return fma(u, fma(e, e, e), u) * w;   // w last: an infinite one gives a signed infinity
}

// Where val_chord<true> stands for the reference's expressions: q >= 1e-3
// (the + 1e-16 terms it leaves out are below 4e-13 of the value), and
// 2e-6 off mp = 4: at the antipode the reference's (2g + q) and (g^2 - 1)
// cancel to rounding noise (4e-10 of p2 at this line, in pairs whose value is
// among the smallest; the line is as close as the test below can draw it,
// because with a band of 0.01 a warp of scattered targets meets it with one
// source in twelve: 17.7 ms for 10,000 targets x 655,362 sources).  False for
// NaN.  On the value's upper word, a positive double's order: the ALU's work,
// not two comparisons on the FP64 pipe.
__device__ __forceinline__ bool chord_plain(double mp) {
    constexpr unsigned kLo = 0x3EB0C6F7u + 1u, kHi = 0x400FFFFFu;   // above 1e-6's, the last below 4's
    return (unsigned)__double2hiint(mp) - kLo < kHi - kLo;
}

// sal_grad_gfunc's val / kCons in the reference's operation order: g clamped,
// mp = 2 - 2g, the two denominators and the two numerators (these carry the
// cancellations that make the self pair pure rounding noise), p1 + p2 over one
// common denominator.
__device__ __forceinline__ double val_ref(double g) {
    g = fmax(fmin(g, 1.0), -1.0);
    const double g2 = __dmul_rn(2.0, g);
    const double mp = __dsub_rn(2.0, g2);
    const double sqp = __dsqrt_rn(mp);
    const double d1 = __dadd_rn(__dmul_rn(sqp, mp), 1e-16);
    const double n2 = __dmul_rn(kC2, __dadd_rn(g2, sqp));
    const double d2 = __dadd_rn(__dmul_rn(2.0, __dsub_rn(__dmul_rn(g, g), 1.0)), 1e-16);
    return __ddiv_rn(fma(kC1, d2, n2 * d1), d1 * d2);
}

// K pairs of the reference kernel (sources s[0], s[stride], ...) as the
// treecode evaluates them: g and 2 - 2g in the reference's operation order,
// then val_chord, K independent chains side by side; or, if any of the K is
// one of the rare pairs (the self pair, near duplicates, antipodes) whose
// value is the reference's rounding noise, one after another with val_ref for
// those.  Adds (nx, ny) val w / kCons into (ax, ay); the constant and the
// target factor 1/sqrt(1 - tz^2) are applied once per target.
template <int K>
__device__ __forceinline__ void gref_near(const Tgt &t, const double4 *s, int stride, double &ax, double &ay) {
    double gxy[K], g[K], mp[K];
    bool plain = true;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double4 q = s[k * stride];
        gxy[k] = __dadd_rn(__dmul_rn(t.x, q.x), __dmul_rn(t.y, q.y));
        g[k] = __dadd_rn(gxy[k], __dmul_rn(t.z, q.z));
        mp[k] = fma(-2.0, g[k], 2.0);   // 2 g is exact: rounds as 2 - 2g
        plain = plain && chord_plain(mp[k]);
    }
    if (plain) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const double4 q = s[k * stride];
            const double val = val_chord<true>(mp[k], q.w);
            ax = fma(fma(-t.y, q.x, t.x * q.y), val, ax);
            ay = fma(fma(-t.z, gxy[k], q.z * t.omx32), val, ay);
        }
    } else {
#pragma unroll 1
        for (int k = 0; k < K; ++k) {
            const double4 q = s[k * stride];
            const double gk = __dadd_rn(__dadd_rn(__dmul_rn(t.x, q.x), __dmul_rn(t.y, q.y)), __dmul_rn(t.z, q.z));
            const double m = fma(-2.0, gk, 2.0);
            const double val = chord_plain(m) ? val_chord<true>(m, q.w) : val_ref(gk) * q.w;
            const double nx = __dsub_rn(__dmul_rn(t.x, q.y), __dmul_rn(t.y, q.x));
            const double ny = __dsub_rn(__dmul_rn(q.z, t.omx32),
                                        __dmul_rn(t.z, __dadd_rn(__dmul_rn(t.x, q.x), __dmul_rn(t.y, q.y))));
            ax = fma(nx, val, ax);
            ay = fma(ny, val, ay);
        }
    }
}

// A pair that EvalBounds has shown to be plain: the dot product fused, and
// Sum val w s as a vector, from which the two components follow once per
// target (nx = tx Ay - ty Ax, ny = (1 - tz^2) Az - tz (tx Ax + ty Ay)).  The
// vector cancels by the chord on projection, and no chord is below 0.012, so
// its rounding stays below 1e-13 of a sum of thousands of pairs.  mt = -2 t.
// 20 FP64 instructions against 27 of gref_near's plain branch.
// K sources s[0], s[stride], ...: independent chains side by side.
template <int K>
__device__ __forceinline__ void gref_far(const double (&mt)[3], const double4 *s, int stride, double (&A)[3]) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double4 q = s[k * stride];
        const double mp = fma(mt[0], q.x, fma(mt[1], q.y, fma(mt[2], q.z, 2.0)));
        const double v = val_chord<false>(mp, q.w);
        A[0] = fma(v, q.x, A[0]);
        A[1] = fma(v, q.y, A[1]);
        A[2] = fma(v, q.z, A[2]);
    }
}

// K pairs of a Cartesian proxy target (x, y, z) with sources s[0], s[stride],
// ...: adds val w (s - x) / kCons, with val's removable antipodal singularity
// cancelled analytically (val_chord's form) and mp = |s - x|^2 from coordinate
// differences, not from 2 - 2 t.s.  Independent chains side by side; with a
// pair closer than 1e-3 among them, which keeps the two + 1e-16 of the
// denominators (a source on the target gives a finite value, times a zero
// displacement), one after another.
template <int K>
__device__ __forceinline__ void cart_pairs(double x, double y, double z, const double4 *s, int stride,
                                           double (&A)[3]) {
    double mp[K];
    bool plain = true;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double4 q = s[k * stride];
        const double dx = q.x - x, dy = q.y - y, dz = q.z - z;
        mp[k] = fma(dx, dx, fma(dy, dy, dz * dz));
        plain = plain && mp[k] >= 1e-6;
    }
    if (plain) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const double4 q = s[k * stride];
            const double v = val_chord<true>(mp[k], q.w);
            A[0] = fma(v, q.x - x, A[0]);
            A[1] = fma(v, q.y - y, A[1]);
            A[2] = fma(v, q.z - z, A[2]);
        }
    } else {
#pragma unroll 1
        for (int k = 0; k < K; ++k) {
            const double4 q = s[k * stride];
            const double dx = q.x - x, dy = q.y - y, dz = q.z - z, m = fma(dx, dx, fma(dy, dy, dz * dz));
            double v;
            if (m >= 1e-6) {
                v = val_chord<true>(m, q.w);
            } else {
                const double c = __dsqrt_rn(m), d1 = c * m + 1e-16, d2 = m * (2.0 + c) + 1e-16;
                v = __ddiv_rn(kC1 * d2 - 2.0 * kC2 * (1.0 + c) * d1, d1 * d2) * q.w;
            }
            A[0] = fma(v, dx, A[0]);
            A[1] = fma(v, dy, A[1]);
            A[2] = fma(v, dz, A[2]);
        }
    }
}

// bli_coeffs, bli_module.f90:6-26 (0-based index i0 of degree d).
__device__ __forceinline__ double bli_coeff(int i0, int d) {
    if (d == 0) return 1.0;
    double s = (i0 & 1) ? -1.0 : 1.0;
    if (i0 == 0) return 0.5;
    if (i0 == d) return 0.5 * s;
    return s;
}

// One dimension of interp_vals_bli, bli_module.f90:67-105: the exact-node
// test, then the second barycentric form normalised by its denominator.
__device__ __forceinline__ void bli_basis(double x, const double *nodes, int n, double *f) {
    bool found = false;
    for (int i = 0; i < n; ++i) {
        f[i] = 0.0;
        if (fabs(__dsub_rn(x, nodes[i])) < 1e-16) { found = true; f[i] = 1.0; }
    }
    if (!found) {
        double denom = 0.0;
        for (int i = 0; i < n; ++i) {
            double v = __ddiv_rn(bli_coeff(i, n - 1), __dsub_rn(x, nodes[i]));
            f[i] = v;
            denom = __dadd_rn(denom, v);
        }
        for (int i = 0; i < n; ++i) f[i] = __ddiv_rn(f[i], denom);
    }
}

// bli_basis for N = d + 1 nodes in registers, with fast_rcp for the divisions.
template <int N>
__device__ __forceinline__ void bli_basis_n(double x, const double *nodes, double (&f)[N]) {
    double denom = 0.0;
    int at = -1;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const double dx = __dsub_rn(x, nodes[i]);
        if (fabs(dx) < 1e-16) at = i;
        const double c = (i & 1 ? -1.0 : 1.0) * (i == 0 || i == N - 1 ? 0.5 : 1.0);
        f[i] = c * fast_rcp(dx);
        denom += f[i];
    }
    const double r = fast_rcp(denom);
#pragma unroll
    for (int i = 0; i < N; ++i) f[i] = at < 0 ? f[i] * r : (i == at ? 1.0 : 0.0);
}

// ----------------------------------------------------------------- argument blocks
struct EvalArgs {
    const double4 *pool;     // sources: points then source proxies, (x, y, z, w); leaf targets
    const EvalUnit *units;   // of this launch, one CTA each
    const EvalStage *stages;
    const EvalItem *items;
    const uint32_t *masks;
    const double4 *tgt_proxy;   // P target proxies per target slot
    int P;
    int kinds;               // leaf units: bit k set evaluates sources of kind k (0 points, 1 proxies)
    const int32_t *perm;     // pool position -> caller index
    double *out_x, *out_y;   // caller order, overwritten (leaf units with out < 0)
    double2 *leaf_part;      // leaf units' partial sums (x, y)
    double4 *proxy_part;     // proxy units' partial sums, P per unit
    int *err;
    uint32_t polls;          // poll limit of every staging wait (0: kDefaultPolls)
    int skip_last;           // fault injection: the last stage's copies of every leaf unit are not issued
};

struct FinArgs {
    const LeafFin *fin;
    const int32_t *down_slots;
    const double4 *pool;     // leaf targets
    const double2 *xieta;    // per pool position
    const double *records;   // DOWN records, rec_stride doubles each
    int rec_stride;
    const double2 *leaf_part;
    const int32_t *perm;
    double *out_x, *out_y;
};

struct UpArgs {
    const double4 *pool;
    const double2 *xieta;
    const UpUnit *units;
    const double *nodes;     // per source slot 2(d+1) nodes
    double *partial;         // P per unit
};

// launches (implemented in kernels.cu)
void launch_prep(const double4 *xyz, const double *area, const double *ssh, const int32_t *perm, int n, double4 *pool,
                 cudaStream_t st);
void launch_upward(const UpArgs &a, int d, int nunits, cudaStream_t st);
void launch_upward_finalize(const int32_t *unit_beg, const double *partial, int nslots, int d, int transposed,
                            double4 *pool_proxy, cudaStream_t st);
void launch_eval(int form, const EvalArgs &a, int nunits, cudaStream_t st);
void launch_leaf_fin(int form, int d, const FinArgs &a, int nfin, cudaStream_t st);
void launch_proxy_finalize(const int32_t *unit_beg, const double4 *partial, int nslots, int P, int rec_stride,
                           double *records, cudaStream_t st);
void launch_direct(const double *xs, const double *ys, const double *zs, const double *w, int n,
                   const int32_t *targets, int nt, double *out_x, double *out_y, double *scratch, int nchunks,
                   cudaStream_t st);
int direct_chunks(int n, int nt);
void launch_extract_w(const double4 *pool_proxy, int count, double *out, cudaStream_t st);
void launch_insert_w(const double *w, int count, double4 *pool_proxy, cudaStream_t st);

}  // namespace dev
}  // namespace sal
