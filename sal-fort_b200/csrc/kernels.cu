// FP64 kernels of the SAL-gradient treecode for sm_100a.
//
// All passes are compute-bound on the FP64 pipe: every staged source tile is
// reused by every target of its group (up to 256), so HBM traffic per pair is
// a few bytes against ~60 FP64 operations.
#include <cuda_runtime.h>

#include "kernels.cuh"

namespace sal {
namespace dev {

// ------------------------------------------------------------------ prep
// Per-solve source weights w = area * ssh in pool order (the factor
// area(j)*ssh(j) of fast_sum_module.f90:69-70).
__global__ void prep_kernel(const double4 *__restrict__ xyz, const double *__restrict__ area,
                            const double *__restrict__ ssh, const int32_t *__restrict__ perm, int n,
                            double4 *__restrict__ pool) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double4 p = xyz[i];
    p.w = area[i] * ssh[perm[i]];
    pool[i] = p;
}

void launch_prep(const double4 *xyz, const double *area, const double *ssh, const int32_t *perm, int n, double4 *pool,
                 cudaStream_t st) {
    if (n <= 0) return;
    prep_kernel<<<(n + 255) / 256, 256, 0, st>>>(xyz, area, ssh, perm, n, pool);
}

// ------------------------------------------------------------------ upward pass
// Proxy weights of one (source slot, chunk) unit: W[j + k N] = sum over the
// chunk's points of xi_basis_j * eta_basis_k * w (fast_sum_module.f90:99-111).
// The threads form the xi bases and the eta bases times w of a tile of points
// in shared memory; then thread (kb, g) adds three eta rows 3 kb.. of points
// g, g + 64, ...: N + 3 shared loads feed 3 N multiply-adds, and a warp's 32
// points are summed with shuffles once per unit.  Bound by the FP64 pipe and
// the shared loads together; the bases use fast_rcp (18 IEEE divisions a point
// at d = 8 were most of the pass).
constexpr int kUpTile = 128;
template <int N>
__global__ void __launch_bounds__(64 * ((N + 2) / 3)) upward_kernel(UpArgs a) {
    constexpr int KB = (N + 2) / 3, T = 64 * KB, P = N * N, NS = N | 1;   // odd row strides: no bank conflicts
    __shared__ double fx[kUpTile][NS];
    __shared__ double fe[kUpTile][NS];
    __shared__ double nod[2 * N];
    __shared__ double red[KB][2][3 * N];
    const UpUnit u = a.units[blockIdx.x];
    const int tid = threadIdx.x, kb = tid >> 6, g = tid & 63;
    if (tid < 2 * N) nod[tid] = a.nodes[(size_t)u.slot * 2 * N + tid];
    double acc[3][N];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int j = 0; j < N; ++j) acc[r][j] = 0.0;
    for (int b = u.beg; b < u.end; b += kUpTile) {
        const int m = min(kUpTile, u.end - b);
        __syncthreads();
        for (int e = tid; e < 2 * m; e += T) {
            const int s = e < m ? e : e - m;
            const double2 xe = a.xieta[b + s];
            const double w = e < m ? 1.0 : a.pool[b + s].w;
            double f[N];
            bli_basis_n<N>(e < m ? xe.x : xe.y, e < m ? nod : nod + N, f);
            double *o = e < m ? fx[s] : fe[s];
#pragma unroll
            for (int i = 0; i < N; ++i) o[i] = f[i] * w;
        }
        __syncthreads();
        for (int s = g; s < m; s += 64) {
            double h[3];
#pragma unroll
            for (int r = 0; r < 3; ++r) h[r] = 3 * kb + r < N ? fe[s][3 * kb + r] : 0.0;
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const double v = fx[s][j];
#pragma unroll
                for (int r = 0; r < 3; ++r) acc[r][j] = fma(v, h[r], acc[r][j]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int j = 0; j < N; ++j) {
            double v = acc[r][j];
#pragma unroll
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if ((tid & 31) == 0) red[kb][(tid >> 5) & 1][r * N + j] = v;
        }
    __syncthreads();
    for (int p = tid; p < P; p += T) {
        const int k = p / N, j = p % N;
        const double *q = red[k / 3][0] + (k % 3) * N + j;
        a.partial[(size_t)blockIdx.x * P + p] = q[0] + q[3 * N];
    }
}

// One instantiation per N = d + 1 from 2 to kMaxDegree + 1.
#define SAL_DEGREE_DISPATCH(fn, d, ...)                  \
    switch ((d) + 1) {                                   \
        case 2: fn<2>(__VA_ARGS__); break;               \
        case 3: fn<3>(__VA_ARGS__); break;               \
        case 4: fn<4>(__VA_ARGS__); break;               \
        case 5: fn<5>(__VA_ARGS__); break;               \
        case 6: fn<6>(__VA_ARGS__); break;               \
        case 7: fn<7>(__VA_ARGS__); break;               \
        case 8: fn<8>(__VA_ARGS__); break;               \
        case 9: fn<9>(__VA_ARGS__); break;               \
        case 10: fn<10>(__VA_ARGS__); break;             \
        case 11: fn<11>(__VA_ARGS__); break;             \
        case 12: fn<12>(__VA_ARGS__); break;             \
        case 13: fn<13>(__VA_ARGS__); break;             \
        case 14: fn<14>(__VA_ARGS__); break;             \
        case 15: fn<15>(__VA_ARGS__); break;             \
        default: break;                                  \
    }
static_assert(kMaxDegree + 1 == 15, "the dispatch covers every degree");

template <int N>
static void launch_upward_n(const UpArgs &a, int nunits, cudaStream_t st) {
    upward_kernel<N><<<nunits, 64 * ((N + 2) / 3), 0, st>>>(a);
}

void launch_upward(const UpArgs &a, int d, int nunits, cudaStream_t st) {
    if (nunits <= 0) return;
    SAL_DEGREE_DISPATCH(launch_upward_n, d, a, nunits, st)
}

// Sums each slot's unit partials in unit order into the w of its pool
// proxies.  transposed != 0 stores W[k + j n] at proxy j + k n, the layout
// mom6_fast_sum_module.f90:63-70 produces.
__global__ void upward_finalize_kernel(const int32_t *__restrict__ unit_beg, const double *__restrict__ partial,
                                       int nslots, int d, int transposed, double4 *__restrict__ pool_proxy) {
    const int n = d + 1, P = n * n;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nslots * P) return;
    const int s = (int)(t / P), p = (int)(t % P);
    const int j = p % n, k = p / n;
    const int src = transposed ? (k + j * n) : p;
    double acc = 0.0;
    for (int u = unit_beg[s]; u < unit_beg[s + 1]; ++u) acc += partial[(size_t)u * P + src];
    pool_proxy[(size_t)s * P + p].w = acc;
}

void launch_upward_finalize(const int32_t *unit_beg, const double *partial, int nslots, int d, int transposed,
                            double4 *pool_proxy, cudaStream_t st) {
    long long tot = (long long)nslots * (d + 1) * (d + 1);
    if (tot <= 0) return;
    upward_finalize_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(unit_beg, partial, nslots, d, transposed,
                                                                          pool_proxy);
}

// ------------------------------------------------------------------ targets x staged sources
// One CTA per unit: the targets of a leaf, or a target slot's proxies, against
// the unit's stages.  A stage is up to 256 sources gathered from up to 32 pool
// ranges; lane i of warp 0 copies range i (one bulk copy each, completing on
// the stage's mbarrier) into a ring of kRing buffers, two stages ahead, so a
// warp that is through with a stage goes on without a CTA-wide barrier.
// Targets and source splits fill the threads without gaps: thread tid has
// target tid % nt and sources tid / nt, tid / nt + nsplit, ...; the splits are
// summed in a fixed order at the end, so results are deterministic.  Stages
// are near (gref_near: the reference's operation order where its rounding
// noise counts) or far (gref_far).
//   Leaf units and FORM 0 proxies: the reference kernel.  FORM 1 proxies: the
//   Cartesian sum val (s - x) w with the antipode-stable val.
// Bound by the FP64 pipe (two cycles an instruction and warp on each of the
// four schedulers).
constexpr int kEvalThreads = 256, kEvalCtas = 3, kIlp = 2, kNearIlp = 2, kRing = 4, kAhead = 2;

template <int FORM>
__global__ void __launch_bounds__(kEvalThreads, kEvalCtas) eval_kernel(EvalArgs a) {
    __shared__ __align__(128) double4 buf[kRing][kMaxStage];
    __shared__ __align__(8) uint64_t full[kRing], empty[kRing];
    __shared__ int abort_;
    volatile int *abort = &abort_;
    const EvalUnit U = a.units[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nt = U.nt, nsplit = kEvalThreads / nt;
    const int ti = tid % nt, sp = tid / nt;
    const bool active = sp < nsplit;
    const bool cart = FORM == 1 && U.proxy;
    const int sb = (U.proxy || (a.kinds & 1)) ? U.sb : U.sm, se = (U.proxy || (a.kinds & 2)) ? U.se : U.sm;
    const int ns = se - sb;
    const uint32_t polls = a.polls ? a.polls : kDefaultPolls;
    const int nissue = (a.skip_last && !U.proxy) ? ns - 1 : ns;
    Tgt T;
    double mt[3] = {0.0, 0.0, 0.0};
    if (active) {
        const double4 c = U.proxy ? a.tgt_proxy[(size_t)U.tgt * a.P + ti] : a.pool[U.tgt + ti];
        tgt_init(T, c.x, c.y, c.z);
    } else {
        tgt_init(T, 0.0, 0.0, 0.5);
        T.live = false;
    }
    mt[0] = -2.0 * T.x;
    mt[1] = -2.0 * T.y;
    mt[2] = -2.0 * T.z;
    const bool work = active && (T.live || cart);
    if (tid == 0) {
        for (int i = 0; i < kRing; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], kEvalThreads / 32);
        }
        fence_mbar_init();
        abort_ = 0;
    }
    __syncthreads();
    // warp 0: stage k's copies, once every warp is through with the stage that
    // last used its buffer.  Nothing is issued after a wait gave up.
    int issued = 0;
    auto issue = [&](int k) {
        const int b = k % kRing;
        if (k >= kRing && !*abort &&
            !mbar_wait_bounded(&empty[b], (uint32_t)((k / kRing - 1) & 1), a.err, kDefaultPolls))
            *abort = 1;
        // fault injection (tests of the time-out path): the unit's last stage
        // is never issued, so its wait runs out with no copy in flight
        if (__any_sync(0xffffffffu, k >= nissue || *abort)) return;
        issued = k + 1;
        fence_proxy_async();
        const EvalStage S = a.stages[sb + k];
        if (lane == 0) mbar_expect_tx(&full[b], (uint32_t)S.cnt * 32u);
        __syncwarp();
        if (lane < S.ie - S.ib) {
            const EvalItem it = a.items[S.ib + lane];
            bulk_g2s(&buf[b][it.dst], a.pool + it.off, (uint32_t)it.cnt * 32u, &full[b]);
        }
        __syncwarp();
    };
    if (warp == 0)
        for (int k = 0; k < kAhead && k < ns; ++k) issue(k);
    double A[3] = {0.0, 0.0, 0.0};   // far pairs: Sum val w s; Cartesian proxies: Sum val w (s - x)
    double ax = 0.0, ay = 0.0;       // near pairs
    for (int k = 0; k < ns; ++k) {
        if (warp == 0 && k + kAhead < ns) issue(k + kAhead);
        const int b = k % kRing;
        const EvalStage S = a.stages[sb + k];
        if (!*abort && !mbar_wait_bounded(&full[b], (uint32_t)((k / kRing) & 1), a.err, polls)) *abort = 1;
        const double4 *src = buf[b];
        // several pairs at a time: independent chains
        auto range = [&](int beg, int end) {
            int s = beg + sp;
            if (cart) {
                for (; s < end; s += nsplit) {
                    const double4 q = src[s];
                    const double dx = q.x - T.x, dy = q.y - T.y, dz = q.z - T.z;
                    const double v = vstable(fma(dx, dx, fma(dy, dy, dz * dz))) * q.w;
                    A[0] = fma(v, dx, A[0]);
                    A[1] = fma(v, dy, A[1]);
                    A[2] = fma(v, dz, A[2]);
                }
            } else if (S.flags & kEvalNear) {
                for (; s + (kNearIlp - 1) * nsplit < end; s += kNearIlp * nsplit) gref_near<kNearIlp>(T, src + s, nsplit, ax, ay);
                for (; s < end; s += nsplit) gref_near<1>(T, src + s, nsplit, ax, ay);
            } else {
                for (; s + (kIlp - 1) * nsplit < end; s += kIlp * nsplit) {
#pragma unroll
                    for (int u = 0; u < kIlp; ++u) gref_far(mt, src[s + u * nsplit], A);
                }
                for (; s < end; s += nsplit) gref_far(mt, src[s], A);
            }
        };
        if (!(S.flags & kEvalMasked)) {
            if (work) range(0, S.cnt);
        } else {
            for (int i = S.ib; i < S.ie; ++i) {
                const EvalItem it = a.items[i];
                if (work && ((a.masks[it.mask + (ti >> 5)] >> (ti & 31)) & 1u)) range(it.dst, it.dst + it.cnt);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[b]);
    }
    // the kernel's constant; leaves and reference proxies: the projection of
    // the far pairs' vector and the target factor 1/sqrt(1 - tz^2) (zero
    // inside the pole guard)
    if (cart) {
        ax = kCons * A[0];
        ay = kCons * A[1];
        A[2] *= kCons;
    } else {
        const double tf = T.live ? kCons * T.inv_mp2 : 0.0;
        ax = tf * (ax + (T.x * A[1] - T.y * A[0]));
        ay = tf * (ay + (T.omx32 * A[2] - T.z * (T.x * A[0] + T.y * A[1])));
        A[2] = 0.0;
    }
    __syncthreads();   // every stage is consumed: the ring holds the reduction
    double *red = reinterpret_cast<double *>(buf);
    if (active) {
        red[3 * tid] = ax;
        red[3 * tid + 1] = ay;
        red[3 * tid + 2] = A[2];
    }
    if (*abort && tid == 0) {
        // a wait gave up: copies still in flight get a last bounded wait
        // before their buffers go (their values are lost anyway)
        for (int k = max(0, issued - kRing); k < issued; ++k)
            mbar_wait_bounded(&full[k % kRing], (uint32_t)((k / kRing) & 1), a.err, kDefaultPolls);
    }
    __syncthreads();
    if (active && sp == 0) {
        double rx = 0.0, ry = 0.0, rz = 0.0;
        for (int s = 0; s < nsplit; ++s) {
            rx += red[3 * (s * nt + ti)];
            ry += red[3 * (s * nt + ti) + 1];
            rz += red[3 * (s * nt + ti) + 2];
        }
        if (U.proxy) {
            a.proxy_part[(size_t)U.out * a.P + ti] = make_double4(rx, ry, rz, 0.0);
        } else if (U.out >= 0) {
            a.leaf_part[(size_t)U.out + ti] = make_double2(rx, ry);
        } else {
            const int idx = a.perm[U.tgt + ti];
            a.out_x[idx] = rx;
            a.out_y[idx] = ry;
        }
    }
}
static_assert(sizeof(double) * 3 * kEvalThreads <= sizeof(double4) * kRing * kMaxStage, "the reduction fits the ring");

void launch_eval(int form, const EvalArgs &a, int nunits, cudaStream_t st) {
    if (nunits <= 0) return;
    if (form == 0) eval_kernel<0><<<nunits, kEvalThreads, 0, st>>>(a);
    else eval_kernel<1><<<nunits, kEvalThreads, 0, st>>>(a);
}

// ------------------------------------------------------------------ leaf ends
// One CTA per leaf: its units' partial sums in unit order, plus the
// interpolation of its target slots' proxy potentials (interp_vals_bli and
// the loops of fast_sum_module.f90:186-199).  FORM 0 interpolates east/north
// components, FORM 1 the Cartesian vector, projected on the target's frame.
// Thread tid has target tid % nt and the eta rows tid / nt, + nsplit, ... of
// every slot, whose record (potentials, nodes) the CTA copies to shared
// memory.
constexpr int kFinThreads = 256;
template <int N, int FORM>
__global__ void __launch_bounds__(kFinThreads) leaf_fin_kernel(FinArgs a) {
    constexpr int P = N * N;
    __shared__ double4 rec[P + (2 * N + 3) / 4];
    __shared__ double red[3][kFinThreads];
    const LeafFin L = a.fin[blockIdx.x];
    const int tid = threadIdx.x, nt = L.nt, nsplit = kFinThreads / nt, ti = tid % nt, sp = tid / nt;
    const bool active = sp < nsplit;
    const double2 xe = active ? a.xieta[L.tgt + ti] : make_double2(0.0, 0.0);
    double ux = 0.0, uy = 0.0, uz = 0.0;
    for (int e = L.db; e < L.de; ++e) {
        const double4 *src = reinterpret_cast<const double4 *>(a.records + (size_t)a.down_slots[e] * a.rec_stride);
        __syncthreads();
        for (int i = tid; i < a.rec_stride / 4; i += kFinThreads) rec[i] = src[i];
        __syncthreads();
        if (active) {
            const double *nodes = reinterpret_cast<const double *>(rec + P);
            double fx[N], fe[N];
            bli_basis_n<N>(xe.x, nodes, fx);
            bli_basis_n<N>(xe.y, nodes + N, fe);
            int turn = sp;   // eta row k is this thread's when turn is 0
#pragma unroll
            for (int k = 0; k < N; ++k) {
                if (turn == 0) {
                    double rx = 0.0, ry = 0.0, rz = 0.0;
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        const double4 ph = rec[j + k * N];
                        rx = fma(fx[j], ph.x, rx);
                        ry = fma(fx[j], ph.y, ry);
                        if (FORM == 1) rz = fma(fx[j], ph.z, rz);
                    }
                    ux = fma(fe[k], rx, ux);
                    uy = fma(fe[k], ry, uy);
                    if (FORM == 1) uz = fma(fe[k], rz, uz);
                    turn = nsplit;
                }
                --turn;
            }
        }
    }
    red[0][tid] = ux;
    red[1][tid] = uy;
    if (FORM == 1) red[2][tid] = uz;
    __syncthreads();
    if (!active || sp != 0) return;
    for (int s = 1; s < nsplit; ++s) {
        ux += red[0][s * nt + ti];
        uy += red[1][s * nt + ti];
        if (FORM == 1) uz += red[2][s * nt + ti];
    }
    if (FORM == 1) {
        const double4 c = a.pool[L.tgt + ti];
        Tgt T;
        tgt_init(T, c.x, c.y, c.z);
        const double tf = T.live ? T.inv_mp2 : 0.0;
        const double ex = (T.x * uy - T.y * ux) * tf;
        uy = (uz * T.omx32 - T.z * (T.x * ux + T.y * uy)) * tf;
        ux = ex;
    }
    for (int k = 0; k < L.parts; ++k) {
        const double2 v = a.leaf_part[(size_t)L.part + (size_t)k * nt + ti];
        ux += v.x;
        uy += v.y;
    }
    const int idx = a.perm[L.tgt + ti];
    a.out_x[idx] = ux;
    a.out_y[idx] = uy;
}

template <int N>
static void launch_leaf_fin_n(int form, const FinArgs &a, int nfin, cudaStream_t st) {
    if (form == 0) leaf_fin_kernel<N, 0><<<nfin, kFinThreads, 0, st>>>(a);
    else leaf_fin_kernel<N, 1><<<nfin, kFinThreads, 0, st>>>(a);
}

void launch_leaf_fin(int form, int d, const FinArgs &a, int nfin, cudaStream_t st) {
    if (nfin <= 0) return;
    SAL_DEGREE_DISPATCH(launch_leaf_fin_n, d, form, a, nfin, st)
}

// Sums each target slot's unit partials in unit order into its record.
__global__ void proxy_finalize_kernel(const int32_t *__restrict__ unit_beg, const double4 *__restrict__ partial,
                                      int nslots, int P, int rec_stride, double *__restrict__ records) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nslots * P) return;
    const int s = (int)(t / P), p = (int)(t % P);
    double x = 0.0, y = 0.0, z = 0.0;
    for (int u = unit_beg[s]; u < unit_beg[s + 1]; ++u) {
        const double4 v = partial[(size_t)u * P + p];
        x += v.x;
        y += v.y;
        z += v.z;
    }
    double4 *rec = reinterpret_cast<double4 *>(records + (size_t)s * rec_stride);
    rec[p] = make_double4(x, y, z, 0.0);
}

void launch_proxy_finalize(const int32_t *unit_beg, const double4 *partial, int nslots, int P, int rec_stride,
                           double *records, cudaStream_t st) {
    long long tot = (long long)nslots * P;
    if (tot <= 0) return;
    proxy_finalize_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(unit_beg, partial, nslots, P, rec_stride,
                                                                         records);
}

// ------------------------------------------------------------------ direct sum
// FP64 direct O(N^2) sum at sampled targets with the reference kernel, sources
// split into chunks (blockIdx.y) whose partial sums are added in chunk order.
constexpr int kDirectTile = 128;
__global__ void __launch_bounds__(kDirectTile) direct_kernel(const double *__restrict__ xs, const double *__restrict__ ys,
                                                             const double *__restrict__ zs, const double *__restrict__ w,
                                                             int n, const int32_t *__restrict__ targets, int nt,
                                                             int chunk, double *__restrict__ partial) {
    __shared__ double4 S[kDirectTile];
    const int k = blockIdx.x * kDirectTile + threadIdx.x;
    const int s0 = blockIdx.y * chunk, s1 = min(n, s0 + chunk);
    Tgt T;
    if (k < nt) {
        const int ti = targets[k];
        tgt_init(T, xs[ti], ys[ti], zs[ti]);
    } else {
        tgt_init(T, 0.0, 0.0, 0.5);
        T.live = false;
    }
    double ax = 0.0, ay = 0.0;
    for (int b = s0; b < s1; b += kDirectTile) {
        const int m = min(kDirectTile, s1 - b);
        if (threadIdx.x < m) {
            const int s = b + threadIdx.x;
            S[threadIdx.x] = make_double4(xs[s], ys[s], zs[s], w[s]);
        }
        __syncthreads();
        if (T.live)
            for (int s = 0; s < m; ++s) {
                double gx, gy;
                gref_exact(T, S[s].x, S[s].y, S[s].z, gx, gy);
                ax += gx * S[s].w;
                ay += gy * S[s].w;
            }
        __syncthreads();
    }
    if (k < nt) {
        partial[((size_t)blockIdx.y * nt + k) * 2] = ax;
        partial[((size_t)blockIdx.y * nt + k) * 2 + 1] = ay;
    }
}

__global__ void direct_reduce_kernel(const double *__restrict__ partial, int nt, int nchunks, double *__restrict__ ox,
                                     double *__restrict__ oy) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nt) return;
    double x = 0.0, y = 0.0;
    for (int c = 0; c < nchunks; ++c) {
        x += partial[((size_t)c * nt + k) * 2];
        y += partial[((size_t)c * nt + k) * 2 + 1];
    }
    ox[k] = x;
    oy[k] = y;
}

int direct_chunks(int n) { return max(1, min(64, (n + 32767) / 32768)); }

void launch_direct(const double *xs, const double *ys, const double *zs, const double *w, int n,
                   const int32_t *targets, int nt, double *out_x, double *out_y, double *scratch, int nchunks,
                   cudaStream_t st) {
    if (nt <= 0) return;
    const int chunk = (n + nchunks - 1) / nchunks;
    dim3 grid((nt + kDirectTile - 1) / kDirectTile, nchunks);
    direct_kernel<<<grid, kDirectTile, 0, st>>>(xs, ys, zs, w, n, targets, nt, chunk, scratch);
    direct_reduce_kernel<<<(nt + 255) / 256, 256, 0, st>>>(scratch, nt, nchunks, out_x, out_y);
}

// ------------------------------------------------------------------ proxy weight transfer
__global__ void extract_w_kernel(const double4 *__restrict__ pp, int count, double *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) out[i] = pp[i].w;
}
__global__ void insert_w_kernel(const double *__restrict__ w, int count, double4 *__restrict__ pp) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) pp[i].w = w[i];
}
void launch_extract_w(const double4 *pool_proxy, int count, double *out, cudaStream_t st) {
    if (count > 0) extract_w_kernel<<<(count + 255) / 256, 256, 0, st>>>(pool_proxy, count, out);
}
void launch_insert_w(const double *w, int count, double4 *pool_proxy, cudaStream_t st) {
    if (count > 0) insert_w_kernel<<<(count + 255) / 256, 256, 0, st>>>(w, count, pool_proxy);
}

}  // namespace dev
}  // namespace sal
