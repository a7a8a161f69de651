// FP64 kernels of the SAL-gradient treecode for sm_100a.
//
// All passes are compute-bound on the FP64 pipe: every staged source tile is
// reused by every target of its group (up to 256), so HBM traffic per pair is
// a few bytes against 20 FP64 instructions (far pairs) or 27 (near ones).
#include <cmath>
#include <cuda_runtime.h>

#include "eval_cut.hpp"
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
    after_previous();
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
    launch_next(upward_kernel<N>, nunits, 64 * ((N + 2) / 3), 0, st, a);
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
    after_previous();
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
    launch_next(upward_finalize_kernel, (unsigned)((tot + 255) / 256), 256, 0, st, unit_beg, partial, nslots, d, transposed,
                                                                          pool_proxy);
}

// ------------------------------------------------------------------ targets x staged sources
// One CTA per unit: the targets of a leaf, or a target slot's proxies, against
// the unit's stages.  A stage is up to 256 sources gathered from up to 32 pool
// ranges; lane i of warp 0 copies range i (one bulk copy each, completing on
// the stage's mbarrier) into a ring of kRing buffers, two stages ahead, so a
// warp that is through with a stage goes on without a CTA-wide barrier.
// Every warp has the same share of the unit's pairs: each target is taken F
// times, each time for one residue of the sources mod F (F from the plan, so
// that the nt F lanes fill up to one chunk of 32 lanes a warp with little
// waste), and a last chunk of m <= 16 lanes takes 32 / m residues more.  The
// (chunk, source) plane is cut into one equal run per warp: a fraction of the
// sources of at most two chunks, the same ones in every stage, whose sums the
// warp keeps (eval_cut.hpp).  (One thread per target and whole source splits
// left a leaf of 148 targets with 5 of 8 warps at work, two of them on one
// scheduler: 62 % of the FP64 pipe.)  The sums are added in a fixed order at the
// end, so results are deterministic.  Stages are near (gref_near: the reference's
// operation order where its rounding noise counts) or far (gref_far).
//   Leaf units and FORM 0 proxies: the reference kernel.  FORM 1 proxies: the
//   Cartesian sum val (s - x) w with the antipode-stable val.
// Bound by the FP64 pipe: an instruction with three register operands takes
// about 2.5 cycles of a scheduler's pipe (50 for a far pair's 20, in a loop of
// nothing else), and 8 pairs at a time on 4 warps a scheduler come closest to
// that (24 warps of 80 registers and 4 pairs: 3 % slower).
constexpr int kEvalThreads = 256, kEvalCtas = 2, kIlp = 8, kNearIlp = 4, kRing = 4, kAhead = 2;
constexpr int kSlots = kEvalSlots;
static_assert(kEvalWarps == kEvalThreads / 32, "eval_cut.hpp deals to the warps of a CTA");

// The far pairs of one lane once more, pair by pair as the near ones: for sums
// that are not finite.  The vector of gref_far turns an infinite weight, or one
// whose products overflow, into NaN at its projection, where the pair itself is
// a signed infinity or finite.  From the pool, nothing staged; a sum that is NaN
// already (a NaN weight) stays so and ends it.
__device__ __noinline__ void far_again(const double4 *pool, const EvalStage *stages, const EvalItem *items,
                                       const uint32_t *masks, int sb, int se, const EvalShare &sh, double x, double y,
                                       double z, double &ax, double &ay) {
    Tgt T;
    T.x = x;
    T.y = y;
    T.z = z;
    T.omx32 = tgt_omx32(z);
    for (int k = sb; k < se; ++k) {
        const EvalStage S = stages[k];
        if (S.flags & kEvalNear) continue;
        int s = 0, e = 0;
        for (int v = S.ib; v < S.ie; ++v) {
            const EvalItem it = items[v];
            if (S.flags & kEvalMasked) {
                if (!((masks[it.mask + (sh.ti >> 5)] >> (sh.ti & 31)) & 1u)) continue;
                sh.sources(it.cnt, s, e);
                s += it.dst;
                e += it.dst;
            } else if (v == S.ib) {
                sh.sources(S.cnt, s, e);
            }
            for (; s < min(e, it.dst + it.cnt); s += sh.step) gref_near<1>(T, pool + it.off + (s - it.dst), 1, ax, ay);
        }
        if (ax != ax && ay != ay) return;
    }
}

template <int FORM>
__global__ void __launch_bounds__(kEvalThreads, kEvalCtas) eval_kernel(EvalArgs a) {
    after_previous();
    __shared__ __align__(128) double4 buf[kRing][kMaxStage];
    __shared__ __align__(8) uint64_t full[kRing], empty[kRing];
    __shared__ int abort_;
    volatile int *abort = &abort_;
    const EvalUnit U = a.units[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool cart = FORM == 1 && U.proxy;
    const int sb = (U.proxy || (a.kinds & 1)) ? U.sb : U.sm, se = (U.proxy || (a.kinds & 2)) ? U.se : U.sm;
    const int ns = se - sb;
    const uint32_t polls = a.polls ? a.polls : kDefaultPolls;
    const int nissue = (a.skip_last && !U.proxy) ? ns - 1 : ns;
    const EvalCut cut(U.nt, U.fold);
    // the slots' state; a stage's range takes one slot into registers
    struct Slot {
        double x, y, z;            // the target
        double A[3], ax, ay;       // sums: far pairs Sum val w s (Cartesian proxies Sum val w (s - x)); near pairs
        EvalShare sh;              // the lane's sources
        bool work;
    } slot[kSlots];
#pragma unroll 1
    for (int i = 0; i < kSlots; ++i) {
        Slot w{};
        w.sh = eval_share(cut, warp, lane, i);
        if (w.sh.work) {
            const double4 q = U.proxy ? a.tgt_proxy[(size_t)U.tgt * a.P + w.sh.ti] : a.pool[U.tgt + w.sh.ti];
            w.x = q.x;
            w.y = q.y;
            w.z = q.z;
            w.work = cart || tgt_live(q.z);
        }
        slot[i] = w;
    }
    if (tid == 0) {
        for (int i = 0; i < kRing; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], kEvalWarps);
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
    for (int k = 0; k < ns; ++k) {
        if (warp == 0 && k + kAhead < ns) issue(k + kAhead);
        const int b = k % kRing;
        const EvalStage S = a.stages[sb + k];
        if (!*abort && !mbar_wait_bounded(&full[b], (uint32_t)((k / kRing) & 1), a.err, polls)) *abort = 1;
        const double4 *src = buf[b];
        const bool near = S.flags & kEvalNear, masked = S.flags & kEvalMasked;
#pragma unroll 1
        for (int i = 0; i < kSlots; ++i) {
            if (!slot[i].work) continue;
            const double x = slot[i].x, y = slot[i].y, z = slot[i].z;
            const EvalShare sh = slot[i].sh;
            const int step = sh.step;
            double A[3] = {slot[i].A[0], slot[i].A[1], slot[i].A[2]}, ax = slot[i].ax, ay = slot[i].ay;
            // an unmasked stage is one run of sources, a masked one a run per item
#pragma unroll 1
            for (int v = masked ? S.ib : S.ie - 1; v < S.ie; ++v) {
                int beg = 0, n = S.cnt;
                if (masked) {
                    const EvalItem it = a.items[v];
                    if (!((a.masks[it.mask + (sh.ti >> 5)] >> (sh.ti & 31)) & 1u)) continue;
                    beg = it.dst;
                    n = it.cnt;
                }
                // this run's share of the blocks of `step` sources
                int s, e;
                sh.sources(n, s, e);
                s += beg;
                e += beg;
                if (cart) {
                    for (; s + (kNearIlp - 1) * step < e; s += kNearIlp * step)
                        cart_pairs<kNearIlp>(x, y, z, src + s, step, A);
                    for (; s < e; s += step) cart_pairs<1>(x, y, z, src + s, step, A);
                } else if (near) {
                    Tgt T;
                    T.x = x;
                    T.y = y;
                    T.z = z;
                    T.omx32 = tgt_omx32(z);
                    for (; s + (kNearIlp - 1) * step < e; s += kNearIlp * step) gref_near<kNearIlp>(T, src + s, step, ax, ay);
                    for (; s < e; s += step) gref_near<1>(T, src + s, step, ax, ay);
                } else {
                    // several pairs at a time: independent chains
                    const double mt[3] = {-2.0 * x, -2.0 * y, -2.0 * z};
                    for (; s + (kIlp - 1) * step < e; s += kIlp * step) gref_far<kIlp>(mt, src + s, step, A);
                    if (s + (kIlp / 2 - 1) * step < e) {
                        gref_far<kIlp / 2>(mt, src + s, step, A);
                        s += kIlp / 2 * step;
                    }
                    for (; s < e; s += step) gref_far<1>(mt, src + s, step, A);
                }
            }
            slot[i].A[0] = A[0];
            slot[i].A[1] = A[1];
            slot[i].A[2] = A[2];
            slot[i].ax = ax;
            slot[i].ay = ay;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[b]);
    }
    __syncthreads();   // every stage is consumed: the ring holds the warps' sums
    double *red = reinterpret_cast<double *>(buf);   // [warp][slot][component][lane]
#pragma unroll 1
    for (int i = 0; i < kSlots; ++i) {
        // the kernel's constant; leaves and reference proxies: the projection
        // of the far pairs' vector and the target factor 1/sqrt(1 - tz^2)
        // (zero inside the pole guard, and in slots without work)
        Slot &w = slot[i];
        double rx = 0.0, ry = 0.0, rz = 0.0;
        if (cart) {
            rx = kCons * w.A[0];
            ry = kCons * w.A[1];
            rz = kCons * w.A[2];
        } else if (w.work) {
            if (!(fabs(w.A[0]) + fabs(w.A[1]) + fabs(w.A[2]) < INFINITY)) {
                w.A[0] = w.A[1] = w.A[2] = 0.0;
                far_again(a.pool, a.stages, a.items, a.masks, sb, se, w.sh, w.x, w.y, w.z, w.ax, w.ay);
            }
            Tgt T;
            tgt_init(T, w.x, w.y, w.z);
            const double tf = kCons * T.inv_mp2;
            rx = tf * (w.ax + (T.x * w.A[1] - T.y * w.A[0]));
            ry = tf * (w.ay + (T.omx32 * w.A[2] - T.z * (T.x * w.A[0] + T.y * w.A[1])));
        }
        double *o = red + ((warp * kSlots + i) * 3) * 32 + lane;
        o[0] = rx;
        o[32] = ry;
        o[64] = rz;
    }
    if (*abort && tid == 0) {
        // a wait gave up: copies still in flight get a last bounded wait
        // before their buffers go (their values are lost anyway)
        for (int k = max(0, issued - kRing); k < issued; ++k)
            mbar_wait_bounded(&full[k % kRing], (uint32_t)((k / kRing) & 1), a.err, kDefaultPolls);
    }
    __syncthreads();
    // lane tid of the folded set: the warps whose runs meet its chunk, in
    // order; then each target's F lanes, in order
    double *fold = red + 3 * 32 * kSlots * kEvalWarps;
    double rx = 0.0, ry = 0.0, rz = 0.0;
    if (tid < cut.nid) {
        const int c = tid >> 5, n = c == cut.nch - 1 ? cut.nlast : 32, r = c == cut.nch - 1 ? cut.rlast : 1;
        for (int v = 0; v < kEvalWarps; ++v) {
            const int i = cut.slot_of(v, c);
            if (i < 0 || i >= kSlots) continue;
            const double *o = red + ((v * kSlots + i) * 3) * 32 + lane;
            for (int k = 0; k < r; ++k) {
                rx += o[k * n];
                ry += o[k * n + 32];
                rz += o[k * n + 64];
            }
        }
    }
    if (U.fold > 1) {
        fold[tid] = rx;
        fold[kEvalThreads + tid] = ry;
        fold[2 * kEvalThreads + tid] = rz;
        __syncthreads();
        if (tid < U.nt)
            for (int id = tid + U.nt; id < cut.nid; id += U.nt) {
                rx += fold[id];
                ry += fold[kEvalThreads + id];
                rz += fold[2 * kEvalThreads + id];
            }
    }
    if (tid < U.nt) {
        if (U.proxy) {
            a.proxy_part[(size_t)U.out * a.P + tid] = make_double4(rx, ry, rz, 0.0);
        } else if (U.out >= 0) {
            a.leaf_part[(size_t)U.out + tid] = make_double2(rx, ry);
        } else {
            const int idx = a.perm[U.tgt + tid];
            a.out_x[idx] = rx;
            a.out_y[idx] = ry;
        }
    }
}
static_assert(sizeof(double) * 3 * (kSlots + 1) * kEvalThreads <= sizeof(double4) * kRing * kMaxStage,
              "the warps' sums and the folded lanes' fit the ring");
static_assert(32 * kEvalMaxChunks <= kEvalThreads, "a thread per lane of the folded set");
static_assert(kEvalThreads >= kMaxStage, "a thread per target at the end (leaves and proxy sets hold at most 256)");

void launch_eval(int form, const EvalArgs &a, int nunits, cudaStream_t st) {
    if (nunits <= 0) return;
    if (form == 0) launch_next(eval_kernel<0>, nunits, kEvalThreads, 0, st, a);
    else launch_next(eval_kernel<1>, nunits, kEvalThreads, 0, st, a);
}

// ------------------------------------------------------------------ leaf ends
// One CTA per leaf: its units' partial sums in unit order, plus the
// interpolation of its target slots' proxy potentials (interp_vals_bli and
// the loops of fast_sum_module.f90:186-199).  FORM 0 interpolates east/north
// components, FORM 1 the Cartesian vector, projected on the target's frame.
// The records (potentials, nodes) of up to kFinSlots slots come to shared
// memory at a time; thread tid has target tid % nt and every (256 / nt)-th
// (slot, eta row) of them, so that small leaves' slots run side by side.
constexpr int kFinThreads = 256, kFinSlots = 4;
template <int N, int FORM>
__global__ void __launch_bounds__(kFinThreads) leaf_fin_kernel(FinArgs a) {
    after_previous();
    constexpr int P = N * N, R = P + (2 * N + 3) / 4;   // double4 per record
    __shared__ double4 rec[kFinSlots][R];
    __shared__ double red[3][kFinThreads];
    const LeafFin L = a.fin[blockIdx.x];
    const int tid = threadIdx.x, nt = L.nt, nsplit = kFinThreads / nt, ti = tid % nt, sp = tid / nt;
    const bool active = sp < nsplit;
    const double2 xe = active ? a.xieta[L.tgt + ti] : make_double2(0.0, 0.0);
    double ux = 0.0, uy = 0.0, uz = 0.0;
    for (int e0 = L.db; e0 < L.de; e0 += kFinSlots) {
        const int ne = min(kFinSlots, L.de - e0);
        __syncthreads();
        for (int i = tid; i < ne * R; i += kFinThreads)
            rec[i / R][i % R] = reinterpret_cast<const double4 *>(
                a.records + (size_t)a.down_slots[e0 + i / R] * a.rec_stride)[i % R];
        __syncthreads();
        if (!active) continue;
        int turn = sp;   // the next (slot, eta row) is this thread's when turn is 0
        for (int e = 0; e < ne; ++e) {
            if (turn >= N) {   // none of this slot's rows
                turn -= N;
                continue;
            }
            const double4 *rc = rec[e];
            const double *nodes = reinterpret_cast<const double *>(rc + P);
            double fx[N], fe[N];
            bli_basis_n<N>(xe.x, nodes, fx);
            bli_basis_n<N>(xe.y, nodes + N, fe);
#pragma unroll
            for (int k = 0; k < N; ++k) {
                if (turn == 0) {
                    double rx = 0.0, ry = 0.0, rz = 0.0;
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        const double4 ph = rc[j + k * N];
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
    if (form == 0) launch_next(leaf_fin_kernel<N, 0>, nfin, kFinThreads, 0, st, a);
    else launch_next(leaf_fin_kernel<N, 1>, nfin, kFinThreads, 0, st, a);
}

void launch_leaf_fin(int form, int d, const FinArgs &a, int nfin, cudaStream_t st) {
    if (nfin <= 0) return;
    SAL_DEGREE_DISPATCH(launch_leaf_fin_n, d, form, a, nfin, st)
}

// Sums each target slot's unit partials in unit order into its record.
__global__ void proxy_finalize_kernel(const int32_t *__restrict__ unit_beg, const double4 *__restrict__ partial,
                                      int nslots, int P, int rec_stride, double *__restrict__ records) {
    after_previous();
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
    launch_next(proxy_finalize_kernel, (unsigned)((tot + 255) / 256), 256, 0, st, unit_beg, partial, nslots, P, rec_stride,
                                                                         records);
}

// ------------------------------------------------------------------ direct sum
// FP64 direct O(N^2) sum at sampled targets with the reference kernel: one
// target per thread, sources staged through shared memory, gref_near 4 pairs
// at a time (g in the reference's operation order, val_ref for the self pair
// and the other pairs whose value is rounding noise).  Bound by the FP64 pipe:
// 27 instructions a pair (10,000 targets x 655,362 sources: 12.3 ms, 71 cycles
// a pair and scheduler of the 68 that a loop of nothing else takes), where
// IEEE division and square root took about 110 (31.4 ms).  The sources are split into
// chunks (blockIdx.y) whose partial sums are added in a fixed order.
constexpr int kDirectThreads = 128, kDirectTile = 256, kDirectCtas = 5, kDirectIlp = 4;
__global__ void __launch_bounds__(kDirectThreads, kDirectCtas)
    direct_kernel(const double *__restrict__ xs, const double *__restrict__ ys, const double *__restrict__ zs,
                  const double *__restrict__ w, int n, const int32_t *__restrict__ targets, int nt, int chunk,
                  double *__restrict__ partial) {
    __shared__ __align__(16) double4 S2[2][kDirectTile];
    const int k = blockIdx.x * kDirectThreads + threadIdx.x;
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
    // the next tile is copied (8 bytes at a time: the four arrays have no other
    // common alignment) while this one is summed
    auto fetch = [&](int b, int buf) {
        for (int i = threadIdx.x; i < min(kDirectTile, s1 - b); i += kDirectThreads) {
            double *o = reinterpret_cast<double *>(&S2[buf][i]);
            cp_async8(o, xs + b + i);
            cp_async8(o + 1, ys + b + i);
            cp_async8(o + 2, zs + b + i);
            cp_async8(o + 3, w + b + i);
        }
        cp_async_commit();
    };
    fetch(s0, 0);
    int buf = 0;
    for (int b = s0; b < s1; b += kDirectTile, buf ^= 1) {
        cp_async_wait_all();
        __syncthreads();   // this tile is here, and every warp is through with the other buffer
        if (b + kDirectTile < s1) fetch(b + kDirectTile, buf ^ 1);
        if (T.live) {
            const double4 *S = S2[buf];
            const int m = min(kDirectTile, s1 - b);
            int s = 0;
            for (; s + kDirectIlp <= m; s += kDirectIlp) gref_near<kDirectIlp>(T, S + s, 1, ax, ay);
            for (; s < m; ++s) gref_near<1>(T, S + s, 1, ax, ay);
        }
    }
    cp_async_wait_all();
    if (k < nt) {
        const double tf = T.live ? kCons * T.inv_mp2 : 0.0;
        partial[((size_t)blockIdx.y * nt + k) * 2] = ax * tf;
        partial[((size_t)blockIdx.y * nt + k) * 2 + 1] = ay * tf;
    }
}

// One warp per target: lane l adds chunks l, l + 32, ..., then the lanes' sums.
__global__ void direct_reduce_kernel(const double2 *__restrict__ partial, int nt, int nchunks, double *__restrict__ ox,
                                     double *__restrict__ oy) {
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (k >= nt) return;
    double x = 0.0, y = 0.0;
    for (int c = lane; c < nchunks; c += 32) {
        const double2 v = partial[(size_t)c * nt + k];
        x += v.x;
        y += v.y;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        y += __shfl_xor_sync(0xffffffffu, y, o);
    }
    if (lane == 0) {
        ox[k] = x;
        oy[k] = y;
    }
}

// Source chunks of a direct sum: up to 8 waves of CTAs, the last one nearly
// full, and chunks of 1,024 sources at least.
int direct_chunks(int n, int nt) {
    const int tb = max(1, (nt + kDirectThreads - 1) / kDirectThreads);
    return max(1, min(8 * 148 * kDirectCtas / tb, n / 1024));
}

void launch_direct(const double *xs, const double *ys, const double *zs, const double *w, int n,
                   const int32_t *targets, int nt, double *out_x, double *out_y, double *scratch, int nchunks,
                   cudaStream_t st) {
    if (nt <= 0) return;
    const int chunk = (n + nchunks - 1) / nchunks;
    dim3 grid((nt + kDirectThreads - 1) / kDirectThreads, nchunks);
    direct_kernel<<<grid, kDirectThreads, 0, st>>>(xs, ys, zs, w, n, targets, nt, chunk, scratch);
    direct_reduce_kernel<<<(nt + 7) / 8, 256, 0, st>>>(reinterpret_cast<const double2 *>(scratch), nt, nchunks, out_x,
                                                       out_y);
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
