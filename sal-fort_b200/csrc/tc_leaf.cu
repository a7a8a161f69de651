// Leaf pass (MODE 0) and proxy pass (MODE 1) of the batched form on the
// 5th-generation tensor cores (tcgen05).  The proxy pass is the same machine
// with the Chebyshev proxies of a target slot as targets (at most 85 per
// group), three Cartesian components val (s - x) instead of the projected
// east / north ones (3 x 85 columns fill N = 256), no self pairs, no DOWN
// items, and the group's end written to its unit's partial rows.  The leaf
// pass is described below.
//
// One CTA per SM at a time, each walking leaf groups of up to 128 targets
// (fuller ones first) with a stride of the grid size.  A group's work is a list of
// items (<= 64 sources, or <= 64 Cartesian rows of a DOWN interpolation), cut
// into stages of 32 K columns (four k-steps of 8).  The contraction is
//     D[field part, target component] += W[field part, k] * T[k, target component]
// with M = 128 weight rows (64 fields, TF32 hi and lo parts, ordered so that
// field f's hi row 32(f/16) + f%16 and lo row +16 share a warp) and N = 2 half
// kernel-tile columns (east of the group's targets, rounded up to half, a
// multiple of 16, then north): per k-step two MMAs, W * T_hi and W * T_lo, give
// all four hi/lo cross products.  An MMA of N = 256 takes 128 cycles, a small
// group's in proportion, if one elected thread issues it with descriptors from
// uniform registers; issued under `lane == 0` each cost 144 cycles and more
// (207 in this kernel, whatever N: half of the MMA warp's time).  Elected
// issue and narrow groups: leaf pass 34.9 -> 33.5 ms at 2.3M cells x 64
// fields, where the producers' tile arithmetic is what the MMA warp then waits
// for; with waits that suspend, records, teams and the plan's DOWN bases 26.6.
// Warp roles:
//   warps 0-7   producers.  A task is one k-step of a 32-target row block:
//               8 kernel-tile entries per component and row in FP32, split
//               into TF32 hi + lo, stored to shared memory in the canonical
//               K-major layout (the MMA's B operand).  Two teams of four
//               warps take the stages in turn, a stage's tasks dealt so that
//               small groups use every warp (see the producer branch).  The self pair enters as the tile's diagonal entry:
//               the reference kernel's FP64 value at distance zero (rounding
//               noise).  The sources' FP32 coordinates (per k-step x[8] y[8]
//               z[8]) come from shared memory, copied there by the loader.
//   warp 8      issues the MMAs.
//   warp 9      loads, per stage, the weight tiles (pre-split TF32 hi / lo,
//               written once per solve by split_store_kernel) and the
//               sources' coordinates (leaf and proxy passes) or BLI factors
//               (upward pass), with bulk copies into a 4-deep ring, and
//               writes the stage's record (centre offset, flags) beside them.
//   warps 10-13 fold finished accumulator chains into the running sums and
//               write the outputs (warp w: tensor memory lanes 32(w%4)..+31).
// FP16 leaf pass (sal_tune.f16): the same machine with kind::f16 MMAs, 16
// sources per MMA.  A stage is 64 sources (eight units of 8, the split
// store's granularity; an odd unit count is completed with a zero unit);
// kernel tiles and weight tiles are FP16 hi + lo (11 + 11 bits, as TF32 hi +
// lo), in the same shared-memory bytes, so each stage carries twice the
// sources for the same MMA count and stores.  FP16's range needs scales:
// every target's kernel values are multiplied by a power of two that takes
// its largest one (computed once per plan) to at most 2^12, every field's
// source weights and its potentials by powers of two of their own (per
// solve), and the fold divides them out of each chain; DOWN items (O(1)
// interpolation weights against potentials) form chains of their own.
// Kernel-tile store (sal_tune.tile_store, FP16 leaf pass): the kernel tiles
// depend on the grid alone.  A recording launch (TS 1) computes them and also
// writes them to device memory; a replaying launch (TS 2) has the loader copy
// each stage's tiles and weights into two shared-memory byte rings, and the
// idle producer warps fold beside the fold warps; a partial replay (TS 3)
// has a team's first producer warp copy the stored items' tiles into the ring
// slot while the producers compute the others.  All three give the computing launch's
// results bit for bit.
// The tensor cores accumulate with truncation, so one chain over all of a
// target's sources would bias the result toward zero: a chain ends after about
// 32 k-steps (plan flag kTcFlush) and is folded into the group's running sums
// with round-to-nearest FP32 adds.  The running sums live in tensor memory
// (columns 256-511, the accumulator's row layout) next to the accumulator
// (columns 0-255); shared memory holds only the operand rings.  The next chain
// starts once the fold warps have read the accumulator; the two-stage
// kernel-tile ring lets the producers run on meanwhile.
#include <cuda_fp16.h>
#include <algorithm>
#include <cuda_runtime.h>

#include "kernels.cuh"
#include "mixed.cuh"

namespace sal {
namespace mix {

using dev::smem_u32;

namespace {

constexpr int kFoldWarps = 4;                     // one per tensor memory lane quarter
constexpr int kProdWarps = 8;
constexpr int kMmaWarp = kProdWarps, kLoadWarp = kProdWarps + 1;
constexpr int kThreads = (kProdWarps + 2 + kFoldWarps) * 32;   // 448
constexpr int kF = 64;                            // fields
constexpr int kStageK = kTcStage;                 // K columns per stage (four k-steps of 8)
constexpr int kStageKs = kStageK / 8;             // k-steps per stage
constexpr int kKStages = 2;                       // kernel-tile ring
constexpr int kWStages = 4;                       // weight / upward-factor ring
constexpr int kAuxFloats = kStageKs * 16 * (kMaxDegree + 1);   // upward factors of a stage's k-steps
constexpr int kTileFloats = 2048;                 // kernel tile of one k-step: 256 rows x 8, one of hi / lo
constexpr int kWStepFloats = 1024;                // weight tile of one k-step: 128 rows x 8
constexpr int kTmemCols = 512;
constexpr int kKmap = 3 * (kMaxDegree + 1) * (kMaxDegree + 1) + 64;
constexpr uint32_t kWaitPolls = 1u << 24, kPollNs = 20000;
constexpr uint64_t kWaitNs = 2000000000ull;
constexpr float kC1F = (float)dev::kC1;
constexpr float kTwoC2F = (float)(2.0 * dev::kC2);

static_assert(kTcChunk % kStageK == 0, "items are whole stages");

// instruction descriptor: D F32, A/B TF32 (or FP16, format 0, 16 sources per
// MMA), both K-major, M = 128; N (columns, a multiple of 16) by idesc_n
constexpr uint32_t kIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(128 >> 4) << 24);
constexpr uint32_t kIdescF16 = (1u << 4) | ((uint32_t)(128 >> 4) << 24);
__device__ __forceinline__ uint32_t idesc_n(uint32_t idesc, int n) { return idesc | ((uint32_t)(n >> 3) << 17); }
// FP16 leaf pass: a stage is 64 sources, eight units of 8 (a unit is one
// TF32 k-step: the split store's granularity); a unit of the FP16 weight store
// is 128 rows x 8 halves, 8-row groups 128 B apart (2 KB)
constexpr int kStageKF16 = 64;
constexpr int kW16UnitBytes = 2048;
// FP16 operands are scaled by powers of two to at most 2^12 (FP16 max 65504)
constexpr int kF16TopExp = 12;
static_assert(kStageKF16 == kTcChunk, "an FP16 stage is one item: the tile store's layout");
// TcSmem::rec flags: units (8 sources) of the stage, its item's kind << 4
// (kRecDown: 2), the end of an accumulator chain, the group's own points among
// the sources
constexpr int kRecUnits = 15, kRecDown = 32, kRecFlush = 64, kRecSelf = 128;

// Replay of the kernel-tile store: the stages' kernel tiles and weight tiles
// go into two byte rings (a stage takes its own size, so the small groups'
// stages do not hold whole 64 KB slots), with up to kRStages stages in
// flight.  A stage's tiles are packed: per MMA step and hi / lo, the group's
// east rows then its north rows (rows rounded up to 16), which are the rows an
// MMA reads.
constexpr int kRStages = 8;
constexpr int kTRingBytes = 180 * 1024;
constexpr int kWRingBytes = 44 * 1024;

// Shared memory of one CTA.  Computing launches: a kKStages-deep ring of
// 64 KB kernel-tile stages, a kWStages-deep weight ring and the producers'
// buffers (source coordinates / upward factors per weight stage, DOWN bases,
// the DOWN row map).  Replay: the two byte rings and the offsets of the
// stages in flight.
template <int TS>
struct TcSmem {
    static constexpr bool kReplay = TS == 2;
    static constexpr int KS = kReplay ? kRStages : kKStages;   // kernel-tile stage slots
    static constexpr int WS = kReplay ? 1 : kWStages;          // weight stage slots
    static constexpr size_t kKtBytes = kReplay ? (size_t)kTRingBytes : (size_t)kKStages * kStageKs * 2 * kTileFloats * 4;
    static constexpr size_t kWtBytes = kReplay ? (size_t)kWRingBytes : (size_t)kWStages * kStageKs * kWStepFloats * 4;
    unsigned char ring[kKtBytes + kWtBytes];
    float aux[kReplay ? 1 : kWStages][kReplay ? 4 : kAuxFloats];   // per stage: BLI factors F[n][8] G[n][8] per k-step
    float fx[kReplay ? 1 : kTcRows][kMaxDegree + 1];              // per target row: BLI bases in the current DOWN slot
    float fe[kReplay ? 1 : kTcRows][kMaxDegree + 1];
    int kmap[kReplay ? 1 : kKmap];
    alignas(16) float cs[kTcRows];                                // folds: the group's column scales (DOWN chains)
    // computing launches, per weight stage, its item as the loader saw it: (dx,
    // dy, dz, flags: kRec*) and (off, row0)
    float4 rec[kReplay ? 1 : kWStages];
    int2 rec2[kReplay ? 1 : kWStages];
    uint32_t toff[KS], tlen[KS], woff[KS], wlen[KS];             // replay: each stage slot's ranges in the rings
    // partial replay: the copies of a slot's tiles, and the parity of the slot's
    // last one (+ 2: there was one)
    uint64_t kcopy[kKStages];
    uint32_t clast[kKStages];
    uint64_t kfull[KS], kempty[KS], wfull[WS], wempty[WS], accfull, accfree, fin;
    uint32_t tmem_base;
    int abort;
    // computing launches: kernel tile (stage slot, k-step, hi / lo), weight stage jb
    __device__ __forceinline__ float *Kt(uint32_t slot, int s, int h) {
        return reinterpret_cast<float *>(ring + (((size_t)slot * kStageKs + s) * 2 + h) * kTileFloats * 4);
    }
    __device__ __forceinline__ float *Wt(uint32_t jb) {
        return reinterpret_cast<float *>(ring + kKtBytes + (size_t)jb * kStageKs * kWStepFloats * 4);
    }
};
template <int TS> constexpr size_t tc_smem_need() { return sizeof(TcSmem<TS>) + 1024; }


// Packed FP32x2 arithmetic (two kernel-tile columns per instruction).
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;"
        : "=l"(r)
        : "l"(*reinterpret_cast<unsigned long long *>(&a)), "l"(*reinterpret_cast<unsigned long long *>(&b)));
    return *reinterpret_cast<float2 *>(&r);
}
__device__ __forceinline__ float2 f2(float x) { return make_float2(x, x); }
__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float tf32_hi(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// The same for kernel-tile values, in two integer instructions (the conversion
// takes about four): half a unit of the last kept bit added to the magnitude, the
// rest cut off.  (A NaN's hi may lose it; its lo = v - hi is NaN then.)
__device__ __forceinline__ float tf32_hi_tile(float x) {
    return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
}

// Hint: fetch a global range into L2 ahead of its bulk copy (16-byte
// aligned, a multiple of 16 bytes).
__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

using dev::mbar_arrive;
// Bounded wait on an mbarrier phase; on time-out raises the error flag and
// the CTA-wide abort flag (later waits then give up at once).  A phase that
// has already completed costs one poll and no read of the flag: every
// shared-memory round trip is on the producers' critical path.  After that a
// poll suspends the warp for up to kPollNs: polls without a time hint come back
// early, and the six waiting warps' loops took more issue slots than the
// producers' arithmetic.  The limits are kWaitNs and kWaitPolls.
__device__ __forceinline__ bool wait_bounded(uint64_t *bar, uint32_t parity, volatile int *abort, int *err) {
    if (dev::mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = dev::global_ns();
    for (uint32_t it = 0; it < kWaitPolls; ++it) {
        if (*abort) return false;
        if (dev::mbar_try_wait_ns(bar, parity, kPollNs)) return true;
        if (dev::global_ns() - t0 > kWaitNs) break;
    }
    *abort = 1;
    atomicExch(err, dev::kErrTimeout);
    return false;
}
// The same for a warp that keeps a failure: the usual case, a phase that is
// complete, touches nothing but the barrier.
__device__ __forceinline__ void wait_or_die(uint64_t *bar, uint32_t parity, volatile int *abort, int *err, bool &dead) {
    if (dev::mbar_try_wait(bar, parity)) return;
    if (!wait_bounded(bar, parity, abort, err)) dead = true;
}
// Bounded wait that ignores the abort flag (drains copies and MMAs in flight
// before the CTA exits).
__device__ __forceinline__ void wait_drain(uint64_t *bar, uint32_t parity, int *err) {
    const uint64_t t0 = dev::global_ns();
    for (uint32_t it = 0; it < kWaitPolls; ++it) {
        if (dev::mbar_try_wait_ns(bar, parity, kPollNs)) return;
        if (dev::global_ns() - t0 > kWaitNs) break;
    }
    atomicExch(err, dev::kErrTimeout);
}

__device__ __forceinline__ void mbar_arrive_n(uint64_t *bar, uint32_t n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}
// Named barrier 1 over the producer warps.
__device__ __forceinline__ void producers_sync(int threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor, canonical K-major layout without swizzle:
// 8-row x 16-byte core matrices, LBO = 128 B between the two K halves of an
// 8-row group, SBO = 256 B between 8-row groups; version 1 (bits 46-47).
__device__ __forceinline__ uint64_t smem_desc(const void *p) {
    const uint64_t addr = smem_u32(p);
    return ((addr >> 4) & 0x3FFFull) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) |
           (1ull << 46);
}

// One thread of the (converged) warp.  MMAs issued under it take their
// descriptors from uniform registers; under `lane == 0` each issue cost 144
// cycles (measured, whatever M and N), more than the MMA itself (N = 256: 128).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// D[tmem] (+)= A[smem] * B[smem], FP16 operands, 16 sources
__device__ __forceinline__ void mma_ss_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Descriptor of an FP16 weight tile of two store units (16 sources): K core
// matrices one unit (2 KB) apart, 8-row groups 128 B apart.
__device__ __forceinline__ uint64_t smem_desc_w16(const void *p) {
    const uint64_t addr = smem_u32(p);
    return ((addr >> 4) & 0x3FFFull) | ((uint64_t)(kW16UnitBytes >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) |
           (1ull << 46);
}
// FP16 hi + lo of two values, packed as half2 words: hi = round(v), lo =
// round(v - hi).  (Rounding hi with cvt.rna.tf32 first, then converting both
// halves, measured 4.6 % slower in the leaf pass.)
__device__ __forceinline__ void split_f16x2(float a, float b, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 back = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - back.x, b - back.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}
// The power of two that takes a magnitude m to at most 2^kF16TopExp (1 for
// m = 0), and its inverse.
__host__ __device__ inline float f16_scale(float m) {
    if (!(m > 0.f)) return 1.f;
    int e;
    frexpf(m, &e);   // m < 2^e
    e = kF16TopExp - e;
    e = e < -120 ? -120 : (e > 120 ? 120 : e);
    return ldexpf(1.f, e);
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16};" ::"r"(taddr),
        "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
        "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
        "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])),
        "r"(__float_as_uint(v[11])), "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])),
        "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15]))
        : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float (&v)[32]) {
    uint32_t r[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(v[i]);
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// BLI basis (FP64, stored as FP32) of one coordinate of a target over one
// axis's Chebyshev nodes.  Out of line: its local array stays out of the
// stage loop's registers.
__device__ __noinline__ void down_basis(double x, const double *nodes, int n, float *out) {
    double f[kMaxDegree + 1];
    dev::bli_basis(x, nodes, n, f);
    for (int i = 0; i < n; ++i) out[i] = (float)f[i];
}

// Byte offset of element (row, k) of a canonical K-major tile without
// swizzle (8-row x 16-byte core matrices, K halves 128 B apart, 8-row groups
// 256 B apart), k < 8.
__host__ __device__ constexpr int canon(int row, int k) {
    return (row >> 3) * 256 + (k >> 2) * 128 + (row & 7) * 16 + (k & 3) * 4;
}
// Weight-tile row of field f's hi (part 0) or lo (part 1) TF32 part: the two
// rows of a field sit in one 32-lane quarter of the accumulator, 16 apart.
__host__ __device__ constexpr int wrow(int f, int part) { return 32 * (f >> 4) + 16 * part + (f & 15); }

}  // namespace

// Writes one finished 16-column chunk x (this lane's accumulator row, the
// running sum already added) to its destination at a group's end.  Lanes
// 0-15 hold fields' hi rows, lanes 16-31 the same fields' lo rows; per
// column pair, lanes 0-15 write the even column and lanes 16-31 the odd one,
// so hi + lo of a field meet in one lane.
template <int MODE>
__device__ __forceinline__ void emit_chunk(const float (&x)[16], int c0, int f, int odd, int nt, int idk, double *out,
                                           bool wr, float *part, int half) {
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const float lo_even = __shfl_down_sync(0xffffffffu, x[2 * m], 16);
        const float hi_odd = __shfl_up_sync(0xffffffffu, x[2 * m + 1], 16);
        const int j = c0 + 2 * m + odd;   // column
        if (MODE == 0) {
            const int t = j >= half ? j - half : j;
            const int ti = __shfl_sync(0xffffffffu, idk, t & 31);
            const double v = odd ? (double)hi_odd + (double)x[2 * m + 1] : (double)x[2 * m] + (double)lo_even;
            if (wr && t < nt) out[ti] = v;
        } else {
            const float v = odd ? hi_odd + x[2 * m + 1] : x[2 * m] + lo_even;
            if (MODE == 2) {
                // upward rows: column j is proxy row0 + j; the unit's partial
                // holds one row of 64 fields per proxy
                if (wr && j < nt) part[(size_t)j * kF + f] = v;
            } else {
                // proxy rows: column j = 85c + r is component c of proxy r; the
                // unit's partial holds (proxy, component) rows of 64 fields
                const int c = j / kTcProxyRows, r = j - c * kTcProxyRows;
                if (wr && c < 3 && r < nt) part[((size_t)r * 3 + c) * kF + f] = v;
            }
        }
    }
}

// Folds a finished accumulator chain into the running sums (warp-collective;
// this warp's lane quarter q: fields 16q..16q+15, hi rows in lanes 0-15 and
// lo rows in lanes 16-31).  The running sums live in tensor memory next to
// the accumulator (columns 256-511, same row layout): running sum (+)= chain
// with round-to-nearest FP32 adds (the group's first chain stores).  At a
// group's end only the chunks that hold targets are folded, and emit_sums
// writes them out after the accumulator has been handed back to the MMA
// warp, so the next group's first chain overlaps the output writes.
// MODE 0 (leaf): columns half c + t are component c (east, north) of target
// t (half = the group's rows rounded up to 16).  MODE 1 (proxy): columns 85c + r are
// Cartesian component c of proxy r.  MODE 2 (upward): columns j < 128 are
// proxies row0 + j.
//
// FP16 leaf pass (scaled, the same in every lane): the chain's operands were
// scaled by powers of two, the weight rows of field f by 1 / fsc and (kernel
// chains) the kernel tile's column of target t by tscale[tgt + t] (DOWN
// chains: unscaled columns).  The running sums are kept in the columns'
// scaled domain: a kernel chain adds chain x fsc, a DOWN chain chain x fsc x
// tscale, and emit_sums multiplies by tinv = 1 / tscale.  Powers of two
// commute with rounding, so this gives the unscaled sums' bits while kernel
// chains (all but one or a few per group) need no per-column factors.
// Several warps of one lane quarter can share a fold: warp part_i of nparts
// takes the chunk pairs (2p, 2p + 1) with p % nparts == part_i, and emits
// the same chunks.

// Chunks of 16 columns a fold covers: per component, at a group's end only
// those that hold targets; a pair (2p, 2p + 1) at a time.
template <int MODE>
__device__ __forceinline__ int fold_per(bool end, int nt, int half) {
    return (MODE != 1 && end) ? (nt + 15) / 16 : (MODE == 0 ? half / 16 : 8);
}

// The MMA warp waits for the fold, so it is short: the chunks are contiguous
// columns (16 i), taken 32 at a time; a kernel chain's factor is a power of
// two, so factor and add are one packed fused multiply-add with the same bits;
// and the next chain columns are on their way while a result is stored (16
// columns at a time 4,300 cycles a chain of a full group and 1,750 of one row
// block, so 4,000 and 1,100).
template <int MODE>
__device__ __noinline__ void fold_chain(uint32_t td, int lane, bool end, bool first, int nt, bool scaled, float fsc,
                                        bool down, float4 tsc, float *cs, int half, int part_i, int nparts) {
    // DOWN chains: the targets' scales, which every fold warp writes to shared
    // memory for itself (the same values; the next such chain's are written
    // after every warp has handed this one's accumulator back)
    if (MODE == 0 && scaled && down) {
        cs[lane] = tsc.x;
        cs[32 + lane] = tsc.y;
        cs[64 + lane] = tsc.z;
        cs[96 + lane] = tsc.w;
        __syncwarp();
    }
    const int per = fold_per<MODE>(end, nt, half);
    const int ncol = 16 * (MODE == 2 ? per : 2 * per);   // component c's chunk j is columns half c + 16 j, half = 16 per
    const float2 f2v = f2(scaled && !down ? fsc : 1.f);
    // DOWN chains: the field's factor, then the column's
    auto unscale = [&](float *x, int c) {
        const float2 *sc = reinterpret_cast<const float2 *>(cs + (c >= half ? c - half : c));
#pragma unroll
        for (int m = 0; m < 16; m += 2) {
            const float2 v = __fmul2_rn(__fmul2_rn(make_float2(x[m], x[m + 1]), f2(fsc)), sc[m >> 1]);
            x[m] = v.x;
            x[m + 1] = v.y;
        }
    };
    auto add = [&](float *x, const float *r) {   // 2 columns
        float2 v = make_float2(x[0], x[1]);
        v = first ? __fmul2_rn(v, f2v) : __ffma2_rn(v, f2v, make_float2(r[0], r[1]));
        x[0] = v.x;
        x[1] = v.y;
    };
    float x[32], r[32];
#pragma unroll
    for (int m = 0; m < 32; ++m) r[m] = 0.f;
    int c = 32 * part_i;
    if (c + 32 <= ncol) tmem_ld32(td + c, x);
#pragma unroll 1
    for (; c + 32 <= ncol; c += 32 * nparts) {
        if (!first) tmem_ld32(td + 256 + c, r);
        tmem_wait_ld();
        if (MODE == 0 && scaled && down) {
            unscale(x, c);
            unscale(x + 16, c + 16);
        }
        float y[32];
#pragma unroll
        for (int m = 0; m < 32; ++m) y[m] = x[m];
#pragma unroll
        for (int m = 0; m < 32; m += 2) add(y + m, r + m);
        if (c + 32 * nparts + 32 <= ncol) tmem_ld32(td + c + 32 * nparts, x);
        tmem_st32(td + 256 + c, y);
    }
    if (c < ncol) {   // an odd chunk left
        float x1[16], r1[16];
        tmem_ld16(td + c, x1);
        if (!first) tmem_ld16(td + 256 + c, r1);
        else
#pragma unroll
            for (int m = 0; m < 16; ++m) r1[m] = 0.f;
        tmem_wait_ld();
        if (MODE == 0 && scaled && down) unscale(x1, c);
#pragma unroll
        for (int m = 0; m < 16; m += 2) add(x1 + m, r1 + m);
        tmem_st16(td + 256 + c, x1);
    }
    tmem_wait_st();
}

// A group's end: its running sums (this warp's chunks of fold_chain) to the
// destinations, hi + lo added in FP64: MODE 0 the caller's outputs, MODE 1 /
// 2 the unit's partial rows `part`.
template <int MODE>
__device__ __noinline__ void emit_sums(uint32_t td, int q, int lane, int tgt, int nt, const int32_t *__restrict__ perm,
                                       double *out_x, double *out_y, int64_t ld_out, int f0, int nf, bool skip,
                                       float *part, bool scaled, const float *__restrict__ tinv, int half, int part_i,
                                       int nparts) {
    const int f = 16 * q + (lane & 15), odd = lane >> 4;
    float cse[4] = {1.f, 1.f, 1.f, 1.f};   // per target slot 32k + lane: its scale's inverse
    if (MODE == 0 && scaled)
#pragma unroll
        for (int k = 0; k < 4; ++k) cse[k] = 32 * k + lane < nt ? tinv[tgt + 32 * k + lane] : 1.f;
    int idx[4] = {0, 0, 0, 0};   // caller index of target slot 32k + lane
    if (MODE == 0)
#pragma unroll
        for (int k = 0; k < 4; ++k) idx[k] = 32 * k + lane < nt ? perm[tgt + 32 * k + lane] : 0;
    const bool wr = (MODE != 0 || f0 + f < nf) && !skip;
    double *ox = MODE == 0 ? out_x + (size_t)(f0 + f) * ld_out : nullptr;
    double *oy = MODE == 0 ? out_y + (size_t)(f0 + f) * ld_out : nullptr;
    const int per = fold_per<MODE>(true, nt, half);
    const int nchunk = MODE == 2 ? per : 2 * per;
    auto col = [&](int i) { return (i / per) * half + (i % per) * 16; };
    float x[16];
#pragma unroll 1
    for (int i = 2 * part_i; i < nchunk; i += 2 * nparts)
#pragma unroll 1
        for (int h = i; h < i + 2 && h < nchunk; ++h) {
            const int c = col(h);
            tmem_ld16(td + 256 + c, x);
            tmem_wait_ld();
            const int b = c >= half ? c - half : c, k = b >> 5;
            if (MODE == 0 && scaled) {
                // out of the columns' scaled domain
                const float src = k == 0 ? cse[0] : k == 1 ? cse[1] : k == 2 ? cse[2] : cse[3];
#pragma unroll
                for (int m = 0; m < 16; ++m) x[m] *= __shfl_sync(0xffffffffu, src, (b & 31) + m);
            }
            const int idk = k == 0 ? idx[0] : k == 1 ? idx[1] : k == 2 ? idx[2] : idx[3];
            emit_chunk<MODE>(x, c, f, odd, nt, idk, c < half ? ox : oy, wr, part, half);
        }
}

// Outputs of target t of a leaf group without sources: its self pair alone.
__device__ __noinline__ void self_only(const TcArgs &a, const MixGroup &G, int t) {
    const int pos = G.tgt + t, idx = a.perm[pos];
    const double2 sk = a.selfk[pos];
    for (int f = 0; f < kF && a.f0 + f < a.nf; ++f) {
        const double w = (double)a.wF[(size_t)pos * kF + f];
        a.out_x[(size_t)(a.f0 + f) * a.ld_out + idx] = sk.x * w;
        a.out_y[(size_t)(a.f0 + f) * a.ld_out + idx] = sk.y * w;
    }
}

// A warp's window on a group's item records, 32 at a time: lane i holds
// record k0 + i, and the next 32 are loaded one batch ahead, so a warp that
// walks items faster than a global load returns (the MMA, loader and fold
// warps) does not wait on one load per item.  k must be warp-uniform and
// non-decreasing.
struct ItemWindow {
    const TcItem *items;
    int k0, ie;
    TcItem cur, nxt;
    __device__ __forceinline__ void start(const TcItem *it, int ib, int e, int lane) {
        items = it;
        k0 = ib;
        ie = e;
        cur = ib + lane < e ? it[ib + lane] : TcItem{};
        nxt = ib + 32 + lane < e ? it[ib + 32 + lane] : TcItem{};
    }
    __device__ __forceinline__ void seek(int k, int lane) {
        while (k >= k0 + 32) {
            cur = nxt;
            k0 += 32;
            nxt = k0 + 32 + lane < ie ? items[k0 + 32 + lane] : TcItem{};
        }
    }
    __device__ __forceinline__ TcItem get(int k, int lane) {
        seek(k, lane);
        const int l = k - k0;
        TcItem r;
        r.off = __shfl_sync(0xffffffffu, cur.off, l);
        r.cnt = __shfl_sync(0xffffffffu, cur.cnt, l);
        r.kb = __shfl_sync(0xffffffffu, cur.kb, l);
        r.kind = __shfl_sync(0xffffffffu, cur.kind, l);
        r.dx = __shfl_sync(0xffffffffu, cur.dx, l);
        r.dy = __shfl_sync(0xffffffffu, cur.dy, l);
        r.dz = __shfl_sync(0xffffffffu, cur.dz, l);
        r.row0 = __shfl_sync(0xffffffffu, cur.row0, l);
        return r;
    }
    __device__ __forceinline__ int kind(int k, int lane) {
        seek(k, lane);
        return __shfl_sync(0xffffffffu, cur.kind, k - k0);
    }
};

// JOINT: one launch over the groups of several grids (of one degree): group
// gi belongs to the grid k with J.beg[k] <= gi < J.beg[k + 1] and carries
// that grid's arguments.  Otherwise J.g[0] is the only grid.
// TS (FP16 leaf pass, one grid): 0 the producers compute the kernel tiles;
// 1 they compute them and also record them in the grid's kernel-tile store;
// 2 the loader copies them from the store into the kernel-tile ring and the
// producers only write the outputs of groups without sources.
template <int MODE, bool JOINT, bool F16, int TS = 0>
__global__ void __launch_bounds__(kThreads, 1) tc_leaf_kernel(const __grid_constant__ TcJoint J, int *err) {
    dev::after_previous();
    static_assert(!F16 || MODE == 0, "FP16 operands in the leaf pass only");
    static_assert(TS == 0 || (MODE == 0 && F16 && !JOINT), "kernel-tile store: FP16 leaf pass of one grid");
    constexpr int SK = F16 ? kStageKF16 : kStageK;   // sources per stage
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    constexpr int KS = TcSmem<TS>::KS, WS = TcSmem<TS>::WS;
    TcSmem<TS> &sm = *reinterpret_cast<TcSmem<TS> *>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n = J.g[0].d + 1, P = J.g[0].P;
    const int total = JOINT ? J.beg[J.ngrids] : J.g[0].ngroups;
    // the grid of joint group gi
    auto grid_of = [&](int gi) -> int {
        int k = 0;
        if (JOINT)
            while (k + 1 < J.ngrids && gi >= J.beg[k + 1]) ++k;
        return k;
    };
    volatile int *abort = &sm.abort;

    // ------------------------------------------------------------ set-up
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&sm.tmem_base)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int j = 0; j < KS; ++j) {
            // replay: the loader's arrival and its copies' bytes fill a stage
            dev::mbar_init(&sm.kfull[j], TS == 2 ? 1 : kProdWarps);
            dev::mbar_init(&sm.kempty[j], 1);
        }
        for (int j = 0; j < WS; ++j) {
            dev::mbar_init(&sm.wfull[j], 1);
            dev::mbar_init(&sm.wempty[j], 1);
        }
        for (int j = 0; j < kKStages; ++j) {
            dev::mbar_init(&sm.kcopy[j], 1);
            sm.clast[j] = 0;
        }
        dev::mbar_init(&sm.accfull, 1);
        // replay: the idle producer warps fold too, three warps per lane quarter
        dev::mbar_init(&sm.accfree, TS == 2 ? kFoldWarps + kProdWarps : kFoldWarps);
        dev::mbar_init(&sm.fin, 1);
        dev::fence_mbar_init();
        sm.abort = 0;
    }
    for (int k = tid; TS != 2 && k < kKmap; k += kThreads) {
        const int kk = k < 3 * P ? k : 0;
        const int p = kk / 3;
        sm.kmap[k] = (p % n) | ((p / n) << 8) | ((kk % 3) << 16);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sm.tmem_base;
    uint32_t st = 0;   // stages this CTA has gone through
    // Set by a producer or MMA warp's first wait that gave up, and kept: from then
    // on it uses no stage's buffers and signals no stage (the abort flag ends the
    // others' waits).  Beyond a stage that was never issued the barriers' parities
    // mean nothing (a slot that missed a lap looks full), and an arrival out of
    // turn, a team's for two among DOWN stages' for one, can take a barrier's count
    // below zero, which is a fault.
    bool dead = false;

    if (TS != 2 && warp < kProdWarps) {
        // ============================================================ producers
        // A stage's tasks are (row block of 32 targets, unit) pairs, one
        // 8-source unit of 32 rows each (a TF32 stage has 4 units, an FP16
        // stage 8).  The stages are dealt to two teams of four warps in turn,
        // and within a team (DOWN stages: over all eight warps w)
        //   3-4 row blocks: warp w takes row block w % 4, all units
        //                   (DOWN: units w / 4 + 2i)
        //   2 row blocks:   row block w % 2, units w / 2 + 2i (w / 2 + 4i)
        //   1 row block:    units w + 4i (unit w)
        // so that a group of few row blocks uses every warp.
        // The source coordinates of a stage's k-steps (x[8] y[8] z[8] each,
        // relative to their panel's centre) arrive in shared memory with the
        // stage's weights: the loader warp copies them up to WS stages
        // ahead, so no global-memory latency sits in a producer task.
        uint32_t cpar = 0;   // partial replay: per slot, the parity of its next copy
        for (int gi = blockIdx.x; gi < total; gi += gridDim.x) {
            const int gk = grid_of(gi);
            const TcArgs &a = J.g[gk];
            const MixGroup G = a.groups[gi - J.beg[gk]];
            const int ni = G.ie - G.ib;
            const int rb = (G.nt + 31) >> 5;
            const int wb = rb >= 3 ? (warp & 3) : rb == 2 ? (warp & 1) : 0;            // row block
            const int kfirst8 = rb >= 3 ? (warp >> 2) : rb == 2 ? (warp >> 1) : warp;    // first k-step
            const int kstride8 = rb >= 3 ? 2 : rb == 2 ? 4 : 8;
            const int row = 32 * wb + lane;
            const bool active = 32 * wb < G.nt, rvalid = row < G.nt;
            // leaf: east / north of target t at rows t, half + t of a kernel tile
            // (half: the targets rounded up to 16)
            const int half = (G.nt + 15) & ~15;
            const bool row_in_tile = row < half;
            // FP16 tiles: byte offset of the row's first K core matrix (8-row
            // groups 256 B apart, the two K halves 128 B apart)
            const int oe16 = (row >> 3) * 256 + (row & 7) * 16;
            // the row's target relative to the leaf centre and its east /
            // north unit vectors (zero at the poles, as the reference's guard)
            float tl0 = 0.f, tl1 = 0.f, tl2 = 0.f, el0 = 0.f, el1 = 0.f, ep0 = 0.f, ep1 = 0.f, ep2 = 0.f;
            // FP16 leaf pass: this row's power-of-two scale of kernel values
            const float tsc = (F16 && rvalid) ? a.tscale[G.tgt + row] : 1.f;
            if (MODE == 0 && rvalid) {
                const double4 c = a.tgt[G.tgt + row];
                tl0 = (float)(c.x - G.cx);
                tl1 = (float)(c.y - G.cy);
                tl2 = (float)(c.z - G.cz);
                if ((fabs(c.z - 1.0) > 1e-15) && (fabs(c.z + 1.0) > 1e-15)) {
                    const double omz = 1.0 - c.z * c.z, inv = 1.0 / sqrt(omz);
                    el0 = (float)(-c.y * inv);
                    el1 = (float)(c.x * inv);
                    ep0 = (float)(-c.z * c.x * inv);
                    ep1 = (float)(-c.z * c.y * inv);
                    ep2 = (float)(omz * inv);
                }
            }
            if (ni == 0) {
                // no sources: the self pair alone (thread t: target t)
                if (MODE == 0 && tid < G.nt && !*abort) self_only(a, G, tid);
                continue;
            }
            // the kernel values' projections; FP16: with the row's scale in them
            const float2 el0v = f2(el0 * tsc), el1v = f2(el1 * tsc), ep0v = f2(ep0 * tsc), ep1v = f2(ep1 * tsc),
                         ep2v = f2(ep2 * tsc);
            int cur_slot = -1;
            // the self pair (FP64 value / kernel constant, the weight carries the constant)
            const int my_pos = G.tgt + row;
            float self_e = 0.f, self_n = 0.f;
            if (MODE == 0 && rvalid) {
                const double2 sk = a.selfk[my_pos];
                self_e = (float)sk.x * tsc;
                self_n = (float)sk.y * tsc;
            }
            // record: the group's tiles in the store, stage after stage; per
            // MMA step four chunks (hi, lo x east, north) of the group's rows
            // rounded up to 16, each the bytes of the ring's rows
            const size_t cb = (size_t)half * 32;
            unsigned char *gtile = (TS == 1 || TS == 3) ? a.ktile + a.ktile_off[gi - J.beg[gk]] : nullptr;
            if constexpr (F16) {
                // FP16: an item is one stage, and its record comes to shared
                // memory with its weights: the loop costs a warp about as much
                // per stage as a task does, so it holds nothing else.  The
                // group's point and proxy items (all before its DOWN items) are
                // dealt to two teams of four warps, stage by stage: a team's
                // warps take twice the tasks of every other stage, and pay
                // for half the stages.  DOWN items are every warp's.  A
                // team's warp counts for two arrivals.
                const int team = warp >> 2, tw = warp & 3;
                const int ndown = G.ndown;   // DOWN items, at the list's end
#pragma unroll 1
                for (int k = 0; k < ni; ++k, ++st) {
                    const bool down = k >= ni - ndown;
                    // an item the kernel-tile store holds (one in tile_every)
                    const bool stored = (TS == 1 || TS == 3) && k % a.tile_every == a.tile_every - 1;
                    const uint32_t cpar_st = (cpar >> (st % KS)) & 1;   // its copy's phase of kcopy
                    if (TS == 3 && stored) cpar ^= 1u << (st % KS);
                    if (!down && (st & 1) != (uint32_t)team) {
                        if (stored) gtile += (size_t)4 * ((((a.items[G.ib + k].cnt + 7) >> 3) + 1) >> 1) * cb;
                        continue;
                    }
                    const uint32_t arrivals = down ? 1 : 2;
                    const uint32_t slot = st % KS, kpar = ((st / KS) - 1) & 1, jb = st % WS;
                    bool slot_free = st < (uint32_t)KS;
                    wait_or_die(&sm.wfull[jb], (st / WS) & 1, abort, err, dead);
                    const float4 rec = sm.rec[jb];
                    const int flags = dead ? 0 : __float_as_int(rec.w), nks = flags & kRecUnits;
                    if (TS == 3 && stored) {
                        // replay: the stage's first warp copies its chunks (MMA step
                        // q / 4, hi / lo, east / north) into the ring slot once the MMAs
                        // that last read it are done, on a barrier of the copies' own
                        const int nq = 4 * ((nks + 1) >> 1);
                        if (!slot_free) wait_or_die(&sm.kempty[slot], kpar, abort, err, dead);
                        if ((down ? warp == 0 : tw == 0) && __all_sync(0xffffffffu, !dead)) {
                            if (lane == 0) dev::mbar_expect_tx(&sm.kcopy[slot], (uint32_t)(nq * cb));
                            __syncwarp();
                            if (lane < nq)
                                dev::bulk_g2s_hint(
                                    reinterpret_cast<unsigned char *>(sm.Kt(slot, lane >> 2, (lane >> 1) & 1)) + (lane & 1) * cb,
                                    gtile + (size_t)lane * cb, (uint32_t)cb, &sm.kcopy[slot], dev::l2_evict_first());
                            if (lane == 0) sm.clast[slot] = 2u | cpar_st;
                        }
                        __syncwarp();
                        if (lane == 0 && !dead) mbar_arrive_n(&sm.kfull[slot], arrivals);
                        gtile += (size_t)nq * cb;
                        continue;
                    }
                    const float2 tx2 = f2(tl0 - rec.x), ty2 = f2(tl1 - rec.y), tz2 = f2(tl2 - rec.z);
                    // the sources' x[8] y[8] z[8] per unit (the same address in every
                    // lane: shared-memory broadcasts), and this row's place in the tile
                    const float2 *crd = reinterpret_cast<const float2 *>(sm.aux[jb]);
                    char *tile = reinterpret_cast<char *>(sm.Kt(slot, 0, 0)) + oe16;
                    // a K task's kernel values (units kk, kk + dk, ...), two columns per
                    // packed instruction, as FP16 hi + lo words o[task] = {east hi, east
                    // lo, north hi, north lo}, packed as they are computed: 4 K
                    // independent chains in one block of code
                    auto pairs16 = [&]<int K>(int kk, int dk, uint32_t (&o)[K][4][4]) {
#pragma unroll
                        for (int c2 = 0; c2 < 4; ++c2)
#pragma unroll
                            for (int t = 0; t < K; ++t) {
                                const float2 *cr = crd + 12 * (kk + t * dk) + c2;
                                const float2 dx = sub2(cr[0], tx2), dy = sub2(cr[4], ty2), dz = sub2(cr[8], tz2);
                                // + 1e-20: mp = 0 only for a source on the target itself (or
                                // a repeated point), and the floor keeps the value finite;
                                // chords of neighbours (mp >= 1e-12) do not see it
                                const float2 mp = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, f2(1e-20f))));
                                const float2 r = make_float2(rsqrt_approx(mp.x), rsqrt_approx(mp.y));
                                const float2 w = __fadd2_rn(__fmul2_rn(mp, r), f2(2.f));
                                const float2 u = make_float2(rcp_approx(w.x), rcp_approx(w.y));
                                const float2 inner = __ffma2_rn(f2(kC1F), r, __ffma2_rn(f2(kTwoC2F), u, f2(-kTwoC2F)));
                                const float2 v = __fmul2_rn(inner, __fmul2_rn(r, r));
                                const float2 pe = __ffma2_rn(el1v, dy, __fmul2_rn(el0v, dx));
                                const float2 pn = __ffma2_rn(ep2v, dz, __ffma2_rn(ep1v, dy, __fmul2_rn(ep0v, dx)));
                                const float2 e2 = __fmul2_rn(v, pe), n2 = __fmul2_rn(v, pn);
                                split_f16x2(e2.x, e2.y, o[t][0][c2], o[t][1][c2]);
                                split_f16x2(n2.x, n2.y, o[t][2][c2], o[t][3][c2]);
                            }
                    };
                    // unit kk is K half kk & 1 of MMA step kk / 2, the row's 8 values
                    // one 16-byte core-matrix row
                    auto store16 = [&](int kk, const uint32_t (&o)[4][4]) {
                        if (!row_in_tile) return;
                        char *t = tile + (kk >> 1) * (2 * kTileFloats * 4) + 128 * (kk & 1);
                        const uint4 eh = make_uint4(o[0][0], o[0][1], o[0][2], o[0][3]), el = make_uint4(o[1][0], o[1][1], o[1][2], o[1][3]);
                        const uint4 nh = make_uint4(o[2][0], o[2][1], o[2][2], o[2][3]), nl = make_uint4(o[3][0], o[3][1], o[3][2], o[3][3]);
                        *reinterpret_cast<uint4 *>(t) = eh;
                        *reinterpret_cast<uint4 *>(t + kTileFloats * 4) = el;
                        *reinterpret_cast<uint4 *>(t + half * 32) = nh;
                        *reinterpret_cast<uint4 *>(t + half * 32 + kTileFloats * 4) = nl;
                        if (TS == 1 && stored) {
                            unsigned char *g = gtile + (size_t)(kk >> 1) * 4 * cb + oe16 + 128 * (kk & 1);
                            *reinterpret_cast<uint4 *>(g) = eh;
                            *reinterpret_cast<uint4 *>(g + cb) = nh;
                            *reinterpret_cast<uint4 *>(g + 2 * cb) = el;
                            *reinterpret_cast<uint4 *>(g + 3 * cb) = nl;
                        }
                    };
                    // the MMAs that last read the slot must be done before the first
                    // store into it
                    auto claim = [&]() {
                        if (!slot_free) wait_or_die(&sm.kempty[slot], kpar, abort, err, dead);
                        slot_free = true;
                    };
                    // units: a team's warp w takes row block w (w % 2, 0), units i (w / 2
                    // + 2i, w + 4i) of a group of 3-4 (2, 1) row blocks
                    const int kstride = down ? kstride8 : rb >= 3 ? 1 : rb == 2 ? 2 : 4;
                    int kk = !active ? nks + 1 : down ? kfirst8 : rb >= 3 ? 0 : rb == 2 ? tw >> 1 : tw;
                    if (!(flags & (kRecDown | kRecSelf))) {
#pragma unroll 1
                        for (; kk + kstride < nks; kk += 2 * kstride) {
                            uint32_t o[2][4][4];
                            pairs16(kk, kstride, o);
                            claim();
                            store16(kk, o[0]);
                            store16(kk + kstride, o[1]);
                        }
                    }
                    if (down) {
                        // the tree passes have one slot a group (every warp must come to
                        // the same barriers, so not by the record, which a time-out may
                        // have left unread)
                        const int slot_id = a.dbasis ? 0 : a.items[G.ib + k].off;
                        if (slot_id != cur_slot) {
                            // BLI bases of every target row in the new slot: thread
                            // t < 128 the xi basis of target t, thread 128 + t its
                            // eta basis
                            cur_slot = slot_id;
                            producers_sync(32 * kProdWarps);
                            const int brow = tid & (kTcRows - 1);
                            if (brow < G.nt) {
                                float *o = tid < kTcRows ? sm.fx[brow] : sm.fe[brow];
                                if (a.dbasis) {
                                    // tree passes: a target has one slot, its bases are in the
                                    // plan's store
                                    const float *src = a.dbasis + (size_t)(G.tgt + brow) * 2 * n + (tid < kTcRows ? 0 : n);
                                    for (int i = 0; i < n; ++i) o[i] = src[i];
                                } else {
                                    const double2 e = a.xieta[G.tgt + brow];
                                    const double *nodes = a.tgt_nodes + (size_t)slot_id * 2 * n;
                                    down_basis(tid < kTcRows ? e.x : e.y, tid < kTcRows ? nodes : nodes + n, n, o);
                                }
                            }
                            producers_sync(32 * kProdWarps);
                        }
                    }
#pragma unroll 1
                    for (; kk < ((nks + 1) & ~1); kk += kstride) {
                        uint32_t o[1][4][4];
                        if (kk >= nks) {
                            // an odd last unit's partner in its 16-source MMA step
#pragma unroll
                            for (int c = 0; c < 4; ++c) o[0][0][c] = o[0][1][c] = o[0][2][c] = o[0][3][c] = 0u;
                        } else if (flags & kRecDown) {
                            // BLI basis of the target x its unit vector's component of the
                            // Cartesian row: the unit's rows r0 .. r0 + 7 are components
                            // r % 3 of proxies r / 3, four proxies at most (rows past
                            // 3 P meet zero weights)
                            const int r0 = sm.rec2[jb].y + 8 * kk, p0 = r0 / 3, ph = r0 - 3 * p0;
                            float bv[4];
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                const int km = sm.kmap[3 * (p0 + q < P ? p0 + q : 0)];
                                bv[q] = sm.fx[row][km & 255] * sm.fe[row][(km >> 8) & 255];
                            }
                            auto fill = [&]<int PH>() {
#pragma unroll
                                for (int c2 = 0; c2 < 4; ++c2) {
                                    float e[2], nn[2];
#pragma unroll
                                    for (int c = 0; c < 2; ++c) {
                                        constexpr int kThree = 3;
                                        const int x = PH + 2 * c2 + c, comp = x % kThree;
                                        const float b = bv[x / kThree];
                                        e[c] = comp == 2 ? 0.f : b * (comp == 0 ? el0 : el1);
                                        nn[c] = b * (comp == 0 ? ep0 : (comp == 1 ? ep1 : ep2));
                                    }
                                    split_f16x2(e[0], e[1], o[0][0][c2], o[0][1][c2]);
                                    split_f16x2(nn[0], nn[1], o[0][2][c2], o[0][3][c2]);
                                }
                            };
                            if (ph == 0) fill.template operator()<0>();
                            else if (ph == 1) fill.template operator()<1>();
                            else fill.template operator()<2>();
                        } else {
                            pairs16(kk, 0, o);
                        }
                        claim();
                        store16(kk, o[0]);
                        if (flags & kRecSelf) {
                            // the target itself among these 8 sources: the self pair's
                            // halves over the tile entry just stored
                            const int cs = my_pos - (sm.rec2[jb].x + 8 * kk);
                            if (row_in_tile && kk < nks && (unsigned)cs < 8u) {
                                uint32_t h, l;
                                split_f16x2(self_e, self_n, h, l);
                                char *t = tile + (kk >> 1) * (2 * kTileFloats * 4) + 128 * (kk & 1) + 2 * cs;
                                *reinterpret_cast<uint16_t *>(t) = (uint16_t)h;
                                *reinterpret_cast<uint16_t *>(t + kTileFloats * 4) = (uint16_t)l;
                                *reinterpret_cast<uint16_t *>(t + half * 32) = (uint16_t)(h >> 16);
                                *reinterpret_cast<uint16_t *>(t + half * 32 + kTileFloats * 4) = (uint16_t)(l >> 16);
                                if (TS == 1 && stored) {
                                    unsigned char *g = gtile + (size_t)(kk >> 1) * 4 * cb + oe16 + 128 * (kk & 1) + 2 * cs;
                                    *reinterpret_cast<uint16_t *>(g) = (uint16_t)h;
                                    *reinterpret_cast<uint16_t *>(g + cb) = (uint16_t)(h >> 16);
                                    *reinterpret_cast<uint16_t *>(g + 2 * cb) = (uint16_t)l;
                                    *reinterpret_cast<uint16_t *>(g + 3 * cb) = (uint16_t)(l >> 16);
                                }
                            }
                        }
                    }
                    // warps that wrote nothing: their arrival must still not run a
                    // ring phase ahead of the MMAs
                    claim();
                    dev::fence_proxy_async();
                    __syncwarp();
                    if (lane == 0 && !dead) mbar_arrive_n(&sm.kfull[slot], arrivals);
                    if (TS == 1 && stored) gtile += (size_t)4 * ((nks + 1) >> 1) * cb;
                }
                continue;
            }
            // TF32 stages: the same two teams.  Leaf pass: a stage's tasks to a
            // team's warps by row block, as above.  Proxy and upward pass: warp w of
            // the team takes unit w for all row blocks.  (Tasks dealt over eight
            // warps left two idle at three row blocks, with an item record from
            // global memory and a wait a stage for each.  Proxy passes of a solve
            // at 2.3M cells x 64 fields: that 7.44 ms, teams 6.85, tf32_hi_tile
            // 6.47, two row blocks side by side 6.28; half units over all eight
            // warps, every stage: 7.08 with the first of these.)
            constexpr int kB = MODE == 0 ? 1 : MODE == 1 ? (kTcProxyRows + 31) / 32 : kTcRows / 32;   // row blocks of a task
            const int team = warp >> 2, tw = warp & 3;
            const int n_all = G.nst, n_kern = G.nst - G.nstd;
            float tl[kB][3];   // targets relative to the group's centre
            int up_i[kB], up_j[kB];   // upward: proxy row0 + row = up_i + up_j n
#pragma unroll
            for (int b = 0; b < kB; ++b) {
                const int r = 32 * b + lane;
                tl[b][0] = tl0; tl[b][1] = tl1; tl[b][2] = tl2;
                up_i[b] = up_j[b] = 0;
                if (MODE == 1) {
                    const double4 c = a.tgt[(size_t)G.tgt * P + G.row0 + (r < G.nt ? r : 0)];
                    tl[b][0] = (float)(c.x - G.cx);
                    tl[b][1] = (float)(c.y - G.cy);
                    tl[b][2] = (float)(c.z - G.cz);
                }
                if (MODE == 2) {
                    const int p = G.row0 + (r < G.nt ? r : 0);
                    up_i[b] = p % n;
                    up_j[b] = p / n;
                }
            }
            // canonical offsets (floats) of row block 0's rows in a kernel tile (a
            // row block is 256 floats on): leaf east / north at rows t, half + t;
            // proxy x / y / z at 85 c + r
            const int oe = canon(MODE == 0 ? row : lane, 0) >> 2;
            const int on = canon(MODE == 0 ? half + row : kTcProxyRows + lane, 0) >> 2;
            const int oz = canon(MODE == 0 ? 0 : 2 * kTcProxyRows + lane, 0) >> 2;
#pragma unroll 1
            for (int k = 0; k < n_all; ++k, ++st) {
                const bool down = MODE == 0 && k >= n_kern;
                if (!down && (st & 1) != (uint32_t)team) continue;
                const uint32_t slot = st % KS, kpar = ((st / KS) - 1) & 1, jb = st % WS;
                bool slot_free = st < (uint32_t)KS;
                wait_or_die(&sm.wfull[jb], (st / WS) & 1, abort, err, dead);
                const float4 rec = sm.rec[jb];
                const int flags = dead ? 0 : __float_as_int(rec.w), nks = flags & kRecUnits;
                // the MMAs that last read the slot must be done before the first
                // store into it
                auto claim = [&]() {
                    if (!slot_free) wait_or_die(&sm.kempty[slot], kpar, abort, err, dead);
                    slot_free = true;
                };
                // kernel value x displacement (leaf: projected east, north; proxy: the
                // Cartesian vector val (s - x)) of two columns for row block b; crd: the
                // columns' x, and 4, 8 further on y and z (the same address in every lane:
                // shared-memory broadcasts)
                auto pair = [&](const float2 *crd, float2 tx2, float2 ty2, float2 tz2, float *vx, float *vy, float *vz) {
                    const float2 dx = sub2(crd[0], tx2), dy = sub2(crd[4], ty2), dz = sub2(crd[8], tz2);
                    // + 1e-20: mp = 0 only for a source on the target itself (or
                    // a repeated point), and the floor keeps the value finite;
                    // chords of neighbours (mp >= 1e-12) do not see it
                    const float2 mp = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, f2(1e-20f))));
                    const float2 r = make_float2(rsqrt_approx(mp.x), rsqrt_approx(mp.y));
                    const float2 w = __fadd2_rn(__fmul2_rn(mp, r), f2(2.f));
                    const float2 u = make_float2(rcp_approx(w.x), rcp_approx(w.y));
                    const float2 inner = __ffma2_rn(f2(kC1F), r, __ffma2_rn(f2(kTwoC2F), u, f2(-kTwoC2F)));
                    const float2 v = __fmul2_rn(inner, __fmul2_rn(r, r));
                    float2 a, b;
                    if (MODE == 0) {
                        a = __fmul2_rn(v, __ffma2_rn(el1v, dy, __fmul2_rn(el0v, dx)));
                        b = __fmul2_rn(v, __ffma2_rn(ep2v, dz, __ffma2_rn(ep1v, dy, __fmul2_rn(ep0v, dx))));
                    } else {
                        const float2 c = __fmul2_rn(v, dz);
                        a = __fmul2_rn(v, dx);
                        b = __fmul2_rn(v, dy);
                        vz[0] = c.x;
                        vz[1] = c.y;
                    }
                    vx[0] = a.x;
                    vx[1] = a.y;
                    vy[0] = b.x;
                    vy[1] = b.y;
                };
                // four values of a row into a tile (hi; lo kTileFloats on): TF32 hi + lo
                // (the tensor cores read lo's top 11 bits)
                auto store = [&](float *th, const float *v) {
                    const float4 h = make_float4(tf32_hi_tile(v[0]), tf32_hi_tile(v[1]), tf32_hi_tile(v[2]), tf32_hi_tile(v[3]));
                    const float2 l01 = sub2(make_float2(v[0], v[1]), make_float2(h.x, h.y));
                    const float2 l23 = sub2(make_float2(v[2], v[3]), make_float2(h.z, h.w));
                    *reinterpret_cast<float4 *>(th) = h;
                    *reinterpret_cast<float4 *>(th + kTileFloats) = make_float4(l01.x, l01.y, l23.x, l23.y);
                };
                if constexpr (MODE == 0) {
                    // a DOWN slot's 3 P rows are slot_stages stages
                    const int slot_stages = (3 * P + SK - 1) / SK;
                    if (down && (k - n_kern) % slot_stages == 0) {
                        // BLI bases of every target row in the new slot: thread t < 128
                        // the xi basis of target t, thread 128 + t its eta basis
                        const int slot_items = (3 * P + kTcChunk - 1) / kTcChunk;
                        const int slot_id = a.items[G.ie - G.ndown + (k - n_kern) / slot_stages * slot_items].off;
                        producers_sync(32 * kProdWarps);
                        const int brow = tid & (kTcRows - 1);
                        if (brow < G.nt) {
                            const double2 e = a.xieta[G.tgt + brow];
                            const double *nodes = a.tgt_nodes + (size_t)slot_id * 2 * n;
                            down_basis(tid < kTcRows ? e.x : e.y, tid < kTcRows ? nodes : nodes + n, n,
                                       tid < kTcRows ? sm.fx[brow] : sm.fe[brow]);
                        }
                        producers_sync(32 * kProdWarps);
                    }
                    const int kstride = down ? kstride8 : rb >= 3 ? 1 : rb == 2 ? 2 : 4;
                    // units kk, kk + kstride, ... (K of them) of this row
                    auto units = [&]<int K>(int kk) {
                        float ve[K][8], vn[K][8];
#pragma unroll
                        for (int i = 0; i < K; ++i) {
                            const int u = kk + i * kstride;
                            if (down) {
                                // BLI basis of the target x its unit vector's component of
                                // the Cartesian row
                                const int *km0 = sm.kmap + sm.rec2[jb].y + 8 * u;
                                const float *fxr = sm.fx[row], *fer = sm.fe[row];
#pragma unroll
                                for (int c = 0; c < 8; ++c) {
                                    const int km = km0[c];
                                    const float b = fxr[km & 255] * fer[(km >> 8) & 255];
                                    const int comp = km >> 16;
                                    ve[i][c] = comp == 2 ? 0.f : b * (comp == 0 ? el0 : el1);
                                    vn[i][c] = b * (comp == 0 ? ep0 : (comp == 1 ? ep1 : ep2));
                                }
                            } else {
                                const float2 *crd = reinterpret_cast<const float2 *>(sm.aux[jb]) + 12 * u;
                                const float2 tx2 = f2(tl0 - rec.x), ty2 = f2(tl1 - rec.y), tz2 = f2(tl2 - rec.z);
#pragma unroll
                                for (int c2 = 0; c2 < 4; ++c2)
                                    pair(crd + c2, tx2, ty2, tz2, ve[i] + 2 * c2, vn[i] + 2 * c2, nullptr);
                                if (flags & kRecSelf) {
                                    // the target itself among these 8 sources: the self pair
                                    const int cs = my_pos - (sm.rec2[jb].x + 8 * u);
#pragma unroll
                                    for (int c = 0; c < 8; ++c)
                                        if (c == cs) { ve[i][c] = self_e; vn[i][c] = self_n; }
                                }
                            }
                        }
                        claim();
                        if (!row_in_tile) return;
#pragma unroll
                        for (int i = 0; i < K; ++i) {
                            float *th = sm.Kt(slot, kk + i * kstride, 0);
                            store(th + oe, ve[i]);
                            store(th + oe + 32, ve[i] + 4);
                            store(th + on, vn[i]);
                            store(th + on + 32, vn[i] + 4);
                        }
                    };
                    int kk = !active ? nks : down ? kfirst8 : rb >= 3 ? 0 : rb == 2 ? tw >> 1 : tw;
                    if (!(flags & (kRecDown | kRecSelf))) {
#pragma unroll 1
                        for (; kk + kstride < nks; kk += 2 * kstride) units.template operator()<2>(kk);
                    }
#pragma unroll 1
                    for (; kk < nks; kk += kstride) units.template operator()<1>(kk);
                } else if (tw < nks) {
                    // unit tw for row blocks b0, b0 + 1 (NB of them side by side: the
                    // second's arithmetic fills the first's latencies), then the next
                    auto blocks = [&]<int NB>(int b0) {
                        float v[NB][3][8];
#pragma unroll
                        for (int i = 0; i < NB; ++i) {
                            const int b = b0 + i;
                            if (MODE == 1) {
                                const float2 *crd = reinterpret_cast<const float2 *>(sm.aux[jb]) + 12 * tw;
                                const float2 tx2 = f2(tl[b][0] - rec.x), ty2 = f2(tl[b][1] - rec.y), tz2 = f2(tl[b][2] - rec.z);
#pragma unroll
                                for (int c2 = 0; c2 < 4; ++c2)
                                    pair(crd + c2, tx2, ty2, tz2, v[i][0] + 2 * c2, v[i][1] + 2 * c2, v[i][2] + 2 * c2);
                            } else {
                                // upward: the BLI basis of proxy (i, j) at the 8 points, F_i(xi)
                                // G_j(eta) from the per-point factors
                                const float *Fb = sm.aux[jb] + 16 * n * tw;
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    const float4 f = *reinterpret_cast<const float4 *>(Fb + 8 * up_i[b] + 4 * h);
                                    const float4 g = *reinterpret_cast<const float4 *>(Fb + 8 * n + 8 * up_j[b] + 4 * h);
                                    v[i][0][4 * h] = f.x * g.x;
                                    v[i][0][4 * h + 1] = f.y * g.y;
                                    v[i][0][4 * h + 2] = f.z * g.z;
                                    v[i][0][4 * h + 3] = f.w * g.w;
                                }
                            }
                        }
                        claim();
#pragma unroll
                        for (int i = 0; i < NB; ++i) {
                            const int b = b0 + i;
                            if (MODE == 1 && 32 * b + lane >= kTcProxyRows) break;
                            float *th = sm.Kt(slot, tw, 0) + 256 * b;
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                store(th + oe + 32 * h, v[i][0] + 4 * h);
                                if (MODE == 1) {
                                    store(th + on + 32 * h, v[i][1] + 4 * h);
                                    store(th + oz + 32 * h, v[i][2] + 4 * h);
                                }
                            }
                        }
                    };
                    blocks.template operator()<2>(0);
                    if (rb > 2) blocks.template operator()<kB - 2>(2);
                }
                // warps that wrote nothing: their arrival must still not run a ring
                // phase ahead of the MMAs
                claim();
                dev::fence_proxy_async();
                __syncwarp();
                if (lane == 0 && !dead) mbar_arrive_n(&sm.kfull[slot], down ? 1 : 2);
            }
        }
    } else if (warp == kMmaWarp) {
        // ============================================================ MMA issue
        uint32_t cc = 0;           // chains started
        uint32_t cpar = 0;         // partial replay: as the producers'
        bool chain_open = false;
        for (int gi = blockIdx.x; gi < total; gi += gridDim.x) {
            const int gk = grid_of(gi);
            const TcArgs &a = J.g[gk];
            const MixGroup G = a.groups[gi - J.beg[gk]];
            // computing launches take a stage's units and chain end from the
            // loader's record; a replay's stage is an item
            constexpr bool kRec = TS != 2;
            ItemWindow w;
            if (!kRec) w.start(a.items, G.ib, G.ie, lane);
            const int nstages = F16 ? G.ie - G.ib : G.nst;
            // the group's columns: component c of target t is column half c + t
            // (half: the targets rounded up to 16), so small groups' MMAs are
            // narrow; the proxy pass has three components of 85 rows, the
            // upward pass one of 128
            const int half = (G.nt + 15) & ~15;
            const uint32_t idesc = idesc_n(F16 ? kIdescF16 : kIdesc, MODE == 0 ? 2 * half : MODE == 1 ? 256 : 128);
            // replay: bytes of one packed tile (east rows, then north rows)
            const uint32_t ptile = 2u * (uint32_t)half * 32u;
            for (int k = 0; k < nstages; ++k, ++st) {
                TcItem it{};
                if (!kRec) it = w.get(G.ib + k, lane);
                bool flush = it.kind & kTcFlush;
                const uint32_t slot = st % KS, jb = st % WS;
                // replay: the stage's one barrier covers its weight and kernel tiles
                // (polled together: the one's latency hides the other's)
                const bool wf = TS == 2 || dev::mbar_try_wait(&sm.wfull[jb], (st / WS) & 1);
                const bool kf = dev::mbar_try_wait(&sm.kfull[slot], (st / KS) & 1);
                if (!kf) wait_or_die(&sm.kfull[slot], (st / KS) & 1, abort, err, dead);
                if (!wf) wait_or_die(&sm.wfull[jb], (st / WS) & 1, abort, err, dead);
                if (TS == 3 && k % a.tile_every == a.tile_every - 1) {
                    wait_or_die(&sm.kcopy[slot], (cpar >> slot) & 1, abort, err, dead);
                    cpar ^= 1u << slot;
                }
                // a new chain overwrites the accumulator, whose last chain
                // (cc - 1) the fold warps must have read
                if (!chain_open && cc >= 1) wait_or_die(&sm.accfree, (cc - 1) & 1, abort, err, dead);
                dead = __any_sync(0xffffffffu, dead);
                tc_fence_after();
                int nks = (it.cnt + 7) >> 3;
                if (kRec) {
                    const int flags = __float_as_int(sm.rec[jb].w);
                    nks = flags & kRecUnits;
                    flush = flags & kRecFlush;
                }
                flush = flush && !dead;
                const uint32_t open = chain_open ? 1u : 0u;
                if (!dead && elect_one()) {
                    if constexpr (TS == 2) {
                        // packed tiles of MMA step s: hi at (2s) ptile, lo at (2s + 1) ptile
                        const uint64_t aw = smem_desc_w16(sm.ring + TcSmem<TS>::kKtBytes + sm.woff[slot]);
                        const uint64_t bt = smem_desc(sm.ring + sm.toff[slot]);
#pragma unroll
                        for (int s = 0; s < SK / 16; ++s)
                            if (2 * s < nks) {
                                const uint64_t a = aw + s * (2 * kW16UnitBytes >> 4), bh = bt + 2 * s * (ptile >> 4);
                                mma_ss_f16(tmem, a, bh, idesc, s ? 1u : open);
                                mma_ss_f16(tmem, a, bh + (ptile >> 4), idesc, 1u);
                            }
                    } else {
                        // FP16: 16 sources per MMA (weight units 2s and 2s + 1); TF32: 8
                        constexpr uint32_t kStepW = kWStepFloats * 4 >> 4, kStepT = kTileFloats * 4 >> 4;
                        const uint64_t aw = F16 ? smem_desc_w16(sm.Wt(jb)) : smem_desc(sm.Wt(jb));
                        const uint64_t bt = smem_desc(sm.Kt(slot, 0, 0));
#pragma unroll
                        for (int s = 0; s < kStageKs; ++s)
                            if ((F16 ? 2 : 1) * s < nks) {
                                const uint64_t a = aw + s * kStepW, bh = bt + 2 * s * kStepT;
                                if (F16) {
                                    mma_ss_f16(tmem, a, bh, idesc, s ? 1u : open);
                                    mma_ss_f16(tmem, a, bh + kStepT, idesc, 1u);
                                } else {
                                    mma_ss(tmem, a, bh, idesc, s ? 1u : open);
                                    mma_ss(tmem, a, bh + kStepT, idesc, 1u);
                                }
                            }
                    }
                    mma_commit(&sm.kempty[slot]);
                    if (TS != 2) mma_commit(&sm.wempty[jb]);
                }
                chain_open = true;
                __syncwarp();
                if (flush) {
                    if (elect_one()) mma_commit(&sm.accfull);
                    __syncwarp();
                    chain_open = false;
                    ++cc;
                }
            }
        }
        // every MMA issued by this CTA completes before tensor memory is freed
        if (elect_one()) mma_commit(&sm.fin);
        if (lane == 0) wait_drain(&sm.fin, 0, err);
        __syncwarp();
    } else if (warp == kLoadWarp) {
        // ============================================================ loads
        // replay: ring heads, the oldest stage still in flight
        uint32_t thead = 0, whead = 0, oldest = 0;
        // After a wait that gave up nothing more is expected or issued: a phase
        // whose bytes never come would hold the drain below for its whole limit.
        // Test hook: nothing from stage inject - 1 on.
        bool live = true;
        uint32_t issued = 0;   // stages issued
        const uint32_t stop = J.g[0].inject ? J.g[0].inject - 1 : 0xffffffffu;
        for (int gi = blockIdx.x; gi < total; gi += gridDim.x) {
            const int gk = grid_of(gi);
            const TcArgs &a = J.g[gk];
            const MixGroup G = a.groups[gi - J.beg[gk]];
            ItemWindow w;
            w.start(a.items, G.ib, G.ie, lane);
            // replay: the group's recorded tiles, stage after stage (per MMA
            // step, hi then lo, each the group's east rows then its north
            // rows, rounded up to 16 rows of 32 bytes)
            const unsigned char *tsrc = TS == 2 ? a.ktile + a.ktile_off[gi - J.beg[gk]] : nullptr;
            const uint32_t cb = (uint32_t)((G.nt + 15) & ~15) * 32u;
            if constexpr (TS != 2) {
                // Lane l holds item k0 + l of the window: it writes its stages'
                // records itself, and the copies need a few of its numbers only.
                // (The whole record by shuffles, twice, and an L2 prefetch of the
                // next item's tiles, made this warp the slowest of a small group's
                // stage: 1,240 cycles.)
#pragma unroll 1
                for (int k = G.ib; k < G.ie; ++k) {
                    w.seek(k, lane);
                    const int l = k - w.k0;
                    const TcItem &it = w.cur;
                    const int kind = it.kind & 3;
                    const bool self = MODE == 0 && kind == 0 && it.off < G.tgt + G.nt && G.tgt < it.off + it.cnt;
                    const int iflags = kind << 4 | ((it.kind & kTcFlush) ? kRecFlush : 0) | (self ? kRecSelf : 0);
                    // F16: an item is one stage
                    const int kb = __shfl_sync(0xffffffffu, it.kb, l), down = __shfl_sync(0xffffffffu, kind, l) == 2;
                    const int cnt = __shfl_sync(0xffffffffu, it.cnt, l);
                    const int row0 = MODE == 2 ? __shfl_sync(0xffffffffu, it.row0, l) : 0;
#pragma unroll 1
                    for (int b = 0; b < cnt; b += SK, ++st) {
                        const uint32_t jb = st % WS, ub = st / WS;
                        const uint32_t nks = (uint32_t)(min(SK, cnt - b) + 7) >> 3;
                        bool ok = true;
                        if (ub > 0) ok = wait_bounded(&sm.wempty[jb], (ub - 1) & 1, abort, err);
                        if (lane == l) {
                            // before the arrival that its readers wait for; a chain ends
                            // with an item's last stage
                            const int flags = (int)nks | (b + SK < cnt ? iflags & ~kRecFlush : iflags);
                            sm.rec[jb] = make_float4(it.dx, it.dy, it.dz, __int_as_float(flags));
                            sm.rec2[jb] = make_int2(kind == 2 ? it.off : it.off + b, it.row0 + b);
                        }
                        live = __all_sync(0xffffffffu, ok) && live && st < stop;
                        if (live) issued = st + 1;
                        __syncwarp();
                        if (live && elect_one()) {
                            // FP16: whole 16-source MMA steps (the store has a spare unit at
                            // its end).  With the weights come the point and proxy sources'
                            // coordinates (24 floats per unit; DOWN rows need none), or the
                            // upward pass's BLI factors.
                            const uint32_t wbytes = F16 ? ((nks + 1) & ~1u) * kW16UnitBytes : nks * kWStepFloats * 4u;
                            const uint32_t lbytes = MODE == 2 ? nks * 64u * n : down ? 0u : nks * 96u;
                            const size_t u = (size_t)kb + b / 8;
                            dev::mbar_expect_tx(&sm.wfull[jb], wbytes + lbytes);
                            if (lbytes)
                                dev::bulk_g2s(sm.aux[jb],
                                              MODE == 2 ? (const void *)(a.basis + ((size_t)row0 + b / 8) * 16 * n)
                                                        : (const void *)(a.sxyz + u * 24),
                                              lbytes, &sm.wfull[jb]);
                            dev::bulk_g2s(sm.Wt(jb),
                                          F16 ? (const void *)(static_cast<const char *>(a.bstore16) + u * kW16UnitBytes)
                                              : (const void *)(a.bstore + u * kWStepFloats),
                                          wbytes, &sm.wfull[jb]);
                        }
                        __syncwarp();
                    }
                }
            } else {
                for (int k = G.ib; k < G.ie; ++k, ++st) {
                    const TcItem it = w.get(k, lane);
                    if (k + 1 < G.ie) {
                        // the next item's weight tiles into L2 while this item's stage runs
                        const TcItem nxt = w.get(k + 1, lane);
                        const uint32_t nks = (uint32_t)(nxt.cnt + 7) >> 3;
                        if (elect_one())
                            prefetch_l2(static_cast<const char *>(a.bstore16) + (size_t)nxt.kb * kW16UnitBytes,
                                        ((nks + 1) & ~1u) * kW16UnitBytes);
                    }
                    // the stage's kernel tiles and weight tiles, each one bulk copy
                    // into its ring (from the start of a ring when they do not fit
                    // before its end), once the stage slot and both ranges are free:
                    // stages retire in order
                    const uint32_t nsteps = (uint32_t)(((it.cnt + 7) >> 3) + 1) >> 1;
                    const uint32_t sb = nsteps * 4u * cb, wb = nsteps * 2u * kW16UnitBytes;
                    const uint32_t tpos = thead + sb > (uint32_t)kTRingBytes ? 0u : thead;
                    const uint32_t wpos = whead + wb > (uint32_t)kWRingBytes ? 0u : whead;
                    while (oldest < st) {
                        bool clash = st - oldest >= (uint32_t)KS;
                        for (uint32_t x = oldest; !clash && x < st; ++x) {
                            const uint32_t xs = x % KS;
                            const uint32_t t0 = sm.toff[xs], t1 = t0 + sm.tlen[xs];
                            const uint32_t w0 = sm.woff[xs], w1 = w0 + sm.wlen[xs];
                            clash = (tpos < t1 && t0 < tpos + sb) || (wpos < w1 && w0 < wpos + wb);
                        }
                        if (!clash) break;
                        wait_bounded(&sm.kempty[oldest % KS], (oldest / KS) & 1, abort, err);
                        ++oldest;
                    }
                    const uint32_t slot = st % KS;
                    live = __all_sync(0xffffffffu, !*abort) && live && st < stop;
                    if (live) issued = st + 1;
                    if (live && elect_one()) {
                        sm.toff[slot] = tpos;
                        sm.tlen[slot] = sb;
                        sm.woff[slot] = wpos;
                        sm.wlen[slot] = wb;
                        // the offsets are written before the arrival the MMA warp waits on
                        dev::mbar_expect_tx(&sm.kfull[slot], sb + wb);
                        // the tiles are read once per solve: they leave L2 first, to
                        // the weight tiles, which other groups read again
                        dev::bulk_g2s_hint(sm.ring + tpos, tsrc, sb, &sm.kfull[slot], dev::l2_evict_first());
                        dev::bulk_g2s_hint(sm.ring + TcSmem<TS>::kKtBytes + wpos,
                                           static_cast<const char *>(a.bstore16) + (size_t)it.kb * kW16UnitBytes,
                                           wb, &sm.kfull[slot], dev::l2_evict_last());
                    }
                    __syncwarp();
                    tsrc += sb;
                    thead = tpos + sb;
                    whead = wpos + wb;
                }
            }
        }
        // no bulk copy may still be landing when the CTA exits
        if (lane == 0)
            for (uint32_t x = issued > (TS == 2 ? KS : WS) ? issued - (TS == 2 ? KS : WS) : 0; x < issued; ++x) {
                if (TS == 2) wait_drain(&sm.kfull[x % KS], (x / KS) & 1, err);
                else wait_drain(&sm.wfull[x % WS], (x / WS) & 1, err);
            }
        __syncwarp();
    }
    else {
        // ============================================================ folds
        // (replay: warps 0-7 and 10-13, fold part 0, 1 or 2 of their lane
        // quarter warp % 4; otherwise warps 10-13)
        const int q = warp & 3;
        const uint32_t tq = tmem + ((uint32_t)(32 * q) << 16);
        const int part_i = TS == 2 ? (warp < 4 ? 0 : warp < kProdWarps ? 1 : 2) : 0, nparts = TS == 2 ? 3 : 1;
        uint32_t cc = 0;   // chains folded
        for (int gi = blockIdx.x; gi < total; gi += gridDim.x) {
            const int gk = grid_of(gi);
            const TcArgs &a = J.g[gk];
            const MixGroup G = a.groups[gi - J.beg[gk]];
            if (TS == 2 && G.ib == G.ie) {
                // a group without sources: the self pairs, by warps 0-7
                if (tid < G.nt && !*abort) self_only(a, G, tid);
                continue;
            }
            bool first = true;
            const int half = MODE == 0 ? (G.nt + 15) & ~15 : 128;   // columns per component
            // everything a fold needs from global memory is read before its chain is
            // awaited: the MMA warp waits for the fold
            float fsc_kern = 1.f, fsc_down = 1.f;
            if (F16) {
                fsc_kern = 1.f / f16_scale(__uint_as_float(a.fmax[16 * q + (lane & 15)]));
                fsc_down = 1.f / f16_scale(__uint_as_float(a.fmax[kF + 16 * q + (lane & 15)]));
            }
            ItemWindow w;
            w.start(a.items, G.ib, G.ie, lane);
            for (int k = G.ib; k < G.ie; ++k) {
                const int kind = w.kind(k, lane);
                if (!(kind & kTcFlush)) continue;
                // FP16: the chain's weight rows are the fields' source weights
                // (scaled per field) against scaled kernel columns, or their
                // potentials (scaled per field) against unscaled DOWN columns
                const bool down_chain = (kind & 3) == 2;
                const float fsc = !F16 ? 1.f : down_chain ? fsc_down : fsc_kern;
                const bool end = k == G.ie - 1;
                float4 tsc = make_float4(1.f, 1.f, 1.f, 1.f);   // DOWN chains: scales of targets 32 k + lane
                if (MODE == 0 && F16 && down_chain) {
                    tsc.x = lane < G.nt ? a.tscale[G.tgt + lane] : 1.f;
                    tsc.y = 32 + lane < G.nt ? a.tscale[G.tgt + 32 + lane] : 1.f;
                    tsc.z = 64 + lane < G.nt ? a.tscale[G.tgt + 64 + lane] : 1.f;
                    tsc.w = 96 + lane < G.nt ? a.tscale[G.tgt + 96 + lane] : 1.f;
                }
                wait_bounded(&sm.accfull, cc & 1, abort, err);
                tc_fence_after();
                fold_chain<MODE>(tq, lane, end, first, G.nt, F16, fsc, down_chain, tsc, sm.cs, half, part_i, nparts);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.accfree);
                // the next group's first chain may run into the accumulator meanwhile
                if (end)
                    emit_sums<MODE>(tq, q, lane, G.tgt, G.nt, a.perm, a.out_x, a.out_y, a.ld_out, a.f0, a.nf,
                                    *abort != 0,
                                    MODE == 1   ? a.partial + ((size_t)G.out * P + G.row0) * 3 * kF
                                    : MODE == 2 ? a.partial + ((size_t)G.out * P + G.row0) * kF
                                                : nullptr,
                                    F16, a.tinv, half, part_i, nparts);
                first = false;
                ++cc;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    // a wait gave up: copies that the MMA warp did not wait for
    if (TS == 3 && tid == 32 && *abort)
        for (int j = 0; j < kKStages; ++j)
            if (sm.clast[j]) wait_drain(&sm.kcopy[j], sm.clast[j] & 1, err);
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

// Row of a split store entry s: weight row s, potential row -2 - s, or (-1, a
// padding row: the caller puts zeros) the first weight row, so that a thread's
// eight loads need no branches and are in flight together.
__device__ __forceinline__ const float *store_row(int32_t s, const float *wF, const float *phiF) {
    return s <= -2 ? phiF + (size_t)(-2 - s) * kF : wF + (size_t)(s >= 0 ? s : 0) * kF;
}

// Split weight store (k-steps [k0, k1) of it, with bsrc and bstore offset
// by the caller): per k-step of 8 store rows, the 64-field rows as one
// 128-row TF32 tile (field f's hi part at row wrow(f, 0), lo part at
// wrow(f, 1)) in the canonical no-swizzle K-major layout.  One thread per
// (k-step, field).
__global__ void split_store_kernel(const int32_t *__restrict__ bsrc, int64_t nk, const float *__restrict__ wF,
                                   const float *__restrict__ phiF, float *__restrict__ bstore) {
    dev::after_previous();
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nk * kF) return;
    const int64_t ks = t / kF;
    const int f = (int)(t % kF);
    float hi[8], lo[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int32_t s = bsrc[ks * 8 + r];
        const float x = store_row(s, wF, phiF)[f], v = s == -1 ? 0.f : x;
        hi[r] = tf32_hi(v);
        lo[r] = tf32_hi(v - hi[r]);
    }
    float *base = bstore + ks * kWStepFloats;
    const int oh = canon(wrow(f, 0), 0) >> 2, ol = canon(wrow(f, 1), 0) >> 2;
    *reinterpret_cast<float4 *>(base + oh) = make_float4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<float4 *>(base + oh + 32) = make_float4(hi[4], hi[5], hi[6], hi[7]);
    *reinterpret_cast<float4 *>(base + ol) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    *reinterpret_cast<float4 *>(base + ol + 32) = make_float4(lo[4], lo[5], lo[6], lo[7]);
}

// FP16 leaf pass: per field the largest |value| of the weight rows (blockIdx.y
// 0, out[f]) and of the potential rows (1, out[64 + f]): one float4 of 4 fields
// per thread and row, contiguous reads, merged as float bits with atomicMax
// (non-negative floats order as their bits).
__global__ void field_max_kernel(const float4 *__restrict__ w, int64_t nw, const float4 *__restrict__ phi, int64_t np,
                                 unsigned *__restrict__ out) {
    dev::after_previous();
    __shared__ float part[16][kF];
    const float4 *x = blockIdx.y ? phi : w;
    const int64_t nrows = blockIdx.y ? np : nw;
    const int c4 = threadIdx.x & 15;
    float m0 = 0.f, m1 = 0.f, m2 = 0.f, m3 = 0.f;
#pragma unroll 4
    for (int64_t r = (int64_t)blockIdx.x * 16 + (threadIdx.x >> 4); r < nrows; r += (int64_t)gridDim.x * 16) {
        const float4 v = x[r * 16 + c4];
        m0 = fmaxf(m0, fabsf(v.x));
        m1 = fmaxf(m1, fabsf(v.y));
        m2 = fmaxf(m2, fabsf(v.z));
        m3 = fmaxf(m3, fabsf(v.w));
    }
    part[threadIdx.x >> 4][4 * c4] = m0;
    part[threadIdx.x >> 4][4 * c4 + 1] = m1;
    part[threadIdx.x >> 4][4 * c4 + 2] = m2;
    part[threadIdx.x >> 4][4 * c4 + 3] = m3;
    __syncthreads();
    if (threadIdx.x < kF) {
        float m = 0.f;
        for (int i = 0; i < 16; ++i) m = fmaxf(m, part[i][threadIdx.x]);
        atomicMax(out + blockIdx.y * kF + threadIdx.x, __float_as_uint(m));
    }
}

// FP16 hi/lo weight store: per unit of 8 store rows, the 64-field rows as
// one 128-row FP16 tile (field f's hi part at row wrow(f, 0), lo at
// wrow(f, 1); row m at byte (m / 8) 128 + (m % 8) 16, 8 halves), source
// weights scaled by their field's power of two, potentials by theirs.  Bound by
// memory: thread (unit, field) reads its field of the unit's rows (a warp: 128
// contiguous bytes a row) and writes 16 bytes of hi and lo each beside its
// neighbours'; kStoreUnits units a thread, for its two scales.  At 655,362
// cells (0.96 GB) 255 -> 155 us: the eight rows' loads stood behind a branch
// each (see store_row).
constexpr int kStoreUnits = 4;
__global__ void __launch_bounds__(256) split_store16_kernel(const int4 *__restrict__ bsrc, int64_t nu,
                                                            const float *__restrict__ wF, const float *__restrict__ phiF,
                                                            const unsigned *__restrict__ fmax,
                                                            unsigned char *__restrict__ out) {
    dev::after_previous();
    const int f = threadIdx.x & (kF - 1);
    const int64_t u0 = ((int64_t)blockIdx.x * (256 / kF) + (threadIdx.x >> 6)) * kStoreUnits;
    const float sw = f16_scale(__uint_as_float(fmax[f])), sp = f16_scale(__uint_as_float(fmax[kF + f]));
    const int mh = wrow(f, 0), ml = wrow(f, 1);
    const int oh = (mh >> 3) * 128 + (mh & 7) * 16, ol = (ml >> 3) * 128 + (ml & 7) * 16;
#pragma unroll 2
    for (int i = 0; i < kStoreUnits; ++i) {
        const int64_t u = u0 + i;
        if (u >= nu) return;
        const int4 s0 = bsrc[2 * u], s1 = bsrc[2 * u + 1];
        const int src[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
        float v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int s = src[r];
            const float x = store_row(s, wF, phiF)[f] * (s >= 0 ? sw : sp);
            v[r] = s == -1 ? 0.f : x;
        }
        uint4 hi, lo;
        split_f16x2(v[0], v[1], hi.x, lo.x);
        split_f16x2(v[2], v[3], hi.y, lo.y);
        split_f16x2(v[4], v[5], hi.z, lo.z);
        split_f16x2(v[6], v[7], hi.w, lo.w);
        unsigned char *base = out + u * kW16UnitBytes;
        *reinterpret_cast<uint4 *>(base + oh) = hi;
        *reinterpret_cast<uint4 *>(base + ol) = lo;
    }
}

// FP16 leaf pass: per target the power of two that takes its largest kernel
// value (east or north, over its PP and PC sources, with the leaf pass's own
// FP32 arithmetic, and its self pair) to at most 2^12, and the inverse.  One
// block per leaf group, thread t its target t.  Once per plan.
__global__ void target_scales_kernel(const TcArgs a, float *__restrict__ tscale, float *__restrict__ tinv) {
    const MixGroup G = a.groups[blockIdx.x];
    const int row = threadIdx.x;
    if (row >= G.nt) return;
    const double4 c = a.tgt[G.tgt + row];
    const float tl0 = (float)(c.x - G.cx), tl1 = (float)(c.y - G.cy), tl2 = (float)(c.z - G.cz);
    float el0 = 0.f, el1 = 0.f, ep0 = 0.f, ep1 = 0.f, ep2 = 0.f;
    if ((fabs(c.z - 1.0) > 1e-15) && (fabs(c.z + 1.0) > 1e-15)) {
        const double omz = 1.0 - c.z * c.z, inv = 1.0 / sqrt(omz);
        el0 = (float)(-c.y * inv);
        el1 = (float)(c.x * inv);
        ep0 = (float)(-c.z * c.x * inv);
        ep1 = (float)(-c.z * c.y * inv);
        ep2 = (float)(omz * inv);
    }
    const double2 sk = a.selfk[G.tgt + row];
    float m = fmaxf(fabsf((float)sk.x), fabsf((float)sk.y));
    for (int k = G.ib; k < G.ie; ++k) {
        const TcItem it = a.items[k];
        if ((it.kind & 3) == 2) continue;
        const float tx = tl0 - it.dx, ty = tl1 - it.dy, tz = tl2 - it.dz;
        for (int i = 0; i < it.cnt; ++i) {
            const float *u = a.sxyz + (size_t)(it.kb + (i >> 3)) * 24;
            const float dx = u[i & 7] - tx, dy = u[8 + (i & 7)] - ty, dz = u[16 + (i & 7)] - tz;
            const float mp = fmaxf(dz * dz + (dy * dy + dx * dx), 1e-20f);
            const float r = rsqrt_approx(mp);
            const float uu = rcp_approx(mp * r + 2.f);
            const float v = (kC1F * r + (kTwoC2F * uu - kTwoC2F)) * (r * r);
            const float pe = el0 * dx + el1 * dy, pn = ep0 * dx + ep1 * dy + ep2 * dz;
            m = fmaxf(m, fmaxf(fabsf(v * pe), fabsf(v * pn)));
        }
    }
    const float sc = f16_scale(m);
    tscale[G.tgt + row] = sc;
    tinv[G.tgt + row] = 1.f / sc;
}

// Tree passes: per target of a leaf group, the BLI bases (xi, then eta; n
// floats each) over the nodes of the group's one DOWN slot, as down_basis gives
// them.  One block per leaf group, thread t its target t.  Once per plan.
__global__ void down_basis_store_kernel(const TcArgs a, float *__restrict__ out) {
    const MixGroup G = a.groups[blockIdx.x];
    const int row = threadIdx.x, n = a.d + 1;
    if (row >= G.nt || G.ndown == 0) return;
    const double *nodes = a.tgt_nodes + (size_t)a.items[G.ie - 1].off * 2 * n;
    const double2 e = a.xieta[G.tgt + row];
    float *o = out + (size_t)(G.tgt + row) * 2 * n;
    down_basis(e.x, nodes, n, o);
    down_basis(e.y, nodes + n, n, o + n);
}

// Per pool row, the FP32 coordinates relative to the centre of the row's own
// panel (a leaf for points, the slot panel for proxies).  One block per range.
__global__ void source_local_kernel(const double4 *__restrict__ pool, const int2 *__restrict__ ranges,
                                    const double4 *__restrict__ centres, float4 *__restrict__ sloc) {
    const int2 r = ranges[blockIdx.x];
    const double4 c = centres[blockIdx.x];
    for (int p = r.x + threadIdx.x; p < r.y; p += blockDim.x) {
        const double4 s = pool[p];
        sloc[p] = make_float4((float)(s.x - c.x), (float)(s.y - c.y), (float)(s.z - c.z), 0.f);
    }
}

// Source coordinates per k-step of the split store: x[8], y[8], z[8] of its
// rows (a far dummy point for padding rows, which carry zero weights).
__global__ void source_ksteps_kernel(const int32_t *__restrict__ bsrc, int64_t nks, const float4 *__restrict__ sloc,
                                     float *__restrict__ sxyz) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nks * 8) return;
    const int64_t ks = t >> 3;
    const int i = (int)(t & 7);
    const int32_t r = bsrc[t];
    const float4 p = r >= 0 ? sloc[r] : make_float4(4.f, 4.f, 4.f, 0.f);
    sxyz[ks * 24 + i] = p.x;
    sxyz[ks * 24 + 8 + i] = p.y;
    sxyz[ks * 24 + 16 + i] = p.z;
}

// Basis store of the upward pass: per k-step b of an upward item (slot s,
// pool rows first..first+cnt-1), the FP64 BLI factors of its 8 points over the
// slot panel's nodes, rounded to FP32: F[i][8] (xi nodes) then G[j][8] (eta
// nodes); zero for padding rows.  One thread per (k-step, point).
__global__ void basis_store_kernel(const int32_t *__restrict__ bas, int64_t nbk, const double2 *__restrict__ xieta,
                                   const double *__restrict__ src_nodes, int n, float *__restrict__ basis) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nbk * 8) return;
    const int64_t b = t >> 3;
    const int i = (int)(t & 7);
    const int s = bas[3 * b], first = bas[3 * b + 1], cnt = bas[3 * b + 2];
    float *F = basis + b * 16 * n, *G = F + 8 * n;
    if (i >= cnt) {
        for (int k = 0; k < n; ++k) F[8 * k + i] = G[8 * k + i] = 0.f;
        return;
    }
    const double2 e = xieta[first + i];
    const double *nodes = src_nodes + (size_t)s * 2 * n;
    double f[kMaxDegree + 1];
    dev::bli_basis(e.x, nodes, n, f);
    for (int k = 0; k < n; ++k) F[8 * k + i] = (float)f[k];
    dev::bli_basis(e.y, nodes + n, n, f);
    for (int k = 0; k < n; ++k) G[8 * k + i] = (float)f[k];
}

// Per pool point, the self pair of sal_grad_gfunc (fast_sum_module.f90:9-31)
// in FP64 divided by the kernel constant: the leaf epilogue multiplies it by
// the point's FP32 weight row, which carries the constant.
__global__ void self_pair_kernel(const double4 *__restrict__ pool, int n, double2 *__restrict__ selfk) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const double4 c = pool[p];
    dev::Tgt T;
    dev::tgt_init(T, c.x, c.y, c.z);
    double sx = 0.0, sy = 0.0;
    if (T.live) dev::gref_exact(T, c.x, c.y, c.z, sx, sy);
    selfk[p] = make_double2(sx / dev::kCons, sy / dev::kCons);
}

static_assert(tc_smem_need<0>() <= 227 * 1024 && tc_smem_need<2>() <= 227 * 1024,
              "the leaf kernel's shared memory fits one SM");

// Dynamic shared memory of a launch: above half of the SM's, so one CTA per
// SM, which owns all 512 tensor memory columns.
template <int TS>
static size_t tc_smem_launch() {
    return tc_smem_need<TS>() > 120 * 1024 ? tc_smem_need<TS>() : 120 * 1024;
}
size_t tc_smem_bytes() { return tc_smem_launch<0>(); }

template <int MODE, bool JOINT, bool F16 = false, int TS = 0>
static void launch_tc(const TcJoint &J, int nsm, int cta_groups, int *err, cudaStream_t st) {
    const int total = J.beg[J.ngrids];
    if (total <= 0) return;
    const size_t smem = tc_smem_launch<TS>();
    static std::atomic<unsigned long long> done{0};
    smem_attr_once((const void *)tc_leaf_kernel<MODE, JOINT, F16, TS>, (int)smem, done);
    // every SM busy, but no CTA longer than cta_groups groups: with short
    // CTAs, kernels of other streams (higher-priority grids) get SMs as CTAs
    // retire
    const int per = cta_groups > 0 ? cta_groups : 1;
    int grid = (total + per - 1) / per;
    if (grid < nsm) grid = total < nsm ? total : nsm;
    if constexpr (JOINT) tc_leaf_kernel<MODE, JOINT, F16, TS><<<grid, kThreads, smem, st>>>(J, err);
    else dev::launch_next(tc_leaf_kernel<MODE, JOINT, F16, TS>, grid, kThreads, smem, st, J, err);
}

template <int MODE, bool F16 = false, int TS = 0>
static void launch_tc(const TcArgs &a, int nsm, int cta_groups, int *err, cudaStream_t st) {
    TcJoint J{};
    J.g[0] = a;
    J.ngrids = 1;
    J.beg[0] = 0;
    J.beg[1] = a.ngroups;
    launch_tc<MODE, false, F16, TS>(J, nsm, cta_groups, err, st);
}

void launch_tc_leaf_joint(const TcArgs *grids, int ngrids, int nsm, int cta_groups, int *err, cudaStream_t st) {
    TcJoint J{};
    J.ngrids = ngrids;
    J.beg[0] = 0;
    for (int k = 0; k < ngrids; ++k) {
        J.g[k] = grids[k];
        J.beg[k + 1] = J.beg[k] + grids[k].ngroups;
    }
    // the caller checks that all grids use one operand precision
    if (grids[0].bstore16)
        launch_tc<0, true, true>(J, nsm, cta_groups, err, st);
    else
        launch_tc<0, true, false>(J, nsm, cta_groups, err, st);
}

void launch_tc_leaf(const TcArgs &a, int nsm, int cg, int *err, cudaStream_t st, int tiles) {
    if (a.bstore16 && a.ktile && tiles == 1)
        launch_tc<0, true, 1>(a, nsm, cg, err, st);
    else if (a.bstore16 && a.ktile && tiles == 2)
        launch_tc<0, true, 2>(a, nsm, cg, err, st);
    else if (a.bstore16 && a.ktile && tiles == 3)
        launch_tc<0, true, 3>(a, nsm, cg, err, st);
    else if (a.bstore16)
        launch_tc<0, true>(a, nsm, cg, err, st);
    else
        launch_tc<0, false>(a, nsm, cg, err, st);
}
void launch_tc_proxy(const TcArgs &a, int nsm, int cg, int *err, cudaStream_t st) { launch_tc<1>(a, nsm, cg, err, st); }
void launch_tc_upward(const TcArgs &a, int nsm, int cg, int *err, cudaStream_t st) { launch_tc<2>(a, nsm, cg, err, st); }

void launch_split_store(const int32_t *bsrc, int64_t k0, int64_t k1, const float *wF, const float *phiF,
                        float *bstore, cudaStream_t st) {
    const int64_t nk = k1 - k0;
    if (nk <= 0) return;
    const int64_t threads = nk * kF;
    dev::launch_next(split_store_kernel, (unsigned)((threads + 255) / 256), 256, 0, st, bsrc + k0 * 8, nk, wF, phiF,
                                                                          bstore + k0 * kWStepFloats);
}

void launch_field_max(const float *wF, int64_t nw, const float *phiF, int64_t np, unsigned *fmax, cudaStream_t st) {
    const int64_t blocks = (std::max(nw, np) + 15) / 16;
    if (blocks > 0)
        field_max_kernel<<<dim3((unsigned)std::min<int64_t>(blocks, 148 * 8), 2), 256, 0, st>>>(
            reinterpret_cast<const float4 *>(wF), nw, reinterpret_cast<const float4 *>(phiF), np, fmax);
}

void launch_split_store16(const int32_t *bsrc, int64_t nunits, const float *wF, const float *phiF,
                          const unsigned *fmax, void *bstore16, cudaStream_t st) {
    if (nunits <= 0) return;
    constexpr int64_t per = 256 / kF * kStoreUnits;   // units a block
    dev::launch_next(split_store16_kernel, (unsigned)((nunits + per - 1) / per), 256, 0, st,
                     reinterpret_cast<const int4 *>(bsrc), nunits, wF, phiF, fmax, static_cast<unsigned char *>(bstore16));
}

void launch_target_scales(const TcArgs &a, float *tscale, float *tinv, cudaStream_t st) {
    if (a.ngroups > 0) target_scales_kernel<<<a.ngroups, kTcRows, 0, st>>>(a, tscale, tinv);
}

void launch_down_basis(const TcArgs &a, float *out, cudaStream_t st) {
    if (a.ngroups > 0) down_basis_store_kernel<<<a.ngroups, kTcRows, 0, st>>>(a, out);
}

void launch_source_local(const double4 *pool, const int2 *ranges, const double4 *centres, int nranges, float4 *sloc,
                         cudaStream_t st) {
    if (nranges > 0) source_local_kernel<<<nranges, 128, 0, st>>>(pool, ranges, centres, sloc);
}

void launch_source_ksteps(const int32_t *bsrc, int64_t nks, const float4 *sloc, float *sxyz, cudaStream_t st) {
    if (nks > 0) source_ksteps_kernel<<<(unsigned)((nks * 8 + 255) / 256), 256, 0, st>>>(bsrc, nks, sloc, sxyz);
}

void launch_basis_store(const int32_t *bas, int64_t nbk, const double2 *xieta, const double *src_nodes, int n,
                        float *basis, cudaStream_t st) {
    if (nbk > 0)
        basis_store_kernel<<<(unsigned)((nbk * 8 + 255) / 256), 256, 0, st>>>(bas, nbk, xieta, src_nodes, n, basis);
}

void launch_self_pair(const double4 *pool, int n, double2 *selfk, cudaStream_t st) {
    if (n > 0) self_pair_kernel<<<(n + 255) / 256, 256, 0, st>>>(pool, n, selfk);
}

}  // namespace mix
}  // namespace sal
