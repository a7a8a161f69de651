// How a unit's pairs of the FP64 evaluation pass are dealt to the warps of its
// CTA (kernels.cu eval_kernel): cut in integers, so that a run ends exactly where
// the next one begins whatever the compiler fuses (cut in floats, 1,969 shapes of
// targets and sources lose or double a block of sources if one of the two
// differences at a boundary is fused), and shared with the host, where a test
// counts the pairs of every shape.
//
// Each of nt targets is taken `fold` times, for one residue of the sources mod
// fold each: nt fold lanes in chunks of 32.  A last chunk of m <= 16 lanes takes
// 32 / m residues more, side by side, and so weighs less.  The (chunk, source)
// plane is cut into one equal run per warp, which meets two chunks at most: its
// slots.
#pragma once
#include <cmath>
#include <cstdint>

#ifdef __CUDACC__
#define SAL_HD __host__ __device__ __forceinline__
#else
#define SAL_HD inline
#endif

namespace sal {

constexpr int kEvalWarps = 8, kEvalSlots = 2;
constexpr int kEvalMaxChunks = 8;   // one a warp; 256 targets fill 8 unfolded
static_assert(kEvalMaxChunks <= kEvalWarps && kEvalSlots == 2, "a warp's run is a chunk at most: it meets two");

struct EvalCut {
    int nt, fold;
    int nid, nch;         // lanes, chunks
    int nlast, rlast;     // the last chunk: lanes, residues side by side
    SAL_HD EvalCut(int nt_, int fold_) : nt(nt_), fold(fold_) {
        nid = nt * fold;
        nch = (nid + 31) >> 5;
        nlast = nid - 32 * (nch - 1);
        rlast = 32 / nlast;
    }
    // positions in the plane: 8 rlast a full chunk, 8 the last one; warp w's run
    // is [start(w), start(w + 1))
    SAL_HD int chunk() const { return kEvalWarps * rlast; }
    SAL_HD int start(int warp) const { return warp * ((nch - 1) * rlast + 1); }
    SAL_HD int first_chunk(int warp) const {
        const int c = start(warp) / chunk();
        return c < nch - 1 ? c : nch - 1;
    }
    // which slot of a warp holds chunk c; -1 or kEvalSlots and more: none
    SAL_HD int slot_of(int warp, int c) const {
        const int p = start(warp) - c * chunk();
        return p >= 0 ? (p < chunk() || c == nch - 1 ? 0 : -1) : p >= -chunk() ? 1 : kEvalSlots;
    }
};

// One lane's part of a chunk.
struct EvalShare {
    int ti, res, step;      // target; residue and modulus of its sources
    float f0, f1, rstep;    // this run's part [f0, f1) of the chunk's blocks of `step` sources, 1 / step
    int work;
    // of n <= 256 sources this lane's: the first, `step` apart, and their end.
    // Products that nothing is added to: there is one way to round them.
    SAL_HD void sources(int n, int &beg, int &end) const {
        const float nb = floorf(((float)(n + step) - 0.5f) * rstep);   // ceil(n / step)
        const int e = (int)(nb * f1) * step;
        beg = (int)(nb * f0) * step + res;
        end = e < n ? e : n;
    }
};
SAL_HD EvalShare eval_share(const EvalCut &u, int warp, int lane, int slot) {
    const int c = u.first_chunk(warp) + slot;
    const bool last = c == u.nch - 1;
    const int n = last ? u.nlast : 32, r = last ? u.rlast : 1, id = 32 * c + lane % n;
    const int span = last ? kEvalWarps : u.chunk(), base = c * u.chunk();
    const int lo = u.start(warp) - base, hi = u.start(warp + 1) - base;
    EvalShare s;
    s.ti = id % u.nt;
    s.res = id / u.nt + u.fold * (lane / n);
    s.step = u.fold * r;
    s.rstep = 1.f / (float)s.step;
    s.f0 = (float)(lo < 0 ? 0 : lo) / (float)span;
    s.f1 = (float)(hi < span ? hi : span) / (float)span;
    s.work = c < u.nch && s.res < s.step && s.f0 < s.f1;
    return s;
}

// How often a set of nt targets is taken (EvalUnit::fold): the number that
// leaves the fewest idle lanes in chunks of 32, up to one chunk a warp (81
// proxies: 3 x 81 lanes fill 8 chunks to 95 %, 84 % unfolded).  More chunks
// than warps were no faster at 2.3M cells (148 targets in 19 chunks: 19.9 ms
// for the leaf units, as unfolded): what the lanes gain, the state that a warp
// swaps per chunk and stage takes back.
inline int32_t eval_fold(int32_t nt) {
    int32_t best = 1;
    double least = 1e30;
    for (int32_t f = 1; f <= 8; ++f) {
        const int32_t nid = nt * f, nch = (nid + 31) / 32, nlast = nid - 32 * (nch - 1);
        if (nch > kEvalMaxChunks && f > 1) break;
        const double c = (nch - 1 + 1.0 / (32 / nlast)) * 32.0 / nid;   // the last chunk takes 32 / nlast residues at once
        if (c < least - 1e-12) { least = c; best = f; }
    }
    return best;
}

}  // namespace sal
