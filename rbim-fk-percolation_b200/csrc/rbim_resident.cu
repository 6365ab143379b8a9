// Resident engine: one lattice per CTA, held in shared memory for every sweep
// of a call.  A persistent grid pulls chains from a work queue (an atomic
// counter in global memory), loads the chain's spin and coupling planes, runs
// its sweeps entirely on chip and writes back only the spin plane, the bin
// sums and the optional per-sweep records.
//
// Labelling runs in two stages so that a whole L = 256 lattice fits one CTA:
//  1. the open lattice (every bond except the 2L that close the periodic
//     boundary) is labelled with a union-find of 16-bit parents: inside the
//     open rectangle every cycle is contractible, so no image offsets are
//     needed and each open cluster's root is its smallest site;
//  2. the roots of the open clusters that touch a seam bond are hashed into a
//     small table whose union-find words carry image offsets; the seam bonds
//     are unioned there, and a seam bond that closes a loop with nonzero
//     summed offset winds around the torus (the exact test of the reference,
//     src/rbim/_unionfind.py:104-124).  Each merged open root is then pointed
//     at the smallest open root of its full cluster.
//
// This replaces, per chain, the loop of run_single_realization
// (src/rbim/simulation.py:196-242) around sw_sweep
// (src/rbim/swendsen_wang.py:103-172).
#include <algorithm>

#include "rbim_internal.h"
#include "rbim_phases.cuh"

namespace rbim {

namespace {

constexpr uint32_t kMaxResidentSites = 65536;  // 16-bit parents
// Dynamic shared memory budget: the 227 KB per-CTA limit minus room for the
// kernels' static shared scratch.
constexpr size_t kMaxSmem = 227 * 1024 - 8 * 1024;
constexpr uint32_t kHashEmpty = 0xFFFFFFFFu;
// Shared memory of one SM, and what a CTA takes beside its dynamic part: the
// per-CTA reservation of 1 KB and the static scratch (Red<512>, 0.8 KB), when
// deciding how many CTAs fit an SM.
constexpr size_t kSmemPerSm = 228 * 1024;
constexpr size_t kStaticSmem = 1024 + 832;

__host__ __device__ constexpr size_t align16(size_t v) { return (v + 15) & ~size_t(15); }

__host__ __device__ constexpr uint32_t hash_size(uint32_t l_max)
{
    // A slot for every end of the 2L seam bonds; few of them are ever taken
    // (bonds inside one open cluster need none, clusters have several ends),
    // and every slot is reset and looked at in every sweep.
    uint32_t h = 32;
    while (h < 4u * l_max) h *= 2;
    return h;
}

}  // namespace

// Optional per-phase cycle accounting (profiling builds only, compiled with
// -DRBIM_PROFILE_PHASES): thread 0 adds the cycles since the previous mark to
// a per-phase counter at each barrier.  No work is skipped.
#ifdef RBIM_PROFILE_PHASES
__device__ unsigned long long g_phase_cycles[16];
__device__ __forceinline__ void phase_mark(int k)
{
    __shared__ long long s_t;
    if (threadIdx.x == 0) {
        const long long now = clock64();
        if (k >= 0) atomicAdd(&g_phase_cycles[k], (unsigned long long)(now - s_t));
        s_t = now;
    }
}
#define RBIM_PHASE_MARK(k) phase_mark(k)
__device__ unsigned long long g_event_counts[8];
#define RBIM_COUNT(k, v) atomicAdd(&g_event_counts[k], (unsigned long long)(v))
#define RBIM_PROF_ONLY(...) __VA_ARGS__
#else
#define RBIM_PHASE_MARK(k) ((void)0)
#define RBIM_COUNT(k, v) ((void)0)
#define RBIM_PROF_ONLY(...)
#endif

}  // namespace rbim

#include "rbim_open.cuh"

namespace rbim {

// Seam union-find word: parent slot (12 bits) | wx (10 bits) | wy (10 bits),
// offsets modulo 1024 (exact for L < 1024, see rbim_device.cuh).
struct SeamWord {
    using T = uint32_t;
    __device__ __forceinline__ static uint32_t parent(T w) { return w & 0xFFFu; }
    __device__ __forceinline__ static int ox(T w) { return ((int)(w << 10)) >> 22; }
    __device__ __forceinline__ static int oy(T w) { return ((int)w) >> 22; }
    __device__ __forceinline__ static T make(uint32_t p, int x, int y)
    {
        return (p & 0xFFFu) | ((uint32_t)(x & 0x3FF) << 12) | ((uint32_t)(y & 0x3FF) << 22);
    }
    __device__ __forceinline__ static bool nonzero(int v) { return (v & 0x3FF) != 0; }
};

// Shared-memory layout for lattices of up to l_max x l_max sites; constexpr so
// that the launches of the common size classes get it as a compile-time
// constant (the kernel's shared-memory views then need no registers).
__host__ __device__ constexpr ResidentLayout resident_layout_c(uint32_t l_max, int threads)
{
    ResidentLayout ly{};
    ly.l_max = l_max;
    ly.n_max = l_max * l_max;
    const uint32_t nw = (ly.n_max + 31u) / 32u;
    ly.nw_max = (nw + 3u) & ~3u;
    ly.hs = hash_size(l_max);
    size_t off = 0;
    ly.off_uf = off;
    off = align16(off + 2ull * ly.n_max);
    const size_t plane = 4ull * (ly.nw_max + 4u);
    ly.off_S = off;
    off += plane;
    ly.off_JH = off;
    off += plane;
    ly.off_JV = off;
    off += plane;
    ly.off_OH = off;
    off += plane;
    ly.off_OV = off;
    off += plane;
    ly.off_FLIP = off;
    off += plane;
    ly.off_ROOT = off;
    off += plane;
    // Row-end masks, for the CTA sizes of the small lattices: several rows end
    // in a word there (16384 lattices, us a sweep with the plane / with masks
    // computed by the reciprocal: L = 32 207 / 211, 44 398 / 404, 64 588 / 592,
    // 40 365 / 366, 16, 24, 48 and 56 the same). Larger CTAs compute them:
    // without the plane a fourth CTA of 256 threads fits an SM at L = 127 and
    // 128 (-8 %).
    ly.off_RE = off;
    if (threads <= 128) off += plane;
    ly.off_SEAMV = off;
    off = align16(off + 4ull * (((l_max + 31u) / 32u) + 4u));
    ly.off_HK = off;
    off += 4ull * ly.hs;
    ly.off_HW = off;
    off += 4ull * ly.hs;
    // The warps' union lists, in the seam tables' memory (reset after the
    // unions) where that gives every warp at least 128 entries, else beside it:
    // 256 entries in CTAs that have the SM to themselves, 32 in others.
    const uint32_t nwarps = (uint32_t)threads / 32u;
    ly.off_LIST = ly.off_HK;
    ly.seg = 4u * ly.hs / nwarps;
    if (ly.seg < 128u || threads == 1024) {
        ly.off_LIST = off;
        ly.seg = threads == 1024 ? 256u : 32u;
        off += 2ull * ly.seg * nwarps;
    }
    ly.bytes = align16(off);
    return ly;
}

ResidentLayout resident_layout(uint32_t l_max, int threads) { return resident_layout_c(l_max, threads); }

int resident_max_l()
{
    int best = 3;
    for (int L = 3; L <= 256; ++L) {
        if ((uint32_t)(L * L) > kMaxResidentSites) break;
        if (resident_layout(L, 1024).bytes <= kMaxSmem) best = L;
    }
    return best;
}

int resident_default_threads(int l_max)
{
    // At 64 registers a thread an SM holds 1024 of this kernel's threads
    // whatever the CTA size, and several small CTAs per SM hide each other's
    // barrier waits better than one large one; so the CTA is as small as the
    // lattice allows before its per-thread work grows long and its shared
    // memory keeps threads off the SM.  Measured on B200, cycles a site and SM
    // with half / this / twice the threads: L = 32: - / 4.2 / 4.5; L = 40: 5.0
    // / 4.2 / 5.0; L = 48: 4.0 / 4.1 / 4.9; L = 64: 3.0 / 2.7 / 3.3; L = 72: 3.1
    // / 3.0 / 4.6; L = 124: 3.2 / 2.1 / 2.8; L = 144: 2.6 / 2.6 / 3.3; L = 192:
    // 3.1 / 2.6 / 2.8, and above, where one CTA of 512 threads would have the
    // SM to itself, L = 224: 5.4 / 3.4 / 2.6.
    if (l_max <= 32) return 32;
    if (l_max <= 44) return 64;
    if (l_max <= 64) return 128;
    if (l_max <= 128) return 256;
    if (2 * (resident_layout_c((uint32_t)l_max, 512).bytes + kStaticSmem) <= kSmemPerSm) return 512;
    return 1024;
}

// Shared scratch of one CTA.
template <int NT>
struct Red {
    uint32_t k1[NT / 32], k2[NT / 32];
    uint32_t unsat[NT / 32], downs[NT / 32], roots[NT / 32], in[NT / 32], in_downs[NT / 32];
    int mc[NT / 32], mc2[NT / 32];
    int item, wrap, err;
    // State of the chain being processed; only thread 0 updates it.
    Acc acc;
    long long cur_bin;
    rbim_chain_t ch;
};

// Blocks per SM the register budget is tuned for (64 registers per thread).
template <int NT>
struct MinBlocks {
    static constexpr int value = NT >= 1024 ? 1 : 1024 / NT;
};

// Per-CTA view of the shared-memory arrays of one lattice.
struct Res {
    Lat<Word16> t;
    uint32_t *HK;  // seam hash keys: open root site, or kHashEmpty
    uint32_t *HW;  // seam union-find words (SeamWord)
    uint32_t hs, hs_log2;
    unsigned short *LIST;  // union lists, `seg` entries per warp
    uint32_t seg;
};

// walk_cap > 0 lowers the per-walk bound (and with it the per-thread loop
// bounds, 64 walks' worth) from N + 64 steps to walk_cap: the chain
// descriptor's test hook that makes the bounds fire on a small lattice.
template <int NT>
__device__ __forceinline__ Res make_res(unsigned char *smem, const ResidentLayout &ly, uint32_t L, Red<NT> &red,
                                        int64_t walk_cap = 0)
{
    Res r;
    Lat<Word16> &t = r.t;
    t.g = Geom{L, L * L, (L * L + 31u) / 32u};
    t.uf.w = (unsigned short *)(smem + ly.off_uf);
    t.uf.sa = (uint32_t)__cvta_generic_to_shared(t.uf.w);
    t.S = (uint32_t *)(smem + ly.off_S);
    t.JH = (const uint32_t *)(smem + ly.off_JH);
    t.JV = (const uint32_t *)(smem + ly.off_JV);
    t.OH = (uint32_t *)(smem + ly.off_OH);
    t.OV = (uint32_t *)(smem + ly.off_OV);
    t.FLIP = (uint32_t *)(smem + ly.off_FLIP);
    t.ROOT = (uint32_t *)(smem + ly.off_ROOT);
    t.NEED = t.ROOT;  // read by the unions, before the roots are recorded
    t.RE = NT <= 128 ? (const uint32_t *)(smem + ly.off_RE) : nullptr;
    t.inv = NT <= 128 ? 0u : 0xFFFFFFFFu / L + 1u;
    t.SEAMV = (uint32_t *)(smem + ly.off_SEAMV);
    t.wrap = &red.wrap;
    t.err = &red.err;
    t.cap = (walk_cap > 0 && walk_cap < (int64_t)(t.g.N + 64u)) ? (uint32_t)walk_cap : t.g.N + 64u;
    r.HK = (uint32_t *)(smem + ly.off_HK);
    r.HW = (uint32_t *)(smem + ly.off_HW);
    r.hs = ly.hs;
    r.hs_log2 = 31u - __clz(ly.hs);
    r.LIST = (unsigned short *)(smem + ly.off_LIST);
    r.seg = ly.seg;
    return r;
}

// The row-end masks (once per chain).
template <int NT>
__device__ __forceinline__ void init_row_ends(const Lat<Word16> &t, uint32_t tid)
{
    if (NT > 128) return;
    uint32_t *re = const_cast<uint32_t *>(t.RE);
    for (uint32_t w = tid; w < t.g.NW; w += NT) re[w] = t.g.row_end(w);
}

__device__ __forceinline__ uint32_t hash_insert(const Res &r, uint32_t key, int *err)
{
    uint32_t h = (key * 0x9E3779B1u) >> (32u - r.hs_log2);
    for (uint32_t it = 0; it < r.hs; ++it) {
        const uint32_t old = atomicCAS(r.HK + h, kHashEmpty, key);
        if (old == kHashEmpty || old == key) return h;
        h = (h + 1u) & (r.hs - 1u);
    }
    atomicOr(err, kErrUnionCap);
    return 0;
}

// Union of two seam nodes across a seam bond with seam crossing (ex, ey); the
// node whose open root is larger is hooked under the other.
__device__ __forceinline__ void seam_union(const Res &r, uint32_t na, uint32_t nb, int ex, int ey, int *wrap,
                                           uint32_t cap, int *err)
{
    const UF<SeamWord> hw{r.HW};
    for (uint32_t it = 0; it < cap; ++it) {
        const FindResult fa = uf_find<SeamWord>(hw, na, cap, err);
        const FindResult fb = uf_find<SeamWord>(hw, nb, cap, err);
        if (fa.root == fb.root) {
            int f = 0;
            if (SeamWord::nonzero(ex + fb.ax - fa.ax)) f |= 1;
            if (SeamWord::nonzero(ey + fb.ay - fa.ay)) f |= 2;
            if (f) atomicOr(wrap, f);
            return;
        }
        const uint32_t ka = r.HK[fa.root], kb = r.HK[fb.root];
        if (ka < kb) {
            const uint32_t expect = SeamWord::make(fb.root, 0, 0);
            if (hw.cas(fb.root, expect, SeamWord::make(fa.root, fa.ax - ex - fb.ax, fa.ay - ey - fb.ay)) == expect)
                return;
        } else {
            const uint32_t expect = SeamWord::make(fa.root, 0, 0);
            if (hw.cas(fa.root, expect, SeamWord::make(fb.root, fb.ax + ex - fa.ax, fb.ay + ey - fa.ay)) == expect)
                return;
        }
    }
    atomicOr(err, kErrUnionCap);
}

// Seam table reset (before the seam phase): each warp resets the 1 / nwarps of
// the two tables that its union list may have used, after its unions.
__device__ __forceinline__ void seam_reset(const Res &r, uint32_t warp, uint32_t nwarps)
{
    const uint32_t per = 2u * r.hs / nwarps, end = (warp + 1u) * per;
    for (uint32_t k = warp * per + (threadIdx.x & 31u); k < end; k += 32u)
        r.HK[k] = k < r.hs ? kHashEmpty : SeamWord::make(k - r.hs, 0, 0);  // HW follows HK
}

// (b) Seam bonds: x seam (x = L-1 -> 0, crossing (1,0)) and y seam
// (y = L-1 -> 0, crossing (0,1)).  The open union-find is final here.  A bond
// inside one open cluster closes a loop that winds once (no path inside the
// open lattice crosses a seam) and needs no node; one that joins the same two
// open clusters with the same crossing as the lane before closes a loop of
// winding zero.
__device__ __forceinline__ void phase_seam(const Res &r, uint32_t tid, uint32_t nthreads)
{
    const Lat<Word16> &t = r.t;
    const Geom &g = t.g;
    const uint32_t lane = tid & 31u;
    for (uint32_t i0 = tid & ~31u; i0 < 2u * g.L; i0 += nthreads) {
        const uint32_t i = i0 + lane;
        uint32_t a = 0, b = 0;
        int ex = 0, ey = 0;
        if (i < g.L) {
            a = g.N - g.L + i;
            b = i;
            ex = (t.OH[a >> 5] >> (a & 31u)) & 1u;
        } else if (i < 2u * g.L) {
            const uint32_t x = i - g.L;
            b = x * g.L;
            a = b + g.L - 1u;
            ey = (t.SEAMV[x >> 5] >> (x & 31u)) & 1u;
        }
        bool live = ex | ey;
        if (live) {
            for (uint32_t it = 0;; ++it) {
                const uint32_t pa = t.uf.ld(a), pb = t.uf.ld(b);
                if (pa == a && pb == b) break;
                a = pa;
                b = pb;
                if (it >= t.cap) {
                    atomicOr(t.err, kErrFindCap);
                    break;
                }
            }
            if (a == b) {
                atomicOr(t.wrap, ex | 2 * ey);
                live = false;
            }
        }
        const uint32_t what = live ? (a << 16 | b) : 0u;  // a != b, so never 0
        const uint32_t before = __shfl_up_sync(0xFFFFFFFFu, what, 1);
        const int ex_before = __shfl_up_sync(0xFFFFFFFFu, ex, 1);
        if (!live || (lane > 0u && before == what && ex_before == ex)) continue;
        const uint32_t na = hash_insert(r, a, t.err);
        const uint32_t nb = hash_insert(r, b, t.err);
        seam_union(r, na, nb, ex, ey, t.wrap, t.cap, t.err);
    }
}

// (b) Point every merged open root at the smallest open root of its cluster.
__device__ __forceinline__ void phase_seam_propagate(const Res &r, uint32_t tid, uint32_t nthreads)
{
    const UF<SeamWord> hw{r.HW};
    for (uint32_t k = tid; k < r.hs; k += nthreads) {
        const uint32_t key = r.HK[k];
        if (key == kHashEmpty) continue;
        const uint32_t g = uf_root_ro<SeamWord>(hw, k, r.hs + 1u, r.t.err);
        if (g != k) r.t.uf.st(key, (unsigned short)r.HK[g]);
    }
}

// Phases as separate (non-inlined) functions, for the CTA sizes where that
// measured faster on B200 (fewer registers live across the phase than inline;
// the larger CTAs lose up to 15 % by it).  us a sweep of 16384 lattices,
// inline against separate: measurement in one-warp CTAs, L = 32: 222 / 203;
// heads with 64 threads, L = 40: 371 / 354; heads and roots with 128 threads,
// L = 64: 597 / 576.
template <int NT, bool kFew>
static __device__ __noinline__ void separate_heads(const Lat<Word16> &t, uint32_t warp)
{
    phase_heads_open<kFew>(t, warp, NT / 32);
}

template <int NT, bool kSweep, int K>
static __device__ __noinline__ void separate_roots(const Lat<Word16> &t, uint32_t *in, uint32_t root, uint32_t warp)
{
    roots_flip_sites<kSweep, K>(t, in, root, warp, NT / 32);
}

// The labelling stages shared by the sweep and label kernels, from occupied
// bond planes to final roots (every site's word at its root, the ROOT plane);
// barriers between stages.  kSweep: the clusters are flipped, and in measured
// sweeps the sites of the cluster most likely to be the largest are left in
// the OH plane (free once the seams are done) and its root returned.
template <int NT, bool kFew, bool kSweep>
__device__ __forceinline__ uint32_t resident_label(const Res &r, bool measure)
{
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    constexpr uint32_t nwarps = NT / 32;
    // Words a warp takes at a time in the roots pass.  Measured on B200, cycles
    // a site and SM with 1 / 2 / 4 / 8 words: L = 256 (1024 threads) 2.69 /
    // 2.53 / 2.46 / 2.49, L = 64 (128) 3.18 / 3.04 / 2.98 / 3.11, L = 32 (one
    // warp, many CTAs hide each other's latency) 5.70 / 5.92 / 6.12 / 6.26.
    constexpr int kWords = NT <= 64 ? 1 : 4;
    unsigned short *list = r.LIST + warp * r.seg;
    if constexpr (NT == 64 || NT == 128)
        separate_heads<NT, kFew>(r.t, warp);
    else
        phase_heads_open<kFew>(r.t, warp, nwarps);
    __syncthreads();
    RBIM_PHASE_MARK(1);
    phase_union_open<kFew>(r.t, list, r.seg, warp, nwarps);
    seam_reset(r, warp, nwarps);
    __syncthreads();
    RBIM_PHASE_MARK(2);
    phase_seam(r, tid, NT);
    __syncthreads();
    RBIM_PHASE_MARK(3);
    phase_seam_propagate(r, tid, NT);
    for (uint32_t i = tid; i < (r.t.g.L + 31u) / 32u; i += NT) r.t.SEAMV[i] = 0u;
    __syncthreads();
    RBIM_PHASE_MARK(4);
    const uint32_t likely = kSweep && measure ? likely_largest(r.t) : 0u;
    uint32_t *members = kSweep && measure ? r.t.OH : nullptr;
    if constexpr (NT == 128)
        separate_roots<NT, kSweep, kWords>(r.t, members, likely, warp);
    else
        roots_flip_sites<kSweep, kWords>(r.t, members, likely, warp, nwarps);
    __syncthreads();
    RBIM_PHASE_MARK(5);
    return likely;
}

// Measurement of one sweep after resident_label: energy, magnetization,
// n_clusters, S1, S2, |M_C1| and, with `second` (records requested), |M_C2|
// (reference sw_sweep, src/rbim/swendsen_wang.py:146-172).  The cluster rooted
// at `likely`, whose sites are the set bits of OH, is counted and its
// magnetization summed by popcounts; when it turns out to be the largest (as
// it does whenever one cluster dominates) no pass for |M_C1| is needed.  Ends
// with a barrier.  Thread 0 returns the record in rec.
template <int NT>
__device__ __forceinline__ void resident_measure(const Res &res, Red<NT> &red, uint32_t likely,
                                                 long long rec[kRecLen], bool second)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    constexpr uint32_t nwarps = NT / 32;
    const Lat<Word16> &t = res.t;
    const Geom &g = t.g;
    unsigned short *u16 = t.uf.w;

    // Energy and magnetization of the flipped spins; clusters; size and down
    // spins of the likely largest.
    uint32_t unsat = 0, downs = 0, ncl = 0, in = 0, in_downs = 0;
    measure_energy(t, tid, NT, unsat, downs);
    for (uint32_t w = tid; w < g.NW; w += NT) {
        const uint32_t c = t.OH[w];
        ncl += __popc(t.ROOT[w]);
        in += __popc(c);
        in_downs += __popc(c & t.S[w]);
    }
    unsat = __reduce_add_sync(0xFFFFFFFFu, unsat);
    downs = __reduce_add_sync(0xFFFFFFFFu, downs);
    ncl = __reduce_add_sync(0xFFFFFFFFu, ncl);
    in = __reduce_add_sync(0xFFFFFFFFu, in);
    in_downs = __reduce_add_sync(0xFFFFFFFFu, in_downs);
    if (lane == 0) {
        red.unsat[warp] = unsat;
        red.downs[warp] = downs;
        red.roots[warp] = ncl;
        red.in[warp] = in;
        red.in_downs[warp] = in_downs;
    }
    RBIM_PHASE_MARK(6);
    // Cluster sizes minus one into the root words, on top of the index each
    // holds; the likely largest cluster is counted above.
    count_pieces(t, u16, t.OH, warp, nwarps);
    __syncthreads();
    RBIM_PHASE_MARK(7);
    // Every warp sums the per-warp partials itself (no barrier needed after).
    const bool live = lane < nwarps;
    const uint32_t unsat_t = __reduce_add_sync(0xFFFFFFFFu, live ? red.unsat[lane] : 0u);
    const uint32_t downs_t = __reduce_add_sync(0xFFFFFFFFu, live ? red.downs[lane] : 0u);
    ncl = __reduce_add_sync(0xFFFFFFFFu, live ? red.roots[lane] : 0u);
    in = __reduce_add_sync(0xFFFFFFFFu, live ? red.in[lane] : 0u);
    in_downs = __reduce_add_sync(0xFFFFFFFFu, live ? red.in_downs[lane] : 0u);
    const long long M = (long long)g.N - 2ll * (long long)downs_t;
    long long mc_total = M, mc2_total = 0;
    uint32_t size1 = g.N, size2 = 0u;
    if (ncl > 1) {
        uint32_t k1 = 0, k2 = 0;
        for (uint32_t w = tid; w < g.NW; w += NT) {
            uint32_t roots = t.ROOT[w];
            while (roots) {
                const uint32_t b = __ffs(roots) - 1u;
                roots &= roots - 1u;
                const uint32_t r = (w << 5) + b;
                const uint32_t size = r == likely ? in : counted_size(u16, r);
                top2_merge(k1, k2, (size << 16) | (0xFFFFu - r), 0u);
            }
        }
        warp_top2(k1, k2);
        if (lane == 0) {
            red.k1[warp] = k1;
            red.k2[warp] = k2;
        }
        __syncthreads();
        uint32_t a1 = live ? red.k1[lane] : 0u, a2 = live ? red.k2[lane] : 0u;
        warp_top2(a1, a2);
        RBIM_PHASE_MARK(8);
        const uint32_t g1 = 0xFFFFu - (a1 & 0xFFFFu), g2 = 0xFFFFu - (a2 & 0xFFFFu);
        size1 = a1 >> 16;
        size2 = a2 >> 16;
        mc_total = (long long)in - 2ll * (long long)in_downs;
        if (g1 != likely || second) {
            // Lanes are sites; every site's word holds its root (a root's own
            // word its size, so roots are known by their ROOT bit).  Two words
            // per iteration keep two load chains in flight.
            int mc = 0, mc2 = 0;
            for (uint32_t w0 = warp; w0 < g.NW; w0 += 2u * nwarps) {
                const uint32_t w1 = w0 + nwarps;
                const uint32_t n0 = (w0 << 5) + lane, n1 = (w1 << 5) + lane;
                const uint32_t rt0 = t.ROOT[w0], rt1 = w1 < g.NW ? t.ROOT[w1] : 0u;
                const bool ok0 = n0 < g.N, ok1 = n1 < g.N;
                const uint32_t p0 = ok0 ? (uint32_t)u16[n0] : 0u, p1 = ok1 ? (uint32_t)u16[n1] : 0u;
                const uint32_t r0 = ((rt0 >> lane) & 1u) ? n0 : p0, r1 = ((rt1 >> lane) & 1u) ? n1 : p1;
                const uint32_t m0 = __ballot_sync(0xFFFFFFFFu, ok0 && r0 == g1);
                const uint32_t m1 = __ballot_sync(0xFFFFFFFFu, ok1 && r1 == g1);
                const uint32_t s0 = t.S[w0], s1 = w1 < g.NW ? t.S[w1] : 0u;
                if (lane == 0) mc += (int)__popc(m0) - 2 * (int)__popc(m0 & s0) + (int)__popc(m1) - 2 * (int)__popc(m1 & s1);
                if (second) {
                    const uint32_t q0 = __ballot_sync(0xFFFFFFFFu, ok0 && r0 == g2);
                    const uint32_t q1 = __ballot_sync(0xFFFFFFFFu, ok1 && r1 == g2);
                    if (lane == 0) mc2 += (int)__popc(q0) - 2 * (int)__popc(q0 & s0) + (int)__popc(q1) -
                                          2 * (int)__popc(q1 & s1);
                }
            }
            if (lane == 0) {
                red.mc[warp] = mc;
                red.mc2[warp] = mc2;
            }
            __syncthreads();
            RBIM_PHASE_MARK(9);
            mc_total = (int)__reduce_add_sync(0xFFFFFFFFu, (uint32_t)(live ? red.mc[lane] : 0));
            mc2_total = (int)__reduce_add_sync(0xFFFFFFFFu, (uint32_t)(live ? red.mc2[lane] : 0));
        }
    }
    if (tid == 0) {
        rec[0] = 2ll * (long long)unsat_t - 2ll * (long long)g.N;
        rec[1] = M;
        rec[2] = ncl;
        rec[3] = size1;
        rec[4] = mc_total < 0 ? -mc_total : mc_total;
        rec[5] = size2;
        rec[6] = mc2_total < 0 ? -mc2_total : mc2_total;
        rec[7] = red.wrap & 1;
        rec[8] = (red.wrap >> 1) & 1;
    }
    __syncthreads();
}

template <int NT>
static __device__ __noinline__ void separate_measure(const Res &res, Red<NT> &red, uint32_t likely,
                                                     long long rec[kRecLen], bool second)
{
    resident_measure<NT>(res, red, likely, rec, second);
}

// LC > 0: the launch's layout is resident_layout_c(LC, NT), a compile-time
// constant; LC == 0: the layout passed in.
template <int NT, int LC>
__global__ void __launch_bounds__(NT, MinBlocks<NT>::value)
    k_resident_sweeps(rbim_chain_t *chains, int n_chains, uint32_t *spin_pool, const uint32_t *coupling_pool,
                      long long *acc_i, double *acc_f, int32_t *records, int n_sweeps, int *queue, int *status,
                      ResidentLayout ly_arg)
{
    constexpr ResidentLayout kly = resident_layout_c(LC > 0 ? LC : 16, NT);
    const ResidentLayout ly = LC > 0 ? kly : ly_arg;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Red<NT> red;
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    constexpr uint32_t nwarps = NT / 32;

    if (tid == 0) red.err = 0;
    for (;;) {
        if (tid == 0) {
            red.item = atomicAdd(queue, 1);
            if (red.item < n_chains) {
                red.ch = chains[red.item];
                red.cur_bin = -1;
            }
        }
        __syncthreads();
        const int item = red.item;
        if (item >= n_chains) break;
        const rbim_chain_t &ch = red.ch;
        if (ch.L < 3 || ch.L > (int64_t)ly.l_max || ch.sweeps_per_bin < 1 || ch.n_bins < 0 || ch.n_therm < 0 ||
            ch.walk_cap < 0) {
            if (tid == 0) atomicOr(status, kErrBadChain);
            __syncthreads();
            continue;
        }
        const uint32_t L = (uint32_t)ch.L;
        const Res res = make_res<NT>(smem, ly, L, red, ch.walk_cap);
        const Lat<Word16> &t = res.t;
        const Geom g = t.g;
        const uint32_t nwp = (g.NW + 3u) & ~3u;

        // Load the chain's planes (16-byte aligned, whole padded planes).
        {
            const uint4 *gs = (const uint4 *)(spin_pool + ch.spin_off);
            const uint4 *gh = (const uint4 *)(coupling_pool + ch.coupling_off);
            const uint4 *gv = (const uint4 *)(coupling_pool + ch.coupling_off + nwp);
            for (uint32_t i = tid; i < nwp / 4u; i += NT) {
                ((uint4 *)t.S)[i] = gs[i];
                ((uint4 *)t.JH)[i] = gh[i];
                ((uint4 *)t.JV)[i] = gv[i];
            }
            for (uint32_t i = tid; i < (L + 31u) / 32u; i += NT) t.SEAMV[i] = 0u;
            init_row_ends<NT>(t, tid);
        }
        const uint64_t t_end = (uint64_t)ch.n_therm + (uint64_t)ch.n_bins * (uint64_t)ch.sweeps_per_bin;
        uint64_t sweep = ch.sweep;
        const uint64_t stop = min(t_end, sweep + (uint64_t)max(n_sweeps, 0));
        __syncthreads();

        for (; sweep < stop; ++sweep) {
            const bool measure = sweep >= (uint64_t)ch.n_therm;
            if (tid == 0) red.wrap = 0;
            RBIM_PHASE_MARK(-1);
            phase_activate<Word16>(t, make_rng(ch.key, sweep, ch.thr), warp, nwarps, tid, NT);
            __syncthreads();
            RBIM_PHASE_MARK(0);
            const uint32_t likely = resident_label<NT, NT >= 512 && LC == 0, true>(res, measure);
            if (measure) {
                long long rec[kRecLen];
                const bool want_rec = records && ch.rec_off >= 0;
                if constexpr (NT == 32)
                    separate_measure<NT>(res, red, likely, rec, want_rec);
                else
                    resident_measure<NT>(res, red, likely, rec, want_rec);
                if (tid == 0) {
                    const long long idx = (long long)(sweep - (uint64_t)ch.n_therm);
                    const long long bin = idx / ch.sweeps_per_bin;
                    if (bin != red.cur_bin) {
                        if (red.cur_bin >= 0)
                            red.acc.store(acc_i + (ch.acc_off + red.cur_bin) * kAccInt,
                                          acc_f + (ch.acc_off + red.cur_bin) * kAccF64);
                        // Resume from the stored sums so that additions stay in
                        // sweep order whatever the split into calls.
                        red.acc.load(acc_i + (ch.acc_off + bin) * kAccInt, acc_f + (ch.acc_off + bin) * kAccF64);
                        red.cur_bin = bin;
                    }
                    red.acc.add(rec[0], rec[1], rec[2], rec[3], rec[4], rec[5], (int)rec[7], (int)rec[8]);
                    if (want_rec) {
                        int32_t *row = records + (ch.rec_off + idx) * kRecLen;
#pragma unroll
                        for (int k = 0; k < kRecLen; ++k) row[k] = (int32_t)rec[k];
                    }
                }
                RBIM_PHASE_MARK(10);
            }
        }
        if (tid == 0) {
            if (red.cur_bin >= 0)
                red.acc.store(acc_i + (ch.acc_off + red.cur_bin) * kAccInt,
                              acc_f + (ch.acc_off + red.cur_bin) * kAccF64);
            chains[item].sweep = stop;
        }
        // Write the spin plane back.
        {
            uint4 *gs = (uint4 *)(spin_pool + ch.spin_off);
            for (uint32_t i = tid; i < nwp / 4u; i += NT) gs[i] = ((const uint4 *)t.S)[i];
        }
        __syncthreads();
    }
    if (tid == 0 && red.err) atomicOr(status, red.err);
}

// Labelling only: frozen occupation bytes in, canonical labels out.
template <int NT>
__global__ void __launch_bounds__(NT, MinBlocks<NT>::value)
    k_resident_label(uint32_t L, const uint8_t *occ, int32_t *labels, int32_t *n_clusters, uint8_t *wraps,
                     int *status, ResidentLayout ly)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Red<NT> red;
    __shared__ uint32_t s_scan[NT];
    const uint32_t tid = threadIdx.x;
    const size_t lat = blockIdx.x;
    if (tid == 0) {
        red.err = 0;
        red.wrap = 0;
    }
    const Res res = make_res<NT>(smem, ly, L, red);
    const Lat<Word16> &t = res.t;
    const Geom g = t.g;
    const uint8_t *o = occ + lat * 2ull * g.N;
    for (uint32_t i = tid; i < (L + 31u) / 32u; i += NT) t.SEAMV[i] = 0u;
    init_row_ends<NT>(t, tid);
    __syncthreads();
    for (uint32_t w = tid; w < g.NW; w += NT) {
        uint32_t h = 0, v = 0;
        for (uint32_t b = 0; b < 32u; ++b) {
            const uint32_t n = (w << 5) + b;
            if (n >= g.N) break;
            h |= (o[2ull * n] ? 1u : 0u) << b;
            v |= (o[2ull * n + 1] ? 1u : 0u) << b;
        }
        const uint32_t re = t.row_end(w);
        t.OH[w] = h;
        t.OV[w] = v & ~re;
        uint32_t seam = v & re;
        while (seam) {
            const uint32_t b = __ffs(seam) - 1u;
            seam &= seam - 1u;
            const uint32_t x = t.row((w << 5) + b);
            atomicOr(t.SEAMV + (x >> 5), 1u << (x & 31u));
        }
    }
    __syncthreads();
    (void)resident_label<NT, false, false>(res, false);
    // Exclusive prefix of root counts over words -> FLIP plane (rank base).
    const uint32_t per = (g.NW + NT - 1u) / NT;
    const uint32_t w0 = tid * per, w1 = min(g.NW, w0 + per);
    uint32_t local = 0;
    for (uint32_t w = w0; w < w1; ++w) local += __popc(t.ROOT[w]);
    s_scan[tid] = local;
    __syncthreads();
    for (uint32_t off = 1; off < NT; off <<= 1) {
        const uint32_t v = tid >= off ? s_scan[tid - off] : 0u;
        __syncthreads();
        s_scan[tid] += v;
        __syncthreads();
    }
    uint32_t base = s_scan[tid] - local;
    for (uint32_t w = w0; w < w1; ++w) {
        t.FLIP[w] = base;
        base += __popc(t.ROOT[w]);
    }
    __syncthreads();
    int32_t *lab = labels + lat * (size_t)g.N;
    for (uint32_t n = tid; n < g.N; n += NT) {
        const uint32_t r = Word16::parent(t.uf.ld(n));
        lab[n] = (int32_t)(t.FLIP[r >> 5] + __popc(t.ROOT[r >> 5] & ((1u << (r & 31u)) - 1u)));
    }
    if (tid == 0) {
        n_clusters[lat] = (int32_t)s_scan[NT - 1];
        wraps[2 * lat] = (uint8_t)(red.wrap & 1);
        wraps[2 * lat + 1] = (uint8_t)((red.wrap >> 1) & 1);
        if (red.err) atomicOr(status, red.err);
    }
}

namespace {

template <int NT, int LC>
cudaError_t launch_sweeps_lc(const rbim_chain_t *chains, int n_chains, int l_max, uint32_t *spin_pool,
                             const uint32_t *coupling_pool, long long *acc_i, double *acc_f, int32_t *rec,
                             int n_sweeps, int grid, int *queue, int *status, cudaStream_t stream)
{
    const ResidentLayout ly = LC > 0 ? resident_layout_c(LC, NT) : resident_layout(l_max, NT);
    cudaError_t e = cudaFuncSetAttribute(k_resident_sweeps<NT, LC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)ly.bytes);
    if (e != cudaSuccess) return e;
    if (grid <= 0) {
        int per_sm = 0, sms = 0, dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (n_chains > sms) {
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_resident_sweeps<NT, LC>, NT, ly.bytes);
            if (e != cudaSuccess) return e;
        }
        grid = std::max(1, per_sm) * std::max(1, sms);
    }
    grid = std::min(grid, n_chains);
    e = cudaMemsetAsync(queue, 0, sizeof(int), stream);
    if (e != cudaSuccess) return e;
    k_resident_sweeps<NT, LC><<<grid, NT, ly.bytes, stream>>>(const_cast<rbim_chain_t *>(chains), n_chains, spin_pool,
                                                          coupling_pool, acc_i, acc_f, rec, n_sweeps, queue,
                                                          status, ly);
    return cudaGetLastError();
}

// Size classes with a compile-time layout:
// 128 < L <= 256 (1024 threads), 96 < L <= 128 and 128 < L <= 176 (512), 64 <
// L <= 96 and 96 < L <= 128 (256).  Below L = 64 (CTAs of 64 and 128 threads) the
// run-time layout measured 5-7% faster than a compile-time one on B200.
template <int NT>
cudaError_t launch_sweeps_nt(const rbim_chain_t *chains, int n_chains, int l_max, uint32_t *spin_pool,
                             const uint32_t *coupling_pool, long long *acc_i, double *acc_f, int32_t *rec,
                             int n_sweeps, int grid, int *queue, int *status, cudaStream_t stream)
{
    if constexpr (NT == 1024) {
        if (l_max > 128 && l_max <= 256)
            return launch_sweeps_lc<NT, 256>(chains, n_chains, l_max, spin_pool, coupling_pool, acc_i, acc_f, rec,
                                             n_sweeps, grid, queue, status, stream);
    }
    if constexpr (NT == 512) {
        if (l_max > 96 && l_max <= 128)
            return launch_sweeps_lc<NT, 128>(chains, n_chains, l_max, spin_pool, coupling_pool, acc_i, acc_f, rec,
                                             n_sweeps, grid, queue, status, stream);
        if (l_max > 128 && l_max <= 176 && 2 * (resident_layout_c(176, 512).bytes + kStaticSmem) <= kSmemPerSm)
            return launch_sweeps_lc<NT, 176>(chains, n_chains, l_max, spin_pool, coupling_pool, acc_i, acc_f, rec,
                                             n_sweeps, grid, queue, status, stream);
    }
    if constexpr (NT == 256) {
        if (l_max > 64 && l_max <= 96)
            return launch_sweeps_lc<NT, 96>(chains, n_chains, l_max, spin_pool, coupling_pool, acc_i, acc_f, rec,
                                            n_sweeps, grid, queue, status, stream);
        if (l_max > 96 && l_max <= 128)
            return launch_sweeps_lc<NT, 128>(chains, n_chains, l_max, spin_pool, coupling_pool, acc_i, acc_f, rec,
                                             n_sweeps, grid, queue, status, stream);
    }
    return launch_sweeps_lc<NT, 0>(chains, n_chains, l_max, spin_pool, coupling_pool, acc_i, acc_f, rec, n_sweeps,
                                   grid, queue, status, stream);
}

template <int NT>
cudaError_t launch_label_nt(int L, int n_lattices, const uint8_t *occ, int32_t *labels, int32_t *ncl,
                            uint8_t *wraps, int *status, cudaStream_t stream)
{
    const ResidentLayout ly = resident_layout(L, NT);
    cudaError_t e = cudaFuncSetAttribute(k_resident_label<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)ly.bytes);
    if (e != cudaSuccess) return e;
    k_resident_label<NT><<<n_lattices, NT, ly.bytes, stream>>>(L, occ, labels, ncl, wraps, status, ly);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_resident_sweeps(const rbim_chain_t *chains, int n_chains, int l_max, uint32_t *spin_pool,
                                   const uint32_t *coupling_pool, long long *acc_i, double *acc_f, int32_t *rec,
                                   int n_sweeps, int threads, int grid, int *queue, int *status,
                                   cudaStream_t stream)
{
    if (threads <= 0) threads = resident_default_threads(l_max);
    switch (threads) {
    case 32:
        return launch_sweeps_nt<32>(chains, n_chains, l_max, spin_pool, coupling_pool, acc_i, acc_f, rec, n_sweeps,
                                    grid, queue, status, stream);
    case 64:
        return launch_sweeps_nt<64>(chains, n_chains, l_max, spin_pool, coupling_pool, acc_i, acc_f, rec, n_sweeps,
                                    grid, queue, status, stream);
    case 128:
        return launch_sweeps_nt<128>(chains, n_chains, l_max, spin_pool, coupling_pool, acc_i, acc_f, rec, n_sweeps,
                                     grid, queue, status, stream);
    case 256:
        return launch_sweeps_nt<256>(chains, n_chains, l_max, spin_pool, coupling_pool, acc_i, acc_f, rec, n_sweeps,
                                     grid, queue, status, stream);
    case 512:
        return launch_sweeps_nt<512>(chains, n_chains, l_max, spin_pool, coupling_pool, acc_i, acc_f, rec, n_sweeps,
                                     grid, queue, status, stream);
    case 1024:
        return launch_sweeps_nt<1024>(chains, n_chains, l_max, spin_pool, coupling_pool, acc_i, acc_f, rec,
                                      n_sweeps, grid, queue, status, stream);
    default:
        return cudaErrorInvalidValue;
    }
}

cudaError_t launch_resident_label(int L, int n_lattices, const uint8_t *occ, int32_t *labels, int32_t *n_clusters,
                                  uint8_t *wraps, int threads, int *status, cudaStream_t stream)
{
    // The labelling kernel keeps at least two warps per CTA.
    if (threads <= 0) threads = std::max(64, resident_default_threads(L));
    switch (threads) {
    case 64:
        return launch_label_nt<64>(L, n_lattices, occ, labels, n_clusters, wraps, status, stream);
    case 128:
        return launch_label_nt<128>(L, n_lattices, occ, labels, n_clusters, wraps, status, stream);
    case 256:
        return launch_label_nt<256>(L, n_lattices, occ, labels, n_clusters, wraps, status, stream);
    case 512:
        return launch_label_nt<512>(L, n_lattices, occ, labels, n_clusters, wraps, status, stream);
    case 1024:
        return launch_label_nt<1024>(L, n_lattices, occ, labels, n_clusters, wraps, status, stream);
    default:
        return cudaErrorInvalidValue;
    }
}

}  // namespace rbim

#ifdef RBIM_PROFILE_PHASES
// Profiling builds only: copy out (and optionally reset) the per-phase cycle
// counters of the resident engine.
extern "C" int rbim_profile_phase_cycles(unsigned long long *out, int reset)
{
    cudaError_t e = cudaMemcpyFromSymbol(out, rbim::g_phase_cycles, sizeof(unsigned long long) * 16);
    if (e == cudaSuccess && reset) {
        const unsigned long long z[16] = {};
        e = cudaMemcpyToSymbol(rbim::g_phase_cycles, z, sizeof(z));
    }
    return e == cudaSuccess ? 0 : -2;
}

// Profiling builds only: event counters (0 unions, 1 find steps, 2 failed CAS).
extern "C" int rbim_profile_event_counts(unsigned long long *out, int reset)
{
    cudaError_t e = cudaMemcpyFromSymbol(out, rbim::g_event_counts, sizeof(unsigned long long) * 8);
    if (e == cudaSuccess && reset) {
        const unsigned long long z[8] = {};
        e = cudaMemcpyToSymbol(rbim::g_event_counts, z, sizeof(z));
    }
    return e == cudaSuccess ? 0 : -2;
}
#endif
