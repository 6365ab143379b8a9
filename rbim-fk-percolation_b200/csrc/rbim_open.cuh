// Open-lattice labelling on a 16-bit shared-memory union-find, shared by the
// resident engine (one lattice per CTA) and the cluster engine (one tile of a
// lattice per CTA).  Inside an open region of the lattice (no bond that
// crosses a periodic seam) every cycle is contractible, so the union-find
// words carry parents only and each open cluster's root is its smallest site.
//
// A lattice context here is a Lat<Word16> whose Geom covers the sites held by
// the CTA; sites whose x-bond leaves that range (the last L sites) are left to
// the caller's seam or boundary stage.
#pragma once

#include "rbim_phases.cuh"

#ifndef RBIM_COUNT
#ifdef RBIM_PROFILE_PHASES
#define RBIM_COUNT(k, v) ((void)(v))
#define RBIM_PROF_ONLY(...) __VA_ARGS__
#else
#define RBIM_COUNT(k, v) ((void)0)
#define RBIM_PROF_ONLY(...)
#endif
#endif

namespace rbim {

// Open-lattice union-find word: the parent site only.
struct Word16 {
    using T = unsigned short;
    __device__ __forceinline__ static uint32_t parent(T w) { return w; }
    __device__ __forceinline__ static int ox(T) { return 0; }
    __device__ __forceinline__ static int oy(T) { return 0; }
    __device__ __forceinline__ static T make(uint32_t p, int, int) { return (T)p; }
    __device__ __forceinline__ static T count_inc(uint32_t c) { return (T)c; }
};

// The open union-find lives in shared memory: access it through 32-bit
// shared-window addresses with explicit ld/st/atom.shared instructions.
template <>
struct UF<Word16> {
    using T = unsigned short;
    T *w;          // generic pointer (for code that indexes the array directly)
    uint32_t sa;   // shared-window address of w
    __device__ __forceinline__ T ld(uint32_t i) const
    {
        T v;
        asm volatile("ld.volatile.shared.u16 %0, [%1];" : "=h"(v) : "r"(sa + 2u * i) : "memory");
        return v;
    }
    // Shared memory is coherent within the CTA: the same load as ld.
    __device__ __forceinline__ T ldc(uint32_t i) const { return ld(i); }
    __device__ __forceinline__ void st(uint32_t i, T v) const
    {
        asm volatile("st.volatile.shared.u16 [%0], %1;" ::"r"(sa + 2u * i), "h"(v) : "memory");
    }
    // The parents of sites i and i + 1 (i even) in one 32-bit store: v holds
    // site i's in its low half.
    __device__ __forceinline__ void st2(uint32_t i, uint32_t v) const
    {
        asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(sa + 2u * i), "r"(v) : "memory");
    }
    // Hooks root hi under lo; false when hi is no longer a root, or when the
    // other parent in its 32-bit word changed meanwhile.
    __device__ __forceinline__ bool hook(uint32_t hi, uint32_t lo) const
    {
        const uint32_t at = (sa + 2u * hi) & ~3u, sh = 16u * (hi & 1u);
        uint32_t cur, old;
        asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(cur) : "r"(at) : "memory");
        if (((cur >> sh) & 0xFFFFu) != hi) return false;
        asm volatile("atom.shared.cas.b32 %0, [%1], %2, %3;"
                     : "=r"(old)
                     : "r"(at), "r"(cur), "r"(cur ^ ((hi ^ lo) << sh))
                     : "memory");
        return old == cur;
    }
    __device__ __forceinline__ void add(uint32_t i, T v) const { uf_atomic_add(w + i, v); }
};

// Bits reached by filling upwards from the seeds s (a subset of p) through
// consecutive bits of p: adding a seed to its run of ones carries through the
// run's end, and the carry clears the bits it passes.
__device__ __forceinline__ uint32_t fill_up(uint32_t s, uint32_t p) { return p & (~(p + s) | s); }

// The up-bonds of word w (bit b: the x-bond from site n - L to n = 32w + b)
// that the labelling needs, split in links and unions.
struct UpBonds {
    uint32_t heads;   // run heads of the word
    uint32_t above;   // run heads of the sites n - L
    uint32_t link;    // bonds that link their run's head to the run above
    uint32_t linked;  // those heads
    uint32_t need;    // bonds left to the unions
};

__device__ __forceinline__ UpBonds up_bonds(const Lat<Word16> &t, uint32_t w)
{
    const Geom &g = t.g;
    UpBonds r;
    const uint32_t valid = g.valid(w);
    r.heads = head_mask(t.OV, w, valid);
    r.above = 0u;
    r.link = 0u;
    r.linked = 0u;
    r.need = 0u;
    if ((w << 5) + 31u < g.L) return r;  // the first row has no up-bonds
    // Bits u - 1 .. u + 31 of OH and u - 1 .. u + 30 of OV (words before the
    // planes read as zero), u = 32w - L the site above bit 0.
    const int u = (int)(w << 5) - (int)g.L, q = u - 1;
    const int qw = q >> 5;
    const uint32_t sh = (uint32_t)q & 31u;
    const uint32_t h0 = qw >= 0 ? t.OH[qw] : 0u, h1 = t.OH[qw + 1];
    const uint32_t v0 = qw >= 0 ? t.OV[qw] : 0u, v1 = t.OV[qw + 1];
    const uint32_t up1 = __funnelshift_r(h0, h1, sh);  // bit 0: the up-bond of the site before the word
    const uint32_t up = ((up1 >> 1) | ((h1 >> sh) << 31)) & valid;
    r.above = ~__funnelshift_r(v0, v1, sh);
    // One bond per pair of runs: a bond is redundant after another one between
    // the same two runs (no head of either row between them).
    const uint32_t p = ~(r.heads | r.above);
    const uint32_t c = up & ~fill_up(((up << 1) | (up1 & 1u)) & p, p);
    // The first bond of each run headed in this word whose upper run's head is
    // also in view links the two heads.
    const uint32_t k = c & (r.heads | (0u - r.heads)) & (r.above | (0u - r.above));
    const uint32_t in_run = ~r.heads;
    r.link = k & ~fill_up((k << 1) & in_run, in_run);
    r.need = c & ~r.link;
    // From each link down its run to the head, with the bits reversed.
    const uint32_t back = __brev(r.link), run = __brev(in_run);
    r.linked = r.heads & __brev(back | (fill_up(back & run, run) << 1));
    return r;
}

// Words of the band of a warp: the words are split in equal contiguous bands,
// one per warp.
struct Band {
    uint32_t first, end;
};

__device__ __forceinline__ Band warp_band(uint32_t NW, uint32_t warp, uint32_t nwarps)
{
    const uint32_t per = (NW + nwarps - 1u) / nwarps;
    const uint32_t first = min(NW, warp * per);
    return {first, min(NW, first + per)};
}

// Parent of one site of a word (`le`: the bits up to the site's): the last run
// head of the word up to it, or for a head with a link the head above the
// link, or that head's own parent when it was written before (`done` sites
// from band0 on).  A site whose run began in an earlier word points at the
// word's predecessor n0 - 1, which is in its run.  n0: the word's first site.
__device__ __forceinline__ uint32_t open_parent(const UF<Word16> &uf, const UpBonds &ub, uint32_t n0, uint32_t le,
                                                uint32_t L, uint32_t band0, uint32_t done)
{
    const uint32_t f = ub.link & ~(le >> 1);  // a linked head's link is the lowest of f
    const bool linked = ub.linked & (le ^ (le >> 1));
    const uint32_t m = linked ? ub.above & (f ^ (f - 1u)) : ub.heads & le;
    uint32_t p = (linked ? n0 - L : n0) + 31u - __clz(m);
    if (linked && p - band0 < done) p = uf.ld(p);
    return p;
}

// (b) Union-find initialisation: every site points at the head of its run of
// occupied y-bonds (through the last site of the word before, when the run
// began there), and a run head with an occupied x-bond to the row above at
// the run above, with plain stores (a head takes one such link, to a smaller
// site, so nothing can race).  A warp writes its band of consecutive words two
// by two (lanes 0-15 one word, 16-31 the next, two sites a lane, one 32-bit
// store; sites past N are not written); a link whose upper head was written in
// an earlier step takes that head's own parent, so inside a band the link
// trees stay one level deep, and a link into the band above (written by
// another warp meanwhile) takes the upper head itself.  The bonds that are
// left go to NEED for the unions: at L = 256 about 9 k of 28 k bonds.
//
// Per group of 32 words, lane j finds the heads and up-bonds of word j.  Bound
// by the integer pipe, so what can be done on whole words is done there.  kFew:
// for launches whose warps may have a single word, which all lanes then look
// at.  kCount: the number of heads is added to *total.
template <bool kFew, bool kCount = false>
__device__ __forceinline__ void phase_heads_open(const Lat<Word16> &t, uint32_t warp, uint32_t nwarps,
                                                 uint32_t *total = nullptr)
{
    const uint32_t lane = threadIdx.x & 31u;
    const Geom &g = t.g;
    const Band band = warp_band(g.NW, warp, nwarps);
    if (kFew && band.end - band.first == 1u) {
        const uint32_t w = band.first, n0 = w << 5;
        const UpBonds ub = up_bonds(t, w);
        if (lane == 0) t.NEED[w] = ub.need;
        const uint32_t p = open_parent(t.uf, ub, n0, mask_le(lane), g.L, 0u, 0u);
        if (n0 + lane < g.N) t.uf.st(n0 + lane, (unsigned short)p);
        return;
    }
    const uint32_t band0 = band.first << 5, b0 = 2u * (lane & 15u), le0 = mask_le(b0), le1 = 2u * le0 + 1u;
    uint32_t heads = 0;
    for (uint32_t base = band.first; base < band.end; base += 32u) {
        const uint32_t wj = base + lane;
        UpBonds ub{};
        if (wj < band.end) {
            ub = up_bonds(t, wj);
            t.NEED[wj] = ub.need;
        }
        if (kCount) heads += __popc(ub.heads);
        const uint32_t count = min(32u, band.end - base);
        for (uint32_t j = 0; j < count; j += 2u) {
            const uint32_t jj = j + (lane >> 4);
            UpBonds w;
            w.heads = __shfl_sync(0xFFFFFFFFu, ub.heads, jj);
            w.above = __shfl_sync(0xFFFFFFFFu, ub.above, jj);
            w.link = __shfl_sync(0xFFFFFFFFu, ub.link, jj);
            w.linked = __shfl_sync(0xFFFFFFFFu, ub.linked, jj);
            const uint32_t n0 = (base + jj) << 5, n = n0 + b0;
            const uint32_t done = ((base + j) << 5) - band0;  // sites of the band written in earlier steps
            const uint32_t p0 = open_parent(t.uf, w, n0, le0, g.L, band0, done);
            const uint32_t p1 = open_parent(t.uf, w, n0, le1, g.L, band0, done);
            if (jj < count) {
                if (n + 1u < g.N)
                    t.uf.st2(n, p0 | (p1 << 16));
                else if (n < g.N)
                    t.uf.st(n, (unsigned short)p0);
            }
            __syncwarp();  // later rows read these words
        }
    }
    if (kCount) {
        heads = __reduce_add_sync(0xFFFFFFFFu, heads);
        if (lane == 0) atomicAdd(total, heads);
    }
}

// One path-halving step of a walk at x, without branches: returns the next
// position and sets `done` when x's parent or grandparent is the root (the
// returned position is then the root).
__device__ __forceinline__ uint32_t halving_step(const UF<Word16> &uf, uint32_t x, bool &done)
{
    const uint32_t p = uf.ld(x);
    const uint32_t gp = uf.ld(p);
    const bool x_root = p == x, p_root = gp == p;
    if (!x_root && !p_root) uf.st(x, (unsigned short)gp);
    done = x_root || p_root;
    return x_root ? x : (p_root ? p : gp);
}

// Lists the set bits of a group of `count` words (lane j holds what is left of
// word j in `bits`) in the warp's `list` of `seg` entries, in order, an entry
// being 32 j + bit; the bits listed are cleared.  Returns the number of
// entries.  kFew: up to eight words are listed bit by lane.
template <bool kFew>
__device__ __forceinline__ uint32_t list_bits(uint32_t &bits, uint32_t count, unsigned short *list, uint32_t seg,
                                              uint32_t lane)
{
    uint32_t total = 0;
    if (kFew && count <= 8u) {
        for (uint32_t j = 0; j < count; ++j) {
            const uint32_t b = __shfl_sync(0xFFFFFFFFu, bits, j);
            const uint32_t k = total + __popc(b & (mask_le(lane) >> 1));
            const bool put = ((b >> lane) & 1u) && k < seg;
            if (put) list[k] = (unsigned short)((j << 5) + lane);
            const uint32_t left = b & ~__ballot_sync(0xFFFFFFFFu, put);
            if (lane == j) bits = left;
            total += __popc(b);
        }
        total = min(total, seg);
    } else {
        const uint32_t mine = __popc(bits);
        uint32_t sum = mine;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, sum, o);
            if (lane >= o) sum += v;
        }
        for (uint32_t k = sum - mine; bits && k < seg; ++k) {
            list[k] = (unsigned short)((lane << 5) + __ffs(bits) - 1u);
            bits &= bits - 1u;
        }
        total = min(__shfl_sync(0xFFFFFFFFu, sum, 31), seg);
    }
    __syncwarp();
    return total;
}

// (b) Open-lattice unions across the x-bonds that phase_heads_open left in
// NEED: the larger root is hooked under the smaller with a CAS, finds use path
// halving, and a union whose CAS loses a race goes on from the two roots it
// found.  Bonds per word vary, so each warp lists the bonds of 32 words at a
// time and its lanes then take every 32nd of them, in one flat loop: both walks of a bond advance in the same iteration and a lane takes its next bond
// as soon as its union is done.  The CAS works on the 32-bit word that holds
// the root's parent; losing it to a change of the other half only repeats it.
//
// kFew: for launches whose warps may have few words (one lattice or tile on
// many threads), which are listed at once; the code for it costs 4 % at
// L = 64 where it is never taken.
template <bool kFew>
__device__ __forceinline__ void phase_union_open(const Lat<Word16> &t, unsigned short *list, uint32_t seg,
                                                 uint32_t warp, uint32_t nwarps)
{
    const Geom &g = t.g;
    const UF<Word16> &uf = t.uf;
    const uint32_t lane = threadIdx.x & 31u;
    const Band band = warp_band(g.NW, warp, nwarps);
    const uint32_t cap = 64u * t.cap;  // 64 walks of t.cap steps (64 N + 4096 by default)
    uint32_t it = 0;
    RBIM_PROF_ONLY(uint32_t n_bonds = 0; uint32_t n_fails = 0);
    for (uint32_t base = band.first; base < band.end; base += 32u) {
        const uint32_t count = min(32u, band.end - base);
        uint32_t pend = lane < count ? t.NEED[base + lane] : 0u;
        while (__any_sync(0xFFFFFFFFu, pend != 0u)) {
            // The bonds of a single word need no list: lane b takes bit b.
            const bool one = kFew && count == 1u;
            uint32_t total;
            if (one) {
                total = (__shfl_sync(0xFFFFFFFFu, pend, 0) >> lane) & 1u ? lane + 1u : 0u;
                pend = 0u;
            } else {
                total = list_bits<kFew>(pend, count, list, seg, lane);
            }
            uint32_t xa = 0, xb = 0;
            bool fetch = true;
            for (uint32_t i = lane;; ++it) {
                if (fetch) {
                    if (i >= total) break;
                    xb = (base << 5) + (one ? lane : (uint32_t)list[i]);
                    xa = xb - g.L;
                    i += 32u;
                    fetch = false;
                    RBIM_PROF_ONLY(++n_bonds);
                }
                if (it >= cap) {
                    atomicOr(t.err, kErrUnionCap);
                    break;
                }
                bool da, db;
                xa = halving_step(uf, xa, da);
                xb = halving_step(uf, xb, db);
                if (da && db) {
                    // Both walks are at roots.
                    fetch = xa == xb || uf.hook(max(xa, xb), min(xa, xb));
                    RBIM_PROF_ONLY(n_fails += fetch ? 0u : 1u);
                }
            }
            __syncwarp();
        }
    }
#ifdef RBIM_PROFILE_PHASES
    {
        uint32_t mx = it, sm = it;
        for (int o = 16; o > 0; o >>= 1) {
            mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
            sm += __shfl_xor_sync(0xFFFFFFFFu, sm, o);
        }
        uint32_t nb = n_bonds, nf = n_fails;
        for (int o = 16; o > 0; o >>= 1) {
            nb += __shfl_xor_sync(0xFFFFFFFFu, nb, o);
            nf += __shfl_xor_sync(0xFFFFFFFFu, nf, o);
        }
        if (lane == 0) {
            RBIM_COUNT(3, mx);
            RBIM_COUNT(4, sm);
            RBIM_COUNT(0, nb);
            RBIM_COUNT(2, nf);
        }
    }
#endif
}

// Run pieces: the sites of a word split into maximal runs of occupied
// y-bonds; every piece starts at a run head or at bit 0 of the word and all
// its sites share one root.  Bits of the pieces' first sites.
__device__ __forceinline__ uint32_t piece_leaders(const Lat<Word16> &t, uint32_t w, uint32_t valid)
{
    return (head_mask(t.OV, w, valid) | 1u) & valid;
}

// Add v to the 16-bit word i through its 32-bit container.  The sum must stay
// below 65536: a carry out of the low half would change the next site's word.
__device__ __forceinline__ void add16(unsigned short *base, uint32_t i, uint32_t v)
{
    atomicAdd((unsigned int *)(base + (i & ~1u)), v << (16u * (i & 1u)));
}

// Cluster sizes into the root words (every piece leader's word holds its
// root): one add per run piece, the sites of a word split into maximal runs
// sharing a root.  With at least 32 words per warp each lane takes a word and
// walks its pieces from the top, so that a piece ends where the last one
// began; with fewer the lanes are the sites of a word.
// skip (or null): plane of the sites of one cluster, counted by popcounts
// elsewhere; without it the largest cluster's root would take most of the
// adds, one after the other.
// Each root m's word holds its own index on entry (a root points at itself, so
// counting onto it needs no zeroing pass), and the piece that starts at the
// root adds one less: the word ends as m + size - 1 (counted_size decodes it),
// below 65536 since m is the smallest of its cluster's at most 65536 sites.
__device__ __forceinline__ void count_pieces(const Lat<Word16> &t, unsigned short *u16, const uint32_t *skip,
                                             uint32_t warp, uint32_t nwarps)
{
    const Geom &g = t.g;
    const uint32_t lane = threadIdx.x & 31u;
    if (g.NW >= 32u * nwarps) {
        for (uint32_t w = (warp << 5) + lane; w < g.NW; w += nwarps << 5) {
            const uint32_t valid = g.valid(w), roots = t.ROOT[w], sk = skip ? skip[w] : 0u;
            // Where counted pieces begin or end: not between two skipped ones.
            uint32_t cut = piece_leaders(t, w, valid) & ~(sk & ((sk << 1) | 1u));
            uint32_t end = 32u - __clz(valid);
            while (cut) {
                const uint32_t b = 31u - __clz(cut), bit = 1u << b;
                cut ^= bit;
                if (!(sk & bit)) {
                    const uint32_t n = (w << 5) + b;
                    const bool is_root = roots & bit;
                    const uint32_t r = is_root ? n : (uint32_t)u16[n];
                    add16(u16, r, end - b - (is_root ? 1u : 0u));
                }
                end = b;
            }
        }
    } else {
        for (uint32_t w = warp; w < g.NW; w += nwarps) {
            const uint32_t valid = g.valid(w);
            const uint32_t lead = piece_leaders(t, w, valid);
            const uint32_t todo = skip ? lead & ~skip[w] : lead;
            if ((todo >> lane) & 1u) {
                const uint32_t n = (w << 5) + lane;
                const uint32_t next = lead & ~mask_le(lane);
                const uint32_t end = next ? (uint32_t)(__ffs(next) - 1) : (uint32_t)__popc(valid);
                const bool is_root = (t.ROOT[w] >> lane) & 1u;
                const uint32_t r = is_root ? n : (uint32_t)u16[n];
                add16(u16, r, end - lane - (is_root ? 1u : 0u));
            }
        }
    }
}

// Size of the cluster of root m after count_pieces.
__device__ __forceinline__ uint32_t counted_size(const unsigned short *u16, uint32_t m)
{
    return (((uint32_t)u16[m] - m) & 0xFFFFu) + 1u;
}

// The root most likely to have the largest cluster: of 32 sites spread over
// the lattice, the root that most of them share (the smallest such root).
// Every warp finds the same one, by read-only walks.
__device__ __forceinline__ uint32_t likely_largest(const Lat<Word16> &t)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t r = uf_root_ro<Word16>(t.uf, (uint32_t)(((2u * lane + 1u) * t.g.N) >> 6), t.cap, t.err);
    const uint32_t same = __popc(__match_any_sync(0xFFFFFFFFu, r));
    return 0xFFFFu - (__reduce_max_sync(0xFFFFFFFFu, (same << 16) | (0xFFFFu - r)) & 0xFFFFu);
}

// Roots and cluster flip in one pass, one lane per site and K consecutive
// words at a time (K independent chains of loads): all lanes walk up to their
// roots together (a word's walks end within a step or two of each other, and
// the sites of a run or of one cluster load the same words), the site's word
// gets its root, and ballots give the word's ROOT bits, its flips (kFlip) and,
// with `in`, its sites in the cluster rooted at `root`.  Walks of other warps
// running at the same time may read a site's old parent or its root; both are
// ancestors, and roots' words never change.
//
// Bound by the latency and bank conflicts of the gathers.  Every lane works
// (one lane per word with a walk per run piece left half of them idle: 64 k
// cycles per L = 256 sweep on one SM, 39 k this way), and leaving out the loads
// of lanes that have arrived costs more in branches than it saves (71 k).
template <bool kFlip, int K>
__device__ __forceinline__ void roots_flip_sites(const Lat<Word16> &t, uint32_t *in, uint32_t root, uint32_t warp,
                                                 uint32_t nwarps)
{
    const uint32_t lane = threadIdx.x & 31u;
    const Geom &g = t.g;
    const UF<Word16> &uf = t.uf;
    for (uint32_t w0 = K * warp; w0 < g.NW; w0 += K * nwarps) {
        const uint32_t n0 = (w0 << 5) + lane;
        // Lanes past the lattice walk from site 0, which is a root.  Two steps
        // a vote, the first two without one (hardly any group ends there).
        uint32_t p[K], r[K];
#pragma unroll
        for (int k = 0; k < K; ++k) r[k] = uf.ld(n0 + 32u * k < g.N ? n0 + 32u * k : 0u);
        for (uint32_t it = 0;; ++it) {
#pragma unroll
            for (int k = 0; k < K; ++k) p[k] = uf.ld(r[k]);
#pragma unroll
            for (int k = 0; k < K; ++k) r[k] = uf.ld(p[k]);
            if (it == 0) continue;
            bool moved = false;
#pragma unroll
            for (int k = 0; k < K; ++k) moved |= p[k] != r[k];
            if (!__any_sync(0xFFFFFFFFu, moved)) break;
            if (it > t.cap) {
                if (moved) atomicOr(t.err, kErrFindCap);
                break;
            }
        }
        uint32_t roots = 0, flips = 0, members = 0;  // lane k: of word w0 + k
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const uint32_t n = n0 + 32u * k;
            const bool ok = n < g.N;
            if (ok) uf.st(n, (unsigned short)r[k]);
            const uint32_t b = __ballot_sync(0xFFFFFFFFu, ok && r[k] == n);
            const uint32_t f = kFlip ? __ballot_sync(0xFFFFFFFFu, ok && ((t.FLIP[r[k] >> 5] >> (r[k] & 31u)) & 1u)) : 0u;
            const uint32_t c = __ballot_sync(0xFFFFFFFFu, ok && r[k] == root);
            if (lane == k) {
                roots = b;
                flips = f;
                members = c;
            }
        }
        if (lane < K && w0 + lane < g.NW) {
            t.ROOT[w0 + lane] = roots;
            if (kFlip) t.S[w0 + lane] ^= flips;
            if (in) in[w0 + lane] = members;
        }
    }
}

}  // namespace rbim
