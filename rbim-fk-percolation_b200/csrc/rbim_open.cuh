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

// Parent of one site of a word: the last run head up to it (`le`: the bits up
// to the site's), or for a head whose run has a link the head above the link,
// or that head's own parent when it was written before (`done` sites from
// band0 on).  h, link, above: the word's UpBonds; before: 1 + the last head
// before the word; n0: the word's first site.
__device__ __forceinline__ uint32_t open_parent(const UF<Word16> &uf, uint32_t h, uint32_t before, uint32_t link,
                                                uint32_t above, uint32_t n0, uint32_t le, uint32_t L, uint32_t band0,
                                                uint32_t done)
{
    const uint32_t f = link & ~(le >> 1);  // the lowest of f is the link of a run headed here ...
    const uint32_t upto = f ^ (f - 1u);
    const bool linked = f && (h & (le ^ (le >> 1))) && !(h & upto & ~le);  // ... if no other head comes before
    const uint32_t m = linked ? above & upto : h & le;
    uint32_t p = (linked ? n0 - L : n0) + 31u - __clz(m);
    if (!m) p = before - 1u;
    if (linked && p - band0 < done) p = uf.ld(p);
    return p;
}

// 1 + the last run head before word w (0: there is none).
__device__ __forceinline__ uint32_t last_head_before(const Lat<Word16> &t, uint32_t w)
{
    // Site 0 always heads a run, so this walk back ends.
    while (w-- > 0) {
        const uint32_t h = head_mask(t.OV, w, 0xFFFFFFFFu);
        if (h) return (w << 5) + 32u - __clz(h);
    }
    return 0u;
}

// (b) Union-find initialisation: every site points at the head of its run of
// occupied y-bonds, and a run head with an occupied x-bond to the row above at
// the run above, with plain stores (a head takes one such link, to a smaller
// site, so nothing can race).  A warp writes its band of consecutive words two
// by two (lanes 0-15 one word, 16-31 the next, two sites a lane, one 32-bit
// store; sites past N are not written); a link whose upper head was written in
// an earlier step takes that head's own parent, so inside a band the link
// trees stay one level deep, and a link into the band above (written by
// another warp meanwhile) takes the upper head itself.  The bonds that are
// left go to NEED for the unions: at L = 256 about 9 k of 28 k bonds.
//
// Per group of 32 words, lane j finds the heads and up-bonds of word j, and a
// max-scan over the lanes gives every word the last head before it.  kFew: for
// launches whose warps may have a single word, which all lanes then look at.
template <bool kFew>
__device__ __forceinline__ void phase_heads_open(const Lat<Word16> &t, uint32_t warp, uint32_t nwarps)
{
    const uint32_t lane = threadIdx.x & 31u;
    const Geom &g = t.g;
    const Band band = warp_band(g.NW, warp, nwarps);
    if (kFew && band.end - band.first == 1u) {
        const uint32_t w = band.first, n0 = w << 5;
        const UpBonds ub = up_bonds(t, w);
        if (lane == 0) t.NEED[w] = ub.need;
        const uint32_t before = (ub.heads & 1u) ? 0u : last_head_before(t, w);
        const uint32_t p = open_parent(t.uf, ub.heads, before, ub.link, ub.above, n0, mask_le(lane), g.L, 0u, 0u);
        if (n0 + lane < g.N) t.uf.st(n0 + lane, (unsigned short)p);
        return;
    }
    const uint32_t band0 = band.first << 5, b0 = 2u * (lane & 15u), le0 = mask_le(b0);
    for (uint32_t base = band.first; base < band.end; base += 32u) {
        const uint32_t wj = base + lane;
        UpBonds ub{};
        if (wj < band.end) {
            ub = up_bonds(t, wj);
            t.NEED[wj] = ub.need;
        }
        const uint32_t h = ub.heads;
        const uint32_t pre = lane == 0 && !(h & 1u) ? last_head_before(t, base) : 0u;
        const uint32_t count = min(32u, band.end - base);
        uint32_t incl = max(h ? (wj << 5) + 32u - __clz(h) : 0u, pre);
        for (uint32_t o = 1; o < count; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl = max(incl, v);
        }
        // Last head before word j: the scan of lanes < j, or pre for j = 0.
        uint32_t before = __shfl_up_sync(0xFFFFFFFFu, incl, 1);
        if (lane == 0) before = pre;
        for (uint32_t j = 0; j < count; j += 2u) {
            const uint32_t jj = j + (lane >> 4);
            const uint32_t hj = __shfl_sync(0xFFFFFFFFu, h, jj);
            const uint32_t cj = __shfl_sync(0xFFFFFFFFu, before, jj);
            const uint32_t lj = __shfl_sync(0xFFFFFFFFu, ub.link, jj);
            const uint32_t aj = __shfl_sync(0xFFFFFFFFu, ub.above, jj);
            const uint32_t n0 = (base + jj) << 5, n = n0 + b0;
            const uint32_t done = ((base + j) << 5) - band0;  // sites of the band written in earlier steps
            const uint32_t p0 = open_parent(t.uf, hj, cj, lj, aj, n0, le0, g.L, band0, done);
            const uint32_t p1 = open_parent(t.uf, hj, cj, lj, aj, n0, 2u * le0 + 1u, g.L, band0, done);
            if (jj < count) {
                if (n + 1u < g.N)
                    t.uf.st2(n, p0 | (p1 << 16));
                else if (n < g.N)
                    t.uf.st(n, (unsigned short)p0);
            }
            __syncwarp();  // later rows read these words
        }
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

// (c) Roots of the run heads (see phase_roots), as a flat per-thread loop
// over the heads of the thread's slices: read-only walks, each head's final
// root written by the head's own thread.  ROOT must be zero on entry.
// Returns the number of roots this thread found.
// Next head of the thread's slices into (h, x), or false when there is none.
__device__ __forceinline__ bool next_head(const Lat<Word16> &t, const Slices &sl, uint32_t nthreads, uint32_t &item,
                                          uint32_t &pending, uint32_t &base, uint32_t &h)
{
    while (!pending && item < sl.items) {
        const uint32_t w = sl.word(item);
        pending = head_mask(t.OV, w, t.g.valid(w)) & sl.mask(item);
        base = w << 5;
        item += nthreads;
    }
    if (!pending) return false;
    h = base + (uint32_t)(__ffs(pending) - 1);
    pending &= pending - 1u;
    return true;
}

__device__ __forceinline__ uint32_t phase_roots_flat(const Lat<Word16> &t, uint32_t tid, uint32_t nthreads)
{
    const Geom &g = t.g;
    const Slices sl = make_slices(g.NW, nthreads);
    uint32_t item = tid, pending = 0, base = 0, nroots = 0;
    // Two walks in flight per thread: heads h0, h1 at positions x0, x1.
    uint32_t h0 = 0, h1 = 0, x0 = 0, x1 = 0;
    bool a0 = next_head(t, sl, nthreads, item, pending, base, h0);
    bool a1 = a0 && next_head(t, sl, nthreads, item, pending, base, h1);
    x0 = h0;
    x1 = h1;
    const uint32_t cap = 64u * t.cap;  // 64 walks of t.cap steps (64 N + 4096 by default)
    for (uint32_t it = 0; a0 || a1; ++it) {
        if (it >= cap) {
            atomicOr(t.err, kErrFindCap);
            break;
        }
        const uint32_t p0 = t.uf.ld(x0), p1 = t.uf.ld(x1);
        const bool r0 = a0 && p0 == x0, r1 = a1 && p1 == x1;
        x0 = p0;
        x1 = p1;
        if (r0) {
            if (x0 != h0) {
                t.uf.st(h0, (unsigned short)x0);
            } else {
                atomicOr(t.ROOT + (h0 >> 5), 1u << (h0 & 31u));
                ++nroots;
            }
            a0 = next_head(t, sl, nthreads, item, pending, base, h0);
            x0 = h0;
        }
        if (r1) {
            if (x1 != h1) {
                t.uf.st(h1, (unsigned short)x1);
            } else {
                atomicOr(t.ROOT + (h1 >> 5), 1u << (h1 & 31u));
                ++nroots;
            }
            a1 = next_head(t, sl, nthreads, item, pending, base, h1);
            x1 = h1;
        }
    }
    return nroots;
}

__device__ __forceinline__ uint32_t warp_sum(uint32_t v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

// Run pieces: the sites of a word split into maximal runs of occupied
// y-bonds; every piece starts at a run head or at bit 0 of the word and all
// its sites share one root.  Bits of the pieces' first sites.
__device__ __forceinline__ uint32_t piece_leaders(const Lat<Word16> &t, uint32_t w, uint32_t valid)
{
    return (head_mask(t.OV, w, valid) | 1u) & valid;
}

// Add v to the 16-bit word i through its 32-bit container (no carry can
// leave the half: cluster sizes stay below 65536 whenever counts are taken).
__device__ __forceinline__ void add16(unsigned short *base, uint32_t i, uint32_t v)
{
    atomicAdd((unsigned int *)(base + (i & ~1u)), v << (16u * (i & 1u)));
}

// Cluster sizes into the root words (after the sites pass, every non-root
// site's word holds its root): one add per run piece, the sites of a word
// split into maximal runs sharing a root.  With at least 32 words per warp,
// each lane takes a word of its warp's block of 32 and walks the word's
// pieces, summing consecutive pieces of one root in a register; at the end
// of the block the lanes holding the same root add their sums in one atomic,
// so a giant cluster sees one add per block instead of one per piece.
// kMinusOne: the piece that starts at the root adds one less, so that a root
// word holds size - 1 (a tile of 65536 sites then still fits 16 bits).
// Each root word must hold zero or the root's own index on entry (a root
// points at itself, so counting onto it needs no zeroing pass; the caller
// then subtracts the index).
template <bool kMinusOne>
__device__ __forceinline__ void count_pieces(const Lat<Word16> &t, unsigned short *u16, uint32_t warp,
                                             uint32_t nwarps)
{
    const Geom &g = t.g;
    const uint32_t lane = threadIdx.x & 31u;
    if (g.NW >= 32u * nwarps) {
        for (uint32_t w0 = warp << 5; w0 < g.NW; w0 += nwarps << 5) {
            const uint32_t w = w0 + lane;
            uint32_t acc_r = 0xFFFFFFFFu, acc = 0;
            if (w < g.NW) {
                const uint32_t valid = g.valid(w);
                uint32_t lead = piece_leaders(t, w, valid);
                const uint32_t roots = t.ROOT[w];
                const uint32_t nv = (uint32_t)__popc(valid);
                while (lead) {
                    const uint32_t b = __ffs(lead) - 1u;
                    lead &= lead - 1u;
                    const uint32_t end = lead ? (uint32_t)(__ffs(lead) - 1) : nv;
                    const uint32_t n = (w << 5) + b;
                    const bool is_root = (roots >> b) & 1u;
                    const uint32_t r = is_root ? n : (uint32_t)u16[n];
                    if (r != acc_r) {
                        if (acc) add16(u16, acc_r, acc);
                        acc_r = r;
                        acc = 0;
                    }
                    acc += end - b - ((kMinusOne && is_root) ? 1u : 0u);
                }
            }
            const uint32_t grp = __match_any_sync(0xFFFFFFFFu, acc_r);
            const uint32_t sum = __reduce_add_sync(grp, acc);
            if (acc_r != 0xFFFFFFFFu && lane == (uint32_t)(__ffs(grp) - 1) && sum) add16(u16, acc_r, sum);
        }
    } else {
        for (uint32_t w = warp; w < g.NW; w += nwarps) {
            const uint32_t valid = g.valid(w);
            const uint32_t lead = piece_leaders(t, w, valid);
            if ((lead >> lane) & 1u) {
                const uint32_t n = (w << 5) + lane;
                const uint32_t next = lead & ~mask_le(lane);
                const uint32_t end = next ? (uint32_t)(__ffs(next) - 1) : (uint32_t)__popc(valid);
                const bool is_root = (t.ROOT[w] >> lane) & 1u;
                const uint32_t r = is_root ? n : (uint32_t)u16[n];
                add16(u16, r, end - lane - ((kMinusOne && is_root) ? 1u : 0u));
            }
        }
    }
}

// Root of any site n once the roots pass is done: every parent is a run head
// (heads are the initial parents, roots are heads, and hooks, path halving
// and the seam merge only ever point at roots or grandparents) and every head
// then points at its root (a root at itself), so two loads reach it.
__device__ __forceinline__ uint32_t piece_root(const unsigned short *u16, uint32_t n) { return u16[u16[n]]; }

// The cluster flip of a sweep, one lane per word and one root lookup per run
// piece instead of per site: the sites of a word split into pieces (maximal
// runs of occupied y-bonds cut at the word boundary) that share a root, and a
// piece flips as a whole when its root's FLIP bit is set.  With
// `leader_roots` the leader of every piece that does not head its run (bit 0
// of a word inside a run) also gets its root written, so that afterwards the
// word of every piece leader holds its root, which the cluster-size count and
// the |M_C| pass read.  Non-head words are nobody's parent, so the writes do
// not disturb the lookups of other lanes.
__device__ __forceinline__ void flip_pieces(const Lat<Word16> &t, uint32_t tid, uint32_t nthreads,
                                                     bool leader_roots)
{
    const Geom &g = t.g;
    unsigned short *u16 = t.uf.w;
    for (uint32_t w = tid; w < g.NW; w += nthreads) {
        const uint32_t valid = g.valid(w);
        const uint32_t heads = head_mask(t.OV, w, valid);
        uint32_t lead = (heads | 1u) & valid;
        const uint32_t nv = (uint32_t)__popc(valid);
        uint32_t fl = 0;
        while (lead) {
            const uint32_t b = __ffs(lead) - 1u;
            lead &= lead - 1u;
            const uint32_t end = lead ? (uint32_t)(__ffs(lead) - 1) : nv;
            const uint32_t n = (w << 5) + b;
            const uint32_t r = piece_root(u16, n);
            if ((t.FLIP[r >> 5] >> (r & 31u)) & 1u) fl |= (end - b == 32u) ? 0xFFFFFFFFu : (((1u << (end - b)) - 1u) << b);
            if (leader_roots && !((heads >> b) & 1u)) u16[n] = (unsigned short)r;
        }
        if (fl) t.S[w] ^= fl;
    }
}

// Roots and cluster flip of a sweep in one pass, one lane per word and one
// walk per run piece (the sites of a word split into pieces -- maximal runs
// of occupied y-bonds cut at the word boundary -- that share a root).  A
// piece's leader walks read-only up to its root; the root is then written
// into the leader's word (for a run head this is the final compression the
// separate roots pass would make, and the count and |M_C| passes read it
// for every leader), the piece flips as a whole with its root's FLIP bit,
// and a leader that is its own root sets its ROOT bit.  Walks of other lanes
// running at the same time may read a head's old parent or its final root;
// both are ancestors, so every walk ends at the right root.  Roots' words are
// never written.  Returns the number of roots this thread found.
__device__ __forceinline__ uint32_t roots_flip_pieces(const Lat<Word16> &t, uint32_t tid, uint32_t nthreads)
{
    const Geom &g = t.g;
    const UF<Word16> &uf = t.uf;
    uint32_t nroots = 0;
    for (uint32_t w = tid; w < g.NW; w += nthreads) {
        const uint32_t valid = g.valid(w);
        uint32_t lead = (head_mask(t.OV, w, valid) | 1u) & valid;
        const uint32_t nv = (uint32_t)__popc(valid);
        uint32_t fl = 0, rootbits = 0;
        while (lead) {
            const uint32_t b = __ffs(lead) - 1u;
            lead &= lead - 1u;
            const uint32_t end = lead ? (uint32_t)(__ffs(lead) - 1) : nv;
            const uint32_t n = (w << 5) + b;
            uint32_t x = uf.ld(n);
            for (uint32_t it = 0;; ++it) {
                const uint32_t p = uf.ld(x);
                if (p == x) break;
                if (it >= t.cap) {
                    atomicOr(t.err, kErrFindCap);
                    break;
                }
                x = p;
            }
            if (x == n) {
                rootbits |= 1u << b;
                ++nroots;
            } else {
                uf.st(n, (unsigned short)x);
            }
            if ((t.FLIP[x >> 5] >> (x & 31u)) & 1u) fl |= (end - b == 32u) ? 0xFFFFFFFFu : (((1u << (end - b)) - 1u) << b);
        }
        t.ROOT[w] = rootbits;
        if (fl) t.S[w] ^= fl;
    }
    return nroots;
}

}  // namespace rbim
