// bsgs.cu -- baby-step giant-step search, a group of 32 to 1024 threads per prime.
//
// Replaces the reference's giantfull/giantparity kernels (kernels/giant.cl:77-323).
// For one prime p with per-prime record (see setup.cu), searched by a group of
// GS = 32 << c threads (class c, chosen per prime by the set-up):
//   baby phase   y_j = s^j for j in [0,Q'), Q' = 16*GS: thread t forms
//                y_{16t..16t+15} from its start A[t%32]*B[t/32] as two chains
//                (doublings when b^e is 2 or 4, else one modular product per
//                step) and enters each into the group's filter.  y_j = 1 for
//                some 0 < j <= Q' detects ord(s) <= Q' (giant.cl:123-134).
//   giant phase  gamma = T_i * S^q for q in [0,Mg): item (i,g) walks q in
//                [g*Lc, (g+1)*Lc) from T_i * S^(g*Lc); a thread runs two items
//                at a time, one modular product and one filter probe per step
//                (giant.cl:170-192).  s^j == gamma gives n = nmin + off_i +
//                e*((q+1)*Q' - 1 - j), where s = b^e and off_i is target i's
//                class of n mod e (setup.cu; e = 2 is the reference's parity
//                split).
//   small order  ord(s) <= Q': each target is looked up once and every n in
//                range with the same residue mod e*ord is claimed (giant.cl:146-168).
//   claims       atomicAnd on the term's bitmap bit; the first claimer appends
//                {p, n, seq} to the factor buffer (giant.cl:21-39,158-162).
//
// The filter holds the baby values as a blocked Bloom filter in shared memory:
// 48 words per thread, i.e. three words per baby value; a value sets three bits
// of one word (one atomicOr without a result) and a probe tests them (one
// 4-byte load).  It never misses a value; about one probe in 2000 passes for a
// value that is not there.  Passing probes go on a queue and are checked exactly
// once the giant steps are done, 16 lanes each: with anchors x_t = s^(16t), t =
// 0..GS, in an index that then takes the filter's place, gamma = s^j for some j =
// 16t - l, 0 <= l < 16, exactly when gamma * s^l is an anchor, so lane l forms gamma
// * s^l and looks it up.  The search is exact for every 64-bit value (the reference's
// split lo32/hi32 table cannot find values whose low 32 bits are zero,
// giant.cl:46,63).
//
// What bounds it: issue.  A random 4-byte shared-memory access of a warp, load or
// atomic, takes 3.55 cycles of the SM's shared-memory pipe, a 16-byte one 10.2,
// and the ALU and FP64 pipes take two cycles per warp instruction (measured).
// A step is about 8 FP64, 8 ALU and 3 IMAD instructions and one such access,
// 14 to 16 cycles of an SM quarter on each of these resources, and its 22 issue
// slots come first: mixed streams of instructions that each hold their pipe for
// two cycles issue one in 1.5 cycles at best (measured), and the kernel issues in
// 65% of all cycles.  100 sequences, n-range 6*10^6, p near 2^50: 13.7 ns per
// prime for 9200 steps (28.1 for 12100 with an exact table of 16-byte buckets of
// fingerprints, whose probes and three-store inserts took 5600 shared-memory
// cycles per prime against 2200 now, and with one group size for all primes of a
// job); p near 2^58, 61 sequences: 15.8 (26.8); 68 sequences over an n-range of
// 10^5: 2.1 (4.0).  One test for two steps of both chains (the least of the four
// probes' missing bits) instead of one each took 14.1 to 13.9 and 17.0 to 16.1 (then) of
// these.  Three bits per value and three words per value: with two bits a pass
// comes four times as often and costs more than the third bit's two
// instructions; the filter fills what two CTAs of 512 threads have of shared
// memory.  A group of Q'/16 threads per prime instead of the whole CTA keeps 16
// baby and about as many giant steps per thread whatever the prime's work.
#include "mont.cuh"
#include "rs_internal.h"

#include <type_traits>

namespace rs {

constexpr u32 HMUL = 0x9E3779B1u;
constexpr u32 FILTER_WPT = 48;         // filter words per thread of the group

// Hash of a residue's 64 bits: word of an nw-word filter (top bits of h) and
// the three bits it sets there (from the low bits of h; they may coincide).
// Both halves are folded in because the baby chain for small bases is a run of
// doublings that repeat shifted patterns (as doubles: one mantissa).
__device__ __forceinline__ u32 val_hash(u64 v) { return ((u32)v ^ (u32)(v >> 32)) * HMUL; }
__device__ __forceinline__ u32 filter_mask(u32 h)
{
    return (1u << (h & 31)) | (1u << ((h >> 5) & 31)) | (1u << ((h >> 10) & 31));
}

// 2x mod p for p < 2^63 (2x cannot wrap): one compare, one predicated subtract
__device__ __forceinline__ u64 dbl63(u64 x, u64 p)
{
    x += x;
    return (x >= p) ? x - p : x;
}

// ---- arithmetic by step kind (MODE) ----
// V: a residue as the chains hold it; Fix: a fixed multiplier.  MODE 2 (p below
// FP_BOUND = 2^51): plain residues, exact in doubles.  MODE 1 (p < 2^63):
// Montgomery form, products by a fixed multiplier by Shoup's method.  MODE 0:
// Montgomery throughout.
template <int MODE>
struct Ring {
    typedef u64 V;
    u64 p, q;
    struct Fix { u64 w, wq; };
    __device__ __forceinline__ explicit Ring(const PrimeHdr &h) : p(h.p), q(h.q) {}
    static __device__ __forceinline__ V val(u64 b) { return b; }
    static __device__ __forceinline__ u64 bits(V v) { return v; }
    static __device__ __forceinline__ V one(const PrimeHdr &h) { return h.one; }
    static __device__ __forceinline__ Fix baby(const PrimeHdr &h) { return MODE == 1 ? Fix{h.sp, h.sw} : Fix{h.s, 0}; }
    static __device__ __forceinline__ Fix giant(const PrimeHdr &h) { return MODE == 1 ? Fix{h.Sp, h.Sw} : Fix{h.S, 0}; }
    __device__ __forceinline__ V mul(V a, V b) const { return mmul(a, b, p, q); }
    __device__ __forceinline__ V step(V x, const Fix &f) const
    {
        return MODE == 1 ? shoup_mul(x, f.w, f.wq, p) : mmul(x, f.w, p, q);
    }
    __device__ __forceinline__ V dbl(V x) const { return MODE == 1 ? dbl63(x, p) : madd(x, x, p); }
};
template <>
struct Ring<2> {
    typedef double V;
    double p, pinv;
    struct Fix { double w, wq; };
    __device__ __forceinline__ explicit Ring(const PrimeHdr &h)
        : p(fp_exact(h.p)), pinv(bits_double(h.q)) {}
    static __device__ __forceinline__ V val(u64 b) { return bits_double(b); }
    static __device__ __forceinline__ u64 bits(V v) { return double_bits(v); }
    static __device__ __forceinline__ V one(const PrimeHdr &) { return 1.0; }
    static __device__ __forceinline__ Fix baby(const PrimeHdr &h) { return Fix{val(h.s), val(h.sw)}; }
    static __device__ __forceinline__ Fix giant(const PrimeHdr &h) { return Fix{val(h.S), val(h.Sw)}; }
    __device__ __forceinline__ V mul(V a, V b) const { return fp_mul(a, b, p, pinv); }
    __device__ __forceinline__ V step(V x, const Fix &f) const { return fp_mulfix(x, f.w, f.wq, p); }
    __device__ __forceinline__ V dbl(V x) const { return fp_dbl(x, p); }
};

// ---- TMA 1D bulk copies and mbarriers (record header prefetch) ----
__device__ __forceinline__ u32 smem_u32(const void *p) { return (u32)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(u64 *bar, u32 count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(u64 *bar, u32 bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// global -> this CTA's shared memory, completion counted on bar (no multicast)
__device__ __forceinline__ void bulk_load(void *dst, const void *src, u32 bytes, u64 *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void l2_prefetch(const void *src, u32 bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(u64 *bar, u32 parity)
{
    u32 ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Barrier of group gid of the CTA: a warp by itself, else a named barrier over
// its gs threads (1 to 15; barrier 0 is the whole CTA's, so groups of 64 need a
// CTA of at most 960 threads).
__device__ __forceinline__ void group_sync(u32 gid, u32 gs)
{
    if (gs == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(gid + 1), "r"(gs) : "memory");
}

constexpr u32 WAIT_BOUND = 1u << 24;   // default try_wait rounds before a copy is declared lost
constexpr u32 NONE = 0xFFFFFFFFu;

// ---- a group's slice of the CTA's dynamic shared memory ----
// Slice | anchors start[GS + 1] (+1 pad) | filter words | queue of GS/2 filter
// passes.  The index of the anchors takes the filter's place once the giant
// steps are done.
// The rare paths are __noinline__ functions that take the slice and a few
// scalars, so the hot loops stay small.
struct Slice {
    PrimeHdr hdr[2];             // this prime's header and the next one's
    u32 idx[2];                  // their record indices (NONE: no more primes)
    u32 claim;                   // the prime after them, claimed ahead
    u32 order;                   // ord(s) when it is at most Q', else NONE
    u32 abort;                   // a record wait gave up
    u32 nq;                      // filter passes put on the queue
    u32 w0, w1, t0, t1;          // this pass: giant steps [t0, t1) of the chunks of items [w0, w1)
    u64 zt;                      // S^t0
    u64 pw[16];                  // s^l, l < 16
};
static_assert(sizeof(Slice) % 16 == 0, "slices start on 16-byte boundaries");
__device__ __forceinline__ u64 *slice_start(Slice *s) { return reinterpret_cast<u64 *>(s + 1); }
__device__ __forceinline__ u32 *slice_filter(Slice *s, u32 gs) { return reinterpret_cast<u32 *>(slice_start(s) + gs + 2); }
constexpr u32 INDEX_PT = 16;           // index slots per anchor
static_assert(INDEX_PT <= FILTER_WPT, "the index lies in the filter's words");
// queue of filter passes: {value bits, item, giant step}
__device__ __forceinline__ uint4 *slice_queue(Slice *s, u32 gs) { return reinterpret_cast<uint4 *>(slice_filter(s, gs) + FILTER_WPT * gs); }
__host__ __device__ constexpr size_t slice_bytes(u32 gs)
{
    return sizeof(Slice) + (gs + 2) * 8 + (size_t)FILTER_WPT * gs * 4 + gs / 2 * 16;
}
static_assert(slice_bytes(32) % 16 == 0, "slices start on 16-byte boundaries");
// the slices of TPB/gs groups take the most room for gs = 32
template <int TPB>
constexpr size_t smem_bytes() { return slice_bytes(32) * (TPB / 32); }

extern __shared__ __align__(128) unsigned char smem_raw[];
__shared__ unsigned long long s_cands, s_dups, s_facs;   // per-CTA totals
__shared__ unsigned long long s_baby, s_giant, s_small;

// One more for each of the warp's lanes here together, by one atomic (a 64-bit add in
// shared memory by every lane to the same word: 38 cycles of an SM per claim).
__device__ __forceinline__ void count(unsigned long long *total)
{
    const u32 here = __activemask();
    if ((threadIdx.x & 31) == (u32)__ffs((int)here) - 1) atomicAdd(total, (unsigned long long)__popc(here));
}

// First claimer of term (seq, n) clears its bitmap bit and appends the factor.
__device__ __forceinline__ void claim(const BsgsArgs &a, u64 p, u32 seq, u32 n)
{
    const u32 o = n - a.nmin;
    u32 *w = a.bitmap + (size_t)seq * a.words + (o >> 5);
    const u32 mask = 1u << (o & 31);
    const u32 old = atomicAnd(w, ~mask);
    if (old & mask) {
        const u32 f = atomicAdd(a.factor_ctr, 1u);
        count(&s_facs);
        if (f < a.factor_cap) {
            FactorRec r;
            r.p = p; r.n = n; r.seq = seq;
            a.factors[f] = r;
        } else {
            atomicOr(a.err, ERR_FACTOR_OVERFLOW);
        }
    } else {
        count(&s_dups);
    }
}

// Builds the group's index of anchors (open addressing over 16 GS slots, t + 1
// in a slot, 0: empty) in the filter's place, and pw[l] = s^l for l < 16.
// Called by the whole group after the last use of the filter; the checks below
// follow it.
template <int MODE>
__device__ __noinline__ void build_index(Slice *sl, const PrimeHdr *H, u32 gid, u32 gs, u32 gt)
{
    typedef typename Ring<MODE>::V V;
    u32 *idx = slice_filter(sl, gs);
    u64 *start = slice_start(sl);
    for (u32 i = gt; i < INDEX_PT / 4 * gs; i += gs) reinterpret_cast<uint4 *>(idx)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (gt < 16) {
        const Ring<MODE> R(*H);
        V x = Ring<MODE>::val(H->s), r = (gt & 1) ? x : Ring<MODE>::one(*H);
        for (u32 k = 1; k < 4; ++k) {
            x = R.mul(x, x);
            const V t = R.mul(r, x);
            r = ((gt >> k) & 1) ? t : r;
        }
        sl->pw[gt] = Ring<MODE>::bits(r);
    }
    group_sync(gid, gs);
    // anchors t = gt, and by the first thread the one past the end, s^Q'; at most
    // GS + 1 entries, so the walks end.  Of equal ones (ord(s) <= Q') one is enough:
    // all of them, in one run of slots, made every walk as long as the run.
    for (u32 t = gt; t < gs + 1; t += gs) {
        const u64 v = (t == gs) ? H->S : start[t];
        if (t == gs) start[gs] = v;
        u32 k = __umulhi(val_hash(v), INDEX_PT * gs);
        for (u32 e; (e = atomicCAS(&idx[k], 0u, t + 1)) != 0u && start[e - 1] != v;) k = (k + 1) & (INDEX_PT * gs - 1);
    }
    group_sync(gid, gs);
}

// The anchor equal to v, or NONE.
__device__ __forceinline__ u32 anchor_find(const u32 *idx, const u64 *start, u32 gs, u64 v)
{
    u32 k = __umulhi(val_hash(v), INDEX_PT * gs);
    for (u32 n = 0; n < INDEX_PT * gs; ++n) {
        const u32 e = idx[k];
        if (e == 0) return NONE;
        if (start[e - 1] == v) return e - 1;
        k = (k + 1) & (INDEX_PT * gs - 1);
    }
    return NONE;
}

// Exact discrete logarithm of gamma (uniform over the warp) to the base s among
// the group's anchors: lane l < 16 looks gamma * s^l up.  Returns 16t - l, in
// (-16, Q'], of the first lane that finds an anchor t, or NO_LOG.  When ord(s) >
// Q' the anchors differ, and gamma = s^j with 0 <= j < Q' is found as exactly
// that j.  Called by a whole warp.
constexpr int NO_LOG = -1000;
template <int MODE>
__device__ __forceinline__ int warp_find(const Ring<MODE> &R, Slice *sl, u32 gs, typename Ring<MODE>::V gamma)
{
    const u32 lane = threadIdx.x & 31;
    u32 t = NONE;
    if (lane < 16)
        t = anchor_find(slice_filter(sl, gs), slice_start(sl), gs,
                        Ring<MODE>::bits(R.mul(gamma, Ring<MODE>::val(sl->pw[lane]))));
    const u32 found = __ballot_sync(0xFFFFFFFFu, t != NONE);
    if (!found) return NO_LOG;
    const u32 src = __ffs((int)found) - 1;
    return (int)(16 * __shfl_sync(0xFFFFFFFFu, t, src)) - (int)src;
}

// Item w of a prime's giant phase: chunk g of target i, w = g*numk + i, by the
// float reciprocal in the header: (w + 1/2)/numk lies at least 1/(2 numk) from
// an integer and errs by under 2^-21 of itself (w < 2^17).
__device__ __forceinline__ void item_of(u32 w, const PrimeHdr *H, u32 &g, u32 &i)
{
    g = (u32)(((float)w + 0.5f) * H->rk);
    i = w - g * H->numk;
}

// One sixteenth of a filter pass's exact check: if gamma * s^l is anchor t, gamma =
// s^j with j = 16t - l.  Returns j when it lies in [0, Q'), else NONE.
template <int MODE>
__device__ __forceinline__ u32 log_at(const Ring<MODE> &R, Slice *sl, u32 gs, u64 gamma, u32 l)
{
    const u32 a = anchor_find(slice_filter(sl, gs), slice_start(sl), gs,
                              Ring<MODE>::bits(R.mul(Ring<MODE>::val(gamma), Ring<MODE>::val(sl->pw[l]))));
    const u32 j = 16 * a - l;                              // (negative: past the end as well)
    return (a != NONE && j < 16 * gs) ? j : NONE;
}

// Claims the term of item w's giant step t (of its chunk), whose value is s^j: n =
// nmin + off + e*((q+1)Q'-1-j).
__device__ __forceinline__ void claim_step(const PrimeHdr *H, u32 gs, u32 j, u32 w, u32 t, const BsgsArgs *args,
                                           const unsigned short *meta)
{
    u32 g, i;
    item_of(w, H, g, i);
    const u32 m = meta[i];
    const u64 u = (u64)(g * H->Lc + t + 1) * (16 * gs) - 1 - j;
    const u64 n = (u64)args->nmin + (m >> 7) + (u64)H->e * u;
    if (n <= args->nmax) claim(*args, H->p, m & 0x7Fu, (u32)n);
}

// Pass seg of a prime whose chunks are longer than a pass should be: `piece` steps of
// one round's chunks.  Returns the round.
template <int MODE>
__device__ __noinline__ u32 cut_chunk(Slice *sl, const PrimeHdr *H, u32 seg)
{
    typedef typename Ring<MODE>::V V;
    const Ring<MODE> R(*H);
    const u32 n = (H->Lc + H->piece - 1) / H->piece, r = seg / n, t0 = (seg - r * n) * H->piece;
    sl->t0 = t0;
    sl->t1 = min(t0 + H->piece, H->Lc);
    V z = Ring<MODE>::one(*H), x = Ring<MODE>::val(H->S);
    for (u32 k = t0; k; k >>= 1) {
        if (k & 1) z = R.mul(z, x);
        x = R.mul(x, x);
    }
    sl->zt = Ring<MODE>::bits(z);
    return r;
}
// What pass seg of a prime walks (Slice): `rounds` rounds of 2 GS items and their whole
// chunks, or a part of one round's.  By the group's first thread.
template <int MODE>
__device__ __forceinline__ void start_pass(Slice *sl, const PrimeHdr *H, u32 gs, u32 seg)
{
    sl->t0 = 0;
    sl->t1 = H->Lc;
    if (H->piece < H->Lc) seg = cut_chunk<MODE>(sl, H, seg);
    const u32 per = H->rounds * 2 * gs;
    sl->w0 = seg * per;
    sl->w1 = min((seg + 1) * per, H->numk * H->G);
}

// Value of item w at the pass's first giant step: T_i * S^(g*Lc + t0).
template <int MODE>
__device__ __forceinline__ typename Ring<MODE>::V item_start(const Ring<MODE> &R, u32 w, const Slice *sl, const PrimeHdr *H,
                                                             const u64 *tb, const u64 *tg)
{
    typedef typename Ring<MODE>::V V;
    u32 g, i;
    item_of(w, H, g, i);
    V z = Ring<MODE>::val(tb[64 + (g & 31)]);
    if (H->G > 32) z = R.mul(z, Ring<MODE>::val(tb[96 + (g >> 5)]));
    if (sl->t0) z = R.mul(z, Ring<MODE>::val(sl->zt));
    return R.mul(Ring<MODE>::val(tg[i]), z);
}

// More filter passes than the queue holds (p not far above Q', where most are
// true): the pass's giant steps again, one item per thread, each value checked by
// its own thread.
template <int MODE>
__device__ __noinline__ void giant_unqueued(Slice *sl, const PrimeHdr *H, u32 gs, u32 gt, const u64 *tb, const u64 *tg,
                                            const BsgsArgs *args, const unsigned short *meta)
{
    typedef typename Ring<MODE>::V V;
    const Ring<MODE> R(*H);
    const typename Ring<MODE>::Fix f = Ring<MODE>::giant(*H);
    for (u32 w = sl->w0 + gt; w < sl->w1; w += gs) {
        V g = item_start<MODE>(R, w, sl, H, tb, tg);
        for (u32 t = sl->t0; t < sl->t1; ++t, g = R.step(g, f)) {
            u32 j = NONE;                                  // (claimed past the loop: by all lanes of a warp together)
            for (u32 l = 0; l < 16 && j == NONE; ++l) j = log_at<MODE>(R, sl, gs, Ring<MODE>::bits(g), l);
            if (j != NONE) claim_step(H, gs, j, w, t, args, meta);
        }
    }
}

// ord(s) <= Q': each target is looked up once, warps of the group taking targets in
// turn, and every n in range with the same residue mod e*ord is claimed
// (giant.cl:146-168): blocks of 32 claims of all targets, dealt to the warps in turn,
// as there may be fewer targets than warps, of 10^5 claims each (100 sequences, n-range
// 6*10^6, the primes from 100 to 1000: 17.4 ms with a warp per target, 13.3 so).  The
// targets' first u lie in the filter's words past the index.  Called by the whole group.
template <int MODE>
__device__ __noinline__ void small_order_search(Slice *sl, const PrimeHdr *H, const BsgsArgs *args, u32 gid, u32 gs, u32 gt,
                                                const u64 *__restrict__ tgt, const unsigned short *__restrict__ meta)
{
    static_assert((FILTER_WPT - INDEX_PT) * 32 >= KMAX, "room for the targets' first u");
    const Ring<MODE> R(*H);
    const u32 lane = gt & 31, warps = gs >> 5, numk = H->numk;
    const u32 Q = 16 * gs, order = sl->order;
    u32 *first = slice_filter(sl, gs) + INDEX_PT * gs;
    for (u32 i = gt >> 5; i < numk; i += warps) {
        const int j = warp_find<MODE>(R, sl, gs, Ring<MODE>::val(tgt[i]));
        if (lane == 0) {
            first[i] = (j == NO_LOG) ? NONE : (u32)((int)(Q - 1 + order) - j) % order;
            if (j != NO_LOG) atomicAdd(&s_cands, 1ull);
        }
    }
    group_sync(gid, gs);
    // u < ceil(L/e), blocks of 32*order of them
    const u64 span = 32ull * order;
    const u32 blocks = (u32)((args->nmax - args->nmin) / H->e / span) + 1;
    for (u32 i = 0, k = gt >> 5;; k += warps) {
        while (i < numk && (first[i] == NONE || k >= blocks)) {
            if (first[i] != NONE) k -= blocks;
            ++i;
        }
        if (i >= numk) return;
        const u32 m = meta[i];
        const u64 n = (u64)args->nmin + (m >> 7) + (u64)H->e * (first[i] + lane * order + k * span);
        if (n <= args->nmax) claim(*args, H->p, m & 0x7Fu, (u32)n);
    }
}

// The least j in (0, Q'] with y_j = 1 among this thread's chain, merged into
// the group's order (only called when some value's hash equals that of 1).
template <int MODE>
__device__ __noinline__ void order_check(Slice *sl, const PrimeHdr *H, u32 j0, u64 x0)
{
    const Ring<MODE> R(*H);
    const typename Ring<MODE>::V s = Ring<MODE>::val(H->s);
    const u64 one = Ring<MODE>::bits(Ring<MODE>::one(*H));
    typename Ring<MODE>::V x = Ring<MODE>::val(x0);
    for (u32 j = j0 + 1; j <= j0 + 16; ++j) {
        x = R.mul(x, s);
        if (Ring<MODE>::bits(x) == one) {
            atomicMin(&sl->order, j);
            return;
        }
    }
}

// The primes of one launch, sorted by class into lists of record indices
// (setup.cu, BsgsLists): count[c] primes of class c at lists + c*stride.  CTAs of TPB
// threads work through the classes from the largest down; a class of GS
// threads per prime runs TPB/GS groups side by side, each claiming the next
// prime of the class when it finishes one.  taken[c] starts at zero.
// MODE: 2 = every prime below FP_BOUND = 2^51 (FP64 steps), 1 = every prime
// below 2^63 (Shoup steps), 0 = every prime at or above 2^63 (Montgomery
// steps).  1024 / TPB CTAs share an SM, so the bound keeps each thread at 64
// registers.  BATCH: the primes of several jobs; each prime's job arguments
// come from job_args.
template <int TPB, int MODE, bool BATCH>
__global__ void __launch_bounds__(TPB, 1024 / TPB)
    k_bsgs(BsgsArgs a, const PrimeHdr *__restrict__ hdr, const u64 *__restrict__ tabs, const u64 *__restrict__ tgt,
           const unsigned short *__restrict__ meta, const u32 *__restrict__ lists, u32 stride,
           const u32 *__restrict__ count, u32 *taken, const BsgsArgs *__restrict__ job_args)
{
    typedef Ring<MODE> RM;
    typedef typename RM::V V;
    // (the integer products' longer code runs slower unrolled further: 8% at p
    // near 2^64)
    constexpr int BABY_UNROLL = MODE == 2 ? 8 : 2, GIANT_UNROLL = MODE == 2 ? 2 : 1;
    __shared__ __align__(8) u64 s_bar[TPB / 32][2];               // record copies of each group (by its first warp)
    __shared__ __align__(8) u64 s_dead;                           // never completed (failure test)
    __shared__ u32 s_par[TPB / 32][2];                            // parity of each barrier's next phase
    __shared__ BsgsArgs s_args;
    __shared__ u32 s_abort;
    const u32 wait_bound = a.wait_bound ? a.wait_bound : WAIT_BOUND;
    const u32 tid = threadIdx.x;
    if ((tid & 31) == 0) {
        mbar_init(&s_bar[tid >> 5][0], 1);
        mbar_init(&s_bar[tid >> 5][1], 1);
        s_par[tid >> 5][0] = s_par[tid >> 5][1] = 0;
    }
    if (tid == 0) {
        mbar_init(&s_dead, 1);
        s_args = a;
        s_abort = 0;
        s_cands = s_dups = s_facs = 0;
        s_baby = s_giant = s_small = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");

    for (int c = NCLASS - 1; c >= 0; --c) {
        const u32 gs = 32u << c;
        const u32 n = count[c];
        if (gs > TPB || n == 0) continue;
        __syncthreads();                                          // slices of the previous class are free
        const bool stop = s_abort != 0;
        __syncthreads();                                          // (the flag is read before any group can set it again)
        if (stop) break;
        const u32 gid = tid / gs, gt = tid & (gs - 1), w0 = gid * (gs >> 5);
        const u32 ngroups = gridDim.x * (TPB / gs);
        Slice *sl = reinterpret_cast<Slice *>(smem_raw + gid * slice_bytes(gs));
        u64 *start = slice_start(sl);
        u32 *filt = slice_filter(sl, gs);
        const u32 nw = FILTER_WPT * gs;
        const u32 *list = lists + (BATCH ? count[3 * NCLASS + c] : c * stride);
        auto fetch = [&](u32 buf, u32 r) {                        // group's first thread only
            mbar_expect_tx(&s_bar[w0][buf], (u32)sizeof(PrimeHdr));
            bulk_load(&sl->hdr[buf], hdr + r, (u32)sizeof(PrimeHdr), &s_bar[w0][buf]);
            l2_prefetch(tabs + (size_t)r * TABS, TABS * 8);
            l2_prefetch(tgt + (size_t)r * KSTRIDE, KSTRIDE * 8);
            l2_prefetch(meta + (size_t)r * KSTRIDE, KSTRIDE * 2);
        };
        // the first prime of each group is fixed, the others are claimed in order
        // (past the end there is nothing: NONE)
        auto claimed = [&](u32 k) -> u32 { return k < n ? list[k] : NONE; };
        if (gt == 0) {
            const u32 r = claimed(blockIdx.x + gid * gridDim.x);
            sl->idx[0] = r;
            sl->claim = NONE;
            sl->abort = 0;
            if (r != NONE) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                fetch(0, r);
                sl->claim = claimed(ngroups + atomicAdd(&taken[c], 1u));
            }
        }
        group_sync(gid, gs);

        // one pass of the loop per prime, or per segment seg of a prime with a long
        // giant phase (every segment fills the filter again; start_pass says what it walks)
        for (u32 it = 0, seg = 0;;) {
            const u32 buf = it & 1;
            const u32 r = sl->idx[buf];
            if (r == NONE) break;
            // the starts' table entries, and an empty filter while they arrive
            const u64 *tb = tabs + (size_t)r * TABS;
            const u64 ta = tb[gt & 31], tB = tb[32 + (gt >> 5)];
            {
                uint4 *z = reinterpret_cast<uint4 *>(filt);
                const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (u32 i = 0; i < FILTER_WPT / 4; ++i) z[i * gs + gt] = zero;
            }
            // this prime's header was fetched one prime ago; the wait is bounded.
            // A failure test sends the first wait to s_dead, which no copy or
            // arrival ever completes, so the bound runs out.
            if (seg == 0) {
                const bool dead = (a.test_stall != 0) && (it == 0);
                u64 *bar = dead ? &s_dead : &s_bar[w0][buf];
                const u32 want = dead ? 0u : s_par[w0][buf];
                u32 tries = 0;
                while (!mbar_try_wait(bar, want)) {
                    if (++tries > wait_bound) { sl->abort = 1; break; }
                }
            }
            if (gt == 0) {
                sl->order = NONE;
                sl->nq = 0;
                if (!sl->abort) start_pass<MODE>(sl, &sl->hdr[buf], gs, seg);   // (the header is here)
            }
            group_sync(gid, gs);
            if (sl->abort) {
                // The group stops before fetching another record, so the only copy
                // that can still be in flight is the one waited for: report, then
                // let it land (bounded by the default) before the CTA's shared
                // memory is released.
                if (gt == 0) {
                    atomicOr(a.err, ERR_TMA_TIMEOUT);
                    s_abort = 1;
                    u32 tries = 0;
                    while (tries < WAIT_BOUND && !mbar_try_wait(&s_bar[w0][buf], s_par[w0][buf])) ++tries;
                }
                break;
            }
            if (gt == 0 && seg == 0) {
                s_par[w0][buf] ^= 1;
                const u32 nxt = sl->claim;
                sl->idx[buf ^ 1] = nxt;
                if (nxt != NONE) {                                // hdr[buf^1] was last read before the barrier
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    fetch(buf ^ 1, nxt);
                }
            }
            const PrimeHdr *H = &sl->hdr[buf];
            const RM R(*H);
            // The last thread claims the prime after next.  The claim, issued here,
            // and the load of its record index, issued after the baby steps, are
            // taken up a phase later, so no warp waits for them.
            const bool claimer = (gt == gs - 1) && seg == 0;
            u32 ahead = NONE;
            if (claimer) ahead = ngroups + atomicAdd(&taken[c], 1u);
            // ---- baby steps y_j = s^j, j < Q' = 16 GS, entered as they are produced ----
            {
                const V x0 = R.mul(RM::val(ta), RM::val(tB));     // s^(16 gt)
                start[gt] = RM::bits(x0);
                // two chains, j in [16 gt, 16 gt + 8) and the next 8, so that the
                // two products of a step are independent; the step kind is uniform
                // per prime and chosen once.  A value whose hash equals that of 1
                // is a candidate for y_j = 1, j > 0: the values after each step,
                // j = 16 gt + 1 .. 16 gt + 16, are compared.
                const typename RM::Fix f = RM::baby(*H);
                const u32 h1 = val_hash(RM::bits(RM::one(*H)));
                V xa = x0, xb = R.mul(x0, RM::val(H->u8));
                bool unit = false;
                auto babies = [&](auto kind) {
                    constexpr int K = decltype(kind)::value;      // 2, 4: doublings; 1: product by s
                    auto step = [&](V v) -> V {
                        if (K == 1) return R.step(v, f);
                        v = R.dbl(v);
                        return (K == 4) ? R.dbl(v) : v;
                    };
                    u32 ha = val_hash(RM::bits(xa)), hb = val_hash(RM::bits(xb));
#pragma unroll BABY_UNROLL
                    for (int i = 0; i < 8; ++i) {
                        atomicOr(&filt[__umulhi(ha, nw)], filter_mask(ha));
                        atomicOr(&filt[__umulhi(hb, nw)], filter_mask(hb));
                        xa = step(xa);
                        xb = step(xb);
                        ha = val_hash(RM::bits(xa));
                        hb = val_hash(RM::bits(xb));
                        unit |= (ha == h1) | (hb == h1);
                    }
                };
                const u32 smul = H->smul;
                if (smul == 2) babies(std::integral_constant<int, 2>{});
                else if (smul == 4) babies(std::integral_constant<int, 4>{});
                else babies(std::integral_constant<int, 1>{});
                if (unit) order_check<MODE>(sl, H, 16 * gt, start[gt]);
            }
            if (claimer) ahead = claimed(ahead);
            group_sync(gid, gs);
            const u64 *tg = tgt + (size_t)r * KSTRIDE;
            const u32 order = sl->order;                          // (the first thread resets it for the next pass)
            if (order == NONE) {
                // ---- giant steps: items (target i, chunk g), two per thread at a time ----
                const u32 wend = sl->w1, nitems = H->numk * H->G;
                const typename RM::Fix f = RM::giant(*H);
                // a filter pass of giant step t of item w goes on the queue (a lane
                // past the last item repeats it, and its passes are that item's own)
                auto pass = [&](V g, u32 w, u32 t) {
                    if (w >= nitems) return;
                    const u64 v = RM::bits(g);
                    const u32 k = atomicAdd(&sl->nq, 1u);
                    if (k < gs / 2) slice_queue(sl, gs)[k] = make_uint4((u32)v, (u32)(v >> 32), w, t);
                };
                for (u32 w = sl->w0 + gt; (w & ~31u) < wend; w += 2 * gs) {
                    V gA = item_start<MODE>(R, min(w, nitems - 1), sl, H, tb, tg);
                    const u32 t1 = sl->t1;
                    u32 t = sl->t0;
                    if ((w & ~31u) + gs < nitems) {
                        V gB = item_start<MODE>(R, min(w + gs, nitems - 1), sl, H, tb, tg);
                        // two steps of both chains per test of the four probes
#pragma unroll GIANT_UNROLL
                        for (; t + 1 < t1; t += 2) {
                            const u32 ha = val_hash(RM::bits(gA)), hb = val_hash(RM::bits(gB));
                            const u32 fa = filt[__umulhi(ha, nw)], fb = filt[__umulhi(hb, nw)];
                            const V nA = R.step(gA, f), nB = R.step(gB, f);
                            const u32 hc = val_hash(RM::bits(nA)), hd = val_hash(RM::bits(nB));
                            const u32 fc = filt[__umulhi(hc, nw)], fd = filt[__umulhi(hd, nw)];
                            const V mA = R.step(nA, f), mB = R.step(nB, f);
                            // the bits each probe misses: none for a pass
                            const u32 a = filter_mask(ha) & ~fa, b = filter_mask(hb) & ~fb, c2 = filter_mask(hc) & ~fc,
                                      d = filter_mask(hd) & ~fd;
                            if (__any_sync(0xFFFFFFFFu, min(min(a, b), min(c2, d)) == 0)) {
                                if (a == 0) pass(gA, w, t);
                                if (b == 0) pass(gB, w + gs, t);
                                if (c2 == 0) pass(nA, w, t + 1);
                                if (d == 0) pass(nB, w + gs, t + 1);
                            }
                            gA = mA;
                            gB = mB;
                        }
                        if (t < t1) {
                            const u32 ha = val_hash(RM::bits(gA)), hb = val_hash(RM::bits(gB));
                            if ((filter_mask(ha) & ~filt[__umulhi(ha, nw)]) == 0) pass(gA, w, t);
                            if ((filter_mask(hb) & ~filt[__umulhi(hb, nw)]) == 0) pass(gB, w + gs, t);
                        }
                    } else {
                        for (; t < t1; ++t) {
                            const u32 ha = val_hash(RM::bits(gA));
                            const u32 fa = filt[__umulhi(ha, nw)];
                            const V nA = R.step(gA, f);
                            if ((filter_mask(ha) & ~fa) == 0) pass(gA, w, t);
                            gA = nA;
                        }
                    }
                }
            } else {
                build_index<MODE>(sl, H, gid, gs, gt);
                small_order_search<MODE>(sl, H, BATCH ? job_args + H->job : &s_args, gid, gs, gt, tg,
                                         meta + (size_t)r * KSTRIDE);
            }
            if (claimer) sl->claim = ahead;
            group_sync(gid, gs);
            // the queued filter passes, 16 lanes each
            const u32 nq = sl->nq;
            if (nq) {
                build_index<MODE>(sl, H, gid, gs, gt);
                const BsgsArgs *args = BATCH ? job_args + H->job : &s_args;
                const unsigned short *mt = meta + (size_t)r * KSTRIDE;
                if (nq <= gs / 2) {
                    for (u32 k = gt >> 4; k < nq; k += gs >> 4) {
                        const uint4 x = slice_queue(sl, gs)[k];
                        const u32 j = log_at<MODE>(RM(*H), sl, gs, ((u64)x.y << 32) | x.x, gt & 15);
                        if (j != NONE) claim_step(H, gs, j, x.z, x.w, args, mt);
                    }
                } else {
                    giant_unqueued<MODE>(sl, H, gs, gt, tb, tg, args, mt);
                }
                if (gt == 0) atomicAdd(&s_cands, (unsigned long long)nq);
                group_sync(gid, gs);
            }
            if (++seg < H->nseg && order == NONE) continue;
            if (gt == 0) {
                atomicAdd(&s_baby, (unsigned long long)min(order, 16 * gs));
                if (order == NONE) atomicAdd(&s_giant, (unsigned long long)H->numk * H->Mg);
                else atomicAdd(&s_small, 1ull);
            }
            seg = 0;
            ++it;
        }
    }
    __syncthreads();
    if (tid == 0) {
        atomicAdd(&a.stats[ST_BABY], s_baby);
        atomicAdd(&a.stats[ST_GIANT], s_giant);
        atomicAdd(&a.stats[ST_SMALLORDER], s_small);
        atomicAdd(&a.stats[ST_CANDIDATES], s_cands);
        atomicAdd(&a.stats[ST_DUPS], s_dups);
        atomicAdd(&a.stats[ST_FACTORS], s_facs);
        atomicAdd(&a.stats[ST_HITS], s_dups + s_facs);
    }
}

template <int TPB, int MODE, bool BATCH>
static cudaError_t launch_shape(const BsgsArgs &a, const PrimeHdr *hdr, const u64 *tabs, const u64 *tgt,
                               const unsigned short *meta, const BsgsLists &L, int sms, cudaStream_t st,
                               const BsgsArgs *job_args)
{
    auto kern = k_bsgs<TPB, MODE, BATCH>;
    kern<<<(unsigned)(sms * (1024 / TPB)), TPB, smem_bytes<TPB>(), st>>>(a, hdr, tabs, tgt, meta, L.list, L.stride,
                                                                        L.ctl, L.ctl + NCLASS, job_args);
    return cudaGetLastError();
}

template <bool BATCH>
static cudaError_t launch_any(const BsgsArgs &a, const PrimeHdr *hdr, const u64 *tabs, const u64 *tgt,
                              const unsigned short *meta, const BsgsLists &L, int mode, u32 tpb, int sms,
                              cudaStream_t st, const BsgsArgs *job_args)
{
    if (tpb == 1024)
        return mode == 2 ? launch_shape<1024, 2, BATCH>(a, hdr, tabs, tgt, meta, L, sms, st, job_args)
             : mode == 1 ? launch_shape<1024, 1, BATCH>(a, hdr, tabs, tgt, meta, L, sms, st, job_args)
                         : launch_shape<1024, 0, BATCH>(a, hdr, tabs, tgt, meta, L, sms, st, job_args);
    return mode == 2 ? launch_shape<512, 2, BATCH>(a, hdr, tabs, tgt, meta, L, sms, st, job_args)
         : mode == 1 ? launch_shape<512, 1, BATCH>(a, hdr, tabs, tgt, meta, L, sms, st, job_args)
                     : launch_shape<512, 0, BATCH>(a, hdr, tabs, tgt, meta, L, sms, st, job_args);
}

size_t bsgs_smem_bytes() { return smem_bytes<1024>(); }

cudaError_t bsgs_prepare()
{
    cudaError_t e = cudaSuccess;
    auto set = [&](const void *k, size_t bytes) {
        const cudaError_t r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e == cudaSuccess) e = r;
    };
#define RS_BSGS_SET(TPB, MODE)                                                  \
    set((const void *)k_bsgs<TPB, MODE, false>, smem_bytes<TPB>());             \
    set((const void *)k_bsgs<TPB, MODE, true>, smem_bytes<TPB>());
    RS_BSGS_SET(512, 0) RS_BSGS_SET(512, 1) RS_BSGS_SET(512, 2)
    RS_BSGS_SET(1024, 0) RS_BSGS_SET(1024, 1) RS_BSGS_SET(1024, 2)
#undef RS_BSGS_SET
    return e;
}

cudaError_t launch_bsgs(const BsgsArgs &a, const PrimeHdr *hdr, const u64 *tabs, const u64 *tgt,
                        const unsigned short *meta, const BsgsLists &L, u64 pmin, u64 pmax, int geom, int sms,
                        cudaStream_t st)
{
    const u64 TOP = 1ull << 63;
    if (pmin < TOP && pmax > TOP) return cudaErrorInvalidValue;   // the caller splits launches at 2^63
    if (pmin < FP_BOUND && pmax > FP_BOUND) return cudaErrorInvalidValue;   // and at FP_BOUND
    if (geom < 0 || geom >= NGEOM) return cudaErrorInvalidValue;
    const int mode = (pmax <= FP_BOUND) ? 2 : (pmax <= TOP) ? 1 : 0;
    return launch_any<false>(a, hdr, tabs, tgt, meta, L, mode, BSGS_GEOMS[geom].tpb, sms, st, nullptr);
}

cudaError_t launch_bsgs_batch(const BsgsArgs &a, const BsgsArgs *job_args, const PrimeHdr *hdr, const u64 *tabs,
                              const u64 *tgt, const unsigned short *meta, const BsgsLists &L, int group, int sms,
                              cudaStream_t st)
{
    return launch_any<true>(a, hdr, tabs, tgt, meta, L, group % 3, group >= 3 ? 1024 : 512, sms, st, job_args);
}

// prefix[0] = 0, prefix[k+1] = prefix[k] + counter `which` of range slot k
// (capped at rcap) when it is active, else + 0.  One block of 256 threads: each
// sums a contiguous run of slots, a block scan offsets the runs.
__global__ void __launch_bounds__(256) k_batch_prefix(const BatchRange *ranges, u32 nr, const u32 *ctrs, u32 rcap,
                                                      u32 *prefix, int which)
{
    __shared__ u32 part[256];
    const u32 t = threadIdx.x;
    const u32 per = (nr + 255) / 256;
    const u32 k0 = t * per, k1 = min(k0 + per, nr);
    auto cnt = [&](u32 k) -> u32 {
        return ranges[k].active ? min(ctrs[k * BR_CTRS + which], rcap) : 0u;
    };
    u32 sum = 0;
    for (u32 k = k0; k < k1; ++k) sum += cnt(k);
    part[t] = sum;
    __syncthreads();
    for (u32 o = 1; o < 256; o <<= 1) {           // inclusive Hillis-Steele scan
        const u32 v = (t >= o) ? part[t - o] : 0u;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    u32 acc = part[t] - sum;                      // exclusive prefix of this run
    if (t == 0) prefix[0] = 0;
    for (u32 k = k0; k < k1; ++k) {
        acc += cnt(k);
        prefix[k + 1] = acc;
    }
}

cudaError_t launch_batch_prefix_all(const BatchRange *ranges, u32 nr, int which, u32 cap, const u32 *ctrs,
                                    u32 *prefix, cudaStream_t st)
{
    k_batch_prefix<<<1, 256, 0, st>>>(ranges, nr, ctrs, cap, prefix, which);
    return cudaGetLastError();
}

}  // namespace rs
