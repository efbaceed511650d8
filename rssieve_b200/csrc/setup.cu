// setup.cu -- per-prime set-up for the BSGS search.
//
// Replaces the reference's setup and sort kernels (kernels/setup.cl:89-209,
// kernels/sort.cl:11-104).  The arithmetic is re-derived rather than ported.
//
// Term k*b^n + c (c = +-1) is divisible by p iff k*b^n == -c (mod p).  Write
// n = nmin + off + e*u with a split modulus e (one table of powers of s = b^e
// serves every sequence) and u = (q+1)*Q - 1 - j with baby index j in [0,Q)
// and giant index q.  Then
//      s^j == T * S^q,   T = -c * k * b^(nmin + off + e*(Q-1)),   S = s^Q,
// so the baby table holds s^j and no modular inverse is needed (the reference
// batch-inverts every k and b^Q, setup.cl:133-166).
//
// Residue classes of n.  The reference splits n by parity when b is a
// quadratic non-residue mod p (e = 2) and filters with d-th power residues
// (setup.cl:22-87).  Here both come from one character of larger order.  Let D
// be the part of p-1 made of the primes up to 251, and chi(x) = x^((p-1)/D),
// which maps onto the D-th roots of unity.  If k*b^n == -c then
//      chi(b)^n = chi(-c) / chi(k),
// so (1) a target is impossible unless chi(-c)/chi(k) lies in the subgroup
// generated by chi(b), of order eo (the reference's filters are the cases
// d | D of this), and (2) n mod e is fixed, for every divisor e of eo, by the
// discrete logarithm of h = chi(b)^(eo/e) -- a table of e values.  e is the
// largest divisor of eo up to 256 (64 for small jobs, JobDev::split).  Both take
// one power per sequence, z = k^E with E = (p-1)/D * eo/e: the logarithm of
// (-c)^E / z to the base h exists exactly when (chi(-c)/chi(k))^eo = 1, the groups
// being cyclic.  Every n the reference finds satisfies both, so the eliminated
// terms are the same, while each sequence's giant steps
// shrink from L/Q to L/(e*Q) (e = 2 is the reference's parity case; at the
// 2^50 p-range of the 100-sequence job e averages well above 2).
// Primes dividing b or any k, and primes where no k survives, are skipped for
// every sequence as setup.cl:156-162,205-208 do.
//
// Kernel 1 (one thread per prime) does the per-prime scalars; kernel 2 (one
// warp per prime, lanes over k; with 16 sequences or fewer, 4 to 16 lanes per
// prime) classifies the sequences, chooses the prime's class, i.e. its baby-step
// count Q', and writes the compacted targets;
// kernel 3 (one thread per prime) writes the giant-step split and the baby-
// and giant-step start tables.  Per-prime work that is the same for every
// sequence runs one prime per thread, where it costs 1/32 of the issue slots
// it would take in the warp-per-prime kernel.
#include "mont.cuh"
#include "rs_internal.h"

#include <type_traits>
#include <utility>

namespace rs {

constexpr u32 SPLIT_MAX = 256;       // largest split modulus e of any job (at most 512: 9 bits of offset per target)
static_assert(SPLIT_MAX <= 512 && SPLIT_MAX % 32 == 0, "offsets and tables of powers");

// The primes whose powers make up D, the smooth part of p-1.
constexpr u32 SMOOTH[] = {
    2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67, 71, 73, 79,
    83, 89, 97, 101, 103, 107, 109, 113, 127, 131, 137, 139, 149, 151, 157, 163, 167, 173,
    179, 181, 191, 193, 197, 199, 211, 223, 227, 229, 233, 239, 241, 251};
constexpr int NSMOOTH = sizeof(SMOOTH) / sizeof(SMOOTH[0]);
constexpr int NSMALL = 18;           // those up to 61
static_assert(NSMOOTH <= 64 && SMOOTH[NSMALL - 1] == 61, "a prime's smooth factors are a 64-bit mask");
static_assert(SMOOTH[NSMOOTH - 1] <= SPLIT_MAX, "the reciprocals' table covers them");

struct PrimeAux {        // kernel 1 -> kernels 2 and 3; residues in the step kind's form (PrimeHdr)
    u64 E;               // the classes' exponent: z = k^E has order dividing e times the index filtered on
    u64 r2;              // R^2 mod p (p >= FP_BOUND)
    u64 b;               // b
    u64 hm1;             // h^-1, h = b^E of order e
    u64 wr0[NCLASS];     // per class, Q'_c = 512 << c: b^(nmin + e(Q'_c - 1))
    u64 S[NCLASS];       //   and s^Q'_c
};
static_assert(sizeof(PrimeAux) == SETUP_AUX, "the engine and the batch allocate it");

// ---- arithmetic of the set-up: plain residues in doubles below FP_BOUND, else
// Montgomery residues ----
template <bool FP>
struct Field;
template <>
struct Field<true> {
    typedef double V;
    double p, pinv;
    __device__ __forceinline__ explicit Field(u64 pi) : p(fp_exact(pi)) { pinv = 1.0 / p; }
    __device__ __forceinline__ Field(const PrimeHdr &h, const PrimeAux &) : p(fp_exact(h.p)), pinv(bits_double(h.q)) {}
    static __device__ __forceinline__ V val(u64 b) { return bits_double(b); }
    static __device__ __forceinline__ u64 bits(V v) { return double_bits(v); }
    __device__ __forceinline__ V one() const { return 1.0; }
    __device__ __forceinline__ V of_int(u64 x) const { return fp_exact(x); }        // x < p
    __device__ __forceinline__ V mul(V a, V b) const { return fp_mul(a, b, p, pinv); }
    __device__ __forceinline__ V neg(V a) const { return p - a; }                  // a != 0
    // products inside a power: any signed residue in (-p, p)
    static constexpr bool lazy = true;
    template <bool LAZY> __device__ __forceinline__ V pmul(V a, V b) const { return fp_mul_signed(a, b, p, pinv); }
    template <bool LAZY> __device__ __forceinline__ V psqr(V a) const { return fp_mul_signed(a, a, p, pinv); }
    template <bool LAZY> __device__ __forceinline__ V pend(V a) const { return (a < 0.0) ? a + p : a; }
};
template <>
struct Field<false> {
    typedef u64 V;
    Mont M;
    bool lazy;           // p < 2^62: products inside a power stay in [0, 2p)
    __device__ __forceinline__ explicit Field(u64 pi) : M(mont_init(pi)), lazy(pi >> 62 == 0) {}
    __device__ __forceinline__ Field(const PrimeHdr &h, const PrimeAux &x) : lazy(h.p >> 62 == 0)
    {
        M.p = h.p; M.q = h.q; M.one = h.one; M.r2 = x.r2;
    }
    static __device__ __forceinline__ V val(u64 b) { return b; }
    static __device__ __forceinline__ u64 bits(V v) { return v; }
    __device__ __forceinline__ V one() const { return M.one; }
    __device__ __forceinline__ V of_int(u64 x) const { return to_mont(x, M); }
    __device__ __forceinline__ V mul(V a, V b) const { return mmul(a, b, M.p, M.q); }
    __device__ __forceinline__ V neg(V a) const { return M.p - a; }
    template <bool LAZY> __device__ __forceinline__ V pmul(V a, V b) const
    {
        return LAZY ? mmul_lazy(a, b, M.p, M.q) : mmul(a, b, M.p, M.q);
    }
    template <bool LAZY> __device__ __forceinline__ V psqr(V a) const
    {
        return LAZY ? msqr_lazy(a, M.p, M.q) : mmul(a, a, M.p, M.q);
    }
    template <bool LAZY> __device__ __forceinline__ V pend(V a) const { return LAZY ? mred(a, M.p) : a; }
};

// x^e, every lane its own e (1 or more): two bits of e at a time, the digit's
// power (1, x, x^2, x^3) chosen by selects, so lanes do not diverge on their
// bits: 1.5 products per bit.
template <bool FP, bool LAZY>
__device__ __forceinline__ typename Field<FP>::V power_as(const Field<FP> &F, typename Field<FP>::V x, u64 e)
{
    typedef typename Field<FP>::V V;
    const V one = F.one(), x2 = F.template psqr<LAZY>(x), x3 = F.template pmul<LAZY>(x2, x);
    int i = (63 - __clzll(e)) & ~1;
    auto digit = [&]() -> V {
        const u32 d = (u32)(e >> i) & 3u;
        const V lo = (d & 1) ? x : one, hi = (d & 1) ? x3 : x2;
        return (d & 2) ? hi : lo;
    };
    V a = digit();
    for (i -= 2; i >= 0; i -= 2) {
        a = F.template psqr<LAZY>(F.template psqr<LAZY>(a));
        a = F.template pmul<LAZY>(a, digit());
    }
    return F.template pend<LAZY>(a);
}
// The same for e of 0 or more.  Out of line: one copy keeps the kernels small enough
// for the instruction cache.
template <bool FP>
__device__ __noinline__ typename Field<FP>::V power(const Field<FP> F, typename Field<FP>::V x, u64 e)
{
    if (e == 0) return F.one();
    return (FP || F.lazy) ? power_as<FP, true>(F, x, e) : power_as<FP, false>(F, x, e);
}

// The SMOOTH primes of index FROM to END-1 that divide x, as a mask of their
// indices.  No branches: the tests are independent.  Below 2^52 x is held in a
// double: q = x/L rounded; x - q*L, exact in the fma, is zero exactly when L divides
// x.  Else x is reduced by products of primes below 2^32, and those remainders by
// the primes.
template <int I>
__device__ __forceinline__ u64 divides_fp(double x)
{
    constexpr u32 L = SMOOTH[I];
    return fma(-fp_round_prod(x, 1.0 / L), (double)L, x) == 0.0 ? 1ull << I : 0ull;
}
template <int FROM, size_t... I>
__device__ __forceinline__ u64 smooth_mask(double x, std::index_sequence<I...>)
{
    return (divides_fp<FROM + (int)I>(x) | ...);
}
template <int FROM, int END>
__device__ __forceinline__ u64 smooth_mask(double x) { return smooth_mask<FROM>(x, std::make_index_sequence<END - FROM>()); }

__host__ __device__ constexpr int group_end(int from, int end)
{
    u64 m = 1;
    while (from < end && m * SMOOTH[from] < (1ull << 32)) m *= SMOOTH[from++];
    return from;
}
__host__ __device__ constexpr u32 group_product(int from, int end)
{
    u32 m = 1;
    for (; from < end; ++from) m *= SMOOTH[from];
    return m;
}
template <int I>
__device__ __forceinline__ u64 divides(u32 r)
{
    constexpr u32 L = SMOOTH[I];
    return r % L == 0 ? 1ull << I : 0ull;
}
template <int FROM, size_t... I>
__device__ __forceinline__ u64 group_mask(u32 r, std::index_sequence<I...>)
{
    return (divides<FROM + (int)I>(r) | ...);
}
template <int FROM, int END>
__device__ __forceinline__ u64 smooth_mask(u64 x)
{
    constexpr int J = group_end(FROM, END);
    constexpr u32 P = group_product(FROM, J);
    u64 m = group_mask<FROM>((u32)(x % P), std::make_index_sequence<J - FROM>());
    if constexpr (J < END) m |= smooth_mask<J, END>(x);
    return m;
}

// SMOOTH and the reciprocals of 1..SPLIT_MAX as tables
struct SetupTables {
    u32 smooth[NSMOOTH];
    double inv[SPLIT_MAX + 1];
};
constexpr SetupTables make_tables()
{
    SetupTables t{};
    for (int i = 0; i < NSMOOTH; ++i) t.smooth[i] = SMOOTH[i];
    for (u32 d = 1; d <= SPLIT_MAX; ++d) t.inv[d] = 1.0 / (double)d;
    return t;
}
__constant__ SetupTables c_tab = make_tables();

// x with every factor l (at most SPLIT_MAX) removed
__device__ __forceinline__ u64 without(u64 x, u32 l)
{
    if (x >> 52) {
        while (x % l == 0) x /= l;
        return x;
    }
    const double inv = c_tab.inv[l];
    double y = fp_exact(x);
    for (;;) {
        const double q = fp_round_prod(y, inv);
        if (fma(-q, (double)l, y) != 0.0) return fp_int(y);
        y = q;
    }
}

// Largest divisor of eo that is at most most (a multiple of 4); four candidates
// at a time, so that their tests overlap.
__device__ __forceinline__ u32 split_modulus(u64 eo, u32 most)
{
    if (eo <= most) return (u32)eo;
    if (eo >> 52) {
        u32 d = most;
        while (eo % d != 0) --d;
        return d;
    }
    const double x = fp_exact(eo);
    auto divides = [&](u32 d) { return fma(-fp_round_prod(x, c_tab.inv[d]), (double)d, x) == 0.0; };
    for (u32 d = most;; d -= 4) {
        const bool a = divides(d), b = divides(d - 1), c = divides(d - 2), e = divides(d - 3);
        if (a | b | c | e) return a ? d : b ? d - 1 : c ? d - 2 : d - 3;
    }
}

// b^e when it is 2 or 4 (baby steps by doublings), else 0.
__device__ __forceinline__ u32 doubling_power(u32 b, u32 e)
{
    if (e == 1) return b == 2 || b == 4 ? b : 0;
    return e == 2 && b == 2 ? 4 : 0;
}

// Per-prime constants of prime p into record t, with the powers that depend on
// the baby-step count for each of the classes kernel 2 chooses from.
template <bool FP>
__device__ __forceinline__ void setup_prime_one(const JobDev *__restrict__ job, u64 p, u32 t, u32 jb,
                                                PrimeHdr *__restrict__ hdr, PrimeAux *__restrict__ aux)
{
    typedef Field<FP> F;
    typedef typename F::V V;
    const u32 b = job->base;
    const u64 bp = (b < p) ? b : b % p;
    if (bp == 0) {                                        // p | b: no term is divisible by p
        PrimeHdr H{};                                     // (kernels 2 and 3 read its job and e)
        H.job = jb;
        H.e = 1;
        hdr[t] = H;
        return;
    }
    const F f(p);
    const V bv = f.of_int(bp);
    // D = smooth part of p-1, x = (p-1)/D, mask: its primes (small searches stop at 61)
    const int v2 = __ffsll((long long)(p - 1)) - 1;
    const u64 odd = (p - 1) >> v2;
    typename std::conditional<FP, double, u64>::type o;
    if constexpr (FP) o = fp_exact(odd);
    else o = odd;
    u64 mask = smooth_mask<1, NSMALL>(o);
    if (job->split > 64) mask |= smooth_mask<NSMALL, NSMOOTH>(o);
    u64 x = odd;
    for (u64 m = mask; m; m &= m - 1) x = without(x, c_tab.smooth[__ffsll((long long)m) - 1]);
    const u64 D = (p - 1) / x;
    mask |= 1;                                            // p is odd
    // chi(b) = b^x and its order eo | D, one prime of D at a time: the power by
    // D without that prime has the order's part of it
    const V g = power<FP>(f, bv, x);
    const u64 one = F::bits(f.one());
    u64 eo = 1;
    while (mask) {
        const u32 l = c_tab.smooth[__ffsll((long long)mask) - 1];
        mask &= mask - 1;
        V y = power<FP>(f, g, without(D, l));
        for (int i = 0; i < 64 && F::bits(y) != one; ++i) {
            y = power<FP>(f, y, l);
            eo *= l;
        }
    }
    const u32 e = split_modulus(eo, job->split);
    const u64 xe = eo / e;
    PrimeHdr H;
    PrimeAux X;
    X.E = x * xe;
    X.b = F::bits(bv);
    X.hm1 = F::bits(power<FP>(f, g, xe * (e - 1)));
    const V s = power<FP>(f, bv, e);
    // s^(Q'-1) by t <- t^2 * s from s^511, Q' = 512 << c
    const V bn = power<FP>(f, bv, job->nmin);
    V tq = power<FP>(f, s, 511);
#pragma unroll 1
    for (int c = 0; c < NCLASS; ++c) {
        if (c) tq = f.mul(f.mul(tq, tq), s);
        X.wr0[c] = F::bits(f.mul(bn, tq));
        X.S[c] = F::bits(f.mul(tq, s));
    }
    H.p = p;
    H.s = F::bits(s);
    H.S = 0; H.Sw = 0; H.Sp = 0; H.u8 = 0;
    if constexpr (FP) {
        X.r2 = 0;
        H.q = double_bits(f.pinv);
        H.one = double_bits(1.0);
        H.sw = double_bits(s / f.p);
        H.sp = 0;
    } else {
        X.r2 = f.M.r2;
        H.q = f.M.q;
        H.one = f.M.one;
        H.sw = 0; H.sp = 0;
        if (!(p >> 63)) {                                 // Shoup multiplier of the baby steps below 2^63
            H.sp = from_mont(s, f.M);
            H.sw = shoup_of_mont(s, f.M.q);
        }
    }
    H.numk = 0; H.e = e; H.G = 0; H.Lc = 0; H.job = jb; H.Mg = 0; H.cls = 0;
    H.smul = doubling_power(b, e);
    H.rk = 0; H.nseg = 0; H.rounds = 0; H.piece = 0;
    hdr[t] = H;
    aux[t] = X;
}

// Which primes a launch holds: all at or above FP_BOUND, all below, or (batch
// rounds) both.
enum Kind { INT_PRIMES = 0, FP_PRIMES = 1, ANY_PRIMES = 2 };

// Kernel 1.  Single job: primes[first, first+count) into records [0, count).
// Batch (BATCH): the primes of every range as one index space (prefix: prefix
// sums of the ranges' prime counts); prime i of range r is record r*rcap + i,
// with its job's sequences.  rec_of[i] keeps that record index, so kernels 2
// and 3 need no search over the prefix sums.
template <int KIND>
__device__ __forceinline__ void setup_prime_any(const JobDev *__restrict__ job, u64 p, u32 t, u32 jb,
                                                PrimeHdr *__restrict__ hdr, PrimeAux *__restrict__ aux)
{
    if (KIND == FP_PRIMES || (KIND == ANY_PRIMES && p < FP_BOUND)) setup_prime_one<true>(job, p, t, jb, hdr, aux);
    else setup_prime_one<false>(job, p, t, jb, hdr, aux);
}
template <int KIND>
__global__ void __launch_bounds__(128, 8) k_setup_prime(const JobDev *__restrict__ jobs, const u64 *__restrict__ primes,
                                                     u32 first, u32 count, PrimeHdr *__restrict__ hdr,
                                                     PrimeAux *__restrict__ aux,
                                                     const BatchRange *__restrict__ ranges,
                                                     const u32 *__restrict__ prefix, u32 nr, u32 rcap,
                                                     u32 *__restrict__ rec_of)
{
    const u32 stride = gridDim.x * blockDim.x;
    if constexpr (KIND == ANY_PRIMES) {
        const u32 total = prefix[nr];
        for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
            const u32 r = prefix_find(prefix, nr, i);
            const u32 rec = r * rcap + (i - prefix[r]);
            const u32 jb = ranges[r].job;
            rec_of[i] = rec;
            setup_prime_any<KIND>(jobs + jb, primes[rec], rec, jb, hdr, aux);
        }
    } else {
        for (u32 t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += stride)
            setup_prime_any<KIND>(jobs, primes[first + t], t, 0, hdr, aux);
    }
}

// A batch's BSGS group of prime p of a job of geometry gm.
__device__ __forceinline__ u32 list_group(const JobGeom &gm, u64 p)
{
    return gm.group + (p < FP_BOUND ? 2u : (p >> 63) ? 0u : 1u);
}

// Class for a prime with nk targets of Le giant-step units each: the c among
// gm.classes that minimises 1.5 Q' + nk*ceil(Le/Q') with Q' = 512 << c, baby
// steps, the work of the 32 << c threads that does not depend on their steps
// (clearing the filter, start values; about eight steps each) and giant steps.
// Where solutions are many (`claims` of them expected, as ord(s) divides E), each
// also costs a group's 32 << c threads a claim, about 16 steps' time, and with Q' < E
// an exact check as well, 64; with Q' >= E ord(s) is found among the baby steps and
// there are no giant steps.  (By giant steps alone, 100 sequences, n-range 6*10^6:
// p from 100 to 1000 75 ms, now 13; from 10^6 to 2*10^6 10.2, now 7.8.)
template <bool CLAIMS>
__device__ __forceinline__ u32 best_class(const JobGeom &gm, u32 nk, u32 Le, u64 E, float claims)
{
    u32 best_c = 0;
    float best = 3.0e38f;
#pragma unroll
    for (u32 c = 0; c < NCLASS; ++c) {
        const u32 lq = 9 + c;
        const u32 mg = ((Le - 1) >> lq) + 1;
        float cost = (float)nk * (float)mg;
        if (CLAIMS) cost = E > (1u << lq) ? cost + 64.0f * claims / (float)(1u << c) : 16.0f * claims / (float)(1u << c);
        cost += 1.5f * (float)(1u << lq);
        if (((gm.classes >> c) & 1u) && cost < best) { best = cost; best_c = c; }
    }
    return best_c;
}
__device__ __noinline__ u32 class_of_many(const JobGeom gm, u32 nk, u32 Le, u64 E)
{
    return best_class<true>(gm, nk, Le, E, (float)nk * (float)Le / (float)E);
}
__device__ __forceinline__ u32 choose_class(const JobGeom &gm, u32 nk, u32 Le, u64 E)
{
    return (u64)nk * Le < E ? best_class<false>(gm, nk, Le, E, 0.0f) : class_of_many(gm, nk, Le, E);
}

// a[r] = x[r]^ex for r < R, the chains interleaved.  UNIFORM: ex (>= 1) is the
// same for every lane, so the loop branches on it: by two-bit digits, 1.375 products
// per bit, or for integers, whose products cost more than the loop, by a sliding
// window of two bits, 1.33.  Else as power().
template <bool FP, int R, bool UNIFORM, bool LAZY>
__device__ __forceinline__ void power_chains_as(const Field<FP> &F, typename Field<FP>::V (&a)[2],
                                                const typename Field<FP>::V (&x)[2], u64 ex)
{
    typedef typename Field<FP>::V V;
    V x2[2], x3[2];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        x2[r] = F.template psqr<LAZY>(x[r]);
        x3[r] = F.template pmul<LAZY>(x2[r], x[r]);
    }
    if constexpr (UNIFORM && FP) {
        // the exponent's digits from the top, two bits each, at the top of t
        const u32 n = (65 - __clzll(ex)) >> 1;             // digits
        u64 t = ex << (64 - 2 * n);
        u32 d = (u32)(t >> 62);                            // 1..3
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = d == 1 ? x[r] : d == 2 ? x2[r] : x3[r];
#pragma unroll 1
        for (u32 i = 1; i < n; ++i) {
            t <<= 2;
            d = (u32)(t >> 62);
#pragma unroll
            for (int r = 0; r < R; ++r) a[r] = F.template psqr<LAZY>(a[r]);
#pragma unroll
            for (int r = 0; r < R; ++r) a[r] = F.template psqr<LAZY>(a[r]);
            if (d & 1) {
                if (d & 2) {
#pragma unroll
                    for (int r = 0; r < R; ++r) a[r] = F.template pmul<LAZY>(a[r], x3[r]);
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) a[r] = F.template pmul<LAZY>(a[r], x[r]);
                }
            } else if (d) {
#pragma unroll
                for (int r = 0; r < R; ++r) a[r] = F.template pmul<LAZY>(a[r], x2[r]);
            }
        }
    } else if constexpr (UNIFORM) {
        int i = 63 - __clzll(ex);
        const bool two = i > 0 && ((ex >> (i - 1)) & 1);
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = two ? x3[r] : x[r];
        i -= two ? 2 : 1;
        while (i >= 0) {
#pragma unroll
            for (int r = 0; r < R; ++r) a[r] = F.template psqr<LAZY>(a[r]);
            if ((ex >> i) & 1) {
                if (i > 0 && ((ex >> (i - 1)) & 1)) {
                    --i;
#pragma unroll
                    for (int r = 0; r < R; ++r) a[r] = F.template pmul<LAZY>(F.template psqr<LAZY>(a[r]), x3[r]);
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) a[r] = F.template pmul<LAZY>(a[r], x[r]);
                }
            }
            --i;
        }
    } else {
        const V one = F.one();
        int i = (63 - __clzll(ex)) & ~1;
        auto digit = [&](int r) -> V {
            const u32 d = (u32)(ex >> i) & 3u;
            const V lo = (d & 1) ? x[r] : one, hi = (d & 1) ? x3[r] : x2[r];
            return (d & 2) ? hi : lo;
        };
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = digit(r);
        for (i -= 2; i >= 0; i -= 2) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                a[r] = F.template pmul<LAZY>(F.template psqr<LAZY>(F.template psqr<LAZY>(a[r])), digit(r));
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) a[r] = F.template pend<LAZY>(a[r]);
}
// (Two chains per lane: four would not fit 64 registers.  Issue and the FP64 pipe
// bound the FP64 form: 100 sequences near 2^50, a launch of 30000 primes, take 5.1 ns
// per prime at 71% issue, FP64 62% busy (4.7 in launches of 120000); 7.8 with an exponentiation per sequence to D alone, a second one
// for the rest of the order, and Montgomery conversions around both.)
template <bool FP, int R, bool UNIFORM>
__device__ __forceinline__ void power_chains(const Field<FP> &F, typename Field<FP>::V (&a)[2],
                                             const typename Field<FP>::V (&x)[2], u64 ex)
{
    if (FP || F.lazy) power_chains_as<FP, R, UNIFORM, true>(F, a, x, ex);
    else power_chains_as<FP, R, UNIFORM, false>(F, a, x, ex);
}

// Shared memory of a sub-warp of GL lanes in kernel 2: the values h^(-r), r <
// min(e, TAB) (all of them for GL = 32; the others look a class up in several turns,
// which with 64 entries cost GL = 32 a third of the kernel), the class lookup over
// them (open addressing, r + 1 in a 16-bit slot, 0: empty), powers of b, and the
// targets' parts until the baby-step count is known.
template <u32 GL>
struct KScratch {
    static constexpr u32 KM = GL == 32 ? 128 : GL;       // sequences
    static constexpr u32 TAB = GL == 4 ? 32 : GL < 32 ? 64 : SPLIT_MAX, CLS_SLOTS = GL < 32 ? 2 * TAB : 4 * TAB;
    u64 hv[TAB];
    u64 part[KM];
    u64 b1[GL == 32 ? 32 : 1], b2[GL == 32 ? 16 : 1];
    alignas(16) unsigned short slot[CLS_SLOTS];
    unsigned short meta[KM];
};

__device__ __forceinline__ u32 cls_hash(u64 v, u32 mask)
{
    return ((((u32)v ^ (u32)(v >> 32)) * 0x9E3779B1u) >> 20) & mask;
}

// The powers of four primes' last sequences together.  With K = 32R + m sequences,
// 0 < m <= REST_MAX, a warp's last round of lanes would leave 32 - m of them idle
// (for odd R it runs beside another round, as the second chain of its lanes, where
// it costs little: shares_rest says no);
// here m8 = 8*ceil(m/8) lanes take a prime's m sequences, so that m8/8 rounds serve
// four primes (each lane its own exponent, 1.5 products per bit against 1.375).
// z = k^E goes to the target row of its record until setup_k_one takes it up.
// Records rec[0..3] (rec[q] valid for q < n), all of one job and step kind.  Called
// by the whole warp.
// Measured: 68 sequences near 2^50.6 4.15 -> 3.62 ns per prime, 20 below 2^64 6.44 ->
// 6.00; 100 (R = 3) 4.76 -> 4.83.
constexpr u32 REST_MAX = 24;
__host__ __device__ __forceinline__ bool shares_rest(u32 kcount)
{
    const u32 m = kcount & 31;
    return m != 0 && m <= REST_MAX && ((kcount >> 5) & 1) == 0;
}
template <bool FP>
__device__ __forceinline__ void rest_powers(const JobDev *__restrict__ job, u32 rec, u32 n, const PrimeHdr *hdr,
                                            const PrimeAux *aux, u64 *tgt)
{
    typedef Field<FP> F;
    const u32 lane = threadIdx.x & 31, m = job->kcount & 31, base = job->kcount - m, m8 = (m + 7) & ~7u;
    const u32 alive = __ballot_sync(0xFFFFFFFFu, lane < n && hdr[rec].p != 0);
    if (!alive) return;
    const u32 any = __ffs((int)alive) - 1;
#pragma unroll 1
    for (u32 c = lane; c < 4 * m8; c += 32) {              // (4*m8 is a multiple of 32: the warp stays whole)
        const u32 q = c / m8, j = c - q * m8;
        // (lane q holds rec[q]; a lane without work repeats the first live prime's)
        const u32 w = __shfl_sync(0xFFFFFFFFu, rec, q), w0 = __shfl_sync(0xFFFFFFFFu, rec, any);
        const bool ok = j < m && q < n && hdr[w].p != 0;
        const u32 wv = ok ? w : w0;
        const F f(hdr[wv], aux[wv]);
        const u64 p = hdr[wv].p, kv = job->k[base + (j < m ? j : 0)];
        const u64 z = F::bits(power<FP>(f, f.of_int((kv < p) ? kv : kv % p), ok ? aux[wv].E : 1));
        if (ok) tgt[(size_t)wv * KSTRIDE + j] = z;
    }
    __syncwarp();
}

// Sequence classes, targets and baby-step count of record w, by GL lanes (lane l
// of them) of a warp; live: the record exists and is not skipped.  GL = 32: up to
// 128 sequences, four rounds of lanes (rest: the last, partial round's powers are in
// the record's target row); GL < 32: at most GL sequences, 32/GL primes side by side
// in a warp.  Called by the whole warp.  Returns the prime's class, or NCLASS when it
// is skipped.
template <bool FP, u32 GL>
__device__ __forceinline__ u32 setup_k_one(const JobDev *__restrict__ job, u32 w, u32 l, bool live,
                                            PrimeHdr *__restrict__ hdr, const PrimeAux *__restrict__ aux,
                                            u64 *tgt, unsigned short *__restrict__ meta,
                                            u64 *__restrict__ stats, const JobGeom &gm, bool rest, KScratch<GL> &sc)
{
    typedef Field<FP> F;
    typedef typename F::V V;
    const u32 lane = threadIdx.x & 31;
    const u32 sub = lane & ~(GL - 1);                      // the sub-warp's first lane
    const u32 gmask = GL == 32 ? 0xFFFFFFFFu : ((1u << (GL & 31)) - 1u) << sub;
    const PrimeAux &X = aux[w];
    const F f(hdr[w], X);
    // (without a live record only the loops' ends matter: a skipped one has no X)
    const u64 p = live ? hdr[w].p : ~0ull, E = live ? X.E : 1;
    const u32 K = job->kcount, e = live ? hdr[w].e : 1;
    // class table: lane l forms h^(-l) by a multiplicative scan over the GL lanes,
    // then every GL-th value from there by products with h^(-GL)
    constexpr u32 TAB = KScratch<GL>::TAB, CLS_SLOTS = KScratch<GL>::CLS_SLOTS;
    const u32 ne = min(e, TAB);
    // (four slots or more per entry for a whole warp's prime: the warp inserts in as
    // many turns as its slowest lane; a power of two, at least 64)
    const u32 nslot = GL < 32 ? CLS_SLOTS : max(64u, 1u << (34 - __clz(ne - 1 | 15)));
    const u32 smask = nslot - 1;
    V hT = f.one();                                        // h^(-TAB), for e > TAB
    __syncwarp();                                          // the previous prime's readers are done
    for (u32 i = l; i < nslot / 8; i += GL) reinterpret_cast<uint4 *>(sc.slot)[i] = make_uint4(0u, 0u, 0u, 0u);
    {
        const V hm1 = F::val(X.hm1);
        V hv = (l == 0) ? f.one() : hm1;
#pragma unroll 1
        for (u32 o = 1; o < GL; o <<= 1) {
            const V hu = F::val(__shfl_up_sync(0xFFFFFFFFu, F::bits(hv), o, GL));
            const V m = f.mul(hv, hu);
            hv = (l >= o) ? m : hv;
        }
        const V hG = f.mul(F::val(__shfl_sync(0xFFFFFFFFu, F::bits(hv), GL - 1, GL)), hm1);
        if constexpr (SPLIT_MAX > TAB) {
            hT = hG;
#pragma unroll 1
            for (u32 n = GL; n < TAB; n *= 2) hT = f.mul(hT, hT);
        }
        __syncwarp();
        // (sub-warps of different e stay together: every lane loops until the last is done)
        for (u32 r = l; __any_sync(0xFFFFFFFFu, live && r < ne); r += GL) {
            const u64 v = F::bits(hv);
            bool pend = live && r < ne;
            if (pend) sc.hv[r] = v;
            u32 s = cls_hash(v, smask);
            while (__any_sync(0xFFFFFFFFu, pend)) {
                if (pend && sc.slot[s] == 0) sc.slot[s] = (unsigned short)(r + 1);
                __syncwarp();
                if (pend) {
                    if (sc.slot[s] == r + 1) pend = false;
                    else s = (s + 1) & smask;
                }
                __syncwarp();
            }
            hv = f.mul(hv, hG);
        }
    }
    if constexpr (GL == 32) {                              // b^l, and b^(32 j) for e > 32
        const V b1 = F::val(X.b);
        V bv = (lane == 0) ? f.one() : b1;
#pragma unroll 1
        for (u32 o = 1; o < 32; o <<= 1) {
            const V bu = F::val(__shfl_up_sync(0xFFFFFFFFu, F::bits(bv), o));
            const V m = f.mul(bv, bu);
            bv = (lane >= o) ? m : bv;
        }
        sc.b1[lane] = F::bits(bv);
        if (e > 32) {
            const V b32 = f.mul(F::val(__shfl_sync(0xFFFFFFFFu, F::bits(bv), 31)), b1);
            V v = (lane == 0) ? f.one() : b32;
#pragma unroll 1
            for (u32 o = 1; o < SPLIT_MAX / 32; o <<= 1) {
                const V u = F::val(__shfl_up_sync(0xFFFFFFFFu, F::bits(v), o));
                const V m = f.mul(v, u);
                v = (lane >= o) ? m : v;
            }
            if (lane < SPLIT_MAX / 32) sc.b2[lane] = F::bits(v);
        }
    }
    __syncwarp();
    // z = k^E of every sequence, two rounds of lanes at a time, and its class: n == r
    // (mod e) where z * h^r == (-c)^E, i.e. h^(-r) == z or, for c = +1 and odd E,
    // == p - z (z is a unit); no such r: no term is divisible.  r is looked up as
    // r0 - TAB*j: z * h^(-TAB*j) == h^(-r0).  A kept sequence's k * b^off
    // (negated for c = +1) and meta are compacted.
    const u32 nmod = job->nmin % e;
    u32 nk = 0;
    bool divk = false;
    auto classify = [&](u32 i, u64 kr, V z) {
        bool keep = false;
        u32 off = 0;
        V u = z;
        if (live && i < K) {
            if (kr == 0) {
                divk = true;
            } else {
                const bool plus = job->c[i] == 1;
                V y = (plus && (E & 1)) ? f.neg(z) : z;
                u32 r0 = 0;
                for (u32 j = 0; j < e && !keep; j += TAB) {
                    const u64 v = F::bits(y);
                    u32 s = cls_hash(v, smask);
                    while ((r0 = sc.slot[s]) != 0) {
                        if (sc.hv[r0 - 1] == v) {
                            keep = true;
                            off = r0 - 1 + e - nmod;       // (GL = 32: j = 0)
                            if constexpr (GL < 32) off = (off + e - j) % e;
                            else if (off >= e) off -= e;
                            break;
                        }
                        s = (s + 1) & smask;
                    }
                    if (SPLIT_MAX > TAB && !keep) y = f.mul(y, hT);
                }
                if (keep) {
                    u = f.of_int(kr);
                    if constexpr (GL == 32) {
                        u = f.mul(u, F::val(sc.b1[off & 31]));
                        if (off >= 32) u = f.mul(u, F::val(sc.b2[off >> 5]));
                    }
                    if (plus) u = f.neg(u);
                }
            }
        }
        if constexpr (GL < 32) {
            const V bo = power<FP>(f, F::val(X.b), off);
            if (keep) u = f.mul(u, bo);
        }
        const u32 km = __ballot_sync(0xFFFFFFFFu, keep) & gmask;
        if (keep) {
            const u32 pos = nk + __popc(km & ((1u << lane) - 1));
            sc.part[pos] = F::bits(u);
            sc.meta[pos] = (unsigned short)(i | (off << 7));
        }
        nk += __popc(km);
    };
    if constexpr (GL == 32) {
        const u32 R = rest ? K / 32 : (K + 31) / 32;
#pragma unroll 1
        for (u32 r0 = 0; r0 < R; r0 += 2) {
            V x[2], z[2];
            u64 kr[2];
#pragma unroll
            for (u32 h = 0; h < 2; ++h) {
                const u32 i = lane + 32 * (r0 + h);
                const u64 kv = (i < K) ? job->k[i] : 1;
                kr[h] = (kv < p) ? kv : kv % p;
                x[h] = f.of_int(kr[h]);
            }
            if (r0 + 1 < R) {
                power_chains<FP, 2, true>(f, z, x, E);
#pragma unroll 1
                for (u32 h = 0; h < 2; ++h) classify(lane + 32 * (r0 + h), h ? kr[1] : kr[0], h ? z[1] : z[0]);
            } else {
                power_chains<FP, 1, true>(f, z, x, E);
                classify(lane + 32 * r0, kr[0], z[0]);
            }
        }
        if (rest) {
            const u32 i = lane + 32 * R;
            const u64 kv = (i < K) ? job->k[i] : 1;
            classify(i, (kv < p) ? kv : kv % p, (i < K) ? F::val(tgt[(size_t)w * KSTRIDE + lane]) : f.one());
        }
    } else {
        const u64 kv = (l < K) ? job->k[l] : 1;
        const u64 kr = (kv < p) ? kv : kv % p;
        V x[2] = {f.of_int(kr), f.one()}, z[2];
        power_chains<FP, 1, false>(f, z, x, E);
        classify(l, kr, z[0]);
    }
    divk = (__ballot_sync(0xFFFFFFFFu, divk) & gmask) != 0;
    const bool skip = divk || nk == 0;
    if (live && skip && l == 0) {
        hdr[w].p = 0;
        atomicAdd(&stats[ST_SKIPPED], 1ull);
    }
    __syncwarp();                                          // the compacted parts are written
    if (!live || skip) return NCLASS;
    // baby steps for this prime (the giant-step tables follow in kernel 3), and the
    // targets T = -c * k * b^(nmin + off + e(Q'-1))
    const u32 cls = choose_class(gm, nk, (job->L - 1) / e + 1, E);
    const V wr0 = F::val(X.wr0[cls]);
    for (u32 j = l; j < nk; j += GL) {
        tgt[(size_t)w * KSTRIDE + j] = F::bits(f.mul(F::val(sc.part[j]), wr0));
        meta[(size_t)w * KSTRIDE + j] = sc.meta[j];
    }
    if (l == 0) {
        hdr[w].numk = nk;
        hdr[w].cls = cls;
    }
    return cls;
}

// Giant phase of nk targets with Mg giant steps each, over a group of gs
// threads: items of G chunks of Lc = ceil(Mg/G) steps per target, a round of
// 2 gs items at a time, `rounds` rounds per segment.  With h half rounds (one
// item per thread) G = gs*h/nk; of h = 1..8 the one with the least h * (Lc + 3),
// an odd h counting half a round more (an item's start values cost about three
// steps, and an odd half round runs one chain per thread instead of two).  A
// segment is checked for filter passes at its end: the filter passes one value
// in 2000 that is not there, and Q'/E of all values are there (they and the s^j lie
// in the group of order E, PrimeAux), so a segment of `run` steps per chain (48
// unless E is small) fills at most a quarter of the queue, GS/8 passes (with Q'/p
// for the share that is there, queues overflowed up to p of 10^8: 100 sequences,
// n-range 6*10^6, p from 2*10^6 to 8*10^6, 124 ns per prime, now 65); longer giant
// phases are cut into chunks and segments of that length.  G is at most 1024 (the
// start tables), and a target's last chunk is never empty.  A chunk that is longer all
// the same (Mg above 1024 times the length) is walked in several segments, `piece`
// steps of one round's chunks in each: one sequence, n-range 2^32, Q' = 1024 near 2^47
// took 339 us per prime with segments of whole chunks, every queue overflowing.
__device__ __forceinline__ void giant_split(u32 gs, u32 nk, u32 Mg, float E, u32 &G, u32 &Lc, u32 &nseg, u32 &rounds,
                                            u32 &piece)
{
    const float fill = fmaxf(1.0f, 1.0f / (16.0f * (5.0e-4f + 16.0f * (float)gs / E)));
    const u32 run = (u32)fminf(48.0f, fill);
    u32 best = 0xFFFFFFFFu, hb = 0;
    for (u32 h = 1; h <= 8; ++h) {
        u32 g = gs * h / nk;
        if (g < 1) continue;
        g = min(min(g, Mg), 1024u);
        const u32 lc = (Mg + g - 1) / g, cost = (2 * h + (h & 1)) * (lc + 3);
        if (cost < best) {
            best = cost;
            hb = h;
            Lc = lc;
        }
        if (g == Mg) break;                               // one step per item already
    }
    if (((hb + 1) >> 1) * Lc > run) Lc = (Mg + min((Mg + run - 1) / run, 1024u) - 1) / min((Mg + run - 1) / run, 1024u);
    G = (Mg + Lc - 1) / Lc;
    const u32 total = (nk * G + 2 * gs - 1) / (2 * gs);   // rounds
    rounds = min(total, max(run / Lc, 1u));
    nseg = (total + rounds - 1) / rounds;
    // (a round of half the items leaves twice the room)
    const u32 most = (u32)(nk * G <= gs ? 2.0f * fill : fill), pieces = (Lc + most - 1) / most;
    piece = (Lc + pieces - 1) / pieces;
    nseg *= (Lc + piece - 1) / piece;                     // (1 for more rounds than one: then 2*Lc <= run)
}

// Baby- and giant-step tables of record t (one thread): giant steps per target
// Mg = ceil(ceil(L/e)/Q'), G chunks of Lc steps per target, A[l] = s^(16l),
// B[l] = s^(512l) (baby starts), Z1[l] = S^(Lc*l), Z2[l] = S^(32*Lc*l) (giant
// starts) with S = s^Q', and the multipliers' quotients, in the form of the
// prime's step kind (PrimeHdr).  Adds the prime's targets and its search kind
// to the thread's tallies.  Each table is only as long as the BSGS kernel
// reads it: A[t % 32] and B[t / 32] for the group's threads t, Z1[g % 32] and
// Z2[g / 32] for the giant chunks g < G.
template <bool FP>
__device__ __forceinline__ void setup_tabs_one(const JobDev *__restrict__ job, u32 t, PrimeHdr *__restrict__ hdr,
                                               const PrimeAux *__restrict__ aux, u64 *__restrict__ tabs,
                                               u64 (*tile)[33], bool run, u32 &n_targets, u32 &n_full, u32 &n_split)
{
    const u32 lane = threadIdx.x & 31;
    typedef Field<FP> F;
    typedef typename F::V V;
    PrimeHdr &h = hdr[t];
    const F f(h, aux[t]);
    const u32 e = run ? h.e : 1, nk = run ? h.numk : 1, cls = run ? h.cls : 0, gs = 32u << cls, lq = 9 + cls;
    // (L - 1 and not L + e - 1: an n-range may be 2^32 - 1 long; without run job is not the record's)
    const u32 Le = run ? (job->L - 1) / e + 1 : 1;
    const u32 Mg = ((Le - 1) >> lq) + 1;
    u32 G, Lc, nseg, rounds, piece;
    giant_split(gs, nk, Mg, (float)aux[t].E, G, Lc, nseg, rounds, piece);
    const V s = F::val(h.s), S = F::val(aux[t].S[cls]);          // (not a record's when !run: never stored)
    V u8 = f.mul(s, s);
    u8 = f.mul(u8, u8);
    u8 = f.mul(u8, u8);
    const V u = f.mul(u8, u8), z = power<FP>(f, S, Lc);
    const u32 nb = gs >> 5, nz1 = min(G, 32u), nz2 = (G + 31) >> 5;
    // n powers of x into row `lane` of the warp's tile, then the rows out to the
    // lanes' records at offset o, a row at a time (one thread's own stores would
    // touch a line each); returns x^n (z^32 is needed only when G > 32, and then
    // the Z1 table runs to 32 entries)
    auto table = [&](V x, u32 n, u32 o) -> V {
        if (!run) n = 0;
        V a = f.one();
        for (u32 l = 0; __any_sync(0xFFFFFFFFu, l < n); ++l) {
            if (l >= n) continue;
            tile[lane][l] = F::bits(a);
            a = f.mul(a, x);
        }
        __syncwarp();
#pragma unroll 4
        for (u32 r = 0; r < 32; ++r) {
            const u32 tr = __shfl_sync(0xFFFFFFFFu, t, r), nr = __shfl_sync(0xFFFFFFFFu, n, r);
            if (lane < nr) tabs[(size_t)tr * TABS + o + lane] = tile[r][lane];
        }
        __syncwarp();
        return a;
    };
    const V u32p = table(u, 32, 0);
    const V z32 = table(z, nz1, 64);
    table(u32p, nb, 32);
    table(z32, nz2, 96);
    if (!run) return;
    h.G = G;
    h.Lc = Lc;
    h.Mg = Mg;
    h.rk = 1.0f / (float)nk;
    h.nseg = nseg;
    h.rounds = rounds;
    h.piece = piece;
    h.S = F::bits(S);
    h.u8 = F::bits(u8);
    if constexpr (FP) {
        h.Sw = double_bits(S / f.p);
    } else if (!(f.M.p >> 63)) {                           // Shoup multiplier of the giant steps below 2^63
        h.Sp = from_mont(S, f.M);
        h.Sw = shoup_of_mont(S, f.M.q);
    }
    n_targets += nk;
    if (e >= 2) ++n_split; else ++n_full;
}

// Kernel 3: one thread per prime (indexing as kernel 1); then the record's index
// goes on the list of its class (ANY_PRIMES: of its job's group and step kind, with the
// lists' starts from kernel 2's counts).
template <int KIND>
__global__ void __launch_bounds__(128, 8) k_setup_tabs(const JobDev *__restrict__ jobs, PrimeHdr *__restrict__ hdr,
                                                    const PrimeAux *__restrict__ aux, u32 count,
                                                    u64 *__restrict__ tabs, u64 *__restrict__ stats,
                                                    u32 *__restrict__ lists, u32 list_stride, u32 *list_ctl,
                                                    const JobGeom *__restrict__ geoms,
                                                    const u32 *__restrict__ prefix, u32 nr,
                                                    const u32 *__restrict__ rec_of)
{
    constexpr bool BATCH = KIND == ANY_PRIMES;
    const u32 stride = gridDim.x * blockDim.x;
    const u32 lane = threadIdx.x & 31;
    const u32 total = BATCH ? prefix[nr] : count;
    __shared__ u64 s_tile[128 / 32][32][33];
    u64 (*tile)[33] = s_tile[threadIdx.x >> 5];
    __shared__ u32 s_first[BATCH ? NGROUP * NCLASS : 1];
    if constexpr (BATCH) {
        const u32 k = threadIdx.x;
        if (k < NGROUP * NCLASS) {
            u32 first = 0;
            for (u32 l = 0; l < k; ++l) first += list_ctl[l / NCLASS * LIST_CTL + 2 * NCLASS + l % NCLASS];
            s_first[k] = first;
            if (blockIdx.x == 0) list_ctl[k / NCLASS * LIST_CTL + 3 * NCLASS + k % NCLASS] = first;
        }
        __syncthreads();
    }
    u32 nt = 0, nf = 0, ns = 0;
    // i0 is uniform over the warp, so that the list claims below stay whole
    for (u32 i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < total; i0 += stride) {
        const u32 i = i0 + lane;
        const u32 rec = (i < total) ? (BATCH ? rec_of[i] : i) : 0;
        const bool live = i < total && hdr[rec].p != 0;
        u32 key = 0xFFFFFFFFu;                             // list of the record: group * NCLASS + class
        const u64 p = hdr[rec].p;
        const u32 jb = BATCH && live ? hdr[rec].job : 0;   // (past the end rec 0 may never have been written)
        const bool fp = KIND == FP_PRIMES || (BATCH && p < FP_BOUND);
        if (KIND != INT_PRIMES && __any_sync(0xFFFFFFFFu, live && fp))
            setup_tabs_one<true>(jobs + jb, rec, hdr, aux, tabs, tile, live && fp, nt, nf, ns);
        if (KIND != FP_PRIMES && __any_sync(0xFFFFFFFFu, live && !fp))
            setup_tabs_one<false>(jobs + jb, rec, hdr, aux, tabs, tile, live && !fp, nt, nf, ns);
        if (live) {
            key = (BATCH ? list_group(geoms[jb], p) : 0u) * NCLASS + hdr[rec].cls;
        }
        const u32 same = __match_any_sync(0xFFFFFFFFu, key);
        const u32 lead = __ffs((int)same) - 1;
        u32 base = 0;
        if (live && lane == lead) base = atomicAdd(&list_ctl[key / NCLASS * LIST_CTL + key % NCLASS], __popc(same));
        base = __shfl_sync(0xFFFFFFFFu, base, lead);
        if (live) lists[(BATCH ? s_first[key] : key * list_stride) + base + __popc(same & ((1u << lane) - 1))] = rec;
    }
    // one atomic per warp and counter
    nt = __reduce_add_sync(0xFFFFFFFFu, nt);
    nf = __reduce_add_sync(0xFFFFFFFFu, nf);
    ns = __reduce_add_sync(0xFFFFFFFFu, ns);
    if (lane == 0) {
        if (nt) atomicAdd(&stats[ST_TARGETS], (u64)nt);
        if (nf) atomicAdd(&stats[ST_FULL], (u64)nf);
        if (ns) atomicAdd(&stats[ST_PARITY], (u64)ns);
    }
}


// Kernel 2: GL lanes per prime.  KIND as kernel 1.  BATCH: the primes of KIND of a
// batch round, GL = 32 (one launch per kind: with both in one kernel its registers
// spilled: 11.9 against 10.2 ms on twelve jobs).
template <int KIND, u32 GL, bool BATCH = false>
__global__ void __launch_bounds__(SETUP_TPB, 4) k_setup_k(const JobDev *__restrict__ jobs, PrimeHdr *__restrict__ hdr,
                                                       const PrimeAux *__restrict__ aux, u32 count, bool four,
                                                       u64 *tgt, unsigned short *__restrict__ meta,
                                                       u64 *__restrict__ stats, JobGeom gm,
                                                       const JobGeom *__restrict__ geoms,
                                                       const u32 *__restrict__ prefix, u32 nr,
                                                       const u32 *__restrict__ rec_of, u32 *list_ctl)
{
    __shared__ KScratch<GL> s_sc[SETUP_TPB / GL];
    const u32 l = threadIdx.x & (GL - 1);
    KScratch<GL> &sc = s_sc[threadIdx.x / GL];
    const u32 stride = gridDim.x * (SETUP_TPB / GL);
    u32 i = (blockIdx.x * SETUP_TPB + threadIdx.x) / GL;
    if constexpr (GL == 32) {
        // four consecutive primes per warp when the sequences leave a partial round
        // that they can share, else one.  A round of a batch only knows its primes here:
        // four as in launch_setup_kind when every warp of the grid then still has some
        // (100 sequences near 2^58, a round of 430 primes: 354 us with four at any
        // size, 283 with one).
        static_assert(KIND != ANY_PRIMES, "a warp holds primes of one step kind");
        const u32 total = BATCH ? prefix[nr] : count;
        const u32 per = four && (!BATCH || total >= 4 * stride) ? 4 : 1;
        for (i *= per; i < total; i += stride * per) {
            const u32 n = min(per, total - i);
            // lane q: prime q (mine: of this launch's kind; a skipped one, p = 0, counts
            // as FP)
            u32 rec = 0, jb = 0;
            bool mine = false, rest = false;
            if (l < n) {
                rec = BATCH ? rec_of[i + l] : i + l;
                if (BATCH) jb = hdr[rec].job;
                mine = !BATCH || (hdr[rec].p < FP_BOUND) == (KIND == FP_PRIMES);
            }
            const u32 todo = __ballot_sync(0xFFFFFFFFu, mine);
            if (per == 4 && todo) {
                const u32 j0 = __shfl_sync(0xFFFFFFFFu, jb, 0);
                rest = shares_rest(jobs[j0].kcount) && __all_sync(0xFFFFFFFFu, l >= n || (mine && jb == j0));
                if (rest) rest_powers<KIND == FP_PRIMES>(jobs + j0, rec, n, hdr, aux, tgt);
            }
#pragma unroll 1
            for (u32 t = todo; t; t &= t - 1) {
                const u32 q = __ffs((int)t) - 1;
                const u32 w = __shfl_sync(0xFFFFFFFFu, rec, q), j = __shfl_sync(0xFFFFFFFFu, jb, q);
                if (hdr[w].p == 0) {
                    if (l == 0) atomicAdd(&stats[ST_SKIPPED], 1ull);
                    continue;
                }
                const u32 cls = setup_k_one<KIND == FP_PRIMES, GL>(jobs + j, w, l, true, hdr, aux, tgt, meta, stats,
                                                                   BATCH ? geoms[j] : gm, rest, sc);
                if (BATCH && l == 0 && cls < NCLASS)       // the length of the list that kernel 3 puts it on
                    atomicAdd(&list_ctl[list_group(geoms[j], hdr[w].p) * LIST_CTL + 2 * NCLASS + cls], 1u);
            }
        }
    } else {
        // (the warp stays until the last of its sub-warps' primes is done)
        for (; __any_sync(0xFFFFFFFFu, i < count); i += stride) {
            const bool in = i < count;
            const bool live = in && hdr[i].p != 0;
            if (in && !live && l == 0) atomicAdd(&stats[ST_SKIPPED], 1ull);
            if (!__any_sync(0xFFFFFFFFu, live)) continue;
            setup_k_one<KIND == FP_PRIMES, GL>(jobs, in ? i : 0, l, live, hdr, aux, tgt, meta, stats, gm, false, sc);
        }
    }
}

template <int KIND>
static cudaError_t launch_setup_kind(const JobDev *job, u32 kcount, const u64 *primes, u32 first, u32 count,
                                     PrimeHdr *hdr, PrimeAux *aux, u64 *tabs, u64 *tgt, unsigned short *meta,
                                     const BsgsLists &lists, u64 *stats, const JobGeom &gm, int sms, cudaStream_t st)
{
    k_setup_prime<KIND><<<(count + 127) / 128, 128, 0, st>>>(job, primes, first, count, hdr, aux, nullptr, nullptr, 0, 0,
                                                             nullptr);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    auto go = [&](auto gl) {
        constexpr u32 GL = decltype(gl)::value;
        // four primes share a partial round of lanes when there are enough of them to
        // fill the chip all the same (4 CTAs of 8 warps per SM)
        const bool four = GL == 32 && shares_rest(kcount) && count >= 4u * 4 * 8 * (u32)sms;
        const u32 ppb = SETUP_TPB / GL * (four ? 4 : 1);   // primes per block
        k_setup_k<KIND, GL><<<(count + ppb - 1) / ppb, SETUP_TPB, 0, st>>>(job, hdr, aux, count, four, tgt, meta, stats,
                                                                          gm, nullptr, nullptr, 0, nullptr, nullptr);
    };
    if (kcount <= 4) go(std::integral_constant<u32, 4>{});
    else if (kcount <= 8) go(std::integral_constant<u32, 8>{});
    else if (kcount <= 16) go(std::integral_constant<u32, 16>{});
    else go(std::integral_constant<u32, 32>{});
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_setup_tabs<KIND><<<(count + 127) / 128, 128, 0, st>>>(job, hdr, aux, count, tabs, stats, lists.list, lists.stride,
                                                            lists.ctl, nullptr, nullptr, 0, nullptr);
    return cudaGetLastError();
}

cudaError_t launch_setup(const JobDev *job, u32 kcount, const u64 *primes, u32 first, u32 count, u64 pmax, PrimeHdr *hdr,
                         void *aux, u64 *tabs, u64 *tgt, unsigned short *meta, const BsgsLists &lists, u64 *stats,
                         int geom, int sms, cudaStream_t st)
{
    if (count == 0) return cudaSuccess;
    const JobGeom gm = job_geom(geom);
    PrimeAux *x = (PrimeAux *)aux;
    return pmax <= FP_BOUND
               ? launch_setup_kind<FP_PRIMES>(job, kcount, primes, first, count, hdr, x, tabs, tgt, meta, lists, stats, gm, sms,
                                            st)
               : launch_setup_kind<INT_PRIMES>(job, kcount, primes, first, count, hdr, x, tabs, tgt, meta, lists, stats, gm, sms,
                                            st);
}

cudaError_t launch_setup_batch(const JobDev *jobs, const JobGeom *geoms, const BatchRange *ranges, const u64 *primes,
                               u32 rcap, const u32 *prefix_p, u32 nranges, PrimeHdr *hdr, void *aux, u64 *tabs,
                               u64 *tgt, unsigned short *meta, const BsgsLists &lists, u64 *stats, u32 *rec_of, int sms,
                               cudaStream_t st)
{
    JobGeom gm{};
    // full-device grids; the kernels stride over the primes of every range
    k_setup_prime<ANY_PRIMES><<<sms * 8, 128, 0, st>>>(jobs, primes, 0, 0, hdr, (PrimeAux *)aux, ranges, prefix_p, nranges,
                                                       rcap, rec_of);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // FP_PRIMES first: it also takes the records without a search from kernel 1 (p = 0 is
    // below FP_BOUND), and the records that the other launch drops must not be among them
    k_setup_k<FP_PRIMES, 32, true><<<sms * 4, SETUP_TPB, 0, st>>>(jobs, hdr, (const PrimeAux *)aux, 0, true, tgt, meta,
                                                                  stats, gm, geoms, prefix_p, nranges, rec_of, lists.ctl);
    k_setup_k<INT_PRIMES, 32, true><<<sms * 4, SETUP_TPB, 0, st>>>(jobs, hdr, (const PrimeAux *)aux, 0, true, tgt, meta,
                                                                   stats, gm, geoms, prefix_p, nranges, rec_of, lists.ctl);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_setup_tabs<ANY_PRIMES><<<sms * 8, 128, 0, st>>>(jobs, hdr, (const PrimeAux *)aux, 0, tabs, stats, lists.list,
                                                      lists.stride, lists.ctl, geoms, prefix_p, nranges, rec_of);
    return cudaGetLastError();
}

}  // namespace rs
