// rs_internal.h -- device data layout shared by the kernels and the engine.
//
// Per job (a set of <= 100 sequences k_i*b^n+c_i sharing b, and an n-range)
// the device holds a JobDev descriptor, the candidate bitmap and a factor
// buffer.  Per segment of the p-range the device holds the generated primes;
// per chunk of primes the setup kernel writes one record per prime (header,
// power tables, BSGS targets) that the BSGS kernel consumes.
#pragma once
#include <cstdint>
#include <vector>
#include <cuda_runtime.h>

namespace rs {

typedef unsigned long long u64;
typedef unsigned int u32;
typedef unsigned char u8;

constexpr int KMAX = 100;            // sequences per job (inputfile.cpp:356-361)
constexpr int KSTRIDE = 112;         // padded per-prime target stride (16-byte multiple for bulk copies)
constexpr int TABS = 128;            // u64 power-table entries per prime

// BSGS classes: a prime of class c is searched by a group of 32 << c threads
// with Q' = 512 << c baby steps.  A geometry bounds the classes that the set-up
// chooses from, per prime, by its maximum q, and fixes the CTAs: 1024 / tpb of
// tpb threads share an SM, each working through the classes.
constexpr int NCLASS = 6;
struct BsgsGeom {
    u32 q, tpb, classes;     // classes: bit c set when class c may be chosen
};
constexpr int NGEOM = 5;
constexpr BsgsGeom BSGS_GEOMS[NGEOM] = {
    {16384, 1024, 0x3D},     // (16 groups of 64 threads would need more than the 15 named barriers)
    {8192, 512, 0x1F},
    {4096, 512, 0x0F},
    {2048, 512, 0x07},
    {1024, 512, 0x03},
};
constexpr int geom_index(u32 q)
{
    return q == 16384 ? 0 : q == 8192 ? 1 : q == 4096 ? 2 : q == 2048 ? 3 : q == 1024 ? 4 : -1;
}

// Model cost of one prime for a geometry, in steps: over primes, the targets
// that survive the prefilter times their giant steps' n-range shrink the work
// kcount*L by D, the part of p-1 made of small primes (as far as the split uses
// it); SPLIT lists ten quantiles of D.  Each prime takes the best class: 1.5 Q'
// (baby steps and the work per thread that does not depend on the job) plus the
// giant steps.
inline double geom_model_cost(int g, u32 kcount, u32 L)
{
    constexpr double SPLIT[10] = {2, 2, 4, 6, 10, 16, 30, 60, 120, 230};
    double sum = 0;
    for (double d : SPLIT) {
        double best = 1e300;
        for (int c = 0; c < NCLASS; ++c) {
            if (!((BSGS_GEOMS[g].classes >> c) & 1)) continue;
            const double q = (double)(512 << c), v = 1.5 * q + (double)kcount * (double)L / (d * q);
            if (v < best) best = v;
        }
        sum += best;
    }
    // (1024-thread CTAs run alone on an SM, so nothing covers their barriers: 12% on
    // the 100-sequence job, 5.6% slower where this cost says 6% faster)
    return sum / 10 * (BSGS_GEOMS[g].tpb == 1024 ? 1.12 : 1.0);
}
inline int geom_model_best(u32 kcount, u32 L)
{
    int best = 0;
    for (int g = 1; g < NGEOM; ++g)
        if (geom_model_cost(g, kcount, L) < geom_model_cost(best, kcount, L)) best = g;
    return best;
}
// Measured geometries per device and job shape (base, kcount, L), shared by the
// single-job contexts and the batches of the process; -1 when none is recorded.
inline u64 job_shape_key(u32 base, u32 kcount, u32 L)
{
    return ((u64)base << 40) ^ ((u64)kcount << 32) ^ (u64)L;
}
int tuned_geom_get(int device, u64 shape);
void tuned_geom_put(int device, u64 shape, int geom);
constexpr int SETUP_TPB = 256;              // 8 warps per block
constexpr int SIEVE_TPB = 512;
constexpr int SIEVE_WORDS = 4096;           // 2^17 odd numbers per sieve block at most
constexpr u64 MR_BOUND = 4295098369ULL;     // 65537^2: below it the sieve by all primes < 2^16 is exact

// error bits (JobDev-independent, one word per context)
constexpr u32 ERR_PRIME_OVERFLOW = 1u;      // segment produced more primes than the buffer holds
constexpr u32 ERR_CAND_OVERFLOW = 2u;
constexpr u32 ERR_FACTOR_OVERFLOW = 8u;     // factor buffer full (cannot happen: sized to the bitmap)
constexpr u32 ERR_TMA_TIMEOUT = 16u;        // a bulk copy did not complete within the wait bound
constexpr u32 ERR_SIEVE_TABLE = 32u;        // the sieving-prime table is missing (does not start with 3)

// statistics counters (u64)
enum Stat {
    ST_PRIMES = 0,        // primes generated (and tested)
    ST_SKIPPED,           // primes dividing b or some k, or with no solvable k (setup.cl:156-162,205-208)
    ST_FULL,              // primes searched over every n (split modulus e = 1)
    ST_PARITY,            // primes searched over one class of n mod e per sequence (e >= 2; e = 2: parity)
    ST_TARGETS,           // sum over primes of surviving k
    ST_BABY,              // baby steps executed
    ST_GIANT,             // giant steps executed (one modular product and one probe each)
    ST_SMALLORDER,        // primes with ord(b^e) < Q
    ST_CANDIDATES,        // filter passes checked exactly
    ST_HITS,              // verified solutions p | k*b^n+c with n in range
    ST_FACTORS,           // bitmap claims won
    ST_DUPS,              // solutions whose bitmap bit was already clear
    ST_SIEVE_CANDS,       // sieve survivors given to Miller-Rabin
    ST_COUNT
};

struct JobDev {
    u32 base, kcount, nmin, nmax;
    u32 L;               // nmax - nmin + 1
    u32 words;           // bitmap words per sequence
    u32 split;           // largest split modulus (split_limit)
    u64 k[KMAX];
    int c[KMAX];
    u32 *bitmap;         // kcount * words
};
// A larger split modulus e means fewer giant steps and a longer class table per
// prime.  With a warp per prime (more than 16 sequences) 256 always pays: 100
// sequences over 6*10^6, 26.0 -> 21.8 ns per prime against 64; 68 over 10^5, 8.5
// -> 8.4.  With 4 to 16 lanes per prime the table weighs more, and small searches keep
// 64: in sequences * n-range both take the same time at 6*10^6 for one sequence, 8*10^6
// for 4, 10^7 for 8 and 1.4*10^7 for 16 (p of 2^40 to 2^63; within 2% for all step
// kinds), at 2*10^6 64 is ahead by 3 to 8%, at 2*10^7 256 by 2 to 7%.
constexpr u32 split_limit(u32 kcount, u32 L)
{
    return kcount > 16 || (u64)kcount * L > 6000000 + 500000 * kcount ? 256u : 64u;
}

// Below FP_BOUND = 2^51 the BSGS steps run on the FP64 pipe (fp_mulfix in
// mont.cuh): residues are exact integers in doubles, and a product by a fixed
// multiplier w takes its quotient from the double w/p.  The set-up's residues and
// products are of the same kind.
constexpr u64 FP_BOUND = 1ull << 51;

// A prime's record header.  Residues are held by step kind: below FP_BOUND each is
// a plain one, as the bits of the double that holds it; from there on residues are
// in Montgomery form unless said otherwise.
struct PrimeHdr {        // 128 bytes (a 16-byte multiple: copied by TMA bulk copies)
    u64 p;               // 0 = skipped
    u64 q;               // p^-1 mod 2^64; below FP_BOUND the bits of 1/p
    u64 one;             // 1
    u64 s;               // b^e, e = the split modulus (n runs over one class mod e per target)
    u64 sw;              // floor(sp*2^64/p), for Shoup's products (0 when p >= 2^63); below FP_BOUND s/p
    u64 sp;              // b^e as a plain integer for FP_BOUND <= p < 2^63, else 0
    u64 S, Sw, Sp;       // the same for s^Q', Q' = this prime's baby-step count
    u64 u8;              // s^8: start offset of a thread's second baby chain
    u32 numk;            // surviving targets
    u32 e;               // split modulus, 1..256
    u32 G, Lc;           // giant phase: G chunks of Lc giant steps per target
    u32 smul;            // 2 or 4 when b^e is (baby steps by doublings), else 0
    u32 job;             // job index within a batch (0 for a single job)
    u32 Mg;              // giant steps per target: ceil(ceil(L/e)/Q')
    u32 cls;             // class: Q' = 512 << cls, 32 << cls threads
    float rk;            // 1/numk
    u32 nseg, rounds;    // segments of a long giant phase: rounds of 2 * (32 << cls) items each
    u32 piece;           // giant steps of a chunk per segment: Lc, or less with a single round
};
static_assert(sizeof(PrimeHdr) == 128, "PrimeHdr is copied in 16-byte units");

struct FactorRec {       // one claimed term: p | k[seq]*b^n + c[seq]
    u64 p;
    u32 n;
    u32 seq;
};

struct BsgsArgs {
    u32 base, nmin, nmax, words;
    u32 *bitmap;
    FactorRec *factors;
    u32 *factor_ctr;
    u32 factor_cap;
    u64 *stats;
    u32 *err;
    u32 wait_bound;      // try_wait rounds before a record copy counts as lost (0: WAIT_BOUND)
    u32 test_stall;      // 1: each CTA's first record wait is on a barrier that nothing completes
};

// ---- batches: many jobs, each with one or more p-ranges, advanced in rounds ----
// A range's window of one round, written on the device by k_batch_windows.
struct BatchWin {
    u64 lo, hi;          // this round's [lo, hi) (lo == hi: the range is done)
    u64 base_odd, nodd;  // odd values base_odd + 2i, i < nodd, covering [lo, hi)
};
struct BatchRange {      // device state of one range slot
    u64 p_cur, p_end;    // next window start, end of the range
    u32 job;             // job slot it belongs to
    u8 active;           // slot in use
    u8 pad_[3];
};
// per-range counters of a round: [0] sieve survivors, [1] primes, [2] pad, [3] pad
constexpr int BR_CTRS = 4;
// per-job BSGS geometry as the set-up kernels need it
struct JobGeom {
    u32 classes;         // classes to choose from (bit c)
    u32 group;           // a batch's BSGS launch of the job's primes: this (0, or 3 for 1024-thread CTAs)
                         // plus the step kind (2 FP64, 1 Shoup, 0 Montgomery)
};
constexpr int NGROUP = 6;
inline JobGeom job_geom(int g)
{
    JobGeom G;
    G.classes = BSGS_GEOMS[g].classes;
    G.group = BSGS_GEOMS[g].tpb == 1024 ? 3u : 0u;
    return G;
}
// One BSGS launch's primes, sorted by class: ctl[c] record indices of class c
// at list + c*stride (a batch's group: at list + ctl[3*NCLASS + c]); ctl[NCLASS + c]
// counts those taken.  A batch's groups share one list, so that it needs one entry per
// record and not one per record, group and class: ctl[2*NCLASS + c] counts the class
// before the list is written, which gives the starts.  All of ctl is zero at the start.
struct BsgsLists {
    u32 *list;
    u32 stride;
    u32 *ctl;
};
constexpr u32 LIST_CTL = 4 * NCLASS;        // u32 of ctl per group
// Set-up scratch of one prime.  Nothing of it is read once the set-up is done, and the
// prime generator's lists are not read once it begins: they share memory.
constexpr size_t SETUP_AUX = 32 + 16 * NCLASS;

// Index i of work spread over nr ranges with prefix sums prefix[0..nr]:
// the range k with prefix[k] <= i < prefix[k+1] (i < prefix[nr]).
__device__ __forceinline__ u32 prefix_find(const u32 *prefix, u32 nr, u32 i)
{
    u32 lo = 0, hi = nr;
    while (hi - lo > 1) {
        const u32 mid = (lo + hi) >> 1;
        if (prefix[mid] <= i) lo = mid; else hi = mid;
    }
    return lo;
}

// launch wrappers (sieve.cu, setup.cu, bsgs.cu)
cudaError_t launch_sieve(u64 base_odd, u64 nodd, const u32 *sp, u32 nsp, u64 *cands, u32 cand_cap, u32 *ctrs, u32 *err,
                         int sms, cudaStream_t st);
// Baillie-PSW in two passes (base 2 into mid, then Lucas over mid); mid holds
// cand_cap values and *mid_ctr starts at zero
cudaError_t launch_mr2(const u64 *cands, const u32 *ctrs, u32 cand_cap, u64 *primes, u32 prime_cap, u32 *prime_ctr,
                       u64 *mid, u32 *mid_ctr, u32 *err, int sms, cudaStream_t st);
// (lists: NCLASS lists of at least count records; the counts in lists.ctl start at
// zero; the primes lie below pmax, entirely on one side of FP_BOUND)
cudaError_t launch_setup(const JobDev *job, u32 kcount, const u64 *primes, u32 first, u32 count, u64 pmax, PrimeHdr *hdr,
                         void *aux, u64 *tabs, u64 *tgt, unsigned short *meta, const BsgsLists &lists, u64 *stats,
                         int geom, int sms, cudaStream_t st);
// every prime of the launch lies in [pmin, pmax), entirely below or entirely at or above 2^63
cudaError_t launch_bsgs(const BsgsArgs &a, const PrimeHdr *hdr, const u64 *tabs, const u64 *tgt,
                        const unsigned short *meta, const BsgsLists &lists, u64 pmin, u64 pmax, int geom, int sms,
                        cudaStream_t st);
size_t bsgs_smem_bytes();     // dynamic shared memory of the largest CTA
cudaError_t bsgs_prepare();   // per device, before the first launch
cudaError_t launch_mulmod_peak(u64 *out, int blocks, int iters, cudaStream_t st);
cudaError_t launch_widemul_peak(u64 *out, int blocks, int iters, cudaStream_t st);
cudaError_t launch_fpmul_peak(u64 *out, int blocks, int iters, cudaStream_t st);

// batch rounds (sieve.cu, setup.cu, bsgs.cu)
// win[r]: primes range slot r should cover this round (0: none); capped at 0.6*rcap
cudaError_t launch_batch_windows(BatchRange *ranges, BatchWin *wins, const u32 *win, u32 nranges, u32 rcap, u32 *ctrs,
                                 cudaStream_t st);
cudaError_t launch_sieve_batch(const BatchWin *wins, u32 nranges, u32 max_blocks, const u32 *sp, u32 nsp, u64 *cands,
                               u32 ccap, u32 *ctrs, u32 *err, cudaStream_t st);
// Baillie-PSW over the survivors of all ranges (prefix_c: their counts'
// prefix sums) in two passes: base-2 strong probable primes of every range
// (value and range) into mid, then the Lucas test over it; primes go to their
// range's slots; *mid_ctr starts at zero
cudaError_t launch_mr_batch2(const u64 *cands, u32 ccap, u64 *primes, u32 rcap, u32 *ctrs, u32 nranges,
                             const u32 *prefix_c, u64 *mid, u32 *mid_r, u32 mid_cap, u32 *mid_ctr, u32 *err, int sms,
                             cudaStream_t st);
// set-up of the primes of all ranges (prefix_p: prefix sums of their counts;
// rec_of and lists.list: room for one record index per prime, nranges * rcap); group
// g's part of lists.ctl starts at LIST_CTL*g
cudaError_t launch_setup_batch(const JobDev *jobs, const JobGeom *geoms, const BatchRange *ranges, const u64 *primes,
                               u32 rcap, const u32 *prefix_p, u32 nranges, PrimeHdr *hdr, void *aux, u64 *tabs,
                               u64 *tgt, unsigned short *meta, const BsgsLists &lists, u64 *stats, u32 *rec_of, int sms,
                               cudaStream_t st);
// prefix over every active range of counter `which` (0: survivors, 1: primes), each capped at cap
cudaError_t launch_batch_prefix_all(const BatchRange *ranges, u32 nr, int which, u32 cap, const u32 *ctrs,
                                    u32 *prefix, cudaStream_t st);
// one launch per group over its own lists
cudaError_t launch_bsgs_batch(const BsgsArgs &a, const BsgsArgs *job_args, const PrimeHdr *hdr, const u64 *tabs,
                              const u64 *tgt, const unsigned short *meta, const BsgsLists &lists, int group, int sms,
                              cudaStream_t st);

}  // namespace rs

// host helpers shared by engine.cu and batch.cu
struct rs_seqs;
std::vector<rs::u32> rs_small_primes();                       // odd primes below 2^16, ascending
void jobdev_from_seqs(const rs_seqs *s, rs::JobDev *out);    // JobDev of a job (bitmap pointer null)
