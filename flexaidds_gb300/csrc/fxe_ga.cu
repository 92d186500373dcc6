// fxe_ga.cu — the GA generation on the device: breeding (roulette selection, crossover,
// mutation on the int32 genes) and replacement, one block per job, for populations kept in HBM.
//
// Semantics follow the reference's operators:
//   * fitness of the population sorted by energy (calculate_fitness, LIB/gaboom.cpp:1627-1760):
//     LINEAR P - i; PSHARE (the reference's default) (P - i) / niche count, the niche count
//     summing 1 - (rmsp / sig_share)^alpha over the chromosomes within sig_share; SMFREE the
//     blend of rank and Boltzmann weight over the same niche count. Under PSHARE the population
//     is walked in fitness order after a generation (LIB/gaboom.cpp:498-499);
//   * roulette_wheel: r = u * sum(fitness), the first index whose running fitness sum exceeds r
//     (LIB/gaboom.cpp:1158-1186);
//   * the reproduce loop (LIB/gaboom.cpp:909-1000): pairs of parents, adaptive probabilities
//     (adapt_prob, :848-880) when asked, crossover with probability crossprob, both children
//     mutated, until nnew children exist;
//   * crossover: the reference's two-point bit crossover over the genes' 32-bit strings, with
//     its choice of genes and bit points, inside genes or at gene boundaries
//     (LIB/gaboom.cpp:2517-2614);
//   * mutate: every bit of every gene flipped with probability mutprob (LIB/gaboom.cpp:2620-2641);
//   * replacement (LIB/gaboom.cpp:1023-1033): BOOM merges parents and children and keeps the best
//     P; STEADY puts the children in place of the worst parents.
// The reference draws from a random_device-seeded generator, so its trajectories cannot be
// replayed; here every draw is a counter-based hash of (job seed, generation, child, draw), so a
// job's trajectory depends on its seed alone — the same whether it runs alone or among others.
// Duplicate rejection (LIB/gaboom.cpp:977-1018 and the populate loop, :1936-1978): children and
// initial chromosomes whose hash_genes signature the job has seen are dropped, as by the
// reference's default (duplicates = false).
#include <cstdint>

#include "fxe_common.cuh"
#include "fxe_dmath.cuh"
#include "fxe_sort.cuh"

namespace fxe {

// SplitMix64 finaliser (Steele, Lea and Flood, OOPSLA 2014) of a 64-bit counter.
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// The 53 random bits of draw `k` of stream `s` of a job.
__device__ __forceinline__ uint64_t uniform_bits(uint64_t seed, uint64_t s, uint64_t k) {
    return mix64(seed ^ mix64(s * 0x100000001B3ull + k)) >> 11;
}

// Uniform double in [0, 1) for draw `k` of stream `s` of a job: its 53 bits times 2^-53 (both
// steps exact).
__device__ __forceinline__ double uniform(uint64_t seed, uint64_t s, uint64_t k) {
    return (double)uniform_bits(seed, s, k) * 0x1.0p-53;
}

// The integer form of the test u < p for draws u = b 2^-53 (b < 2^53 an integer): u < p exactly
// when b < ceil(p 2^53), the scaling by 2^53 being exact. Tests with it stay on the integer units
// (a mutation makes 32 such tests per gene).
__device__ __forceinline__ uint64_t draw_threshold(double p) {
    const double t = p * 0x1.0p53;
    if (t >= 0x1.0p53) return 1ull << 53;            // p >= 1: every draw is below
    return t > 0.0 ? (uint64_t)ceil(t) : 0ull;       // p <= 0 or NaN: no draw is
}

constexpr int kGaThreads = 256;
// The one-block-per-job sorts (replacement, fitness).
constexpr int kGaSortThreads = kSortThreads;
constexpr int kGaMaxPop = 2048;

// Order-preserving 64-bit image of a double that is not a NaN: the images compare as unsigned
// integers in the order the values compare (-0 and +0, which compare equal, share one image), so
// the sorts below run on the integer units rather than on the narrow double-precision pipe.
__device__ __forceinline__ uint64_t order_key(double x) {
    uint64_t b = (uint64_t)__double_as_longlong(x);
    if ((b << 1) == 0) b = 0;
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// roulette_wheel (LIB/gaboom.cpp:1158-1186) over the fitness in roulette order: the first
// position whose running sum exceeds r = u * total, the last position if none does, and a
// uniform position when the total is not positive.
__device__ __forceinline__ int roulette(const GaJob& J, double u) {
    const int P = J.P;
    const double tot = J.fstat[0];
    if (!(tot > 0.0)) return (int)(u * (double)P) % P;
    const double r = u * tot;
    int lo = 0, hi = P - 1;   // smallest k with fcum[k] > r
    if (!(J.fcum[P - 1] > r)) return P - 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (J.fcum[mid] > r) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// genetoic (LIB/gaboom.cpp:2887-2906): the first running bin total at or above u.
__device__ __forceinline__ double gene_ic(const GaJob& J, int g, int32_t gene) {
    const double u = gene / (2147483647.0 + 1.0);
    // the totals are positive: as signed 64-bit integers their bit patterns compare with u's as
    // the values do (a negative gene's u lies below them all), on the integer units
    const long long ub = __double_as_longlong(u);
    int lo = J.dec_off[g], hi = J.dec_off[g + 1];
    const int base = lo;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__double_as_longlong(J.dec_tab[mid]) < ub) lo = mid + 1;
        else hi = mid;
    }
    return J.gene_min[g] + J.gene_del[g] * (double)(lo - base);
}

// hash_genes (LIB/gaboom.cpp:1040-1045) with the C++ library's identity hash of int32.
__device__ __forceinline__ uint64_t signature(const GaJob& J, const int32_t* genes) {
    uint64_t h = 0;
    for (int i = 0; i < J.ng; ++i) {
        const int32_t v = (int32_t)(gene_ic(J, i, genes[i]) + 0.5);
        h ^= (uint64_t)(int64_t)v + 0x9e3779b9ull + (h << 6) + (h >> 2);
    }
    return h;
}

// The signature set: open addressing in HBM; 0 marks an empty slot of the table, so the signature
// 0 is kept in gen[4] instead.
// Whether a signature is in the set (no insertion).
__device__ bool seen_contains(const GaJob& J, uint64_t h) {
    if (h == 0) return J.gen[4] != 0;
    unsigned long long i = mix64(h) & J.hmask;
    for (unsigned long long n = 0; n <= J.hmask; ++n, i = (i + 1) & J.hmask) {
        const uint64_t v = J.seen[i];
        if (v == h) return true;
        if (v == 0) return false;
    }
    return false;
}

// Inserts a signature the set does not hold, safe beside other threads inserting other
// signatures (the table's layout may differ from one-at-a-time insertion; membership does not).
__device__ void seen_insert_concurrent(const GaJob& J, uint64_t h) {
    if (h == 0) {
        J.gen[4] = 1;
        return;
    }
    unsigned long long i = mix64(h) & J.hmask;
    for (unsigned long long n = 0; n <= J.hmask; ++n, i = (i + 1) & J.hmask) {
        const unsigned long long prev = atomicCAS(reinterpret_cast<unsigned long long*>(J.seen) + i, 0ull,
                                                  (unsigned long long)h);
        if (prev == 0ull || prev == h) return;
    }
}

__device__ __forceinline__ int32_t uniform_gene(const GaJob& J, uint64_t i) {
    return (int32_t)(mix64(J.seed ^ mix64(0xFFFFFFFFull * 977 + i)) >> 33);
}

// Initial candidates c0 .. c0 + 2 npairs - 1: uniform genes in [0, 2^31) like the reference's
// RandomInt over MAX_RANDOM_VALUE; candidate c's gene q is draw c * ng + q. A rotamer gene is
// drawn only with its side chain's probability, else 0 (rotamer 0, the input conformation;
// generate_random_individual, LIB/gaboom.cpp:1875-1895), that chance being draw c * ng + q of
// stream kInitRotStream.
constexpr uint64_t kInitRotStream = 0xFFFFFFFEull;

// (the candidates first, first + stride, ... of the batch: the threads of a block, or of a grid)
__device__ void initial_candidates(const GaJob& J, long long c0, int npairs, int first, int stride) {
    const int ng = J.ng;
    for (int c = first; c < 2 * npairs; c += stride) {
        int32_t* g = J.cand + (size_t)c * ng;
        for (int q = 0; q < ng; ++q) {
            const uint64_t i = (uint64_t)(c0 + c) * ng + q;
            const float pr = J.gene_prob[q];
            g[q] = pr < 0.0f || uniform(J.seed, kInitRotStream, i) < (double)pr ? uniform_gene(J, i) : 0;
        }
        J.cand_sig[c] = signature(J, g);
    }
}

__global__ void __launch_bounds__(kGaThreads) ga_init_kernel(const GaJob* __restrict__ all, const int* __restrict__ run) {
    const GaJob& J = all[run[blockIdx.y]];
    initial_candidates(J, 0, min(J.ncand, J.gen[1]), blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// adapt_prob (LIB/gaboom.cpp:848-880) for parents of fitness f1 and f2.
__device__ __forceinline__ void adapt_prob(const GaJob& J, double f1, double f2, double fit_max, double fit_avg, double* crossp,
                                           double* mutp) {
    const double hi = f1 > f2 ? f1 : f2, lo = f1 > f2 ? f2 : f1;
    double denom = fit_max - fit_avg;
    if (denom < 1e-15) denom = 1e-15;   // GA_FITNESS_DENOM_FLOOR, LIB/ga_constants.h:38
    *crossp = hi > fit_avg ? J.k[0] * (fit_max - hi) / denom : J.k[2];
    *mutp = lo > fit_avg ? J.k[1] * (fit_max - lo) / denom : J.k[3];
}

// The crossover's draws (LIB/gaboom.cpp:2527-2598): whether it happens, its genes and bit points.
struct Crossover {
    bool on;
    int gen_a, gen_b, pnt_a, pnt_b;
};
template <typename Draw>
__device__ __forceinline__ Crossover draw_crossover(const GaJob& J, Draw&& draw, double crossp) {
    const int ng = J.ng;
    Crossover x{false, 0, 0, 0, 0};
    if (!(draw() < crossp)) return x;
    x.on = true;
    x.gen_a = (int)(draw() * (double)ng);
    x.gen_b = (int)(draw() * (double)ng);
    if (x.gen_a >= ng) x.gen_a = ng - 1;
    if (x.gen_b >= ng) x.gen_b = ng - 1;
    if (J.intragenes) {
        x.pnt_a = (int)(draw() * 32.0);
        x.pnt_b = (int)(draw() * 32.0);
        if (x.gen_a > x.gen_b) {
            const int tg = x.gen_a, tp = x.pnt_a;
            x.gen_a = x.gen_b; x.pnt_a = x.pnt_b;
            x.gen_b = tg; x.pnt_b = tp;
        }
        if (x.gen_a == x.gen_b && x.pnt_a < x.pnt_b) {
            const int tp = x.pnt_b;
            x.pnt_b = x.pnt_a;
            x.pnt_a = tp;
        }
    } else {
        if (x.gen_a > x.gen_b) {
            const int tg = x.gen_a;
            x.gen_a = x.gen_b;
            x.gen_b = tg;
        }
        if (x.gen_a != x.gen_b) {
            x.pnt_a = draw() < 0.5 ? 32 : 0;
            x.pnt_b = draw() < 0.5 ? 32 : 0;
            if (x.gen_b - x.gen_a == 1 && x.pnt_a == 0 && x.pnt_b == 32) x.pnt_b = x.pnt_a;
        } else {
            x.pnt_a = 32;
            x.pnt_b = 0;
        }
    }
    return x;
}

// One pair of children: two roulette draws, optional adaptive probabilities, crossover with
// probability crossp, both children mutated bit by bit. draw() gives the next uniform in [0, 1)
// of the pair's draws, in the order the reference makes them.
template <typename Draw>
__device__ __forceinline__ void breed_pair_with(const GaJob& J, Draw&& draw, int32_t* john, int32_t* mary) {
    const int ng = J.ng;
    // fitness_stats (LIB/gaboom.cpp:818-840) of the population
    const double fit_max = J.fstat[1], fit_avg = J.fstat[2];
    const int pa = roulette(J, draw());
    const int pb = roulette(J, draw());
    const int a = J.ford[pa], b = J.ford[pb];
    double crossp = J.cross_rate, mutp = J.mut_rate;
    if (J.adaptive) adapt_prob(J, J.fit[pa], J.fit[pb], fit_max, fit_avg, &crossp, &mutp);
    int32_t* m = mary;
    for (int q = 0; q < ng; ++q) {
        john[q] = J.pop[(size_t)a * ng + q];
        m[q] = J.pop[(size_t)b * ng + q];
    }
    const Crossover x = draw_crossover(J, draw, crossp);
    if (x.on) {
        const int gen_a = x.gen_a, gen_b = x.gen_b;
        for (int j = gen_a; j <= gen_b; ++j) {
            const int np = j == gen_a ? x.pnt_a : 32;
            // the reference's mask: 1, then np times optr |= optr << 1
            const uint32_t optr = np >= 31 ? 0xFFFFFFFFu : ((2u << np) - 1u);
            const uint32_t uj = (uint32_t)john[j], um = (uint32_t)m[j];
            john[j] = (int32_t)((uj & ~optr) | (um & optr));
            m[j] = (int32_t)((uj & optr) | (um & ~optr));
        }
        if (x.pnt_b > 0) {
            const int np = x.pnt_b - 1;
            const uint32_t optr = np >= 31 ? 0xFFFFFFFFu : ((2u << np) - 1u);
            const uint32_t uj = (uint32_t)john[gen_b], um = (uint32_t)m[gen_b];
            john[gen_b] = (int32_t)((uj & ~optr) | (um & optr));
            m[gen_b] = (int32_t)((uj & optr) | (um & ~optr));
        }
    }
    // mutate both children (LIB/gaboom.cpp:2620-2641): the genes before the rotamer genes, then
    // each rotamer gene with its side chain's probability (LIB/gaboom.cpp:944-966)
    for (int c = 0; c < 2; ++c) {
        int32_t* ch = c == 0 ? john : m;
        for (int q = 0; q < ng; ++q) {
            const float pr = J.gene_prob[q];
            if (pr >= 0.0f && !(draw() < (double)pr)) continue;
            uint32_t optr = 0u;
            for (int bit = 0; bit < 32; ++bit)
                if (draw() < mutp) optr |= 1u << bit;
            ch[q] ^= (int32_t)optr;
        }
    }
}

// The draws of one pair: its counter-based stream.
struct StreamDraws {
    uint64_t seed, st, d;
    __device__ __forceinline__ double operator()() { return uniform(seed, st, d++); }
};

// One gene of a child after the crossover of breed_pair_with: its own value u and its mate's.
__device__ __forceinline__ uint32_t crossed(uint32_t own, uint32_t mate, int np) {
    const uint32_t optr = np >= 31 ? 0xFFFFFFFFu : ((2u << np) - 1u);
    return (own & ~optr) | (mate & optr);
}

// Pair k of the children of generation g + 1, from the generation's counter-based stream, by one
// warp: breed_pair_with's draws in its order, the genes spread over the lanes (genes lane and
// lane + 32; ng <= 64) and a gene's 32 mutation draws one per lane. A thread per pair made 1,216 draws
// one after another on nine SMs (184 us per generation of 2,000; 32 by warps, which spread over the device).
// cand: the pair's two chromosomes; sig: their signatures.
__device__ void breed_pair_warp(const GaJob& J, int g, int k, int lane, int32_t* cand, uint64_t* sig) {
    const int ng = J.ng;
    StreamDraws draw{J.seed, ((uint64_t)(g + 1) << 32) + (uint64_t)k, 0};   // streams of generation g + 1
    const double fit_max = J.fstat[1], fit_avg = J.fstat[2];
    const int pa = roulette(J, draw());
    const int pb = roulette(J, draw());
    const int a = J.ford[pa], b = J.ford[pb];
    double crossp = J.cross_rate, mutp = J.mut_rate;
    if (J.adaptive) adapt_prob(J, J.fit[pa], J.fit[pb], fit_max, fit_avg, &crossp, &mutp);
    const uint64_t mut = draw_threshold(mutp);
    const Crossover x = draw_crossover(J, draw, crossp);
    uint32_t c0[2] = {0u, 0u}, c1[2] = {0u, 0u};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int q = lane + 32 * h;
        if (q < ng) {
            uint32_t u = (uint32_t)J.pop[(size_t)a * ng + q], v = (uint32_t)J.pop[(size_t)b * ng + q];
            if (x.on) {
                if (q >= x.gen_a && q <= x.gen_b) {
                    const int np = q == x.gen_a ? x.pnt_a : 32;
                    const uint32_t t = crossed(u, v, np);
                    v = crossed(v, u, np);
                    u = t;
                }
                if (q == x.gen_b && x.pnt_b > 0) {
                    const uint32_t t = crossed(u, v, x.pnt_b - 1);
                    v = crossed(v, u, x.pnt_b - 1);
                    u = t;
                }
            }
            c0[h] = u;
            c1[h] = v;
        }
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        uint32_t* const ch = c == 0 ? c0 : c1;
        for (int q = 0; q < ng; ++q) {
            const float pr = J.gene_prob[q];
            if (pr >= 0.0f && !(draw() < (double)pr)) continue;
            const uint32_t optr = __ballot_sync(0xffffffffu, uniform_bits(draw.seed, draw.st, draw.d + lane) < mut);
            draw.d += 32;
            if (lane == (q & 31)) {
                if (q < 32) ch[0] ^= optr;
                else ch[1] ^= optr;
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (lane + 32 * h < ng) cand[c * ng + lane + 32 * h] = (int32_t)ch[h];
        // hash_genes of the child (see signature): the lanes decode, the fold is in gene order
        uint64_t sg = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int q = lane + 32 * h;
            const int32_t v = q < ng ? (int32_t)(gene_ic(J, q, (int32_t)ch[h]) + 0.5) : 0;
            for (int i = 32 * h; i < ng && i < 32 * h + 32; ++i)
                sg ^= (uint64_t)(int64_t)__shfl_sync(0xffffffffu, v, i & 31) + 0x9e3779b9ull + (sg << 6) + (sg >> 2);
        }
        if (lane == 0) sig[c] = sg;
    }
}

// Pairs k0 .. k0 + npairs - 1 of the running generation's children as candidates, with their
// signatures: the pairs first, first + stride, ... of the batch, one warp each (of a block, or of a grid).
__device__ void bred_candidates(const GaJob& J, int g, long long k0, int npairs, int first, int stride, int lane) {
    for (int k = first; k < npairs; k += stride)
        breed_pair_warp(J, g, (int)(k0 + k), lane, J.cand + (size_t)(2 * k) * J.ng, J.cand_sig + 2 * k);
}

__global__ void __launch_bounds__(kGaThreads) ga_breed_kernel(const GaJob* __restrict__ all, const int* __restrict__ run) {
    const GaJob& J = all[run[blockIdx.y]];
    bred_candidates(J, J.gen[0], 0, min(J.ncand, J.gen[1]), (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)),
                    (int)(gridDim.x * (blockDim.x >> 5)), threadIdx.x & 31);
}

// Blocks per job of the first candidate batch (pairs up to P + 8 with P <= 2048; one pair per thread).
constexpr int kGaBatchBlocks = (2048 + 8 + kGaThreads - 1) / kGaThreads;
// Blocks per job of the breeding kernel: a warp per pair, over the device's SMs when a job runs alone.
constexpr int kBreedBlocks = (2048 + 8) / (kGaThreads / 32);

constexpr int kGaMaxBatches = 16;   // candidate batches before duplicates are let through

// Acceptance in the reference's order (child 1, then child 2 of each pair, until the generation
// has nnew children; the initial population: P chromosomes): a candidate is taken unless its
// signature was seen before in the job, and taken signatures join the set. Walked one candidate
// at a time, candidate c is taken exactly when its signature is in neither the set the batch
// started from nor at an earlier candidate of the batch (an earlier copy joined the set or was in
// it), up to the candidate that completes the generation; candidates after it are not looked at.
// So the block decides all of a batch's candidates at once: the first occurrences by a hash table of
// (signature, lowest index) in shared memory, the set by read-only probes, the cut by an ordered
// scan; then it copies the taken ones into place and inserts their signatures. (A bitonic sort of the
// signatures in the table's place took most of the kernel's 145 us at 2,000 children; 41 us so.) When a batch runs
// out, the block breeds the next batch of pairs. After kGaMaxBatches batches candidates are taken
// as they come (counted in gen[2]), where the reference would loop until mutation finds new genes.
// gen[1] sizes the next generation's first batch from what this one used; gen[3] counts rejected
// candidates.
constexpr int kAcceptThreads = 1024;
constexpr int kAcceptMax = 2 * (kGaMaxPop + 8);    // candidates of a batch
constexpr int kAcceptTable = 8192;                 // hash slots: at most two thirds of them taken
static_assert(2 * kAcceptTable >= 3 * kAcceptMax && kAcceptTable <= 65536, "slots to spare, named by 16 bits");
constexpr size_t kAcceptSmem = (size_t)kAcceptTable * (sizeof(uint64_t) + sizeof(int)) + (size_t)kAcceptMax * (sizeof(uint16_t) + 1);

template <bool kInitial>
__global__ void __launch_bounds__(kAcceptThreads) ga_accept_kernel(const GaJob* __restrict__ all, const int* __restrict__ run) {
    extern __shared__ __align__(16) unsigned char acc_smem[];
    unsigned long long* hkey = reinterpret_cast<unsigned long long*>(acc_smem);
    int* hidx = reinterpret_cast<int*>(hkey + kAcceptTable);
    uint16_t* place = reinterpret_cast<uint16_t*>(hidx + kAcceptTable);   // a candidate's slot, then its rank
    uint8_t* take = reinterpret_cast<uint8_t*>(place + kAcceptMax);
    __shared__ int s_zero;
    __shared__ int wsum[kAcceptThreads / 32];
    __shared__ int s_cut, s_taken, s_rej;
    const GaJob& J = all[run[blockIdx.x]];
    const int ng = J.ng, g = J.gen[0];
    const int need = kInitial ? J.P : J.nnew;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int npairs = min(J.ncand, J.gen[1]);
    long long base = 0;   // candidate index of the batch's first entry
    int i = 0, used = 0, forced = 0, rejected = 0;
    for (int batch = 0;; ++batch) {
        const bool force = !J.reject || batch >= kGaMaxBatches;
        const int ncb = 2 * npairs;
        // 1. which candidates would be taken (before the cut)
        if (force) {
            for (int c = tid; c < ncb; c += kAcceptThreads) take[c] = 1;
        } else {
            for (int k = tid; k < kAcceptTable; k += kAcceptThreads) {
                hkey[k] = 0ull;
                hidx[k] = 0x7fffffff;
            }
            if (tid == 0) s_zero = 0x7fffffff;
            __syncthreads();
            // (0 marks an empty slot: that signature has a counter of its own)
            for (int c = tid; c < ncb; c += kAcceptThreads) {
                const unsigned long long h = J.cand_sig[c];
                if (h == 0ull) {
                    atomicMin(&s_zero, c);
                    continue;
                }
                int i = (int)(mix64(h) & (kAcceptTable - 1));
                for (int n = 0; n < kAcceptTable; ++n, i = (i + 1) & (kAcceptTable - 1)) {
                    const unsigned long long prev = atomicCAS(&hkey[i], 0ull, h);
                    if (prev == 0ull || prev == h) break;
                }
                atomicMin(&hidx[i], c);
                place[c] = (uint16_t)i;
            }
            __syncthreads();
            for (int c = tid; c < ncb; c += kAcceptThreads) {
                const unsigned long long h = J.cand_sig[c];
                const bool first = (h == 0ull ? s_zero : hidx[place[c]]) == c;
                take[c] = first && !seen_contains(J, h) ? 1 : 0;
            }
        }
        __syncthreads();
        // 2. the cut: the candidate that takes the generation to `need`, by an ordered scan over
        // contiguous runs of candidates per thread
        const int per = (ncb + kAcceptThreads - 1) / kAcceptThreads;
        const int c0 = tid * per, c1 = min(ncb, c0 + per);
        int cnt = 0;
        for (int c = c0; c < c1; ++c) cnt += take[c];
        int inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) wsum[warp] = inc;
        if (tid == 0) {
            s_cut = ncb;
            s_taken = 0;
            s_rej = 0;
        }
        __syncthreads();
        int wbase = 0;
        for (int w = 0; w < warp; ++w) wbase += wsum[w];
        const int left = need - i;
        int rank = wbase + inc - cnt;   // taken candidates before c0
        for (int c = c0; c < c1; ++c)
            if (take[c]) {
                if (rank == left - 1) s_cut = c;   // (one thread holds the cut, if any)
                ++rank;
            }
        __syncthreads();
        const int cut = s_cut;                  // last candidate looked at (ncb: none)
        // 3. copy the taken candidates up to the cut into place, insert their signatures, count
        int my_taken = 0, my_rej = 0;
        rank = wbase + inc - cnt;
        for (int c = c0; c < c1 && c <= cut; ++c) {
            if (c >= ncb) break;
            if (take[c]) {
                place[c] = (uint16_t)rank;
                if (!force) seen_insert_concurrent(J, J.cand_sig[c]);
                ++rank;
                ++my_taken;
            } else {
                ++my_rej;
            }
        }
        if (my_taken) atomicAdd(&s_taken, my_taken);
        if (my_rej) atomicAdd(&s_rej, my_rej);
        __syncthreads();
        const int n_copy = min(cut + 1, ncb) * ng;
        const unsigned inv = ng > 1 ? 0xffffffffu / (unsigned)ng + 1u : 0u;   // t / ng for these small t
        for (int t = tid; t < n_copy; t += kAcceptThreads) {
            const int c = ng > 1 ? (int)__umulhi((unsigned)t, inv) : t;
            if (take[c]) J.child[(size_t)(i + place[c]) * ng + (t - c * ng)] = J.cand[t];
        }
        const int taken = s_taken;
        if (J.reject && force) forced += taken;
        rejected += s_rej;
        i += taken;
        used = (int)(base + cut + 1);
        const bool done = i == need;
        __syncthreads();
        if (done) break;
        base += 2 * npairs;
        npairs = J.ncand;
        if (kInitial) initial_candidates(J, base, npairs, threadIdx.x, blockDim.x);
        else bred_candidates(J, g, base >> 1, npairs, warp, kAcceptThreads / 32, lane);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        int next;
        if (kInitial) {
            next = (J.nnew + 1) / 2 + J.nnew / 16 + 8;
        } else {
            const int pairs = (used + 1) / 2;
            next = pairs + pairs / 4 + 8;
        }
        J.gen[1] = min(J.ncand, next);
        J.gen[2] += forced;
        J.gen[3] += rejected;
    }
}

// Selection. kInitial: the evaluated initial population becomes generation 0. Otherwise the
// replacement: BOOM merges the P parents and nnew children, STEADY keeps the best P - nnew
// parents with the children in the places of the worst (child i at place P - 1 - i); the merged
// set is ordered by energy (equal energies by place, parents first), the best P kept, saved as the
// generation's snapshot, and the generation counter advanced. The parents are in order already: the
// children are sorted, and every entry's place in the merged order is its own place plus the entries
// of the other list before it, found by binary search (2,000 and 2,000: 52 us; 82 when all 4,000 were
// sorted).
template <bool kInitial>
__global__ void __launch_bounds__(kGaSortThreads) ga_select_kernel(GaJob* __restrict__ all, const int* __restrict__ run) {
    extern __shared__ __align__(16) unsigned char sel_smem[];
    uint64_t* const ckey = reinterpret_cast<uint64_t*>(sel_smem);   // the children, sorted
    uint64_t* const pkey = ckey + kGaMaxPop;                        // the parents
    int* const cidx = reinterpret_cast<int*>(pkey + kGaMaxPop);
    int* const idx = cidx + kGaMaxPop;                              // the entry at each new place
    GaJob& J = all[run[blockIdx.x]];
    const int P = J.P, ng = J.ng, nnew = J.nnew;
    const int g = J.gen[0];
    int32_t* const pop = J.pop;
    int32_t* const nxt = J.pop_next;
    double* const pe = J.pop_e;
    double* const nxt_e = J.pop_e_next;
    // entries: parents [0, np_), then children; idx >= np_ names a child
    const int np_ = kInitial ? 0 : (J.steady ? P - nnew : P);
    const int nc = kInitial ? P : nnew;
    for (int i = threadIdx.x; i < nc; i += blockDim.x) {
        const int id = np_ + i;
        // STEADY: the place P-1-c holds child c
        const int c = kInitial ? id : (J.steady ? (P - 1 - id) : i);
        double e = J.child_cf[c].evalue;
        if (e != e) e = INFINITY;   // a NaN energy sorts last
        ckey[i] = order_key(e);
        cidx[i] = id;
    }
    for (int i = threadIdx.x; i < np_; i += blockDim.x) pkey[i] = order_key(pe[i]);
    block_sort(ckey, cidx, nc);
    for (int i = threadIdx.x; i < np_; i += blockDim.x) {
        const uint64_t k = pkey[i];
        int lo = 0, hi = nc;   // children below k
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (ckey[mid] < k) lo = mid + 1;
            else hi = mid;
        }
        if (i + lo < P) idx[i + lo] = i;
    }
    for (int i = threadIdx.x; i < nc; i += blockDim.x) {
        const uint64_t k = ckey[i];
        int lo = 0, hi = np_;   // parents at or below k
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (pkey[mid] <= k) lo = mid + 1;
            else hi = mid;
        }
        if (i + lo < P) idx[i + lo] = cidx[i];
    }
    __syncthreads();
    // the new population, and (after a generation) its snapshot for the ensemble
    int32_t* const sg = kInitial ? nullptr : J.snap + (size_t)g * P * ng;
    double* const se = kInitial ? nullptr : J.snap_e + (size_t)g * P;
    const unsigned inv = ng > 1 ? 0xffffffffu / (unsigned)ng + 1u : 0u;   // t / ng for these small t
    for (int t = threadIdx.x; t < P * ng; t += blockDim.x) {
        const int r = ng > 1 ? (int)__umulhi((unsigned)t, inv) : t, q = t - r * ng;
        const int src = idx[r];
        const int c = kInitial ? src : (J.steady ? (P - 1 - src) : (src - np_));
        const int32_t v = src < np_ ? pop[(size_t)src * ng + q] : J.child[(size_t)c * ng + q];
        nxt[t] = v;
        if (!kInitial) sg[t] = v;
    }
    for (int r = threadIdx.x; r < P; r += blockDim.x) {
        const int src = idx[r];
        const int c = kInitial ? src : (J.steady ? (P - 1 - src) : (src - np_));
        double e = src < np_ ? pe[src] : J.child_cf[c].evalue;
        if (e != e) e = INFINITY;
        nxt_e[r] = e;
        if (!kInitial) se[r] = e;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        J.pop = nxt;
        J.pop_next = pop;
        J.pop_e = nxt_e;
        J.pop_e_next = pe;
        if (!kInitial) J.gen[0] = g + 1;
    }
}

// ICs of the (new) population, clamped into the gene limits as eval_chromosome leaves them in
// the genes (LIB/gaboom.cpp:1845-1866), for the niche counts. A block per SM: each value is a chain of
// look-ups (2,000 chromosomes of 19 genes: 69 us on eight blocks, 12 so).
__global__ void __launch_bounds__(kGaThreads) ga_decode_kernel(const GaJob* __restrict__ all, const int* __restrict__ run) {
    const GaJob& J = all[run[blockIdx.y]];
    if (J.fitness == kFitLinear) return;
    const int n = J.P * J.ng;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int q = t % J.ng;
        double v = gene_ic(J, q, J.pop[t]);
        if (v > J.gene_max[q]) v = J.gene_max[q];
        else if (v < J.gene_min[q]) v = J.gene_min[q];
        J.pic[t] = v;
    }
}

constexpr int kNicheRows = 8;              // chromosomes of a block
constexpr int kNicheChunk = 256;           // others taken at a time (one per thread)
constexpr int kNicheBlocks = (kGaMaxPop + kNicheRows - 1) / kNicheRows;

// Niche count of chromosome i: the sum over all j of 1 - (rmsp / sig_share)^alpha where rmsp
// (calc_rmsp, LIB/gaboom.cpp:2874-2885: root mean square of the IC differences) is within
// sig_share (LIB/gaboom.cpp:1652-1661). A pair beyond sig_share adds 0, which changes no sum of
// these non-negative terms, so only the pairs within it, in j order, need the double arithmetic:
// every pair's distance is formed in single precision with a bound on its error, the pairs not
// surely beyond sig_share are listed and evaluated in double by full warps, and each row's terms
// are added in j order, the block's eight rows on eight lanes. The FP64 unit (2 lanes per clock and
// SM) bounded the form that evaluated every pair in double: 0.87 ms per generation at P = 2,000, 0.11 so.
//
// Bound: with coordinates truncated to float (2^-23 of them) the distance's square root moves by at
// most 2^-23 (|x_i| + |x_j|) and its rounding by 2^-21 of it, so a pair whose float distance is above
// sqrt(ng) sig + 2^-22 (|x_i|_1 + |x_j|_1), by one part in 10^5, is beyond sig_share also in double.
__global__ void __launch_bounds__(kNicheChunk) ga_niche_kernel(const GaJob* __restrict__ all, const int* __restrict__ run) {
    __shared__ float xi[kNicheRows][64];
    __shared__ float ni[kNicheRows];
    __shared__ uint32_t mask[kNicheRows][kNicheChunk / 32];   // pairs listed
    __shared__ uint16_t list[kNicheRows * kNicheChunk];
    __shared__ double term[kNicheRows][kNicheChunk + 1];
    __shared__ int n_list;
    const GaJob& J = all[run[blockIdx.y]];
    const int ng = J.ng, P = J.P, i0 = blockIdx.x * kNicheRows;
    if (J.fitness == kFitLinear || i0 >= P) return;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int rows = min(kNicheRows, P - i0);
    const double sig = J.sig_share, alpha = J.share_alpha;
    const float lim0 = (float)(sqrt((double)ng) * sig) * 1.00001f;
    const bool f32 = ng <= 64;          // (longer rows than the staging's: every pair in double)
    for (int k = t; f32 && k < rows * ng; k += kNicheChunk) {
        const int r = k / ng;
        xi[r][k - r * ng] = d2f_trunc(J.pic[(size_t)i0 * ng + k]);
    }
    __syncthreads();
    if (t < rows) {
        float n = 0.0f;
        for (int q = 0; f32 && q < ng; ++q) n += fabsf(xi[t][q]);
        ni[t] = n;
    }
    double sum = 0.0;   // warp 0, lane r: row r
    for (int j0 = 0; j0 < P; j0 += kNicheChunk) {
        const int j = j0 + t;
        float acc[kNicheRows];
#pragma unroll
        for (int r = 0; r < kNicheRows; ++r) acc[r] = 0.0f;
        float nj = 0.0f;
        if (t == 0) n_list = 0;
        __syncthreads();
        if (f32 && j < P) {
            const double* xj = J.pic + (size_t)j * ng;
            for (int q = 0; q < ng; ++q) {
                const float x = d2f_trunc(xj[q]);
                nj += fabsf(x);
#pragma unroll
                for (int r = 0; r < kNicheRows; ++r) {
                    const float d = xi[r][q] - x;
                    acc[r] = fmaf(d, d, acc[r]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < kNicheRows; ++r) {
            const float lim = lim0 + 0x1.0p-22f * 1.00001f * (r < rows ? ni[r] + nj : 0.0f);
            const bool near = j < P && r < rows && !(f32 && acc[r] > lim * lim * 1.00002f);
            const unsigned m = __ballot_sync(0xffffffffu, near);
            int at = 0;
            if (lane == 0) {
                mask[r][warp] = m;
                if (m) at = atomicAdd(&n_list, __popc(m));
            }
            at = __shfl_sync(0xffffffffu, at, 0);
            if (near) list[at + __popc(m & lanemask_lt())] = (uint16_t)(r << 8 | t);
        }
        __syncthreads();
        const int n = n_list;
        for (int k = t; k < n; k += kNicheChunk) {
            const int r = list[k] >> 8, c = list[k] & 255;
            const double* a = J.pic + (size_t)(i0 + r) * ng;
            const double* b = J.pic + (size_t)(j0 + c) * ng;
            double s = 0.0;
            for (int q = 0; q < ng; ++q) {
                const double dq = a[q] - b[q];
                s = __fma_rn(dq, dq, s);
            }
            bool slow;
            double v = div_short(s, (double)ng, &slow);
            if (slow) v = plain_div(s, (double)ng);
            double d = sqrt_short(v, &slow);
            if (slow) d = plain_sqrt(v);
            double w = 0.0;
            if (d <= sig) {
                double x = div_short(d, sig, &slow);
                if (slow) x = plain_div(d, sig);
                w = 1.0 - (alpha == 1.0 ? x : pow(x, alpha));
            }
            term[r][c] = w;
        }
        __syncthreads();
        if (warp == 0 && lane < rows) {
            for (int w = 0; w < kNicheChunk / 32; ++w)
                for (uint32_t m = mask[lane][w]; m; m &= m - 1) sum += term[lane][32 * w + __ffs(m) - 1];
        }
        __syncthreads();
    }
    if (warp == 0 && lane < rows) J.share[i0 + lane] = sum;
}

// Running sums of the fitness in roulette order (roullete_wheel's walk, LIB/gaboom.cpp:1158-1186)
// and fitness_stats' total, maximum and mean (LIB/gaboom.cpp:818-840), in order.
__device__ void fitness_sums(const GaJob& J, const double* fit, int P) {
    // (fitness_stats' total adds the same terms in the same order as the running sum: one sum;
    // the largest value, the first of equal ones, is found on the order keys, off the
    // double-precision pipe)
    double cum = 0.0;
    uint64_t mk = order_key(fit[0]);
    int mi = 0;
#pragma unroll 8
    for (int i = 0; i < P; ++i) {
        const double f = fit[i];
        cum += f;
        J.fcum[i] = cum;
        const uint64_t k = order_key(f);
        const bool nan = ((uint64_t)__double_as_longlong(f) << 1) > (0x7FF0000000000000ull << 1);
        if (k > mk && !nan) {   // (a NaN never compares greater)
            mk = k;
            mi = i;
        }
    }
    J.fstat[0] = cum;
    J.fstat[1] = fit[mi];
    J.fstat[2] = cum / (double)P;
}

// Fitness of the population (sorted by energy), the roulette order, running sums and
// fitness_stats. kInitial: the initial population, walked in energy order whatever the model. The
// running sum is a chain of additions in the reference's order (70 cycles each): one thread makes
// nothing else, out of and into shared memory, while the block finds the maximum.
template <bool kInitial>
__global__ void __launch_bounds__(kGaSortThreads) ga_fitness_kernel(const GaJob* __restrict__ all, const int* __restrict__ run) {
    // the fitness (then its running sums), the sort keys (then the sorted fitness) and the order
    extern __shared__ __align__(16) unsigned char fit_smem[];
    double* const fval = reinterpret_cast<double*>(fit_smem);
    uint64_t* const key = reinterpret_cast<uint64_t*>(fval + kGaMaxPop);
    int* const idx = reinterpret_cast<int*>(key + kGaMaxPop);
    __shared__ uint64_t max_key[kGaSortThreads / 32];
    __shared__ int max_at[kGaSortThreads / 32];
    const GaJob& J = all[run[blockIdx.x]];
    const int P = J.P, model = J.fitness;
    const bool rank_only = model == kFitLinear || (model == kFitSmfree && !(J.beta > 0.0));
    double e0 = J.pop_e[0];
    if (!isfinite(e0)) e0 = 0.0;
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
        double f = (double)(P - i);
        if (!rank_only) {
            if (model == kFitPshare) {
                f = f / J.share[i];
            } else {
                // SMFREE (LIB/gaboom.cpp:1666-1736): the Boltzmann weight over the largest one
                // (that of the lowest energy)
                const double e = J.pop_e[i];
                const double bw = isfinite(e) && isfinite(J.pop_e[0]) ? exp(-J.beta * (e - e0)) : 0.0;
                const double blended = (1.0 - J.ent_w) * (f / (double)P) + J.ent_w * bw;
                f = blended * (double)P / J.share[i];
            }
        }
        fval[i] = f;
        idx[i] = i;
    }
    __syncthreads();
    const bool sorted = !kInitial && model == kFitPshare;
    if (sorted) {
        // QuickSort by fitness, descending (LIB/gaboom.cpp:499); equal fitness keeps energy order
        for (int i = threadIdx.x; i < P; i += blockDim.x) key[i] = order_key(-fval[i]);
        block_sort(key, idx, P);
    }
    double* const fs = reinterpret_cast<double*>(key);   // the fitness in roulette order
    double mine[2] = {0.0, 0.0};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int i = threadIdx.x + kGaSortThreads * e;
        if (i < P) mine[e] = fval[sorted ? idx[i] : i];
    }
    __syncthreads();
    // the largest value, the first of equal ones, on the order keys (a NaN never compares greater;
    // one in the first place stays)
    uint64_t mk = 0;
    int mi = 0x7fffffff;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int i = threadIdx.x + kGaSortThreads * e;
        if (i >= P) continue;
        const double f = mine[e];
        fs[i] = f;
        J.fit[i] = f;
        J.ford[i] = idx[i];
        const bool nan = ((uint64_t)__double_as_longlong(f) << 1) > (0x7FF0000000000000ull << 1);
        const uint64_t k = i == 0 && nan ? ~0ull : order_key(f);
        if ((!nan || i == 0) && (k > mk || (k == mk && i < mi))) {
            mk = k;
            mi = i;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t k2 = __shfl_xor_sync(0xffffffffu, (unsigned long long)mk, o);
        const int i2 = __shfl_xor_sync(0xffffffffu, mi, o);
        if (k2 > mk || (k2 == mk && i2 < mi)) {
            mk = k2;
            mi = i2;
        }
    }
    if ((threadIdx.x & 31) == 0) {
        max_key[threadIdx.x >> 5] = mk;
        max_at[threadIdx.x >> 5] = mi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kGaSortThreads / 32; ++w)
            if (max_key[w] > mk || (max_key[w] == mk && max_at[w] < mi)) {
                mk = max_key[w];
                mi = max_at[w];
            }
        double cum = 0.0;
#pragma unroll 8
        for (int i = 0; i < P; ++i) {
            cum += fs[i];
            fval[i] = cum;
        }
        J.fstat[0] = cum;
        J.fstat[1] = fs[mi];
        J.fstat[2] = cum / (double)P;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < P; i += blockDim.x) J.fcum[i] = fval[i];
}

constexpr int kDecodeBlocks = 152;
constexpr size_t kFitSmem = (size_t)kGaMaxPop * (2 * sizeof(uint64_t) + sizeof(int));
constexpr size_t kSelSmem = (size_t)kGaMaxPop * (2 * sizeof(uint64_t) + 2 * sizeof(int));

// The acceptance and selection kernels' shared memory (at or beyond the default 48 KB), allowed once
// per device.
static void ga_smem_attributes() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
    static bool done[64] = {false};
    if (done[dev]) return;
    cudaFuncSetAttribute(ga_accept_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAcceptSmem);
    cudaFuncSetAttribute(ga_accept_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAcceptSmem);
    cudaFuncSetAttribute(ga_select_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSelSmem);
    cudaFuncSetAttribute(ga_select_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSelSmem);
    cudaFuncSetAttribute(ga_fitness_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFitSmem);
    cudaFuncSetAttribute(ga_fitness_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFitSmem);
    done[dev] = true;
}

void launch_ga_fitness(const GaJob* all, const int* run, int n_jobs, bool initial, cudaStream_t st) {
    // (a gene's decode is a chain of table reads: a thread each keeps more of them in flight)
    ga_decode_kernel<<<dim3(kDecodeBlocks, n_jobs), kGaThreads, 0, st>>>(all, run);
    ga_niche_kernel<<<dim3(kNicheBlocks, n_jobs), kNicheChunk, 0, st>>>(all, run);
    if (initial) ga_fitness_kernel<true><<<n_jobs, kGaSortThreads, kFitSmem, st>>>(all, run);
    else ga_fitness_kernel<false><<<n_jobs, kGaSortThreads, kFitSmem, st>>>(all, run);
}

void launch_ga_init(const GaJob* all, const int* run, int n_jobs, cudaStream_t st) {
    ga_init_kernel<<<dim3(2 * kGaBatchBlocks, n_jobs), kGaThreads, 0, st>>>(all, run);
    ga_smem_attributes();
    ga_accept_kernel<true><<<n_jobs, kAcceptThreads, kAcceptSmem, st>>>(all, run);
}
void launch_ga_breed(const GaJob* all, const int* run, int n_jobs, cudaStream_t st) {
    ga_breed_kernel<<<dim3(kBreedBlocks, n_jobs), kGaThreads, 0, st>>>(all, run);
    ga_smem_attributes();
    ga_accept_kernel<false><<<n_jobs, kAcceptThreads, kAcceptSmem, st>>>(all, run);
}
// Breeding with the caller's draws (fxe_ga_breed_draws): J.fit and J.ford given, one block forms
// the running sums and fitness_stats, then one thread per pair breeds from its row of draws.
__global__ void ga_draws_stats_kernel(const GaJob* __restrict__ J) {
    if (threadIdx.x == 0 && blockIdx.x == 0) fitness_sums(*J, J->fit, J->P);
}

__global__ void __launch_bounds__(kGaThreads) ga_breed_draws_kernel(const GaJob* __restrict__ Jp, const double* __restrict__ draws,
                                                                    long long stride, int n_pairs, int* __restrict__ used) {
    const GaJob& J = *Jp;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_pairs) return;
    // the draws of one pair: its row of the caller's draws
    struct RowDraws {
        const double* row;
        long long stride, d;
        bool over;
        __device__ double operator()() {
            if (d >= stride) { over = true; return 0.0; }
            return row[d++];
        }
    } draw{draws + (size_t)k * stride, stride, 0, false};
    int32_t* john = J.child + (size_t)(2 * k) * J.ng;
    breed_pair_with(J, draw, john, john + J.ng);
    used[k] = draw.over ? -1 : (int)draw.d;
}

void launch_ga_breed_draws(const GaJob* J, const double* draws, long long stride, int n_pairs, int* used,
                           cudaStream_t st) {
    ga_draws_stats_kernel<<<1, 32, 0, st>>>(J);
    ga_breed_draws_kernel<<<(n_pairs + kGaThreads - 1) / kGaThreads, kGaThreads, 0, st>>>(J, draws, stride, n_pairs, used);
}

// Niche counts of a population whose ICs are given (fxe_ga_niche_counts): the generation's kernel
// on one job.
void launch_ga_niche(const GaJob* all, const int* run, cudaStream_t st) {
    ga_niche_kernel<<<dim3(kNicheBlocks, 1), kNicheChunk, 0, st>>>(all, run);
}

void launch_ga_select(GaJob* all, const int* run, int n_jobs, bool initial, cudaStream_t st) {
    ga_smem_attributes();
    if (initial) ga_select_kernel<true><<<n_jobs, kGaSortThreads, kSelSmem, st>>>(all, run);
    else ga_select_kernel<false><<<n_jobs, kGaSortThreads, kSelSmem, st>>>(all, run);
}

}  // namespace fxe
