// fxe_ensemble.cu — the GA ensemble the reference hands to statmech, assembled on the device:
// every generation's population (the snapshots, LIB/gaboom.cpp:494), sorted by energy
// (QuickSort, :520; ties here keep snapshot order), then remove_dups (:2728-2747): a chromosome is
// dropped when every decoded gene lies within 0.1 of the last chromosome kept.
//
// Sort: least-significant-digit radix sort of the energies' order-preserving 64-bit images, 8 bits
// a pass (8 passes), each pass a launch that counts every block's digits and one that scatters, stable
// (each block adds up the counts before its own, and ranks its elements by warp match and per-warp
// counts), so equal energies keep their input order.
//
// remove_dups is a chain: whether chromosome i is kept depends on which one was kept last. Runs of
// identical chromosomes (a survivor sits in the population for many generations) are collapsed
// first: a chromosome identical to its predecessor is always dropped and never becomes the last one
// kept. Over the remaining run heads, next(t) = the first later head that is not within 0.1 of head
// t (a bounded scan per thread, then one warp per unresolved head scanning 32 at a time); the kept
// heads are the path 0, next(0), next(next(0)), .... The heads are cut into segments that fit a block's
// shared memory: one launch finds by pointer jumping where the path leaves the segment from each of its
// heads, the next follows those exits to its segment (past 608 segments one thread does it for all, in a
// launch between) and marks the path inside.
//
// What bounds the assembly is its number of dependent launches more than the bytes (12 per chromosome
// and pass, the genes once): 4-bit digits with a three-launch scan each and log2(n) launches of pointer
// jumping made 130 of them.
#include <cstdint>

#include "fxe_place.cuh"

namespace fxe {

constexpr int kEnsThreads = 256;
constexpr int kScanThreads = 1024;
constexpr int kNearScan = 32;          // heads a thread tests before handing its head to a warp
constexpr double kDupTol = 0.1;        // LIB/gaboom.cpp:2737

// Order-preserving image of a double (NaN placed after +infinity, -0 with +0).
__device__ __forceinline__ unsigned long long order_key(double e) {
    if (e != e) return 0xFFFFFFFFFFFFFFFFull;
    if (e == 0.0) return 0x8000000000000000ull;   // -0 and +0 compare equal
    const unsigned long long b = (unsigned long long)__double_as_longlong(e);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// --- exclusive scan of int counts (n entries, total written to out[n]) -------------------------

__device__ __forceinline__ int block_excl_scan(int v, int* wsum, int* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        int s = lane < nw ? wsum[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < nw) wsum[lane] = s;
    }
    __syncthreads();
    const int before = w > 0 ? wsum[w - 1] : 0;
    *total = wsum[nw - 1];
    __syncthreads();
    return before + x - v;
}

__global__ void __launch_bounds__(kScanThreads) scan_block_kernel(const int* __restrict__ in, int* __restrict__ out, long long n,
                                                                  int* __restrict__ bsum) {
    __shared__ int wsum[32];
    const long long i = blockIdx.x * (long long)kScanThreads + threadIdx.x;
    const int v = i < n ? in[i] : 0;
    int tot;
    const int ex = block_excl_scan(v, wsum, &tot);
    if (i < n) out[i] = ex;
    if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

// One block: exclusive scan of the nb block sums in place, the grand total to *total.
__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(int* __restrict__ bsum, int nb, int* __restrict__ total) {
    __shared__ int wsum[32];
    const int per = (nb + kScanThreads - 1) / kScanThreads;
    const int b0 = threadIdx.x * per;
    int s = 0;
    for (int k = 0; k < per && b0 + k < nb; ++k) s += bsum[b0 + k];
    int tot;
    int run = block_excl_scan(s, wsum, &tot);
    for (int k = 0; k < per && b0 + k < nb; ++k) {
        const int v = bsum[b0 + k];
        bsum[b0 + k] = run;
        run += v;
    }
    if (threadIdx.x == 0) *total = tot;
}

__global__ void scan_add_kernel(int* __restrict__ out, long long n, const int* __restrict__ bsum) {
    const long long i = blockIdx.x * (long long)kScanThreads + threadIdx.x;
    if (i < n) out[i] += bsum[blockIdx.x];
}

// tmp: at least scan_tmp_ints(n) ints. out: n + 1 ints (out[n] = the total).
static long long scan_blocks(long long n) { return (n + kScanThreads - 1) / kScanThreads; }
long long scan_tmp_ints(long long n) { return scan_blocks(n > 0 ? n : 1) + 1; }

void scan_ints(const int* in, int* out, long long n, int* tmp, cudaStream_t st) {
    const long long nb = scan_blocks(n > 0 ? n : 1);
    scan_block_kernel<<<(unsigned)nb, kScanThreads, 0, st>>>(in, out, n, tmp);
    scan_sums_kernel<<<1, kScanThreads, 0, st>>>(tmp, (int)nb, out + n);
    scan_add_kernel<<<(unsigned)nb, kScanThreads, 0, st>>>(out, n, tmp);
}

// --- radix sort passes --------------------------------------------------------------------------

constexpr int kRadix = 256;
constexpr int kRadixItems = 8;                                // keys a thread holds
constexpr int kRadixTile = kEnsThreads * kRadixItems;
constexpr int kRadixBlocks = 4 * 152;                         // at most; then a block takes several tiles
static_assert(kEnsThreads == kRadix, "a digit per thread");

static long long radix_tiles_per_block(long long n) {
    const long long tiles = (n + kRadixTile - 1) / kRadixTile;
    return (tiles + kRadixBlocks - 1) / kRadixBlocks;
}
static int radix_blocks(long long n) {
    const long long per = radix_tiles_per_block(n) * kRadixTile;
    return (int)((n + per - 1) / per);
}

// The digit counts of each block's run of `per` keys, hist[block * kRadix + digit]. kFirst: the keys
// are formed from the energies and stored.
template <bool kFirst>
__global__ void __launch_bounds__(kEnsThreads)
radix_count_kernel(const double* __restrict__ e, unsigned long long* __restrict__ key, long long n, long long per, int shift,
                   int* __restrict__ hist) {
    __shared__ int cnt[kEnsThreads / 32][kRadix];
    const int w = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < kEnsThreads / 32 * kRadix; k += kEnsThreads) (&cnt[0][0])[k] = 0;
    __syncthreads();
    const long long lo = (long long)blockIdx.x * per, hi = lo + per < n ? lo + per : n;
    for (long long i0 = lo; i0 < hi; i0 += kRadixTile) {
        unsigned long long k[kRadixItems];
#pragma unroll
        for (int j = 0; j < kRadixItems; ++j) {
            const long long i = i0 + j * kEnsThreads + threadIdx.x;
            if (i < hi) k[j] = kFirst ? order_key(e[i]) : key[i];
        }
#pragma unroll
        for (int j = 0; j < kRadixItems; ++j) {
            const long long i = i0 + j * kEnsThreads + threadIdx.x;
            if (i < hi) {
                if (kFirst) key[i] = k[j];
                atomicAdd(&cnt[w][(int)((k[j] >> shift) & (kRadix - 1))], 1);
            }
        }
    }
    __syncthreads();
    int s = 0;
#pragma unroll
    for (int u = 0; u < kEnsThreads / 32; ++u) s += cnt[u][threadIdx.x];
    hist[blockIdx.x * kRadix + threadIdx.x] = s;
}

// Scatters each block's keys and values to their places, stable: a tile's elements in the order warp,
// item, lane, which is their order in the tile. vin null: the values are the indices.
__global__ void __launch_bounds__(kEnsThreads)
radix_scatter_kernel(const unsigned long long* __restrict__ kin, const int* __restrict__ vin, unsigned long long* __restrict__ kout,
                     int* __restrict__ vout, long long n, long long per, int shift, const int* __restrict__ hist) {
    __shared__ int wcnt[kEnsThreads / 32][kRadix + 1];      // (digit kRadix: past the end)
    __shared__ int wsum[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // where the block's first key of each digit goes
    int all = 0, before = 0;
#pragma unroll 8
    for (int b = 0; b < (int)gridDim.x; ++b) {
        const int c = hist[b * kRadix + threadIdx.x];
        all += c;
        before += b < (int)blockIdx.x ? c : 0;
    }
    int total;
    int off = block_excl_scan(all, wsum, &total) + before;      // of digit threadIdx.x
    const long long lo = (long long)blockIdx.x * per, hi = lo + per < n ? lo + per : n;
    for (long long i0 = lo; i0 < hi; i0 += kRadixTile) {
        const long long first = i0 + w * 32 * kRadixItems + lane;
        unsigned long long k[kRadixItems];
        int v[kRadixItems], rank[kRadixItems];
#pragma unroll
        for (int j = 0; j < kRadixItems; ++j) {
            const long long i = first + 32 * j;
            k[j] = i < hi ? kin[i] : 0ull;
            v[j] = i < hi ? (vin ? vin[i] : (int)i) : 0;
        }
        for (int d = lane; d <= kRadix; d += 32) wcnt[w][d] = 0;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < kRadixItems; ++j) {
            const int dg = first + 32 * j < hi ? (int)((k[j] >> shift) & (kRadix - 1)) : kRadix;
            const unsigned peers = __match_any_sync(0xffffffffu, dg);
            const int base = wcnt[w][dg], under = __popc(peers & lanemask_lt());
            rank[j] = base + under;
            __syncwarp();
            if (under == 0) wcnt[w][dg] = base + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kEnsThreads / 32; ++u) {
            const int c = wcnt[u][threadIdx.x];
            wcnt[u][threadIdx.x] = off;
            off += c;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kRadixItems; ++j) {
            if (first + 32 * j >= hi) continue;
            const long long dst = (long long)wcnt[w][(int)((k[j] >> shift) & (kRadix - 1))] + rank[j];
            kout[dst] = k[j];
            vout[dst] = v[j];
        }
        __syncthreads();
    }
}

// --- the chain over run heads -------------------------------------------------------------------

__device__ __forceinline__ bool within_tol(const double* __restrict__ a, const double* __restrict__ b, int ng) {
    for (int q = 0; q < ng; ++q)
        if (!(fabs(a[q] - b[q]) < kDupTol)) return false;
    return true;
}

// x / ng for a flat index x of [n][ng] (in 32 bits where they suffice).
__device__ __forceinline__ long long row_of(long long x, int ng, bool small) {
    return small ? (long long)((unsigned)x / (unsigned)ng) : x / ng;
}

// head[p] (zeroed before) = 1 where sorted chromosome p differs from p - 1 in some decoded gene.
__global__ void ens_heads_kernel(const double* __restrict__ ic, long long n, int ng, int* __restrict__ head) {
    const long long total = n * ng;
    const bool small = total <= 0xffffffffll;
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < total; x += (long long)gridDim.x * blockDim.x)
        if (x < ng || ic[x] != ic[x - ng]) head[row_of(x, ng, small)] = 1;
}

// H[t]: the sorted position of head t.
__global__ void ens_compact_kernel(const int* __restrict__ flag, const int* __restrict__ pos, long long n, int* __restrict__ out) {
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x)
        if (flag[p]) out[pos[p]] = (int)p;
}

__global__ void ens_next_kernel(const double* __restrict__ ic, int ng, const int* __restrict__ H, const int* __restrict__ Mp,
                                int* __restrict__ nxt, int* __restrict__ far_list, int* __restrict__ far_n) {
    const int M = *Mp;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < M; t += gridDim.x * blockDim.x) {
        const double* a = ic + (long long)H[t] * ng;
        int r = -1;
        const int last = t + kNearScan < M - 1 ? t + kNearScan : M - 1;
        for (int s = t + 1; s <= last; ++s)
            if (!within_tol(ic + (long long)H[s] * ng, a, ng)) { r = s; break; }
        if (r < 0) {
            if (last >= M - 1) r = M;
            else far_list[atomicAdd(far_n, 1)] = t;
        }
        nxt[t] = r;
    }
}

// One warp per head whose next head lies beyond the bounded scan: 32 later heads at a time.
__global__ void ens_next_far_kernel(const double* __restrict__ ic, int ng, const int* __restrict__ H, const int* __restrict__ Mp,
                                    int* __restrict__ nxt, const int* __restrict__ far_list, const int* __restrict__ far_n) {
    const int M = *Mp, nf = *far_n;
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    for (int u = blockIdx.x * wpb + (threadIdx.x >> 5); u < nf; u += gridDim.x * wpb) {
        const int t = far_list[u];
        const double* a = ic + (long long)H[t] * ng;
        int r = M;
        for (int base = t + kNearScan + 1; base < M; base += 32) {
            const int s = base + lane;
            const bool hit = s < M && !within_tol(ic + (long long)H[s] * ng, a, ng);
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            if (m) {
                r = base + __ffs(m) - 1;
                break;
            }
        }
        if (lane == 0) nxt[t] = r;
    }
}

constexpr int kSegment = 8192;         // heads of a segment
constexpr int kSegThreads = 1024;
constexpr int kSegItems = kSegment / kSegThreads;
constexpr size_t kSegSmem = sizeof(int) * kSegment + kSegment;

// out[t]: the first head past t's segment on the path from t (M: none), by pointer jumping inside the
// segment, at most log2(kSegment) rounds.
__global__ void __launch_bounds__(kSegThreads)
ens_exits_kernel(const int* __restrict__ nxt, const int* __restrict__ Mp, int* __restrict__ out) {
    extern __shared__ int jump[];
    const int M = *Mp;
    const long long base = (long long)blockIdx.x * kSegment;
    if (base >= M) return;
    const long long end = base + kSegment < M ? base + kSegment : M;
    int j[kSegItems];
#pragma unroll
    for (int k = 0; k < kSegItems; ++k) {
        const long long t = base + k * kSegThreads + threadIdx.x;
        j[k] = t < end ? nxt[t] : M;
        jump[k * kSegThreads + threadIdx.x] = j[k];
    }
    __syncthreads();
    for (;;) {
        bool more = false;
#pragma unroll
        for (int k = 0; k < kSegItems; ++k)
            if (j[k] < end) {
                j[k] = jump[j[k] - base];
                more = true;
            }
        if (!__syncthreads_or(more)) break;
#pragma unroll
        for (int k = 0; k < kSegItems; ++k) jump[k * kSegThreads + threadIdx.x] = j[k];
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < kSegItems; ++k) {
        const long long t = base + k * kSegThreads + threadIdx.x;
        if (t < end) out[t] = j[k];
    }
}

// Up to this many segments each block of ens_mark_kernel follows the exits to its own segment; beyond,
// one thread follows them once for all (the walks of S blocks are S^2 / 2 dependent loads, two blocks an
// SM at a time, so that they cost more than one walk from about 600 segments up). 300,000,000
// chromosomes, 36,622 segments: 693 ms the call with every block walking, 358 ms so (20,000,000: 21.5
// and 20.6; 4,000,000: 4.8 either way).
constexpr int kOwnWalk = 608;

// entry[s]: the first head on the path from head 0 that lies in segment s or past it.
__global__ void ens_entries_kernel(const int* __restrict__ exits, const int* __restrict__ Mp, int* __restrict__ entry) {
    const int M = *Mp;
    int t = 0;
    for (long long base = 0; base < M; base += kSegment) {
        entry[base / kSegment] = t;
        if (t < base + kSegment) t = exits[t];
    }
}

// flag[t] = 1 for the heads on the path from head 0, 0 for the others and for t from M to n: each block
// takes its segment's entry (entries null: follows the exits to it), then marks by pointer jumping inside
// (every marked head marks the head 2^r steps along).
__global__ void __launch_bounds__(kSegThreads)
ens_mark_kernel(const int* __restrict__ nxt, const int* __restrict__ exits, const int* __restrict__ entries,
                const int* __restrict__ Mp, long long n, int* __restrict__ flag) {
    extern __shared__ int jump[];
    volatile uint8_t* on = reinterpret_cast<uint8_t*>(jump + kSegment);
    __shared__ int entry;
    const int M = *Mp;
    const long long base = (long long)blockIdx.x * kSegment;
    const long long end = base + kSegment < M ? base + kSegment : M;
    if (base < M) {
        if (threadIdx.x == 0) {
            int t = entries ? entries[blockIdx.x] : 0;
            while (t < base) t = exits[t];
            entry = t;
        }
        int j[kSegItems];
#pragma unroll
        for (int k = 0; k < kSegItems; ++k) {
            const int at = k * kSegThreads + threadIdx.x;
            j[k] = base + at < end ? nxt[base + at] : M;
            jump[at] = j[k];
            on[at] = 0;
        }
        __syncthreads();
        if (threadIdx.x == 0 && entry < end) on[entry - base] = 1;
        __syncthreads();
        for (;;) {
            bool more = false;
            uint8_t mark = 0;
#pragma unroll
            for (int k = 0; k < kSegItems; ++k)
                if (on[k * kSegThreads + threadIdx.x]) mark |= 1u << k;
            __syncthreads();       // (a round marks from the heads marked before it)
#pragma unroll
            for (int k = 0; k < kSegItems; ++k)
                if (j[k] < end) {
                    if (mark >> k & 1) on[j[k] - base] = 1;
                    j[k] = jump[j[k] - base];
                    more = true;
                }
            if (!__syncthreads_or(more)) break;
#pragma unroll
            for (int k = 0; k < kSegItems; ++k) jump[k * kSegThreads + threadIdx.x] = j[k];
            __syncthreads();
        }
    }
#pragma unroll
    for (int k = 0; k < kSegItems; ++k) {
        const int at = k * kSegThreads + threadIdx.x;
        if (base + at < n) flag[base + at] = base + at < end ? (int)on[at] : 0;
    }
}

// Sorted ICs from ICs given in input order.
__global__ void ens_gather_ic_kernel(const double* __restrict__ ic_in, const int* __restrict__ order, long long n, int ng,
                                     double* __restrict__ ic_out) {
    const long long total = n * ng;
    const bool small = total <= 0xffffffffll;
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < total; x += (long long)gridDim.x * blockDim.x) {
        const long long p = row_of(x, ng, small);
        const int q = (int)(x - p * ng);
        ic_out[x] = ic_in[(long long)order[p] * ng + q];
    }
}

// Sorted ICs decoded from int32 genes in input order, clamped as eval_chromosome leaves them.
__global__ void ens_decode_kernel(DevSystem S, const int32_t* __restrict__ genes, const int* __restrict__ order, long long n,
                                  double* __restrict__ ic_out) {
    const int ng = S.n_genes;
    const long long total = n * ng;
    const bool small = total <= 0xffffffffll;
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < total; x += (long long)gridDim.x * blockDim.x) {
        const long long p = row_of(x, ng, small);
        const int q = (int)(x - p * ng);
        double v = S.gene_min[q] + S.gene_del[q] * (double)gene_bin(S, q, genes[(long long)order[p] * ng + q]);
        if (v > S.gene_max[q]) v = S.gene_max[q];
        else if (v < S.gene_min[q]) v = S.gene_min[q];
        ic_out[x] = v;
    }
}

// The kept chromosomes: their sorted positions (kept_pos) -> input indices, energies and ICs.
__global__ void ens_emit_kernel(const int* __restrict__ H, const int* __restrict__ flag, const int* __restrict__ pos,
                                const int* __restrict__ Mp, const int* __restrict__ order, const double* __restrict__ e_in,
                                const double* __restrict__ ic_sorted, int ng, long long* __restrict__ idx_out,
                                double* __restrict__ e_out, double* __restrict__ ic_out) {
    const int M = *Mp;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < M; t += gridDim.x * blockDim.x) {
        if (!flag[t]) continue;
        const int k = pos[t];
        const int p = H[t];
        const int src = order[p];
        if (idx_out) idx_out[k] = src;
        if (e_out) e_out[k] = e_in[src];
        if (ic_out)
            for (int q = 0; q < ng; ++q) ic_out[(long long)k * ng + q] = ic_sorted[(long long)p * ng + q];
    }
}

// --- driver ---------------------------------------------------------------------------------

static unsigned grid_for(long long n, int threads) {
    long long b = (n + threads - 1) / threads;
    if (b > 16384) b = 16384;
    return (unsigned)(b > 0 ? b : 1);
}

// The scratch buffers of one assembly, carved from one allocation in a fixed order; with base
// null only the size is counted (ensemble_scratch_bytes), so sizing and carving cannot disagree.
struct EnsScratch {
    unsigned long long *k0, *k1;
    int *v0, *v1, *hist, *stmp, *head;
    double* ics;
    int* cnt;
    size_t bytes = 0;

    template <typename T>
    T* take(unsigned char* base, size_t count) {
        T* q = base ? reinterpret_cast<T*>(base + bytes) : nullptr;
        bytes += (count * sizeof(T) + 255) & ~(size_t)255;
        return q;
    }
    void carve(unsigned char* base, long long n, int ng) {
        bytes = 0;
        k0 = take<unsigned long long>(base, n);
        k1 = take<unsigned long long>(base, n);
        v0 = take<int>(base, n);
        v1 = take<int>(base, n);
        hist = take<int>(base, (size_t)kRadix * radix_blocks(n));
        stmp = take<int>(base, scan_tmp_ints(n + 1));
        ics = take<double>(base, (size_t)n * ng);
        head = take<int>(base, 5 * (n + 1));           // head flags, positions, H, next, exits (far list)
        cnt = take<int>(base, 4);                      // M, far count
    }
};

size_t ensemble_scratch_bytes(long long n, int ng) {
    EnsScratch s;
    s.carve(nullptr, n > 0 ? n : 1, ng);
    return s.bytes;
}

// Sorts n energies, collapses identical runs, runs the chain and writes the kept chromosomes
// (input indices, energies, ICs; each may be null) in energy order; *d_kept (device) gets their
// count. ICs come from ic_in (n * ng, input order) or, when null, from genes decoded with S.
// scratch: ensemble_scratch_bytes(n, ng) bytes.
cudaError_t launch_ensemble(long long n, int ng, const double* e_in, const double* ic_in, const DevSystem* S,
                            const int32_t* genes, void* scratch, long long* idx_out, double* e_out, double* ic_out,
                            int* d_kept, cudaStream_t st) {
    if (n <= 0) return cudaMemsetAsync(d_kept, 0, sizeof(int), st);
    EnsScratch sc;
    sc.carve(static_cast<unsigned char*>(scratch), n, ng);
    unsigned long long *k0 = sc.k0, *k1 = sc.k1;
    int *v0 = sc.v0, *v1 = sc.v1;
    int* hist = sc.hist;
    int* stmp = sc.stmp;
    double* ics = sc.ics;
    int* head = sc.head;
    int* hpos = head + (n + 1);
    int* H = hpos + (n + 1);
    int* nxt = H + (n + 1);
    int* exits = nxt + (n + 1);
    int* cnt = sc.cnt;                                       // [0] M, [1] far count
    int* kept_flag = head;                                   // reused once the heads are compacted
    int* kept_pos = hpos;

    const int nb = radix_blocks(n);
    const long long per = radix_tiles_per_block(n) * kRadixTile;
    for (int pass = 0; pass < 8; ++pass) {
        const int shift = 8 * pass;
        if (pass == 0) radix_count_kernel<true><<<nb, kEnsThreads, 0, st>>>(e_in, k0, n, per, shift, hist);
        else radix_count_kernel<false><<<nb, kEnsThreads, 0, st>>>(nullptr, k0, n, per, shift, hist);
        radix_scatter_kernel<<<nb, kEnsThreads, 0, st>>>(k0, pass == 0 ? nullptr : v0, k1, v1, n, per, shift, hist);
        unsigned long long* tk = k0; k0 = k1; k1 = tk;
        int* tv = v0; v0 = v1; v1 = tv;
    }
    // v0: input index at each sorted position
    if (ic_in) ens_gather_ic_kernel<<<grid_for(n * ng, kEnsThreads), kEnsThreads, 0, st>>>(ic_in, v0, n, ng, ics);
    else ens_decode_kernel<<<grid_for(n * ng, kEnsThreads), kEnsThreads, 0, st>>>(*S, genes, v0, n, ics);
    cudaError_t e = cudaMemsetAsync(head, 0, sizeof(int) * (size_t)n, st);
    if (e != cudaSuccess) return e;
    ens_heads_kernel<<<grid_for(n * ng, kEnsThreads), kEnsThreads, 0, st>>>(ics, n, ng, head);
    scan_ints(head, hpos, n, stmp, st);
    ens_compact_kernel<<<grid_for(n, kEnsThreads), kEnsThreads, 0, st>>>(head, hpos, n, H);
    e = cudaMemcpyAsync(cnt, hpos + n, sizeof(int), cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(cnt + 1, 0, sizeof(int), st)) != cudaSuccess) return e;
    // heads: at most n; the kernels read M from the device
    ens_next_kernel<<<grid_for(n, kEnsThreads), kEnsThreads, 0, st>>>(ics, ng, H, cnt, nxt, exits, cnt + 1);
    ens_next_far_kernel<<<grid_for(n * 32, kEnsThreads), kEnsThreads, 0, st>>>(ics, ng, H, cnt, nxt, exits, cnt + 1);
    const unsigned segments = (unsigned)((n + kSegment - 1) / kSegment);
    ens_exits_kernel<<<segments, kSegThreads, kSegSmem, st>>>(nxt, cnt, exits);
    int* entries = nullptr;
    if (segments > kOwnWalk) {
        entries = stmp;      // (an int per 1,024 chromosomes, free between the scans)
        ens_entries_kernel<<<1, 1, 0, st>>>(exits, cnt, entries);
    }
    ens_mark_kernel<<<segments, kSegThreads, kSegSmem, st>>>(nxt, exits, entries, cnt, n, kept_flag);
    scan_ints(kept_flag, kept_pos, n, stmp, st);
    ens_emit_kernel<<<grid_for(n, kEnsThreads), kEnsThreads, 0, st>>>(H, kept_flag, kept_pos, cnt, v0, e_in, ics, ng, idx_out,
                                                                      e_out, ic_out);
    if ((e = cudaMemcpyAsync(d_kept, kept_pos + n, sizeof(int), cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace fxe
