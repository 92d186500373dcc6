// fxe_thermo.cu — FP64 canonical-ensemble reduction (StatMechEngine::compute,
// LIB/statmech.cpp:73-174, and boltzmann_weights, :178-201).
//
// One pass over the energies: every thread keeps an online log-sum-exp state
// (running max m of the log-weights lw = ln n - beta E, s = sum exp(lw - m), and the first and
// second energy moments weighted the same way); blocks merge their threads' states and write one
// partial each; the host merges the partials. This equals the reference's three passes
// (max-shifted log-sum-exp of LIB/UnifiedHardwareDispatch.cpp:800-843, then the moments with
// p = exp(lw - lnZ)) up to rounding, and reads each energy once.
#include <climits>
#include <cmath>

#include "fxe_common.cuh"

namespace fxe {

constexpr int kThermoThreads = 256;

struct LseState {
    double m, s, e1, e2;
};

// One energy into the state. Both cases take exp(-|lw - m|): the rescale factor of the sums when
// lw is a new maximum, the weight of the energy otherwise; one exp per energy and no divergent
// exp between the lanes of a warp. (With no energy yet, m = -inf and the factor is exp(-inf) = 0.)
__device__ __forceinline__ void lse_push(LseState& st, double lw, double e) {
    const double d = lw - st.m;
    const double x = exp(-fabs(d));
    if (d > 0.0) {
        st.s = st.s * x + 1.0;
        st.e1 = st.e1 * x + e;
        st.e2 = st.e2 * x + e * e;
        st.m = lw;
    } else {
        st.s += x;
        st.e1 += x * e;
        st.e2 += x * e * e;
    }
}

// The block's states merged, max first: the block's maximum M by shuffles, then each thread's
// sums rescaled once by exp(m - M) and added up (one exp per thread instead of one per merge).
// Every thread of the block calls it; thread 0 gets the result.
__device__ LseState block_merge(const LseState& st) {
    __shared__ double wm[kThermoThreads / 32];
    __shared__ double ws[3][kThermoThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double m = st.m;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) wm[warp] = m;
    __syncthreads();
    double M = wm[0];
    for (int w = 1; w < kThermoThreads / 32; ++w) M = fmax(M, wm[w]);
    const double f = st.m == -INFINITY ? 0.0 : exp(st.m - M);
    double a = st.s * f, b = st.e1 * f, c = st.e2 * f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if (lane == 0) {
        ws[0][warp] = a;
        ws[1][warp] = b;
        ws[2][warp] = c;
    }
    __syncthreads();
    LseState t{M, 0.0, 0.0, 0.0};
    if (threadIdx.x == 0)
        for (int w = 0; w < kThermoThreads / 32; ++w) {
            t.s += ws[0][w];
            t.e1 += ws[1][w];
            t.e2 += ws[2][w];
        }
    return t;
}

__global__ void __launch_bounds__(kThermoThreads)
thermo_partial_kernel(const double* __restrict__ e, const int32_t* __restrict__ mult, long n,
                      double beta, LsePart* __restrict__ part) {
    LseState st{-INFINITY, 0.0, 0.0, 0.0};
    const long stride = (long)gridDim.x * blockDim.x;
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const double ei = e[i];
        const double lw = (mult ? log((double)mult[i]) : 0.0) - beta * ei;
        lse_push(st, lw, ei);
    }
    const LseState t = block_merge(st);
    if (threadIdx.x == 0) part[blockIdx.x] = {t.m, t.s, t.e1, t.e2};
}

__global__ void thermo_weights_kernel(const double* __restrict__ e, const int32_t* __restrict__ mult,
                                      long n, double beta, double lnZ, double* __restrict__ w) {
    const long stride = (long)gridDim.x * blockDim.x;
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const double lw = (mult ? log((double)mult[i]) : 0.0) - beta * e[i];
        w[i] = exp(lw - lnZ);
    }
}

int thermo_blocks(long n, int sms) {
    long b = (n + kThermoThreads - 1) / kThermoThreads;
    const long cap = (long)sms * 8;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

void launch_thermo_partial(const double* e, const int32_t* mult, long n, double beta, LsePart* part,
                           int blocks, cudaStream_t st) {
    thermo_partial_kernel<<<blocks, kThermoThreads, 0, st>>>(e, mult, n, beta, part);
}

void launch_thermo_weights(const double* e, const int32_t* mult, long n, double beta, double lnZ,
                           double* w, int blocks, cudaStream_t st) {
    thermo_weights_kernel<<<blocks, kThermoThreads, 0, st>>>(e, mult, n, beta, lnZ, w);
}

// Host merge of the block partials into the reference's Thermodynamics record.
void thermo_finish(const LsePart* part, int nb, double T, fxe_thermo* out) {
    const double kB = 0.001987206;  // LIB/statmech.h:26
    double M = -INFINITY;
    for (int b = 0; b < nb; ++b) M = part[b].m > M ? part[b].m : M;
    double s = 0.0, e1 = 0.0, e2 = 0.0;
    for (int b = 0; b < nb; ++b) {
        if (part[b].m == -INFINITY) continue;
        const double f = std::exp(part[b].m - M);
        s += part[b].s * f;
        e1 += part[b].e1 * f;
        e2 += part[b].e2 * f;
    }
    const double lnZ = M + std::log(s);
    const double Ea = e1 / s, E2 = e2 / s;
    const double kT = kB * T;
    const double var = E2 - Ea * Ea;
    out->temperature = T;
    out->log_Z = lnZ;
    out->free_energy = -kT * lnZ;
    out->mean_energy = Ea;
    out->mean_energy_sq = E2;
    out->heat_capacity = var / (kT * kT);
    out->entropy = (Ea - out->free_energy) / T;
    out->std_energy = std::sqrt(var > 0.0 ? var : 0.0);
}

}  // namespace fxe

// ------------------------------------------------------------------------------------------
// Fixed-scratch variant: the same reduction with the block partials in a file-scope device
// array and the merge on the device, for callers that may not allocate (see
// fxe_thermo_compute_device_fixed in include/fxe.h).
// ------------------------------------------------------------------------------------------
namespace fxe {

constexpr int kFixedBlocks = 4 * 152;   // at most

// One partial per block, and after them one slot for the count of finished blocks; every slot a
// call reads is written (or, the count, cleared) by that call first, so nothing here needs to
// start at zero.
static __device__ __align__(256) LsePart g_fixed_part[kFixedBlocks + 1];

cudaError_t fixed_scratch_address(LsePart** p) {
    return cudaGetSymbolAddress(reinterpret_cast<void**>(p), g_fixed_part);
}

// exp(x) for |x| < 700 by the table method (P. T. P. Tang, ACM Transactions on Mathematical Software
// 15, 1989): x = (256 j + i) ln2 / 256 + r with |r| < ln2 / 512, exp(x) = 2^j 2^(i/256) (1 + p(r)), p
// the Taylor polynomial to r^4 (the next term is below 4e-17). Nine FP64 instructions.
static __device__ const unsigned long long kExp2Table[256] = {   // 2^(i/256), rounded to nearest
    0x3ff0000000000000ull, 0x3ff00b1afa5abcbfull, 0x3ff0163da9fb3335ull, 0x3ff02168143b0281ull, 0x3ff02c9a3e778061ull, 0x3ff037d42e11bbccull,
    0x3ff04315e86e7f85ull, 0x3ff04e5f72f654b1ull, 0x3ff059b0d3158574ull, 0x3ff0650a0e3c1f89ull, 0x3ff0706b29ddf6deull, 0x3ff07bd42b72a836ull,
    0x3ff0874518759bc8ull, 0x3ff092bdf66607e0ull, 0x3ff09e3ecac6f383ull, 0x3ff0a9c79b1f3919ull, 0x3ff0b5586cf9890full, 0x3ff0c0f145e46c85ull,
    0x3ff0cc922b7247f7ull, 0x3ff0d83b23395decull, 0x3ff0e3ec32d3d1a2ull, 0x3ff0efa55fdfa9c5ull, 0x3ff0fb66affed31bull, 0x3ff1073028d7233eull,
    0x3ff11301d0125b51ull, 0x3ff11edbab5e2ab6ull, 0x3ff12abdc06c31ccull, 0x3ff136a814f204abull, 0x3ff1429aaea92de0ull, 0x3ff14e95934f312eull,
    0x3ff15a98c8a58e51ull, 0x3ff166a45471c3c2ull, 0x3ff172b83c7d517bull, 0x3ff17ed48695bbc0ull, 0x3ff18af9388c8deaull, 0x3ff1972658375d2full,
    0x3ff1a35beb6fcb75ull, 0x3ff1af99f8138a1cull, 0x3ff1bbe084045cd4ull, 0x3ff1c82f95281c6bull, 0x3ff1d4873168b9aaull, 0x3ff1e0e75eb44027ull,
    0x3ff1ed5022fcd91dull, 0x3ff1f9c18438ce4dull, 0x3ff2063b88628cd6ull, 0x3ff212be3578a819ull, 0x3ff21f49917ddc96ull, 0x3ff22bdda27912d1ull,
    0x3ff2387a6e756238ull, 0x3ff2451ffb82140aull, 0x3ff251ce4fb2a63full, 0x3ff25e85711ece75ull, 0x3ff26b4565e27cddull, 0x3ff2780e341ddf29ull,
    0x3ff284dfe1f56381ull, 0x3ff291ba7591bb70ull, 0x3ff29e9df51fdee1ull, 0x3ff2ab8a66d10f13ull, 0x3ff2b87fd0dad990ull, 0x3ff2c57e39771b2full,
    0x3ff2d285a6e4030bull, 0x3ff2df961f641589ull, 0x3ff2ecafa93e2f56ull, 0x3ff2f9d24abd886bull, 0x3ff306fe0a31b715ull, 0x3ff31432edeeb2fdull,
    0x3ff32170fc4cd831ull, 0x3ff32eb83ba8ea32ull, 0x3ff33c08b26416ffull, 0x3ff3496266e3fa2dull, 0x3ff356c55f929ff1ull, 0x3ff36431a2de883bull,
    0x3ff371a7373aa9cbull, 0x3ff37f26231e754aull, 0x3ff38cae6d05d866ull, 0x3ff39a401b7140efull, 0x3ff3a7db34e59ff7ull, 0x3ff3b57fbfec6cf4ull,
    0x3ff3c32dc313a8e5ull, 0x3ff3d0e544ede173ull, 0x3ff3dea64c123422ull, 0x3ff3ec70df1c5175ull, 0x3ff3fa4504ac801cull, 0x3ff40822c367a024ull,
    0x3ff4160a21f72e2aull, 0x3ff423fb2709468aull, 0x3ff431f5d950a897ull, 0x3ff43ffa3f84b9d4ull, 0x3ff44e086061892dull, 0x3ff45c2042a7d232ull,
    0x3ff46a41ed1d0057ull, 0x3ff4786d668b3237ull, 0x3ff486a2b5c13cd0ull, 0x3ff494e1e192aed2ull, 0x3ff4a32af0d7d3deull, 0x3ff4b17dea6db7d7ull,
    0x3ff4bfdad5362a27ull, 0x3ff4ce41b817c114ull, 0x3ff4dcb299fddd0dull, 0x3ff4eb2d81d8abffull, 0x3ff4f9b2769d2ca7ull, 0x3ff508417f4531eeull,
    0x3ff516daa2cf6642ull, 0x3ff5257de83f4eefull, 0x3ff5342b569d4f82ull, 0x3ff542e2f4f6ad27ull, 0x3ff551a4ca5d920full, 0x3ff56070dde910d2ull,
    0x3ff56f4736b527daull, 0x3ff57e27dbe2c4cfull, 0x3ff58d12d497c7fdull, 0x3ff59c0827ff07ccull, 0x3ff5ab07dd485429ull, 0x3ff5ba11fba87a03ull,
    0x3ff5c9268a5946b7ull, 0x3ff5d84590998b93ull, 0x3ff5e76f15ad2148ull, 0x3ff5f6a320dceb71ull, 0x3ff605e1b976dc09ull, 0x3ff6152ae6cdf6f4ull,
    0x3ff6247eb03a5585ull, 0x3ff633dd1d1929fdull, 0x3ff6434634ccc320ull, 0x3ff652b9febc8fb7ull, 0x3ff6623882552225ull, 0x3ff671c1c70833f6ull,
    0x3ff68155d44ca973ull, 0x3ff690f4b19e9538ull, 0x3ff6a09e667f3bcdull, 0x3ff6b052fa75173eull, 0x3ff6c012750bdabfull, 0x3ff6cfdcddd47645ull,
    0x3ff6dfb23c651a2full, 0x3ff6ef9298593ae5ull, 0x3ff6ff7df9519484ull, 0x3ff70f7466f42e87ull, 0x3ff71f75e8ec5f74ull, 0x3ff72f8286ead08aull,
    0x3ff73f9a48a58174ull, 0x3ff74fbd35d7cbfdull, 0x3ff75feb564267c9ull, 0x3ff77024b1ab6e09ull, 0x3ff780694fde5d3full, 0x3ff790b938ac1cf6ull,
    0x3ff7a11473eb0187ull, 0x3ff7b17b0976cfdbull, 0x3ff7c1ed0130c132ull, 0x3ff7d26a62ff86f0ull, 0x3ff7e2f336cf4e62ull, 0x3ff7f3878491c491ull,
    0x3ff80427543e1a12ull, 0x3ff814d2add106d9ull, 0x3ff82589994cce13ull, 0x3ff8364c1eb941f7ull, 0x3ff8471a4623c7adull, 0x3ff857f4179f5b21ull,
    0x3ff868d99b4492edull, 0x3ff879cad931a436ull, 0x3ff88ac7d98a6699ull, 0x3ff89bd0a478580full, 0x3ff8ace5422aa0dbull, 0x3ff8be05bad61778ull,
    0x3ff8cf3216b5448cull, 0x3ff8e06a5e0866d9ull, 0x3ff8f1ae99157736ull, 0x3ff902fed0282c8aull, 0x3ff9145b0b91ffc6ull, 0x3ff925c353aa2fe2ull,
    0x3ff93737b0cdc5e5ull, 0x3ff948b82b5f98e5ull, 0x3ff95a44cbc8520full, 0x3ff96bdd9a7670b3ull, 0x3ff97d829fde4e50ull, 0x3ff98f33e47a22a2ull,
    0x3ff9a0f170ca07baull, 0x3ff9b2bb4d53fe0dull, 0x3ff9c49182a3f090ull, 0x3ff9d674194bb8d5ull, 0x3ff9e86319e32323ull, 0x3ff9fa5e8d07f29eull,
    0x3ffa0c667b5de565ull, 0x3ffa1e7aed8eb8bbull, 0x3ffa309bec4a2d33ull, 0x3ffa42c980460ad8ull, 0x3ffa5503b23e255dull, 0x3ffa674a8af46052ull,
    0x3ffa799e1330b358ull, 0x3ffa8bfe53c12e59ull, 0x3ffa9e6b5579fdbfull, 0x3ffab0e521356ebaull, 0x3ffac36bbfd3f37aull, 0x3ffad5ff3a3c2774ull,
    0x3ffae89f995ad3adull, 0x3ffafb4ce622f2ffull, 0x3ffb0e07298db666ull, 0x3ffb20ce6c9a8952ull, 0x3ffb33a2b84f15fbull, 0x3ffb468415b749b1ull,
    0x3ffb59728de5593aull, 0x3ffb6c6e29f1c52aull, 0x3ffb7f76f2fb5e47ull, 0x3ffb928cf22749e4ull, 0x3ffba5b030a1064aull, 0x3ffbb8e0b79a6f1full,
    0x3ffbcc1e904bc1d2ull, 0x3ffbdf69c3f3a207ull, 0x3ffbf2c25bd71e09ull, 0x3ffc06286141b33dull, 0x3ffc199bdd85529cull, 0x3ffc2d1cd9fa652cull,
    0x3ffc40ab5fffd07aull, 0x3ffc544778fafb22ull, 0x3ffc67f12e57d14bull, 0x3ffc7ba88988c933ull, 0x3ffc8f6d9406e7b5ull, 0x3ffca3405751c4dbull,
    0x3ffcb720dcef9069ull, 0x3ffccb0f2e6d1675ull, 0x3ffcdf0b555dc3faull, 0x3ffcf3155b5bab74ull, 0x3ffd072d4a07897cull, 0x3ffd1b532b08c968ull,
    0x3ffd2f87080d89f2ull, 0x3ffd43c8eacaa1d6ull, 0x3ffd5818dcfba487ull, 0x3ffd6c76e862e6d3ull, 0x3ffd80e316c98398ull, 0x3ffd955d71ff6075ull,
    0x3ffda9e603db3285ull, 0x3ffdbe7cd63a8315ull, 0x3ffdd321f301b460ull, 0x3ffde7d5641c0658ull, 0x3ffdfc97337b9b5full, 0x3ffe11676b197d17ull,
    0x3ffe264614f5a129ull, 0x3ffe3b333b16ee12ull, 0x3ffe502ee78b3ff6ull, 0x3ffe653924676d76ull, 0x3ffe7a51fbc74c83ull, 0x3ffe8f7977cdb740ull,
    0x3ffea4afa2a490daull, 0x3ffeb9f4867cca6eull, 0x3ffecf482d8e67f1ull, 0x3ffee4aaa2188510ull, 0x3ffefa1bee615a27ull, 0x3fff0f9c1cb6412aull,
    0x3fff252b376bba97ull, 0x3fff3ac948dd7274ull, 0x3fff50765b6e4540ull, 0x3fff6632798844f8ull, 0x3fff7bfdad9cbe14ull, 0x3fff91d802243c89ull,
    0x3fffa7c1819e90d8ull, 0x3fffbdba3692d514ull, 0x3fffd3c22b8f71f1ull, 0x3fffe9d96b2a23d9ull};

__device__ __forceinline__ double exp_short(double x, const double* tab) {
    constexpr double kShift = 6755399441055744.0;   // 1.5 * 2^52: the sum's low bits are the integer
    double k = fma(x, 0x1.71547652b82fep+8, kShift);
    const int ki = __double2loint(k);
    k -= kShift;
    const double r = fma(k, -0x1.abc9e3b39803fp-64, fma(k, -0x1.62e42fefa39efp-9, x));
    const double c = fma(fma(fma(r, 1.0 / 24.0, 1.0 / 6.0), r, 0.5), r, 1.0) * r;
    const double t = tab[ki & 255];
    const double T = __hiloint2double(__double2hiint(t) + (ki >> 8) * 0x100000, __double2loint(t));
    return fma(T, c, T);
}

// The library's exp, for arguments outside exp_short's range (called, so that the loop does not carry
// it).
__device__ __noinline__ double exp_any(double x) { return exp(x); }

// A double's bits as an integer that orders like it (its own inverse).
__device__ __forceinline__ long long order_bits(long long b) { return b ^ ((b >> 63) & 0x7fffffffffffffffll); }

// The smallest of the block's keys, for every thread.
__device__ __forceinline__ long long block_min(long long k, long long* warp_min) {
    const int hi = (int)(k >> 32), mh = __reduce_min_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_min_sync(0xffffffffu, hi == mh ? (unsigned)k : 0xffffffffu);
    if ((threadIdx.x & 31) == 0) warp_min[threadIdx.x >> 5] = ((long long)mh << 32) | ml;
    __syncthreads();
    long long r = warp_min[0];
#pragma unroll
    for (int w = 1; w < kThermoThreads / 32; ++w) r = min(r, warp_min[w]);
    __syncthreads();
    return r;
}

// The block's sums of states with one maximum, for thread 0. Six additions a thread: the lanes split the
// three sums among them after the first two exchanges.
__device__ __forceinline__ LseState block_sums(const LseState& st, double (*ws)[kThermoThreads / 32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool up = lane & 16, mid = lane & 8;
    double x = (up ? st.e1 : st.s) + __shfl_xor_sync(0xffffffffu, up ? st.s : st.e1, 16);
    const double y = st.e2 + __shfl_xor_sync(0xffffffffu, st.e2, 16);
    x = (mid ? y : x) + __shfl_xor_sync(0xffffffffu, mid ? x : y, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0 || lane == 8 || lane == 16) ws[lane == 0 ? 0 : lane == 16 ? 1 : 2][warp] = x;
    __syncthreads();
    LseState t{st.m, 0.0, 0.0, 0.0};
    if (threadIdx.x == 0)
        for (int w = 0; w < kThermoThreads / 32; ++w) {
            t.s += ws[0][w];
            t.e1 += ws[1][w];
            t.e2 += ws[2][w];
        }
    return t;
}

// The fixed-scratch reduction in one launch: each block covers a contiguous run of per_block energies,
// kFixedChunk per thread at a time. A chunk's largest log-weight is found first, on the integer
// units, so that the sums are rescaled at most once per chunk and every energy costs one exp_short
// and four more FP64 instructions. The last block to finish (a counter in the scratch, cleared before
// the launch) merges the partials and writes the record.
// Bound by the FP64 unit (one warp instruction per 64 cycles and SM quarter): with the library's exp
// and a running maximum per thread an energy cost 55 of its instructions, 98 us for 1,000,000 energies;
// 47 us so (14 instructions an energy are 24 us).
constexpr int kFixedChunk = 8;

template <bool kMult>
__global__ void __launch_bounds__(kThermoThreads, 4)
thermo_fixed_kernel(const double* __restrict__ e, const int32_t* __restrict__ mult, long n, long per_block,
                    double beta, double T, LsePart* __restrict__ part, unsigned* __restrict__ done,
                    fxe_thermo* __restrict__ out) {
    __shared__ double tab[256];
    __shared__ long long warp_min[kThermoThreads / 32];
    __shared__ double ws[3][kThermoThreads / 32];
    static_assert(kThermoThreads == 256, "a table entry per thread");
    tab[threadIdx.x] = __longlong_as_double((long long)kExp2Table[threadIdx.x]);
    const long lo = (long)blockIdx.x * per_block;
    const long hi = lo + per_block < n ? lo + per_block : n;
    LseState st{-INFINITY, 0.0, 0.0, 0.0};
    #pragma unroll 1
    for (long i0 = lo; i0 < hi; i0 += (long)kFixedChunk * kThermoThreads) {
        double ev[kFixedChunk], lw[kMult ? kFixedChunk : 1];
        long long key = LLONG_MAX;      // orders like the negative of the log-weight
#pragma unroll
        for (int j = 0; j < kFixedChunk; ++j) {
            const long i = i0 + (long)j * kThermoThreads + threadIdx.x;
            ev[j] = i < hi ? e[i] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < kFixedChunk; ++j) {
            const long i = i0 + (long)j * kThermoThreads + threadIdx.x;
            if (i >= hi) continue;
            if (kMult) lw[j] = log((double)mult[i]) - beta * ev[j];
            key = min(key, order_bits(__double_as_longlong(kMult ? -lw[kMult ? j : 0] : ev[j])));
        }
        const double least = __longlong_as_double(order_bits(block_min(key, warp_min)));
        const double m = kMult ? -least : -(beta * least);
        if (!(m <= st.m)) {      // (the same for the whole block)
            const double f = st.m == -INFINITY ? 0.0 : exp_any(st.m - m);
            st.s *= f;
            st.e1 *= f;
            st.e2 *= f;
            st.m = m;
        }
#pragma unroll
        for (int j = 0; j < kFixedChunk; ++j) {
            const long i = i0 + (long)j * kThermoThreads + threadIdx.x;
            if (i >= hi) continue;
            const double x = kMult ? lw[kMult ? j : 0] - st.m : fma(-beta, ev[j], -st.m);
            double w;
            if ((__double2hiint(x) & 0x7fffffff) < 0x4085e000) {   // |x| < 700
                w = exp_short(x, tab);
            } else {
                const double l = kMult ? lw[kMult ? j : 0] : -(beta * ev[j]);
                if (l == -INFINITY) continue;
                w = exp_any(l - st.m);
            }
            const double we = w * ev[j];
            st.s += w;
            st.e1 += we;
            st.e2 = fma(we, ev[j], st.e2);
        }
    }
    __shared__ bool last;
    const LseState t = block_sums(st, ws);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = {t.m, t.s, t.e1, t.e2};
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // the last block: every partial, rescaled to their largest maximum, then the block's
    const int nb = (int)gridDim.x;
    long long key = LLONG_MAX;
    for (int b = threadIdx.x; b < nb; b += kThermoThreads)
        key = min(key, order_bits(__double_as_longlong(-((volatile LsePart*)part)[b].m)));
    LseState sp{-__longlong_as_double(order_bits(block_min(key, warp_min))), 0.0, 0.0, 0.0};
    for (int b = threadIdx.x; b < nb; b += kThermoThreads) {
        const volatile LsePart* q = (volatile LsePart*)part + b;
        const double qm = q->m;
        if (qm == -INFINITY) continue;
        const double x = qm - sp.m;
        const double f = (__double2hiint(x) & 0x7fffffff) < 0x4085e000 ? exp_short(x, tab) : exp_any(x);
        sp.s += q->s * f;
        sp.e1 += q->e1 * f;
        sp.e2 += q->e2 * f;
    }
    const LseState r = block_sums(sp, ws);
    if (threadIdx.x == 0) {
        const double kB = 0.001987206;  // LIB/statmech.h:26
        const double lnZ = r.m + log(r.s);
        const double Ea = r.e1 / r.s, E2 = r.e2 / r.s;
        const double kT = kB * T;
        const double var = E2 - Ea * Ea;
        fxe_thermo rec;
        rec.temperature = T;
        rec.log_Z = lnZ;
        rec.free_energy = -kT * lnZ;
        rec.mean_energy = Ea;
        rec.mean_energy_sq = E2;
        rec.heat_capacity = var / (kT * kT);
        rec.entropy = (Ea - rec.free_energy) / T;
        rec.std_energy = sqrt(var > 0.0 ? var : 0.0);
        *out = rec;
    }
}

// Blocks of the fixed-scratch pass: one energy per thread, up to four blocks per SM (the device's
// full set at 64 registers); past 1,245,184 energies a block takes several chunks.
void launch_thermo_fixed(const double* e, const int32_t* mult, long n, double beta, double T,
                         LsePart* scratch, fxe_thermo* d_out, cudaStream_t st) {
    long nb = (n + kThermoThreads - 1) / kThermoThreads;
    if (nb > kFixedBlocks) nb = kFixedBlocks;
    if (nb < 1) nb = 1;
    // whole warps
    const long per_block = ((n + nb - 1) / nb + 31) & ~31l;
    nb = (n + per_block - 1) / per_block;
    unsigned* done = reinterpret_cast<unsigned*>(scratch + kFixedBlocks);
    cudaMemsetAsync(done, 0, sizeof(unsigned), st);
    auto* kernel = mult ? thermo_fixed_kernel<true> : thermo_fixed_kernel<false>;
    kernel<<<(int)nb, kThermoThreads, 0, st>>>(e, mult, n, per_block, beta, T, scratch, done, d_out);
}

}  // namespace fxe
