// Device samplers (the reference's Sampler, aoa-ntt src/cuda/sampler.cu:
// 13-230: sample_uniform, sample_DG, sample_Z0, sample_hw), on a documented
// counter-based generator so that every draw is reproducible from
// (seed, stream, index) on any device or on the host:
//   Philox4x32-10 (Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as
//   easy as 1, 2, 3", SC 2011): 10 rounds over a 128-bit counter with a
//   64-bit key; round: (hi0, lo0) = M0 * c0, (hi1, lo1) = M1 * c2,
//   c = (hi1 ^ c1 ^ k0, lo1, hi0 ^ c3 ^ k1, lo0); key += (W0, W1).
// Counter of draw i in stream s: (i mod 2^32, i >> 32, s mod 2^32, s >> 32);
// key = seed.  Outputs:
//   uniform   residue of limb l at coefficient i = (x3 x2 x1 x0 as a 128-bit
//             integer) mod q, counter index l * N + i (bias < 2^-64; the
//             reference reduces one 64-bit Sobol draw, biased up to q / 2^64)
//   gaussian  Box-Muller on the draw's two 64-bit halves (53-bit uniforms),
//             rounded to the nearest integer (sample_DG rounds a normal draw)
//   ternary   exactly hw entries +-1 at the positions of the hw smallest keys
//             (draw word 0, then the index: no ties), sign from draw bit
//             32; the rest 0 (sample_hw: hw = 64; sample_Z0: hw = N/2)
#include "aoa_internal.h"
#include "async.cuh"

using namespace aoa;

namespace {

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

constexpr uint32_t kPhiloxM0 = 0xD2511F53u, kPhiloxM1 = 0xCD9E8D57u;
constexpr uint32_t kPhiloxW0 = 0x9E3779B9u, kPhiloxW1 = 0xBB67AE85u;

__device__ __forceinline__ uint4 philox(uint64_t index, uint64_t stream, uint64_t seed) {
  uint32_t c0 = (uint32_t)index, c1 = (uint32_t)(index >> 32), c2 = (uint32_t)stream, c3 = (uint32_t)(stream >> 32);
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
  for (int r = 0; r < 10; r++) {
    const uint32_t lo0 = kPhiloxM0 * c0, hi0 = __umulhi(kPhiloxM0, c0);
    const uint32_t lo1 = kPhiloxM1 * c2, hi1 = __umulhi(kPhiloxM1, c2);
    const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
    c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    k0 += kPhiloxW0;
    k1 += kPhiloxW1;
  }
  return make_uint4(c0, c1, c2, c3);
}

__global__ void sample_uniform_kernel(uint64_t* out, long N, int nlimbs, int first_prime, const PrimeConst* pc,
                                      uint64_t seed, uint64_t stream) {
  const long total = N * nlimbs;
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
    const uint4 r = philox((uint64_t)t, stream, seed);
    const uint64_t lo = ((uint64_t)r.y << 32) | r.x, hi = ((uint64_t)r.w << 32) | r.z;
    out[t] = reduce128(lo, hi, pc[first_prime + t / N]);
  }
}

__global__ void sample_gaussian_kernel(int64_t* out, long n, double sigma, uint64_t seed, uint64_t stream) {
  pdl_begin();
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    const uint4 r = philox((uint64_t)t, stream, seed);
    const uint64_t a = ((uint64_t)r.y << 32) | r.x, b = ((uint64_t)r.w << 32) | r.z;
    const double u1 = ((double)(a >> 11) + 1.0) * 0x1.0p-53;        // (0, 1]
    const double u2 = (double)(b >> 11) * 0x1.0p-53;                // [0, 1)
    const double z = sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
    out[t] = (int64_t)llrint(z * sigma);
  }
}

// Radix select of the hw smallest 64-bit keys (random word 0 in the high 32
// bits, the index in the low bits, so all keys differ) by one cluster of eight
// CTAs, 11 bits a pass: every CTA counts its share of the keys, and after a
// cluster barrier each sums the eight histograms through distributed shared
// memory and finds the same digit.  The passes end when every key under the
// prefix is taken, as a rule after the random word's three.  The keys are drawn
// once (up to kSelCache per CTA) while the stream's previous kernel ends.  One
// CTA drawing every key again in each of eight 8-bit passes took 76 us for
// 2^14 keys.
constexpr int kSelThreads = 1024, kSelCtas = 8, kSelBins = 2048;
constexpr long kSelCache = 16384;

__global__ void __cluster_dims__(kSelCtas, 1, 1) __launch_bounds__(kSelThreads)
sample_ternary_kernel(int64_t* out, long n, long hw, uint64_t seed, uint64_t stream) {
  extern __shared__ uint64_t words[];        // random word 0, sign in bit 32
  __shared__ __align__(8) unsigned hist[kSelBins];
  __shared__ unsigned warp_sum[32];
  __shared__ unsigned found_bin, found_need, found_count;
  const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
  const long chunk = (n + kSelCtas - 1) / kSelCtas;
  const long i0 = blockIdx.x * chunk, cnt = max(0L, min(chunk, n - i0));
  const bool cached = chunk <= kSelCache;
  auto draw = [&](long t) {
    const uint4 r = philox((uint64_t)(i0 + t), stream, seed);
    return (uint64_t)r.x | ((uint64_t)(r.y & 1) << 32);
  };
  auto word = [&](long t) { return cached ? words[t] : draw(t); };
  if (cached)
    for (long t = tid; t < cnt; t += kSelThreads) words[t] = draw(t);   // read by the same thread only
  uint64_t prefix = 0, mask = 0, kth = 0;
  unsigned need = (unsigned)hw;              // keys still to take under the current prefix
  const uint32_t h_addr = smem_u32(hist);
  constexpr int kShift[6] = {53, 42, 32, 21, 10, 0};
  for (int d = 0; d < 6 && need > 0; d++) {
    const int shift = kShift[d], width = d % 3 == 2 ? 10 : 11;
    for (int i = tid; i < kSelBins; i += kSelThreads) hist[i] = 0;
    __syncthreads();
    for (long t = tid; t < cnt; t += kSelThreads) {
      const uint64_t k = (word(t) << 32) | (uint64_t)(i0 + t);
      if ((k & mask) == prefix) atomicAdd(&hist[(k >> shift) & ((1u << width) - 1)], 1u);
    }
    cluster_barrier();
    unsigned c0 = 0, c1 = 0;                 // bins 2 tid, 2 tid + 1 of the whole cluster
    for (int r = 0; r < kSelCtas; r++) {
      uint32_t a, x, y;
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(h_addr + tid * 8), "r"(r));
      asm volatile("ld.shared::cluster.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(a));
      c0 += x;
      c1 += y;
    }
    unsigned incl = c0 + c1;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned v = __shfl_up_sync(~0u, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    unsigned before = incl - c0 - c1;        // keys in lower bins
    for (int w = 0; w < warp; w++) before += warp_sum[w];
    if (before < need && need <= before + c0) {
      found_bin = 2 * tid;
      found_need = need - before;
      found_count = c0;
    } else if (before + c0 < need && need <= before + c0 + c1) {
      found_bin = 2 * tid + 1;
      found_need = need - before - c0;
      found_count = c1;
    }
    cluster_barrier();                       // every histogram is read; the digit is visible
    prefix |= (uint64_t)found_bin << shift;
    mask |= (uint64_t)((1u << width) - 1) << shift;
    kth = prefix | ((1ull << shift) - 1);
    need = found_need;
    if (found_count == need) break;          // every key under the prefix is taken
  }
  pdl_begin();
  for (long t = tid; t < cnt; t += kSelThreads) {
    const uint64_t w = word(t), k = (w << 32) | (uint64_t)(i0 + t);
    out[i0 + t] = hw > 0 && k <= kth ? ((w >> 32) ? -1 : 1) : 0;
  }
}

__global__ void signed_to_residues_kernel(const int64_t* in, uint64_t* out, long N, int nlimbs, int first_prime,
                                          const PrimeConst* pc) {
  const long total = N * nlimbs;
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
    const uint64_t q = pc[first_prime + t / N].q;
    const int64_t v = in[t % N];
    const uint64_t m = (uint64_t)(v < 0 ? -v : v) % q;
    out[t] = v < 0 ? (m ? q - m : 0) : m;
  }
}

}  // namespace

extern "C" {

// small signed integers (a secret, noise) -> [nlimbs][N] canonical residues
// under primes first_prime .. (the cast of sample_hw / sample_DG)
int aoa_signed_to_residues(aoa_ctx* c, const int64_t* d_in, uint64_t* d_out, int first_prime, int nlimbs) {
  if (!c || !d_in || !d_out) return fail(AOA_ERR_BAD_PARAM, "null argument");
  return guarded([&] {
    const Engine& E = *c->c.E;
    if (first_prime < 0 || nlimbs < 1 || first_prime + nlimbs > E.nprimes)
      throw AoaError(AOA_ERR_BAD_PARAM, "prime range out of bounds");
    signed_to_residues_kernel<<<2 * E.num_sms, 256, 0, c->c.stream>>>(d_in, d_out, E.N, nlimbs, first_prime, E.d_pc);
    note_launch();
    AOA_CHECK_LAUNCH();
  });
}

int aoa_sample_uniform(aoa_ctx* c, uint64_t* d_out, int first_prime, int nlimbs, uint64_t seed, uint64_t stream) {
  if (!c || !d_out) return fail(AOA_ERR_BAD_PARAM, "null argument");
  return guarded([&] {
    const Engine& E = *c->c.E;
    if (first_prime < 0 || nlimbs < 1 || first_prime + nlimbs > E.nprimes)
      throw AoaError(AOA_ERR_BAD_PARAM, "prime range out of bounds");
    sample_uniform_kernel<<<4 * E.num_sms, 256, 0, c->c.stream>>>(d_out, E.N, nlimbs, first_prime, E.d_pc, seed,
                                                                   stream);
    note_launch();
    AOA_CHECK_LAUNCH();
  });
}

int aoa_sample_gaussian(aoa_ctx* c, int64_t* d_out, long n, double sigma, uint64_t seed, uint64_t stream) {
  if (!c || !d_out || n < 0 || !(sigma >= 0)) return fail(AOA_ERR_BAD_PARAM, "bad argument");
  return guarded([&] {
    if (n == 0) return;
    launch_pdl(sample_gaussian_kernel, 2 * c->c.E->num_sms, 256, 0, c->c.stream, d_out, n, sigma, seed, stream);
    AOA_CHECK_LAUNCH();
  });
}

int aoa_sample_ternary(aoa_ctx* c, int64_t* d_out, long n, long hw, uint64_t seed, uint64_t stream) {
  if (!c || !d_out || n < 0 || hw < 0 || hw > n || n > (1L << 31)) return fail(AOA_ERR_BAD_PARAM, "bad argument");
  return guarded([&] {
    if (n == 0) return;
    const long chunk = (n + kSelCtas - 1) / kSelCtas;
    const size_t smem = chunk <= kSelCache ? (size_t)chunk * 8 : 0;
    AOA_CUDA(cudaFuncSetAttribute(sample_ternary_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(kSelCache * 8)));
    launch_pdl(sample_ternary_kernel, kSelCtas, kSelThreads, smem, c->c.stream, d_out, n, hw, seed, stream);
    AOA_CHECK_LAUNCH();
  });
}

}  // extern "C"
