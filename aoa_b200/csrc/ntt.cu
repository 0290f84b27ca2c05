// Entry points of the limb transforms: the split of a call into launches
// (butterfly kinds, chunks, passes) and the small rings.  Kernels and their
// contract: ntt_kernels.cuh.
#include "ntt_kernels.cuh"

namespace aoa {

AOA_NTT_KIND(extern, kButterflyCanonical)
AOA_NTT_KIND(extern, kButterflyLazy)
AOA_NTT_KIND(extern, kButterflyLazyQ1)

void ntt_init(Engine& E) {
  allow_kind<kButterflyCanonical>();
  allow_kind<kButterflyLazy>();
  allow_kind<kButterflyLazyQ1>();
  allow_wo_kernels();
  limb_init(E);
  int sms = 0;
  AOA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, E.device));
  E.num_sms = sms;
}

// the same epilogue as a separate pass over transformed data (small rings)
__global__ void ntt_epilogue_kernel(const uint64_t* data, long poly_stride, int npolys, int nlimbs, int first_prime,
                                    int prime_shift, const PrimeConst* pc, int log_n, const __grid_constant__ NttEpi e) {
  pdl_begin();
  const long N = 1L << log_n;
  const long total = (long)npolys * nlimbs * N;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const long c = i % N;
    const int limb = (int)((i / N) % nlimbs);
    const long p = i / N / nlimbs;
    const int prime = first_prime + (limb >> prime_shift);
    epi_store(e, N, p, limb, prime, c, data[(p * poly_stride + limb) * N + c], pc[prime]);
  }
}

// Small transforms (N < 1024): one CTA per item, the whole limb in shared
// memory, one radix-2 stage per step, canonical (strict) butterflies with the
// same merged tables as the large kernels.
__global__ void ntt_small(NttBatch b, bool fwd) {
  pdl_begin();
  extern __shared__ __align__(16) uint64_t xs[];
  const int N = 1 << b.log_n;
  for (int j = blockIdx.x; j < b.nitems; j += gridDim.x) {
    const int limb = j / b.npolys, p = j % b.npolys;
    const int prime = b.prime_of(limb);
    uint64_t* x = b.data + ((long)p * b.poly_stride + limb) * N;
    const PrimeConst& P = b.pc[prime];
    const uint64_t q = P.q;
    const ShoupW* tw = (fwd ? b.tw : b.itw) + (long)prime * N;
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += blockDim.x) xs[i] = x[i];
    __syncthreads();
    if (fwd) {
      for (int m = 1; m < N; m <<= 1) {
        const int t = N / (2 * m);
        for (int bf = threadIdx.x; bf < N / 2; bf += blockDim.x) {
          const int g = bf / t, l = bf % t, i0 = 2 * g * t + l;
          const uint64_t u = xs[i0], v = shoup(xs[i0 + t], tw[m + g], q);
          xs[i0] = add_mod(u, v, q);
          xs[i0 + t] = sub_mod(u, v, q);
        }
        __syncthreads();
      }
      for (int i = threadIdx.x; i < N; i += blockDim.x) x[i] = xs[i];
    } else {
      for (int m = N / 2; m >= 1; m >>= 1) {
        const int t = N / (2 * m);
        for (int bf = threadIdx.x; bf < N / 2; bf += blockDim.x) {
          const int g = bf / t, l = bf % t, i0 = 2 * g * t + l;
          const uint64_t u = xs[i0], v = xs[i0 + t];
          xs[i0] = add_mod(u, v, q);
          xs[i0 + t] = shoup(sub_mod(u, v, q), tw[m + g], q);
        }
        __syncthreads();
      }
      for (int i = threadIdx.x; i < N; i += blockDim.x) x[i] = shoup(xs[i], P.ninv, P.ninv_sh, q);
    }
  }
}

// the transforms move tiles with bulk / tensor-map copies, which need 16-byte
// aligned addresses: limbs start at data + multiples of N words (N >= 2^10)
static void check_alignment(const uint64_t* data, const NttIo* io) {
  if (((uintptr_t)data & 15) || (io && io->src && ((uintptr_t)io->src & 15)))
    throw AoaError(AOA_ERR_BAD_PARAM, "ntt: device data must be 16-byte aligned");
}

static LimbUse limb_use(const NttTables& T, int first_prime, int nlimbs, int gap, bool forward) {
  auto kind_at = [&](int l) {
    return T.prime_kind ? (int)T.prime_kind[first_prime + (l >> T.prime_shift) + (l ? gap : 0)] : T.kind;
  };
  bool one_lazy = kind_at(0) != kButterflyCanonical;
  for (int l = 1; l < nlimbs && one_lazy && T.prime_kind; l++) one_lazy = kind_at(l) == kind_at(0);
  return !one_lazy ? kLimbOther : T.prime_shift ? kLimbCyclic : forward ? kLimbForward : kLimbOther;
}

// Transform limbs [0, nlimbs) of npolys polys (layout [npolys][poly_stride][N],
// N = 2^T.log_n) with the tables T; limb l under prime first_prime +
// (l >> T.prime_shift).  Large transforms are split into chunks of whole polys
// of at most tune.ntt_chunk_bytes, column and row pass per chunk.
void ntt_batch_tables(const Engine& E, const NttTables& T, uint64_t* data, int npolys, int first_prime, int nlimbs,
                      long poly_stride, bool forward, cudaStream_t st, const NttIo* io) {
  if (npolys <= 0 || nlimbs <= 0) return;
  const int gap = io && nlimbs > 1 ? io->prime_gap : 0;
  if (first_prime < 0 || first_prime + ((nlimbs - 1) >> T.prime_shift) + gap >= E.nprimes)
    throw AoaError(AOA_ERR_BAD_PARAM, "ntt: prime range out of bounds");
  if ((!io || io->epi.mode == kEpiStore) &&
      limb_serves(E, T.log_n, (long)npolys * nlimbs, limb_use(T, first_prime, nlimbs, gap, forward))) {
    check_alignment(data, io);
    limb_transform(E, T, data, npolys, first_prime, nlimbs, poly_stride, forward, io ? *io : NttIo{}, st);
    return;
  }
  if (T.prime_kind && T.log_n >= 10) {
    // Primes of different butterfly kinds (the reference's prime sets put a
    // 63-bit q0 before its 45..55-bit buckets): the limbs run in maximal runs
    // of one kind, the lazy kernels for primes below 2^kLazyPrimeBits (with
    // the shorter remainder where q = 1 mod 2^32), the canonical ones for the
    // rest.  Runs start at prime boundaries; each run's data, source and
    // epilogue limbs are offset by its first limb.
    const long n = 1L << T.log_n;
    auto kind_at = [&](int l) { return (int)T.prime_kind[first_prime + (l >> T.prime_shift) + (l ? gap : 0)]; };
    for (int l0 = 0; l0 < nlimbs;) {
      const int kind = kind_at(l0);
      int l1 = l0 + 1;
      while (l1 < nlimbs && kind_at(l1) == kind) l1++;
      NttTables T2 = T;
      T2.kind = kind;
      T2.prime_kind = nullptr;
      if (l0 == 0 && l1 == nlimbs) {
        ntt_batch_tables(E, T2, data, npolys, first_prime, nlimbs, poly_stride, forward, st, io);
        return;
      }
      NttIo run;
      if (io) run = *io;
      if (run.src) run.src += (long)l0 * n;
      run.epi.limb_base += l0;
      run.part = true;
      if (l0) run.prime_gap = 0;                 // it is in the run's first prime
      ntt_batch_tables(E, T2, data + (long)l0 * n, npolys, first_prime + (l0 >> T.prime_shift) + (l0 ? gap : 0),
                       l1 - l0, poly_stride, forward, st, &run);
      l0 = l1;
    }
    return;
  }
  const NttEpi no_epi{};
  const NttEpi& epi = io ? io->epi : no_epi;
  if (epi.mode != kEpiStore && !forward) throw AoaError(AOA_ERR_BAD_PARAM, "ntt: epilogues are for forward transforms");
  check_alignment(data, io);
  NttBatch b;
  b.tw = T.tw; b.itw = T.itw; b.pc = T.pc; b.err = E.d_err;
  b.spin = E.tune.spin_limit;
  b.log_n = T.log_n;
  b.log_c = T.log_n / 2 + T.split;
  b.log_c = std::max(std::max(5, T.log_n - 10), std::min(std::min(10, T.log_n - 5), b.log_c));
  b.log_r = T.log_n - b.log_c;
  b.first_prime = first_prime; b.prime_shift = T.prime_shift; b.poly_stride = poly_stride;
  b.src = nullptr; b.src_poly_stride = 0; b.poly_base = 0; b.use_tma = 0;
  b.unscaled = io && io->unscaled;
  b.alone = !(io && io->part);
  b.prime_gap = gap;
  const long n = 1L << T.log_n;
  if ((b.unscaled && forward) || ((b.unscaled || gap) && T.log_n < 10))
    throw AoaError(AOA_ERR_BAD_PARAM, "ntt: only inverses of N >= 2^10 leave N^-1 out");
  if (T.log_n < 10) {
    // small rings: the out-of-place source is copied first and the epilogue
    // runs as its own pass
    if (io && io->src)
      AOA_CUDA(cudaMemcpy2DAsync(data, poly_stride * n * 8, io->src, io->src_poly_stride * n * 8,
                                 (size_t)nlimbs * n * 8, npolys, cudaMemcpyDeviceToDevice, st));
    b.npolys = npolys;
    b.nitems = npolys * nlimbs;
    b.data = data;
    const int grid = std::min(b.nitems, 8 * E.num_sms);
    launch_pdl(ntt_small, grid, std::max(32, std::min((int)n / 2, 256)), n * 8, st, b, forward);
    if (epi.mode != kEpiStore) {
      launch_pdl(ntt_epilogue_kernel, 2 * E.num_sms, 256, 0, st, data, poly_stride, npolys, nlimbs, first_prime,
                                                         T.prime_shift, T.pc, T.log_n, epi);
    }
    AOA_CHECK_LAUNCH();
    return;
  }
  const long limb_bytes = 8 * n;
  const long chunk = std::max(1L, E.tune.ntt_chunk_bytes / (limb_bytes * nlimbs));
  for (long c0 = 0; c0 < npolys; c0 += chunk) {
    const int np = (int)std::min<long>(chunk, npolys - c0);
    b.npolys = np;
    b.nitems = np * nlimbs;
    b.data = data + c0 * poly_stride * n;
    b.poly_base = (int)c0;
    NttBatch first = b;                    // the first pass may read out of place
    if (io && io->src) {
      first.src = io->src + c0 * io->src_poly_stride * n;
      first.src_poly_stride = io->src_poly_stride;
    }
    switch (T.kind) {
#define AOA_KIND(K)                                                                   \
  case K:                                                                             \
    if (forward) { run_cols<K>(E, first, true, st); run_rows<K>(E, b, true, st, epi); }  \
    else { run_rows<K>(E, first, false, st, no_epi); run_cols<K>(E, b, false, st); }     \
    break;
      AOA_KIND(kButterflyCanonical) AOA_KIND(kButterflyLazy) AOA_KIND(kButterflyLazyQ1)
#undef AOA_KIND
      default: throw AoaError(AOA_ERR_BAD_PARAM, "ntt: unknown butterfly kind");
    }
  }
  AOA_CHECK_LAUNCH();
}

// Negacyclic limb transforms of the engine's ring (psi^bitrev tables).
void ntt_batch(const Engine& E, uint64_t* data, int npolys, int first_prime, int nlimbs,
               long poly_stride, bool forward, cudaStream_t st) {
  NttTables T;
  T.tw = E.d_tw; T.itw = E.d_itw; T.pc = E.d_pc;
  T.log_n = E.log_n; T.prime_shift = 0; T.kind = std::max(E.ntt_kind, 0);
  T.split = E.tune.ntt_split;
  if (E.ntt_kind < 0) T.prime_kind = E.prime_kind.data();
  ntt_batch_tables(E, T, data, npolys, first_prime, nlimbs, poly_stride, forward, st, nullptr);
}

// Limb transforms with a fused source and / or epilogue (NttIo).
void ntt_batch_io(const Engine& E, uint64_t* data, int npolys, int first_prime, int nlimbs, long poly_stride,
                  bool forward, const NttIo& io, cudaStream_t st) {
  NttTables T;
  T.tw = E.d_tw; T.itw = E.d_itw; T.pc = E.d_pc;
  T.log_n = E.log_n; T.prime_shift = 0; T.kind = std::max(E.ntt_kind, 0);
  T.split = E.tune.ntt_split;
  if (E.ntt_kind < 0) T.prime_kind = E.prime_kind.data();
  ntt_batch_tables(E, T, data, npolys, first_prime, nlimbs, poly_stride, forward, st, &io);
}

}  // namespace aoa
