// Whole-limb transforms of the smaller rings (N = 2^10 .. 2^15): one launch per
// transform, with the work around it in the same launch.
//
// A call on few limbs of a small ring is bound by latency: two passes are two
// launches whose CTAs each load, transform a few microseconds' worth and store.
// Here a thread-block cluster of CL CTAs holds one limb in its shared memory:
// CTA r transforms C / CL columns, sends every row to the CTA that owns it
// (st.shared::cluster), and after one cluster barrier transforms R / CL rows;
// the inverse runs the other way.  The butterflies, their bounds and the tables
// are the pass kernels' (ntt_kernels.cuh), so residues are identical; stages
// run two at a time on words in shared memory.  The limb's prime picks canonical or lazy butterflies inside
// the kernel (a cluster's CTAs share it), so limbs of a 63-bit q_0 and of
// 55-bit primes run side by side instead of in launches of one kind.
//
// Modes fuse what surrounds a transform in HMult and in the automorphisms:
//   kLimbFwd, kLimbInv    plain, in place or from a source
//   kLimbInvUnscaled      the inverse without N^-1 (NttIo::unscaled), as in the
//                         fused inverses whose limbs go on to a basis conversion
//   kLimbTensorInv        d2 = a1 b1, its inverse (ModUp's input)
//   kLimbGaloisInv        permuted c0; permuted c1 and its inverse
//   kLimbKey              forward of a ModUp limb, key product, inverse: one
//                         cluster per (limb, output poly), the forward done by
//                         both; limb `kl` of a rescaling HMult is the top Q
//                         limb of d + d2 key B^-1 (inverse only)
//   kLimbFinish           forward of the corrections, HMult's Q limbs out
//   kLimbGaloisFinish     the same for an automorphism
#include "ks_math.cuh"
#include "ntt_kernels.cuh"

namespace aoa {

namespace {

template <int LR_, int LC_, int LCL_>
struct Limb {
  static constexpr int LR = LR_, LC = LC_;
  static constexpr int R = 1 << LR, C = 1 << LC, CL = 1 << LCL_;
  static constexpr long N = (long)R * C;
  static constexpr int W = C / CL, RW = R / CL;        // columns, rows of a CTA
  static constexpr int M = (int)(N / CL);              // words of a CTA
  static constexpr int P = M / 4 < 512 ? M / 4 : 512;  // threads
  static constexpr int TW = R + RW * (C - 1);          // staged twiddles of one direction: column's, rows' by level
  static constexpr size_t smem(int dirs) { return (size_t)M * 16 + (size_t)dirs * TW * 16; }
  static_assert(LR % 2 == 0 && W >= 4, "column rounds are radix 4");
};

enum {
  kLimbFwd, kLimbInv, kLimbInvUnscaled, kLimbTensorInv, kLimbGaloisInv, kLimbKey, kLimbFinish, kLimbGaloisFinish
};
constexpr bool limb_has_fwd(int mode) { return mode == kLimbFwd || mode >= kLimbKey; }
constexpr bool limb_has_inv(int mode) { return mode >= kLimbInv && mode <= kLimbKey; }

struct LimbArgs {
  uint64_t* data;          // transformed limbs: item (p, l) at data + (p poly_stride + l) N
  long poly_stride;
  const uint64_t* src;     // read from here instead (same form)
  long src_poly_stride;
  const ShoupW *tw, *itw;
  const PrimeConst* pc;
  unsigned* err;
  int npolys, first_prime, prime_shift, prime_gap, spin;   // primes of the limbs as in NttBatch
};

struct NoEnds {};
struct TensorEnds {        // a1 b1 of op p -> D2 + p half
  CtPtrs ptr;
  long half;
  uint64_t* D2;
};
struct GaloisEnds {        // polys 2n: c0 of op p -> R + p half; c1 of op p - n -> R + p half and its inverse
  CtPtrs ptr;
  GaloisList g;
  long half;
  uint64_t* R;
  int n;
};
struct KeyEnds {           // polys 2n: part p / n of op p % n
  KeyPtrs keys;
  long key_half;
  int n, kl;
  // the top limb (index kl)
  CtPtrs ptr;
  long half;
  const uint64_t* D2;
  const ShoupW* binv;
  int level;
  uint64_t* U;             // poly p at U + p N
};
struct FinishEnds {
  CtPtrs ptr;
  long half;
  const uint64_t* D2;
  const uint64_t* key;
  long key_half;
  OutPtrs outp;
  int n;
  const ShoupW *binv, *resc;
};
struct GaloisFinishEnds {
  const uint64_t* R;
  long half;
  KeyPtrs keys;
  long key_half;
  OutPtrs outp;
  int n;
  bool add;                // add to the outputs' words
  const ShoupW* binv;
};
template <int MODE> struct EndsOf { using T = NoEnds; };
template <> struct EndsOf<kLimbTensorInv> { using T = TensorEnds; };
template <> struct EndsOf<kLimbGaloisInv> { using T = GaloisEnds; };
template <> struct EndsOf<kLimbKey> { using T = KeyEnds; };
template <> struct EndsOf<kLimbFinish> { using T = FinishEnds; };
template <> struct EndsOf<kLimbGaloisFinish> { using T = GaloisFinishEnds; };

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void sts64_cluster(uint32_t a, uint64_t v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}

__device__ __forceinline__ long galois_source(long p, long g, int log_n) {   // automorph_ntt_batch's permutation
  const uint32_t br = __brev((uint32_t)p) >> (32 - log_n);
  const long e = ((2L * br + 1) * g) & ((2L << log_n) - 1);
  return (long)(__brev((uint32_t)((e - 1) >> 1)) >> (32 - log_n));
}

// Addresses of a CTA's buffers and twiddles (shared memory).
struct LimbSmem {
  uint32_t col, row, tf, ti;             // tiles [R][W] and [RW][C]; twiddles forward and inverse
};

// Word i of a row sits at i ^ 5 ((i / 16) mod 4): the radix-4 rounds of spans
// 1 and 4 then spread a warp's words over all banks.
__device__ __forceinline__ int row_word(int i) { return i ^ (((i >> 4) & 3) * 5); }

// Two forward stages on words d apart: pairs (0, 2), (1, 3) by w0, then (0, 1)
// by w1 and (2, 3) by w2.
template <int KIND>
__device__ __forceinline__ void ct4(uint64_t (&v)[4], ShoupW w0, ShoupW w1, ShoupW w2, uint64_t q) {
  Bf<KIND>::ct(v[0], v[2], w0, q, true);
  Bf<KIND>::ct(v[1], v[3], w0, q, true);
  Bf<KIND>::ct(v[0], v[1], w1, q, false);
  Bf<KIND>::ct(v[2], v[3], w2, q, false);
}

// The rounds are loops with one copy of their code: a CTA runs each instruction
// a few times only, so an unrolled transform (radix-16 rounds in registers) is
// bound by instruction fetch, 1.6 times slower for HMult at N = 2^12.
template <class L, int KIND>
__device__ __forceinline__ void limb_fwd(const LimbSmem& s, uint32_t rank, uint64_t q) {
  const int tid = threadIdx.x;
  // columns: radix-4 rounds over the rows; the last one sends its words to the rows' CTAs
#pragma unroll 1
  for (int st = 0; st < L::LR; st += 2) {
    const int ld = L::LR - 2 - st, d = 1 << ld;
    const bool last = st == L::LR - 2;
    if (last) cluster_wait();              // every CTA of the cluster has started
#pragma unroll 1
    for (int G = tid; G < L::M / 4; G += L::P) {
      const int w = G % L::W, g = G / L::W, hi = g >> ld, r0 = (hi << (ld + 2)) + (g & (d - 1));
      const uint32_t a = s.col + (r0 * L::W + w) * 8, step = (uint32_t)d * (L::W * 8);
      uint64_t v[4];
#pragma unroll
      for (int j = 0; j < 4; j++) v[j] = lds64(a + j * step);
      const uint32_t t = s.tf + (2 << st) * 16 + 2 * hi * 16;
      ct4<KIND>(v, ldsw(s.tf + ((1 << st) + hi) * 16), ldsw(t), ldsw(t + 16), q);
      if (!last) {
#pragma unroll
        for (int j = 0; j < 4; j++) sts64(a + j * step, v[j]);
      } else {
        const uint32_t c = s.row + row_word(rank * L::W + w) * 8;
#pragma unroll
        for (int j = 0; j < 4; j++)
          sts64_cluster(cluster_addr(c + ((r0 + j) % L::RW) * (L::C * 8), (r0 + j) / L::RW), v[j]);
      }
    }
    if (!last) __syncthreads();
  }
  cluster_arrive();
  cluster_wait();
  // rows: level st of row r has its 2^st twiddles at RW (2^st - 1) + (r 2^st)
  const uint32_t tr = s.tf + L::R * 16;
#pragma unroll 1
  for (int st = 0; st + 1 < L::LC; st += 2) {
    const int ld = L::LC - 2 - st, d = 1 << ld;
#pragma unroll 1
    for (int G = tid; G < L::M / 4; G += L::P) {
      const int g = G % (L::C / 4), r = G / (L::C / 4), hi = g >> ld, i0 = (hi << (ld + 2)) + (g & (d - 1));
      const uint32_t a = s.row + r * (L::C * 8);
      uint64_t v[4];
#pragma unroll
      for (int j = 0; j < 4; j++) v[j] = lds64(a + row_word(i0 + j * d) * 8);
      const uint32_t t0 = tr + (L::RW * ((1 << st) - 1) + (r << st) + hi) * 16;
      const uint32_t t1 = tr + (L::RW * ((2 << st) - 1) + (r << (st + 1)) + 2 * hi) * 16;
      ct4<KIND>(v, ldsw(t0), ldsw(t1), ldsw(t1 + 16), q);
#pragma unroll
      for (int j = 0; j < 4; j++) sts64(a + row_word(i0 + j * d) * 8, v[j]);
    }
    __syncthreads();
  }
  if (L::LC % 2) {                         // an odd last stage
    constexpr int st = L::LC - 1;
#pragma unroll 1
    for (int G = tid; G < L::M / 2; G += L::P) {
      const int hi = G % (L::C / 2), r = G / (L::C / 2);
      const uint32_t a = s.row + (r * L::C + row_word(2 * hi)) * 8, b = s.row + (r * L::C + row_word(2 * hi + 1)) * 8;
      uint64_t x = lds64(a), y = lds64(b);
      Bf<KIND>::ct(x, y, ldsw(tr + (L::RW * ((1 << st) - 1) + (r << st) + hi) * 16), q, true);
      sts64(a, x);
      sts64(b, y);
    }
    __syncthreads();
  }
}

// The row tile (words below 8q on lazy primes) to the finished inverse limb at
// x.  WAIT: the barrier that every CTA of the cluster arrives at when it starts
// is still to be waited for (a forward transform has done so, and its own
// barrier has every column tile read).
template <class L, int KIND, bool WAIT, bool UNSCALED>
__device__ __forceinline__ void limb_inv(const LimbSmem& s, uint32_t rank, uint64_t* x, const PrimeConst& P) {
  const int tid = threadIdx.x;
  const uint64_t q = P.q;
  const uint32_t tr = s.ti + L::R * 16;
  if (L::LC % 2) {
    constexpr int st = L::LC - 1;
#pragma unroll 1
    for (int G = tid; G < L::M / 2; G += L::P) {
      const int hi = G % (L::C / 2), r = G / (L::C / 2);
      const uint32_t a = s.row + (r * L::C + row_word(2 * hi)) * 8, b = s.row + (r * L::C + row_word(2 * hi + 1)) * 8;
      uint64_t u = lds64(a), y = lds64(b);
      Bf<KIND>::gs(u, y, ldsw(tr + (L::RW * ((1 << st) - 1) + (r << st) + hi) * 16), q, 8);
      sts64(a, u);
      sts64(b, y);
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int st = L::LC - L::LC % 2 - 2; st >= 0; st -= 2) {
    const int ld = L::LC - 2 - st, d = 1 << ld;
    if (WAIT && st == 0) cluster_wait();
#pragma unroll 1
    for (int G = tid; G < L::M / 4; G += L::P) {
      const int g = G % (L::C / 4), r = G / (L::C / 4), hi = g >> ld, i0 = (hi << (ld + 2)) + (g & (d - 1));
      const uint32_t a = s.row + r * (L::C * 8);
      uint64_t v[4];
#pragma unroll
      for (int j = 0; j < 4; j++) v[j] = lds64(a + row_word(i0 + j * d) * 8);
      const ShoupW w0 = ldsw(tr + (L::RW * ((1 << st) - 1) + (r << st) + hi) * 16);
      const uint32_t t1 = tr + (L::RW * ((2 << st) - 1) + (r << (st + 1)) + 2 * hi) * 16;
      Bf<KIND>::gs(v[0], v[1], ldsw(t1), q, 8);
      Bf<KIND>::gs(v[2], v[3], ldsw(t1 + 16), q, 8);
      Bf<KIND>::gs(v[0], v[2], w0, q, 8);
      Bf<KIND>::gs(v[1], v[3], w0, q, 8);
      if (st) {
#pragma unroll
        for (int j = 0; j < 4; j++) sts64(a + row_word(i0 + j * d) * 8, v[j]);
      } else {                             // to the columns' CTAs
        const uint32_t c = s.col + (rank * L::RW + r) * (L::W * 8);
#pragma unroll
        for (int j = 0; j < 4; j++)
          sts64_cluster(cluster_addr(c + ((i0 + j * d) % L::W) * 8, (i0 + j * d) / L::W), v[j]);
      }
    }
    if (st) __syncthreads();
  }
  cluster_arrive();
  cluster_wait();
  const ShoupW ninv{P.ninv, P.ninv_sh}, ninv_w1{P.ninv_w1, P.ninv_w1_sh};
#pragma unroll 1
  for (int st = L::LR - 2; st >= 0; st -= 2) {
    const int ld = L::LR - 2 - st, d = 1 << ld;
#pragma unroll 1
    for (int G = tid; G < L::M / 4; G += L::P) {
      const int w = G % L::W, g = G / L::W, hi = g >> ld, r0 = (hi << (ld + 2)) + (g & (d - 1));
      const uint32_t a = s.col + (r0 * L::W + w) * 8, step = (uint32_t)d * (L::W * 8);
      uint64_t v[4];
#pragma unroll
      for (int j = 0; j < 4; j++) v[j] = lds64(a + j * step);
      const uint32_t t = s.ti + (2 << st) * 16 + 2 * hi * 16;
      Bf<KIND>::gs(v[0], v[1], ldsw(t), q, 8);
      Bf<KIND>::gs(v[2], v[3], ldsw(t + 16), q, 8);
      if (st) {
        const ShoupW w0 = ldsw(s.ti + ((1 << st) + hi) * 16);
        Bf<KIND>::gs(v[0], v[2], w0, q, 8);
        Bf<KIND>::gs(v[1], v[3], w0, q, 8);
#pragma unroll
        for (int j = 0; j < 4; j++) sts64(a + j * step, v[j]);
      } else {                             // the last stage, with N^-1 or left unscaled
        if constexpr (UNSCALED) {
          const ShoupW w0 = ldsw(s.ti + 16);
          Bf<KIND>::gs_unscaled(v[0], v[2], w0, q);
          Bf<KIND>::gs_unscaled(v[1], v[3], w0, q);
        } else {
          Bf<KIND>::gs_last(v[0], v[2], ninv, ninv_w1, q);
          Bf<KIND>::gs_last(v[1], v[3], ninv, ninv_w1, q);
        }
        uint64_t* o = x + rank * L::W + w;
#pragma unroll
        for (int j = 0; j < 4; j++) o[(long)(r0 + j * d) * L::C] = v[j];
      }
    }
    if (st) __syncthreads();
  }
}

template <class L, int KIND, int MODE>
__device__ __forceinline__ void limb_run(const LimbArgs& a, const typename EndsOf<MODE>::T& e, const LimbSmem& s,
                                         uint32_t rank, int limb, int p, const PrimeConst& P, int prime) {
  const int tid = threadIdx.x;
  const uint64_t q = P.q;
  const long limb_off = (long)limb * L::N;
  const long row0 = (long)rank * L::M;                     // the CTA's first coefficient (its rows are contiguous)
  uint64_t* x = a.data + (long)p * a.poly_stride * L::N + limb_off;
  auto word = [&](int i) { return s.row + ((i & ~(L::C - 1)) + row_word(i & (L::C - 1))) * 8; };
  [[maybe_unused]] int z = p;
  [[maybe_unused]] bool second = false;
  if constexpr (MODE == kLimbGaloisInv || MODE == kLimbKey || MODE == kLimbFinish || MODE == kLimbGaloisFinish) {
    second = p >= e.n;
    z = second ? p - e.n : p;
  }
  if constexpr (MODE == kLimbKey) {
    if (limb == e.kl) {
      // the top Q limb of d + d2 key B^-1
      const long top = (long)e.level * L::N + row0;
      const uint64_t *A = e.ptr.a[z] + top, *B = e.ptr.b[z] + top, *D = e.D2 + (long)z * e.half + top;
      const uint64_t* key = e.keys.k[z] + (second ? e.key_half : 0) + top;
      const ShoupW bi = e.binv[e.level];
      const bool fit = sums_fit(P);
#pragma unroll 1
      for (int i = tid; i < L::M; i += L::P) {
        const uint64_t k = shoup(key[i], bi, q);
        sts64(word(i), second ? ks_sum3(A[i], A[e.half + i], B[i], B[e.half + i], D[i], k, fit, P)
                              : ks_sum2(A[i], B[i], D[i], k, fit, P));
      }
      __syncthreads();
      limb_inv<L, KIND, true, false>(s, rank, e.U + (long)p * L::N, P);
      return;
    }
    limb_fwd<L, KIND>(s, rank, q);
    const uint64_t* key = e.keys.k[z] + (second ? e.key_half : 0) + (long)prime * L::N + row0;
#pragma unroll 2
    for (int i = tid; i < L::M; i += L::P)
      sts64(word(i), mul_mod(Bf<KIND>::fwd_out(lds64(word(i)), q), key[i], P));
    __syncthreads();
    limb_inv<L, KIND, false, true>(s, rank, x, P);
  } else if constexpr (MODE == kLimbFwd) {
    limb_fwd<L, KIND>(s, rank, q);
#pragma unroll 2
    for (int i = tid; i < L::M; i += L::P) x[row0 + i] = Bf<KIND>::fwd_out(lds64(word(i)), q);
  } else if constexpr (MODE == kLimbFinish) {
    limb_fwd<L, KIND>(s, rank, q);
    const long o = limb_off + row0;
    const uint64_t *A = e.ptr.a[z] + o, *B = e.ptr.b[z] + o, *D = e.D2 + (long)z * e.half + o;
    const uint64_t* key = e.key + (second ? e.key_half : 0) + o;
    uint64_t* out = e.outp.p[p] + o;
    const ShoupW bi = e.binv[limb], rs = e.resc ? e.resc[limb] : bi;
    const bool fit = sums_fit(P);
#pragma unroll 2
    for (int i = tid; i < L::M; i += L::P) {
      const uint64_t y = Bf<KIND>::fwd_out(lds64(word(i)), q), k = shoup(key[i], bi, q);
      const uint64_t sum = second ? ks_sum3(A[i], A[e.half + i], B[i], B[e.half + i], D[i], k, fit, P)
                                  : ks_sum2(A[i], B[i], D[i], k, fit, P);
      out[i] = e.resc ? shoup(sub_mod(sum, y, q), rs, q) : sub_mod(sum, shoup(y, bi, q), q);
    }
  } else if constexpr (MODE == kLimbGaloisFinish) {
    limb_fwd<L, KIND>(s, rank, q);
    const long o = limb_off + row0;
    const uint64_t *R0 = e.R + (long)z * e.half + o, *X = e.R + (long)(e.n + z) * e.half + o;
    const uint64_t* key = e.keys.k[z] + (second ? e.key_half : 0) + o;
    uint64_t* out = e.outp.p[p] + o;
    const ShoupW bi = e.binv[limb];
#pragma unroll 2
    for (int i = tid; i < L::M; i += L::P) {
      const uint64_t y = Bf<KIND>::fwd_out(lds64(word(i)), q);
      const uint64_t d = shoup(sub_mod(mul_mod(X[i], key[i], P), y, q), bi, q);
      const uint64_t c = second ? d : add_mod(R0[i], d, q);
      out[i] = e.add ? add_mod(out[i], c, q) : c;
    }
  } else {
    if constexpr (MODE == kLimbInv || MODE == kLimbInvUnscaled) {
      const uint64_t* src = (a.src ? a.src + (long)p * a.src_poly_stride * L::N + limb_off : x) + row0;
#pragma unroll 4
      for (int i = tid; i < L::M; i += L::P) sts64(word(i), src[i]);
    } else if constexpr (MODE == kLimbTensorInv) {
      const long o = limb_off + row0;
      const uint64_t *A = e.ptr.a[p] + e.half + o, *B = e.ptr.b[p] + e.half + o;
      uint64_t* D = e.D2 + (long)p * e.half + o;
#pragma unroll 2
      for (int i = tid; i < L::M; i += L::P) {
        const uint64_t d = mul_mod(A[i], B[i], P);
        D[i] = d;
        sts64(word(i), d);
      }
    } else {
      const uint64_t* in = e.ptr.a[z] + (second ? e.half : 0) + limb_off;
      uint64_t* R = e.R + (long)p * e.half + limb_off + row0;
      const long g = e.g.g[z];
#pragma unroll 2
      for (int i = tid; i < L::M; i += L::P) {
        const uint64_t d = in[galois_source(row0 + i, g, L::LR + L::LC)];
        R[i] = d;
        if (second) sts64(word(i), d);
      }
      if (!second) {                       // c0: the permutation alone
        cluster_wait();
        return;
      }
      x = a.data + (long)z * a.poly_stride * L::N + limb_off;
    }
    __syncthreads();
    limb_inv<L, KIND, true, MODE != kLimbInv>(s, rank, x, P);
  }
}

template <class L, int MODE>
__global__ void __launch_bounds__(L::P, 1)
limb_kernel(const __grid_constant__ LimbArgs a, const __grid_constant__ typename EndsOf<MODE>::T e) {
  extern __shared__ __align__(128) uint64_t dyn[];
  __shared__ __align__(8) uint64_t mbar[2];                // [0] twiddles, [1] the column tile
  constexpr bool FWD = limb_has_fwd(MODE), INV = limb_has_inv(MODE);
  const int tid = threadIdx.x;
  const uint32_t rank = blockIdx.x % L::CL;
  const int item = blockIdx.x / L::CL, limb = item / a.npolys, p = item % a.npolys;
  int prime = a.first_prime + (limb >> a.prime_shift) + (limb ? a.prime_gap : 0);
  bool fwd = FWD;
  if constexpr (MODE == kLimbKey)
    if (limb == e.kl) {                    // the top Q limb: inverse only
      prime = e.level;
      fwd = false;
    }
  LimbSmem s;
  s.col = smem_u32(dyn);
  s.row = s.col + L::M * 8;
  s.tf = s.row + L::M * 8;
  s.ti = FWD ? s.tf + L::TW * 16 : s.tf;
  if (tid == 0) {
    mbar_init(&mbar[0], 1);
    mbar_init(&mbar[1], 1);
    mbar_init_fence();
    // the twiddles are constants: their copies run while the previous kernel ends
    mbar_expect_tx(&mbar[0], (unsigned)((fwd ? 1 : 0) + (INV ? 1 : 0)) * (L::TW * 16));
    for (int dir = 0; dir < 2; dir++) {
      if (dir ? !INV : !fwd) continue;
      const ShoupW* tw = (dir ? a.itw : a.tw) + (long)prime * L::N;
      uint32_t to = dir ? s.ti : s.tf;
      bulk_g2s(to, tw, L::R * 16, &mbar[0]);
      to += L::R * 16;
      for (int st = 0; st < L::LC; st++) {                 // level st of the CTA's rows is contiguous
        bulk_g2s(to, tw + ((long)(L::R + rank * L::RW) << st), (L::RW << st) * 16, &mbar[0]);
        to += (L::RW << st) * 16;
      }
    }
  }
  __syncthreads();
  cluster_arrive();
  pdl_begin();
  if (fwd) {
    const int sp = MODE == kLimbKey ? p % (a.npolys / 2) : p;
    const uint64_t* src = (a.src ? a.src + sp * a.src_poly_stride * L::N : a.data + sp * a.poly_stride * L::N) +
                          (long)limb * L::N;
    if (tid == 0) mbar_expect_tx(&mbar[1], (unsigned)(L::M * 8));
    for (int r = tid; r < L::R; r += L::P)
      bulk_g2s(s.col + r * (L::W * 8), src + (long)r * L::C + rank * L::W, L::W * 8, &mbar[1]);
  }
  // an expired wait is recorded and waited for once more with the default
  // bound; the CTA goes on (its cluster waits for it) with whatever arrived
  if (!mbar_wait(&mbar[0], 0, a.spin) || (fwd && !mbar_wait(&mbar[1], 0, a.spin))) {
    atomicOr(a.err, kErrWaitTimeout);
    mbar_wait(&mbar[0], 0);
    if (fwd) mbar_wait(&mbar[1], 0);
  }
  __syncwarp();
  const PrimeConst P = a.pc[prime];
  if (lazy_prime(P.q)) limb_run<L, kButterflyLazy, MODE>(a, e, s, rank, limb, p, P, prime);
  else limb_run<L, kButterflyCanonical, MODE>(a, e, s, rank, limb, p, P, prime);
}

template <class L, int MODE>
void limb_launch(const LimbArgs& a, const typename EndsOf<MODE>::T& e, int nlimbs, cudaStream_t st) {
  constexpr size_t smem = L::smem((limb_has_fwd(MODE) ? 1 : 0) + (limb_has_inv(MODE) ? 1 : 0));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(nlimbs * a.npolys * L::CL));
  cfg.blockDim = dim3(L::P);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = L::CL;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  AOA_CUDA(cudaLaunchKernelEx(&cfg, limb_kernel<L, MODE>, a, e));
  note_launch();
}

// the split of each ring
using Limb10 = Limb<4, 6, 1>;
using Limb11 = Limb<6, 5, 1>;
using Limb12 = Limb<6, 6, 2>;
using Limb13 = Limb<6, 7, 2>;
using Limb14 = Limb<8, 6, 2>;
using Limb15 = Limb<8, 7, 3>;

template <int MODE>
void limb_dispatch(int log_n, const LimbArgs& a, const typename EndsOf<MODE>::T& e, int nlimbs, cudaStream_t st) {
  if (nlimbs <= 0 || a.npolys <= 0) return;
  switch (log_n) {
    case 10: limb_launch<Limb10, MODE>(a, e, nlimbs, st); break;
    case 11: limb_launch<Limb11, MODE>(a, e, nlimbs, st); break;
    case 12: limb_launch<Limb12, MODE>(a, e, nlimbs, st); break;
    case 13: limb_launch<Limb13, MODE>(a, e, nlimbs, st); break;
    case 14: limb_launch<Limb14, MODE>(a, e, nlimbs, st); break;
    case 15: limb_launch<Limb15, MODE>(a, e, nlimbs, st); break;
    default: throw AoaError(AOA_ERR_BAD_PARAM, "whole-limb transforms are for N = 2^10 .. 2^15");
  }
}

template <class L, int MODE>
void limb_allow() {
  constexpr size_t smem = L::smem((limb_has_fwd(MODE) ? 1 : 0) + (limb_has_inv(MODE) ? 1 : 0));
  AOA_CUDA(cudaFuncSetAttribute(limb_kernel<L, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
}

template <class L>
void limb_allow_all() {
  limb_allow<L, kLimbFwd>();
  limb_allow<L, kLimbInv>();
  limb_allow<L, kLimbInvUnscaled>();
  limb_allow<L, kLimbTensorInv>();
  limb_allow<L, kLimbGaloisInv>();
  limb_allow<L, kLimbKey>();
  limb_allow<L, kLimbFinish>();
  limb_allow<L, kLimbGaloisFinish>();
}

LimbArgs limb_args(const Engine& E) {
  LimbArgs a{};
  a.tw = E.d_tw;
  a.itw = E.d_itw;
  a.pc = E.d_pc;
  a.err = E.d_err;
  a.spin = E.tune.spin_limit;
  return a;
}

}  // namespace

void limb_init(const Engine&) {
  limb_allow_all<Limb10>();
  limb_allow_all<Limb11>();
  limb_allow_all<Limb12>();
  limb_allow_all<Limb13>();
  limb_allow_all<Limb14>();
  limb_allow_all<Limb15>();
}

// Up to how many limb transforms the whole-limb kernels are faster than the two
// passes, which have the higher throughput once the chip is full.  Measured on
// both sides of each line (us, two passes -> whole limbs, one B200):
//   forward, one lazy kind: 2^11, 1024 limbs 40 -> 31; 2^12, 112 11.1 -> 10.1, 150
//     12.2 -> 13.3, 336 20.7 -> 23.8; 2^13, 64 13.9 -> 12.3, 96 16.4 -> 16.6 (four
//     HMults with 68 limbs 93.0 -> 91.4), 128 18.4 -> 21.6; 2^14, 32 (a cluster of
//     four on every SM) 12.5 -> 11.0, 36 12.6 -> 21.0, 64 21.4 -> 22.1; 2^15, 1 to 8
//     8.5 -> 11.0, but within an HMult of 4 or 5 limbs, whose corrections are 6 or 8,
//     114.4 -> 111.9 and 123.5 -> 118.4;
//   DGT limbs of one lazy kind, with the twist: 2^11, 512 22.3 -> 21.6, 608 24.0 ->
//     26.3; 2^12, 448 forward 37.2 -> 38.7, inverse 41.3 -> 36.2; 2^13, 128 28.3 ->
//     26.3, 160 31.7 -> 34.1; 2^14, 32 16.1 -> 14.4, 48 18.0 -> 26.2; 2^15, 8 17.4
//     -> 13.9, 16 19.7 -> 26.5;
//   other inverses, canonical limbs and calls of several kinds, which take two
//     launches per kind: inverse of one kind 2^12, 448 30.0 -> 27.8, 672 39.3 ->
//     40.0; 2^13, 128 21.3 -> 20.1, 160 22.3 -> 24.6; 2^14, 64 24.3 -> 20.5, 80 26.9
//     -> 30.2; 2^15, 6 8.8 -> 10.6, 8 15.8 -> 10.8, 16 17.4 -> 20.9; forward of
//     63-bit and 55-bit primes 2^12, 448 35.3 -> 32.0, 672 43.9 -> 46.2; 2^13, 128
//     35.1 -> 22.8; 2^14, 64 37.0 -> 24.4; 2^15, 8 29.0 -> 13.5;
//   fused, by the 2 n (kl + 1) key-product limbs of a key switch: HMult 2^12, 320
//     138 -> 103; 2^13, 110 105 -> 98, 150 120 -> 120, 196 168 -> 179; 2^14, 60 113
//     -> 94, 100 142 -> 152; rotation 2^14, 56 110 -> 109, 80 136 -> 140; 2^15, 16
//     83.9 -> 85.8, 24 98 -> 110; HMult 2^15, 20 95 -> 90, 30 107 -> 98.
bool limb_serves(const Engine& E, int log_n, long items, LimbUse use) {
  constexpr long kMost[4][6] = {{1024, 1024, 128, 96, 32, 8},     // kLimbForward; log_n = 10 .. 15
                                {1024, 512, 448, 128, 32, 8},     // kLimbCyclic
                                {1024, 1024, 448, 128, 64, 8},    // kLimbOther
                                {1024, 1024, 320, 112, 56, 20}};  // kLimbFused
  const bool on = E.tune.ntt_whole == 2 || (E.tune.ntt_whole == 1 && E.tune.default_shape());
  return on && log_n >= 10 && log_n <= 15 && items <= kMost[use][log_n - 10];
}

void limb_transform(const Engine& E, const NttTables& T, uint64_t* data, int npolys, int first_prime, int nlimbs,
                    long poly_stride, bool forward, const NttIo& io, cudaStream_t st) {
  LimbArgs a = limb_args(E);
  a.tw = T.tw;
  a.itw = T.itw;
  a.pc = T.pc;
  a.data = data;
  a.poly_stride = poly_stride;
  a.src = io.src;
  a.src_poly_stride = io.src_poly_stride;
  a.prime_gap = io.prime_gap;
  a.npolys = npolys;
  a.first_prime = first_prime;
  a.prime_shift = T.prime_shift;
  if (forward) limb_dispatch<kLimbFwd>(T.log_n, a, NoEnds{}, nlimbs, st);
  else if (io.unscaled) limb_dispatch<kLimbInvUnscaled>(T.log_n, a, NoEnds{}, nlimbs, st);
  else limb_dispatch<kLimbInv>(T.log_n, a, NoEnds{}, nlimbs, st);
}

void limb_tensor_inv(const Engine& E, const CtPtrs& ptr, long half, uint64_t* D2, uint64_t* T, int n, int nlimbs,
                     cudaStream_t st) {
  LimbArgs a = limb_args(E);
  a.data = T;
  a.poly_stride = half >> E.log_n;
  a.npolys = n;
  TensorEnds e;
  e.ptr = ptr;
  e.half = half;
  e.D2 = D2;
  limb_dispatch<kLimbTensorInv>(E.log_n, a, e, nlimbs, st);
}

void limb_galois_inv(const Engine& E, const CtPtrs& ptr, const GaloisList& g, long half, uint64_t* R, uint64_t* T,
                     int n, int nlimbs, cudaStream_t st) {
  LimbArgs a = limb_args(E);
  a.data = T;
  a.poly_stride = half >> E.log_n;
  a.npolys = 2 * n;
  GaloisEnds e;
  e.ptr = ptr;
  e.g = g;
  e.half = half;
  e.R = R;
  e.n = n;
  limb_dispatch<kLimbGaloisInv>(E.log_n, a, e, nlimbs, st);
}

void limb_key(const Engine& E, const uint64_t* UB, uint64_t* KS, long ks_stride, const KeyPtrs& keys, int n,
              const CtPtrs* ptr, long half, const uint64_t* D2, uint64_t* U, int level, cudaStream_t st) {
  LimbArgs a = limb_args(E);
  a.data = KS;
  a.poly_stride = ks_stride >> E.log_n;
  a.src = UB;
  a.src_poly_stride = E.kl;
  a.npolys = 2 * n;
  a.first_prime = E.k;
  KeyEnds e{};
  e.keys = keys;
  e.key_half = (long)E.nprimes * E.N;
  e.n = n;
  e.kl = E.kl;
  if (ptr) {
    e.ptr = *ptr;
    e.half = half;
    e.D2 = D2;
    e.binv = E.rns.moddown_binv;
    e.level = level;
    e.U = U;
  }
  limb_dispatch<kLimbKey>(E.log_n, a, e, E.kl + (ptr ? 1 : 0), st);
}

void limb_finish(const Engine& E, uint64_t* Y, const CtPtrs& ptr, long half, const uint64_t* D2, const uint64_t* key,
                 const OutPtrs& outp, int n, int nlimbs, int rescale_level, cudaStream_t st) {
  LimbArgs a = limb_args(E);
  a.data = Y;
  a.poly_stride = half >> E.log_n;
  a.npolys = 2 * n;
  FinishEnds e;
  e.ptr = ptr;
  e.half = half;
  e.D2 = D2;
  e.key = key;
  e.key_half = (long)E.nprimes * E.N;
  e.outp = outp;
  e.n = n;
  e.binv = E.rns.moddown_binv;
  e.resc = rescale_level > 0 ? E.rns.resc_inv + (long)rescale_level * E.k : nullptr;
  limb_dispatch<kLimbFinish>(E.log_n, a, e, nlimbs, st);
}

void limb_galois_finish(const Engine& E, uint64_t* Y, const uint64_t* R, long half, const KeyPtrs& keys,
                        const OutPtrs& outp, int n, int nlimbs, bool add, cudaStream_t st) {
  LimbArgs a = limb_args(E);
  a.data = Y;
  a.poly_stride = half >> E.log_n;
  a.npolys = 2 * n;
  GaloisFinishEnds e;
  e.R = R;
  e.half = half;
  e.keys = keys;
  e.key_half = (long)E.nprimes * E.N;
  e.outp = outp;
  e.n = n;
  e.add = add;
  e.binv = E.rns.moddown_binv;
  limb_dispatch<kLimbGaloisFinish>(E.log_n, a, e, nlimbs, st);
}

}  // namespace aoa
