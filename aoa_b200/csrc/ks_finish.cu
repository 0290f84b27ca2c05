// The Q limbs of HMult and of the Galois automorphisms, transform domain
// (ckks_mul_without_rescale, aoa-ntt src/ckks/ckks.cpp:300-347; ckks_rotate_left
// & co., ckks.cpp:953-1040).
//
// The key products of the Q limbs never leave the domain the result is in, so
// they are formed where the result is: one pass reads the operands, d2 (or the
// permuted c1), the key and the corrections and writes both output polys.
// Bound by HBM: 9 words per coefficient and product (a0 a1 b0 b1 d2 y0 y1 in,
// c0 c1 out) besides the key, where a tensor kernel writing d0 d1 d2, key
// products written out and a combine kernel reading all of them moved 18.
// A thread holds two neighbouring coefficients (16-byte loads: limbs start at
// multiples of N words of 256-byte aligned allocations) and loops over the
// products of the launch, so that each key word is read and scaled by B^-1
// once for all of them.
#include "async.cuh"
#include "ks_math.cuh"

namespace aoa {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ ulonglong2 ld2(const uint64_t* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ void st2(uint64_t* p, uint64_t x, uint64_t y) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(x, y);
}

// d2 = a1 b1 of op z = blockIdx.z, limb blockIdx.y
__global__ void __launch_bounds__(kThreads) tensor_d2(const __grid_constant__ CtPtrs ptr, long half, uint64_t* D2,
                                                      const PrimeConst* pc, int log_n) {
  pdl_begin();
  const int z = blockIdx.z;
  const PrimeConst P = pc[blockIdx.y];
  const long off = ((long)blockIdx.y << log_n) + ((long)blockIdx.x * kThreads + threadIdx.x) * 2;
  const ulonglong2 x = ld2(ptr.a[z] + half + off), y = ld2(ptr.b[z] + half + off);
  st2(D2 + (long)z * half + off, mul_mod(x.x, y.x, P), mul_mod(x.y, y.y, P));
}

// Limb `level` of d + ModDown's Q part (no correction): U[poly][z] = limb
// `level` of (a0 b0 + d2 kb B^-1, a0 b1 + a1 b0 + d2 ka B^-1), polys u_stride apart
__global__ void __launch_bounds__(kThreads) hmult_top(const __grid_constant__ CtPtrs ptr, long half,
                                                      const uint64_t* D2, const uint64_t* key, long key_half,
                                                      uint64_t* U, long u_stride, int n, int level, const ShoupW* binv,
                                                      const PrimeConst* pc, int log_n) {
  pdl_begin();
  const long N = 1L << log_n;
  const int z = blockIdx.z;
  const PrimeConst P = pc[level];
  const bool fit = sums_fit(P);
  const ShoupW bi = binv[level];
  const long c = (long)blockIdx.x * kThreads + threadIdx.x, off = (long)level * N + c;
  const uint64_t kb = shoup(key[off], bi, P.q), ka = shoup(key[key_half + off], bi, P.q);
  const uint64_t *a = ptr.a[z] + off, *b = ptr.b[z] + off;
  const uint64_t a0 = a[0], a1 = a[half], b0 = b[0], b1 = b[half], d2 = D2[(long)z * half + off];
  U[z * u_stride + c] = ks_sum2(a0, b0, d2, kb, fit, P);
  U[(n + z) * u_stride + c] = ks_sum3(a0, a1, b0, b1, d2, ka, fit, P);
}

// out = (d + d2 key B^-1 - y) q_l^-1 (RESC, y = the merged ModDown + rescale
// correction) or d + (d2 key - y) B^-1, limb blockIdx.y of every op; y of
// (poly, z) at Y + (poly n + z) half.
template <bool RESC>
__global__ void __launch_bounds__(kThreads) hmult_finish(const __grid_constant__ CtPtrs ptr, long half,
                                                         const uint64_t* D2, const uint64_t* key, long key_half,
                                                         const uint64_t* Y, const __grid_constant__ OutPtrs outp,
                                                         int n, const ShoupW* binv, const ShoupW* resc,
                                                         const PrimeConst* pc, int log_n) {
  pdl_begin();
  const int i = blockIdx.y;
  const PrimeConst P = pc[i];
  const uint64_t q = P.q;
  const bool fit = sums_fit(P);
  const ShoupW bi = binv[i], rs = RESC ? resc[i] : bi;
  const long off = ((long)i << log_n) + ((long)blockIdx.x * kThreads + threadIdx.x) * 2;
  ulonglong2 kb = ld2(key + off), ka = ld2(key + key_half + off);
  kb.x = shoup(kb.x, bi, q);
  kb.y = shoup(kb.y, bi, q);
  ka.x = shoup(ka.x, bi, q);
  ka.y = shoup(ka.y, bi, q);
  for (int z = blockIdx.z; z < n; z += gridDim.z) {
    const ulonglong2 a0 = ld2(ptr.a[z] + off), a1 = ld2(ptr.a[z] + half + off);
    const ulonglong2 b0 = ld2(ptr.b[z] + off), b1 = ld2(ptr.b[z] + half + off);
    const ulonglong2 d2 = ld2(D2 + (long)z * half + off);
    const ulonglong2 y0 = ld2(Y + (long)z * half + off), y1 = ld2(Y + (long)(n + z) * half + off);
    const uint64_t c0 = ks_sum2(a0.x, b0.x, d2.x, kb.x, fit, P), e0 = ks_sum2(a0.y, b0.y, d2.y, kb.y, fit, P);
    const uint64_t c1 = ks_sum3(a0.x, a1.x, b0.x, b1.x, d2.x, ka.x, fit, P);
    const uint64_t e1 = ks_sum3(a0.y, a1.y, b0.y, b1.y, d2.y, ka.y, fit, P);
    if (RESC) {
      st2(outp.p[z] + off, shoup(sub_mod(c0, y0.x, q), rs, q), shoup(sub_mod(e0, y0.y, q), rs, q));
      st2(outp.p[n + z] + off, shoup(sub_mod(c1, y1.x, q), rs, q), shoup(sub_mod(e1, y1.y, q), rs, q));
    } else {
      st2(outp.p[z] + off, sub_mod(c0, shoup(y0.x, bi, q), q), sub_mod(e0, shoup(y0.y, bi, q), q));
      st2(outp.p[n + z] + off, sub_mod(c1, shoup(y1.x, bi, q), q), sub_mod(e1, shoup(y1.y, bi, q), q));
    }
  }
}

// out0 = r0 + (x kb - y0) B^-1, out1 = (x ka - y1) B^-1 with r0 = R, x = R + n
// half the permuted polys of op z at op stride half; key of op z keys.k[z].
// add: the outputs' words are added to (a rotate-and-sum step).
template <bool ONE_KEY>
__global__ void __launch_bounds__(kThreads) galois_finish(const uint64_t* R, long half,
                                                          const __grid_constant__ KeyPtrs keys, long key_half,
                                                          const uint64_t* Y, const __grid_constant__ OutPtrs outp,
                                                          int n, bool add, const ShoupW* binv, const PrimeConst* pc,
                                                          int log_n) {
  pdl_begin();
  const int i = blockIdx.y;
  const PrimeConst P = pc[i];
  const uint64_t q = P.q;
  const ShoupW bi = binv[i];
  const long off = ((long)i << log_n) + ((long)blockIdx.x * kThreads + threadIdx.x) * 2;
  ulonglong2 kb, ka;
  if (ONE_KEY) {
    kb = ld2(keys.k[0] + off);
    ka = ld2(keys.k[0] + key_half + off);
  }
  for (int z = blockIdx.z; z < n; z += gridDim.z) {
    if (!ONE_KEY) {
      kb = ld2(keys.k[z] + off);
      ka = ld2(keys.k[z] + key_half + off);
    }
    const ulonglong2 r0 = ld2(R + (long)z * half + off), x = ld2(R + (long)(n + z) * half + off);
    const ulonglong2 y0 = ld2(Y + (long)z * half + off), y1 = ld2(Y + (long)(n + z) * half + off);
    ulonglong2 c0, c1;
    c0.x = add_mod(r0.x, shoup(sub_mod(mul_mod(x.x, kb.x, P), y0.x, q), bi, q), q);
    c0.y = add_mod(r0.y, shoup(sub_mod(mul_mod(x.y, kb.y, P), y0.y, q), bi, q), q);
    c1.x = shoup(sub_mod(mul_mod(x.x, ka.x, P), y1.x, q), bi, q);
    c1.y = shoup(sub_mod(mul_mod(x.y, ka.y, P), y1.y, q), bi, q);
    if (add) {
      const ulonglong2 o0 = ld2(outp.p[z] + off), o1 = ld2(outp.p[n + z] + off);
      c0.x = add_mod(c0.x, o0.x, q);
      c0.y = add_mod(c0.y, o0.y, q);
      c1.x = add_mod(c1.x, o1.x, q);
      c1.y = add_mod(c1.y, o1.y, q);
    }
    st2(outp.p[z] + off, c0.x, c0.y);
    st2(outp.p[n + z] + off, c1.x, c1.y);
  }
}

// ---- Gaussian integers (DGT contexts) ----------------------------------------------
// A limb's planes re | im of H = N/2 words; one thread holds one Gaussian
// integer.  A complex product sum takes one reduction per component for up to
// four word products (4 q^2 in one Barrett step's range, as above).
struct Gi {
  uint64_t r, i;
};
__device__ __forceinline__ Gi gi_ld(const uint64_t* p, int H) { return Gi{p[0], p[H]}; }

__device__ __forceinline__ Gi gi_mulmod(Gi a, Gi b, const PrimeConst& P) {
  const uint64_t q = P.q;
  const uint64_t s1 = mul_mod(a.r, b.r, P), s2 = mul_mod(a.i, b.i, P);
  const uint64_t s3 = mul_mod(add_mod(a.r, a.i, q), add_mod(b.r, b.i, q), P);
  return Gi{sub_mod(s1, s2, q), sub_mod(s3, add_mod(s1, s2, q), q)};
}

// a b + c d mod q
__device__ __forceinline__ Gi gi_sum2(Gi a, Gi b, Gi c, Gi d, bool fit, const PrimeConst& P) {
  const uint64_t q = P.q;
  if (!fit) {
    const Gi x = gi_mulmod(a, b, P), y = gi_mulmod(c, d, P);
    return Gi{add_mod(x.r, y.r, q), add_mod(x.i, y.i, q)};
  }
  Gi s;
  uint64_t lo = a.r * b.r, hi = __umul64hi(a.r, b.r);
  mac_wide(lo, hi, q - a.i, b.i);
  mac_wide(lo, hi, c.r, d.r);
  mac_wide(lo, hi, q - c.i, d.i);
  s.r = barrett_wide(lo, hi, q, P.bar_mu, (uint32_t)P.bar_sh);
  lo = a.r * b.i;
  hi = __umul64hi(a.r, b.i);
  mac_wide(lo, hi, a.i, b.r);
  mac_wide(lo, hi, c.r, d.i);
  mac_wide(lo, hi, c.i, d.r);
  s.i = barrett_wide(lo, hi, q, P.bar_mu, (uint32_t)P.bar_sh);
  return s;
}

__device__ __forceinline__ Gi gi_add(Gi a, Gi b, uint64_t q) { return Gi{add_mod(a.r, b.r, q), add_mod(a.i, b.i, q)}; }
__device__ __forceinline__ Gi gi_scale(Gi a, ShoupW w, uint64_t q) { return Gi{shoup(a.r, w, q), shoup(a.i, w, q)}; }

__global__ void __launch_bounds__(kThreads) gi_tensor_d2(const __grid_constant__ CtPtrs ptr, long half, uint64_t* D2,
                                                         const PrimeConst* pc, int log_n) {
  pdl_begin();
  const int H = 1 << (log_n - 1), z = blockIdx.z;
  const PrimeConst P = pc[blockIdx.y];
  const long off = ((long)blockIdx.y << log_n) + (long)blockIdx.x * kThreads + threadIdx.x;
  const Gi a = gi_ld(ptr.a[z] + half + off, H), b = gi_ld(ptr.b[z] + half + off, H);
  const Gi d = gi_mulmod(a, b, P);
  D2[(long)z * half + off] = d.r;
  D2[(long)z * half + off + H] = d.i;
}

// hmult_top and hmult_finish for Gaussian integers; MODE 0: the top limb (no
// correction, out = U of stride N), 1: rescale, 2: without rescale
template <int MODE>
__global__ void __launch_bounds__(kThreads) gi_finish(const __grid_constant__ CtPtrs ptr, long half,
                                                      const uint64_t* D2, const uint64_t* key, long key_half,
                                                      const uint64_t* Y, const __grid_constant__ OutPtrs outp,
                                                      uint64_t* U, int n, int limb0, const ShoupW* binv,
                                                      const ShoupW* resc, const PrimeConst* pc, int log_n) {
  pdl_begin();
  const int H = 1 << (log_n - 1), i = limb0 + blockIdx.y;
  const PrimeConst P = pc[i];
  const uint64_t q = P.q;
  const bool fit = sums_fit(P);
  const ShoupW bi = binv[i], rs = MODE == 1 ? resc[i] : bi;
  const long c = (long)blockIdx.x * kThreads + threadIdx.x, off = ((long)i << log_n) + c;
  const Gi kb = gi_scale(gi_ld(key + off, H), bi, q), ka = gi_scale(gi_ld(key + key_half + off, H), bi, q);
  for (int z = blockIdx.z; z < n; z += gridDim.z) {
    const Gi a0 = gi_ld(ptr.a[z] + off, H), a1 = gi_ld(ptr.a[z] + half + off, H);
    const Gi b0 = gi_ld(ptr.b[z] + off, H), b1 = gi_ld(ptr.b[z] + half + off, H);
    const Gi d = gi_ld(D2 + (long)z * half + off, H);
    Gi y0{0, 0}, y1{0, 0};
    if (MODE) {
      y0 = gi_ld(Y + (long)z * half + off, H);
      y1 = gi_ld(Y + (long)(n + z) * half + off, H);
    }
    Gi c0 = gi_sum2(a0, b0, d, kb, fit, P);
    Gi c1 = gi_add(gi_sum2(a0, b1, a1, b0, fit, P), gi_mulmod(d, ka, P), q);
    uint64_t *o0 = MODE ? outp.p[z] + off : U + ((long)z << log_n) + c;
    uint64_t *o1 = MODE ? outp.p[n + z] + off : U + ((long)(n + z) << log_n) + c;
    if (MODE == 2) {
      y0 = gi_scale(y0, bi, q);
      y1 = gi_scale(y1, bi, q);
    }
    if (MODE) {
      c0 = Gi{sub_mod(c0.r, y0.r, q), sub_mod(c0.i, y0.i, q)};
      c1 = Gi{sub_mod(c1.r, y1.r, q), sub_mod(c1.i, y1.i, q)};
    }
    if (MODE == 1) {
      c0 = gi_scale(c0, rs, q);
      c1 = gi_scale(c1, rs, q);
    }
    o0[0] = c0.r;
    o0[H] = c0.i;
    o1[0] = c1.r;
    o1[H] = c1.i;
  }
}

// blocks over ops: one thread serves every op of the launch when the limbs
// alone fill the chip, else the ops are spread so that about eight blocks per
// SM are in flight
int op_blocks(const Engine& E, long blocks, int n) {
  const long want = (8L * E.num_sms + blocks - 1) / blocks;
  return (int)std::max(1L, std::min((long)n, want));
}

}  // namespace

void tensor_d2_op(const Engine& E, const CtPtrs& ptr, long half, uint64_t* D2, int n, int nlimbs, cudaStream_t st) {
  launch_pdl(tensor_d2, dim3(E.N / (2 * kThreads), nlimbs, n), kThreads, 0, st, ptr, half, D2, E.d_pc, E.log_n);
}

void hmult_top_op(const Engine& E, const CtPtrs& ptr, long half, const uint64_t* D2, const uint64_t* key, uint64_t* U,
                  long u_stride, int n, int level, cudaStream_t st) {
  launch_pdl(hmult_top, dim3(E.N / kThreads, 1, n), kThreads, 0, st, ptr, half, D2, key, (long)E.nprimes * E.N, U,
             u_stride, n, level, E.rns.moddown_binv, E.d_pc, E.log_n);
}

void hmult_finish_op(const Engine& E, const CtPtrs& ptr, long half, const uint64_t* D2, const uint64_t* key,
                     const uint64_t* Y, const OutPtrs& outp, int n, int nlimbs, int rescale_level, cudaStream_t st) {
  const ShoupW* resc = rescale_level > 0 ? E.rns.resc_inv + (long)rescale_level * E.k : nullptr;
  const long blocks = E.N / (2 * kThreads) * nlimbs;
  const dim3 grid(E.N / (2 * kThreads), nlimbs, op_blocks(E, blocks, n));
  launch_pdl(resc ? hmult_finish<true> : hmult_finish<false>, grid, kThreads, 0, st, ptr, half, D2, key,
             (long)E.nprimes * E.N, Y, outp, n, E.rns.moddown_binv, resc, E.d_pc, E.log_n);
}

void gi_tensor_d2_op(const Engine& E, const CtPtrs& ptr, long half, uint64_t* D2, int n, int nlimbs, cudaStream_t st) {
  launch_pdl(gi_tensor_d2, dim3(E.N / (2 * kThreads), nlimbs, n), kThreads, 0, st, ptr, half, D2, E.d_pc, E.log_n);
}

void gi_hmult_top_op(const Engine& E, const CtPtrs& ptr, long half, const uint64_t* D2, const uint64_t* key,
                     uint64_t* U, int n, int level, cudaStream_t st) {
  launch_pdl(gi_finish<0>, dim3(E.N / (2 * kThreads), 1, n), kThreads, 0, st, ptr, half, D2, key,
             (long)E.nprimes * E.N, nullptr, OutPtrs{}, U, n, level, E.rns.moddown_binv, nullptr, E.d_pc, E.log_n);
}

void gi_hmult_finish_op(const Engine& E, const CtPtrs& ptr, long half, const uint64_t* D2, const uint64_t* key,
                        const uint64_t* Y, const OutPtrs& outp, int n, int nlimbs, int rescale_level,
                        cudaStream_t st) {
  const ShoupW* resc = rescale_level > 0 ? E.rns.resc_inv + (long)rescale_level * E.k : nullptr;
  const long blocks = E.N / (2 * kThreads) * nlimbs;
  launch_pdl(resc ? gi_finish<1> : gi_finish<2>, dim3(E.N / (2 * kThreads), nlimbs, op_blocks(E, blocks, n)), kThreads,
             0, st, ptr, half, D2, key, (long)E.nprimes * E.N, Y, outp, nullptr, n, 0, E.rns.moddown_binv, resc, E.d_pc,
             E.log_n);
}

void galois_finish_op(const Engine& E, const uint64_t* R, long half, const KeyPtrs& keys, bool one_key,
                      const uint64_t* Y, const OutPtrs& outp, int n, int nlimbs, bool add, cudaStream_t st) {
  const long blocks = E.N / (2 * kThreads) * nlimbs;
  const dim3 grid(E.N / (2 * kThreads), nlimbs, op_blocks(E, blocks, n));
  launch_pdl(one_key ? galois_finish<true> : galois_finish<false>, grid, kThreads, 0, st, R, half, keys,
             (long)E.nprimes * E.N, Y, outp, n, add, E.rns.moddown_binv, E.d_pc, E.log_n);
}

}  // namespace aoa
