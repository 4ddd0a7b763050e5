// K3-K8: the sumcheck-family kernels of the prover.
//
//  K3 eq tables:        eq(r, x) = prod_i (x_i ? r_i : 1 + r_i), bit i of x <-> r_i
//                       (zerocheck/univariate_skip.rs:31-87, lincheck.rs:2080-2125);
//                       materialised as lo[x & mask] * hi[x >> s].
//  K4 zerocheck round 1 (univariate skip over the 6 low bits, extract-c form):
//                       P_AB(l) = sum_x eq(r_rest, x) phi8(a^_l(x) b^_l(x)),
//                       P_C(l)  = sum_x eq(r_rest, x) phi8(c^_l(x)), l in Lambda
//                       (univariate_skip.rs:90-160).  The first seven rest
//                       variables carry the fixed inner challenges
//                       (univariate_skip_optimized.rs:136-233): three phi8
//                       subfield constants and four gamma^(2^i)/(1+gamma^(2^i)),
//                       so eq on a 128-row block is phi8(g(xs)) * C * gamma^xm:
//                       the small part is folded in GF(2^8), the medium part is a
//                       shift by xm bits, one general product per block and l.
//  K5 zerocheck multilinear rounds: message (G(1), G(inf)) of
//                       G(X) = sum eq(.) a^(X,.) b^(X,.), LSB binding, fused with
//                       the fold of the previous round (zerocheck.rs:1735-1795,
//                       multilinear.rs:575-657,3194-3330).
//  K6 lincheck:         comb = alpha A^T eq + B^T eq (CSC gather; lincheck.rs:175-200),
//                       z_vec[c] = sum_o eq(x_outer, o) z[c + 2^14 o],
//                       8 top-binding product-sumcheck rounds (lincheck.rs:4968-4990,5880-6050).
//  K7 ring switch:      s_hat_v[r] = sum_i eq(i) bit_r(z_i) (ring_switch.rs:1594-1640);
//                       b_combined[i] = sum_k gamma_k sum_b bit_b(eq_k(i)) eq''_k[b]
//                       (ring_switch.rs:1952-2130, pcs.rs:778-1290).
//  K8 Ligerito:         round messages u0 = sum f0 b0, u2 = sum (f0+f1)(b0+b1) and
//                       LSB folds (pcs/ligerito.rs:4923-5020, 8894-9100).
#include "kernels.cuh"
#include <algorithm>

namespace {
}  // namespace

// ------------------------------------------------------------------ K3 --
// eq tables built on the device: out[i] = scale * prod_j (bit j of i ? r_j : 1 + r_j)
// (the same values as the doubling construction of eq(r, .), field products
// being exact).  A table's cost is the chain of dependent products, about a
// microsecond each, so the chain is kept short: a CTA tabulates variables 0..3
// and 4..7, the next q, and multiplies the rest (its own index bits) in a
// shuffle tree, all at once; an output then takes one product.
// Up to 4 tables a launch (grid y).  Tables of up to 2^18 values take 7 us, one
// of 2^19 40 us; one chain of up to 13 products per thread, and a third launch
// for the tables above 2^12, took 18 + 18 + 4 us (54 us at 2^19).
struct EqVec {
  f128 r[32];
  f128 scale;
  f128* out;
  int n, q;
};
struct EqVecs {
  EqVec v[kMaxEqTables];
};
__global__ void __launch_bounds__(256) k_eq_build(const __grid_constant__ EqVecs V) {
  const EqVec& E = V.v[blockIdx.y];
  const int n = E.n, q = E.q, t = threadIdx.x;
  if (((uint64_t)blockIdx.x << (8 + q)) >> n) return;
  __shared__ f128 T[3][16], H, K[16];
  auto factor = [&](int j, uint32_t bit) { return j < n ? (bit ? E.r[j] : fx(E.r[j], mk(1, 0))) : mk(1, 0); };
  if (t < 48) {  // entry e of the table of variables j0..j0+3
    const int w = t >> 4, e = t & 15, j0 = 4 * w, nv = w < 2 ? 4 : q;
    f128 v = nv ? factor(j0, e & 1) : mk(1, 0);
    for (int j = 1; j < nv; j++) v = fmul(v, factor(j0 + j, (e >> j) & 1));
    T[w][e] = v;
  } else if (t >= 64 && t < 96) {  // the CTA's own index bits, and the scale
    const int l = t - 64, own = max(n - 8 - q, 0);
    f128 v = l < own ? factor(8 + q + l, (blockIdx.x >> l) & 1) : l == own ? E.scale : mk(1, 0);
    for (int m = 1; m <= own; m <<= 1) {  // lane 0 collects lanes 0..2m-1
      f128 o;
      o.lo = shfl_xor64(v.lo, m);
      o.hi = shfl_xor64(v.hi, m);
      v = fmul(v, o);
    }
    if (l == 0) H = v;
  }
  __syncthreads();
  const f128 lo = fmul(T[0][t & 15], T[1][t >> 4]);
  if (t < (1 << q)) K[t] = fmul(T[2][t], H);
  __syncthreads();
  if (n < 8 && (t >> n)) return;
  f128* out = E.out + ((size_t)blockIdx.x << (8 + q)) + t;
  for (int k = 0; k < (1 << q); k++) st(out + ((size_t)k << 8), fmul(lo, K[k]));
}

// out[s + 64 k] = L[s] * e[k]
struct Vec64 {
  f128 v[64];
};
__global__ void k_outer64(Vec64 L, const f128* __restrict__ e, size_t n_e, f128* __restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 64 * n_e) return;
  st(out + i, fmul(L.v[i & 63], ldg(e + (i >> 6))));
}

// The byte tables of a GF(2)-linear map, group g's basis values in the launch's
// parameters: eight selected XORs a value, one CTA a group, bound by the
// launch.  Built on the host, the 128 KiB of the ring switch's tables took a
// 2^10-compression proof more than 15 us (8192 XORs, fresh pages, a copy from
// pageable memory): its proof gained 15 us.
struct SubsetBasis {
  f128 v[256];
};
__global__ void k_subset_tables(const __grid_constant__ SubsetBasis B, f128* __restrict__ out) {
  const unsigned g = blockIdx.x, v = threadIdx.x;
  f128 x = mk(0, 0);
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const f128 y = B.v[8 * g + j];
    if (v >> j & 1) x = fx(x, y);
  }
  st(out + 256 * g + v, x);
}

// out[i] += beta * x[i]
__global__ void k_axpy(f128* __restrict__ out, const f128* __restrict__ x, f128 beta, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  st(out + i, fx(ld(out + i), fmul(ld(x + i), beta)));
}

// out[0] ^= sum_i f[i] g[i]
__global__ void k_inner(const f128* __restrict__ f, const f128* __restrict__ g, size_t n, f128* out, MailArgs mail) {
  u256 acc = zero256();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    acc_wide(acc, mul_wide(ld(f + i), ld(g + i)));
  block_xor_out(reduce(acc), out);
  mail_last(mail, out);
}

// ------------------------------------------------------------------ K5 --
// last fold: 2 -> 1 values per vector
__global__ void k_fold_pair_final(const f128* a_in, const f128* b_in, f128 rho, f128* out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    f128 a0 = a_in[0], a1 = a_in[1], b0 = b_in[0], b1 = b_in[1];
    out[0] = fx(a0, fmul(rho, fx(a0, a1)));
    out[1] = fx(b0, fmul(rho, fx(b0, b1)));
  }
}

void fold_pair_final(const f128* a_in, const f128* b_in, f128 rho, f128* out, cudaStream_t s) {
  count_launch(); k_fold_pair_final<<<1, 32, 0, s>>>(a_in, b_in, rho, out);
}

// ------------------------------------------------------------------ K6 --
// comb[c] = alpha * (A^T eq)[c] + (B^T eq)[c] (+ beta at the pinned column).
// The sums are gathers of 16-byte eq values at the columns' CSC row indices
// (21 M of them for the BLAKE3 block).  A CTA holds one 8-byte half of the
// table (2^14 rows; for 2^15 rows, one 4-byte quarter) in shared memory and a
// warp sums that part of a column, its lanes striding over the nonzeros; a
// second kernel forms the products.  Gathered from global memory, where the
// 256 KiB table misses L1, the sums took 82 us; they take 53 us here (2^14
// compressions; 56 and 43 us with the rows still in L2 from a proof of 2^10).
template <class W>
__global__ void __launch_bounds__(1024) k_lc_sums(const uint32_t* __restrict__ at_ptr,
                                                  const uint16_t* __restrict__ at_row,
                                                  const uint32_t* __restrict__ bt_ptr,
                                                  const uint16_t* __restrict__ bt_row, const W* __restrict__ eq, int k,
                                                  W* __restrict__ sums) {
  extern __shared__ __align__(16) uint8_t lc_sm[];
  W* T = reinterpret_cast<W*>(lc_sm);
  constexpr int kParts = 16 / sizeof(W);
  const int part = blockIdx.y;
  for (int i = threadIdx.x; i < k; i += blockDim.x) T[i] = eq[(size_t)i * kParts + part];
  __syncthreads();
  const int lane = threadIdx.x & 31, warps = (int)(gridDim.x * blockDim.x) >> 5;
  for (int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); c < 2 * k; c += warps) {
    const bool B = c >= k;
    const uint32_t* ptr = (B ? bt_ptr - k : at_ptr) + c;
    const uint16_t* row = B ? bt_row : at_row;
    const uint32_t e = ptr[1];
    W v = 0;
    uint32_t j = ptr[0] + lane;
    for (; j + 96 < e; j += 128) v ^= T[row[j]] ^ T[row[j + 32]] ^ T[row[j + 64]] ^ T[row[j + 96]];
    for (; j < e; j += 32) v ^= T[row[j]];
#pragma unroll
    for (int m = 16; m; m >>= 1) v ^= __shfl_xor_sync(0xffffffffu, v, m);
    if (lane == 0) sums[(size_t)c * kParts + part] = v;
  }
}
// comb: the 2 k sums in, the k values out
__global__ void __launch_bounds__(256) k_lc_comb(f128* comb, f128 alpha, f128 beta, int pin, int k) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= k) return;
  f128 v = fx(fmul(alpha, ld(comb + c)), ld(comb + k + c));
  if (c == pin) v = fx(v, beta);
  st(comb + c, v);
}

// One lincheck round (top binding): with do_fold, fold comb and zv (2 len
// values each) at r into their first len values; with emit, add the
// message over the (folded) pairs (i, i + len/2) into out[0..2):
// q1 = sum c1 z1, qinf = sum (c0 + c1)(z0 + z1).  Thread i < len/2 owns
// outputs i and i + len/2 and reads exactly the four inputs that fold into
// them, so the grid needs no synchronisation; the message is XOR-reduced per
// CTA and added atomically (out must be zero).
__global__ void __launch_bounds__(256) k_lc_round(f128* comb, f128* zv, int len, int do_fold, f128 r, int emit,
                                                  f128* out, MailArgs mail) {
  const int h = len >> 1;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  f128 q1 = mk(0, 0), qi = mk(0, 0);
  if (i < h) {
    f128 c0 = comb[i], c1 = comb[i + h], z0 = zv[i], z1 = zv[i + h];
    if (do_fold) {
      const f128 c0h = comb[i + len], c1h = comb[i + h + len], z0h = zv[i + len], z1h = zv[i + h + len];
      c0 = fx(c0, fmul(r, fx(c0h, c0)));
      c1 = fx(c1, fmul(r, fx(c1h, c1)));
      z0 = fx(z0, fmul(r, fx(z0h, z0)));
      z1 = fx(z1, fmul(r, fx(z1h, z1)));
      comb[i] = c0;
      comb[i + h] = c1;
      zv[i] = z0;
      zv[i + h] = z1;
    }
    if (emit) {
      q1 = fmul(c1, z1);
      qi = fmul(fx(c0, c1), fx(z0, z1));
    }
  }
  if (!emit) return;
  block_xor_out(q1, out);
  block_xor_out(qi, out + 1);
  mail_last(mail, out);
}

// The same round with four lanes a pair (short rounds).
__global__ void __launch_bounds__(256) k_lc_round_quad(f128* comb, f128* zv, int len, int do_fold, f128 r, int emit,
                                                       f128* out, MailArgs mail) {
  const int h = len >> 1, t = blockIdx.x * blockDim.x + threadIdx.x, i = t >> 2, q = t & 3;
  f128 v = mk(0, 0);
  if (i < h) {
    f128* p = (q < 2 ? comb : zv) + i + (q & 1 ? h : 0);
    v = *p;
    if (do_fold) {
      v = fx(v, fmul(r, fx(p[len], v)));
      *p = v;
    }
  }
  if (!emit) return;
  f128 x, y;
  quad_factors<false>(v, q, x, y);
  // odd lanes: sum c1 z1 (out[0]); even lanes: sum (c0 + c1)(z0 + z1) (out[1])
  block_xor_classes<4>(fmul(x, y), out, [](int c) { return c < 2 ? 1 - c : -1; });
  mail_last(mail, out);
}

void lc_comb(const uint32_t* at_ptr, const uint16_t* at_row, const uint32_t* bt_ptr, const uint16_t* bt_row,
             const f128* eq, f128 alpha, f128 beta, int pin, int k, f128* comb, int sms, cudaStream_t s,
             int* ctas) {
  const int parts = k <= (1 << 14) ? 2 : 4;
  const size_t smem = (size_t)k * 16 / parts;
  if (smem > ((size_t)128 << 10)) throw CudaError("lc_comb: at most 2^15 rows");
  // one CTA fits an SM, and it stays for the whole launch
  const dim3 grid(std::max(1, sms / parts), parts);
  if (ctas) *ctas = (int)(grid.x * grid.y);
  count_launch(2);
  if (parts == 2) {
    CK(cudaFuncSetAttribute(k_lc_sums<uint64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 << 10));
    k_lc_sums<uint64_t><<<grid, 1024, smem, s>>>(at_ptr, at_row, bt_ptr, bt_row,
                                                 reinterpret_cast<const uint64_t*>(eq), k,
                                                 reinterpret_cast<uint64_t*>(comb));
  } else {
    CK(cudaFuncSetAttribute(k_lc_sums<uint32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 << 10));
    k_lc_sums<uint32_t><<<grid, 1024, smem, s>>>(at_ptr, at_row, bt_ptr, bt_row,
                                                 reinterpret_cast<const uint32_t*>(eq), k,
                                                 reinterpret_cast<uint32_t*>(comb));
  }
  k_lc_comb<<<(k + 255) / 256, 256, 0, s>>>(comb, alpha, beta, pin, k);
}
void lc_round(f128* comb, f128* zv, int len, bool fold, f128 r, bool emit, f128* out, cudaStream_t s,
              const MailArgs& mail) {
  const int pairs = std::max(1, len / 2);
  count_launch();
  if (pairs <= kQuadPairs)
    k_lc_round_quad<<<(4 * pairs + 255) / 256, 256, 0, s>>>(comb, zv, len, fold, r, emit, out, mail);
  else
    k_lc_round<<<(pairs + 255) / 256, 256, 0, s>>>(comb, zv, len, fold, r, emit, out, mail);
}

// ------------------------------------------------------------------ K7 --
// ------------------------------------------------------------------ K8 --
__global__ void __launch_bounds__(256) k_lig_msg(const f128* __restrict__ f, const f128* __restrict__ b,
                                                 size_t n_pairs, f128* __restrict__ out, MailArgs mail) {
  u256 u0 = zero256(), u2 = zero256();
  for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < n_pairs; j += (size_t)gridDim.x * blockDim.x) {
    f128 f0 = ld(f + 2 * j), f1 = ld(f + 2 * j + 1), b0 = ld(b + 2 * j), b1 = ld(b + 2 * j + 1);
    acc_wide(u0, mul_wide(f0, b0));
    acc_wide(u2, mul_wide(fx(f0, f1), fx(b0, b1)));
  }
  block_xor_out(reduce(u0), out);
  block_xor_out(reduce(u2), out + 1);
  mail_last(mail, out);
}

// fold f and b at r (LSB binding), then emit the next message on the folded
// pair; products by r go through a CTA-resident 8-bit window table
__global__ void __launch_bounds__(256) k_lig_fold_msg(const f128* __restrict__ f, const f128* __restrict__ b,
                                                      f128* __restrict__ fo, f128* __restrict__ bo, f128 r,
                                                      size_t n_pairs_out, int emit, f128* __restrict__ out,
                                                      MailArgs mail) {
  extern __shared__ __align__(16) uint8_t sm[];
  MulTab8* rt = reinterpret_cast<MulTab8*>(sm);
  multab_build(rt, r);
  auto mr = [&](f128 v) { return multab_mul(rt, v); };
  u256 u0 = zero256(), u2 = zero256();
  for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < n_pairs_out; j += (size_t)gridDim.x * blockDim.x) {
    f128 fv[4], bv[4];
#pragma unroll
    for (int k = 0; k < 4; k++) { fv[k] = ld(f + 4 * j + k); bv[k] = ld(b + 4 * j + k); }
    f128 f0 = fx(fv[0], mr(fx(fv[0], fv[1]))), f1 = fx(fv[2], mr(fx(fv[2], fv[3])));
    f128 b0 = fx(bv[0], mr(fx(bv[0], bv[1]))), b1 = fx(bv[2], mr(fx(bv[2], bv[3])));
    st(fo + 2 * j, f0); st(fo + 2 * j + 1, f1);
    st(bo + 2 * j, b0); st(bo + 2 * j + 1, b1);
    if (emit) {
      acc_wide(u0, mul_wide(f0, b0));
      acc_wide(u2, mul_wide(fx(f0, f1), fx(b0, b1)));
    }
  }
  if (emit) {
    block_xor_out(reduce(u0), out);
    block_xor_out(reduce(u2), out + 1);
    mail_last(mail, out);
  }
}

// The same for short rounds: four lanes a pair, products by r without a table
// (building it takes longer than the folds).
__global__ void __launch_bounds__(256) k_lig_fold_quad(const f128* __restrict__ f, const f128* __restrict__ b,
                                                       f128* __restrict__ fo, f128* __restrict__ bo, f128 r,
                                                       int n_pairs_out, int emit, f128* __restrict__ out,
                                                       MailArgs mail) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, j = t >> 2, q = t & 3;
  f128 v = mk(0, 0);
  if (j < n_pairs_out) {
    const f128* p = (q < 2 ? f : b) + 4 * (size_t)j + 2 * (q & 1);
    v = ld(p);
    v = fx(v, fmul(r, fx(v, ld(p + 1))));
    st((q < 2 ? fo : bo) + 2 * (size_t)j + (q & 1), v);
  }
  if (!emit) return;
  f128 x, y;
  quad_factors<true>(v, q, x, y);
  // even lanes: sum f0 b0 (out[0]); odd lanes: sum (f0 + f1)(b0 + b1) (out[1])
  block_xor_classes<4>(fmul(x, y), out, [](int c) { return c < 2 ? c : -1; });
  mail_last(mail, out);
}

// Degree-3 sumcheck round over plain F128 vectors (the zerocheck round of
// zerocheck/multilinear.rs:616-657 in its unstructured form): for the pairs
// (a0, a1) = (a[2j], a[2j+1]), (b0, b1) likewise and eq weight e[j],
//   G(1) = sum_j e[j] a1 b1,  G(inf) = sum_j e[j] (a0 + a1)(b0 + b1),
// optionally after folding the previous round's pairs at rho (LSB binding,
// a' = a0 + rho (a0 + a1); multilinear.rs:3194-3219).  The eq product is
// accumulated unreduced; rho's operand split is built once per thread.
template <bool FOLD>
__global__ void __launch_bounds__(256) k_sc3_round(const f128* __restrict__ a, const f128* __restrict__ b,
                                                   const f128* __restrict__ e, f128* __restrict__ ao,
                                                   f128* __restrict__ bo, f128 rho, size_t n_pairs,
                                                   f128* __restrict__ out) {
  const MulConst R = mulconst(rho);
  u256 g1 = zero256(), gi = zero256();
  for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < n_pairs; j += (size_t)gridDim.x * blockDim.x) {
    f128 a0, a1, b0, b1;
    if (FOLD) {
      f128 av[4], bv[4];
#pragma unroll
      for (int k = 0; k < 4; k++) { av[k] = ld(a + 4 * j + k); bv[k] = ld(b + 4 * j + k); }
      a0 = fx(av[0], fmul_c(fx(av[0], av[1]), R));
      a1 = fx(av[2], fmul_c(fx(av[2], av[3]), R));
      b0 = fx(bv[0], fmul_c(fx(bv[0], bv[1]), R));
      b1 = fx(bv[2], fmul_c(fx(bv[2], bv[3]), R));
      st(ao + 2 * j, a0); st(ao + 2 * j + 1, a1);
      st(bo + 2 * j, b0); st(bo + 2 * j + 1, b1);
    } else {
      a0 = ld(a + 2 * j); a1 = ld(a + 2 * j + 1);
      b0 = ld(b + 2 * j); b1 = ld(b + 2 * j + 1);
    }
    const f128 w = ld(e + j);
    acc_wide(g1, mul_wide(w, fmul(a1, b1)));
    acc_wide(gi, mul_wide(w, fmul(fx(a0, a1), fx(b0, b1))));
  }
  block_xor_out(reduce(g1), out);
  block_xor_out(reduce(gi), out + 1);
}

void sc3_round(const f128* a, const f128* b, const f128* e, f128* ao, f128* bo, const f128* rho, size_t n_pairs,
               f128* out, int grid, cudaStream_t s) {
  count_launch();
  if (rho)
    k_sc3_round<true><<<grid, 256, 0, s>>>(a, b, e, ao, bo, *rho, n_pairs, out);
  else
    k_sc3_round<false><<<grid, 256, 0, s>>>(a, b, e, ao, bo, mk(0, 0), n_pairs, out);
}

// sms: the SMs the launch may fill (one wave of resident CTAs on them)
void lig_msg(const f128* f, const f128* b, size_t n_pairs, f128* out, int sms, cudaStream_t s, const MailArgs& mail) {
  const int grid = resident_grid((const void*)k_lig_msg, 256, 0, sms);
  count_launch(); k_lig_msg<<<grid, 256, 0, s>>>(f, b, n_pairs, out, mail);
}
void lig_fold_msg(const f128* f, const f128* b, f128* fo, f128* bo, f128 r, size_t n_pairs_out, bool emit, f128* out,
                  int sms, cudaStream_t s, const MailArgs& mail) {
  count_launch();
  if (n_pairs_out > (size_t)kQuadPairs) {
    size_t smem = sizeof(MulTab8);
    CK(cudaFuncSetAttribute(k_lig_fold_msg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int grid = resident_grid((const void*)k_lig_fold_msg, 256, smem, sms);
    k_lig_fold_msg<<<grid, 256, smem, s>>>(f, b, fo, bo, r, n_pairs_out, emit, out, mail);
  } else {
    const unsigned grid = std::max(1u, ((unsigned)n_pairs_out * 4 + 255) / 256);
    k_lig_fold_quad<<<grid, 256, 0, s>>>(f, b, fo, bo, r, (int)n_pairs_out, emit, out, mail);
  }
}
void eq_build(const EqTable* tabs, int count, cudaStream_t s) {
  if (count < 1 || count > kMaxEqTables) throw CudaError("eq_build: one to four tables");
  EqVecs V;
  unsigned blocks = 1;
  for (int i = 0; i < count; i++) {
    const EqTable& t = tabs[i];
    if (t.n < 0 || t.n > 31) throw CudaError("eq_build: at most 31 variables");
    EqVec& E = V.v[i];
    for (int j = 0; j < t.n; j++) E.r[j] = t.r[j];
    E.scale = t.scale;
    E.out = t.out;
    E.n = t.n;
    // values per CTA 2^(8 + q): 2^10 CTAs before they grow
    E.q = std::min(4, std::max(0, t.n - 18));
    blocks = std::max(blocks, 1u << std::max(0, t.n - 8 - E.q));
  }
  count_launch();
  k_eq_build<<<dim3(blocks, count), 256, 0, s>>>(V);
}
void eq_build(const f128* r, int n, f128 scale, f128* out, cudaStream_t s) {
  const EqTable t{r, n, scale, out};
  eq_build(&t, 1, s);
}
void outer64(const f128* L, const f128* e, size_t n_e, f128* out, cudaStream_t s) {
  Vec64 V;
  for (int j = 0; j < 64; j++) V.v[j] = L[j];
  count_launch();
  k_outer64<<<(unsigned)((64 * n_e + 255) / 256), 256, 0, s>>>(V, e, n_e, out);
}
void subset_tables(const f128* basis, int groups, f128* out, cudaStream_t s) {
  if (groups < 1 || groups > 32) throw CudaError("subset_tables: 1 to 32 groups");
  SubsetBasis B;
  for (int i = 0; i < 256; i++) B.v[i] = i < 8 * groups ? basis[i] : mk(0, 0);
  count_launch();
  k_subset_tables<<<(unsigned)groups, 256, 0, s>>>(B, out);
}
void axpy(f128* out, const f128* x, f128 beta, size_t n, cudaStream_t s) {
  count_launch(); k_axpy<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(out, x, beta, n);
}
void inner(const f128* f, const f128* g, size_t n, f128* out, int grid, cudaStream_t s, const MailArgs& mail) {
  count_launch(); k_inner<<<grid, 256, 0, s>>>(f, g, n, out, mail);
}
