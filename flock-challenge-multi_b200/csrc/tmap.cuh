// GF(2)-linear maps of 128-bit values on the tensor cores.
//
// A product by a fixed field element (an NTT twiddle, a fold challenge) is a
// 128 x 128 bit matrix applied to the other factor.  tcgen05.mma kind::i8
// applies it to 128 values at a time: the values' bits are spread to bytes
// (A operand, one value per tensor-memory lane, 128 bytes of K), the matrix
// is a byte matrix in shared memory (B operand), and a result bit is the
// parity of a 32-bit count.  Two result bits share one count: the matrix
// byte is m_n + 128 m_n', so bit 0 of the count is the parity of bit n and
// bit 7 that of bit n' (the first count is at most 127 unless a row of the
// matrix is all ones: tensor_safe, ntt.cu, checks the twiddles).
// N is therefore 64, not 128, which halves both the tensor work and the
// extraction, the part that runs on the integer pipe.
//
// Orders (free, since both operands are laid out here):
//  * K byte 16 j + b holds input bit 8 b + j, so a 32-bit word w spreads to
//    (w >> j) & 0x01010101 (tensor-memory column 4 j + word).
//  * Column v = 16 w + 2 k + h of the result holds output bits n = 32 w + 16 h
//    + k and n + 7 (k < 7), or n = 32 w + 16 h + 14 and n + 1 (k = 7).  Two
//    columns are read back per register (tcgen05.ld .pack::16b), so register
//    8 w + k carries bits k, k + 7, k + 16, k + 23 of word w at positions 0,
//    7, 16, 23: one shift and one bit select merge four bits.
//
// The product matrix of t is made of windows of one bit sequence: with
// Q[i] = top bit of t x^i (0 <= i < 255), the entry (n, k) is Q[127 - n + k]
// up to the reduction's low terms: for n < 7 it differs by top bits of the
// product itself, which tm_extract adds back (the fold of bits 121..127 that
// GHASH reduction of an overflow makes).  So a matrix is written from 32
// bytes of Q by funnel shifts, with no field arithmetic.
#pragma once
#include "kernels.cuh"

constexpr int kTmMatBytes = 8192;    // one matrix: 64 rows of 128 bytes, 128-byte swizzle
constexpr int kTmCols = 128;         // tensor-memory columns of one CTA: result 64, operand 32 (x 2)
constexpr uint32_t kTmOperand = 64;  // first operand column

__device__ __forceinline__ uint32_t tm_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ f128 tm_lds(uint32_t a) {
  f128 v;
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.lo), "=l"(v.hi) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void tm_sts(uint32_t a, f128 v) {
  asm volatile("st.shared.v2.u64 [%0], {%1, %2};" ::"r"(a), "l"(v.lo), "l"(v.hi) : "memory");
}
__device__ __forceinline__ uint32_t tm_lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void tm_sts32(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// predicated, without a branch; OFF: bytes added to the address
template <int OFF>
__device__ __forceinline__ void tm_sts_if(uint32_t take, uint32_t a, uint4 v) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.v4.u32 [%1 + %6], {%2, %3, %4, %5};\n\t}" ::"r"(
          take),
      "r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "n"(OFF)
      : "memory");
}
// one thread of a converged warp
__device__ __forceinline__ bool tm_elect() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

// D 32-bit integers, A and B unsigned bytes (K-major), N = 64, M = 128
constexpr uint32_t kTmIdesc = (2u << 4) | ((64u >> 3) << 17) | ((128u >> 4) << 24);

// 128-byte swizzled K-major tile: 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t tm_desc(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
         (2ull << 61);
}

// One warp allocates; the address is in *slot after the next barrier.
__device__ __forceinline__ void tm_alloc(uint32_t* slot) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tm_smem(slot)), "n"(kTmCols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tm_free(uint32_t taddr) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "n"(kTmCols) : "memory");
}
__device__ __forceinline__ void tm_mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tm_smem(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void tm_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tm_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tm_fence_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ bool tm_poll(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(a), "r"(parity)
      : "memory");
  return ok;
}
// Waits for phase `parity`.  When it has not come within `polls` polls, what was
// in flight is waited for kWaitPolls longer, and then the CTA's word `dead` (a
// shared address) is set: false, here and at once in every later wait that finds
// its phase not come.  The CTA starts nothing from then on.
__device__ __forceinline__ bool tm_wait(uint32_t a, uint32_t parity, uint32_t dead, uint32_t polls) {
  if (tm_poll(a, parity)) return true;
  if (tm_lds32(dead)) return false;
  for (uint32_t i = 0; i < polls; i++)
    if (tm_poll(a, parity)) return true;
  for (uint32_t i = 0; i < kWaitPolls; i++)
    if (tm_poll(a, parity)) break;
  tm_sts32(dead, 1);
  return false;
}

// One elected thread: result columns [d, d + 64) of the lanes not masked =
// operand columns [a, a + 32) times the matrix with descriptor desc.
__device__ __forceinline__ void tm_mma(uint32_t d, uint32_t a, uint64_t desc, uint32_t off_lo, uint32_t off_hi) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, {%5, %5, %6, %6}, p;\n\t}" ::"r"(d),
        "r"(a + 8 * k), "l"(desc + (uint64_t)(2 * k)), "r"(kTmIdesc), "r"((uint32_t)k), "r"(off_lo), "r"(off_hi)
        : "memory");
  }
}
__device__ __forceinline__ void tm_mma(uint32_t d, uint32_t a, uint64_t desc) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a + 8 * k), "l"(desc + (uint64_t)(2 * k)), "r"(kTmIdesc), "r"((uint32_t)k)
        : "memory");
  }
}
__device__ __forceinline__ void tm_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

// The thread that started products waits for all of them, on an mbarrier not used
// before (bounded; the end of a CTA that gave up).
__device__ __forceinline__ void tm_drain(uint32_t bar) {
  tm_commit(bar);
  for (uint32_t i = 0; i < kWaitPolls && !tm_poll(bar, 0); i++) {
  }
}

// Powers of two that reach the kernels as parameters: a product by one is an
// IMAD on the otherwise idle FMA pipe, where a shift by a constant would go
// to the integer pipe that bounds the kernels built on this header.
struct TmShifts {
  uint32_t l[15];  // 2^k: a left shift
};
inline TmShifts tm_shifts() {
  TmShifts s;
  for (int k = 0; k < 15; k++) s.l[k] = 1u << k;
  return s;
}

// This thread's value into its lane's operand columns (lane = thread).
__device__ __forceinline__ void tm_put(uint32_t taddr, f128 y) {
  const uint32_t w[4] = {(uint32_t)y.lo, (uint32_t)(y.lo >> 32), (uint32_t)y.hi, (uint32_t)(y.hi >> 32)};
  uint32_t r[32];
#pragma unroll
  for (int j = 0; j < 8; j++)
#pragma unroll
    for (int i = 0; i < 4; i++) r[4 * j + i] = (w[i] >> j) & 0x01010101u;
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tm_put_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// This thread's lane of the result columns, as raw packed counts.
__device__ __forceinline__ void tm_get(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.pack::16b.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

// This thread's lane of 32 columns of 32-bit counts.
__device__ __forceinline__ void tm_get_counts(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

// a & m | c & ~m
__device__ __forceinline__ uint32_t bit_select(uint32_t a, uint32_t c, uint32_t m) { return (a & m) | (c & ~m); }

// The parities of the packed counts, as the map's 128-bit result.
__device__ __forceinline__ f128 tm_extract(const uint32_t (&r)[32], const TmShifts& S) {
  constexpr uint32_t kBits = 0x00810081u;
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    uint32_t x = r[8 * i + 7] * S.l[8];
    x = bit_select(r[8 * i + 7] * S.l[14], x, (1u << 14) | (1u << 30));
    x = bit_select(r[8 * i], x, kBits);
#pragma unroll
    for (int k = 1; k < 7; k++) x = bit_select(r[8 * i + k] * S.l[k], x, kBits << k);
    w[i] = x;
  }
  return mk((uint64_t)w[0] | ((uint64_t)w[1] << 32), (uint64_t)w[2] | ((uint64_t)w[3] << 32));
}
// The low terms of the product's reduction that the window matrix leaves out.
__device__ __forceinline__ f128 tm_finish_product(f128 v) {
  v.lo ^= (v.hi >> 57) ^ (v.hi >> 62) ^ (v.hi >> 63);
  return v;
}

// Q of t: bit i = top bit of t x^i, words 0..7 into q (q[8], q[9] = 0)
__device__ __forceinline__ void tm_sequence(f128 t, uint32_t* q) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint64_t s = __brevll(t.hi);
    q[2 * k] = (uint32_t)s;
    q[2 * k + 1] = (uint32_t)(s >> 32);
    t = reduce256(0, t.lo, t.hi, 0);  // t x^64
  }
  q[8] = q[9] = 0;
}

// 16 bytes at bit offset p of Q, one bit per byte (stride 8 bits), plus 128
// times the same at offset p - D.  q: shared address of the sequence, whose
// words (p - D) / 32 .. + 5 are read.
template <int D>
__device__ __forceinline__ uint4 tm_chunk(uint32_t q, int p) {
  const uint32_t a = q + 4 * ((p - D) >> 5);
  const int e = (p - D) & 31;
  uint32_t w[6], x[5], o[4];
#pragma unroll
  for (int i = 0; i < 6; i++) w[i] = tm_lds32(a + 4 * i);
#pragma unroll
  for (int i = 0; i < 5; i++) x[i] = __funnelshift_r(w[i], w[i + 1], e);
#pragma unroll
  for (int i = 0; i < 4; i++)
    o[i] = (x[i] & 0x01010101u) * 128u + (__funnelshift_r(x[i], x[i + 1], D) & 0x01010101u);
  return make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ uint32_t tm_chunk_off(int row, int j) {
  return (uint32_t)(row * 128 + ((j ^ (row & 7)) << 4));
}
// What each of the 128 threads writes of a product matrix.  The chunk j of the
// row of output bit n is the window at p = 127 - n + j, so a thread computes
// the window of one p and stores it to every row that takes it: with p = 135 -
// 16 h - b (h < 8, b < 16) those are the rows of n = 16 h + k, k = b - 8 + j in
// 0..6.  A warp's lanes hold four successive b, so it has at most seven or
// (the first and last warp) three stores to make, and these two warps write
// the 64 chunks of the rows of bits 14 and 15 mod 16 besides.  Eight
// neighbouring lanes take four b and two h: their rows differ mod 8, so their
// stores meet eight different bank groups.
struct TmRows {
  uint32_t off[7], take;  // shared addresses in the first matrix; bit i: store i exists
  uint32_t off1;          // the second window's
  int p, p1;
  bool wide;  // seven stores and no second window
};
__device__ __forceinline__ TmRows tm_rows(uint32_t mat) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = 4 * warp + (lane & 3), h = 2 * (lane >> 3) + ((lane >> 2) & 1);
  const int j0 = warp == 0 ? 5 : warp == 1 ? 1 : 0;
  TmRows R;
  R.p = 135 - 16 * h - b;
  R.wide = warp == 1 || warp == 2;
  R.take = 0;
#pragma unroll
  for (int i = 0; i < 7; i++) {
    const int j = j0 + i, k = b - 8 + j;
    R.off[i] = mat + tm_chunk_off(16 * (h >> 1) + 2 * k + (h & 1), j);
    if (k >= 0 && k < 7 && j < 8) R.take |= 1u << i;
  }
  const int t = lane + (warp ? 32 : 0), h1 = t >> 3, j1 = t & 7;
  R.off1 = mat + tm_chunk_off(16 * (h1 >> 1) + 14 + (h1 & 1), j1);
  R.p1 = 127 - (16 * h1 + 14) + j1;
  return R;
}
// The product matrix of the element whose sequence is at shared address q, by
// the CTA's 128 threads, OFF bytes after the first matrix.
template <int OFF>
__device__ __forceinline__ void tm_product_matrix(uint32_t q, const TmRows& R) {
  const uint4 v = tm_chunk<7>(q, R.p);
#pragma unroll
  for (int i = 0; i < 3; i++) tm_sts_if<OFF>(R.take & (1u << i), R.off[i], v);
  if (R.wide) {
#pragma unroll
    for (int i = 3; i < 7; i++) tm_sts_if<OFF>(R.take & (1u << i), R.off[i], v);
  } else {
    tm_sts_if<OFF>(1, R.off1, tm_chunk<1>(q, R.p1));
  }
}

// ---- bulk copies of 16-byte aligned rows ----
__device__ __forceinline__ void tm_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tm_load_row(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tm_store_row(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void tm_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// the stores' sources may be overwritten / the stores are done
__device__ __forceinline__ void tm_store_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tm_store_done() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
