// The lincheck's block fold on the tensor cores: z_vec[i] = XOR over blocks o
// with bit i of block o set of eq(x_outer, o), over the 2^k_log-bit blocks of
// the witness (lincheck.rs:2423 partial_fold_packed_z_block_major).
//
// Over the integers it is a matrix product, counts[p][b] = sum_o bit_p(block
// o) bit_b(eq(o)), whose parities are the answer: both operands are 0/1 bytes,
// tcgen05.mma kind::i8 accumulates the counts in tensor memory over all of a
// CTA's blocks, and only the end of a run costs an extraction.  A CTA takes 256
// bits of 64 blocks (rows) per step (two 128 x 128 count tiles): eight warps
// spread the bits to bytes, in the order that (word >> j) & 0x01010101 gives
// (the extraction undoes it), into one of three operand buffers, and a ninth
// starts the tensor cores.  A step is short beside the memory's latency, so a
// thread's words come by cp.async four steps ahead, into slots of its own.
// Both operands are MN-major: a row's bytes are contiguous, as its bits are in
// memory, so nothing is transposed.
// Bound: the chain of a step (copies' arrival, spreading, a barrier, the tensor
// cores' start), with two CTAs an SM to overlap it; then shared memory (the
// operands' stores and the tensor cores' reads, 56 KiB a step).  Measured at
// 2^18 / 2^14 / 2^10 compressions: 747 / 54 / 7.4 us, against 1097 / 90 / 20 us
// for XORs of eq values through 256-entry subset tables (a thread 16 bits of
// every block); the checks on its waits have since added 3 % at 2^18 (710 to 733
// us by the profiler's clock).  The same kernel with round 1's group weights took 1262 us for
// the c column's statistic at 2^18, whose table kernel takes 665 us.
#include "kernels.cuh"
#include "tmap.cuh"
#include <algorithm>

namespace {
constexpr int kRowsStep = 64;
constexpr uint32_t kTileBytes = kRowsStep * 128;    // 64 rows of 128 bytes
constexpr uint32_t kBufBytes = 3 * kTileBytes;      // two tiles of bits, one of weights
constexpr int kBufs = 3, kAhead = 4, kSpreaders = 256, kGemmThreads = kSpreaders + 32;
constexpr uint32_t kSlotBytes = 12;                 // a thread's words of a step: two of bits, one of a weight
constexpr size_t kGemmSmem = 1024 + kBufs * kBufBytes + kAhead * kSpreaders * kSlotBytes + 64;
constexpr int kGemmCols = 256;  // tensor-memory columns: two tiles of 128 counts
// D 32-bit integers, A and B unsigned bytes, both MN-major, M = N = 128
constexpr uint32_t kGemmIdesc = (2u << 4) | (1u << 15) | (1u << 16) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

struct GemmArgs {
  const uint32_t* bits;  // row o at bits + o * row_words
  uint32_t row_words, n_rows, cols;  // cols: 256-bit columns of a row
  const uint32_t* w;  // weights, four words a row
  f128* out;
};

__device__ __forceinline__ void spread(uint32_t w, uint4& lo, uint4& hi) {
  lo = make_uint4(w & 0x01010101u, (w >> 1) & 0x01010101u, (w >> 2) & 0x01010101u, (w >> 3) & 0x01010101u);
  hi = make_uint4((w >> 4) & 0x01010101u, (w >> 5) & 0x01010101u, (w >> 6) & 0x01010101u, (w >> 7) & 0x01010101u);
}
__device__ __forceinline__ void sts128(uint32_t a, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void gemm_mma(uint32_t d, uint64_t a, uint64_t b, bool add) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(kGemmIdesc), "r"((uint32_t)add)
      : "memory");
}

__device__ __forceinline__ void copy4(uint32_t dst, const void* src, bool there) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(there ? 4 : 0) : "memory");
}
__global__ void __launch_bounds__(kGemmThreads, 2) k_lc_zvec(GemmArgs G, WaitLimit W) {
  extern __shared__ __align__(16) uint8_t raw[];
  const uint32_t base = tm_smem(raw) + ((1024 - (tm_smem(raw) & 1023)) & 1023);
  const uint32_t slots = base + kBufs * kBufBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(raw + (slots - tm_smem(raw)) + kAhead * kSpreaders * kSlotBytes);
  uint32_t* addr = reinterpret_cast<uint32_t*>(bars + kBufs + 1);  // [tensor-memory address, dead, taken]
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tm_smem(addr)),
                 "n"(kGemmCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < kBufs + 1; i++) tm_mbar_init(bars + i);  // a buffer's products are done; all are
    addr[1] = addr[2] = 0;
  }
  tm_fence_before();
  __syncthreads();
  tm_fence_after();
  const uint32_t taddr = __shfl_sync(0xffffffffu, *addr, 0), bar = tm_smem(bars);
  const uint32_t dead = tm_smem(addr + 1), taken = tm_smem(addr + 2);

  const uint32_t per_col = (G.n_rows + kRowsStep - 1) / kRowsStep;
  const uint64_t total = (uint64_t)per_col * G.cols;
  const uint32_t s0 = (uint32_t)(total * blockIdx.x / gridDim.x), s1 = (uint32_t)(total * (blockIdx.x + 1) / gridDim.x);
  const uint32_t steps = s1 - s0;
  // step n: buffer n mod kBufs, use n / kBufs of it; column and row block of step s0 + n
  uint32_t col = s0 / per_col, blk = s0 % per_col;

  if (warp == kSpreaders / 32) {
    for (uint32_t n = 0, buf = 0; n < steps; n++) {
      const bool go = W.polls && !tm_lds32(dead);
      // named barrier 1 + buf: the step's operands are in place
      asm volatile("bar.sync %0, %1;" ::"r"(1 + buf), "n"(kGemmThreads) : "memory");
      tm_fence_after();
      const uint32_t A = base + buf * kBufBytes, B = A + 2 * kTileBytes;
      const bool first = n == 0 || blk == 0;
      if (tm_elect() && go) {
#pragma unroll
        for (int k = 0; k < 2; k++)  // 32 rows an instruction
#pragma unroll
          for (int t = 0; t < 2; t++)
            gemm_mma(taddr + 128 * t, tm_desc(A + t * kTileBytes + 4096 * k), tm_desc(B + 4096 * k), !first || k);
        tm_commit(bar + 8 * buf);
      }
      if (lane == 0) tm_sts32(taken, n + 1);
      __syncwarp();
      buf = buf + 1 == kBufs ? 0 : buf + 1;
      if (++blk == per_col) blk = 0;
    }
    // whoever gave up, the products end before their memory is another CTA's
    if (tm_elect()) tm_drain(bar + 8 * kBufs);
    __syncwarp();
  } else {
    const int r0 = tid >> 3, bw = tid & 7;  // two words of bits (rows r0, r0 + 32), one of a weight (row tid / 4)
    const uint32_t slot = slots + tid * kSlotBytes;
    uint32_t lcol = col, lblk = blk;  // the step to fetch next
    auto fetch = [&](uint32_t n) {
      if (n < steps) {
        const uint32_t d = slot + (n % kAhead) * (kSpreaders * kSlotBytes), row = lblk * kRowsStep;
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const uint32_t o = row + r0 + 32 * i;
          const bool there = o < G.n_rows;
          copy4(d + 4 * i, G.bits + (size_t)(there ? o : 0) * G.row_words + lcol * 8 + bw, there);
        }
        const uint32_t o = row + (tid >> 2);
        const bool there = o < G.n_rows;
        copy4(d + 8, G.w + (there ? 4 * (size_t)o + (tid & 3) : 0), there);
        if (++lblk == per_col) {
          lblk = 0;
          lcol++;
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // No wait of this thread ran out, nor did it see another's.  If one did, it
    // goes on to the end with wrong values, and before it arrives waits, in place
    // of the products, for the ninth warp to have taken the barrier's last round:
    // that warp waits for nothing but these arrivals.
    bool live = true;
    for (int i = 0; i < kAhead - 1; i++) fetch(i);
    for (uint32_t n = 0, buf = 0, use = 0; n < steps; n++) {
      fetch(n + kAhead - 1);
      asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory");
      const uint32_t d = slot + (n % kAhead) * (kSpreaders * kSlotBytes);
      const uint32_t x[2] = {tm_lds32(d), tm_lds32(d + 4)}, w = tm_lds32(d + 8);
      const uint32_t A = base + buf * kBufBytes, B = A + 2 * kTileBytes;
      if (use && live) live = tm_wait(bar + 8 * buf, (use - 1) & 1, dead, W.polls);  // its last products have read it
      if (use && !live)
        for (uint32_t i = 0; i < kWaitPolls && tm_lds32(taken) + kBufs <= n; i++) __nanosleep(20);
      uint4 lo, hi;
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int o = r0 + 32 * i, t = bw >> 2, c = 2 * (bw & 3);
        const uint32_t row = A + t * kTileBytes + 128 * o;
        spread(x[i], lo, hi);
        // the two tiles' threads store their chunks in opposite order: different banks
        sts128(row + (((c + t) ^ (o & 7)) << 4), t ? hi : lo);
        sts128(row + (((c + 1 - t) ^ (o & 7)) << 4), t ? lo : hi);
      }
      {
        const int o = tid >> 2, c = 2 * (tid & 3);
        spread(w, lo, hi);
        sts128(B + 128 * o + ((c ^ (o & 7)) << 4), lo);
        sts128(B + 128 * o + (((c + 1) ^ (o & 7)) << 4), hi);
      }
      tm_fence_smem();
      tm_fence_before();  // (a finished column's counts have been read)
      __syncwarp();
      asm volatile("bar.arrive %0, %1;" ::"r"(1 + buf), "n"(kGemmThreads) : "memory");
      if (n + 1 == steps || blk + 1 == per_col) {  // the column's or this CTA's last rows: extract
        if (live) live = tm_wait(bar + 8 * buf, use & 1, dead, W.polls);
        __syncwarp();
        tm_fence_after();
        // warps 0..3 read the first tile, 4..7 the second: row 32 (warp mod 4) + lane
        const uint32_t src = taddr + ((uint32_t)(warp & 3) << 21) + 128 * (warp >> 2);
        uint32_t v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          uint32_t r[32];
          tm_get_counts(src + 32 * q, r);
          v[q] = 0;
#pragma unroll
          for (int c = 0; c < 32; c++) v[q] |= (r[c] & 1u) << (8 * (c & 3) + (c >> 2));
        }
        const uint32_t p = 256 * col + 128 * (warp >> 2) + 32 * (warp & 3) + 8 * (lane & 3) + (lane >> 2);
        atomic_xor128(G.out + p, mk((uint64_t)v[0] | (uint64_t)v[1] << 32, (uint64_t)v[2] | (uint64_t)v[3] << 32));
      }
      if (++buf == kBufs) {
        buf = 0;
        use++;
      }
      if (++blk == per_col) {
        blk = 0;
        col++;
      }
    }
  }
  tm_fence_before();
  __syncthreads();
  if (tid == 0 && tm_lds32(dead)) *W.ran_out = 1;
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "n"(kGemmCols) : "memory");
}

}  // namespace

static uint64_t fold_steps(size_t n_outer, int k_log) {
  return (uint64_t)((n_outer + kRowsStep - 1) / kRowsStep) << (k_log - 8);
}
// the kernel counts rows and steps in 32 bits
bool lc_zvec_fits(size_t n_outer, int k_log) {
  return k_log >= 8 && k_log <= 17 && !(n_outer >> 30) && !(fold_steps(n_outer, k_log) >> 32);
}

// zv[i] ^= XOR over o < n_outer with bit i of o's 2^k_log-bit block set of eqo[o]
// (sms: the SMs the launch may fill, one wave of resident CTAs on them)
void lc_zvec(const f128* z, const f128* eqo, size_t n_outer, int k_log, f128* zv, int sms, cudaStream_t s,
             const WaitLimit& w) {
  if (!w.ran_out) throw CudaError("lc_zvec: a word for its waits");
  if (!lc_zvec_fits(n_outer, k_log)) throw CudaError("lc_zvec: bad shape");
  if (!n_outer) return;
  GemmArgs G{reinterpret_cast<const uint32_t*>(z), 1u << (k_log - 5), (uint32_t)n_outer, 1u << (k_log - 8),
             reinterpret_cast<const uint32_t*>(eqo), zv};
  CK(cudaFuncSetAttribute(k_lc_zvec, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem));
  const uint64_t grid = (uint64_t)resident_grid((const void*)k_lc_zvec, kGemmThreads, kGemmSmem, sms);
  count_launch();
  k_lc_zvec<<<(unsigned)std::max<uint64_t>(1, std::min(grid, fold_steps(n_outer, k_log))), kGemmThreads, kGemmSmem, s>>>(
      G, w);
}
