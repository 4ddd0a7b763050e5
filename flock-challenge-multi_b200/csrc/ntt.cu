// K1: additive NTT over GF(2^128) (LCH novel basis, neighbours-last) on the
// interleaved layout data[pos * lanes + lane], and its transpose.
//
// Semantics: crates/flock-core/src/ntt/additive_ntt_f128.rs — layer l pairs
// positions 2^(log_d - l - 1) apart inside 2^l blocks; butterfly
// u += v * t, v += u with t = twiddle(l, block) = sum over set bits j of the
// block index of W^_{d-l-1}(beta_{d-l+j}) (:2684-2693, :4766-4800).  RS
// encoding at rate 2^-r = replicate the message into 2^r sub-blocks, then
// layers r..d-1 (:2741-2760; commit.rs:1838-1877).  The transposed map (used
// to induce the Ligerito query basis; pcs/ligerito.rs:1579-1600,1987-2056)
// runs layers in reverse with s = u + v, u = s, v = t*s + v.
//
// GPU mapping: each pass covers R <= 10 consecutive layers.  A CTA owns one
// tile = 2^R positions (one per combination of the pass's pair bits, the
// other position bits fixed) x LG consecutive lanes, staged in shared
// memory (LG lanes of one position are contiguous: 16*LG-byte coalesced
// rows); LG is chosen so that two CTAs fit an SM.  The tile's 2^R - 1
// twiddles are derived once into shared memory from the per-layer basis
// values (XOR of at most d values each); block 0 of every layer has the zero
// twiddle and needs no product.
#include "kernels.cuh"
#include "tmap.cuh"
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>
#include "host.hpp"

namespace {
constexpr int kMaxR = 10;  // layers per pass in the default split (the tuner also tries 11)

struct PassArgs {
  f128* data;
  const f128* ev;  // ev[l * 32 + j] = W^_{d-l-1}(beta_{d-l+j}), j < l
  int log_d, lanes, lg_shift, l0, R;
  // The first pass of an RS encode reads its tiles from the message instead
  // of from a replicated codeword: position p of the data holds message
  // position p & src_mask (the rate-2^-r replicate, layer 0..r-1 copies).
  const f128* src = nullptr;
  uint64_t src_mask = 0;
};
__device__ __forceinline__ const f128* tile_src(const PassArgs& p, uint64_t pos) {
  return p.src ? p.src + (pos & p.src_mask) * p.lanes : p.data + pos * p.lanes;
}

__device__ __forceinline__ f128 twiddle(const f128* ev, int l, uint64_t b) {
  f128 t = mk(0, 0);
  for (int j = 0; j < l; j++)
    if ((b >> j) & 1) t = fx(t, ldg(ev + l * 32 + j));
  return t;
}

// One tile of a pass (tile index t_id), staged through the CTA's shared memory.
template <bool TRANSPOSE>
__device__ __forceinline__ void ntt_tile(const PassArgs& p, uint64_t t_id, f128* smem) {
  const int R = p.R, LG = 1 << p.lg_shift;
  f128* tile = smem;                       // [2^R][LG]
  f128* tw = smem + ((size_t)LG << R);     // [2^R - 1] : stage s block k at (1<<s)-1+k
  const int log_d = p.log_d, l0 = p.l0;
  const int lo_bits = log_d - l0 - R;      // position bits below the pair bits
  const int groups = p.lanes >> p.lg_shift;
  const int grp = (int)(t_id % groups);
  t_id /= groups;
  const uint64_t lo = t_id & ((1ull << lo_bits) - 1);
  const uint64_t hi = t_id >> lo_bits;     // l0 bits
  const int n_el = LG << R;
  // load
  uint64_t any = 0;
  for (int e = threadIdx.x; e < n_el; e += blockDim.x) {
    uint64_t pl = (uint64_t)(e >> p.lg_shift);
    uint64_t pos = (hi << (log_d - l0)) | (pl << lo_bits) | lo;
    tile[e] = ld(tile_src(p, pos) + ((size_t)grp << p.lg_shift) + (e & (LG - 1)));
    if (TRANSPOSE) any |= tile[e].lo | tile[e].hi;
  }
  // The transposed transform (the query-basis induction) starts from a vector
  // that is zero outside the queried positions, and a pass maps a zero tile
  // to zeros in place: such tiles are left as they are.
  if (TRANSPOSE && !__syncthreads_or(any != 0)) return;
  for (int k = threadIdx.x; k < (1 << R) - 1; k += blockDim.x) {
    int s = 31 - __clz(k + 1);               // stage
    uint64_t blk = (uint64_t)(k + 1 - (1 << s));
    tw[k] = twiddle(p.ev, l0 + s, (hi << s) | blk);
  }
  __syncthreads();
  // A thread owns one position pair and `per` of its LG lanes (all of them
  // once the tile has as many position pairs as threads): the twiddle's
  // operand split is built once and reused for every lane.  Lanes are
  // visited in an order rotated by the thread index so that the 8 threads
  // of a quarter warp read 8 different 16-byte bank groups.
  const int n_pp = 1 << (R - 1);
  const int per = min(LG, max(1, (n_pp * LG) / (int)blockDim.x));
  const int tpp = LG / per;  // threads per position pair
  const int rs = 3 - p.lg_shift;  // rotate by pq >> rs: distinct bank groups per quarter warp
  for (int stg = 0; stg < R; stg++) {
    const int s = TRANSPOSE ? R - 1 - stg : stg;
    const int hb = R - 1 - s;                // local pair bit
    for (int w = threadIdx.x; w < n_pp * tpp; w += blockDim.x) {
      const int pq = w / tpp, lane0 = (w % tpp) * per;
      const int top = ((pq >> hb) << (hb + 1)) | (pq & ((1 << hb) - 1));
      const int bot = top | (1 << hb);
      const f128 tv = tw[(1 << s) - 1 + (top >> (hb + 1))];
      if (fz(tv)) {  // block 0 of every layer: the twiddle is the empty sum
        for (int k = 0; k < per; k++) {
          const int lane = lane0 + ((k + (pq >> rs)) & (per - 1));
          const int it = (top << p.lg_shift) | lane, ib = (bot << p.lg_shift) | lane;
          if (!TRANSPOSE) tile[ib] = fx(tile[ib], tile[it]);
          else tile[it] = fx(tile[it], tile[ib]);
        }
        continue;
      }
      const MulConst M = mulconst(tv);
      // lane order rotated by the position pair: lane0 + rot covers all 8
      // bank groups over 8 consecutive threads for every `per`
      auto bfly = [&](int lane) {
        f128 u = tile[(top << p.lg_shift) | lane], v = tile[(bot << p.lg_shift) | lane];
        if (!TRANSPOSE) {
          u = fx(u, fmul_c(v, M));
          v = fx(v, u);
        } else {
          u = fx(u, v);
          v = fx(v, fmul_c(u, M));
        }
        tile[(top << p.lg_shift) | lane] = u;
        tile[(bot << p.lg_shift) | lane] = v;
      };
      if (per == 1) {
        bfly(lane0);
      } else {
        for (int k = 0; k < per; k += 2) {  // two independent butterflies per step
          const int l0 = lane0 + ((k + (pq >> rs)) & (per - 1)), l1 = lane0 + ((k + 1 + (pq >> rs)) & (per - 1));
          f128 u0 = tile[(top << p.lg_shift) | l0], v0 = tile[(bot << p.lg_shift) | l0];
          f128 u1 = tile[(top << p.lg_shift) | l1], v1 = tile[(bot << p.lg_shift) | l1];
          if (!TRANSPOSE) {
            u0 = fx(u0, fmul_c(v0, M));
            u1 = fx(u1, fmul_c(v1, M));
            v0 = fx(v0, u0);
            v1 = fx(v1, u1);
          } else {
            u0 = fx(u0, v0);
            u1 = fx(u1, v1);
            v0 = fx(v0, fmul_c(u0, M));
            v1 = fx(v1, fmul_c(u1, M));
          }
          tile[(top << p.lg_shift) | l0] = u0;
          tile[(bot << p.lg_shift) | l0] = v0;
          tile[(top << p.lg_shift) | l1] = u1;
          tile[(bot << p.lg_shift) | l1] = v1;
        }
      }
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < n_el; e += blockDim.x) {
    uint64_t pl = (uint64_t)(e >> p.lg_shift);
    uint64_t pos = (hi << (log_d - l0)) | (pl << lo_bits) | lo;
    st(p.data + pos * p.lanes + ((size_t)grp << p.lg_shift) + (e & (LG - 1)), tile[e]);
  }
}

// ---- warp-per-pair passes: warp-uniform twiddles, table products ----
// A tile holds 2^R positions x 64 lanes.  A warp owns one position pair at a
// time (thread t takes lanes t and t + 32), so the pair's twiddle is uniform
// across the warp in every stage, and the warp multiplies by it through a
// 4-bit window table of the twiddle: entry n of window w is
// t * n(x) * x^(4w), and a product is the XOR of 32 lookups, one per nibble
// of the other factor.  The halves of an entry sit in separate 8-byte arrays
// and window w's entries are permuted by n -> n ^ (w mod 16), so the warp's
// lookups into one window, and the builder's stores, hit 16 distinct bank
// pairs.  A warp's consecutive pairs share the twiddle in all but the last
// stages, and the table is rebuilt only when the twiddle changes.  The
// table lookups load the shared-memory pipe instead of the integer
// multipliers; KIND 2 sends lane t + 32 through the integer product, so both
// pipes work.
size_t pass_w_smem(int R, int threads) {
  return ((size_t)64 << R) * sizeof(f128) + ((size_t)1 << R) * sizeof(f128) + (size_t)(threads / 32) * kTab4Bytes;
}

template <bool TRANSPOSE, int KIND>
__device__ __forceinline__ void ntt_tile_w(const PassArgs& p, uint64_t t_id, f128* smem) {
  const int R = p.R;
  f128* tile = smem;                         // [2^R][64]
  f128* tw = smem + ((size_t)64 << R);       // [2^R - 1], padded to 2^R
  Tab4* tabs = reinterpret_cast<Tab4*>(tw + (1 << R));
  const int log_d = p.log_d, l0 = p.l0;
  const int lo_bits = log_d - l0 - R;
  const int groups = p.lanes >> 6;
  const int grp = (int)(t_id % groups);
  t_id /= groups;
  const uint64_t lo = t_id & ((1ull << lo_bits) - 1);
  const uint64_t hi = t_id >> lo_bits;
  const int n_el = 64 << R;
  uint64_t any = 0;
  for (int e = threadIdx.x; e < n_el; e += blockDim.x) {
    const uint64_t pl = (uint64_t)(e >> 6);
    const uint64_t pos = (hi << (log_d - l0)) | (pl << lo_bits) | lo;
    tile[e] = ld(tile_src(p, pos) + ((size_t)grp << 6) + (e & 63));
    if (TRANSPOSE) any |= tile[e].lo | tile[e].hi;
  }
  if (TRANSPOSE && !__syncthreads_or(any != 0)) return;
  for (int k = threadIdx.x; k < (1 << R) - 1; k += blockDim.x) {
    const int s = 31 - __clz(k + 1);
    const uint64_t blk = (uint64_t)(k + 1 - (1 << s));
    tw[k] = twiddle(p.ev, l0 + s, (hi << s) | blk);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  Tab4* T = tabs + warp;
  const int chunk = (1 << (R - 1)) / nw;  // position pairs per warp per stage (the host keeps nw <= 2^(R-1))
  for (int stg = 0; stg < R; stg++) {
    const int s = TRANSPOSE ? R - 1 - stg : stg;
    const int hb = R - 1 - s;
    int cur = -1;
    MulConst M;  // KIND 2: the class split of the current twiddle
    for (int pq = warp * chunk; pq < (warp + 1) * chunk; pq++) {
      const int top = ((pq >> hb) << (hb + 1)) | (pq & ((1 << hb) - 1));
      const int bot = top | (1 << hb);
      const int k = (1 << s) - 1 + (top >> (hb + 1));
      const f128 tv = tw[k];
      f128* ut = tile + ((size_t)top << 6);
      f128* vt = tile + ((size_t)bot << 6);
      if (fz(tv)) {  // block 0 of every layer: the twiddle is the empty sum
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const int l = lane + 32 * q;
          if (!TRANSPOSE) vt[l] = fx(vt[l], ut[l]);
          else ut[l] = fx(ut[l], vt[l]);
        }
        continue;
      }
      if (k != cur) {
        __syncwarp();  // every lane has finished with the previous table
        tab4_build(T, tv, lane);
        if (KIND == 2) M = mulconst(tv);
        __syncwarp();
        cur = k;
      }
      f128 u0 = ut[lane], v0 = vt[lane], u1 = ut[lane + 32], v1 = vt[lane + 32];
      if (!TRANSPOSE) {
        u0 = fx(u0, tab4_mul(T, v0));
        if (KIND == 1) u1 = fx(u1, tab4_mul(T, v1));
        else u1 = fx(u1, fmul_c(v1, M));
        v0 = fx(v0, u0);
        v1 = fx(v1, u1);
      } else {
        u0 = fx(u0, v0);
        u1 = fx(u1, v1);
        v0 = fx(v0, tab4_mul(T, u0));
        if (KIND == 1) v1 = fx(v1, tab4_mul(T, u1));
        else v1 = fx(v1, fmul_c(u1, M));
      }
      ut[lane] = u0;
      vt[lane] = v0;
      ut[lane + 32] = u1;
      vt[lane + 32] = v1;
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < n_el; e += blockDim.x) {
    const uint64_t pl = (uint64_t)(e >> 6);
    const uint64_t pos = (hi << (log_d - l0)) | (pl << lo_bits) | lo;
    st(p.data + pos * p.lanes + ((size_t)grp << 6) + (e & 63), tile[e]);
  }
}

// ---- tensor-core passes: twiddles as bit matrices ----
// A CTA of 128 threads owns a tile of 2^R positions x 64 lanes.  Thread r of
// a unit takes lane r mod 64 of position pair 2 unit + r / 64; all 128
// products of a unit go through one tcgen05 matrix product (tmap.cuh), with
// the unit's twiddle as a matrix that the CTA writes to shared memory when
// the twiddle changes.  In the last stage the unit's two pairs have their
// own twiddles: two matrices, each product masked to its half of the lanes.
// Four CTAs fit an SM (tile, matrices, 128 of 512 tensor-memory columns), so
// one CTA's barriers and tensor latency hide behind the others.
// Bound: the integer pipe (spreading and merging bits, 96 of about 160 of its
// operations a product; writing matrices 40 more), then the dependent chain of
// a unit, which four CTAs do not quite cover.  Measured, 2^20 positions x 64
// lanes: 7.49 ms, 8.5 10^10 products/s, against 11.80 ms for the table passes
// (their ceiling, the shared-memory pipe, is 7.27 10^10) and 17.9 ms for the
// integer products; 2^16: 0.477 / 0.611 / 0.914 ms; 2^12: 0.046 / 0.070 /
// 0.064 ms.  R = 4 throughout (one pass more, and 15 matrices for 16 units in
// place of 31 for 40) takes 8.27 ms.
constexpr int kMaxRt = 5;
size_t pass_t_smem(int R) {
  return 1024 + 2 * kTmMatBytes + ((size_t)64 << R) * sizeof(f128) + ((size_t)1 << R) * 48 + 64;
}

constexpr int kSeqWords = 12;  // per twiddle: ten of its sequence, whether it is nonzero, padding

struct TmapCta {
  uint32_t tile, seqs, mat;  // shared addresses (mat: two matrices, 1024-byte aligned)
  uint32_t bar;              // mbarriers of the products, of the tile's load, of the end; two words
  uint32_t taddr;            // tensor-memory base
  int warp;
  TmRows rows;
  uint32_t phase = 0, phase_ld = 0;
  __device__ __forceinline__ uint32_t bar_ld() const { return bar + 8; }
  __device__ __forceinline__ uint32_t bar_end() const { return bar + 16; }
  // Set once a wait of the CTA ran out: from then on its threads run through
  // their tiles without waiting, loading or starting products, on wrong values.
  // In shared memory and read off the waits' path: with a flag per thread, tested
  // between the barrier and the products' start, a pass takes 1.3 % longer.
  __device__ __forceinline__ uint32_t dead() const { return bar + 28; }
  __device__ __forceinline__ void wait(uint32_t b, uint32_t& ph, uint32_t polls) {
    tm_wait(b, ph, dead(), polls);
    ph ^= 1;
  }
};

// Stage s of the tile in shared memory.
template <bool LAST>
__device__ __forceinline__ void ntt_stage_t(int R, int s, TmapCta& C, const TmShifts& sh, uint32_t polls) {
  const int tid = threadIdx.x, hb = LAST ? 0 : R - 1 - s;
  const uint32_t sq = C.seqs + 4 * kSeqWords * ((1 << s) - 1);
  const uint32_t my = C.taddr + ((uint32_t)(tid & ~31) << 16);  // this warp's 32 lanes
  // the second half of the threads takes the pair after the first half's
  const uint32_t cell = C.tile + 16 * (tid & 63) + ((uint32_t)(tid >> 6) << (LAST ? 11 : 10));
  const uint32_t v_off = 1024u << hb;
  const int n_units = 1 << (R - 2);
  auto base = [&](int u) -> uint32_t {  // the first position of unit u's first pair, as a tile offset
    return (uint32_t)(LAST ? 4 * u : (((2 * u) >> hb) << (hb + 1)) | ((2 * u) & ((1 << hb) - 1))) << 10;
  };
  int u = 0;
  if (!LAST && !tm_lds32(sq + 40))  // block 0 of a layer can have the zero twiddle (the empty sum)
    for (; u < (1 << hb) / 2; u++) {
      const uint32_t c = cell + base(u);
      tm_sts(c + v_off, fx(tm_lds(c + v_off), tm_lds(c)));
    }
  int cur = -1;
  auto start = [&](int w) {
    const int k = LAST ? 2 * w : (2 * w) >> hb;
    tm_put(my + kTmOperand, tm_lds(cell + base(w) + v_off));
    if (LAST || k != cur) {
      tm_product_matrix<0>(sq + 4 * kSeqWords * k, C.rows);
      if (LAST) tm_product_matrix<kTmMatBytes>(sq + 4 * kSeqWords * (k + 1), C.rows);
      tm_fence_smem();
      cur = k;
    }
    const uint32_t dead = tm_lds32(C.dead());
    tm_put_wait();
    tm_fence_before();
    __syncthreads();
    if (C.warp == 0) {
      tm_fence_after();
      if (tm_elect() && !dead) {
        const uint64_t desc = tm_desc(C.mat);
        if (LAST) {
          tm_mma(C.taddr, C.taddr + kTmOperand, desc, 0, ~0u);
          tm_mma(C.taddr, C.taddr + kTmOperand, desc + (kTmMatBytes >> 4), ~0u, 0);
        } else {
          tm_mma(C.taddr, C.taddr + kTmOperand, desc);
        }
        tm_commit(C.bar);
      }
      __syncwarp();
    }
  };
  // Unit u's counts are read back, the next unit is put in and started, and
  // only then are u's counts turned into products: the tensor cores' latency
  // passes behind the extraction.
  if (u < n_units) start(u);
  for (; u < n_units; u++) {
    C.wait(C.bar, C.phase, polls);
    tm_fence_after();
    uint32_t r[32];
    tm_get(my, r);
    if (u + 1 < n_units) start(u + 1);
    const uint32_t c = cell + base(u);
    const f128 a = fx(tm_lds(c), tm_finish_product(tm_extract(r, sh)));
    tm_sts(c, a);
    tm_sts(c + v_off, fx(tm_lds(c + v_off), a));
  }
  if (LAST) tm_fence_smem();  // the tile is stored by bulk copies
  __syncthreads();
}

// Tile t_id of a pass.  seq_hi: the block prefix whose twiddle sequences are in
// shared memory (~0: none); tiles of one prefix are neighbours, so a CTA that
// runs successive tiles derives them rarely, except in the last pass.
__device__ __forceinline__ void ntt_tile_t(const PassArgs& p, uint64_t t_id, uint32_t* seqs, TmapCta& C,
                                           uint64_t& seq_hi, const TmShifts& sh, uint32_t polls) {
  const int R = p.R;
  const int log_d = p.log_d, l0 = p.l0;
  const int lo_bits = log_d - l0 - R;
  const int groups = p.lanes >> 6;
  const int grp = (int)(t_id % groups);
  t_id /= groups;
  const uint64_t lo = t_id & ((1ull << lo_bits) - 1);
  const uint64_t hi = t_id >> lo_bits;
  const int tid = threadIdx.x;
  const size_t row = ((size_t)tid * p.lanes << lo_bits) + ((size_t)grp << 6);  // thread's position of the tile
  f128* const dst = p.data + ((hi << (log_d - l0)) | lo) * p.lanes + row;
  if (C.warp == 0) {  // a row of 64 values per lane (R <= 5)
    tm_store_read();  // the previous tile has left shared memory
    // (no wait lies between the last tile's end and here: one value for the warp)
    const bool live = __all_sync(0xffffffffu, polls && !tm_lds32(C.dead()));
    if (tid == 0 && live) tm_expect(C.bar_ld(), 1024u << R);
    __syncwarp();
    if (tid < (1 << R) && live)
      tm_load_row(C.tile + 1024 * tid, p.src ? p.src + lo * p.lanes + row : dst, 1024, C.bar_ld());
  }
  if (hi != seq_hi) {
    for (int k = tid; k < (1 << R) - 1; k += 128) {
      const int s = 31 - __clz(k + 1), l = l0 + s;
      const uint64_t blk = (hi << s) | (uint64_t)(k + 1 - (1 << s));
      f128 t = mk(0, 0);
#pragma unroll 4
      for (int j = 0; j < l; j++) {
        const f128 e = ldg(p.ev + l * 32 + j);
        const uint64_t m = 0 - ((blk >> j) & 1);
        t.lo ^= e.lo & m;
        t.hi ^= e.hi & m;
      }
      tm_sequence(t, seqs + kSeqWords * k);
      seqs[kSeqWords * k + 10] = !fz(t);
    }
    seq_hi = hi;
    __syncthreads();
  }
  C.wait(C.bar_ld(), C.phase_ld, polls);
  for (int s = 0; s < R - 1; s++) ntt_stage_t<false>(R, s, C, sh, polls);
  ntt_stage_t<true>(R, R - 1, C, sh, polls);
  if (tid < (1 << R)) {
    tm_store_row(dst, C.tile + 1024 * tid, 1024);
    tm_store_commit();
  }
}

// A tensor pass's CTA: shared memory [matrices | tile | sequences | mbarriers,
// address] for passes of at most R layers, tensor memory, mbarrier.
struct TmapSetup {
  TmapCta cta;
  uint32_t* seqs;
  __device__ __forceinline__ TmapSetup(uint8_t* raw, int R) {
    uint8_t* mat = raw + ((1024 - (tm_smem(raw) & 1023)) & 1023);
    uint8_t* tile = mat + 2 * kTmMatBytes;
    seqs = reinterpret_cast<uint32_t*>(tile + ((size_t)1024 << R));
    uint64_t* bar = reinterpret_cast<uint64_t*>(seqs + ((size_t)kSeqWords << R));
    uint32_t* slot = reinterpret_cast<uint32_t*>(bar + 3);  // [tensor-memory address, dead]
    cta.warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
    if (cta.warp == 0) tm_alloc(slot);
    if (threadIdx.x == 0) {
      for (int i = 0; i < 3; i++) tm_mbar_init(bar + i);
      slot[1] = 0;
    }
    tm_fence_before();
    __syncthreads();
    tm_fence_after();
    cta.tile = tm_smem(tile);
    cta.seqs = tm_smem(seqs);
    cta.mat = tm_smem(mat);
    cta.bar = tm_smem(bar);
    cta.taddr = __shfl_sync(0xffffffffu, *slot, 0);
    cta.rows = tm_rows(cta.mat);
  }
  // true: a wait ran out
  __device__ __forceinline__ bool finish() {
    const bool dead = tm_lds32(cta.dead());  // (set before the last tile's last barrier, if at all)
    // products that were started before the thread that starts them saw the word
    if (dead && cta.warp == 0 && tm_elect()) tm_drain(cta.bar_end());
    tm_store_done();
    tm_fence_before();
    __syncthreads();
    if (cta.warp == 0) tm_free(cta.taddr);
    return dead;
  }
};

// per: successive tiles of a CTA
__global__ void __launch_bounds__(128, 4) k_ntt_pass_t(PassArgs p, uint64_t n_tiles, uint64_t per, TmShifts sh,
                                                       WaitLimit w) {
  extern __shared__ __align__(16) uint8_t raw[];
  TmapSetup S(raw, p.R);
  uint64_t seq_hi = ~0ull;
  const uint64_t t0 = blockIdx.x * per, t1 = min(t0 + per, n_tiles);
  for (uint64_t t = t0; t < t1; t++) ntt_tile_t(p, t, S.seqs, S.cta, seq_hi, sh, w.polls);
  if (S.finish() && threadIdx.x == 0) *w.ran_out = 1;
}

template <bool TRANSPOSE, int KIND>
__global__ void __launch_bounds__(256, 1) k_ntt_pass_w(PassArgs p) {
  extern __shared__ f128 smem[];
  ntt_tile_w<TRANSPOSE, KIND>(p, blockIdx.x, smem);
}

template <bool TRANSPOSE>
__global__ void __launch_bounds__(256, 2) k_ntt_pass(PassArgs p) {
  extern __shared__ f128 smem[];
  ntt_tile<TRANSPOSE>(p, blockIdx.x, smem);
}

// Pass `pass` of every job of a batch: a persistent grid strides over the
// tiles of all jobs (each job's tiles numbered from its tile0[pass]).
__global__ void __launch_bounds__(256, 2) k_ntt_pass_batch(const BatchJob* __restrict__ jobs, int n_jobs, int pass,
                                                           uint64_t total_tiles) {
  extern __shared__ f128 smem[];
  for (uint64_t t = blockIdx.x; t < total_tiles; t += gridDim.x) {
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (jobs[mid].tile0[pass] <= t) lo = mid;
      else hi = mid - 1;
    }
    const BatchJob& J = jobs[lo];
    const NttPass& ps = J.pass[pass];
    PassArgs a{J.cw, J.ev, J.log_d, 64, ps.lgs, ps.l0, ps.R};
    if (pass == 0) {  // rate 1/2: the message fills both halves of the codeword
      a.src = J.z;
      a.src_mask = ((uint64_t)1 << (J.log_d - 1)) - 1;
    }
    __syncthreads();  // the previous tile's stores have read the shared tile
    if (ps.kind == 1) ntt_tile_w<false, 1>(a, t - J.tile0[pass], smem);
    else if (ps.kind == 2) ntt_tile_w<false, 2>(a, t - J.tile0[pass], smem);
    else ntt_tile<false>(a, t - J.tile0[pass], smem);
  }
}

// The same for the jobs whose pass runs on the tensor cores.
__global__ void __launch_bounds__(128, 4) k_ntt_pass_batch_t(const BatchJob* __restrict__ jobs, int n_jobs, int pass,
                                                             uint64_t total_tiles, uint64_t per, int max_R, TmShifts sh,
                                                             uint32_t polls) {
  extern __shared__ __align__(16) uint8_t raw[];
  TmapSetup S(raw, max_R);
  uint64_t seq_hi = ~0ull;
  int job = -1;
  const uint64_t t0 = blockIdx.x * per, t1 = min(t0 + per, total_tiles);
  for (uint64_t t = t0; t < t1; t++) {
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (jobs[mid].tile0t[pass] <= t) lo = mid;
      else hi = mid - 1;
    }
    const BatchJob& J = jobs[lo];
    const NttPass& ps = J.pass[pass];
    PassArgs a{J.cw, J.ev, J.log_d, 64, ps.lgs, ps.l0, ps.R};
    if (pass == 0) {  // rate 1/2: the message fills both halves of the codeword
      a.src = J.z;
      a.src_mask = ((uint64_t)1 << (J.log_d - 1)) - 1;
    }
    if (lo != job) seq_hi = ~0ull;
    job = lo;
    ntt_tile_t(a, t - J.tile0t[pass], S.seqs, S.cta, seq_hi, sh, polls);
  }
  if (S.finish())  // the jobs that had tiles here
    for (int j = threadIdx.x; j < n_jobs; j += 128)
      if (jobs[j].tile0t[pass] < t1 && (j + 1 < n_jobs ? jobs[j + 1].tile0t[pass] : total_tiles) > t0)
        *jobs[j].ran_out = 1;
}

__global__ void k_replicate_batch(const BatchJob* __restrict__ jobs, int n_jobs, uint64_t total) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  int lo = 0, hi = n_jobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].rep0 <= i) lo = mid;
    else hi = mid - 1;
  }
  const BatchJob& J = jobs[lo];
  const uint64_t k = i - J.rep0;  // rate 1/2: the message and one copy
  const f128 v = ld(J.z + k);
  st(J.cw + k, v);
  st(J.cw + J.msg_len + k, v);
}

__global__ void k_replicate(const f128* __restrict__ msg, f128* __restrict__ cw, size_t msg_len, int copies) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= msg_len) return;
  f128 v = ld(msg + i);
  for (int c = 0; c < copies; c++) st(cw + (size_t)c * msg_len + i, v);
}

// SplitMix64 words: the tuner's scratch holds random values, so that the table
// passes' lookups meet the nibble patterns of real data (all-zero data would
// turn every lookup into a broadcast and time those passes too fast)
__global__ void k_fill_random(uint64_t* p, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t z = (i + 1) * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  p[i] = z ^ (z >> 31);
}

__global__ void k_fold_copies(const f128* __restrict__ in, f128* __restrict__ out, size_t len, int copies) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= len) return;
  f128 acc = ld(in + i);
  for (int c = 1; c < copies; c++) acc = fx(acc, ld(in + (size_t)c * len + i));
  st(out + i, acc);
}

// Host-computed per-dimension basis table (additive_ntt_f128.rs:54-87).
std::vector<f128> layer_basis(int dim) {
  std::vector<std::vector<f128>> evals;
  std::vector<f128> basis(dim);
  for (int i = 0; i < dim; i++) basis[i] = mk(i < 64 ? 1ull << i : 0, i < 64 ? 0 : 1ull << (i - 64));
  evals.push_back(basis);
  for (int i = 1; i < dim; i++) {
    std::vector<f128> row;
    const auto& prev = evals[i - 1];
    for (size_t k = 1; k < prev.size(); k++) row.push_back(flock::hmul(prev[k], fx(prev[k], prev[0])));
    evals.push_back(row);
  }
  for (auto& row : evals) {
    f128 inv = flock::hinv(row[0]);
    for (auto& v : row) v = flock::hmul(v, inv);
  }
  std::vector<f128> tab((size_t)32 * 32, mk(0, 0));
  for (int l = 0; l < dim; l++)
    for (int j = 0; j < l; j++) tab[l * 32 + j] = evals[dim - l - 1][1 + j];
  return tab;
}
const f128* device_evals(int dim) {
  static std::mutex mu;
  static std::map<int, f128*> cache;
  std::lock_guard<std::mutex> lk(mu);
  auto it = cache.find(dim);
  if (it != cache.end()) return it->second;
  const std::vector<f128> tab = layer_basis(dim);
  f128* d = nullptr;
  CK(cudaMalloc(&d, tab.size() * sizeof(f128)));
  CK(cudaMemcpy(d, tab.data(), tab.size() * sizeof(f128), cudaMemcpyHostToDevice));
  cache[dim] = d;
  return d;
}

// The tensor-core passes add two counts in one word and need the first to stay
// below 128 (tmap.cuh): a row of a twiddle's matrix may not be all ones.  The
// elements with such a row are s x^-o, where the top bit of s x^k is 1 for
// every k < 128; true when no layer's twiddles (the sums of its basis values)
// contain one.
bool tensor_safe(int dim) {
  static std::mutex mu;
  static std::map<int, bool> cache;
  std::lock_guard<std::mutex> lk(mu);
  auto it = cache.find(dim);
  if (it != cache.end()) return it->second;
  f128 s{};
  for (int low = 0; low < 128; low++) {  // bits 7..127 are the first 121 top bits
    const f128 c = mk(~0ull << 7 | (uint64_t)low, ~0ull);
    f128 t = c;
    bool all = true;
    for (int k = 0; k < 128 && all; k++, t = mul_xk(t, 1)) all = t.hi >> 63;
    if (all) s = c;
  }
  if (fz(s)) return cache[dim] = false;
  const std::vector<f128> tab = layer_basis(dim);
  bool ok = true;
  for (int l = 1; l < dim && ok; l++) {
    std::vector<f128> basis;  // reduced, with distinct leading bits
    auto lead = [](f128 v) { return v.hi ? 127 - __builtin_clzll(v.hi) : 63 - __builtin_clzll(v.lo); };
    auto reduce_by = [&](f128 v) {
      for (const f128& b : basis) {
        const int t = lead(b);
        if ((t < 64 ? v.lo >> t : v.hi >> (t - 64)) & 1) v = fx(v, b);
      }
      return v;
    };
    for (int j = 0; j < l; j++) {
      const f128 v = reduce_by(tab[l * 32 + j]);
      if (!fz(v)) basis.push_back(v);
    }
    f128 t = s;
    for (int o = 0; o < 128 && ok; o++) {
      ok = !fz(reduce_by(t));
      t = t.lo & 1 ? mk((t.lo ^ 0x87) >> 1 | t.hi << 63, t.hi >> 1 | 1ull << 63) : mk(t.lo >> 1 | t.hi << 63, t.hi >> 1);
    }
  }
  return cache[dim] = ok;
}

// ---------------------------------------------------------------- plans --
// A plan is the list of passes (first layer, layer count R, lanes per tile
// 2^lgs, threads per CTA) that covers layers layer_begin..log_d-1.  The
// autotuner times candidate splits of the layers and, for each pass, the
// tile widths and CTA sizes that fit one or two CTAs per SM, and keeps the
// fastest combination per (device, log_d, lanes, layer_begin).

size_t pass_smem(int lgs, int R) { return ((size_t)(1 << lgs) << R) * sizeof(f128) + ((1 << R) - 1) * sizeof(f128); }
constexpr size_t kSmem2 = (size_t)112 << 10;  // two CTAs per SM
constexpr size_t kSmem1 = (size_t)200 << 10;  // one CTA per SM

int max_lgs(int lanes) {
  int g = 0;
  while ((1 << (g + 1)) <= lanes && g < 3) g++;
  return g;
}

std::vector<std::pair<int, int>> balanced_split(int begin, int n_layers, int n_pass) {
  std::vector<std::pair<int, int>> v;
  int l = begin;
  for (int i = 0; i < n_pass; i++) {
    int R = (n_layers - (l - begin) + (n_pass - i) - 1) / (n_pass - i);
    v.push_back({l, R});
    l += R;
  }
  return v;
}

// layer splits to try: the balanced split into the fewest passes of <= 10
// layers, its mirror, a split with one 11-layer pass, and one more pass
std::vector<std::vector<std::pair<int, int>>> candidate_splits(int begin, int n_layers) {
  std::vector<std::vector<std::pair<int, int>>> out;
  auto add = [&](std::vector<std::pair<int, int>> v) {
    for (auto& x : out)
      if (x == v) return;
    for (auto& pr : v)
      if (pr.second < 1 || pr.second > kMaxR + 1) return;
    out.push_back(v);
  };
  const int p0 = (n_layers + kMaxR - 1) / kMaxR;
  auto bal = balanced_split(begin, n_layers, p0);
  add(bal);
  if (p0 >= 2) {  // mirror: the larger passes last
    std::vector<int> Rs;
    for (auto& pr : bal) Rs.push_back(pr.second);
    std::reverse(Rs.begin(), Rs.end());
    std::vector<std::pair<int, int>> v;
    int l = begin;
    for (int R : Rs) { v.push_back({l, R}); l += R; }
    add(v);
  }
  if (n_layers == kMaxR + 1) add({{begin, n_layers}});
  if (p0 == 2 && n_layers > 11) {
    add({{begin, 11}, {begin + 11, n_layers - 11}});
    add({{begin, n_layers - 11}, {begin + n_layers - 11, 11}});
  }
  if (n_layers >= p0 + 1) add(balanced_split(begin, n_layers, p0 + 1));
  return out;
}

// splits for the warp-per-pair passes (at most kMaxRw layers: a 64-lane tile
// and the warps' tables share the CTA's shared memory)
constexpr int kMaxRw = 7;
std::vector<std::vector<std::pair<int, int>>> candidate_splits_w(int begin, int n_layers) {
  std::vector<std::vector<std::pair<int, int>>> out;
  const int p0 = (n_layers + kMaxRw - 1) / kMaxRw;
  for (int np = p0; np <= p0 + 1 && np <= n_layers; np++) {
    auto v = balanced_split(begin, n_layers, np);
    bool ok = true;
    for (auto& pr : v) ok = ok && pr.second >= 4 && pr.second <= kMaxRw;
    if (ok) out.push_back(v);
  }
  return out;
}

// per-pass launch shapes to try: (lgs, threads) of the thread-per-pair passes
std::vector<std::pair<int, int>> candidate_shapes(int lanes, int R) {
  std::vector<std::pair<int, int>> out;
  const int top = max_lgs(lanes);
  int g2 = top;
  while (g2 > 0 && pass_smem(g2, R) > kSmem2) g2--;
  int g1 = top;
  while (g1 > 0 && pass_smem(g1, R) > kSmem1) g1--;
  std::vector<int> gs = {g2};
  if (g2 > 0) gs.push_back(g2 - 1);
  if (g1 > g2) gs.push_back(g1);
  for (int g : gs) {
    if (pass_smem(g, R) > kSmem1) continue;
    const int work = ((1 << g) << R) / 2;  // butterflies per stage
    for (int t : {128, 256}) {
      if (t > std::max(32, work)) continue;
      out.push_back({g, t});
    }
    if (out.empty() || out.back().first != g) out.push_back({g, std::min(256, std::max(32, work))});
  }
  return out;
}

// splits for the tensor-core passes: as few passes of 2 to kMaxRt layers as
// cover the layers, and one more (smaller tiles, more of them in flight)
std::vector<std::vector<std::pair<int, int>>> candidate_splits_t(int lanes, int begin, int n_layers) {
  std::vector<std::vector<std::pair<int, int>>> out;
  if (lanes % 64 || !tensor_safe(begin + n_layers)) return out;
  const int p0 = (n_layers + kMaxRt - 1) / kMaxRt;
  for (int np = p0; np <= p0 + 1 && np <= n_layers; np++) {
    auto v = balanced_split(begin, n_layers, np);
    bool ok = true;
    for (auto& pr : v) ok = ok && pr.second >= 2 && pr.second <= kMaxRt;
    if (ok) out.push_back(v);
  }
  return out;
}

// From 2^kTensorMinLog positions on there are tiles enough for the SMs and the
// tensor-core passes are the fastest of all kinds (2^12 positions x 64 lanes:
// 0.046 ms against 0.057 ms for the best mix of the others; 2^14: 0.121 / 0.167;
// 2^20: 7.49 / 11.8 ms; 2^10: 0.028 against 0.026 ms for the integer products),
// so only their splits are timed there.
constexpr int kTensorMinLog = 12;

// the warp-per-pair shapes of a pass of R layers: (threads, kind) with the
// tile and every warp's table within one CTA's shared memory
std::vector<NttPass> candidate_shapes_w(int lanes, int l0, int R) {
  std::vector<NttPass> out;
  if (lanes % 64 || R < 4 || R > kMaxRw) return out;
  for (int kind : {1, 2})
    for (int t : {64, 128, 256}) {
      if (t / 32 > (1 << (R - 1)) || pass_w_smem(R, t) > kSmem1) continue;
      NttPass p{l0, R, 6, t};
      p.kind = kind;
      out.push_back(p);
    }
  return out;
}

// successive tiles per CTA of a tensor-core pass: enough to share their
// twiddles and hide the CTA's start, few enough that other streams' kernels
// find free SMs soon (a batch's commits run beside other proofs' rounds; CTAs
// that strode over all of a pass held every SM for milliseconds)
uint64_t tiles_per_cta(uint64_t tiles, int sms) {
  return std::max<uint64_t>(1, std::min<uint64_t>(8, tiles / ((uint64_t)sms * 4)));
}

template <bool TR>
void launch_pass_w(const NttPass& ps, const PassArgs& a, uint64_t tiles, cudaStream_t s) {
  auto k = ps.kind == 1 ? k_ntt_pass_w<TR, 1> : k_ntt_pass_w<TR, 2>;
  CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem1));
  count_launch();
  k<<<(unsigned)tiles, ps.threads, pass_w_smem(ps.R, ps.threads), s>>>(a);
}

void launch_pass(const NttPass& ps, f128* data, const f128* ev, int log_d, int lanes, bool transpose,
                 cudaStream_t s, const WaitLimit& w, const f128* src = nullptr) {
  PassArgs a{data, ev, log_d, lanes, ps.lgs, ps.l0, ps.R};
  if (src) {
    a.src = src;
    a.src_mask = ((uint64_t)1 << (log_d - ps.l0)) - 1;
  }
  const size_t smem = pass_smem(ps.lgs, ps.R);
  const uint64_t tiles = ((uint64_t)1 << (log_d - ps.R)) * (uint64_t)(lanes >> ps.lgs);
  if (ps.kind == 3) {
    if (transpose) throw CudaError("ntt: tensor passes run forward only");
    if (!w.ran_out) throw CudaError("ntt: a tensor pass needs a word for its waits");
    CK(cudaFuncSetAttribute(k_ntt_pass_t, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pass_t_smem(kMaxRt)));
    int dev = 0, sms = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const uint64_t per = tiles_per_cta(tiles, sms);
    count_launch();
    k_ntt_pass_t<<<(unsigned)((tiles + per - 1) / per), 128, pass_t_smem(ps.R), s>>>(a, tiles, per, tm_shifts(), w);
    return;
  }
  if (ps.kind) {
    if (transpose) launch_pass_w<true>(ps, a, tiles, s);
    else launch_pass_w<false>(ps, a, tiles, s);
    return;
  }
  // The attribute is the same upper bound for every launch: it is global to
  // the kernel, so a per-launch size set by one host thread could undercut
  // another thread's launch of a larger tile.
  if (transpose) {
    CK(cudaFuncSetAttribute(k_ntt_pass<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem1));
    count_launch(); k_ntt_pass<true><<<(unsigned)tiles, ps.threads, smem, s>>>(a);
  } else {
    CK(cudaFuncSetAttribute(k_ntt_pass<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem1));
    count_launch(); k_ntt_pass<false><<<(unsigned)tiles, ps.threads, smem, s>>>(a);
  }
}

NttPlan default_plan(int log_d, int lanes, int layer_begin) {
  NttPlan plan;
  const int n_layers = log_d - layer_begin;
  if (n_layers <= 0) return plan;
  const auto tensor = candidate_splits_t(lanes, layer_begin, n_layers);
  if (!tensor.empty() && log_d >= kTensorMinLog) {
    for (auto& pr : tensor[0]) plan.push_back({pr.first, pr.second, 6, 128, 3});
    return plan;
  }
  for (auto& pr : balanced_split(layer_begin, n_layers, (n_layers + kMaxR - 1) / kMaxR)) {
    int g = max_lgs(lanes);
    while (g > 0 && pass_smem(g, pr.second) > kSmem2) g--;
    plan.push_back({pr.first, pr.second, g, std::min(256, std::max(32, ((1 << g) << pr.second) / 2))});
  }
  return plan;
}

// every plan the tuner may pick: each candidate split with each launch shape
// applied to all of its passes (for parity tests of the tiling)
std::vector<NttPlan> all_plans(int log_d, int lanes, int layer_begin) {
  std::vector<NttPlan> out;
  const int n_layers = log_d - layer_begin;
  if (n_layers <= 0) return {NttPlan{}};
  for (auto& split : candidate_splits(layer_begin, n_layers)) {
    size_t n_shapes = 0;
    for (auto& pr : split) n_shapes = std::max(n_shapes, candidate_shapes(lanes, pr.second).size());
    for (size_t k = 0; k < n_shapes; k++) {
      NttPlan plan;
      for (auto& pr : split) {
        auto sh = candidate_shapes(lanes, pr.second);
        auto& c = sh[std::min(k, sh.size() - 1)];
        plan.push_back({pr.first, pr.second, c.first, c.second});
      }
      out.push_back(plan);
    }
  }
  for (auto& split : candidate_splits_w(layer_begin, n_layers)) {
    size_t n_shapes = 0;
    for (auto& pr : split) n_shapes = std::max(n_shapes, candidate_shapes_w(lanes, pr.first, pr.second).size());
    for (size_t k = 0; k < n_shapes; k++) {
      NttPlan plan;
      for (auto& pr : split) {
        auto sh = candidate_shapes_w(lanes, pr.first, pr.second);
        if (!sh.empty()) plan.push_back(sh[std::min(k, sh.size() - 1)]);
      }
      if (plan.size() == split.size()) out.push_back(plan);
    }
  }
  for (auto& split : candidate_splits_t(lanes, layer_begin, n_layers)) {
    NttPlan plan;
    for (auto& pr : split) plan.push_back({pr.first, pr.second, 6, 128, 3});
    out.push_back(plan);
  }
  return out;
}

struct PlanKey {
  int device, log_d, lanes, begin;
  bool operator<(const PlanKey& o) const {
    return std::tie(device, log_d, lanes, begin) < std::tie(o.device, o.log_d, o.lanes, o.begin);
  }
};
std::mutex g_plan_mu;
std::map<PlanKey, NttPlan>& tuned_plans() {
  static std::map<PlanKey, NttPlan> m;
  return m;
}

NttPlan plan_for(int log_d, int lanes, int layer_begin) {
  int dev = 0;
  CK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_plan_mu);
  auto it = tuned_plans().find({dev, log_d, lanes, layer_begin});
  return it != tuned_plans().end() ? it->second : default_plan(log_d, lanes, layer_begin);
}

// src != nullptr (forward only): the message whose replicate the first pass
// reads in place of data
void run_plan(const NttPlan& plan, f128* data, int log_d, int lanes, bool transpose, cudaStream_t s,
              const WaitLimit& w, const f128* src = nullptr) {
  if (plan.empty()) return;
  const f128* ev = device_evals(log_d);
  if (transpose)
    for (auto it = plan.rbegin(); it != plan.rend(); ++it) launch_pass(*it, data, ev, log_d, lanes, true, s, w);
  else
    for (size_t i = 0; i < plan.size(); i++)
      launch_pass(plan[i], data, ev, log_d, lanes, false, s, w, i ? nullptr : src);
}

void run_passes(f128* data, int log_d, int lanes, int layer_begin, bool transpose, cudaStream_t s,
                const WaitLimit& w) {
  run_plan(plan_for(log_d, lanes, layer_begin), data, log_d, lanes, transpose, s, w);
}
}  // namespace

void ntt_replicate_batch(const BatchJob* jobs, int n_jobs, uint64_t total, cudaStream_t s) {
  count_launch();
  k_replicate_batch<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(jobs, n_jobs, total);
}
// the batched pass kernel runs 256 threads: a warp-per-pair pass holds 8 tables
size_t ntt_pass_batch_smem(const NttPass& p) { return p.kind ? pass_w_smem(p.R, 256) : pass_smem(p.lgs, p.R); }
void ntt_pass_batch(const BatchJob* jobs, int n_jobs, int pass, uint64_t total_tiles, size_t smem, int grid,
                    cudaStream_t s) {
  if (smem > kSmem1) throw CudaError("ntt_pass_batch: tile larger than the shared-memory bound");
  CK(cudaFuncSetAttribute(k_ntt_pass_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem1));
  count_launch();
  k_ntt_pass_batch<<<(unsigned)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)grid, total_tiles)), 256, smem, s>>>(
      jobs, n_jobs, pass, total_tiles);
}

void ntt_pass_batch_t(const BatchJob* jobs, int n_jobs, int pass, uint64_t total_tiles, int max_R, int sms,
                      cudaStream_t s, unsigned polls) {
  const size_t smem = pass_t_smem(max_R);
  CK(cudaFuncSetAttribute(k_ntt_pass_batch_t, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pass_t_smem(kMaxRt)));
  const uint64_t per = tiles_per_cta(total_tiles, sms);
  count_launch();
  k_ntt_pass_batch_t<<<(unsigned)((total_tiles + per - 1) / per), 128, smem, s>>>(
      jobs, n_jobs, pass, total_tiles, per, max_R, tm_shifts(), polls);
}

NttPlan ntt_autotune(f128* scratch, int log_d, int lanes, int layer_begin, cudaStream_t s, const WaitLimit& w,
                     double* best_ms) {
  int dev = 0;
  CK(cudaGetDevice(&dev));
  const PlanKey key{dev, log_d, lanes, layer_begin};
  {
    std::lock_guard<std::mutex> lk(g_plan_mu);
    auto it = tuned_plans().find(key);
    if (it != tuned_plans().end()) {
      if (best_ms) *best_ms = -1;
      return it->second;
    }
  }
  const int n_layers = log_d - layer_begin;
  if (n_layers <= 0) return {};
  const f128* ev = device_evals(log_d);
  {
    const size_t words = ((size_t)lanes << log_d) * 2;
    count_launch();
    k_fill_random<<<(unsigned)((words + 255) / 256), 256, 0, s>>>(reinterpret_cast<uint64_t*>(scratch), words);
    CK(cudaGetLastError());
  }
  struct Events {
    cudaEvent_t e[2] = {nullptr, nullptr};
    ~Events() {
      for (cudaEvent_t v : e)
        if (v) cudaEventDestroy(v);
    }
  } events;
  cudaEvent_t &e0 = events.e[0], &e1 = events.e[1];
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  // one warm launch, then the best of two timed launches (CUDA events on
  // the launching stream), on the random scratch filled above
  auto time_pass = [&](const NttPass& ps) {
    launch_pass(ps, scratch, ev, log_d, lanes, false, s, w);
    float best = 1e30f;
    for (int r = 0; r < 2; r++) {
      CK(cudaEventRecord(e0, s));
      launch_pass(ps, scratch, ev, log_d, lanes, false, s, w);
      CK(cudaEventRecord(e1, s));
      CK(cudaEventSynchronize(e1));
      check_waits(w);  // the time of a pass that gave up is no time
      float t = 0;
      CK(cudaEventElapsedTime(&t, e0, e1));
      best = std::min(best, t);
    }
    return (double)best;
  };
  std::map<std::pair<int, int>, std::pair<NttPass, double>> best_pass;  // (l0, R) -> fastest shape
  NttPlan best_plan;
  double best_total = 1e300;
  const auto tensor = candidate_splits_t(lanes, layer_begin, n_layers);
  const bool tensor_only = !tensor.empty() && log_d >= kTensorMinLog;
  std::vector<std::vector<std::pair<int, int>>> splits;
  if (!tensor_only) {
    splits = candidate_splits(layer_begin, n_layers);
    for (auto& sp : candidate_splits_w(layer_begin, n_layers))
      if (std::find(splits.begin(), splits.end(), sp) == splits.end()) splits.push_back(sp);
  }
  for (auto& sp : tensor)
    if (std::find(splits.begin(), splits.end(), sp) == splits.end()) splits.push_back(sp);
  for (auto& split : splits) {
    NttPlan plan;
    double total = 0;
    for (auto& pr : split) {
      auto it = best_pass.find(pr);
      if (it == best_pass.end()) {
        NttPass bp{};
        double bt = 1e300;
        std::vector<NttPass> shapes;
        if (!tensor_only) {
          if (pr.second <= kMaxR + 1)
            for (auto& sh : candidate_shapes(lanes, pr.second))
              shapes.push_back({pr.first, pr.second, sh.first, sh.second});
          for (auto& ps : candidate_shapes_w(lanes, pr.first, pr.second)) shapes.push_back(ps);
        }
        if (lanes % 64 == 0 && pr.second >= 2 && pr.second <= kMaxRt && tensor_safe(log_d))
          shapes.push_back({pr.first, pr.second, 6, 128, 3});
        for (auto& ps : shapes) {
          const double t = time_pass(ps);
          if (t < bt) { bt = t; bp = ps; }
        }
        it = best_pass.emplace(pr, std::make_pair(bp, bt)).first;
      }
      plan.push_back(it->second.first);
      total += it->second.second;
    }
    if (total < best_total) { best_total = total; best_plan = plan; }
  }
  std::lock_guard<std::mutex> lk(g_plan_mu);
  tuned_plans()[key] = best_plan;
  if (best_ms) *best_ms = best_total;
  return best_plan;
}

NttPlan ntt_plan(int log_d, int lanes, int layer_begin) { return plan_for(log_d, lanes, layer_begin); }
const f128* ntt_evals(int log_d) { return device_evals(log_d); }

std::string ntt_plan_desc(const NttPlan& plan) {
  std::string d;
  for (auto& ps : plan) {
    if (!d.empty()) d += " + ";
    d += "R" + std::to_string(ps.R) + "@l" + std::to_string(ps.l0) + " x" + std::to_string(1 << ps.lgs) +
         " lanes/" + std::to_string(ps.threads) + "t" + (ps.kind == 1 ? "/tab" : ps.kind == 2 ? "/tab+imad" : ps.kind == 3 ? "/mma" : "");
  }
  return d;
}

size_t ntt_plan_count(int log_d, int lanes, int layer_begin) { return all_plans(log_d, lanes, layer_begin).size(); }
std::string ntt_plan_desc_at(int log_d, int lanes, int layer_begin, size_t index) {
  const auto plans = all_plans(log_d, lanes, layer_begin);
  return index < plans.size() ? ntt_plan_desc(plans[index]) : std::string();
}

void ntt_rs_encode_plan(const f128* msg, f128* cw, int log_msg_pos, int lanes, int log_inv_rate, size_t plan_idx,
                        cudaStream_t s, const WaitLimit& w) {
  const int log_d = log_msg_pos + log_inv_rate;
  auto plans = all_plans(log_d, lanes, log_inv_rate);
  if (plan_idx >= plans.size()) throw std::out_of_range("ntt plan index");
  size_t msg_len = ((size_t)lanes) << log_msg_pos;
  if (plans[plan_idx].empty() || plans[plan_idx][0].l0 != log_inv_rate) {
    count_launch(); k_replicate<<<(unsigned)((msg_len + 255) / 256), 256, 0, s>>>(msg, cw, msg_len, 1 << log_inv_rate);
    run_plan(plans[plan_idx], cw, log_d, lanes, false, s, w);
  } else {
    run_plan(plans[plan_idx], cw, log_d, lanes, false, s, w, msg);
  }
}

void ntt_rs_encode(const f128* msg, f128* cw, int log_msg_pos, int lanes, int log_inv_rate, cudaStream_t s,
                   const WaitLimit& w) {
  const int log_d = log_msg_pos + log_inv_rate;
  const NttPlan plan = plan_for(log_d, lanes, log_inv_rate);
  if (plan.empty()) {  // no butterfly layer: the codeword is the replicate
    size_t msg_len = ((size_t)lanes) << log_msg_pos;
    count_launch(); k_replicate<<<(unsigned)((msg_len + 255) / 256), 256, 0, s>>>(msg, cw, msg_len, 1 << log_inv_rate);
    return;
  }
  run_plan(plan, cw, log_d, lanes, false, s, w, msg);  // the first pass reads the message's replicate in place
}

void ntt_forward(f128* data, int log_d, int lanes, int start_layer, cudaStream_t s, const WaitLimit& w) {
  run_passes(data, log_d, lanes, start_layer, false, s, w);
}

// out[j] (j < 2^log_msg) = sum_q E[q] * (codeword position q of unit message j);
// e is overwritten.
void ntt_transposed_encode(f128* e, f128* out, int log_msg, int log_inv_rate, cudaStream_t s) {
  run_passes(e, log_msg + log_inv_rate, 1, log_inv_rate, true, s, WaitLimit{});  // (no kernel of these waits)
  size_t len = (size_t)1 << log_msg;
  count_launch(); k_fold_copies<<<(unsigned)((len + 255) / 256), 256, 0, s>>>(e, out, len, 1 << log_inv_rate);
}
