// Batched 16-bit-operand GEMM with FP32 accumulation in tensor memory, for sm_100a.
//
//   D[b] = alpha_b * sum_seg A_seg[b] * B_seg[b]^T   (+ beta_b * C[b])
//
// One persistent CTA per SM (or one CTA pair per SM pair: cta_group::2, 256 x 128, 256 x 256 or 256 x 512 tiles),
// warp-specialised:
//   warps 0, 2  TMA producers: 128-byte-swizzled tiles of A (warp 0) and of B (warp 2) into a shared-memory ring
//   warp 1      allocates tensor memory and issues tcgen05.mma (one thread), accumulating in TMEM
//   warps 4..11 epilogue: tcgen05.ld the accumulator (double-buffered, so it overlaps the next chain's
//               MMAs), sum chains in registers, apply the affine epilogue, store FP32 / 16-bit results
// The tensor core adds every 16-deep partial sum into its FP32 accumulator by truncation; over long K
// that bias reaches 1e-5 relative.  Where FP32 accuracy matters (`promote`), accumulation chains are
// kept short in TMEM and summed with round-to-nearest by the epilogue warps.
// Operands may be stored K-major (k contiguous) or MN-major (m or n contiguous: a transposed view, as
// in X^T X); symmetric results can be computed from the tiles that meet the upper triangle only and
// mirrored on store.  "Segments" concatenate several operand planes along K into one accumulator,
// which is how the FP32-accurate product  Ah*Bh + Ah*Bl + Al*Bh  of FP16 hi/lo splits is formed.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "ptx.cuh"

namespace toner {

constexpr int kBM = 128;          // tile rows (UMMA M)
constexpr int kBK = 64;           // 16-bit elements per k-block: one 128-byte swizzle row
constexpr int kUmmaK = 16;        // K per tcgen05.mma for 16-bit operands
constexpr int kMaxSegs = 3;
constexpr int kGemmThreads = 384;      // warpgroup 0: A's TMA warp, MMA warp, B's TMA warp, one idle; warpgroups 1-2: epilogue
constexpr long long kWaitCycles = 4000000000LL;  // about two seconds; a healthy wait is microseconds
constexpr long long kDrainCycles = 2000000LL;    // per stage, after an abort: about a millisecond for copies in flight
constexpr long long kSettleCycles = 200000LL;    // after an abort: a CTA of a pair lets copies it cannot observe land

enum GemmStatus : int { kOk = 0, kTimeoutProducer = 101, kTimeoutMma = 102, kTimeoutEpilogue = 103, kTimeoutSelftest = 199 };

struct GemmParams {
  // operands: one 3-D tensor map (inner, outer, z) each, or an array in global memory with one map per batch
  CUtensorMap a_map, b_map;
  const CUtensorMap* a_maps;   // non-null: separately allocated matrices
  const CUtensorMap* b_maps;
  int a_z_stride, b_z_stride;      // z coordinate = batch * z_stride + seg_z[seg]
  int a_mn, b_mn;                  // 1: stored MN-major (outer index is k), 0: K-major (outer index is m / n)
  int a_seg_z[kMaxSegs], b_seg_z[kMaxSegs];
  int segs;
  int M, N, K, batch;
  int fmt;  // operand format: 0 FP16, 1 BF16
  int tri;  // 1: M == N, only tiles meeting the upper triangle are computed
  int promote;  // > 0: k-blocks per tensor-core accumulation chain; chains are summed in FP32 registers
  int promote_all;  // 0: only the first segment is chained (split products); 1: every segment
  // splits > 1: the accumulation of every tile is divided among that many units.  Each epilogue warp leaves its part of the
  // partial sums in split_part and counts itself in at split_count (zeroed before the launch); the last of a tile's warps
  // adds the parts in the order of the splits -- whoever comes last, so the result is reproducible -- and writes the result.
  int splits;
  float* split_part;
  unsigned int* split_count;
  int raster;   // tile columns per rasterisation group (full schedules): keeps a group's B panels in L2
  // epilogue: d = alpha * acc + beta * C ; alpha, beta optionally scaled per batch from device arrays
  float alpha, beta;
  const float* alpha_a;
  const float* alpha_b;
  const float* beta_v;
  int alpha_b_step;
  const float* C;
  long long ldc, c_bs;
  float* D;
  long long ldd, d_bs;
  void* D16;
  long long ld16, d16_bs;
  int d16_fmt;  // 0 FP16, 1 BF16
  int packed;   // C and D are packed upper triangles (row r starts at r*N - r(r-1)/2 - r ... see packed_off)
  int mirror;   // tri: also store the transposed element
  int upper_d;  // tri + mirror: the FP32 result D is not mirrored (its lower triangle is never read)
  int tma_ok;   // C and every output can be moved by TMA (16-byte bases and strides): *_map below are valid
  int s_lo_z;   // the lo plane of an operand-plane output is s_lo_z batches behind the hi plane in s0_map / s1_map
  float* sumsq;           // per batch: sum of d^2 over the full (mirrored) result
  unsigned int* maxabs;   // per batch: max |d| as FP32 bits
  unsigned int* maxaff;   // per batch: max |aff_a * [r==c] + aff_b * d| as FP32 bits
  float aff_a, aff_b;
  unsigned int* maxres;   // per batch: max |[r==c] - d| as FP32 bits (distance of the result from the identity)
  // optional FP16 hi/lo operand planes of the result, ready to feed the next split-precision product:
  //   S0: planes of s0_scale * (s0_aff_a * [r==c] + d)            S1: planes of s1_scale * (s1_aff_a * [r==c] + s1_aff_b * d)
  // hi plane at S + b * s_bs + r * s_ld + c, lo plane s_plane elements further
  __half* S0;
  __half* S1;
  long long s_ld, s_bs, s_plane;
  float s0_scale, s0_aff_a, s1_scale, s1_aff_a, s1_aff_b;
  // Symmetric matrices of which only the 256 x 256 blocks on and above the diagonal are stored, these whole.  Both operands (kernels
  // with kHalf): a k-block left of an operand's rows' own block is read from its mirror image, MN-major, through the *_turned maps
  // (64 x 64 boxes).  half_out: the operand planes S0 and S1.
  int half_out;
  const int* skip;   // optional, per batch: not zero where the product is left out (its outputs keep what they hold)
  int* status;  // set non-zero if a bounded wait ran out
  unsigned long long* prof;  // optional: eight cycle counters summed over CTAs (see toner_gemm_phase_cycles)
  // 32 x 32 boxes of C and of the outputs, (columns, rows, batch): FP32 with 128-byte, 16-bit with 64-byte swizzle
  CUtensorMap c_map, d_map, h_map, s0_map, s1_map;
  CUtensorMap a_turned, b_turned;
};
constexpr int kHalfShift = 8;   // log2 of the blocks of half-stored matrices: tiles of every size lie in one of them

__host__ __device__ inline long long packed_off(long long r, long long c, long long n) {
  return r * n - r * (r + 1) / 2 + c;
}

// Tiles are TM x BN (TM = 128, or 256 for CTA pairs).
__host__ __device__ inline int gemm_tiles_per_batch(int M, int N, int BN, int tri, int TM = kBM) {
  const int tm = (M + TM - 1) / TM, tn = (N + BN - 1) / BN;
  if (!tri) return tm * tn;
  int total = 0;
  for (int i = 0; i < tm; ++i) {
    const int first = (i * TM) / BN;
    if (first < tn) total += tn - first;
  }
  return total;
}

// kPair: two CTAs of a cluster work on one 256 x BN tile (cta_group::2); each holds 128 rows of A and BN/2
// rows of B per stage: 32 KB for a 256 x 256 tile, where a single CTA's 128 x 256 takes 48.
// BN = 512 (pairs only) is the wide tile: two 256-column MMAs per k-step share the A rows, which cuts the operand
// bytes fetched per flop by a quarter (48 KB per CTA and k-block for twice the work of 32 KB).  Its accumulator
// fills all 512 columns of tensor memory, so there is no second buffer: the epilogue of a tile overlaps the next
// tile's MMAs only half by half.  It pays where the accumulation is long (K in the thousands of k-blocks, as in
// the statistic X^T X, or three plane passes of a wide matrix).
constexpr int kEpiBlockBytes = 32 * 32 * 4;  // one staged 32 x 32 block of the epilogue

template <int BN, bool kPair = false, bool kInter = false>
struct GemmSmem {
  static constexpr bool kWide = kPair && BN == 512;
  static constexpr int kABytes = kBM * kBK * 2;
  static constexpr int kBRows = kPair ? BN / 2 : BN;   // rows of B this CTA loads per stage
  static constexpr int kBBytes = kBRows * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  // A stage's way round -- freed, copied into, multiplied, freed -- takes about 2700 cycles whatever its size, so it is the
  // number of stages that keeps the main loop fed: BF16 8192^3 on 256 x 256 pair tiles 627 cycles per k-block with four, 541
  // with five, 535 with six (its MMAs take 512).  The epilogue wants two blocks a warp in flight where it brings in C and
  // writes two results: 32 x 768^3 Newton-Schulz update 52 us with two or three, 58 with one.  Hence five stages of 32 KB and
  // six of 24 KB with two blocks, four of 48 KB with one.
  // (Interleaved plane products hold two stages until the three products of a k-block have been issued: six.)
  static constexpr int kStages = kInter ? 6 : (kStageBytes > 32 * 1024 ? 4 : (kStageBytes < 32 * 1024 ? 6 : 5));
  static constexpr int kTileBytes = kStages * kStageBytes;
  // 4 KB blocks per epilogue warp
  static constexpr int kEpiBufs = kStageBytes > 32 * 1024 || (kInter && kStageBytes == 32 * 1024) ? 1 : 2;
  static constexpr int kEpiBytes = 8 * kEpiBufs * kEpiBlockBytes;
  static constexpr int kBarBytes = 320;
  static constexpr int kTotal = kTileBytes + kEpiBytes + kBarBytes + 1024;  // 1024: alignment slack
  static constexpr int kTmemCols = kWide ? 512 : 2 * BN;
};

__device__ __forceinline__ void tile_coord(const GemmParams& p, int BN, int TM, int t, int tiles_per_batch, int tiles_n,
                                           int& b, int& tm, int& tn) {
  b = t / tiles_per_batch;
  int r = t - b * tiles_per_batch;
  if (!p.tri) {
    // Column groups of `raster` tiles, rows swept inside a group: the tiles in flight at any moment share
    // a few B panels (resident in L2 for the whole sweep) and stream A panels once per group.
    const int tiles_m = tiles_per_batch / tiles_n;
    const int g = p.raster > 0 ? p.raster : tiles_n;
    const int per_group = g * tiles_m;
    const int group = r / per_group;
    const int in_group = r - group * per_group;
    const int width = min(g, tiles_n - group * g);
    tm = in_group / width;
    tn = group * g + (in_group - tm * width);
    return;
  }
  tm = 0;
  for (;;) {
    const int first = (tm * TM) / BN;
    const int cnt = tiles_n - first;
    if (r < cnt) {
      tn = first + r;
      return;
    }
    r -= cnt;
    ++tm;
  }
}

__device__ __forceinline__ void report(int* status, int code) {
  if (status) atomicCAS(status, 0, code);
}

// Per-tile epilogue state (uniform over the warp).
struct EpilogueTile {
  const float* Cb;
  float* Db;
  uint16_t* Hb;  // 16-bit copy of the result (FP16 or BF16 bits)
  __half* S0b;
  __half* S1b;
  float alpha, beta;
  bool use_c, stats;
};

__device__ __forceinline__ uint16_t to_bits16(float v, int bf16) {
  const __half h = __float2half_rn(v);
  const __nv_bfloat16 g = __float2bfloat16_rn(v);
  return bf16 ? *reinterpret_cast<const uint16_t*>(&g) : *reinterpret_cast<const uint16_t*>(&h);
}

__device__ __forceinline__ uint32_t pack2_16(float a, float b, int bf16) {
  const __half2 h = __floats2half2_rn(a, b);
  const __nv_bfloat162 g = __floats2bfloat162_rn(a, b);
  return bf16 ? *reinterpret_cast<const uint32_t*>(&g) : *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ void store_split1(__half* hi, long long plane, float x) {
  const __half h = __float2half_rn(x);
  hi[0] = h;
  hi[plane] = __float2half_rn(x - __half2float(h));
}

// The epilogue works in 32 x 32 blocks.  A thread has one row of the block in registers (that is how tensor memory is
// read), writes it to a shared-memory block in the layout of a swizzled TMA box -- row by row, or exchanged for the mirrored
// half of a symmetric result -- and one lane stores the box.  No address arithmetic per element, no masks (TMA clips at
// the matrix edge), and the stores run behind the next block.  With two epilogue warps per scheduler it is the number of
// instructions a block takes that bounds short products: staging rows in shared memory, reading them back and storing
// them with 16-byte accesses took about 500 per block and output, 2100 cycles for one FP32 output.
//
// Offsets inside a staged block (base 1024-byte aligned), conflict-free for a lane = row writer:
//   FP32 box, 128-byte rows: 16-byte chunk index ^= row & 7;    16-bit box, 64-byte rows: chunk index ^= (row >> 1) & 3.
struct EpilogueSums {
  float ssq = 0.f, mabs = 0.f, maff = 0.f, mres = 0.f;
};

__device__ __forceinline__ void stage_rows_f32(uint32_t buf, int lane, const float (&v)[32]) {
  const uint32_t at = buf + lane * 128 + ((lane & 7) << 4);
#pragma unroll
  for (int j = 0; j < 8; ++j)
    ptx::sts128(at ^ (j << 4), __float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]), __float_as_uint(v[4 * j + 2]),
                __float_as_uint(v[4 * j + 3]));
}
__device__ __forceinline__ void stage_cols_f32(uint32_t buf, int lane, const float (&v)[32]) {
  const uint32_t at = buf + ((lane >> 2) << 4) + (lane & 3) * 4;
#pragma unroll
  for (int j = 0; j < 32; ++j) ptx::sts32((at ^ ((j & 7) << 4)) + j * 128, __float_as_uint(v[j]));
}
__device__ __forceinline__ void load_row_f32(uint32_t buf, int lane, float4 (&r)[8]) {
  const uint32_t at = buf + lane * 128 + ((lane & 7) << 4);
#pragma unroll
  for (int j = 0; j < 8; ++j) r[j] = ptx::lds128(at ^ (j << 4));
}
// w[k]: the 16-bit elements 2k (low half) and 2k + 1 of this lane's row
__device__ __forceinline__ void stage_rows_16(uint32_t buf, int lane, const uint32_t (&w)[16]) {
  const uint32_t at = buf + lane * 64 + (((lane >> 1) & 3) << 4);
#pragma unroll
  for (int c = 0; c < 4; ++c) ptx::sts128(at ^ (c << 4), w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
}
__device__ __forceinline__ void stage_cols_16(uint32_t buf, int lane, const uint32_t (&w)[16]) {
  const uint32_t at = buf + ((lane >> 3) << 4) + (lane & 7) * 2;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    ptx::sts16((at ^ ((k & 3) << 4)) + k * 128, w[k]);
    ptx::sts16_hi((at ^ ((k & 3) << 4)) + k * 128 + 64, w[k]);
  }
}

// A warp's ring of staged blocks: `bufs` (one or two) of them.  Every acquired block ends in exactly one bulk group,
// committed in the order of acquisition, so "all but the bufs - 1 newest groups have been read" frees the block acquired bufs
// acquisitions ago.
struct EpilogueRing {
  uint32_t base;
  int bufs;
  int next = 0;
  __device__ __forceinline__ uint32_t acquire() {
    if (ptx::elect_one()) {
      if (bufs == 2) ptx::bulk_wait_read<1>();
      else ptx::bulk_wait_read<0>();
    }
    __syncwarp();
    const uint32_t buf = base + next * kEpiBlockBytes;
    next = next + 1 == bufs ? 0 : next + 1;
    return buf;
  }
};

// One block of the result: v holds alpha * accumulator of this lane's row on entry.  `held`: a block of the ring that is
// already this block's own (C arrived in it), 0 if none.  `whole`: a diagonal block of a mirrored symmetric result; it is
// made symmetric from its upper half and written once.
__device__ __forceinline__ void epilogue_block(const GemmParams& p, const EpilogueTile& e, EpilogueRing& ring, float (&v)[32],
                                               uint32_t held, int b, int row_first, int c0, int lane, bool whole,
                                               EpilogueSums& t) {
  auto take = [&]() {
    const uint32_t buf = held ? held : ring.acquire();
    held = 0;
    return buf;
  };
  auto send = [&](auto&& stores) {   // what the lanes staged becomes visible to the copy engine, then one lane stores it
    ptx::fence_proxy_async_smem();
    __syncwarp();
    if (ptx::elect_one()) {
      stores();
      ptx::bulk_commit();
    }
  };
  if (whole) {
    if (!held) held = ring.acquire();
    stage_cols_f32(held, lane, v);
    __syncwarp();
    float4 r[8];
    load_row_f32(held, lane, r);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (4 * j < lane) v[4 * j] = r[j].x;
      if (4 * j + 1 < lane) v[4 * j + 1] = r[j].y;
      if (4 * j + 2 < lane) v[4 * j + 2] = r[j].z;
      if (4 * j + 3 < lane) v[4 * j + 3] = r[j].w;
    }
    __syncwarp();
  }
  const bool image = p.tri && p.mirror && !whole;   // the block below the diagonal is this lane's row as a column
  if (e.stats) {   // (outside the matrix the results are zero: operands and C are read as zero there)
    float s = 0.f, m = 0.f;
    const bool diag = c0 == row_first && row_first + lane < p.M && row_first + lane < p.N;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      s = fmaf(v[j], v[j], s);
      if (diag && j == lane) {   // the diagonal element's distance from the identity and its affine image are its own
        t.mabs = fmaxf(t.mabs, fabsf(v[j]));
        t.maff = fmaxf(t.maff, fabsf(fmaf(p.aff_b, v[j], p.aff_a)));
        t.mres = fmaxf(t.mres, fabsf(1.f - v[j]));
      } else {
        m = fmaxf(m, fabsf(v[j]));
      }
    }
    t.ssq += (p.tri && !whole) ? 2.f * s : s;    // a block above the diagonal counts for its mirror image as well
    t.mabs = fmaxf(t.mabs, m);
    t.maff = fmaxf(t.maff, fabsf(p.aff_b) * m);  // off the diagonal the affine map is a plain scaling
    // and the distance from the identity is |d|; fmaxf drops NaN, the sum of squares does not
    t.mres = fmaxf(t.mres, isfinite(s) ? m : INFINITY);
  }
  if (p.D) {
    const uint32_t buf = take();
    stage_rows_f32(buf, lane, v);
    send([&]() { ptx::tma_store_3d(&p.d_map, buf, c0, row_first, b); });
    if (image && !p.upper_d) {
      const uint32_t tb = take();
      stage_cols_f32(tb, lane, v);
      send([&]() { ptx::tma_store_3d(&p.d_map, tb, row_first, c0, b); });
    }
  }
  if (p.D16) {
    uint32_t w[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) w[k] = pack2_16(v[2 * k], v[2 * k + 1], p.d16_fmt);
    const uint32_t buf = take();
    stage_rows_16(buf, lane, w);
    if (image) stage_cols_16(buf + kEpiBlockBytes / 2, lane, w);
    send([&]() {
      ptx::tma_store_3d(&p.h_map, buf, c0, row_first, b);
      if (image) ptx::tma_store_3d(&p.h_map, buf + kEpiBlockBytes / 2, row_first, c0, b);
    });
  }
  // FP16 hi/lo planes of s * v (+ d on the diagonal): hi = rn(x), lo = rn(x - hi)
  auto planes = [&](const CUtensorMap* map, float s, float d) {
    uint32_t hi[16], lo[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      float x = s * v[2 * k], y = s * v[2 * k + 1];
      if (d != 0.f) {
        if (2 * k == lane) x = fmaf(s, v[2 * k], d);
        if (2 * k + 1 == lane) y = fmaf(s, v[2 * k + 1], d);
      }
      const __half2 h = __floats2half2_rn(x, y);
      const float2 f = __half22float2(h);
      const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
      hi[k] = *reinterpret_cast<const uint32_t*>(&h);
      lo[k] = *reinterpret_cast<const uint32_t*>(&l);
    }
    const uint32_t buf = take();
    stage_rows_16(buf, lane, hi);
    stage_rows_16(buf + kEpiBlockBytes / 2, lane, lo);
    send([&]() {
      ptx::tma_store_3d(map, buf, c0, row_first, b);
      ptx::tma_store_3d(map, buf + kEpiBlockBytes / 2, c0, row_first, b + p.s_lo_z);
    });
    if (image && !(p.half_out && (c0 >> kHalfShift) != (row_first >> kHalfShift))) {
      const uint32_t tb = take();
      stage_cols_16(tb, lane, hi);
      stage_cols_16(tb + kEpiBlockBytes / 2, lane, lo);
      send([&]() {
        ptx::tma_store_3d(map, tb, row_first, c0, b);
        ptx::tma_store_3d(map, tb + kEpiBlockBytes / 2, row_first, c0, b + p.s_lo_z);
      });
    }
  };
  if (p.S0) planes(&p.s0_map, p.s0_scale, c0 == row_first ? p.s0_scale * p.s0_aff_a : 0.f);
  if (p.S1) planes(&p.s1_map, p.s1_scale * p.s1_aff_b, c0 == row_first ? p.s1_scale * p.s1_aff_a : 0.f);
}

// Element of a block staged by stage_rows_f32.
__device__ __forceinline__ int stage_at(int row, int col) { return row * 32 + (((col >> 2) ^ (row & 7)) << 2) + (col & 3); }

// Any other block (packed or unaligned output; a diagonal block of a symmetric result that is not mirrored), from its rows
// staged in FP32: one element per lane with full masking, lane = column, so rows -- also rows of a packed triangle -- are
// still written as contiguous runs; the mirrored half with lane = source row.  C is fetched eight rows at a time.
// v = acc here, not yet scaled.

__device__ __forceinline__ void epilogue_block_scalar(const GemmParams& p, const EpilogueTile& e, float* stage, int row_first,
                                                      int c0, int lane, EpilogueSums& t) {
  const int col = c0 + lane;
  const bool col_ok = col < p.N;
  const bool mirror = p.tri && p.mirror;
  const int rows = min(32, p.M - row_first);
#pragma unroll 1
  for (int i0 = 0; i0 < rows; i0 += 8) {
    float cv[8];
    if (e.use_c) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int row = row_first + i0 + u;
        cv[u] = 0.f;
        if (row < p.M && col_ok && !(p.tri && col < row))
          cv[u] = e.Cb[p.packed ? packed_off(row, col, p.N) : (long long)row * p.ldc + col];
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = i0 + u, row = row_first + i;
      float* const at = stage + stage_at(i, lane);
      float v = 0.f;
      if (row < p.M && col_ok && !(p.tri && col < row)) {
        v = e.alpha * *at;
        if (e.use_c) v = fmaf(e.beta, cv[u], v);
        if (e.Db) e.Db[p.packed ? packed_off(row, col, p.N) : (long long)row * p.ldd + col] = v;
        if (e.Hb) e.Hb[(long long)row * p.ld16 + col] = to_bits16(v, p.d16_fmt);
        const float dg = (col == row) ? 1.f : 0.f;
        if (e.S0b) store_split1(e.S0b + (long long)row * p.s_ld + col, p.s_plane, p.s0_scale * (v + p.s0_aff_a * dg));
        if (e.S1b) store_split1(e.S1b + (long long)row * p.s_ld + col, p.s_plane, p.s1_scale * fmaf(p.s1_aff_b, v, p.s1_aff_a * dg));
        t.mres = isfinite(v) ? fmaxf(t.mres, fabsf(dg - v)) : INFINITY;  // a non-finite result must not pass as converged
        const float w = (p.tri && col > row) ? 2.f : 1.f;
        t.ssq = fmaf(w * v, v, t.ssq);
        t.mabs = fmaxf(t.mabs, fabsf(v));
        t.maff = fmaxf(t.maff, fabsf(fmaf(p.aff_b, v, col == row ? p.aff_a : 0.f)));
      }
      if (mirror) *at = v;  // final value; zero where masked
    }
  }
  if (mirror) {
    __syncwarp();
    const int row = row_first + lane;  // this lane's source row becomes the target column
    const int cols = min(32, p.N - c0);
    if (row < p.M) {
#pragma unroll 1
      for (int j = 0; j < cols; ++j) {
        const int c = c0 + j;
        if (c > row) {
          const float v = stage[stage_at(lane, j)];
          if (e.Db && !p.upper_d) e.Db[(long long)c * p.ldd + row] = v;
          if (e.Hb) e.Hb[(long long)c * p.ld16 + row] = to_bits16(v, p.d16_fmt);
          if (e.S0b) store_split1(e.S0b + (long long)c * p.s_ld + row, p.s_plane, p.s0_scale * v);
          if (e.S1b) store_split1(e.S1b + (long long)c * p.s_ld + row, p.s_plane, p.s1_scale * p.s1_aff_b * v);
        }
      }
    }
  }
  __syncwarp();
}

// kChained: the kernel sums several accumulation chains per tile in registers (p.promote > 0).
// kPair: launched as clusters of two CTAs that share each 256 x BN tile (BN = 128, 256 or 512): both load their halves of
// the operands, the leader CTA's MMA thread issues cta_group::2 MMAs, each CTA's epilogue warps write the
// 128 rows that sit in its own tensor memory.  The pair halves the operand traffic per flop of B.
//
// kInter: the split-precision product Ah Bh + Ah Bl + Al Bh with its three plane products interleaved k-block by k-block: a
// stage with the lo planes of a k-block, a stage with the hi planes, three groups of MMAs over the two, so that each plane
// comes from L2 once instead of one and a half times: three plane products need 64 KB instead of 96 KB beside their 1536
// cycles of MMAs.  Measured plane by plane / interleaved, under the power limit: 12 x 3072^3 symmetric 864 / 744 us, in chains of two
// 876 / 825; 6 x 5632^3 symmetric 2450 / 2170 and 2555 / 2517.
// The cross products of a k-block go into the accumulator before its hi product.  In a chained product they now share the
// chains, which the host therefore makes shorter than c k-blocks, except c = 2 (see the MMA loop), so that no error grows:
// against FP64 at 2048^3, chains of 2 plane by plane and interleaved 4.1e-7; of 8 plane by plane 2.4e-6, of 5 interleaved
// 1.9e-6 (random signs 3.4e-7, 1.5e-6 and 1.4e-6); one chain 1.8e-5 and 1.5e-5.  (GemmParams::segs
// is 1 here: the three products are one.)
template <int BN, bool kChained, bool kPair = false, bool kInter = false, bool kHalf = false>
__global__ void __launch_bounds__(kGemmThreads, 1) gemm_tcgen05_kernel(const __grid_constant__ GemmParams p) {
  using S = GemmSmem<BN, kPair, kInter>;
  static_assert(!kInter || (kPair && BN <= 256), "interleaved plane products: 256 x 256 or 256 x 128 on pairs");
  static_assert((BN == 64 && !kPair) || BN == 128 || BN == 256 || (BN == 512 && kPair && !kChained),
                "tile widths: 64 (single CTAs), 128, 256, or 512 (pairs)");
  constexpr bool kWide = S::kWide;
  constexpr int BNI = kWide ? 256 : BN;                // columns of one MMA instruction
  constexpr int TM = kPair ? 2 * kBM : kBM;            // rows of one scheduled tile
  const uint32_t cta_rank = kPair ? ptx::cluster_ctarank() : 0u;
  const bool leader = cta_rank == 0;
  const int unit = kPair ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;     // which persistent worker this CTA (pair) is
  const int units = kPair ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* const smem = smem_raw + (base - raw);
  // barrier block after the tiles and the epilogue's blocks
  const uint32_t bars = base + S::kTileBytes + S::kEpiBytes;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (S::kStages + s); };
  auto tfull_bar = [&](int s) { return bars + 8u * (2 * S::kStages + s); };
  auto tempty_bar = [&](int s) { return bars + 8u * (2 * S::kStages + 2 + s); };
  auto c_bar = [&](int w) { return bars + 8u * (2 * S::kStages + 4 + w); };   // C blocks of epilogue warp w
  constexpr int kAfterBars = S::kTileBytes + S::kEpiBytes + 8 * (2 * S::kStages + 12);
  static_assert(8 * (2 * S::kStages + 12) + 16 <= S::kBarBytes, "barrier block");
  volatile uint32_t* const tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + kAfterBars);
  volatile int* const abort_flag = reinterpret_cast<volatile int*>(smem + kAfterBars + 8);
  // A role that gives up stops its own CTA and, in a pair, the peer as well, so that neither waits for two more seconds.  The flag
  // is looked at in a wait that is not satisfied at once, and every role soon comes to one: the producers fill and the MMAs use at
  // most the ring's stages without the other, the MMAs two accumulators without the epilogue, and the epilogue those without the
  // MMAs.  The peer's shared memory is valid until the closing cluster barrier, which every thread of both CTAs reaches.
  auto raise_abort = [&]() {
    *abort_flag = 1;
    if constexpr (kPair)
      ptx::st_cluster_u32(ptx::mapa(ptx::smem_u32(const_cast<int*>(abort_flag)), cta_rank ^ 1u), 1u);
  };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_n = (p.N + BN - 1) / BN;
  const int tiles_per_batch = gemm_tiles_per_batch(p.M, p.N, BN, p.tri, TM);
  const int total_tiles = tiles_per_batch * p.batch;
  const int kb_per_seg = (p.K + kBK - 1) / kBK;
  const int num_kb = kb_per_seg * p.segs;
  // Accumulation chains: with promote > 0 the MMA warp starts a fresh TMEM accumulator every `promote`
  // k-blocks of the FIRST segment and the epilogue warps sum the chains in registers.  Later segments
  // (the hi*lo cross terms of a split product, 2^-11 of the first) form one chain each: truncation
  // inside them is far below the result's last bit.  promote_all chains every segment the same way.
  const int chunks_seg0 = p.promote > 0 ? (kb_per_seg + p.promote - 1) / p.promote : 1;
  const int chunks_rest = (p.promote > 0 && p.promote_all) ? chunks_seg0 : 1;
  const int chunks_per_tile = p.promote > 0 ? chunks_seg0 + (p.segs - 1) * chunks_rest : 1;
  // Order of work inside a tile.  When only the first segment is chained, the later segments come FIRST, one
  // long chain each: while the epilogue warps are still writing the previous tile they cannot sum chains, and
  // two long chains give them that time; the short chains of the first segment follow.
  const bool rest_first = p.promote > 0 && !p.promote_all && p.segs > 1;
  auto chunk_range = [&](int ch, int& kb_begin, int& kb_end) {  // k-block indices in processing order
    if (rest_first) {
      const int rest = p.segs - 1;
      if (ch < rest) {
        kb_begin = ch * kb_per_seg;
        kb_end = kb_begin + kb_per_seg;
      } else {
        kb_begin = rest * kb_per_seg + (ch - rest) * p.promote;
        kb_end = min(kb_begin + p.promote, num_kb);
      }
      return;
    }
    int seg = 0, c = ch;
    if (ch >= chunks_seg0) {
      seg = 1 + (ch - chunks_seg0) / chunks_rest;
      c = (ch - chunks_seg0) - (seg - 1) * chunks_rest;
    }
    const bool chained = (seg == 0) || p.promote_all;
    kb_begin = seg * kb_per_seg + (chained ? c * p.promote : 0);
    kb_end = chained ? min(kb_begin + p.promote, (seg + 1) * kb_per_seg) : (seg + 1) * kb_per_seg;
  };
  // Work unit u: split u % splits of tile u / splits, i.e. accumulation chains [ch_lo, ch_hi) -- where there is one chain, a
  // part of it -- and k-blocks [kb_lo, kb_hi) in processing order.
  const int total_units = total_tiles * p.splits;
  struct Unit {
    int tile, split, ch_lo, ch_hi, kb_lo, kb_hi;
  };
  auto unit_of = [&](int u) {
    Unit w;
    w.tile = u / p.splits;
    w.split = u - w.tile * p.splits;
    if (p.promote > 0) {
      w.ch_lo = chunks_per_tile * w.split / p.splits;
      w.ch_hi = chunks_per_tile * (w.split + 1) / p.splits;
      int unused;
      chunk_range(w.ch_lo, w.kb_lo, unused);
      chunk_range(w.ch_hi - 1, unused, w.kb_hi);
    } else {
      w.ch_lo = 0;
      w.ch_hi = 1;
      w.kb_lo = (int)((long long)num_kb * w.split / p.splits);
      w.kb_hi = (int)((long long)num_kb * (w.split + 1) / p.splits);
    }
    return w;
  };
  // (every role asks alike: what is left out is left out by all of them)
  auto left_out = [&](int b) { return p.skip != nullptr && p.skip[b] != 0; };
  if (threadIdx.x == 0) {
    for (int s = 0; s < S::kStages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(tfull_bar(s), 1);
      // one arrival per epilogue warp (of both CTAs of a pair); per half of a wide tile: the four warps that read it
      ptx::mbar_init(tempty_bar(s), kWide ? 8 : (kPair ? 16 : 8));
    }
    for (int w = 0; w < 8; ++w) ptx::mbar_init(c_bar(w), 1);
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    if constexpr (kPair) {
      ptx::tmem_alloc_pair(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), S::kTmemCols);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), S::kTmemCols);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  if constexpr (kPair) ptx::cluster_sync();  // the peer's barriers exist before anything signals them
  else __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  ptx::pdl_begin();   // everything above runs beside the previous kernel

  if (warp < 4) {
  ptx::reg_dec<48>();
  if (warp == 0 || warp == 2) {
    // ------------------------------------------------------------ TMA producers: warp 0 brings A, warp 2 brings B
    // Issuing a copy holds its thread up until the copy engine takes it, hence two threads.
    const bool for_a = warp == 0;
    if (ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      long long prof_wait = 0;
      for (int u = unit; u < total_units && ok; u += units) {
        const Unit w = unit_of(u);
        int b, tm, tn;
        tile_coord(p, BN, TM, w.tile, tiles_per_batch, tiles_n, b, tm, tn);
        if (left_out(b)) continue;
        const CUtensorMap* map = for_a ? &p.a_map : &p.b_map;
        if (for_a ? p.a_maps != nullptr : p.b_maps != nullptr) {
          map = (for_a ? p.a_maps : p.b_maps) + b;
          ptx::fence_tensormap_acquire(map);
        }
        // a pair splits the tile's rows (A) and its columns (B) between its two CTAs
        // (of a wide tile each CTA holds 128 columns of either 256-column half: r0 is its share of the first half)
        const int r0 = for_a ? tm * TM + (int)cta_rank * kBM : tn * BN + (int)cta_rank * (kWide ? BNI / 2 : S::kBRows);
        // fill this operand's part of the next stage with k-block k0 of plane z
        auto fill = [&](int k0, int z) {
          const long long w0 = p.prof ? clock64() : 0;
          const bool got = ptx::mbar_wait_unless(empty_bar(stage), phase ^ 1u, kWaitCycles, abort_flag);
          if (p.prof) prof_wait += clock64() - w0;
          if (!got) {
            report(p.status, kTimeoutProducer);
            raise_abort();
            ok = false;
            return;
          }
          const uint32_t dst = base + stage * S::kStageBytes + (for_a ? 0 : S::kABytes);
          uint32_t bar = full_bar(stage);
          if constexpr (kPair) {
            // Both CTAs' copies report to the leader's barrier, which expects the bytes of the whole pair.
            if (for_a && leader) ptx::mbar_expect_tx(bar, 2 * S::kStageBytes);
            bar = ptx::mapa(bar, 0);
          } else if (for_a) {
            ptx::mbar_expect_tx(bar, S::kStageBytes);
          }
          auto copy = [&](uint32_t to, const CUtensorMap* from, int x, int y) {
            if constexpr (kPair) ptx::tma_load_3d_pair(to, from, bar, x, y, z);
            else ptx::tma_load_3d(to, from, bar, x, y, z);
          };
          // `slabs` times 64 rows from r on: stored MN-major, the mirror image of a half-stored operand's, or K-major
          auto rows = [&](uint32_t to, int r, auto slabs) {
            const bool image = kHalf && (k0 >> kHalfShift) < (r >> kHalfShift);
            if (image || (for_a ? p.a_mn : p.b_mn)) {
              const CUtensorMap* const from = image ? (for_a ? &p.a_turned : &p.b_turned) : map;
#pragma unroll
              for (int s = 0; s < decltype(slabs)::value; ++s) copy(to + s * 8192, from, r + s * 64, k0);
            } else {
              copy(to, map, k0, r);
            }
          };
          constexpr std::integral_constant<int, kBM / 64> kOfA;
          constexpr std::integral_constant<int, (kWide ? 128 : kPair ? S::kBRows : BN) / 64> kOfB;
          if (for_a) {
            rows(dst, r0, kOfA);
          } else {
            rows(dst, r0, kOfB);
            if constexpr (kWide) rows(dst + 16384, r0 + BNI, kOfB);
          }
          if (++stage == S::kStages) {
            stage = 0;
            phase ^= 1u;
          }
        };
        if constexpr (kInter) {
          const int z = b * (for_a ? p.a_z_stride : p.b_z_stride);
          const int z_lo = z + (for_a ? p.a_seg_z[2] : p.b_seg_z[1]), z_hi = z + (for_a ? p.a_seg_z[0] : p.b_seg_z[0]);
          for (int kb = w.kb_lo; kb < w.kb_hi && ok; ++kb) {
            fill(kb * kBK, z_lo);
            if (ok) fill(kb * kBK, z_hi);
          }
        } else {
          for (int kb = w.kb_lo; kb < w.kb_hi && ok;) {
            const int si = kb / kb_per_seg, seg_end = min(w.kb_hi, (si + 1) * kb_per_seg);
            const int seg = rest_first ? (si + 1 == p.segs ? 0 : si + 1) : si;
            const int z = for_a ? b * p.a_z_stride + p.a_seg_z[seg] : b * p.b_z_stride + p.b_seg_z[seg];
            for (; kb < seg_end && ok; ++kb) fill((kb - si * kb_per_seg) * kBK, z);
          }
        }
      }
      if (p.prof && leader && for_a) atomicAdd(p.prof + 3, (unsigned long long)prof_wait);
      if (!ok || *abort_flag) {
        // Copies already issued must land before this CTA gives its shared memory back (the closing barrier waits
        // for threads, not for bulk copies).  Stage s was last filled in this round if s < stage, else in the round
        // before (a stage never filled is "complete" at once: its barrier has not left phase 0).  In a pair every
        // copy of both CTAs reports to the leader's barriers, so the leader waits for them; a barrier whose other
        // half was never issued cannot complete, hence the bound.  Copies this thread cannot account for (the peer or the
        // other producer ran a few stages ahead of it) get a fixed settling time: a copy lands within microseconds.
        if (!kPair || leader) {
          for (int s = 0; s < S::kStages; ++s)
            ptx::mbar_wait(full_bar(s), (s < stage) ? phase : (phase ^ 1u), kDrainCycles);
        }
        const long long t0 = clock64();
        while (clock64() - t0 < kSettleCycles) {
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (of a pair: the leader CTA only)
    // This thread's own instructions, not memory, were what bounded the main loop (half the copies: the same time; a quarter
    // of the MMAs: 666 cycles a k-block instead of 775): it is elected, and the flag of a role that gave up is looked at only
    // while waiting.  8192^3 775 -> 627 cycles a k-block, 541 with five stages: 838 -> 726 us (power-capped; zeros, which draw
    // little power, 770 -> 572 us).
    if (leader && ptx::elect_one()) {
      const uint32_t idesc_k = (1u << 4) | ((uint32_t)p.fmt << 7) | ((uint32_t)p.fmt << 10) | ((uint32_t)(BNI >> 3) << 17) |
                               ((uint32_t)(TM >> 4) << 24);
      // K-major: 8-row groups 1024 B apart, k advances 32 B inside the swizzled row.
      // MN-major: 64-element slabs 8192 B apart (LBO), 8-k-row groups 1024 B apart (SBO), k advances 16 rows = 2048 B.
      // The descriptor's upper word (8-row groups 1024 B apart, version, 128-byte swizzle) never changes; the lower
      // word is the address in 16-byte units plus the leading-dimension offset, so a k-step is an addition.
      const uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
      // Which operands of a k-block are MN-major (of a wide tile, the halves of B): those that are stored so, and of half-stored ones
      // the mirror images.  What follows from it is kept, not worked out for every k-block: that cost Newton-Schulz 1.4 %.
      uint32_t a_lo_const, a_step16, b_lo_const[kWide ? 2 : 1], b_step16[kWide ? 2 : 1], idesc[kWide ? 2 : 1];
      auto orient = [&](bool a_mn, bool b_mn, int j) {
        a_lo_const = (a_mn ? 512u : 1u) << 16;
        a_step16 = a_mn ? 128u : 2u;
        b_lo_const[j] = (b_mn ? 512u : 1u) << 16;
        b_step16[j] = b_mn ? 128u : 2u;
        idesc[j] = idesc_k | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u);
      };
#pragma unroll
      for (int j = 0; j < (kWide ? 2 : 1); ++j) orient(p.a_mn != 0, p.b_mn != 0, j);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t gchunk = 0;  // accumulator hand-offs so far; buffer = gchunk & 1
      bool ok = true;
      long long prof_acc = 0, prof_ops = 0;
      const long long prof_t0 = p.prof ? clock64() : 0;
      for (int u = unit; u < total_units && ok; u += units) {
        const Unit w = unit_of(u);
        if (left_out(w.tile / tiles_per_batch)) continue;
        int a_block = 0, b_block = 0;   // blocks of half-stored operands that the tile's rows of A and of B lie in
        if constexpr (kHalf) {
          int b, tm, tn;
          tile_coord(p, BN, TM, w.tile, tiles_per_batch, tiles_n, b, tm, tn);
          a_block = (tm * TM) >> kHalfShift;
          b_block = (tn * BN) >> kHalfShift;
        }
        auto turn = [&](int kb) {   // (k-blocks in processing order: every segment goes through all of them)
          if (!kHalf) return;
          if (!kInter) {
            if (kb >= kb_per_seg) kb -= kb_per_seg;
            if (kb >= kb_per_seg) kb -= kb_per_seg;
          }
          const int block = (kb * kBK) >> kHalfShift;
#pragma unroll
          for (int j = 0; j < (kWide ? 2 : 1); ++j) orient(block < a_block, block < b_block + j, j);
        };
        for (int ch = w.ch_lo; ch < w.ch_hi && ok; ++ch, ++gchunk) {
          int kb_begin = w.kb_lo, kb_end = w.kb_hi;
          if (p.promote > 0) chunk_range(ch, kb_begin, kb_end);
          // The wide tile has one accumulator of two halves, each with its own "drained" barrier (tempty 0 / 1): the
          // MMAs of the first k-block's first half start as soon as that half has been read out.
          const int buf = kWide ? 0 : (int)(gchunk & 1u);
          const uint32_t acc_parity = (kWide ? (gchunk & 1u) : ((gchunk >> 1) & 1u)) ^ 1u;
          auto wait_drained = [&](int bar) {
            const long long w0 = p.prof ? clock64() : 0;
            const bool got_acc = ptx::mbar_wait_unless(tempty_bar(bar), acc_parity, kWaitCycles, abort_flag);
            if (p.prof) prof_acc += clock64() - w0;
            if (!got_acc) {
              report(p.status, kTimeoutMma);
              raise_abort();
              ok = false;
              return false;
            }
            ptx::tc_fence_after();
            return true;
          };
          if (!wait_drained(buf)) break;
          const uint32_t d_tmem = tmem_base + (uint32_t)(kWide ? 0 : buf * BN);
          // wait for the operands of a stage; its shared-memory address
          auto operands = [&](int st, uint32_t ph) {
            const long long w1 = p.prof ? clock64() : 0;
            const bool got_ops = ptx::mbar_wait_unless(full_bar(st), ph, kWaitCycles, abort_flag);
            if (p.prof) prof_ops += clock64() - w1;
            if (!got_ops) {
              report(p.status, kTimeoutMma);
              raise_abort();
              ok = false;
            }
            ptx::tc_fence_after();
            return base + st * S::kStageBytes;
          };
          // the MMAs of one k-block (columns from 256 * j on), A from stage address sa, B from sb
          auto multiply = [&](uint32_t sa, uint32_t sb, int j, uint32_t fresh) {
            const uint32_t a_lo = ((sa & 0x3FFFFu) >> 4) | a_lo_const;
            const uint32_t b_lo = (((sb + S::kABytes) & 0x3FFFFu) >> 4) | b_lo_const[j];
#pragma unroll
            for (int k = 0; k < kBK / kUmmaK; ++k) {
              const uint64_t da = ((uint64_t)desc_hi << 32) | (a_lo + k * a_step16);
              const uint64_t db = ((uint64_t)desc_hi << 32) | (b_lo + j * ((BNI / 2) * kBK * 2 / 16) + k * b_step16[j]);
              if constexpr (kPair) ptx::mma_f16_pair(d_tmem + j * BNI, da, db, idesc[j], k != 0 ? 1u : fresh);
              else ptx::mma_f16(d_tmem, da, db, idesc[j], k != 0 ? 1u : fresh);
            }
          };
          auto release_stage = [&](int st) {  // frees the stage (in both CTAs of a pair) once the MMAs so far have read it
            if constexpr (kPair) {
              ptx::mma_commit_pair(empty_bar(st));
              ptx::mma_commit_pair(ptx::mapa(empty_bar(st), 1));
            } else {
              ptx::mma_commit(empty_bar(st));
            }
          };
          auto advance = [&]() {
            if (++stage == S::kStages) {
              stage = 0;
              phase ^= 1u;
            }
          };
          // one stage's operands, and its index for release_stage
          auto next_operands = [&](int& st) {
            st = stage;
            const uint32_t at = operands(st, phase);
            if (ok) advance();
            return at;
          };
          if constexpr (kInter) {
            // In chains of two, the cross products of both k-blocks go into the accumulator before the hi products of either:
            // they are added while it is still 2^-11 of what it becomes.  (Otherwise one k-block after the other: holding
            // four stages until the hi products have been issued cost one-chain products 5 %.)
            const bool pairs = kChained && p.promote == 2;
            for (int kb = kb_begin; kb < kb_end; kb += pairs ? 2 : 1) {
              const bool two = pairs && kb + 1 < kb_end;
              int s_lo, s_hi, s_lo1, s_hi1 = 0;
              const uint32_t lo = next_operands(s_lo), hi = ok ? next_operands(s_hi) : 0u;
              if (!ok) break;
              turn(kb);   // (two k-blocks from an even one on lie in one block of 256)
              multiply(hi, lo, 0, kb != kb_begin ? 1u : 0u);   // Ah Bl
              multiply(lo, hi, 0, 1u);                         // Al Bh
              release_stage(s_lo);
              uint32_t hi1 = 0;
              if (two) {
                const uint32_t lo1 = next_operands(s_lo1);
                hi1 = ok ? next_operands(s_hi1) : 0u;
                if (!ok) break;
                multiply(hi1, lo1, 0, 1u);
                multiply(lo1, hi1, 0, 1u);
                release_stage(s_lo1);
              }
              multiply(hi, hi, 0, 1u);
              release_stage(s_hi);
              if (two) {
                multiply(hi1, hi1, 0, 1u);
                release_stage(s_hi1);
              }
            }
          } else {
            for (int kb = kb_begin; kb < kb_end; ++kb) {
              const uint32_t fresh = (kb != kb_begin) ? 1u : 0u;
              int st;
              const uint32_t at = next_operands(st);
              if (!ok) break;
              turn(kb);
              multiply(at, at, 0, fresh);
              if constexpr (kWide) {
                if (kb == kb_begin && !wait_drained(1)) break;
                multiply(at, at, 1, fresh);
              }
              release_stage(st);
            }
          }
          if (ok) {  // this chain's partial sum is complete
            if constexpr (kPair) {
              ptx::mma_commit_pair(tfull_bar(buf));
              ptx::mma_commit_pair(ptx::mapa(tfull_bar(buf), 1));
            } else {
              ptx::mma_commit(tfull_bar(buf));
            }
          }
        }
      }
      if (p.prof) {
        atomicAdd(p.prof + 0, (unsigned long long)(clock64() - prof_t0));
        atomicAdd(p.prof + 1, (unsigned long long)prof_acc);
        atomicAdd(p.prof + 2, (unsigned long long)prof_ops);
        atomicAdd(p.prof + 7, 1ull);
      }
    }
  }
  } else {
    ptx::reg_inc<224>();
    // ------------------------------------------------------------ epilogue (warps 4..11)
    // Warp w may read TMEM lanes [32*(w&3), +32); two warps share a lane group and split the columns.
    constexpr int NCH = BN / 64;  // 32-column chunks per warp
    const int lane_group = warp & 3;
    const int half = (warp - 4) >> 2;
    const int ew = warp - 4;
    // With C the last of the warp's blocks is C's own, where there are several: the next block's C is then on its way while
    // this block's results are staged (a 32 x 32 block of C, D and D16 took 4000 cycles with C fetched after them, 1500 of
    // them the wait for it).  With one block only, C arrives where D will be staged.
    const bool c_apart = S::kEpiBufs > 1 && p.C != nullptr;
    const uint32_t warp_bufs = base + S::kTileBytes + ew * S::kEpiBufs * kEpiBlockBytes;
    EpilogueRing ring{warp_bufs, c_apart ? S::kEpiBufs - 1 : S::kEpiBufs};
    uint32_t c_buf = 0, c_phase = 0;   // block C is arriving in (0: none), parity of its barrier
    constexpr bool chained = kChained;
    // Running sums of the accumulation chains (chained products only), added with round-to-nearest: the
    // tensor core itself adds into its accumulator by truncation.
    float racc[kChained ? NCH * 32 : 1];
    uint32_t gchunk = 0;
    bool alive = true;
    long long prof_wait = 0, prof_out = 0, prof_sum = 0;
    for (int u = unit; u < total_units && alive; u += units) {
      const Unit w = unit_of(u);
      int b, tm, tn;
      tile_coord(p, BN, TM, w.tile, tiles_per_batch, tiles_n, b, tm, tn);
      if (left_out(b)) continue;
      const int m0 = tm * TM + (int)cta_rank * kBM, n0 = tn * BN;  // this CTA's 128 rows of the tile
      const int row_first = m0 + lane_group * 32;
      const int col_first = n0 + half * (BN / 2);
      // 32-column blocks this warp never needs: outside the matrix, or wholly below the diagonal (warp-uniform)
      auto needed = [&](int c0) { return c0 < p.N && row_first < p.M && !(p.tri && c0 + 31 < row_first); };
      auto wait_chain = [&](int buf) {
        const long long w0 = p.prof ? clock64() : 0;
        // every lane observes the barrier itself, so each one is ordered after the MMAs' TMEM writes
        const uint32_t parity = kWide ? (gchunk & 1u) : ((gchunk >> 1) & 1u);
        const int waited = __all_sync(0xffffffffu, ptx::mbar_wait_unless(tfull_bar(buf), parity, kWaitCycles, abort_flag) ? 1 : 0);
        if (!waited) {
          if (lane == 0) {
            report(p.status, kTimeoutEpilogue);
            raise_abort();
          }
          return false;
        }
        ptx::tc_fence_after();
        if (p.prof) prof_wait += clock64() - w0;
        return true;
      };
      auto release = [&](int buf) {  // buffer drained: hand it back to the MMA warp
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (kPair) ptx::mbar_arrive_cluster(ptx::mapa(tempty_bar(buf), 0));  // the leader's MMA thread waits
          else ptx::mbar_arrive(tempty_bar(buf));
        }
      };
      auto tmem_of = [&](int buf) {
        return tmem_base + ((uint32_t)(lane_group * 32) << 16) + (uint32_t)((kWide ? 0 : buf * BN) + half * (BN / 2));
      };

      EpilogueTile e;
      e.alpha = p.alpha;
      e.beta = p.beta;
      if (p.alpha_a) e.alpha *= __ldg(p.alpha_a + b);
      if (p.alpha_b) e.alpha *= __ldg(p.alpha_b + (long long)b * p.alpha_b_step);
      if (p.beta_v) e.beta *= __ldg(p.beta_v + b);
      e.use_c = (p.C != nullptr) && (e.beta != 0.f);
      e.stats = p.sumsq || p.maxabs || p.maxaff || p.maxres;
      // the blocks this warp writes: a contiguous run of its NCH 32-column blocks (warp-uniform)
      int cc_first = 0, cc_end = NCH;
      while (cc_first < NCH && !needed(col_first + cc_first * 32)) ++cc_first;
      while (cc_end > cc_first && !needed(col_first + (cc_end - 1) * 32)) --cc_end;
      // Boxes move by TMA unless an address or stride rules it out; a symmetric result that is not mirrored keeps its lower
      // triangle untouched, which a box across the diagonal would not.
      auto boxed = [&](int c0) { return p.tma_ok && !(p.tri && !p.mirror && c0 <= row_first + 31); };
      // C of a block is fetched as soon as its place is free -- of the tile's first block, while the accumulator is still
      // being formed.
      auto fetch_c = [&](int cc) {
        if (!e.use_c || cc >= cc_end || !boxed(col_first + cc * 32)) return;
        c_buf = c_apart ? warp_bufs + (S::kEpiBufs - 1) * kEpiBlockBytes : ring.acquire();
        if (ptx::elect_one()) {
          ptx::mbar_expect_tx(c_bar(ew), kEpiBlockBytes);
          ptx::tma_load_3d(c_buf, &p.c_map, c_bar(ew), col_first + cc * 32, row_first, b);
        }
      };
      if (p.splits == 1) fetch_c(cc_first);

      if (chained) {
#pragma unroll
        for (int j = 0; j < NCH * 32; ++j) racc[j] = 0.f;
        for (int ch = w.ch_lo; ch < w.ch_hi; ++ch, ++gchunk) {
          const int buf = gchunk & 1u;
          if (!wait_chain(buf)) {
            alive = false;
            break;
          }
          const long long a0 = p.prof ? clock64() : 0;
          const uint32_t taddr = tmem_of(buf);
          // Software pipeline in steps of 16 columns: the next load is in flight while the current one is added.
          // (Blocks wholly below the diagonal are loaded and added too: their sums are simply never written.)
          uint32_t s0[16], s1[16];
          ptx::tmem_ld16(taddr, s0);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int h = 0; h < NCH * 2; ++h) {
            uint32_t* cur = (h & 1) ? s1 : s0;
            uint32_t* nxt = (h & 1) ? s0 : s1;
            if (h + 1 < NCH * 2) ptx::tmem_ld16(taddr + (uint32_t)((h + 1) * 16), nxt);
#pragma unroll
            for (int j = 0; j < 16; ++j) racc[h * 16 + j] += __uint_as_float(cur[j]);
            if (h + 1 < NCH * 2) ptx::tmem_ld_wait();
          }
          release(buf);
          if (p.prof) prof_sum += clock64() - a0;
        }
        if (!alive) break;
      } else if (!wait_chain(kWide ? 0 : (int)(gchunk & 1u))) {
        alive = false;
        break;
      }

      // ---- write the tile: one rolled loop over the warp's 32 x 32 blocks
      const long long o0 = p.prof ? clock64() : 0;
      EpilogueSums sums;
      const uint32_t taddr = tmem_of(kWide ? 0 : (int)(gchunk & 1u));
      // this unit's sums of block cc, one row per lane
      auto take_block = [&](int cc, float (&v)[32]) {
        if constexpr (chained) {
          // the running sums live in registers: static indices only
          auto take_sums = [&](auto first) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = racc[decltype(first)::value + j];
          };
          if (cc == 0) take_sums(std::integral_constant<int, 0>());
          if (cc == 1) take_sums(std::integral_constant<int, (chained && NCH > 1) ? 32 : 0>());
          if (cc == 2) take_sums(std::integral_constant<int, (chained && NCH > 2) ? 64 : 0>());
          if (cc == 3) take_sums(std::integral_constant<int, (chained && NCH > 2) ? 96 : 0>());
        } else {
          uint32_t raw[32];
          ptx::tmem_ld32(taddr + (uint32_t)(cc * 32), raw);
          ptx::tmem_ld_wait();
          // every block has been read: the MMA warp may have the accumulator back (a wide tile: this warp read columns of
          // half `half` only, and that half's barrier counts its four lane groups of both CTAs)
          if (cc == cc_end - 1) release(kWide ? half : (int)(gchunk & 1u));
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(raw[j]);
        }
      };
      // partial sums of (tile, split, warp, block): 32 floats of each lane, 16 bytes of all lanes side by side
      auto part_at = [&](int split, int cc) {
        const long long slot = ((long long)w.tile * p.splits + split) * (kPair ? 16 : 8) + (int)cta_rank * 8 + ew;
        return reinterpret_cast<float4*>(p.split_part) + (slot * NCH + cc) * 256 + lane;
      };
      auto add_parts = [&](int cc, float* v) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0.f;
        for (int split = 0; split < p.splits; ++split) {
          const float4* src = part_at(split, cc);
          constexpr int kAhead = chained ? 4 : 8;   // loads in flight (a chained kernel has its sums in registers as well)
#pragma unroll
          for (int j0 = 0; j0 < 8; j0 += kAhead) {
            float4 r[kAhead];
#pragma unroll
            for (int j = 0; j < kAhead; ++j) r[j] = __ldcg(src + 32 * (j0 + j));
#pragma unroll
            for (int j = 0; j < kAhead; ++j) {
              float* t = v + 4 * (j0 + j);
              t[0] += r[j].x; t[1] += r[j].y; t[2] += r[j].z; t[3] += r[j].w;
            }
          }
        }
      };
      bool mine = true;   // this warp writes the result
      if (p.splits > 1) {
        auto leave_part = [&](int cc, const float* v) {
          float4* dst = part_at(w.split, cc);
#pragma unroll
          for (int j = 0; j < 8; ++j) __stcg(dst + 32 * j, make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
        };
        if constexpr (chained) {
#pragma unroll
          for (int cc = 0; cc < NCH; ++cc)
            if (cc >= cc_first && cc < cc_end) leave_part(cc, racc + 32 * cc);
        } else {
#pragma unroll 1
          for (int cc = cc_first; cc < cc_end; ++cc) {
            float v[32];
            take_block(cc, v);
            leave_part(cc, v);
          }
        }
        __threadfence();
        __syncwarp();
        unsigned int before = 0;
        if (lane == 0) before = atomicAdd(p.split_count + (long long)w.tile * (kPair ? 16 : 8) + (int)cta_rank * 8 + ew, 1u);
        mine = __shfl_sync(0xffffffffu, before, 0) == (unsigned)(p.splits - 1);
        __threadfence();
        if (mine) {
          fetch_c(cc_first);
          if constexpr (chained) {   // the running sums have been handed over: their registers take the totals
#pragma unroll
            for (int cc = 0; cc < NCH; ++cc)
              if (cc >= cc_first && cc < cc_end) add_parts(cc, racc + 32 * cc);
          }
        }
      }
#pragma unroll 1
      for (int cc = cc_first; cc < cc_end && mine; ++cc) {
        const int c0 = col_first + cc * 32;
        float v[32];
        if (chained || p.splits == 1) take_block(cc, v);
        else add_parts(cc, v);
        if (boxed(c0)) {
          uint32_t held = c_buf;
          if (held) {
            const bool got = __all_sync(0xffffffffu, ptx::mbar_wait_unless(c_bar(ew), c_phase, kWaitCycles, abort_flag) ? 1 : 0);
            if (!got) {
              if (lane == 0) {
                report(p.status, kTimeoutEpilogue);
                raise_abort();
              }
              alive = false;
              break;
            }
            c_buf = 0;
            c_phase ^= 1u;
            float4 r[8];
            load_row_f32(held, lane, r);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              v[4 * j] = fmaf(e.beta, r[j].x, e.alpha * v[4 * j]);
              v[4 * j + 1] = fmaf(e.beta, r[j].y, e.alpha * v[4 * j + 1]);
              v[4 * j + 2] = fmaf(e.beta, r[j].z, e.alpha * v[4 * j + 2]);
              v[4 * j + 3] = fmaf(e.beta, r[j].w, e.alpha * v[4 * j + 3]);
            }
            __syncwarp();   // every lane has its row of C: the block is free
            if (c_apart) {
              held = 0;
              fetch_c(cc + 1);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] *= e.alpha;
          }
          epilogue_block(p, e, ring, v, held, b, row_first, c0, lane, p.tri && p.mirror && c0 == row_first, sums);
        } else {
          const uint32_t buf = ring.acquire();
          stage_rows_f32(buf, lane, v);
          __syncwarp();
          e.Cb = p.C ? p.C + (long long)b * p.c_bs : nullptr;
          e.Db = p.D ? p.D + (long long)b * p.d_bs : nullptr;
          e.Hb = p.D16 ? reinterpret_cast<uint16_t*>(p.D16) + (long long)b * p.d16_bs : nullptr;
          e.S0b = p.S0 ? p.S0 + (long long)b * p.s_bs : nullptr;
          e.S1b = p.S1 ? p.S1 + (long long)b * p.s_bs : nullptr;
          epilogue_block_scalar(p, e, reinterpret_cast<float*>(smem + (buf - base)), row_first, c0, lane, sums);
          if (ptx::elect_one()) ptx::bulk_commit();   // (nothing in flight: the ring counts one group per block)
        }
        if (!c_buf) fetch_c(cc + 1);
      }
      if (!alive) break;
      if (!chained) {
        if (cc_first >= cc_end) release(kWide ? half : (int)(gchunk & 1u));   // nothing of this tile is this warp's to read
        ++gchunk;
      }
      if (p.prof) prof_out += clock64() - o0;

      if (e.stats) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          sums.ssq += __shfl_xor_sync(0xffffffffu, sums.ssq, o);
          sums.mabs = fmaxf(sums.mabs, __shfl_xor_sync(0xffffffffu, sums.mabs, o));
          sums.maff = fmaxf(sums.maff, __shfl_xor_sync(0xffffffffu, sums.maff, o));
          sums.mres = fmaxf(sums.mres, __shfl_xor_sync(0xffffffffu, sums.mres, o));
        }
        if (lane == 0) {
          if (p.sumsq) atomicAdd(p.sumsq + b, sums.ssq);  // order of these additions is not fixed
          if (p.maxabs) atomicMax(p.maxabs + b, __float_as_uint(sums.mabs));
          if (p.maxaff) atomicMax(p.maxaff + b, __float_as_uint(sums.maff));
          if (p.maxres) atomicMax(p.maxres + b, __float_as_uint(sums.mres));
        }
      }
    }
    __syncwarp();
    if (ptx::elect_one()) {
      if (c_buf) ptx::mbar_wait(c_bar(ew), c_phase, kDrainCycles);   // (gave up with a block of C on its way)
      ptx::bulk_wait_all();   // the stores have read shared memory and are written before the CTA ends
    }
    if (p.prof && leader && warp == 4 && lane == 0) {
      atomicAdd(p.prof + 4, (unsigned long long)prof_wait);
      atomicAdd(p.prof + 5, (unsigned long long)prof_out);
      atomicAdd(p.prof + 6, (unsigned long long)prof_sum);
    }
  }

  // ---------------------------------------------------------------- teardown
  ptx::tc_fence_before();
  if constexpr (kPair) ptx::cluster_sync();  // neither CTA leaves while the other may still signal or read it
  else __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    if constexpr (kPair) ptx::tmem_dealloc_pair(tmem_base, S::kTmemCols);
    else ptx::tmem_dealloc(tmem_base, S::kTmemCols);
  }
}

}  // namespace toner
