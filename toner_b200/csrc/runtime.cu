// Per-device context, TMA tensor-map cache and the GEMM launcher.
#include "runtime.cuh"

#include "polar_chain.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace toner {

static thread_local std::string g_error;
static std::mutex g_mutex;
static Context g_ctx[16];

// One cached operand description: where its tensor maps sit in the arena, and the upload that put them there.
struct MapEntry {
  int slot = 0;
  cudaStream_t stream = nullptr;  // stream the upload was enqueued on
  cudaEvent_t uploaded = nullptr; // recorded right after the upload
  bool settled = false;           // the upload is known to have finished: no ordering needed any more
};
using MapCache = std::unordered_map<std::string, MapEntry>;

static std::atomic<long long> g_launches{0};
void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

void set_error(const std::string& msg) { g_error = msg; }
int fail(int code, const std::string& msg) {
  g_error = msg;
  return code;
}
const char* last_error() { return g_error.c_str(); }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn g_encode = nullptr;

static int load_encode() {
  if (g_encode) return 0;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
  if (e != cudaSuccess || fn == nullptr || q != cudaDriverEntryPointSuccess)
    return fail(kErrDriver, "cuTensorMapEncodeTiled is not available from the CUDA driver");
  g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  return 0;
}

Context* context() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) {
    set_error("no CUDA device is current: toner_b200 has no CPU path");
    return nullptr;
  }
  // Tensor maps are encoded by the driver on the launching thread, which has no context of its own until the runtime has
  // made a call on it that needs one: a thread's first call may be a product.
  static thread_local int bound = -1;
  if (bound != dev) {
    if (cudaSetDevice(dev) != cudaSuccess) {
      set_error("cudaSetDevice failed");
      return nullptr;
    }
    bound = dev;
  }
  std::lock_guard<std::mutex> lock(g_mutex);
  Context& c = g_ctx[dev];
  if (c.device == dev) return &c;
  if (load_encode()) return nullptr;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) {
    set_error("cudaGetDeviceProperties failed");
    return nullptr;
  }
  if (prop.major != 10) {
    set_error("toner_b200 kernels are built for sm_100a only; device reports sm_" + std::to_string(prop.major) +
              std::to_string(prop.minor));
    return nullptr;
  }
  c.num_sms = prop.multiProcessorCount;
  c.gemm_sms = c.num_sms;
  c.arena_cap = 32768;
  if (cudaMalloc(&c.arena_dev, sizeof(CUtensorMap) * c.arena_cap) != cudaSuccess ||
      cudaMallocHost(&c.arena_host, sizeof(CUtensorMap) * c.arena_cap) != cudaSuccess ||
      cudaMalloc(&c.status_dev, sizeof(int)) != cudaSuccess || cudaMemset(c.status_dev, 0, sizeof(int)) != cudaSuccess) {
    set_error("could not allocate the tensor-map arena");
    return nullptr;
  }
  c.map_cache = new MapCache();
  bool ok = true;
  auto allow = [&ok](auto kernel, int bytes) {
    ok = ok && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
  };
  allow(gemm_tcgen05_kernel<64, false>, GemmSmem<64>::kTotal);
  allow(gemm_tcgen05_kernel<64, true>, GemmSmem<64>::kTotal);
  allow(gemm_tcgen05_kernel<128, false>, GemmSmem<128>::kTotal);
  allow(gemm_tcgen05_kernel<128, true>, GemmSmem<128>::kTotal);
  allow(gemm_tcgen05_kernel<256, false>, GemmSmem<256>::kTotal);
  allow(gemm_tcgen05_kernel<256, true>, GemmSmem<256>::kTotal);
  allow(gemm_tcgen05_kernel<128, false, true, false, true>, GemmSmem<128, true>::kTotal);
  allow(gemm_tcgen05_kernel<128, true, true, false, true>, GemmSmem<128, true>::kTotal);
  allow(gemm_tcgen05_kernel<256, false, true, false, true>, GemmSmem<256, true>::kTotal);
  allow(gemm_tcgen05_kernel<256, true, true, false, true>, GemmSmem<256, true>::kTotal);
  allow(gemm_tcgen05_kernel<512, false, true, false, true>, GemmSmem<512, true>::kTotal);
  allow(gemm_tcgen05_kernel<128, false, true, true, true>, GemmSmem<128, true, true>::kTotal);
  allow(gemm_tcgen05_kernel<128, true, true, true, true>, GemmSmem<128, true, true>::kTotal);
  allow(gemm_tcgen05_kernel<256, false, true, true, true>, GemmSmem<256, true, true>::kTotal);
  allow(gemm_tcgen05_kernel<256, true, true, true, true>, GemmSmem<256, true, true>::kTotal);
  allow(gemm_tcgen05_kernel<128, false, true>, GemmSmem<128, true>::kTotal);
  allow(gemm_tcgen05_kernel<128, true, true>, GemmSmem<128, true>::kTotal);
  allow(gemm_tcgen05_kernel<256, false, true>, GemmSmem<256, true>::kTotal);
  allow(gemm_tcgen05_kernel<256, true, true>, GemmSmem<256, true>::kTotal);
  allow(gemm_tcgen05_kernel<128, false, true, true>, GemmSmem<128, true, true>::kTotal);
  allow(gemm_tcgen05_kernel<128, true, true, true>, GemmSmem<128, true, true>::kTotal);
  allow(gemm_tcgen05_kernel<256, false, true, true>, GemmSmem<256, true, true>::kTotal);
  allow(gemm_tcgen05_kernel<256, true, true, true>, GemmSmem<256, true, true>::kTotal);
  allow(polar_chain_kernel<256, true>, GemmSmem<256, true>::kTotal);
  allow(polar_chain_kernel<128, true>, GemmSmem<128, true>::kTotal);
  allow(polar_chain_kernel<64, false>, GemmSmem<64>::kTotal);
  allow(gemm_tcgen05_kernel<512, false, true>, GemmSmem<512, true>::kTotal);
  if (!ok || !allow_factor_kernels()) {
    set_error("the kernels' shared memory was refused");
    return nullptr;
  }
  c.device = dev;
  return &c;
}

static int encode_one(CUtensorMap* out, const void* base, int rows, int cols, long long ld, long long z_stride, int nz,
                      int box_rows) {
  if (base == nullptr) return fail(kErrArg, "null operand pointer");
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0) return fail(kErrArg, "operand base must be 16-byte aligned");
  if (ld % 8 != 0 || ld < cols) return fail(kErrArg, "operand leading dimension must be a multiple of 8 elements and >= cols");
  if (nz > 1 && z_stride % 8 != 0) return fail(kErrArg, "operand z stride must be a multiple of 8 elements");
  const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)(nz > 0 ? nz : 1)};
  const long long zs = (nz > 1) ? z_stride : (long long)rows * ld;
  const cuuint64_t strides[2] = {(cuuint64_t)ld * 2ull, (cuuint64_t)zs * 2ull};
  const cuuint32_t box[3] = {64u, (cuuint32_t)box_rows, 1u};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  CUresult r = g_encode(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(kErrDriver, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
  return 0;
}

// Map of the 32 x 32 boxes in which the GEMM's epilogue moves C and the results (elt: 4 = FP32, 2 = 16-bit).  False where
// the addresses or strides are not what TMA takes; the epilogue then goes element by element.
static bool encode_box(CUtensorMap* out, const void* base, int rows, int cols, long long ld, long long bs, int nz, int elt) {
  const long long zs = nz > 1 ? bs : (long long)rows * ld;
  if ((reinterpret_cast<uintptr_t>(base) & 15u) || (ld * elt) % 16 || (zs * elt) % 16 || ld < cols || zs <= 0) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)nz};
  const cuuint64_t strides[2] = {(cuuint64_t)(ld * elt), (cuuint64_t)(zs * elt)};
  const cuuint32_t box[3] = {32u, 32u, 1u};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  return g_encode(out, elt == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base),
                  dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  elt == 4 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int get_maps(Context* ctx, const toner_operand& op, int batch, int box_rows, cudaStream_t stream, const CUtensorMap** out) {
  const int count = batch;
  const int brows = op.mn_major ? 64 : box_rows;
  std::string key;
  key.reserve(64 + 8 * count);
  auto put = [&key](const void* p, size_t n) { key.append(reinterpret_cast<const char*>(p), n); };
  put(&op.rows, 4); put(&op.cols, 4); put(&op.ld, 8); put(&op.z_stride, 8); put(&op.nz, 4); put(&brows, 4);
  for (int i = 0; i < batch; ++i) put(&op.list[i], sizeof(void*));
  std::lock_guard<std::mutex> lock(g_mutex);
  auto* cache = static_cast<MapCache*>(ctx->map_cache);
  auto it = cache->find(key);
  if (it != cache->end()) {
    // The maps were uploaded by an asynchronous copy on the stream of the call that first used this operand.  A
    // launch on that stream is ordered after the copy by the stream itself; a launch on any other stream waits for
    // the copy's event (until the copy is known to be done, after which the entry needs no ordering at all).
    MapEntry& e = it->second;
    if (!e.settled) {
      if (cudaEventQuery(e.uploaded) == cudaSuccess) {
        e.settled = true;
      } else {
        (void)cudaGetLastError();  // cudaErrorNotReady is not an error here
        if (e.stream != stream) TONER_CUDA(cudaStreamWaitEvent(stream, e.uploaded, 0));
      }
    }
    *out = ctx->arena_dev + e.slot;
    return 0;
  }
  if (ctx->arena_used + count > ctx->arena_cap) {
    // Start over: wait for everything that may still read old maps, then reuse the arena from slot 0.
    TONER_CUDA(cudaDeviceSynchronize());
    for (auto& kv : *cache)
      if (kv.second.uploaded) cudaEventDestroy(kv.second.uploaded);
    cache->clear();
    ctx->arena_used = 0;
    if (count > ctx->arena_cap) return fail(kErrArg, "too many separately allocated operands in one call");
  }
  const int slot = ctx->arena_used;
  for (int i = 0; i < count; ++i) {
    if (op.list[i] == nullptr) return fail(kErrArg, "null operand pointer");
    int rc = encode_one(ctx->arena_host + slot + i, op.list[i], op.rows, op.cols, op.ld, op.z_stride, 1, brows);
    if (rc) return rc;
  }
  MapEntry e;
  e.slot = slot;
  e.stream = stream;
  TONER_CUDA(cudaEventCreateWithFlags(&e.uploaded, cudaEventDisableTiming));
  TONER_CUDA(cudaMemcpyAsync(ctx->arena_dev + slot, ctx->arena_host + slot, sizeof(CUtensorMap) * count,
                             cudaMemcpyHostToDevice, stream));
  TONER_CUDA(cudaEventRecord(e.uploaded, stream));
  ctx->arena_used += count;
  (*cache)[key] = e;
  *out = ctx->arena_dev + slot;
  return 0;
}

static long long gemm_tiles(const toner_gemm_desc& d, int bn, bool pair) {
  return (long long)gemm_tiles_per_batch(d.m, d.n, bn, d.tri, pair ? 2 * kBM : kBM) * d.batch;
}
static size_t split_part_bytes(const toner_gemm_desc& d, int bn, bool pair, int splits) {
  return (size_t)gemm_tiles(d, bn, pair) * splits * (pair ? 2 * kBM : kBM) * bn * sizeof(float);
}
static size_t split_count_bytes(const toner_gemm_desc& d, int bn, bool pair) {
  return (size_t)gemm_tiles(d, bn, pair) * (pair ? 16 : 8) * sizeof(unsigned int);
}

struct TileChoice {
  int bn;
  bool pair;
  int splits;
  size_t ws_bytes;   // scratch the splits need
};

// Whether a product's three plane products may be interleaved (toner_gemm_desc::interleave); only pair tiles do.
static bool may_interleave(const toner_gemm_desc& d) {
  return d.interleave && d.segs == 3 && !d.promote_all && d.a.seg_z[0] == d.a.seg_z[1] && d.b.seg_z[0] == d.b.seg_z[2];
}

// Which tile, and among how many units a tile's accumulation is divided (only where the caller gave scratch for it).  An
// estimate of the launch in SM cycles decides, from what was measured on the kernel:
//   * a 64-deep k-block takes 512 cycles of 256 x 256 on a pair and of 128 x 128 on one CTA, 384 of 256 x 128 on a pair and of
//     128 x 64, 768 of 128 x 256 -- what their copies take; deep products are faster by a quarter on the small tiles, which they
//     do not use;
//   * interleaved plane products bring two thirds of the operands: 256 x 256 stays bound by its MMAs, 256 x 128 takes 320 (one
//     product of 768 14.6 us plane by plane on 128 x 64, 13.8 interleaved on 256 x 128; twelve 25.5 on 256 x 256, 24.5);
//   * a 32 x 32 block of the epilogue takes a warp 900 cycles plus 450 per box moved, and its boxes take shared memory away
//     from the main loop of the next tile;
//   * tiles of one wave run side by side, and the epilogue of one tile beside the main loop of the next.
// Small problems so get many small tiles (one 768 x 768 product: 128 x 64), a batch that just misses a wave of large tiles
// gets 256 x 128, everything large gets 256 x 256.
static TileChoice choose_tile(const Context* ctx, const toner_gemm_desc& d) {
  struct Config {
    int bn;
    bool pair;
    double per_kb, per_kb_inter;
  };
  static const Config configs[] = {{256, true, 512, 512}, {128, true, 384, 320}, {256, false, 768, 768}, {128, false, 512, 512}, {64, false, 384, 384}};
  const bool inter = may_interleave(d);
  const bool mirror = d.tri && d.mirror;
  const double boxes = (d.c ? 1.2 : 0.0) + (d.d ? (mirror && !d.upper_d ? 2.0 : 1.0) : 0.0) + (d.d16 ? (mirror ? 1.6 : 1.0) : 0.0) +
                       ((d.split0 ? 1.3 : 0.0) + (d.split1 ? 1.3 : 0.0)) * (mirror ? 2.0 : 1.0);
  const double block = 900.0 + 450.0 * boxes, block_smem = 64.0 * boxes;
  const double kb = (double)((d.k + kBK - 1) / kBK) * d.segs;
  const int chains = d.promote > 0 ? ((d.k + kBK - 1) / kBK + d.promote - 1) / d.promote : (int)(kb / 4);
  TileChoice best = {256, true, 1, 0};
  double best_cost = 0.0;
  for (const Config& c : configs) {
    const long long tiles = gemm_tiles(d, c.bn, c.pair);
    const int workers = c.pair ? ctx->gemm_sms / 2 : ctx->gemm_sms;
    const int blocks = c.bn / 64;   // per epilogue warp
    const double main = kb * (inter ? c.per_kb_inter : c.per_kb), epi = blocks * block;
    const double waves = (double)((tiles + workers - 1) / workers);
    const double busy = main + blocks * 8 * block_smem;
    double cost = main + epi + (waves - 1) * (busy > epi ? busy : epi);
    int splits = 1;
    if (d.split_ws && d.segs == 1 && !(d.split_chains && d.promote <= 0)) {
      for (int s = d.split_chains && chains > 2 ? chains : 2; s <= 32 && s <= chains && tiles * s <= workers; ++s) {
        const size_t need = split_part_bytes(d, c.bn, c.pair, s) + split_count_bytes(d, c.bn, c.pair);
        if (need > (size_t)d.split_ws_bytes) break;
        const double parts = 4000.0 + blocks * (800.0 + 400.0 * s);   // writing and adding the parts, the extra memset
        if (main / s + parts + epi < cost) {
          cost = main / s + parts + epi;
          splits = s;
        }
      }
    }
    if (best_cost == 0.0 || cost < best_cost) {
      best_cost = cost;
      best = {c.bn, c.pair, splits, splits > 1 ? split_part_bytes(d, c.bn, c.pair, splits) + split_count_bytes(d, c.bn, c.pair) : 0};
    }
  }
  if (best.bn == 256 && best.pair && best.splits == 1 && d.promote <= 0 && !inter && kb >= ctx->gemm_wide_kb) {
    // The wide tile takes in 48 KB per k-block for twice the work of 32 KB and draws less power for it, but its epilogue is only
    // half hidden and its waves are coarser, and symmetric results have more of it below the diagonal.  Estimates of both, in
    // k-blocks of the pair tile; a k-block takes 1.72 (few waves) to 2 of those (measured wide / pair, three planes symmetric:
    // 2 x 4096^3 0.86, 12 x 3072^3 1.07, 18 x 2048^3 1.10, 6 x 5632^3 1.03, 32 x 512^3 1.15; one plane: 8192^3 0.96, 2 x 4096^3
    // symmetric 0.89, 6 x 5632^3 symmetric with C 1.14).
    auto waves = [&](int bn) {
      const long long t = gemm_tiles(d, bn, true), w = ctx->gemm_sms / 2;
      return (double)((t + w - 1) / w);
    };
    const double epi = 8 * block * 0.6 / 541.0;
    if (waves(512) * (kb * 1.8 + epi) < 0.97 * waves(256) * kb) best.bn = 512;
  }
  return best;
}

size_t gemm_split_bytes(const toner_gemm_desc& desc) {
  Context* ctx = context();
  if (!ctx) return 0;
  toner_gemm_desc d = desc;
  d.split_ws = ctx;                       // any address: the choice only asks whether there is one
  d.split_ws_bytes = (int64_t)256 << 20;  // scratch a caller is asked for at most
  return choose_tile(ctx, d).ws_bytes;
}

// The kernel's parameters for one product on a given tile.
static int gemm_params(Context* ctx, const toner_gemm_desc& d, int bn, bool pair, int splits, bool inter, cudaStream_t stream, GemmParams& p) {
  std::memset(&p, 0, sizeof(p));
  // a pair's CTA loads half a tile's rows of B, at most 128 at a time; MN-major operands always come in 64 x 64 boxes
  auto operand_map = [&](const toner_operand& op, int box_rows, CUtensorMap* map, const CUtensorMap** maps) {
    if (op.list) return get_maps(ctx, op, d.batch, box_rows, stream, maps);
    return encode_one(map, op.base, op.rows, op.cols, op.ld, op.z_stride, op.nz, op.mn_major ? 64 : box_rows);
  };
  int rc = operand_map(d.a, kBM, &p.a_map, &p.a_maps);
  if (rc) return rc;
  rc = operand_map(d.b, pair ? (bn == 128 ? 64 : 128) : bn, &p.b_map, &p.b_maps);
  if (rc) return rc;
  p.a_z_stride = d.a.list ? 0 : d.a.z_step;
  p.b_z_stride = d.b.list ? 0 : d.b.z_step;
  p.a_mn = d.a.mn_major ? 1 : 0;
  p.b_mn = d.b.mn_major ? 1 : 0;
  for (int s = 0; s < kMaxSegs; ++s) {
    p.a_seg_z[s] = d.a.list ? 0 : d.a.seg_z[s];
    p.b_seg_z[s] = d.b.list ? 0 : d.b.seg_z[s];
  }
  p.segs = inter ? 1 : d.segs;
  p.M = d.m; p.N = d.n; p.K = d.k; p.batch = d.batch;
  p.fmt = d.fmt;
  p.tri = d.tri ? 1 : 0;
  p.promote = d.promote > 0 ? (inter && d.promote > 2 ? (2 * d.promote + 1) / 3 : d.promote) : 0;   // (see gemm_tcgen05_kernel)
  p.promote_all = d.promote_all ? 1 : 0;
  p.raster = d.tri ? 0 : (d.raster > 0 ? d.raster : (bn == 512 ? 4 : 8));   // (a group of 2048 columns)
  p.alpha = d.alpha; p.beta = d.beta;
  p.alpha_a = d.alpha_a; p.alpha_b = d.alpha_b; p.beta_v = d.beta_v;
  p.alpha_b_step = d.alpha_b_step > 0 ? d.alpha_b_step : 1;
  p.C = d.c; p.ldc = d.ldc; p.c_bs = d.c_bs;
  p.D = d.d; p.ldd = d.ldd; p.d_bs = d.d_bs;
  p.D16 = d.d16; p.ld16 = d.ld16; p.d16_bs = d.d16_bs; p.d16_fmt = d.d16_fmt;
  p.packed = d.packed ? 1 : 0;
  p.mirror = d.mirror ? 1 : 0;
  p.upper_d = (d.upper_d && d.tri && d.mirror) ? 1 : 0;
  p.tma_ok = !d.packed;
  if (p.tma_ok && d.c) p.tma_ok = encode_box(&p.c_map, d.c, d.m, d.n, d.ldc, d.c_bs, d.batch, 4);
  if (p.tma_ok && d.d) p.tma_ok = encode_box(&p.d_map, d.d, d.m, d.n, d.ldd, d.d_bs, d.batch, 4);
  if (p.tma_ok && d.d16) p.tma_ok = encode_box(&p.h_map, d.d16, d.m, d.n, d.ld16, d.d16_bs, d.batch, 2);
  if (p.tma_ok && (d.split0 || d.split1)) {
    // the lo plane is reached through the batch coordinate: a whole number of batch strides behind the hi plane
    const long long step = d.batch > 1 ? d.split_bs : d.split_plane;
    p.tma_ok = step > 0 && d.split_plane > 0 && d.split_plane % step == 0 && d.split_plane / step < (1 << 30);
    p.s_lo_z = p.tma_ok ? (int)(d.split_plane / step) : 0;
    if (p.tma_ok && d.split0) p.tma_ok = encode_box(&p.s0_map, d.split0, d.m, d.n, d.split_ld, step, p.s_lo_z + d.batch, 2);
    if (p.tma_ok && d.split1) p.tma_ok = encode_box(&p.s1_map, d.split1, d.m, d.n, d.split_ld, step, p.s_lo_z + d.batch, 2);
  }
  p.S0 = static_cast<__half*>(d.split0); p.S1 = static_cast<__half*>(d.split1);
  p.s_ld = d.split_ld; p.s_bs = d.split_bs; p.s_plane = d.split_plane;
  p.s0_scale = d.split0_scale; p.s0_aff_a = d.split0_aff_a; p.s1_scale = d.split1_scale; p.s1_aff_a = d.split1_aff_a; p.s1_aff_b = d.split1_aff_b;
  p.maxres = d.maxres;
  p.sumsq = d.sumsq; p.maxabs = d.maxabs; p.maxaff = d.maxaff;
  p.aff_a = d.aff_a; p.aff_b = d.aff_b;
  p.splits = splits;
  if (splits > 1) {
    const size_t parts = split_part_bytes(d, bn, pair, splits), counts = split_count_bytes(d, bn, pair);
    p.split_part = static_cast<float*>(d.split_ws);
    p.split_count = reinterpret_cast<unsigned int*>(static_cast<char*>(d.split_ws) + parts);
    TONER_CUDA(cudaMemsetAsync(p.split_count, 0, counts, stream));
  }
  p.status = ctx->status_dev;
  p.prof = ctx->prof_dev;
  return 0;
}

int launch_gemm(const toner_gemm_desc& d, cudaStream_t stream, const GemmMore& more) {
  Context* ctx = context();
  if (!ctx) return kErrCuda;
  if (d.m <= 0 || d.n <= 0 || d.k <= 0 || d.batch <= 0) return fail(kErrArg, "gemm: sizes must be positive");
  if (d.segs < 1 || d.segs > kMaxSegs) return fail(kErrArg, "gemm: segs must be 1..3");
  if (d.tri && d.m != d.n) return fail(kErrArg, "gemm: a symmetric result needs m == n");
  if (d.packed && (!d.tri || d.mirror || d.d16)) return fail(kErrArg, "gemm: packed output is upper-triangle FP32 only");
  if (!d.d && !d.d16 && !d.split0 && !d.split1) return fail(kErrArg, "gemm: no output");
  if (d.packed && (d.split0 || d.split1)) return fail(kErrArg, "gemm: operand planes cannot be packed");
  if (reinterpret_cast<uintptr_t>(d.split_ws) & 15u) return fail(kErrArg, "gemm: split_ws must be 16-byte aligned");
  if (d.fmt != 0 && d.fmt != 1) return fail(kErrArg, "gemm: fmt must be 0 (FP16) or 1 (BF16)");

  int bn = d.tile_n, splits = 1;
  bool pair = false;
  if (bn == 0) {
    const TileChoice t = choose_tile(ctx, d);
    bn = t.bn;
    pair = t.pair;
    splits = t.splits;
  } else if (bn == 512) {
    bn = 256;
    pair = true;
  } else if (bn == -128) {
    bn = 128;
    pair = true;
  } else if (bn == 1024) {
    if (d.promote > 0) return fail(kErrArg, "gemm: the wide tile has no chained accumulation");
    bn = 512;
    pair = true;
  }
  if (!(bn == 64 && !pair) && bn != 128 && bn != 256 && !(bn == 512 && pair))
    return fail(kErrArg, "gemm: tile_n must be 0, 64, 128, 256, -128 (256 x 128 on a CTA pair), 512 (256 x 256 on a pair) or 1024 "
                         "(256 x 512 on a pair)");

  if (more.half_in && !pair) {   // (large stacks: pair tiles, of which alone there are kernels for it)
    bn = 128;
    pair = true;
    splits = 1;
  }
  const bool inter = pair && bn <= 256 && may_interleave(d);
  GemmParams p;
  if (int rc = gemm_params(ctx, d, bn, pair, splits, inter, stream, p)) return rc;
  p.skip = more.skip;
  p.half_out = more.half_out ? 1 : 0;
  if (more.half_in) {
    if (d.a.list || d.b.list || d.a.mn_major || d.b.mn_major) return fail(kErrArg, "gemm: half-stored operands are K-major stacks");
    int rc = encode_one(&p.a_turned, d.a.base, d.a.rows, d.a.cols, d.a.ld, d.a.z_stride, d.a.nz, 64);
    if (rc) return rc;
    if (d.b.base == d.a.base) p.b_turned = p.a_turned;
    else rc = encode_one(&p.b_turned, d.b.base, d.b.rows, d.b.cols, d.b.ld, d.b.z_stride, d.b.nz, 64);
    if (rc) return rc;
  }

  const long long total = gemm_tiles(d, bn, pair) * splits;
  if (total > 0x7fffffffLL) return fail(kErrArg, "gemm: too many tiles");
  const bool chained = p.promote > 0;
  const int workers = pair ? ctx->gemm_sms / 2 : ctx->gemm_sms;
  const int grid = (int)(total < workers ? total : workers) * (pair ? 2 : 1);
#define TONER_INTER(BN, CHAINED)                                                                                                        \
  TONER_CUDA(launch(more.half_in ? gemm_tcgen05_kernel<BN, CHAINED, true, true, true> : gemm_tcgen05_kernel<BN, CHAINED, true, true>, grid, \
                    kGemmThreads, GemmSmem<BN, true, true>::kTotal, stream, 2, p))
  if (inter) {
    if (bn == 256 && chained) TONER_INTER(256, true);
    else if (bn == 256) TONER_INTER(256, false);
    else if (chained) TONER_INTER(128, true);
    else TONER_INTER(128, false);
    return 0;
  }
#undef TONER_INTER
#define TONER_GEMM(BN, CHAINED, PAIR)                                                                                                  \
  TONER_CUDA(launch(PAIR && more.half_in ? gemm_tcgen05_kernel<BN, CHAINED, PAIR, false, PAIR> : gemm_tcgen05_kernel<BN, CHAINED, PAIR>, \
                    grid, kGemmThreads, GemmSmem<BN, PAIR>::kTotal, stream, PAIR ? 2 : 0, p))
  if (pair && bn == 512) TONER_GEMM(512, false, true);
  else if (pair && bn == 256 && chained) TONER_GEMM(256, true, true);
  else if (pair && bn == 256) TONER_GEMM(256, false, true);
  else if (pair && chained) TONER_GEMM(128, true, true);
  else if (pair) TONER_GEMM(128, false, true);
  else if (bn == 256 && chained) TONER_GEMM(256, true, false);
  else if (bn == 256) TONER_GEMM(256, false, false);
  else if (bn == 128 && chained) TONER_GEMM(128, true, false);
  else if (bn == 128) TONER_GEMM(128, false, false);
  else if (chained) TONER_GEMM(64, true, false);
  else TONER_GEMM(64, false, false);
#undef TONER_GEMM
  return 0;
}

int launch_polar_chain(const toner_gemm_desc (&ops)[6], int steps, bool in_step, unsigned int* claim, unsigned int* done,
                       cudaStream_t stream, bool* taken) {
  *taken = false;
  Context* ctx = context();
  if (!ctx) return kErrCuda;
  // Deeper products hide their ends behind their own tiles, and one nearly square matrix has nothing to overlap: its tiles wait for
  // each other, and a counter is a slower hand-over than a launch.  Launched / chained, us, ten steps: 768^2 252 / 292, 1280^2
  // 358 / 397, 768 x 3072 378 / 376, 2 x 768^2 262 / 270 and 4 x 1280^2 650 / 541; five steps: 512 x 2048 147 / 137, 768 x 3072
  // 196 / 180, 2 x 768^2 138 / 136.  Depth, ten steps: 2 x 1536^2 574 / 558, 8 x 1536^2 1660 / 1240, 2 x 2048^2 885 / 1155, 24 x
  // 2048^2 8384 / 8424; between them it depends on the shape: 2 x 1664^2 790 / 650, a MuonT step of 2 x 2120 x 1688 2802 / 2933.
  // In an optimizer's step the host prepares the next launches meanwhile: thirty of them take it 91 us, this one 14, and a MuonT
  // step of one 768^2 layer 930 us with them, 880 with it.  There such a matrix is chained from eight steps on.
  constexpr int kChainDepth = 1536, kChainSteps = 8;
  const int depth = ops[2].k;
  const bool alone = (long long)ops[3].batch * std::max(ops[3].m, ops[3].n) < 2LL * depth;
  if (depth > kChainDepth || (alone && !(in_step && steps >= kChainSteps))) return 0;
  struct Config {
    int bn;
    bool pair;
    double per_kb;
  };
  // As in choose_tile, but a product's last wave is filled by the next product's tiles: what counts is the time of a tile, times
  // the tiles a worker gets, and that of a whole tile, first copy to last store, where a product has fewer tiles than workers.
  static const Config configs[] = {{256, true, 541}, {128, true, 400}, {64, false, 384}};
  const Config* best = nullptr;
  double best_cost = 0.0;
  for (const Config& c : configs) {
    double cost = 0.0;
    for (int i : {0, 2, 3}) {
      const toner_gemm_desc& d = ops[i];
      const double boxes = (d.c ? 1.2 : 0.0) + (d.d ? 1.0 : 0.0) + (d.d16 ? (d.tri ? 1.6 : 1.0) : 0.0);
      const double main = (d.k + kBK - 1) / kBK * c.per_kb, epi = c.bn / 64 * (300.0 + 850.0 * boxes);
      const double tiles = (double)gemm_tiles(d, c.bn, c.pair) / (c.pair ? ctx->gemm_sms / 2 : ctx->gemm_sms);
      const double each = std::max(main, epi) + 0.25 * std::min(main, epi);   // (they share the SM's paths to L2)
      cost += std::max(tiles * each, main + epi + 4000.0);
    }
    if (!best || cost < best_cost) {
      best = &c;
      best_cost = cost;
    }
  }
  PolarChain p;
  std::memset(&p, 0, sizeof(p));
  for (int i = 0; i < 6; ++i) {
    if (int rc = gemm_params(ctx, ops[i], best->bn, best->pair, 1, false, stream, p.op[i])) return rc;
    if (!p.op[i].tma_ok) return 0;
  }
  p.steps = steps;
  p.batch = ops[0].batch;
  const int workers = best->pair ? ctx->gemm_sms / 2 : ctx->gemm_sms;
  long long widest = 0;
  for (int i = 0; i < 3; ++i) {
    const toner_gemm_desc& d = ops[i + (i > 0)];
    p.tiles[i] = gemm_tiles_per_batch(d.m, d.n, best->bn, d.tri, best->pair ? 2 * kBM : kBM);
    widest = std::max(widest, (long long)p.tiles[i] * p.batch);
  }
  if (widest * 3 * steps > 0x3fffffffLL) return 0;   // (unit numbers and done[] have 32 bits)
  p.claim = claim;
  p.done = done;
  const int grid = (int)(widest < workers ? widest : workers) * (best->pair ? 2 : 1);
  if (best->bn == 256) TONER_CUDA(launch(polar_chain_kernel<256, true>, grid, kChainThreads, GemmSmem<256, true>::kTotal, stream, 2, p));
  else if (best->bn == 128) TONER_CUDA(launch(polar_chain_kernel<128, true>, grid, kChainThreads, GemmSmem<128, true>::kTotal, stream, 2, p));
  else TONER_CUDA(launch(polar_chain_kernel<64, false>, grid, kChainThreads, GemmSmem<64>::kTotal, stream, 0, p));
  *taken = true;
  return 0;
}

// A wait that nothing will ever satisfy: the barrier expects one arrival and gets none.  The wait gives up after
// `limit_cycles`, reports through the status word like the GEMM's waits do, and the kernel returns normally.
__global__ void bounded_wait_selftest_kernel(long long limit_cycles, int* status) {
  __shared__ unsigned long long bar;
  const uint32_t b = ptx::smem_u32(&bar);
  if (threadIdx.x == 0) {
    ptx::mbar_init(b, 1);
    ptx::fence_mbar_init();
  }
  __syncthreads();
  if (threadIdx.x == 0 && !ptx::mbar_wait(b, 0, limit_cycles)) report(status, kTimeoutSelftest);
}

}  // namespace toner

// ------------------------------------------------------------------ C ABI: library + generic GEMM
extern "C" {

int toner_init(int device) {
  if (cudaSetDevice(device) != cudaSuccess) return toner::fail(toner::kErrCuda, "cudaSetDevice failed");
  return toner::context() ? 0 : toner::kErrCuda;
}

const char* toner_last_error(void) {
  return toner::g_error.c_str();
}

long long toner_launch_count(void) { return toner::g_launches.load(std::memory_order_relaxed); }

int toner_sm_count(void) {
  toner::Context* c = toner::context();
  return c ? c->num_sms : 0;
}

int toner_set_gemm_sm_limit(int32_t sms) {
  toner::Context* c = toner::context();
  if (!c) return toner::kErrCuda;
  if (sms < 0) return toner::fail(toner::kErrArg, "gemm sm limit: must be 0 (all) or a positive count");
  int n = sms == 0 || sms > c->num_sms ? c->num_sms : sms;
  n &= ~1;  // CTA pairs
  c->gemm_sms = n < 2 ? 2 : n;
  return 0;
}

int toner_device_status(void* stream, int* status_out) {
  toner::Context* c = toner::context();
  if (!c) return toner::kErrCuda;
  if (!status_out) return toner::fail(toner::kErrArg, "status_out is null");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int v = 0;
  TONER_CUDA(cudaMemcpyAsync(&v, c->status_dev, sizeof(int), cudaMemcpyDeviceToHost, s));
  TONER_CUDA(cudaStreamSynchronize(s));
  if (v != 0) TONER_CUDA(cudaMemsetAsync(c->status_dev, 0, sizeof(int), s));
  *status_out = v;
  return 0;
}

int toner_status_snapshot(int32_t* host_out, void* stream) {
  toner::Context* c = toner::context();
  if (!c) return toner::kErrCuda;
  if (!host_out) return toner::fail(toner::kErrArg, "status_snapshot: host_out is null");
  TONER_CUDA(cudaMemcpyAsync(host_out, c->status_dev, sizeof(int), cudaMemcpyDeviceToHost, static_cast<cudaStream_t>(stream)));
  return 0;
}

int toner_selftest_bounded_wait(long long limit_cycles, void* stream) {
  toner::Context* c = toner::context();
  if (!c) return toner::kErrCuda;
  if (limit_cycles <= 0 || limit_cycles > 2000000000LL)
    return toner::fail(toner::kErrArg, "selftest: the limit must be between 1 and 2e9 cycles");
  toner::bounded_wait_selftest_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(limit_cycles, c->status_dev);
  toner::count_launch();
  TONER_CUDA(cudaGetLastError());
  return 0;
}

int toner_gemm_phase_cycles(int enable, void* stream, unsigned long long* out8) {
  toner::Context* c = toner::context();
  if (!c) return toner::kErrCuda;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (out8) {
    for (int i = 0; i < 8; ++i) out8[i] = 0;
    if (c->prof_dev) {
      TONER_CUDA(cudaMemcpyAsync(out8, c->prof_dev, 8 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
      TONER_CUDA(cudaStreamSynchronize(s));
      TONER_CUDA(cudaMemsetAsync(c->prof_dev, 0, 8 * sizeof(unsigned long long), s));
    }
  }
  if (enable && !c->prof_dev) {
    TONER_CUDA(cudaMalloc(&c->prof_dev, 8 * sizeof(unsigned long long)));
    TONER_CUDA(cudaMemset(c->prof_dev, 0, 8 * sizeof(unsigned long long)));
  } else if (!enable && c->prof_dev) {
    TONER_CUDA(cudaStreamSynchronize(s));
    TONER_CUDA(cudaFree(c->prof_dev));
    c->prof_dev = nullptr;
  }
  return 0;
}

int toner_gemm(const toner_gemm_desc* desc, void* stream) {
  if (!desc) return toner::fail(toner::kErrArg, "gemm: null descriptor");
  return toner::launch_gemm(*desc, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
