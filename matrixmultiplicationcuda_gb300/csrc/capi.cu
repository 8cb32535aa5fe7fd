// C ABI of libbcsr_spmm: argument checks, error reporting and dispatch.
#include <cudaTypedefs.h>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>
#include "internal.h"

namespace spmm {

namespace {
thread_local std::string g_last_error;
std::mutex g_mu;
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
constexpr int kMaxDevices = 64;
unsigned* g_err_word[kMaxDevices] = {nullptr};
int g_sms[kMaxDevices] = {0};

bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

int current_device() {
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess) return -1;
  return d;
}
}  // namespace

spmm_status fail(spmm_status st, const std::string& msg) {
  g_last_error = msg;
  return st;
}

spmm_status host_fail(spmm_status st, const std::string& msg) { return fail(st, msg); }

void clear_error() { g_last_error.clear(); }

spmm_status cuda_fail(cudaError_t e, const char* what) {
  g_last_error = std::string(what) + ": " + cudaGetErrorString(e);
  return SPMM_ERR_CUDA;
}

int sm_count() {
  int d = current_device();
  if (d < 0 || d >= kMaxDevices) return 1;
  if (g_sms[d] == 0) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d);
    g_sms[d] = n > 0 ? n : 1;
  }
  return g_sms[d];
}

int smem_per_sm() {
  static int cache[kMaxDevices] = {0};
  int d = current_device();
  if (d < 0 || d >= kMaxDevices) return 0;
  if (cache[d] == 0) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMaxSharedMemoryPerMultiprocessor, d);
    cache[d] = n;
  }
  return cache[d];
}

namespace {
// Per-device caches of kernel attributes (keyed by kernel address).
struct FnKey {
  const void* fn;
  int dev, a, b;
  bool operator==(const FnKey& o) const { return fn == o.fn && dev == o.dev && a == o.a && b == o.b; }
};
struct FnVal {
  FnKey k;
  int v;
};
std::vector<FnVal> g_fn_cache;
}  // namespace

cudaError_t ensure_smem_attr(const void* fn, int bytes) {
  const FnKey k{fn, current_device(), bytes, -1};
  {
    std::lock_guard<std::mutex> lk(g_mu);
    for (const FnVal& e : g_fn_cache)
      if (e.k == k) return cudaSuccess;
  }
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) {
    std::lock_guard<std::mutex> lk(g_mu);
    g_fn_cache.push_back({k, 1});
  }
  return e;
}

int max_blocks_per_sm(const void* fn, int threads, size_t smem) {
  const FnKey k{fn, current_device(), threads, (int)smem};
  {
    std::lock_guard<std::mutex> lk(g_mu);
    for (const FnVal& e : g_fn_cache)
      if (e.k == k) return e.v;
  }
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, threads, smem) != cudaSuccess) n = 1;
  std::lock_guard<std::mutex> lk(g_mu);
  g_fn_cache.push_back({k, n});
  return n;
}

bool pdl_enabled() {
  static const bool on = std::getenv("SPMM_NO_PDL") == nullptr;
  return on;
}

unsigned* device_error_word() {
  int d = current_device();
  if (d < 0 || d >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_err_word[d]) {
    void* p = nullptr;
    if (cudaMalloc(&p, 256) != cudaSuccess) return nullptr;
    if (cudaMemset(p, 0, 256) != cudaSuccess) return nullptr;
    g_err_word[d] = static_cast<unsigned*>(p);
  }
  return g_err_word[d];
}

unsigned long long wait_limit_ns() {
  static unsigned long long v = [] {
    const char* s = std::getenv("SPMM_WAIT_LIMIT_NS");
    unsigned long long x = s ? std::strtoull(s, nullptr, 10) : 0ull;
    return x ? x : 1000000000ull;  // one second
  }();
  return v;
}

namespace {
// Encoded tensor maps, reused across calls: an encoding depends only on its
// arguments, and repeated products on the same buffers are the common case.
struct MapKey {
  int rank, dt, swz;
  const void* base;
  uint64_t d0, d1, d2, s0, s1;
  uint32_t b0, b1, b2;
  bool operator==(const MapKey& o) const { return std::memcmp(this, &o, sizeof(MapKey)) == 0; }
};
struct MapEntry {
  MapKey k;
  CUtensorMap map;
};
constexpr int kMapCache = 128;
MapEntry g_maps[kMapCache];
int g_maps_used = 0, g_maps_next = 0;

bool map_lookup(const MapKey& k, CUtensorMap* out) {
  std::lock_guard<std::mutex> lk(g_mu);
  for (int i = 0; i < g_maps_used; ++i)
    if (g_maps[i].k == k) {
      *out = g_maps[i].map;
      return true;
    }
  return false;
}
void map_store(const MapKey& k, const CUtensorMap& m) {
  std::lock_guard<std::mutex> lk(g_mu);
  MapEntry& e = g_maps[g_maps_next];
  e.k = k;
  e.map = m;
  g_maps_next = (g_maps_next + 1) % kMapCache;
  if (g_maps_used < kMapCache) ++g_maps_used;
}
MapKey map_key(int rank, int dt, int swz, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s0,
               uint64_t s1, uint32_t b0, uint32_t b1, uint32_t b2) {
  MapKey k;
  std::memset(&k, 0, sizeof(k));   // padding takes part in the comparison
  k.rank = rank;
  k.dt = dt;
  k.swz = swz;
  k.base = base;
  k.d0 = d0;
  k.d1 = d1;
  k.d2 = d2;
  k.s0 = s0;
  k.s1 = s1;
  k.b0 = b0;
  k.b1 = b1;
  k.b2 = b2;
  return k;
}
}  // namespace

spmm_status encode_tile_map_2d(CUtensorMap* map, CUtensorMapDataType dt, const void* base,
                               uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                               uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swz) {
  const MapKey key = map_key(2, (int)dt, (int)swz, base, inner, outer, 0, row_stride_bytes, 0, box_inner,
                             box_outer, 0);
  if (map_lookup(key, map)) return SPMM_OK;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_encode) {
      cudaDriverEntryPointQueryResult q;
      void* fn = nullptr;
      cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000,
                                                        cudaEnableDefault, &q);
      if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn)
        return fail(SPMM_ERR_CUDA, "cuTensorMapEncodeTiled entry point not available");
      g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
  }
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {row_stride_bytes};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode(map, dt, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(SPMM_ERR_INVALID_ARG,
                "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) +
                    "): B needs a 16-byte aligned base and a row stride that is a multiple of 16 bytes");
  map_store(key, *map);
  return SPMM_OK;
}

spmm_status encode_panel_map_3d(CUtensorMap* map, const void* base, uint64_t N, uint64_t K,
                                uint64_t row_stride_bytes, uint32_t boxes, int elem_bytes) {
  if (elem_bytes != 1 && elem_bytes != 2) return fail(SPMM_ERR_UNSUPPORTED, "panel map: 8- or 16-bit elements");
  const uint64_t W = 128 / (uint64_t)elem_bytes;
  const CUtensorMapDataType dt = elem_bytes == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16;
  if (N % W || boxes == 0 || boxes > 256)
    return fail(SPMM_ERR_UNSUPPORTED, "panel map needs N to be a multiple of 128 bytes of columns");
  const MapKey key = map_key(3, (int)dt, (int)CU_TENSOR_MAP_SWIZZLE_128B, base, W, K, N / W, row_stride_bytes, 128,
                             (uint32_t)W, 16, boxes);
  if (map_lookup(key, map)) return SPMM_OK;
  CUtensorMap probe;
  spmm_status st = encode_tile_map_2d(&probe, dt, base, N, K, row_stride_bytes, (uint32_t)W, 16,
                                      CU_TENSOR_MAP_SWIZZLE_128B);   // resolves the entry point
  if (st != SPMM_OK) return st;
  cuuint64_t dims[3] = {W, K, N / W};
  cuuint64_t strides[2] = {row_stride_bytes, 128};
  cuuint32_t box[3] = {(cuuint32_t)W, 16, boxes};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = g_encode(map, dt, 3, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(SPMM_ERR_UNSUPPORTED, "3-D panel tensor map rejected (" + std::to_string((int)r) + ")");
  map_store(key, *map);
  return SPMM_OK;
}

}  // namespace spmm

using namespace spmm;

extern "C" {

int spmm_abi_version(void) { return 1; }

const char* spmm_last_error(void) { return g_last_error.c_str(); }

int spmm_device_sm_count(void) { return sm_count(); }

spmm_status spmm_device_error_check(void* stream) {
  unsigned* w = device_error_word();
  if (!w) return fail(SPMM_ERR_CUDA, "no device error word");
  SPMM_CUDA_TRY(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
  unsigned v = 0;
  SPMM_CUDA_TRY(cudaMemcpy(&v, w, sizeof(v), cudaMemcpyDeviceToHost));
  if (v) {
    SPMM_CUDA_TRY(cudaMemset(w, 0, sizeof(unsigned)));
    if (v == 64u)   // only the scale check fired: every wait completed
      return fail(SPMM_ERR_INVALID_ARG,
                  "an e4m3 block scale is not a positive normal power of two (the tcgen05 e4m3 kernels take "
                  "each scale as a UE8M0 exponent; spmm_quantize makes such scales)");
    return fail(SPMM_ERR_TIMEOUT, "a device-side pipeline wait timed out (code " + std::to_string(v) + ")");
  }
  return SPMM_OK;
}

}  // extern "C"

namespace spmm {

// What a product with no configuration runs, from its sizes and (nnzb >= 0) the
// number of stored blocks. The lines stand where neither side of one was much
// slower than a single fixed kernel (the 128- or 256-column tcgen05 kernel for 64
// rows, mma.sync with single blocks for 16 and 32): at most 9 %, over 2500 products
// (M to 16384, K 256 to 16384, N 40 to 4096, 0.5 to 300 blocks a row; even, random
// and log-normal rows; replayed ten at a time on one GB300). items: block rows x
// 256-column tiles. Times in us, the line's two sides:
//   64-row blocks, fp16 and bf16:
//     - next to nothing to do (known): mma.sync. 43 rows of one block, N 104: 2.5
//       (64-row pipeline 4.3, tc128 4.8). Not for long rows, whose blocks one CTA
//       takes one by one: one row of 83, N 128: 19.0, tc128 12.4.
//     - as many items as SMs at most: the 64-row pipeline, which gives an item a
//       whole SM. 45 block rows, 97 blocks a row, N 512: 14.8, tc256 21.4; with
//       more its last round is half empty: 237 rows of one block, N 512: 11.8,
//       9.3; 184 rows of 61, N 120: 22.9, tc128 16.4.
//     - 128 columns and fewer: tc128, and the 64-row pipeline (items as above)
//       only for whole 64-column boxes: 83 rows of 39, N 40: 12.2, 10.1.
//     - 512-column tiles from 1024 columns and 256 of them on: 206 rows of 47, N
//       2048: 55 (64-row pipeline 66, tc256 68). Not for the shortest rows (known):
//       230 of 0.7, N 1024: 16.3, tc256 15.3.
//     - more than two items an SM and 8 or more blocks a row (known): the 64-row
//       pipeline (144 rows of 30, N 776: 25.0, 26.5), else tc256 (254 rows of 1.4, N
//       400: 11.8, 10.9). Rows of one or two blocks (known) take the static
//       stride, as a claim costs more than they do: 10.2 against 10.9.
//   split fp16 above 128 columns: the 64-row pipeline, but tc256 for more items
//     than SMs with less than 6 blocks a row or an unknown number (57 rows of two,
//     N 4096: 19.4, 14.0; but 190 rows of 19, N 512: 18.3, 22.8).
//   32- and 16-row blocks: mma.sync, whose CTAs are small, with single blocks
//     unless rows are known to be longer. From 5.5 blocks a row (8 with more items
//     than SMs, 16 then with part boxes below 128 columns) a ring of eight in
//     groups of four: one row of 12, N 64, 32 rows: 3.6, 4.4; 200 rows of 7, N 264:
//     5.6, 5.2; 382 of 11.5, N 72: 8.4, 7.7. Its tile is 128 columns wide: up to
//     64 columns only with few block rows (352 of 8, N 40: 7.9, 5.4; whole boxes
//     to four per SM: 14.8 to 12.6 us at 626 rows of 40, 16 rows, but 11.0 from 10.5
//     at 861 of 23). 16 rows: to two items an SM, the 256-column tile to three (206
//     rows of 25, N 512: 8.3, 128 columns 11.4, single blocks 9.7).
//     The longer the rows and the more the items, the better a tcgen05 CTA's
//     deeper ring: 32 rows, few items: 40 a row (one of 83, N 128 stays; 50 rows of
//     19, N 256: 6.8, 4.8 for the ring of eight), 20 with two an SM, 12 with more,
//     5 with five (8192^2, 5.7 a row, N 1024: 14.4, 16.6). 16 rows: 64 (14 rows of
//     17, N 512: 6.3, 4.1), not between two and three items an SM, where mma.sync's
//     CTAs hold all (322 rows of 21, N 256: 10.5, 7.4), 12 from five (10 from seven)
//     on: 8192^2, 10 a row, N 1024: 20.9, 22.0. Its tile is 256 columns wide, so
//     the last one has to be at least half used.
//   e4m3: mma.sync or, where converts_e4m3 says so, the tcgen05 pipeline with
//     e4m3 converted to fp16; both take any block scale whose products with the
//     block's values fp16 holds (the block-scaled MMA, which a caller may ask for,
//     is faster but needs powers of two). 16 rows and 2048 items or more:
//     mma.sync's 256-column tile (8192^2, 10 %, N 1024: 80 against 102 for 128
//     columns; 2 % and log-normal rows, N 2048: 48 against 59; 16384 x 4096, 2 %, N
//     512: 14.0 against 16.2). With fewer, 128 columns spread long rows further
//     (16384 x 4096, log-normal, N 256: 16.4 against 19.0), as where half of the
//     last 256 would be empty (N 272: 13.2, 14.2).
spmm_config default_config(int bR, spmm_dtype dtype, int M, int N, long long nnzb) {
  spmm_config c;
  std::memset(&c, 0, sizeof(c));
  const double row = nnzb >= 0 && M > 0 ? (double)nnzb * bR / M : -1.0;   // blocks per block row
  const long long sms = sm_count();
  // (rows not known: as with many)
  const long long items = M > 0 ? (long long)(M / bR) * ((N + 255) / 256) : 1ll << 40;
  auto tc = [&](int kernel, int nt, int acc) {
    c.kernel = kernel;
    c.n_tile = nt;
    c.acc_buffers = acc;
    c.schedule = 1;
    c.split_k = 1;
  };
  auto tc256 = [&] {
    tc(2, 256, 2);
    if (row >= 0 && row < 2.5) c.schedule = 0;
  };
  const bool sixteen = dtype == SPMM_F16 || dtype == SPMM_BF16;
  if (bR == 64 && dtype == SPMM_F16_SPLIT) {
    if (N <= 128)
      tc(2, 128, 2);
    else if (items <= sms || row >= 6)
      tc(3, 256, 0);
    else
      tc256();
    return c;
  }
  if (bR == 64 && sixteen && !(nnzb >= 0 && nnzb <= 100 && row <= 8)) {
    if (N <= 128) {
      if (items <= sms && N % 64 == 0)
        tc(3, 256, 0);
      else
        tc(2, 128, 2);
    } else if (!(row >= 0 && row < 2.5) && N >= 1024 && (N % 512 == 0 || N % 512 > 256) &&
               (long long)(M / 64) * ((N + 511) / 512) >= 256) {
      tc(2, 512, 2);
    } else if (items <= sms || (items > 2 * sms && row >= 8)) {
      tc(3, 256, 0);
    } else {
      tc256();
    }
    return c;
  }
  if (bR != 64 && sixteen && N > 128 && (N <= 256 || N > 384)) {   // the last 256-column tile at least half used
    const double long_row = bR == 32 ? (items <= sms ? 40 : items <= 2 * sms ? 20 : items < 5 * sms ? 12 : 5)
                                     : (items > 2 * sms && items <= 3 * sms ? 1e9 : items < 5 * sms ? 64 : items < 7 * sms ? 12 : 10);
    if (row >= long_row) {
      tc(2, 256, 2);
      return c;
    }
  }
  c.kernel = 1;
  c.n_tile = bR == 64 && sixteen ? 64 : mma_default_nt(bR, dtype, N);
  if (dtype == SPMM_E4M3 && bR == 16 && N > 128 && (N <= 256 || N > 384) && M > 0 && items >= 2048) c.n_tile = 256;
  c.stages = 4;
  if (bR != 64 && sixteen && row >= (items <= sms ? 5.5 : N < 128 && N % 64 ? 16 : 8)) {
    if (N <= 128) {
      if (c.n_tile != 64 || N > 64 || M / bR < (N % 64 == 0 ? 4 * sms : sms)) {
        c.n_tile = 128;
        c.stages = 8;
      }
    } else if (bR == 32 || items <= 2 * sms) {
      c.n_tile = 128;
      c.stages = 8;
    } else if (items <= 3 * sms && c.n_tile == 256) {
      c.stages = 8;
    }
  }
  return c;
}

// Whether an e4m3 product of known size runs converted to fp16 in the tcgen05
// pipeline instead of on mma.sync (us, converted against mma.sync):
//   64 rows: 16384^2, 2 % (20 blocks a row), N 512: 25.2, 32.4; 8192^2, 10 %, N
//     1024: 47.4, 69.7; 32 rows: 61.0, 79.5; 8192^2 with log-normal rows, 3 %, N
//     1024: 64 rows 32.0, 40.0, 32 rows 30.5, 41.4.
//   Short rows do not fill its ring, and with few items its last round of CTAs (two
//     an SM) is short of work: 64 rows, 8192^2, 10 a row, N 1024 (512 items): 17.3,
//     19.7, but 93 rows of 10, N 1024 (372): 15.1, 12.5; 32 rows: 166 rows of 11, N
//     1008 (664): 16.7, 13.6, 164 of 52, N 400 (328): 34.5, 30.6, but 314 of 21, N
//     512 (628): 21.3, 22.9, and 212 of 69, N 512 (424): 39, 48.
//   With fewer items than CTAs run at once the longest rows bound both, and
//     mma.sync's narrower tiles spread them further: 64 rows, 8192^2 with
//     log-normal rows, N 512 (256 items): 45.6, 42.0.
//   Its tile is 256 wide: 32 rows, 16384 x 8192, 5 %, N 272: 39.8, 34.8; 94 rows of
//     17, N 784: 17.1, 12.0; long rows: 422 of 55, N 784: 110, 112.
//   16 rows: slower (8192^2, 10 %, N 1024: 108, 80 with mma.sync's 256-column tile).
bool converts_e4m3(int bR, int M, int N, long long nnzb) {
  if (bR == 16 || nnzb < 0 || N <= 128 || (N > 256 && N <= 384)) return false;
  const long long items = (long long)(M / bR) * ((N + 255) / 256), sms = sm_count();
  const double row = (double)nnzb * bR / M;
  const bool whole = N % 256 == 0 || N % 256 > 128;   // the last tile at least half used
  if (!whole && row < 40) return false;
  return items >= 2.5 * sms && (row >= 24 || (items >= 3 * sms && row >= (bR == 64 ? 10 : 16)));
}

}  // namespace spmm

extern "C" {

spmm_status spmm_bcsr_mm(const spmm_bcsr_desc* A, const spmm_dense_desc* B, int N, float* C, int ldc,
                         const spmm_config* cfg, void* stream) {
  return spmm_bcsr_mm_nnzb(A, -1, B, N, C, ldc, cfg, stream);
}

spmm_status spmm_bcsr_mm_nnzb(const spmm_bcsr_desc* A, long long nnzb, const spmm_dense_desc* B, int N, float* C,
                         int ldc, const spmm_config* cfg, void* stream) {
  g_last_error.clear();
  if (!A || !B) return fail(SPMM_ERR_INVALID_ARG, "null descriptor");
  if (A->M < 0 || A->K < 0 || N < 0) return fail(SPMM_ERR_INVALID_ARG, "negative size");
  if (A->bC != 16) return fail(SPMM_ERR_UNSUPPORTED, "block width must be 16");
  if (A->bR != 16 && A->bR != 32 && A->bR != 64)
    return fail(SPMM_ERR_UNSUPPORTED, "block height must be 16, 32 or 64");
  if (A->M % A->bR) return fail(SPMM_ERR_INVALID_ARG, "M must be a multiple of the block height");
  if (A->K % 16) return fail(SPMM_ERR_INVALID_ARG, "K must be a multiple of 16");
  if (A->M == 0 || N == 0) return SPMM_OK;
  if (!A->row_ptr || !C || !B->data) return fail(SPMM_ERR_INVALID_ARG, "null pointer");
  // col_idx / vals may be NULL only when A stores no blocks (they are never read then)
  const bool e4m3 = A->dtype == SPMM_E4M3, split = A->dtype == SPMM_F16_SPLIT;
  if ((int)A->dtype < 0 || (int)A->dtype > 3) return fail(SPMM_ERR_INVALID_ARG, "unknown dtype");
  if (e4m3 && !A->scales) return fail(SPMM_ERR_INVALID_ARG, "E4M3 needs per-block scales");
  if (split && (!A->vals_lo || !B->data_lo))
    return fail(SPMM_ERR_INVALID_ARG, "F16_SPLIT needs the low halves of A and B");
  const int nmul = e4m3 ? 16 : 8;
  if (N % nmul) return fail(SPMM_ERR_UNSUPPORTED, "N must be a multiple of " + std::to_string(nmul));
  if (B->ldb < N || B->ldb % nmul) return fail(SPMM_ERR_MISALIGNED, "ldb must be >= N and a multiple of " + std::to_string(nmul));
  if (ldc < N || ldc % 4) return fail(SPMM_ERR_MISALIGNED, "ldc must be >= N and a multiple of 4");
  if (!aligned(A->vals, 16) || !aligned(B->data, 16) || !aligned(C, 16) ||
      (split && (!aligned(A->vals_lo, 16) || !aligned(B->data_lo, 16))))
    return fail(SPMM_ERR_MISALIGNED, "A values, B and C must be 16-byte aligned");
  if (A->K == 0) {
    // No block columns: C = 0 for the window.
    SPMM_CUDA_TRY(cudaMemset2DAsync(C, (size_t)ldc * 4, 0, (size_t)N * 4, A->M,
                                    static_cast<cudaStream_t>(stream)));
    return SPMM_OK;
  }
  LaunchRequest r;
  r.A = A;
  r.B = B;
  r.N = N;
  r.C = C;
  r.ldc = ldc;
  std::memset(&r.cfg, 0, sizeof(r.cfg));
  if (cfg) r.cfg = *cfg;
  r.stream = static_cast<cudaStream_t>(stream);
  if (r.cfg.kernel == 0) {
    // a configuration without a kernel may still set parts of one
    const spmm_config want = r.cfg;
    const bool plain = want.n_tile == 0 && want.stages == 0 && want.ctas_per_sm == 0 && want.acc_buffers == 0 &&
                       want.schedule == 0 && want.split_k <= 1;
    if (plain) {
      r.cfg = default_config(A->bR, A->dtype, A->M, N, nnzb);
      if (e4m3 && converts_e4m3(A->bR, A->M, N, nnzb)) {
        r.convert = true;
        r.cfg.kernel = 2;
        r.cfg.n_tile = 256;
        r.cfg.stages = 0;
        r.cfg.schedule = 1;
      } else if (e4m3 && nnzb >= 0) {
        // Lines where groups begin to pay: 16 rows of 3 to 8 blocks take 0.92 of the
        // time in groups, 64 rows of 3 to 8 1.00; 32 rows of 5 to 14 with several CTAs
        // on an SM 1.04 (174 rows of 6, N 400: 8.1, 6.9 us in single blocks), else 0.89.
        const bool full = (long long)(A->M / 32) * ((N + 127) / 128) > sm_count();
        r.single_blocks = (double)nnzb * A->bR < (A->bR == 16 ? 2.5 : A->bR == 32 && full ? 14 : 5.5) * A->M;
      }
    } else {
      r.cfg.kernel = A->bR == 64 && !e4m3 ? 2 : 1;
    }
    spmm_status st = r.cfg.kernel == 1 ? launch_mma(r) : r.cfg.kernel == 3 ? launch_tc64(r) : launch_tc(r);
    if (st != SPMM_ERR_UNSUPPORTED || r.cfg.kernel == 1) return st;
    g_last_error.clear();
    r.convert = false;
    r.cfg = want;
    r.cfg.kernel = 0;
    return launch_mma(r);
  }
  if (r.cfg.kernel == 3) return launch_tc64(r);
  if (r.cfg.kernel == 2) return launch_tc(r);
  return launch_mma(r);
}

spmm_status spmm_hcsr_mm(const spmm_bcsr_desc* A, const spmm_csr_desc* R, const spmm_dense_desc* B, int N,
                         float* C, int ldc, const spmm_config* cfg, void* stream) {
  g_last_error.clear();
  if (!A || !R || !B) return fail(SPMM_ERR_INVALID_ARG, "null descriptor");
  if (A->dtype != SPMM_F16) return fail(SPMM_ERR_UNSUPPORTED, "the hybrid product is fp16");
  if (R->M != A->M || R->K != A->K) return fail(SPMM_ERR_INVALID_ARG, "the two parts must have the same shape");
  if (A->M > 0 && !R->row_ptr) return fail(SPMM_ERR_INVALID_ARG, "null CSR row_ptr");
  spmm_config c;
  std::memset(&c, 0, sizeof(c));
  if (cfg)
    c = *cfg;
  else
    c.schedule = 1;   // the grid's pending blocks as items
  if (c.kernel != 0 && c.kernel != 2) return fail(SPMM_ERR_UNSUPPORTED, "the hybrid product runs on kernel 2");
  if (c.split_k > 1) return fail(SPMM_ERR_UNSUPPORTED, "the hybrid product has no split-K");
  c.kernel = 2;
  // the same argument checks as the BCSR product, then the launch with the CSR part
  if (A->M < 0 || A->K < 0 || N < 0) return fail(SPMM_ERR_INVALID_ARG, "negative size");
  if (A->bC != 16 || (A->bR != 16 && A->bR != 32 && A->bR != 64))
    return fail(SPMM_ERR_UNSUPPORTED, "block shape must be 16, 32 or 64 x 16");
  if (A->M % A->bR || A->K % 16) return fail(SPMM_ERR_INVALID_ARG, "M / K not multiples of the block shape");
  if (A->M == 0 || N == 0) return SPMM_OK;
  if (!A->row_ptr || !C || !B->data) return fail(SPMM_ERR_INVALID_ARG, "null pointer");
  if (N % 8) return fail(SPMM_ERR_UNSUPPORTED, "N must be a multiple of 8");
  if (B->ldb < N || B->ldb % 8) return fail(SPMM_ERR_MISALIGNED, "ldb must be >= N and a multiple of 8");
  if (ldc < N || ldc % 4) return fail(SPMM_ERR_MISALIGNED, "ldc must be >= N and a multiple of 4");
  if (!aligned(A->vals, 16) || !aligned(B->data, 16) || !aligned(C, 16))
    return fail(SPMM_ERR_MISALIGNED, "A values, B and C must be 16-byte aligned");
  if (A->K == 0) {
    SPMM_CUDA_TRY(cudaMemset2DAsync(C, (size_t)ldc * 4, 0, (size_t)N * 4, A->M, static_cast<cudaStream_t>(stream)));
    return SPMM_OK;
  }
  LaunchRequest r;
  r.A = A;
  r.B = B;
  r.N = N;
  r.C = C;
  r.ldc = ldc;
  r.cfg = c;
  r.stream = static_cast<cudaStream_t>(stream);
  // The CSR part in a launch of its own runs on every warp of an SM; in the
  // epilogue it has eight, whose B loads wait for L2. us, two launches against
  // the fused one: 4096^2, 10 % blocks, 2 % entries, N 1024: 68.8, 106; 0.5 %
  // entries, N 512: 24.1, 27.6; 1024^2, N 1024: 14.7, 15.0; 4096^2, N 64: 30.3,
  // 31.8; 5 % blocks, 0.1 % entries, N 128: 11.1, 12.0. Two launches cost a calling
  // loop more than the smallest products take: 256 x 288, N 2400: 11.2, 9.1.
  if (!cfg && (long long)A->M * N >= 1 << 18 && N <= 65535 * 256) {
    const spmm_status st = launch_tc(r);
    return st != SPMM_OK ? st : launch_csr_add(*R, *B, N, C, ldc, r.stream);
  }
  r.csr = R;
  return launch_tc(r);
}

static spmm_status ref_launch(int bR, const int* hdr, const int* idx, const void* data,
                              const void* B, float* C, unsigned M, unsigned N, unsigned K,
                              void* stream) {
  spmm_bcsr_desc a;
  std::memset(&a, 0, sizeof(a));
  a.M = (int)M;
  a.K = (int)K;
  a.bR = bR;
  a.bC = 16;
  a.row_ptr = hdr;
  a.col_idx = idx;
  a.vals = data;
  a.dtype = SPMM_F16;
  spmm_dense_desc b;
  std::memset(&b, 0, sizeof(b));
  b.data = B;
  b.scale = 1.0f;
  b.ldb = (int)N;
  return spmm_bcsr_mm(&a, &b, (int)N, C, (int)N, nullptr, stream);
}

spmm_status sparseMatrixMulTensor_launch(const int* hdr, const int* idx, const void* data,
                                         const void* B, float* C, unsigned M, unsigned N,
                                         unsigned K, void* stream) {
  return ref_launch(16, hdr, idx, data, B, C, M, N, K, stream);
}
spmm_status sparseMatrixMulTensor32x16_launch(const int* hdr, const int* idx, const void* data,
                                              const void* B, float* C, unsigned M, unsigned N,
                                              unsigned K, void* stream) {
  return ref_launch(32, hdr, idx, data, B, C, M, N, K, stream);
}
spmm_status sparseMatrixMulTensor64x16_launch(const int* hdr, const int* idx, const void* data,
                                              const void* B, float* C, unsigned M, unsigned N,
                                              unsigned K, void* stream) {
  return ref_launch(64, hdr, idx, data, B, C, M, N, K, stream);
}
// The reference's variant kernels (src/cuda_kernels.cuh:47-99) compute the
// same product as the kernel of their block shape with another warp split or
// staging; each name launches this library's pipeline for that block shape.
#define SPMM_VARIANT_LAUNCHER(NAME, BR)                                                                   \
  spmm_status NAME(const int* hdr, const int* idx, const void* data, const void* B, float* C, unsigned M, \
                   unsigned N, unsigned K, void* stream) {                                                \
    return ref_launch(BR, hdr, idx, data, B, C, M, N, K, stream);                                         \
  }
SPMM_VARIANT_LAUNCHER(sparseMatrixMulTensor_v2_launch, 16)
SPMM_VARIANT_LAUNCHER(sparseMatrixMulTensor_v3_launch, 16)
SPMM_VARIANT_LAUNCHER(sparseMatrixMulTensor_v1_improved_launch, 16)
SPMM_VARIANT_LAUNCHER(sparseMatrixMulTensor32x16_v2_launch, 32)
SPMM_VARIANT_LAUNCHER(sparseMatrixMulTensor32x16_shared_launch, 32)
SPMM_VARIANT_LAUNCHER(sparseMatrixMulTensor32x16_shared_vectorized_launch, 32)
SPMM_VARIANT_LAUNCHER(sparseMatrixMulTensor32x16_v2_shared_vectorized_launch, 32)
SPMM_VARIANT_LAUNCHER(sparseMatrixMulTensor64x16_v2_launch, 64)
SPMM_VARIANT_LAUNCHER(sparseMatrixMulTensor_option2_ldmatrix_sm80_launch, 16)
#undef SPMM_VARIANT_LAUNCHER
// sparseMatrixMulTensor1 (src/cuda_kernels.cu:330-355) multiplies square n x n
// matrices: its one size argument is M, N and K at once.
spmm_status sparseMatrixMulTensor1_launch(const int* hdr, const int* idx, const void* data, const void* B, float* C,
                                          unsigned n, void* stream) {
  return ref_launch(16, hdr, idx, data, B, C, n, n, n, stream);
}
spmm_status sparseMatrixMulTensorAdaptive_launch(const int* hdr, const int* idx, const void* data,
                                                 const void* B, float* C, unsigned M, unsigned N,
                                                 unsigned colBlocksPerRow, unsigned K,
                                                 void* stream) {
  (void)colBlocksPerRow;
  return ref_launch(16, hdr, idx, data, B, C, M, N, K, stream);
}
spmm_status sparseMatrixMulTensorAdaptive32x16_launch(const int* hdr, const int* idx,
                                                      const void* data, const void* B, float* C,
                                                      unsigned M, unsigned N,
                                                      unsigned colBlocksPerRow, unsigned K,
                                                      void* stream) {
  (void)colBlocksPerRow;
  return ref_launch(32, hdr, idx, data, B, C, M, N, K, stream);
}
spmm_status sparseMatrixMulTensorAdaptive64x16_launch(const int* hdr, const int* idx,
                                                      const void* data, const void* B, float* C,
                                                      unsigned M, unsigned N,
                                                      unsigned colBlocksPerRow, unsigned K,
                                                      void* stream) {
  (void)colBlocksPerRow;
  return ref_launch(64, hdr, idx, data, B, C, M, N, K, stream);
}

}  // extern "C"
