#include "tmap.h"

#include <atomic>
#include <memory>
#include <mutex>
#include <new>
#include <unordered_map>
#include <stdarg.h>
#include <string.h>

namespace blr {

static thread_local char g_last_error[512] = "";

void set_last_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
  va_end(ap);
}
const char* last_error() { return g_last_error; }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(p);
    }
  });
  return fn;
}

// Encoding a descriptor costs about a microsecond of host time and a call needs up to 18 of them, while
// the same weights come back call after call: keep the encoded descriptors, keyed by everything
// that went into them (addresses are unique over the devices of a process).  Two levels: a small direct-mapped table per
// thread, which needs no lock and one comparison, in front of the shared map.
struct TmapKey {
  uint64_t v[12];
  bool operator==(const TmapKey& o) const { return memcmp(v, o.v, sizeof(v)) == 0; }
};
static inline uint64_t tmap_hash(const TmapKey& k) {
  uint64_t h = 0x9E3779B97F4A7C15ull;
  for (int i = 0; i < 12; ++i) h = (h ^ k.v[i]) * 0xD6E8FEB86659FD93ull, h ^= h >> 32;
  return h;
}
struct TmapKeyHash {
  size_t operator()(const TmapKey& k) const { return (size_t)tmap_hash(k); }
};
static std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> g_tmap_cache;
static std::mutex g_tmap_mu;

struct TmapSlot {
  TmapKey key;  // v[0] = 0: empty (no descriptor has a null base)
  CUtensorMap map;
};
static constexpr int kTmapSlots = 1024;  // 224 KB per thread that calls the library
static thread_local std::unique_ptr<TmapSlot[]> t_tmap_slots;

int encode_tmap_4d(CUtensorMap* map, CUtensorMapDataType dt, const void* base, const uint64_t dims[4], const uint64_t strides[3],
                   const uint32_t box[4], Swz swz) {
  const TmapKey key = {{(uint64_t)reinterpret_cast<uintptr_t>(base), dims[0], dims[1], dims[2], dims[3], strides[0], strides[1], strides[2],
                        ((uint64_t)box[0] << 32) | box[1], ((uint64_t)box[2] << 32) | box[3], (uint64_t)dt, (uint64_t)swz}};
  // (no exception leaves a C entry point over a table: a host out of memory goes without)
  if (!t_tmap_slots) t_tmap_slots.reset(new (std::nothrow) TmapSlot[kTmapSlots]());
  TmapSlot* slot = t_tmap_slots ? &t_tmap_slots[tmap_hash(key) % kTmapSlots] : nullptr;
  if (base != nullptr && slot != nullptr && slot->key == key) {
    *map = slot->map;
    return BLR_OK;
  }
  auto keep = [&] {
    if (slot == nullptr) return;
    slot->key = key;
    slot->map = *map;
  };
  {
    std::lock_guard<std::mutex> lk(g_tmap_mu);
    auto it = g_tmap_cache.find(key);
    if (it != g_tmap_cache.end()) {
      *map = it->second;
      keep();
      return BLR_OK;
    }
  }
  EncodeTiledFn fn = get_encode_fn();
  BLR_REQUIRE(fn != nullptr, BLR_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  BLR_REQUIRE((reinterpret_cast<uintptr_t>(base) & 15) == 0, BLR_ERR_ALIGN, "tensor base %p is not 16-byte aligned", base);
  BLR_REQUIRE((strides[0] & 15) == 0 && (strides[1] & 15) == 0 && (strides[2] & 15) == 0, BLR_ERR_ALIGN,
              "tensor strides (%llu, %llu bytes) must be multiples of 16", (unsigned long long)strides[0],
              (unsigned long long)strides[1]);
  const int rank = box[3] == 0 ? 3 : 4;
  cuuint64_t gdims[4] = {dims[0], dims[1], dims[2], dims[3]};
  cuuint64_t gstr[3] = {strides[0], strides[1], strides[2]};
  cuuint32_t bx[4] = {box[0], box[1], box[2], box[3]};
  cuuint32_t es[4] = {1, 1, 1, 1};
  CUtensorMapSwizzle s = swz == Swz::B128 ? CU_TENSOR_MAP_SWIZZLE_128B
                         : swz == Swz::B64 ? CU_TENSOR_MAP_SWIZZLE_64B
                         : swz == Swz::B32 ? CU_TENSOR_MAP_SWIZZLE_32B
                                           : CU_TENSOR_MAP_SWIZZLE_NONE;
  CUresult r = fn(map, dt, (cuuint32_t)rank, const_cast<void*>(base), gdims, gstr, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE, s,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  BLR_REQUIRE(r == CUDA_SUCCESS, BLR_ERR_CUDA,
              "cuTensorMapEncodeTiled failed (%d): dims=(%llu,%llu,%llu) strides=(%llu,%llu) box=(%u,%u,%u)", (int)r,
              (unsigned long long)dims[0], (unsigned long long)dims[1], (unsigned long long)dims[2],
              (unsigned long long)strides[0], (unsigned long long)strides[1], box[0], box[1], box[2]);
  {
    std::lock_guard<std::mutex> lk(g_tmap_mu);
    if (g_tmap_cache.size() > 16384) g_tmap_cache.clear();
    try {
      g_tmap_cache.emplace(key, *map);
    } catch (const std::bad_alloc&) {
    }
  }
  keep();
  return BLR_OK;
}

int encode_tmap_3d(CUtensorMap* map, CUtensorMapDataType dt, const void* base, const uint64_t dims[3],
                   const uint64_t strides[2], const uint32_t box[3], Swz swz) {
  const uint64_t d[4] = {dims[0], dims[1], dims[2], 0}, st[3] = {strides[0], strides[1], 0};
  const uint32_t bx[4] = {box[0], box[1], box[2], 0};
  return encode_tmap_4d(map, dt, base, d, st, bx, swz);
}

static DeviceInfo g_devices[64];
static std::atomic<bool> g_device_known[64];

int device_info(DeviceInfo* out) {
  static std::mutex mu;
  int dev = 0;
  BLR_CUDA_OK(cudaGetDevice(&dev));
  BLR_REQUIRE(dev >= 0 && dev < 64, BLR_ERR_ARG, "device ordinal %d out of range", dev);
  if (!g_device_known[dev].load(std::memory_order_acquire)) {
    std::lock_guard<std::mutex> lk(mu);
    DeviceInfo d;
    BLR_CUDA_OK(cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev));
    BLR_CUDA_OK(cudaDeviceGetAttribute(&d.max_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    BLR_CUDA_OK(cudaDeviceGetAttribute(&d.coop, cudaDevAttrCooperativeLaunch, dev));
    d.dev = dev;
    g_devices[dev] = d;
    g_device_known[dev].store(true, std::memory_order_release);
  }
  *out = g_devices[dev];
  return BLR_OK;
}

int sm_count() {
  int n = 0;
  if (cudaGetDevice(&n) != cudaSuccess) {
    (void)cudaGetLastError();
    return 148;
  }
  if (n >= 0 && n < 64 && g_device_known[n].load(std::memory_order_acquire)) return g_devices[n].sm_count;  // (asked several times a call)
  DeviceInfo di;
  return device_info(&di) == BLR_OK && di.sm_count > 0 ? di.sm_count : 148;
}

}  // namespace blr
