// Host side of libfa_b200.so: the C ABI declared in include/fa_b200.h.
// Validates arguments, builds the TMA descriptors, launches the sm_100a kernel on the caller's
// stream.  No exceptions, no torch types, no CPU fallback: a device that is not 10.x is an error.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <mutex>

#include "../../include/fa_b200.h"
#include "add_layernorm_sm100.cuh"
#include "cache_write_sm100.cuh"
#include "fa_decode_sm100.cuh"
#include "fa_fwd_sm100.cuh"
#include "gpt_step_sm100.cuh"
#include "linear_small_sm100.cuh"

namespace {

constexpr int kMaxDevices = 64;

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

struct DeviceState {
  std::once_flag once;
  int init_error = 0;       // value fa_b200_fwd returns if set-up failed
  unsigned int* status = nullptr;  // device address of the watchdog words
  int resident_ctas = 0;           // persistent grid size: CTAs per SM x SM count
  int sm_count = 0;
};

DeviceState g_dev[kMaxDevices];
std::once_flag g_encode_once;
EncodeTiledFn g_encode = nullptr;

// Watchdog words, one set per device that loads the module (a __device__ variable is
// instantiated per device).  Word 0: code, 1: blockIdx.x, 2: threadIdx.x, 3: barrier parity.
__device__ unsigned int g_fa_status[4];

void resolve_encode() {
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) ==
          cudaSuccess &&
      qres == cudaDriverEntryPointSuccess)
    g_encode = reinterpret_cast<EncodeTiledFn>(fn);
}

struct DeviceGuard {
  int prev = -1;
  bool switched = false;
  int error = 0;
  explicit DeviceGuard(int dev) {
    cudaError_t e = cudaGetDevice(&prev);
    if (e != cudaSuccess) { error = static_cast<int>(e); return; }
    if (prev != dev) {
      e = cudaSetDevice(dev);
      if (e != cudaSuccess) { error = static_cast<int>(e); return; }
      switched = true;
    }
  }
  ~DeviceGuard() {
    if (switched) cudaSetDevice(prev);
  }
};

using FwdKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, fa::FwdParams);
template <int kSchedule>
FwdKernel fwd_kernel_of(bool causal, bool ragged) {
  if (causal) return &fa::fa_fwd_kernel<kSchedule, true>;
  return ragged ? &fa::fa_fwd_kernel<kSchedule, false, true> : &fa::fa_fwd_kernel<kSchedule, false>;
}
// Causal sequences from here on take the instantiation with the diagonal tile behind the loop (figures: fa_fwd_kernel).
constexpr int kLongRows = 12288;
FwdKernel fwd_kernel(int schedule, bool causal, bool ragged, bool is_long = false) {
  if (is_long && schedule == fa::kOneItem) return &fa::fa_fwd_kernel<fa::kOneItem, true, false, true>;
  if (is_long && schedule == fa::kDynamic) return &fa::fa_fwd_kernel<fa::kDynamic, true, false, true>;
  return schedule == fa::kOneItem ? fwd_kernel_of<fa::kOneItem>(causal, ragged)
         : schedule == fa::kStatic ? fwd_kernel_of<fa::kStatic>(causal, ragged) : fwd_kernel_of<fa::kDynamic>(causal, ragged);
}

// Runs once per device, with that device current.
void init_device(int dev) {
  DeviceState& st = g_dev[dev];
  cudaDeviceProp prop;
  cudaError_t e = cudaGetDeviceProperties(&prop, dev);
  if (e != cudaSuccess) { st.init_error = static_cast<int>(e); return; }
  if (prop.major != 10) { st.init_error = FA_B200_ERR_ARCH; return; }
  // The kernel moves registers between its warpgroups with setmaxnreg; that only works (and
  // otherwise blocks for ever) if the compiler gave the kernel the launch allocation the budget
  // in fa_fwd_sm100.cuh assumes.  Refuse to launch a build where it did not.
  const void* variants[11];
  {
    int i = 0;
    for (int schedule : {fa::kOneItem, fa::kStatic, fa::kDynamic})
      for (int mask : {0, 1, 2}) variants[i++] = reinterpret_cast<const void*>(fwd_kernel(schedule, mask == 2, mask == 1));
    for (int schedule : {fa::kOneItem, fa::kDynamic}) variants[i++] = reinterpret_cast<const void*>(fwd_kernel(schedule, true, false, true));
  }
  for (const void* fn : variants) {
    cudaFuncAttributes fattr;
    e = cudaFuncGetAttributes(&fattr, fn);
    if (e != cudaSuccess) { st.init_error = static_cast<int>(e); return; }
    if (fattr.numRegs != fa::kLaunchRegs) { st.init_error = FA_B200_ERR_BUILD; return; }
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, fa::kSmemBytes);
    if (e != cudaSuccess) { st.init_error = static_cast<int>(e); return; }
    // Two CTAs of ~100 KB each must fit: ask for the largest shared-memory carveout.
    e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                             cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) { st.init_error = static_cast<int>(e); return; }
    // Two CTAs per SM each allocate half of tensor memory; a third resident CTA would block in
    // tcgen05.alloc until one of them exits.  Shared memory already limits residency to two; make
    // sure of it (a build with a much smaller footprint would break that assumption).
    int resident = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, fn, fa::kNumThreads, fa::kSmemBytes);
    if (e != cudaSuccess) { st.init_error = static_cast<int>(e); return; }
    if (resident < 1 || resident > fa::kCtasPerSm) { st.init_error = FA_B200_ERR_BUILD; return; }
  }
  // The persistent grid is sized for kCtasPerSm per SM whatever the occupancy query answered: it
  // has been seen to answer 1 where the hardware co-schedules 2, and a CTA that has to wait for
  // a slot only starts later -- work items are partitioned by grid stride, no CTA waits on another.
  st.resident_ctas = fa::kCtasPerSm * prop.multiProcessorCount;
  st.sm_count = prop.multiProcessorCount;
  for (const void* fn : {reinterpret_cast<const void*>(&fa::fa_decode_kernel<128, 7, true>),
                         reinterpret_cast<const void*>(&fa::fa_decode_kernel<256, 4, true>),
                         reinterpret_cast<const void*>(&fa::fa_decode_kernel<512, 2, true>)}) {
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) { st.init_error = static_cast<int>(e); return; }
  }
  void* addr = nullptr;
  e = cudaGetSymbolAddress(&addr, g_fa_status);
  if (e != cudaSuccess) { st.init_error = static_cast<int>(e); return; }
  st.status = static_cast<unsigned int*>(addr);
  e = cudaMemset(st.status, 0, 4 * sizeof(unsigned int));
  if (e != cudaSuccess) { st.init_error = static_cast<int>(e); return; }
}

bool stride_ok(const int64_t s[3]) {
  for (int i = 0; i < 3; ++i)
    if (s[i] <= 0 || (s[i] % 8) != 0) return false;
  return true;
}

int encode_map_uncached(CUtensorMap* map, const void* base, const fa_b200_params* p,
                        const int64_t st[3], unsigned box_rows) {
  // dims, innermost first: d, N, H, B.  Strides (bytes) for dims 1..3: row, head, batch.
  const cuuint64_t dims[4] = {static_cast<cuuint64_t>(p->d), static_cast<cuuint64_t>(p->N),
                              static_cast<cuuint64_t>(p->H), static_cast<cuuint64_t>(p->B)};
  const cuuint64_t strides[3] = {static_cast<cuuint64_t>(st[2]) * 2, static_cast<cuuint64_t>(st[1]) * 2,
                                 static_cast<cuuint64_t>(st[0]) * 2};
  const cuuint32_t box[4] = {fa::kHeadDim, box_rows, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : FA_B200_ERR_TENSORMAP;
}

// A tensor map is a pure function of (base, shape, strides, box): the driver call that encodes
// one costs about a microsecond, four of them per launch are a visible share of a small problem's
// launch path, and callers (a model's layers, a benchmark loop) present the same few buffers
// again and again.  Each host thread keeps a small direct-mapped cache of encoded maps; a hit
// needs no lock and can never be stale, because nothing outside the key enters the encoding.
struct MapKey {
  const void* base;
  int32_t B, H, N, box_rows;
  int64_t st[3];
  bool operator==(const MapKey& o) const {
    return base == o.base && B == o.B && H == o.H && N == o.N && box_rows == o.box_rows &&
           st[0] == o.st[0] && st[1] == o.st[1] && st[2] == o.st[2];
  }
};
struct MapSlot {
  MapKey key;
  bool valid = false;
  alignas(64) CUtensorMap map;
};
constexpr int kMapCacheSlots = 64;

int encode_map(CUtensorMap* map, const void* base, const fa_b200_params* p, const int64_t st[3],
               unsigned box_rows = fa::kBlockN) {
  static thread_local MapSlot cache[kMapCacheSlots];
  const MapKey key{base, p->B, p->H, p->N, static_cast<int32_t>(box_rows), {st[0], st[1], st[2]}};
  uint64_t h = reinterpret_cast<uintptr_t>(base) >> 4;
  h ^= (static_cast<uint64_t>(p->N) * 0x9E3779B97F4A7C15ull) ^ (static_cast<uint64_t>(st[2]) << 17) ^
       (static_cast<uint64_t>(box_rows) << 7) ^ (static_cast<uint64_t>(p->B) << 40) ^
       (static_cast<uint64_t>(p->H) << 52);
  h ^= h >> 29;
  MapSlot& slot = cache[(h * 0xBF58476D1CE4E5B9ull) >> 58];
  if (slot.valid && slot.key == key) {
    *map = slot.map;
    return 0;
  }
  const int rc = encode_map_uncached(&slot.map, base, p, st, box_rows);
  slot.valid = rc == 0;
  if (rc != 0) return rc;
  slot.key = key;
  *map = slot.map;
  return 0;
}

// What the next node captured on a stream depends on, where that is one node of one capture.
struct Captured {
  unsigned long long id = 0;      // of the capture: unique in the process
  cudaGraphNode_t node = nullptr;
};
Captured captured_last(cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  const cudaGraphNode_t* deps = nullptr;
  const cudaGraphEdgeData* edges = nullptr;
  size_t count = 0;
  Captured c;
  if (cudaStreamGetCaptureInfo_v3(stream, &status, &id, nullptr, &deps, &edges, &count) != cudaSuccess) {
    cudaGetLastError();
  } else if (status == cudaStreamCaptureStatusActive && count == 1) {
    c.id = id;
    c.node = deps[0];
  }
  return c;
}
thread_local Captured g_ours;     // the node of this thread's last launch, where it was captured

// Launch with programmatic dependent launch (the kernels wait for the previous one before their first
// access to global memory, see pdl_wait): back-to-back launches overlap the start-up of one with the
// end of the other.  On a stream that is for every launch (a prompt of 72 tokens, GPT-2 small: 540 us,
// 654 without).  In a graph it is for launches behind a kernel of this library: behind one that says
// nothing to its dependents, a GEMM, such an edge only costs (a replayed prefill, GPT-2 medium 4 x 111:
// 1153 us with them everywhere, 1142 without; GPT-2 small 4 x 67: 487, 482).
// `cluster` > 1: clusters of that many CTAs along x.
template <class... Params, class... Args>
cudaError_t launch_kernel(void (*kernel)(Params...), dim3 grid, unsigned block, size_t smem, cudaStream_t stream,
                          unsigned cluster, const Args&... args) {
  bool capturing = false, dependent = true;
  if (stream != nullptr) {                         // (the legacy default stream cannot be captured)
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) cudaGetLastError();
    capturing = status == cudaStreamCaptureStatusActive;
  }
  if (capturing) {
    const Captured before = captured_last(stream);
    dependent = before.node != nullptr && before.id == g_ours.id && before.node == g_ours.node;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = dependent ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  const cudaError_t last = cudaGetLastError();     // (clears the sticky copy)
  if (capturing) g_ours = captured_last(stream);
  return e != cudaSuccess ? e : last;
}

// How one forward call is scheduled (the rule behind fa_b200_fwd and fa_b200_fwd_plan).
constexpr long long kOrderBytes = 32ll << 20;   // K and V of the heads that are ordered together (16, 64 MB: equal)
struct FwdPlan {
  int schedule;        // fa::Schedule
  int n_qtiles, kv_tiles;
  long long items;     // B * H * n_qtiles
  unsigned grid;       // launched
  bool early;          // let the next kernel of the stream start while this one runs
};

FwdPlan plan_fwd(const fa_b200_params* p, const DeviceState& st) {
  FwdPlan pl;
  pl.n_qtiles = (p->N + fa::kBlockM - 1) / fa::kBlockM;
  pl.kv_tiles = (p->N + fa::kBlockN - 1) / fa::kBlockN;
  pl.items = static_cast<long long>(p->B) * p->H * pl.n_qtiles;
  const long long slots = st.resident_ctas;
  // Measured on B200 (296 slots), N = 64 .. 16384, 12 .. 800 heads:
  // * No more items than slots, or a third more: one CTA per item.  Nobody has much to take over, and
  //   asking costs 0.4 us (B=4 H=12 N=1024, 384 items: 13.9 us, static 15.4, dynamic 15.7).
  // * Items of up to 4 K/V tiles that make less than two rounds, or of one: static.  (B=8 H=16 N=300,
  //   384 items: 8.5 us, dynamic 9.0, one item 10.3; B=4 H=25 N=512 non-causal: 14.1 against 16.0: who
  //   takes over an item does not know who else is on the SM.)
  //   Two K/V tiles up to 2.7 rounds: static / dynamic at 2.0 rounds N=130 causal 8.9 / 9.4 us, N=200 9.0 / 9.4, full 11.6-11.8 /
  //   11.7-11.8; at 2.07 10.0 / 11.9, 10.3 / 11.9, 13.0 / 14.2-15.0; at 2.2 10.0 / 11.9, 10.4 / 12.2, 13.1 / 15.1; at 2.6 N=200 10.8 /
  //   12.5 and 15.2 / 15.3; but at 3.0 12.8 / 12.5 and 17.8 / 15.9.
  // * Otherwise dynamic (B=32 H=25 N=777: 139 us, static 170, one item 191), except
  //   - non-causal sequences above 3072: one CTA per item, whose tile loop is the smallest code
  //     (B=4 H=25 N=8192: 1.94 ms, dynamic 2.12);
  //   - more items per slot than the item table holds: one CTA per item.
  const bool causal = p->causal != 0;
  pl.schedule = fa::kOneItem;
  if (pl.items > slots * fa::kItemTable) {
  } else if (pl.kv_tiles == 1 || (pl.kv_tiles <= 4 && pl.items < 2 * slots) ||
             (pl.kv_tiles == 2 && 11 * pl.items <= 30 * slots)) {
    if (pl.items > slots) pl.schedule = fa::kStatic;
  } else if (3 * pl.items >= 4 * slots && (causal || pl.kv_tiles <= 24)) {
    pl.schedule = fa::kDynamic;
  }
  pl.grid = static_cast<unsigned>(pl.schedule == fa::kStatic ? slots : pl.items);
  // The next kernel's CTAs are placed when this one says so, around the slots that it holds: where it leaves
  // SMs free, some get two of them and others none, and two share an SM's pipes.  Back to back, early / at the
  // end / a kernel without either (us): N = 8192 full, 64 items 84.3 / 67.2 / 69.8; N = 2048 causal, 256 items
  // 25.7 / 21.6 / 24.7; N = 1300 causal, 385 items 19.1 / 17.7 / 27.0.  So early only
  // - for single tiles, whose time is their start-up (N = 72, 290 items: 5.2 / 5.5 / 8.3), and for up to a quarter
  //   of the SMs, where nobody has to share (N = 512 causal, 12 items 7.4 / 7.6 / 11.6; but N = 1300 full, 44 items
  //   17.4 / 14.8 / 16.5);
  // - where others wait for slots anyway: dynamic; full with more items than SMs (N = 512, 256 items: 9.6 /
  //   10.6 / 12.4); causal with a second wave, as long as it is long enough for its tiles (N = 1024, 384 items
  //   14.4 / 15.2 / 20.6, but 328 items 14.3 / 13.4; N = 640, 330 items 10.5 / 11.3 / 16.5).
  pl.early = pl.kv_tiles == 1 || 4 * pl.items <= st.sm_count || pl.schedule == fa::kDynamic ||
             (causal ? pl.kv_tiles <= 8 && pl.items >= slots + 16 * (pl.kv_tiles - 3) : pl.items > st.sm_count);
#ifdef FA_WAIT_TEST    // the test's problem, one causal head of two tiles, as one CTA: what waits for what is then known
  if (causal && p->B * p->H == 1 && pl.n_qtiles == 2) {
    pl.schedule = fa::kStatic;
    pl.grid = 1;
  }
#endif
  return pl;
}

// Device guard + per-device set-up shared by the forward entry points.
int ready_device(int device, DeviceState** out) {
  DeviceState& st = g_dev[device];
  std::call_once(st.once, init_device, device);
  if (st.init_error) return st.init_error;
  *out = &st;
  return 0;
}

}  // namespace

extern "C" {

int fa_b200_abi_version(void) { return FA_B200_ABI_VERSION; }

int fa_b200_validate(const fa_b200_params* p) {
  if (p == nullptr || p->q == nullptr || p->k == nullptr || p->v == nullptr || p->o == nullptr)
    return FA_B200_ERR_NULL;
  if (p->d != fa::kHeadDim) return FA_B200_ERR_HEAD_DIM;
  if (p->B < 0 || p->H < 0 || p->N < 0) return FA_B200_ERR_SHAPE;
  if (p->N > (1 << 24)) return FA_B200_ERR_SHAPE;
  {
    const long long ctas = static_cast<long long>(p->B) * p->H * ((p->N + 127) / 128);
    if (ctas > 0x7fffffffLL) return FA_B200_ERR_SHAPE;
  }
  if (!stride_ok(p->q_strides) || !stride_ok(p->k_strides) || !stride_ok(p->v_strides) ||
      !stride_ok(p->o_strides))
    return FA_B200_ERR_STRIDE;
  const uintptr_t ptrs[4] = {reinterpret_cast<uintptr_t>(p->q), reinterpret_cast<uintptr_t>(p->k),
                             reinterpret_cast<uintptr_t>(p->v), reinterpret_cast<uintptr_t>(p->o)};
  for (uintptr_t a : ptrs)
    if (a & 15u) return FA_B200_ERR_ALIGN;
  if (p->lse != nullptr && (reinterpret_cast<uintptr_t>(p->lse) & 3u)) return FA_B200_ERR_ALIGN;
  if (!(p->softmax_scale >= 0.0f) || std::isinf(p->softmax_scale)) return FA_B200_ERR_SCALE;
  if (p->device < 0 || p->device >= kMaxDevices) return FA_B200_ERR_DEVICE;
  return FA_B200_OK;
}

int fa_b200_fwd(const fa_b200_params* p) {
  int rc = fa_b200_validate(p);
  if (rc != FA_B200_OK) return rc;
  if (p->B == 0 || p->H == 0 || p->N == 0) return FA_B200_OK;  // nothing to compute

  DeviceGuard guard(p->device);
  if (guard.error) return guard.error;
  DeviceState* stp = nullptr;
  if ((rc = ready_device(p->device, &stp)) != 0) return rc;
  const DeviceState& st = *stp;
  std::call_once(g_encode_once, resolve_encode);
  if (g_encode == nullptr) return FA_B200_ERR_DRIVER;

  CUtensorMap mq, mk, mv, mo;
  if ((rc = encode_map(&mq, p->q, p, p->q_strides)) != 0) return rc;
  if ((rc = encode_map(&mk, p->k, p, p->k_strides)) != 0) return rc;
  if ((rc = encode_map(&mv, p->v, p, p->v_strides)) != 0) return rc;
  if ((rc = encode_map(&mo, p->o, p, p->o_strides, 32)) != 0) return rc;   // one 32-row slab per warp

  const FwdPlan pl = plan_fwd(p, st);
  fa::FwdParams kp;
  kp.lse = p->lse;
  kp.B = p->B;
  kp.H = p->H;
  kp.N = p->N;
  kp.n_qtiles = pl.n_qtiles;
  kp.div_qtiles = fa::make_fast_div(static_cast<uint32_t>(kp.n_qtiles));
  kp.div_heads = fa::make_fast_div(static_cast<uint32_t>(p->H));
  kp.causal = p->causal ? 1 : 0;
  const float scale = p->softmax_scale > 0.0f ? p->softmax_scale : 1.0f / std::sqrt(static_cast<float>(p->d));
  kp.scale_log2 = scale * 1.4426950408889634f;
  kp.status = st.status;
  kp.n_items = static_cast<int>(pl.items);
  kp.early = pl.early ? 1 : 0;
  const int first_wave = static_cast<int>(pl.items < st.resident_ctas ? pl.items : st.resident_ctas);
  kp.mirror_from = st.sm_count;
  kp.mirror_to = kp.causal ? first_wave : 0;
  // causal order: groups of heads whose K and V (N * 256 bytes each) stay in L2 while their tiles run
  const long long heads = static_cast<long long>(p->B) * p->H;
  long long fit = kOrderBytes / (static_cast<long long>(p->N) * 256);
  if (fit < 1) fit = 1;
  const long long groups = (heads + fit - 1) / fit;
  kp.group = static_cast<int>((heads + groups - 1) / groups);
  kp.group_items = kp.group * kp.n_qtiles;
  kp.last_group = static_cast<int>(heads - (heads - 1) / kp.group * kp.group);
  kp.div_group_items = fa::make_fast_div(static_cast<uint32_t>(kp.group_items));
  kp.div_group = fa::make_fast_div(static_cast<uint32_t>(kp.group));
  kp.div_last_group = fa::make_fast_div(static_cast<uint32_t>(kp.last_group));
  const cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  const bool ragged = (p->N % fa::kBlockN) != 0;   // non-causal only: the causal mask covers the columns past N
  const FwdKernel kernel = fwd_kernel(pl.schedule, kp.causal != 0, ragged, kp.causal != 0 && p->N >= kLongRows);
  return static_cast<int>(launch_kernel(kernel, dim3(pl.grid), fa::kNumThreads, fa::kSmemBytes, stream, 1, mq, mk, mv, mo, kp));
}

int fa_b200_fwd_plan(const fa_b200_params* p, int32_t* schedule, int32_t* grid) {
  int rc = fa_b200_validate(p);
  if (rc != FA_B200_OK) return rc;
  if (p->B == 0 || p->H == 0 || p->N == 0) {
    if (schedule != nullptr) *schedule = FA_B200_SCHEDULE_NONE;
    if (grid != nullptr) *grid = 0;
    return FA_B200_OK;
  }
  DeviceGuard guard(p->device);
  if (guard.error) return guard.error;
  DeviceState* stp = nullptr;
  if ((rc = ready_device(p->device, &stp)) != 0) return rc;
  const FwdPlan pl = plan_fwd(p, *stp);
  if (schedule != nullptr)
    *schedule = pl.schedule == fa::kOneItem  ? FA_B200_SCHEDULE_CTA_PER_TILE
                : pl.schedule == fa::kStatic ? FA_B200_SCHEDULE_STATIC
                                             : FA_B200_SCHEDULE_DYNAMIC;
  if (grid != nullptr) *grid = static_cast<int32_t>(pl.grid);
  return FA_B200_OK;
}

// ------------------------------------------------------------------------------------ decode
namespace {

// Bytes of workspace that callers of fa_b200_decode lend, by the rule of the kernels that needed one:
// chunks of a head's keys, 66 floats each.  Today's kernel merges inside a cluster and touches none of
// it; the sizes stay what callers have been told.
constexpr int kDecodeTargetCtas = 592, kDecodeTargetCtasLong = 2368;
constexpr int kDecodeLongLen = 2048;
constexpr int kDecodeChunkRows = 64, kDecodeChunkRowsLong = 512;   // rows per chunk, at least
int64_t decode_workspace(int B, int H, int kv_len, bool fine_for_long) {
  const long long heads = static_cast<long long>(B) * H;
  if (heads == 0 || (heads <= 296 && kv_len <= 4096)) return 0;
  const bool long_cache = fine_for_long && kv_len >= kDecodeLongLen;
  const long long min_rows = long_cache ? kDecodeChunkRowsLong : kDecodeChunkRows;
  long long want = ((long_cache ? kDecodeTargetCtasLong : kDecodeTargetCtas) + heads - 1) / heads;
  const long long most = (kv_len + min_rows - 1) / min_rows;
  want = want > most ? most : (want < 1 ? 1 : want);
  const long long rows = ((kv_len + want - 1) / want + 15) / 16 * 16;
  const long long chunks = (kv_len + rows - 1) / rows;
  return chunks == 1 ? 0 : heads * chunks * fa::kDecodePartial * static_cast<int64_t>(sizeof(float));
}

// How a problem is launched: CTAs per head (a cluster) and their threads.  As many CTAs as are resident
// at seven per SM, the cluster a power of two, no CTA with less than kDecodeMinRows rows; where clusters
// of 16 still leave the chip half empty and a CTA has more rows than it loads at once (threads / 2),
// larger CTAs.  (H = 12, B=1 kv 8192: 12.1 us with 128 threads, 7.5 with 512; H = 25: 14.8, 11.8 with
// 256; from 48 heads on nothing.)
struct DecodeShape {
  int cluster, threads;
};
DecodeShape decode_shape(long long heads, int kv_len, int sm_count) {
  DecodeShape s{1, 128};
  const long long slots = 7LL * sm_count;
  while (s.cluster < fa::kDecodeClusterMax && heads * s.cluster * 2 <= slots && kv_len >= s.cluster * 2 * fa::kDecodeMinRows)
    s.cluster *= 2;
  if (s.cluster == fa::kDecodeClusterMax)
    while (s.threads < 512 && heads * s.cluster * s.threads * 2 <= slots * 128 && kv_len > s.cluster * s.threads / 2)
      s.threads *= 2;
  return s;
}

bool stride_ok_n(const int64_t* s, int n) {
  for (int i = 0; i < n; ++i)
    if (s[i] <= 0 || (s[i] % 8) != 0) return false;
  return true;
}

int decode_validate(const fa_b200_decode_params* p) {
  if (p == nullptr || p->q == nullptr || p->k_cache == nullptr || p->v_cache == nullptr ||
      p->o == nullptr)
    return FA_B200_ERR_NULL;
  if (p->d != fa::kHeadDim) return FA_B200_ERR_HEAD_DIM;
  if (p->B < 0 || p->H < 0 || p->kv_len < 1) return FA_B200_ERR_SHAPE;
  if (static_cast<long long>(p->B) * p->H > 0x7fffffffLL / 64) return FA_B200_ERR_SHAPE;
  if (!stride_ok_n(p->q_strides, 2) || !stride_ok_n(p->o_strides, 2) || !stride_ok_n(p->k_strides, 3) ||
      !stride_ok_n(p->v_strides, 3))
    return FA_B200_ERR_STRIDE;
  const uintptr_t ptrs[4] = {reinterpret_cast<uintptr_t>(p->q), reinterpret_cast<uintptr_t>(p->k_cache),
                             reinterpret_cast<uintptr_t>(p->v_cache), reinterpret_cast<uintptr_t>(p->o)};
  for (uintptr_t a : ptrs)
    if (a & 15u) return FA_B200_ERR_ALIGN;
  if (p->lse != nullptr && (reinterpret_cast<uintptr_t>(p->lse) & 3u)) return FA_B200_ERR_ALIGN;
  if (p->kv_len_device != nullptr && (reinterpret_cast<uintptr_t>(p->kv_len_device) & 3u)) return FA_B200_ERR_ALIGN;
  if ((p->k_new == nullptr) != (p->v_new == nullptr)) return FA_B200_ERR_NULL;
  if (p->k_new != nullptr) {
    if (!stride_ok_n(p->new_strides, 2)) return FA_B200_ERR_STRIDE;
    if ((reinterpret_cast<uintptr_t>(p->k_new) & 15u) || (reinterpret_cast<uintptr_t>(p->v_new) & 15u))
      return FA_B200_ERR_ALIGN;
  }
  if (!(p->softmax_scale >= 0.0f) || std::isinf(p->softmax_scale)) return FA_B200_ERR_SCALE;
  if (p->device < 0 || p->device >= kMaxDevices) return FA_B200_ERR_DEVICE;
  return FA_B200_OK;
}

}  // namespace

int64_t fa_b200_decode_workspace_bytes(int32_t B, int32_t H, int32_t kv_len) {
  if (B < 0 || H < 0 || kv_len < 1) return FA_B200_ERR_SHAPE;
  if (B == 0 || H == 0) return 0;
  return decode_workspace(B, H, kv_len, /*fine_for_long=*/true);
}

extern "C++" {
namespace {

template <int kThreads, int kCtasPerSm>
cudaError_t decode_launch_cluster(const fa::DecodeParams& kp, unsigned heads, int cluster, cudaStream_t stream) {
  return launch_kernel(&fa::fa_decode_kernel<kThreads, kCtasPerSm, true>, dim3(heads * static_cast<unsigned>(cluster)),
                       kThreads, 0, stream, static_cast<unsigned>(cluster), kp);
}

// The launch shared by the decode entry points.  `p` has been validated.
int decode_launch(const fa_b200_decode_params* p) {
  if (p->B == 0 || p->H == 0) return FA_B200_OK;
  DeviceGuard guard(p->device);
  if (guard.error) return guard.error;
  DeviceState* stp = nullptr;
  const int rc = ready_device(p->device, &stp);
  if (rc != 0) return rc;
  fa::DecodeParams kp;
  kp.q = static_cast<const __nv_bfloat16*>(p->q);
  kp.k = static_cast<const __nv_bfloat16*>(p->k_cache);
  kp.v = static_cast<const __nv_bfloat16*>(p->v_cache);
  kp.o = static_cast<__nv_bfloat16*>(p->o);
  kp.lse = p->lse;
  kp.q_sb = p->q_strides[0]; kp.q_sh = p->q_strides[1];
  kp.o_sb = p->o_strides[0]; kp.o_sh = p->o_strides[1];
  kp.k_sb = p->k_strides[0]; kp.k_sh = p->k_strides[1]; kp.k_sn = p->k_strides[2];
  kp.v_sb = p->v_strides[0]; kp.v_sh = p->v_strides[1]; kp.v_sn = p->v_strides[2];
  kp.B = p->B; kp.H = p->H; kp.kv_len = p->kv_len;
  kp.kv_len_ptr = p->kv_len_device;
  kp.k_new = static_cast<const __nv_bfloat16*>(p->k_new);
  kp.v_new = static_cast<const __nv_bfloat16*>(p->v_new);
  kp.new_sb = p->new_strides[0]; kp.new_sh = p->new_strides[1];
  const float scale = p->softmax_scale > 0.0f ? p->softmax_scale : 1.0f / std::sqrt(static_cast<float>(p->d));
  kp.scale_log2 = scale * 1.4426950408889634f;

  const cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  const unsigned heads = static_cast<unsigned>(p->B * p->H);
  const DecodeShape shape = decode_shape(heads, p->kv_len, stp->sm_count);
  kp.cluster_log2 = 0;
  while ((1 << kp.cluster_log2) < shape.cluster) ++kp.cluster_log2;
  if (shape.cluster == 1)
    return static_cast<int>(launch_kernel(&fa::fa_decode_kernel<128, 7, false>, dim3(heads), 128, 0, stream, 1, kp));
  return static_cast<int>(shape.threads == 128   ? decode_launch_cluster<128, 7>(kp, heads, shape.cluster, stream)
                          : shape.threads == 256 ? decode_launch_cluster<256, 4>(kp, heads, shape.cluster, stream)
                                                 : decode_launch_cluster<512, 2>(kp, heads, shape.cluster, stream));
}

}  // namespace
}  // extern "C++"

int fa_b200_decode(const fa_b200_decode_params* p) {
  const int rc = decode_validate(p);
  if (rc != FA_B200_OK) return rc;
  const int64_t need = decode_workspace(p->B, p->H, p->kv_len, /*fine_for_long=*/true);
  if (need > 0 && (p->workspace == nullptr || p->workspace_bytes < need ||
                   (reinterpret_cast<uintptr_t>(p->workspace) & 15u)))
    return FA_B200_ERR_WORKSPACE;
  return decode_launch(p);
}

int fa_b200_decode_direct(const fa_b200_decode_params* p) {
  const int rc = decode_validate(p);
  return rc != FA_B200_OK ? rc : decode_launch(p);
}

int fa_b200_decode_static(const fa_b200_decode_params* p) {
  const int rc = decode_validate(p);
  if (rc != FA_B200_OK) return rc;
  if (decode_workspace(p->B, p->H, p->kv_len, /*fine_for_long=*/false) > static_cast<int64_t>(FA_B200_STATIC_SCRATCH_BYTES))
    return FA_B200_ERR_STATIC_SCRATCH;
  return decode_launch(p);
}

int fa_b200_device_ok(int device) {
  if (device < 0) return FA_B200_ERR_DEVICE;
  int count = 0;
  cudaError_t e = cudaGetDeviceCount(&count);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (device >= count) return FA_B200_ERR_DEVICE;
  int major = 0;
  e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device);
  if (e != cudaSuccess) return static_cast<int>(e);
  return major == 10 ? 1 : 0;
}

int fa_b200_last_status(int device, void* stream) {
  if (device < 0 || device >= kMaxDevices) return FA_B200_ERR_DEVICE;
  DeviceGuard guard(device);
  if (guard.error) return guard.error;
  cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return static_cast<int>(e);
  DeviceState& st = g_dev[device];
  if (st.status == nullptr) return 0;  // no kernel was ever launched on this device
  unsigned int words[4] = {0, 0, 0, 0};
  e = cudaMemcpy(words, st.status, sizeof(words), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (words[0] != 0) {
    std::fprintf(stderr, "fa_b200: watchdog code 0x%x (block %u, thread %u, parity %u)\n", words[0],
                 words[1], words[2], words[3]);
    e = cudaMemset(st.status, 0, sizeof(words));
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  return static_cast<int>(words[0]);
}

// ------------------------------------------------------------------------- add + LayerNorm
extern "C++" {
namespace {

template <int kVec>
cudaError_t launch_add_ln(const fa::AddLnParams& kp, cudaStream_t stream, int sm_count) {
  const long long ctas = (kp.rows + fa::kLnWarpsPerCta - 1) / fa::kLnWarpsPerCta;
  // (from 6 vectors a lane on only where no SM has a third CTA to lose; see the kernel)
  auto kernel = &fa::fa_add_layernorm_kernel<kVec, true>;
  if constexpr (kVec > 5)
    if (ctas > 2 * sm_count) kernel = &fa::fa_add_layernorm_kernel<kVec, false>;
  return launch_kernel(kernel, dim3(static_cast<unsigned>(ctas)), fa::kLnWarpsPerCta * 32, 0, stream, 1, kp);
}

}  // namespace
}  // extern "C++"

int fa_b200_add_layernorm(const fa_b200_add_layernorm_params* p) {
  if (p == nullptr || p->a == nullptr || p->scale == nullptr || p->shift == nullptr ||
      p->norm_out == nullptr)
    return FA_B200_ERR_NULL;
  if (p->rows < 0 || p->cols <= 0 || (p->cols % 8) != 0 ||
      p->cols > fa::kLnMaxVecPerLane * 256)
    return FA_B200_ERR_SHAPE;
  if ((p->rows + fa::kLnWarpsPerCta - 1) / fa::kLnWarpsPerCta > 0x7fffffffLL) return FA_B200_ERR_SHAPE;
  const void* ptrs[6] = {p->a, p->resid, p->scale, p->shift, p->sum_out, p->norm_out};
  for (const void* q : ptrs)
    if (reinterpret_cast<uintptr_t>(q) & 15u) return FA_B200_ERR_ALIGN;
  if (!(p->eps >= 0.0f)) return FA_B200_ERR_SCALE;
  if (p->device < 0 || p->device >= kMaxDevices) return FA_B200_ERR_DEVICE;
  if (p->rows == 0) return FA_B200_OK;

  DeviceGuard guard(p->device);
  if (guard.error) return guard.error;
  DeviceState& st = g_dev[p->device];
  std::call_once(st.once, init_device, p->device);
  if (st.init_error) return st.init_error;

  fa::AddLnParams kp;
  kp.a = static_cast<const __nv_bfloat16*>(p->a);
  kp.resid = static_cast<const __nv_bfloat16*>(p->resid);
  kp.scale = static_cast<const __nv_bfloat16*>(p->scale);
  kp.shift = static_cast<const __nv_bfloat16*>(p->shift);
  kp.sum_out = static_cast<__nv_bfloat16*>(p->sum_out);
  kp.norm_out = static_cast<__nv_bfloat16*>(p->norm_out);
  kp.rows = p->rows;
  kp.cols = p->cols;
  kp.eps = p->eps;
  const cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  cudaError_t e;
  switch ((p->cols + 255) / 256) {   // 16-byte vectors per lane
    case 1: e = launch_add_ln<1>(kp, stream, st.sm_count); break;
    case 2: e = launch_add_ln<2>(kp, stream, st.sm_count); break;
    case 3: e = launch_add_ln<3>(kp, stream, st.sm_count); break;
    case 4: e = launch_add_ln<4>(kp, stream, st.sm_count); break;
    case 5: e = launch_add_ln<5>(kp, stream, st.sm_count); break;
    case 6: e = launch_add_ln<6>(kp, stream, st.sm_count); break;
    case 7: e = launch_add_ln<7>(kp, stream, st.sm_count); break;
    default: e = launch_add_ln<8>(kp, stream, st.sm_count); break;
  }
  return static_cast<int>(e);
}

// ------------------------------------------------------------------------------ cache write
int fa_b200_cache_write(const fa_b200_cache_write_params* p) {
  if (p == nullptr || p->k == nullptr || p->v == nullptr || p->k_cache == nullptr || p->v_cache == nullptr)
    return FA_B200_ERR_NULL;
  if (p->B < 0 || p->N < 0 || p->H < 0) return FA_B200_ERR_SHAPE;
  if (!stride_ok(p->strides) || !stride_ok(p->cache_strides)) return FA_B200_ERR_STRIDE;
  if ((reinterpret_cast<uintptr_t>(p->k) | reinterpret_cast<uintptr_t>(p->v) | reinterpret_cast<uintptr_t>(p->k_cache) |
       reinterpret_cast<uintptr_t>(p->v_cache)) & 15u)
    return FA_B200_ERR_ALIGN;
  if (p->device < 0 || p->device >= kMaxDevices) return FA_B200_ERR_DEVICE;
  fa::CacheWriteParams kp;
  kp.total = 8LL * p->B * p->N * p->H;
  if (kp.total == 0) return FA_B200_OK;
  const long long ctas = (kp.total + fa::kCacheWriteThreads - 1) / fa::kCacheWriteThreads;
  if (ctas > 0x7fffffffLL) return FA_B200_ERR_SHAPE;
  DeviceGuard guard(p->device);
  if (guard.error) return guard.error;
  DeviceState* stp = nullptr;
  const int rc = ready_device(p->device, &stp);
  if (rc != 0) return rc;
  kp.k = static_cast<const __nv_bfloat16*>(p->k);
  kp.v = static_cast<const __nv_bfloat16*>(p->v);
  kp.k_cache = static_cast<__nv_bfloat16*>(p->k_cache);
  kp.v_cache = static_cast<__nv_bfloat16*>(p->v_cache);
  kp.s_b = p->strides[0]; kp.s_n = p->strides[1]; kp.s_h = p->strides[2];
  kp.c_b = p->cache_strides[0]; kp.c_n = p->cache_strides[1]; kp.c_h = p->cache_strides[2];
  kp.N = p->N;
  kp.H = p->H;
  return static_cast<int>(launch_kernel(&fa::fa_cache_write_kernel, dim3(static_cast<unsigned>(ctas)),
                                        fa::kCacheWriteThreads, 0, static_cast<cudaStream_t>(p->stream), 1, kp));
}

// ------------------------------------------------------------------- Linear for a few rows
extern "C++" {
namespace {

constexpr int kLinSmemLimit = 128 * 1024;
std::once_flag g_lin_once[kMaxDevices];
int g_lin_error[kMaxDevices];

template <int kRows>
cudaError_t lin_prepare() {
  cudaError_t e = cudaFuncSetAttribute(
      reinterpret_cast<const void*>(&fa::fa_linear_small_kernel<kRows, fa::kLinUnrollShort>),
      cudaFuncAttributeMaxDynamicSharedMemorySize, kLinSmemLimit);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(
      reinterpret_cast<const void*>(&fa::fa_linear_small_kernel<kRows, fa::kLinUnrollLong>),
      cudaFuncAttributeMaxDynamicSharedMemorySize, kLinSmemLimit);
}
void lin_init(int dev) {   // with `dev` current
  cudaError_t e = lin_prepare<1>();
  if (e == cudaSuccess) e = lin_prepare<2>();
  if (e == cudaSuccess) e = lin_prepare<4>();
  if (e == cudaSuccess) e = lin_prepare<8>();
  g_lin_error[dev] = static_cast<int>(e);
}
template <int kRows>
cudaError_t lin_launch(const fa::LinearSmallParams& kp, cudaStream_t stream, int sm_count) {
  const size_t smem = static_cast<size_t>(kRows) * kp.K * 2;
  // as many CTAs per SM as ~200 KB of shared memory hold (1..8): every CTA stages x once
  long long per_sm = (200 * 1024) / static_cast<long long>(smem > 0 ? smem : 1);
  per_sm = per_sm < 1 ? 1 : (per_sm > 8 ? 8 : per_sm);
  long long ctas = (kp.N + fa::kLinWarps - 1) / fa::kLinWarps;
  if (ctas > per_sm * sm_count) ctas = per_sm * sm_count;
  // more loads in flight per lane pay for long rows and for many columns per warp (measured:
  // the vocabulary head 31 -> 28 us, K = 6400 9.2 -> 8.2 us; the short layers are better with 4)
  if (kp.K > 2048 || kp.N >= 16384)
    fa::fa_linear_small_kernel<kRows, fa::kLinUnrollLong><<<static_cast<unsigned>(ctas), fa::kLinWarps * 32, smem, stream>>>(kp);
  else
    fa::fa_linear_small_kernel<kRows, fa::kLinUnrollShort><<<static_cast<unsigned>(ctas), fa::kLinWarps * 32, smem, stream>>>(kp);
  return cudaGetLastError();
}

}  // namespace
}  // extern "C++"

int fa_b200_linear_small(const fa_b200_linear_small_params* p) {
  if (p == nullptr || p->x == nullptr || p->w == nullptr || p->y == nullptr) return FA_B200_ERR_NULL;
  if (p->M < 1 || p->M > fa::kLinMaxRows || p->N < 0 || p->K <= 0 || (p->K % 8) != 0)
    return FA_B200_ERR_SHAPE;
  const int rows = p->M <= 1 ? 1 : (p->M <= 2 ? 2 : (p->M <= 4 ? 4 : 8));
  if (static_cast<long long>(rows) * p->K * 2 > kLinSmemLimit) return FA_B200_ERR_SHAPE;
  if (p->act != 0 && p->act != 1) return FA_B200_ERR_SHAPE;
  if (p->ldw < p->K || (p->ldw % 8) != 0) return FA_B200_ERR_STRIDE;
  if ((reinterpret_cast<uintptr_t>(p->x) & 15u) || (reinterpret_cast<uintptr_t>(p->w) & 15u) ||
      (reinterpret_cast<uintptr_t>(p->y) & 15u) || (reinterpret_cast<uintptr_t>(p->bias) & 1u))
    return FA_B200_ERR_ALIGN;
  const bool prologue = p->resid != nullptr || p->ln_scale != nullptr || p->sum_out != nullptr;
  if (prologue) {
    if ((p->ln_scale == nullptr) != (p->ln_shift == nullptr)) return FA_B200_ERR_NULL;
    if (p->K > 256 * 8) return FA_B200_ERR_SHAPE;
    const void* extra[4] = {p->resid, p->ln_scale, p->ln_shift, p->sum_out};
    for (const void* q : extra)
      if (reinterpret_cast<uintptr_t>(q) & 15u) return FA_B200_ERR_ALIGN;
    if (p->sum_out != nullptr && (p->sum_out == p->x || p->sum_out == p->resid)) return FA_B200_ERR_ALIAS;
    if (p->ln_scale != nullptr && !(p->eps >= 0.0f)) return FA_B200_ERR_SCALE;
  }
  if (p->device < 0 || p->device >= kMaxDevices) return FA_B200_ERR_DEVICE;
  if (p->N == 0) return FA_B200_OK;

  DeviceGuard guard(p->device);
  if (guard.error) return guard.error;
  DeviceState& st = g_dev[p->device];
  std::call_once(st.once, init_device, p->device);
  if (st.init_error) return st.init_error;
  std::call_once(g_lin_once[p->device], lin_init, p->device);
  if (g_lin_error[p->device]) return g_lin_error[p->device];

  fa::LinearSmallParams kp;
  kp.x = static_cast<const __nv_bfloat16*>(p->x);
  kp.w = static_cast<const __nv_bfloat16*>(p->w);
  kp.bias = static_cast<const __nv_bfloat16*>(p->bias);
  kp.y = static_cast<__nv_bfloat16*>(p->y);
  kp.M = p->M; kp.N = p->N; kp.K = p->K;
  kp.ldw = p->ldw;
  kp.act = p->act;
  kp.resid = static_cast<const __nv_bfloat16*>(p->resid);
  kp.ln_scale = static_cast<const __nv_bfloat16*>(p->ln_scale);
  kp.ln_shift = static_cast<const __nv_bfloat16*>(p->ln_shift);
  kp.sum_out = static_cast<__nv_bfloat16*>(p->sum_out);
  kp.eps = p->eps;
  const cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  cudaError_t e;
  switch (rows) {
    case 1: e = lin_launch<1>(kp, stream, st.sm_count); break;
    case 2: e = lin_launch<2>(kp, stream, st.sm_count); break;
    case 4: e = lin_launch<4>(kp, stream, st.sm_count); break;
    default: e = lin_launch<8>(kp, stream, st.sm_count); break;
  }
  return static_cast<int>(e);
}

// ------------------------------------------------------------------------- generation step
namespace {

constexpr int kStepMaxGrid = 160;      // CTAs, one per SM
std::once_flag g_step_once[kMaxDevices];
int g_step_error[kMaxDevices];

void step_init(int dev) {   // with `dev` current
  cudaFuncAttributes attr;
  cudaError_t e = cudaFuncGetAttributes(&attr, reinterpret_cast<const void*>(&fa::fa_gpt_step_kernel));
  if (e != cudaSuccess) { g_step_error[dev] = static_cast<int>(e); return; }
  if (attr.numRegs != fa::kStepLaunchRegs) { g_step_error[dev] = FA_B200_ERR_BUILD; return; }
  e = cudaFuncSetAttribute(reinterpret_cast<const void*>(&fa::fa_gpt_step_kernel),
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, fa::kStepSmemBytes);
  g_step_error[dev] = static_cast<int>(e);
}

// Byte offsets of the workspace's parts, for `B` sequences of `H` heads.
struct StepWorkspace {
  int64_t best, arrived, x_att, x_mlp, qkv, ctx, h, part_ml, part_o, bytes;
  StepWorkspace(int B, int H) {
    // exchange words [8, C], from 4 KB boundaries: 757 us against 773 per GPT-2 XL step where they began anywhere
    const int64_t words = (8LL * 64 * H * 4 + 4095) / 4096 * 4096, pairs = static_cast<int64_t>(B) * H;
    const int64_t partials = pairs > kStepMaxGrid ? pairs : kStepMaxGrid;          // pairs * splits <= grid where split
    best = 128;                                                  // in front: generation, done
    arrived = best + 128;
    x_att = (arrived + fa::kStepMaxPairs * 4 + 4095) / 4096 * 4096;
    x_mlp = x_att + words;
    qkv = x_mlp + words;
    ctx = qkv + 3 * words;
    h = ctx + words;
    part_ml = h + 4 * words;
    part_o = part_ml + (partials * 8 + 127) / 128 * 128;
    bytes = part_o + partials * 64 * 4;
  }
};

bool step_shape_ok(int B, int H) {
  return B >= 1 && B <= fa::kStepMaxRows && H >= 1 && 64 * H <= fa::kStepMaxWidth && B * H <= 256;
}

}  // namespace

int64_t fa_b200_gpt_step_workspace_bytes(int32_t B, int32_t H) {
  if (!step_shape_ok(B, H)) return FA_B200_ERR_SHAPE;
  return StepWorkspace(B, H).bytes;
}

int fa_b200_gpt_step(const fa_b200_gpt_step_params* p) {
  if (p == nullptr || p->layers == nullptr || p->tok_emb == nullptr || p->pos_emb == nullptr ||
      p->lnf_scale == nullptr || p->lnf_shift == nullptr || p->head_w == nullptr || p->ids == nullptr ||
      p->k_cache == nullptr || p->v_cache == nullptr || p->logits == nullptr)
    return FA_B200_ERR_NULL;
  if (!step_shape_ok(p->B, p->H) || p->n_layers < 1 || p->n_layers > fa::kStepMaxLayers || p->vocab < 1 ||
      p->vocab >= fa::kStepMaxVocab ||
      p->cache_rows < 1 || p->n_positions < 1 || p->cache_rows > (1 << 22))
    return FA_B200_ERR_SHAPE;
  if (p->pos_device == nullptr && (p->pos < 0 || p->pos >= p->cache_rows || p->pos >= p->n_positions))
    return FA_B200_ERR_SHAPE;
  if (!stride_ok(p->cache_strides) || p->cache_strides[1] > 0x7fffffff || p->cache_strides[2] > 0x7fffffff)
    return FA_B200_ERR_STRIDE;
  const void* ptrs[7] = {p->tok_emb, p->pos_emb, p->lnf_scale, p->lnf_shift, p->head_w, p->layers, p->workspace};
  for (const void* q : ptrs)
    if (reinterpret_cast<uintptr_t>(q) & 15u) return FA_B200_ERR_ALIGN;
  for (int l = 0; l < p->n_layers; ++l) {
    if (p->k_cache[l] == nullptr || p->v_cache[l] == nullptr) return FA_B200_ERR_NULL;
    if ((reinterpret_cast<uintptr_t>(p->k_cache[l]) | reinterpret_cast<uintptr_t>(p->v_cache[l])) & 15u)
      return FA_B200_ERR_ALIGN;
  }
  if ((reinterpret_cast<uintptr_t>(p->ids) | reinterpret_cast<uintptr_t>(p->pos_device) |
       reinterpret_cast<uintptr_t>(p->next_ids)) & 7u)
    return FA_B200_ERR_ALIGN;
  if ((reinterpret_cast<uintptr_t>(p->length_device) & 3u) || (reinterpret_cast<uintptr_t>(p->logits) & 1u))
    return FA_B200_ERR_ALIGN;
  if (!(p->eps >= 0.0f)) return FA_B200_ERR_SCALE;
  if (p->device < 0 || p->device >= kMaxDevices) return FA_B200_ERR_DEVICE;
  const StepWorkspace ws(p->B, p->H);
  if (p->workspace == nullptr || p->workspace_bytes < ws.bytes) return FA_B200_ERR_WORKSPACE;

  DeviceGuard guard(p->device);
  if (guard.error) return guard.error;
  DeviceState* stp = nullptr;
  int rc = ready_device(p->device, &stp);
  if (rc != 0) return rc;
  std::call_once(g_step_once[p->device], step_init, p->device);
  if (g_step_error[p->device]) return g_step_error[p->device];

  fa::StepParams kp;
  static_assert(sizeof(fa::StepLayer) == sizeof(fa_b200_gpt_layer), "layer records are passed through");
  auto bf = [](const void* q) { return static_cast<const __nv_bfloat16*>(q); };
  kp.layers = reinterpret_cast<const fa::StepLayer*>(p->layers);
  kp.tok_emb = bf(p->tok_emb); kp.pos_emb = bf(p->pos_emb);
  kp.lnf_g = bf(p->lnf_scale); kp.lnf_b = bf(p->lnf_shift);
  kp.head_w = bf(p->head_w);
  kp.ids = reinterpret_cast<const long long*>(p->ids);
  kp.ids_stride = p->ids_stride;
  kp.pos_ptr = reinterpret_cast<long long*>(p->pos_device);
  kp.len_ptr = p->length_device;
  kp.pos = p->pos;
  kp.advance = p->advance;
  kp.n_layers = p->n_layers;
  kp.C = 64 * p->H; kp.H = p->H; kp.V = p->vocab; kp.M = p->B;
  const int columns = kp.C / fa::kStepUnit;                      // units; even
  kp.lg_chunks = columns > fa::kStepChunkUnits ? 1 : 0;
  kp.stage_units = columns >> kp.lg_chunks;
  kp.stage_pitch = fa::step_pitch(kp.stage_units);
  kp.batch_units = 4 * fa::kStepTake / kp.M;
  kp.inv_c = 1.0f / static_cast<float>(kp.C);
  kp.cache_rows = p->cache_rows;
  kp.n_positions = p->n_positions;
  kp.eps = p->eps;
  kp.scale_log2 = 0.125f * 1.4426950408889634f;                  // 1/sqrt(64) * log2(e)
  kp.c_sb = p->cache_strides[0];
  kp.c_sn = static_cast<int>(p->cache_strides[1]);
  kp.c_sh = static_cast<int>(p->cache_strides[2]);
  unsigned char* w = static_cast<unsigned char*>(p->workspace);
  kp.generation = reinterpret_cast<uint32_t*>(w);
  kp.done = reinterpret_cast<unsigned int*>(w) + 1;
  kp.best = reinterpret_cast<unsigned long long*>(w + ws.best);
  kp.arrived = reinterpret_cast<unsigned int*>(w + ws.arrived);
  kp.x_att = reinterpret_cast<uint32_t*>(w + ws.x_att);
  kp.x_mlp = reinterpret_cast<uint32_t*>(w + ws.x_mlp);
  kp.qkv = reinterpret_cast<uint32_t*>(w + ws.qkv);
  kp.ctx = reinterpret_cast<uint32_t*>(w + ws.ctx);
  kp.h = reinterpret_cast<uint32_t*>(w + ws.h);
  kp.part_ml = reinterpret_cast<float2*>(w + ws.part_ml);
  kp.part_o = reinterpret_cast<float*>(w + ws.part_o);
  kp.next_ids = reinterpret_cast<long long*>(p->next_ids);
  kp.next_stride = p->next_stride;
  kp.logits = static_cast<__nv_bfloat16*>(p->logits);
  kp.status = stp->status;
  for (int l = 0; l < p->n_layers; ++l) {
    kp.k_cache[l] = static_cast<__nv_bfloat16*>(p->k_cache[l]);
    kp.v_cache[l] = static_cast<__nv_bfloat16*>(p->v_cache[l]);
  }
  // at least B * H / 2 CTAs: a CTA then has at most kStepSegs attention units
  const int grid = stp->sm_count < kStepMaxGrid ? stp->sm_count : kStepMaxGrid;
  // (and every CTA has rows of the QKV projection and the MLP: the exchange relies on it)
  if (2 * grid < p->B * p->H || kp.C > fa::kStepTile * grid || 3 * kp.C < grid) return FA_B200_ERR_SHAPE;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(fa::kStepThreads);
  cfg.dynamicSmemBytes = fa::kStepSmemBytes;
  cfg.stream = static_cast<cudaStream_t>(p->stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;     // CTAs wait on one another: all must be resident
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, fa::fa_gpt_step_kernel, kp);
  const cudaError_t last = cudaGetLastError();     // clears the sticky copy of a launch error
  return static_cast<int>(e != cudaSuccess ? e : last);
}

#ifdef FA_TRACE
// Trace builds only: choose the traced CTA / copy the trace buffer to the host (synchronises).
int fa_b200_trace_select(int block) {
  return static_cast<int>(cudaMemcpyToSymbol(fa::g_fa_trace_block, &block, sizeof(int)));
}
int fa_b200_trace_read(unsigned long long* out, int n) {
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return static_cast<int>(e);
  if (n > fa::kTraceSlots) n = fa::kTraceSlots;
  return static_cast<int>(cudaMemcpyFromSymbol(out, fa::g_fa_trace, sizeof(unsigned long long) * n));
}
#endif

const char* fa_b200_strerror(int code) {
  switch (code) {
    case FA_B200_OK: return "ok";
    case FA_B200_ERR_NULL: return "fa_b200: params, q, k, v or o is NULL";
    case FA_B200_ERR_HEAD_DIM: return "fa_b200: head dimension must be 64";
    case FA_B200_ERR_SHAPE: return "fa_b200: B, H, N must be non-negative and within kernel limits";
    case FA_B200_ERR_STRIDE: return "fa_b200: strides must be positive multiples of 8 elements (16 bytes)";
    case FA_B200_ERR_ALIGN: return "fa_b200: q, k, v, o must be 16-byte aligned (lse 4-byte)";
    case FA_B200_ERR_SCALE: return "fa_b200: softmax_scale must be finite and >= 0 (0 selects 1/sqrt(d))";
    case FA_B200_ERR_DEVICE: return "fa_b200: bad device ordinal";
    case FA_B200_ERR_ARCH: return "fa_b200: device is not compute capability 10.x (B200); there is no fallback";
    case FA_B200_ERR_TENSORMAP: return "fa_b200: the driver rejected a TMA tensor map (check strides and sizes)";
    case FA_B200_ERR_DRIVER: return "fa_b200: cuTensorMapEncodeTiled is not available from this driver";
    case FA_B200_ERR_STATIC_SCRATCH: return "fa_b200: this decode problem is past the limit of fa_b200_decode_static, what its original form fitted into a built-in buffer (FA_B200_STATIC_SCRATCH_BYTES); use fa_b200_decode_direct";
    case FA_B200_ERR_ALIAS: return "fa_b200: an output buffer overlaps an input it must not overlap";
    case FA_B200_ERR_WORKSPACE: return "fa_b200: workspace is NULL, too small or (decode) not 16-byte aligned";
    case FA_B200_ERR_BUILD: return "fa_b200: the kernel image does not match this library's launch configuration; rebuild it";
    default: break;
  }
  if (code > static_cast<int>(fa::kWatchdogBase)) {
    switch (code & 0xff) {
      case fa::kWaitQFull: return "fa_b200 watchdog: wait for the Q tile load ran out";
      case fa::kWaitKVFull: return "fa_b200 watchdog: wait for a K/V tile load ran out";
      case fa::kWaitKVEmpty: return "fa_b200 watchdog: wait for a free K/V slot ran out";
      case fa::kWaitSFull: return "fa_b200 watchdog: wait for S = QK^T ran out";
      case fa::kWaitPFull: return "fa_b200 watchdog: wait for P from the softmax warps ran out";
      case fa::kWaitSFree: return "fa_b200 watchdog: wait for the softmax warps to take S ran out";
      case fa::kWaitOFree: return "fa_b200 watchdog: wait for the epilogue to read O ran out";
      case fa::kWaitQEmpty: return "fa_b200 watchdog: wait for the Q slot to be released ran out";
      case fa::kWaitStepFull: return "fa_b200 watchdog: generation step, wait for a weight tile ran out";
      case fa::kWaitStepEmpty: return "fa_b200 watchdog: generation step, wait for a free ring stage ran out";
      case fa::kWaitStepWords: return "fa_b200 watchdog: generation step, wait for another CTA's values ran out";
      case fa::kWaitItem: return "fa_b200 watchdog: wait for the next work item ran out";
      case fa::kWaitOFull: return "fa_b200 watchdog: wait for O += PV ran out";
      default: return "fa_b200 watchdog: a bounded wait ran out";
    }
  }
  if (code > 0) return cudaGetErrorString(static_cast<cudaError_t>(code));
  return "fa_b200: unknown error code";
}

}  // extern "C"
