// Native runtime of the B200 simulation backend: the C ABI declared in
// include/annarchy_b200.h.
//
// It owns, per network: the device arrays of every population/projection
// attribute (by name), the NVRTC-compiled module generated for the network,
// and the per-step launch plan. A step is either the list of plan kernels
// (grid engine; captured once into a CUDA graph of `graph_steps` steps and
// replayed, so a run of n steps costs n/graph_steps graph launches and no
// host round trip per step) or one persistent kernel that advances many
// steps per launch (local engine).
//
// The reference drives its generated CUDA step from the host every step
// and blocks on a device->host copy of the spike count
// (ANNarchy/generator/Template/CUDABaseTemplate.py:328-630); here the spike
// counts and the time counter stay on the device.
#include <cuda.h>
#include <cuda_runtime.h>
#include <nvrtc.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>
#include <algorithm>

#include "../../include/annarchy_b200.h"

extern "C" int anb_bsr_spmm_tc_after(const int* brow_ptr, const int* bcol, const uint16_t* a_tiles,
                                     int n_block_rows, int parts, const uint16_t* x_tiles, int batch,
                                     float* y, int n_post, int* err, void* stream, int pdl);

namespace {

thread_local std::string g_error;

// Driver-API entry points, fetched through the runtime on first use so that
// the library itself does not link libcuda (it then loads, and reports "no
// device", on machines without a GPU driver).
struct Driver {
  bool loaded = false;
  decltype(&cuModuleLoadData) moduleLoadData = nullptr;
  decltype(&cuModuleUnload) moduleUnload = nullptr;
  decltype(&cuModuleGetFunction) moduleGetFunction = nullptr;
  decltype(&cuModuleGetGlobal) moduleGetGlobal = nullptr;
  decltype(&cuLaunchKernel) launchKernel = nullptr;
  decltype(&cuFuncSetAttribute) funcSetAttribute = nullptr;
  decltype(&cuGetErrorString) getErrorString = nullptr;
  decltype(&cuLaunchKernelEx) launchKernelEx = nullptr;
  decltype(&cuOccupancyMaxActiveClusters) maxActiveClusters = nullptr;
  decltype(&cuOccupancyMaxActiveBlocksPerMultiprocessor) maxActiveBlocks = nullptr;
};
Driver g_drv;

template <typename F>
bool entry(const char* name, F* fn) {
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess || !p)
    return false;
  *fn = reinterpret_cast<F>(p);
  return true;
}

bool load_driver() {
  if (g_drv.loaded) return true;
  bool ok = entry("cuModuleLoadData", &g_drv.moduleLoadData) &&
            entry("cuModuleUnload", &g_drv.moduleUnload) &&
            entry("cuModuleGetFunction", &g_drv.moduleGetFunction) &&
            entry("cuModuleGetGlobal", &g_drv.moduleGetGlobal) &&
            entry("cuLaunchKernel", &g_drv.launchKernel) &&
            entry("cuFuncSetAttribute", &g_drv.funcSetAttribute) &&
            entry("cuGetErrorString", &g_drv.getErrorString) &&
            entry("cuLaunchKernelEx", &g_drv.launchKernelEx) &&
            entry("cuOccupancyMaxActiveClusters", &g_drv.maxActiveClusters) &&
            entry("cuOccupancyMaxActiveBlocksPerMultiprocessor", &g_drv.maxActiveBlocks);
  g_drv.loaded = ok;
  return ok;
}

int fail(int code, const std::string& msg) {
  g_error = msg;
  return code;
}

#define ANB_CUDA(call)                                                                \
  do {                                                                                \
    cudaError_t e_ = (call);                                                          \
    if (e_ != cudaSuccess)                                                            \
      return fail(ANB_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));  \
  } while (0)

#define ANB_CU(call)                                                \
  do {                                                              \
    CUresult r_ = (call);                                           \
    if (r_ != CUDA_SUCCESS) {                                       \
      const char* s_ = nullptr;                                     \
      if (g_drv.getErrorString) g_drv.getErrorString(r_, &s_);      \
      return fail(ANB_ERR_CUDA, std::string(#call) + ": " + (s_ ? s_ : "?")); \
    }                                                               \
  } while (0)

struct Array {
  void* ptr = nullptr;
  size_t bytes = 0;
};

// Plan entries that are library operations rather than module kernels.
enum { kOpKernel = 0, kOpBsrTc = 1, kOpBsrShared = 2 };

struct Launch {
  std::string name;
  CUfunction fn = nullptr;
  unsigned grid = 1, block = 1, smem = 0;
  unsigned cluster = 1;  // CTAs per thread-block cluster (launch attribute)
  int group = 0;         // consecutive launches of one nonzero group may run concurrently
  bool cooperative = false;  // all CTAs resident at once (grid-wide barriers)
  int op = kOpKernel;
  // kOpBsrTc: arrays block_row_ptr, block_col, tiles, x, x_tiles, y and the
  // sizes n_block_rows, batch, n_pre, n_post (kOpBsrShared: no x, the runs per block row for n_pre)
  std::string arr[6];
  int iarg[4] = {0, 0, 0, 0};
};

struct TimedLaunch {
  int kernel;
  cudaEvent_t start, stop;
};

struct KernelTime {
  std::string name;
  double total_ms = 0.0;
  int64_t launches = 0;
};

}  // namespace

struct anb_net {
  int device = 0;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  std::map<std::string, Array> arrays;
  CUmodule module = nullptr;
  bool bindings_dirty = true;
  std::vector<Launch> plan;
  Launch local;
  bool has_local = false;
  int graph_steps = 32;
  // plan kernels launched with programmatic stream serialization (each
  // generated kernel waits for its predecessor with griddepcontrol.wait)
  bool pdl = true;
  bool pdl_prev = false;   // the last plan operation was a kernel on the main stream
  cudaGraphExec_t graph = nullptr;
  double dt = 1.0;
  int64_t t = 0;
  bool timing = false;
  std::vector<TimedLaunch> pending;
  std::vector<KernelTime> times;
  std::map<std::string, int> time_index;
  void* flush_buf = nullptr;
  size_t flush_bytes = 0;
  // side streams and fork/join events of concurrent plan groups
  std::vector<cudaStream_t> side;
  std::vector<cudaEvent_t> side_ev;
  cudaEvent_t fork_ev = nullptr;
  // device scratch of anb_monitor_decode (grown on demand)
  long long* dec_rows = nullptr;
  int64_t dec_rows_cap = 0;
  int* dec_out = nullptr;
  int64_t dec_out_cap = 0;
  int64_t dec_last = 0;             // spikes of the last decoding
  int64_t dec_guess = 4096;         // pairs copied along with the next one's counts
  int64_t dec_ready = 0;            // of these, in the stage's second half
  long long* dec_first = nullptr;   // first word of every slot
  int64_t dec_first_cap = 0;
  // pinned staging for device-to-host copies, two halves of kStage bytes
  unsigned char* stage = nullptr;
  cudaEvent_t stage_ev[2] = {nullptr, nullptr};
  std::recursive_mutex stage_mutex; // held while the stage or the decoder's scratch is in use
  // stop conditions of populations (anb_run_until): the kernel of population
  // `pop` writes the device step into stop_flags[pop] when a neuron satisfies
  // the condition ("any") or when one fails it ("all")
  struct Stop {
    int pop;
    Launch l;
    int all;
  };
  std::vector<Stop> stops;
  // recorded state variables declared for anb_estimate_record_size
  struct Record {
    std::string ring;
    int64_t values = 0;
    int value_bytes = 8;
    int64_t period = 1;
  };
  std::vector<Record> records;
  // rates packed into shared bfloat16 tiles at the start of every run; the
  // step's update kernels keep the tiles up to date
  struct Pack {
    std::string x, tiles;
    int batch = 0, n_pre = 0, first_block = 0;
  };
  std::vector<Pack> packs;
};

namespace {

int ensure_device(anb_net* net) {
  ANB_CUDA(cudaSetDevice(net->device));
  return ANB_OK;
}

Array* find(anb_net* net, const char* name) {
  if (!name) return nullptr;
  auto it = net->arrays.find(name);
  return it == net->arrays.end() ? nullptr : &it->second;
}

void drop_graph(anb_net* net) {
  if (net->graph) {
    cudaGraphExecDestroy(net->graph);
    net->graph = nullptr;
  }
}

// Write the device address of every array into the module's __constant__
// pointer of the same name (anb_p_<name>), where the module declares one.
int bind(anb_net* net) {
  if (!net->module || !net->bindings_dirty) return ANB_OK;
  ANB_CUDA(cudaStreamSynchronize(net->stream));
  for (auto& kv : net->arrays) {
    std::string sym = "anb_p_" + kv.first;
    CUdeviceptr dptr = 0;
    size_t sz = 0;
    CUresult r = g_drv.moduleGetGlobal(&dptr, &sz, net->module, sym.c_str());
    if (r == CUDA_ERROR_NOT_FOUND) continue;
    if (r != CUDA_SUCCESS) return fail(ANB_ERR_CUDA, "cuModuleGetGlobal(" + sym + ") failed");
    if (sz != sizeof(void*)) return fail(ANB_ERR_ARG, sym + " is not a pointer");
    void* p = kv.second.ptr;
    ANB_CUDA(cudaMemcpy((void*)dptr, &p, sizeof(void*), cudaMemcpyHostToDevice));
  }
  net->bindings_dirty = false;
  return ANB_OK;
}

// The batched block-sparse product of a plan entry: the rates x (batch x
// n_pre, row-major) packed into bfloat16 tiles, then y (batch x n_post) +=
// x W^T on the tensor cores; a bounded wait that gives up is reported in the
// network's error word.
int launch_bsr_tc(anb_net* net, const Launch& l, cudaStream_t st) {
  void* p[6];
  for (int i = 0; i < 6; ++i) {
    Array* a = find(net, l.arr[i].c_str());
    if (!a) return fail(ANB_ERR_STATE, l.name + ": array " + l.arr[i] + " is missing");
    p[i] = a->ptr;
  }
  Array* err = find(net, "err");
  int rc = anb_bsr_tc_pack_x((const float*)p[3], l.iarg[1], l.iarg[2], (uint16_t*)p[4], st);
  if (rc == 0)
    rc = anb_bsr_spmm_tc((const int*)p[0], (const int*)p[1], (const uint16_t*)p[2], l.iarg[0],
                         (const uint16_t*)p[4], l.iarg[1], (float*)p[5], l.iarg[3],
                         err ? (int*)err->ptr : nullptr, st);
  if (rc == 2) return fail(ANB_ERR_ARG, l.name + ": the block product rejected its sizes");
  if (rc != 0) return fail(ANB_ERR_CUDA, l.name + ": block product launch failed");
  return ANB_OK;
}

int launch_bsr_shared(anb_net* net, const Launch& l, cudaStream_t st, bool pdl) {
  void* p[6] = {};
  for (int i = 0; i < 6; ++i) {
    if (i == 3) continue;
    Array* a = find(net, l.arr[i].c_str());
    if (!a) return fail(ANB_ERR_STATE, l.name + ": array " + l.arr[i] + " is missing");
    p[i] = a->ptr;
  }
  Array* err = find(net, "err");
  const int rc = anb_bsr_spmm_tc_after((const int*)p[0], (const int*)p[1], (const uint16_t*)p[2], l.iarg[0], l.iarg[2],
                                       (const uint16_t*)p[4], l.iarg[1], (float*)p[5], l.iarg[3],
                                       err ? (int*)err->ptr : nullptr, st, pdl ? 1 : 0);
  if (rc == 2) return fail(ANB_ERR_ARG, l.name + ": the block product rejected its sizes");
  if (rc != 0) return fail(ANB_ERR_CUDA, l.name + ": block product launch failed");
  return ANB_OK;
}

int launch(anb_net* net, const Launch& l, void** params, cudaStream_t on = nullptr, bool pdl = false) {
  if (l.op == kOpBsrShared) return launch_bsr_shared(net, l, on ? on : net->stream, pdl);
  if (l.op == kOpBsrTc) return launch_bsr_tc(net, l, on ? on : net->stream);
  if (l.cooperative) {
    CUlaunchAttribute attr;
    std::memset(&attr, 0, sizeof(attr));
    attr.id = CU_LAUNCH_ATTRIBUTE_COOPERATIVE;
    attr.value.cooperative = 1;
    CUlaunchConfig cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDimX = l.grid;
    cfg.gridDimY = 1;
    cfg.gridDimZ = 1;
    cfg.blockDimX = l.block;
    cfg.blockDimY = 1;
    cfg.blockDimZ = 1;
    cfg.sharedMemBytes = l.smem;
    cfg.hStream = (CUstream)(on ? on : net->stream);
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    ANB_CU(g_drv.launchKernelEx(&cfg, l.fn, params, nullptr));
    return ANB_OK;
  }
  if (l.cluster <= 1 && pdl) {
    // may be scheduled while the stream's previous kernel still runs; the
    // kernel's griddepcontrol.wait orders its reads after that kernel
    CUlaunchAttribute attr;
    std::memset(&attr, 0, sizeof(attr));
    attr.id = CU_LAUNCH_ATTRIBUTE_PROGRAMMATIC_STREAM_SERIALIZATION;
    attr.value.programmaticStreamSerializationAllowed = 1;
    CUlaunchConfig cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDimX = l.grid;
    cfg.gridDimY = 1;
    cfg.gridDimZ = 1;
    cfg.blockDimX = l.block;
    cfg.blockDimY = 1;
    cfg.blockDimZ = 1;
    cfg.sharedMemBytes = l.smem;
    cfg.hStream = (CUstream)(on ? on : net->stream);
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    ANB_CU(g_drv.launchKernelEx(&cfg, l.fn, params, nullptr));
    return ANB_OK;
  }
  if (l.cluster <= 1) {
    ANB_CU(g_drv.launchKernel(l.fn, l.grid, 1, 1, l.block, 1, 1, l.smem,
                              (CUstream)(on ? on : net->stream), params, nullptr));
    return ANB_OK;
  }
  CUlaunchAttribute attr;
  std::memset(&attr, 0, sizeof(attr));
  attr.id = CU_LAUNCH_ATTRIBUTE_CLUSTER_DIMENSION;
  attr.value.clusterDim.x = l.cluster;
  attr.value.clusterDim.y = 1;
  attr.value.clusterDim.z = 1;
  CUlaunchConfig cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDimX = l.grid;
  cfg.gridDimY = 1;
  cfg.gridDimZ = 1;
  cfg.blockDimX = l.block;
  cfg.blockDimY = 1;
  cfg.blockDimZ = 1;
  cfg.sharedMemBytes = l.smem;
  cfg.hStream = (CUstream)net->stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  ANB_CU(g_drv.launchKernelEx(&cfg, l.fn, params, nullptr));
  return ANB_OK;
}

int timed_launch(anb_net* net, const Launch& l, void** params) {
  auto it = net->time_index.find(l.name);
  int idx;
  if (it == net->time_index.end()) {
    idx = (int)net->times.size();
    net->time_index[l.name] = idx;
    net->times.push_back(KernelTime{l.name, 0.0, 0});
  } else {
    idx = it->second;
  }
  TimedLaunch tl{idx, nullptr, nullptr};
  ANB_CUDA(cudaEventCreate(&tl.start));
  ANB_CUDA(cudaEventCreate(&tl.stop));
  ANB_CUDA(cudaEventRecord(tl.start, net->stream));
  int rc = launch(net, l, params);
  if (rc != ANB_OK) return rc;
  ANB_CUDA(cudaEventRecord(tl.stop, net->stream));
  net->pending.push_back(tl);
  return ANB_OK;
}

int collect_times(anb_net* net) {
  for (auto& tl : net->pending) {
    float ms = 0.f;
    ANB_CUDA(cudaEventSynchronize(tl.stop));
    ANB_CUDA(cudaEventElapsedTime(&ms, tl.start, tl.stop));
    net->times[tl.kernel].total_ms += ms;
    net->times[tl.kernel].launches += 1;
    cudaEventDestroy(tl.start);
    cudaEventDestroy(tl.stop);
  }
  net->pending.clear();
  return ANB_OK;
}

// k - 1 side streams and their join events (created once per network)
int ensure_side(anb_net* net, size_t k) {
  if (!net->fork_ev) ANB_CUDA(cudaEventCreateWithFlags(&net->fork_ev, cudaEventDisableTiming));
  while (net->side.size() < k) {
    cudaStream_t st;
    cudaEvent_t ev;
    ANB_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    ANB_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    net->side.push_back(st);
    net->side_ev.push_back(ev);
  }
  return ANB_OK;
}

// One step of the plan. A run of consecutive launches sharing a nonzero
// group forks from the network's stream: the first stays on it, the others
// go to side streams that wait for the fork event, and the network's stream
// waits for all of them before the next launch (captured as parallel
// branches when a graph is recorded). Timed runs stay sequential.
int run_plan_once(anb_net* net) {
  const size_t n = net->plan.size();
  for (size_t i = 0; i < n;) {
    const Launch& l = net->plan[i];
    size_t j = i + 1;
    if (l.group != 0 && !net->timing)
      while (j < n && net->plan[j].group == l.group) ++j;
    if (j - i == 1) {
      // programmatic only after a kernel of the main stream (not after the
      // join of parallel branches or a library operation)
      const bool pdl = net->pdl && net->pdl_prev && !net->timing && l.op != kOpBsrTc && l.cluster <= 1;
      int rc = net->timing ? timed_launch(net, l, nullptr) : launch(net, l, nullptr, nullptr, pdl);
      if (rc != ANB_OK) return rc;
      net->pdl_prev = l.op != kOpBsrTc && l.cluster <= 1 && !l.cooperative;
      i = j;
      continue;
    }
    int rc = ensure_side(net, j - i - 1);
    if (rc != ANB_OK) return rc;
    ANB_CUDA(cudaEventRecord(net->fork_ev, net->stream));
    for (size_t q = i + 1; q < j; ++q) {
      cudaStream_t st = net->side[q - i - 1];
      ANB_CUDA(cudaStreamWaitEvent(st, net->fork_ev, 0));
      rc = launch(net, net->plan[q], nullptr, st);
      if (rc != ANB_OK) return rc;
      ANB_CUDA(cudaEventRecord(net->side_ev[q - i - 1], st));
    }
    // the branch on the main stream may start early like a single launch; the
    // side branches wait for the fork event (the previous kernel's end)
    const bool pdl = net->pdl && net->pdl_prev && l.op != kOpBsrTc && l.cluster <= 1;
    rc = launch(net, l, nullptr, nullptr, pdl);
    if (rc != ANB_OK) return rc;
    for (size_t q = i + 1; q < j; ++q) ANB_CUDA(cudaStreamWaitEvent(net->stream, net->side_ev[q - i - 1], 0));
    net->pdl_prev = false;
    i = j;
  }
  return ANB_OK;
}

int build_graph(anb_net* net) {
  if (net->graph) return ANB_OK;
  cudaGraph_t g = nullptr;
  ANB_CUDA(cudaStreamBeginCapture(net->stream, cudaStreamCaptureModeThreadLocal));
  net->pdl_prev = false;
  int rc = ANB_OK;
  for (int s = 0; s < net->graph_steps && rc == ANB_OK; ++s) rc = run_plan_once(net);
  cudaError_t e = cudaStreamEndCapture(net->stream, &g);
  if (rc != ANB_OK) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  if (e != cudaSuccess) return fail(ANB_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(e));
  e = cudaGraphInstantiate(&net->graph, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return fail(ANB_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(e));
  return ANB_OK;
}

constexpr size_t kStage = 1 << 20;

// Pinned stages (2 * kStage bytes) of destroyed networks, for the next ones:
// allocating one takes about 3 ms. At most kSparePins are kept.
constexpr size_t kSparePins = 8;
std::mutex g_pin_mutex;
std::vector<unsigned char*> g_pins;

int take_stage(anb_net* net) {
  for (auto& ev : net->stage_ev)
    if (!ev) ANB_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  {
    std::lock_guard<std::mutex> lock(g_pin_mutex);
    if (!g_pins.empty()) {
      net->stage = g_pins.back();
      g_pins.pop_back();
      return ANB_OK;
    }
  }
  void* p = nullptr;
  ANB_CUDA(cudaHostAlloc(&p, 2 * kStage, cudaHostAllocPortable));
  net->stage = (unsigned char*)p;
  return ANB_OK;
}

// (the network's stream has finished)
void give_stage(anb_net* net) {
  if (!net->stage) return;
  unsigned char* p = net->stage;
  net->stage = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_pin_mutex);
    if (g_pins.size() < kSparePins) {
      g_pins.push_back(p);
      return;
    }
  }
  cudaFreeHost(p);
}

// Device memory to the host after the stream's work. Up to kStaged bytes go
// through the pinned stage, the copy of the next part while this one is moved to
// dst: a copy into pageable memory is staged by the driver in the same way, with
// two more synchronisations (32 KB took 19 us and take 15, 1 MB 87 and 77), and
// leaves nothing in the caches for the conversion that follows most reads (5 MB of
// packed weights and their widening: 1.5 and 2.1 ms). Larger copies are the driver's
// (256 MB into memory in use 13.7 ms, 22 through the stage), with a write to every
// page first: the driver is slow on pages that do not exist yet (256 MB into a
// new array 54 ms, 41 this way and 43 through the stage).
constexpr size_t kStaged = 16 << 20;
int read_staged(anb_net* net, const void* src, void* dst, size_t bytes) {
  if (bytes > kStaged) {
    for (size_t off = 0; off < bytes; off += 4096) static_cast<volatile unsigned char*>(dst)[off] = 0;
    ANB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, net->stream));
    ANB_CUDA(cudaStreamSynchronize(net->stream));
    return ANB_OK;
  }
  // (several threads may read one network's arrays)
  std::lock_guard<std::recursive_mutex> lock(net->stage_mutex);
  const size_t parts = (bytes + kStage - 1) / kStage;
  if (parts > 1) net->dec_ready = 0;   // decoded pairs kept in the second half
  auto issue = [&](size_t i) -> cudaError_t {
    const size_t off = i * kStage, n = bytes - off < kStage ? bytes - off : kStage;
    cudaError_t e = cudaMemcpyAsync(net->stage + (i & 1) * kStage, (const unsigned char*)src + off, n,
                                    cudaMemcpyDeviceToHost, net->stream);
    return e != cudaSuccess ? e : cudaEventRecord(net->stage_ev[i & 1], net->stream);
  };
  ANB_CUDA(issue(0));
  for (size_t i = 0; i < parts; ++i) {
    if (i + 1 < parts) ANB_CUDA(issue(i + 1));
    ANB_CUDA(cudaEventSynchronize(net->stage_ev[i & 1]));
    const size_t off = i * kStage, n = bytes - off < kStage ? bytes - off : kStage;
    std::memcpy((unsigned char*)dst + off, net->stage + (i & 1) * kStage, n);
  }
  return ANB_OK;
}

int write_time(anb_net* net) {
  Array* a = find(net, "t");
  if (!a) return fail(ANB_ERR_STATE, "time counter missing");
  long long t = (long long)net->t;
  ANB_CUDA(cudaMemcpyAsync(a->ptr, &t, sizeof(t), cudaMemcpyHostToDevice, net->stream));
  ANB_CUDA(cudaStreamSynchronize(net->stream));
  return ANB_OK;
}

int create_array(anb_net* net, const std::string& name, size_t bytes) {
  Array* old = find(net, name.c_str());
  if (old) {
    if (old->bytes == bytes) {
      ANB_CUDA(cudaMemsetAsync(old->ptr, 0, bytes ? bytes : 1, net->stream));
      ANB_CUDA(cudaStreamSynchronize(net->stream));
      return ANB_OK;
    }
    ANB_CUDA(cudaStreamSynchronize(net->stream));
    cudaFree(old->ptr);
    net->arrays.erase(name);
  }
  Array a;
  a.bytes = bytes;
  size_t alloc = bytes ? bytes : 16;
  cudaError_t e = cudaMalloc(&a.ptr, alloc);
  if (e != cudaSuccess)
    return fail(ANB_ERR_ALLOC, "cudaMalloc(" + std::to_string(alloc) + ") for " + name + ": " +
                                   cudaGetErrorString(e));
  ANB_CUDA(cudaMemsetAsync(a.ptr, 0, alloc, net->stream));
  ANB_CUDA(cudaStreamSynchronize(net->stream));
  net->arrays[name] = a;
  net->bindings_dirty = true;
  return ANB_OK;
}

}  // namespace

extern "C" {

int anb_abi_version(void) { return 1; }

const char* anb_last_error(void) { return g_error.c_str(); }

int anb_device_count(int* count) {
  if (!count) return fail(ANB_ERR_ARG, "count is NULL");
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  *count = (e == cudaSuccess) ? n : 0;
  return ANB_OK;
}

int anb_device_sm_count(int device, int* count) {
  if (!count) return fail(ANB_ERR_ARG, "count is NULL");
  *count = 0;
  ANB_CUDA(cudaDeviceGetAttribute(count, cudaDevAttrMultiProcessorCount, device));
  return ANB_OK;
}

int anb_create(int device, anb_net** out) {
  if (!out) return fail(ANB_ERR_ARG, "out is NULL");
  *out = nullptr;
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0)
    return fail(ANB_ERR_CUDA, "no CUDA device is available");
  if (device < 0 || device >= n) return fail(ANB_ERR_ARG, "device index out of range");
  std::unique_ptr<anb_net> net(new anb_net());
  net->device = device;
  ANB_CUDA(cudaSetDevice(device));
  ANB_CUDA(cudaFree(nullptr));  // create the primary context for the driver-API calls
  if (!load_driver()) return fail(ANB_ERR_CUDA, "CUDA driver entry points are unavailable");
  ANB_CUDA(cudaStreamCreateWithFlags(&net->own_stream, cudaStreamNonBlocking));
  net->stream = net->own_stream;
  int rc = take_stage(net.get());
  if (rc == ANB_OK) rc = create_array(net.get(), "t", sizeof(long long));
  if (rc == ANB_OK) rc = create_array(net.get(), "dt", sizeof(double));
  if (rc == ANB_OK) rc = create_array(net.get(), "err", 4 * sizeof(int));
  if (rc != ANB_OK) {
    give_stage(net.get());
    return rc;
  }
  *out = net.release();
  return ANB_OK;
}

int anb_destroy(anb_net* net) {
  if (!net) return ANB_OK;
  cudaSetDevice(net->device);
  if (net->stream) cudaStreamSynchronize(net->stream);
  for (auto& tl : net->pending) {
    cudaEventDestroy(tl.start);
    cudaEventDestroy(tl.stop);
  }
  drop_graph(net);
  for (auto st : net->side) cudaStreamDestroy(st);
  for (auto ev : net->side_ev) cudaEventDestroy(ev);
  if (net->fork_ev) cudaEventDestroy(net->fork_ev);
  if (net->flush_buf) cudaFree(net->flush_buf);
  if (net->dec_rows) cudaFree(net->dec_rows);
  if (net->dec_out) cudaFree(net->dec_out);
  if (net->dec_first) cudaFree(net->dec_first);
  give_stage(net);
  for (auto ev : net->stage_ev)
    if (ev) cudaEventDestroy(ev);
  if (net->module) g_drv.moduleUnload(net->module);
  for (auto& kv : net->arrays) cudaFree(kv.second.ptr);
  if (net->own_stream) cudaStreamDestroy(net->own_stream);
  delete net;
  return ANB_OK;
}

int anb_initialize(anb_net* net, double dt) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  if (!(dt > 0.0)) return fail(ANB_ERR_ARG, "dt must be positive");
  int rc = ensure_device(net);
  if (rc) return rc;
  net->dt = dt;
  Array* a = find(net, "dt");
  ANB_CUDA(cudaMemcpyAsync(a->ptr, &dt, sizeof(double), cudaMemcpyHostToDevice, net->stream));
  net->t = 0;
  return write_time(net);
}

int anb_set_time(anb_net* net, int64_t t) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  int rc = ensure_device(net);
  if (rc) return rc;
  net->t = t;
  return write_time(net);
}

int anb_get_time(anb_net* net, int64_t* t) {
  if (!net || !t) return fail(ANB_ERR_ARG, "NULL argument");
  *t = net->t;
  return ANB_OK;
}

int anb_set_stream(anb_net* net, void* cuda_stream) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  int rc = ensure_device(net);
  if (rc) return rc;
  ANB_CUDA(cudaStreamSynchronize(net->stream));
  net->stream = cuda_stream ? (cudaStream_t)cuda_stream : net->own_stream;
  drop_graph(net);
  return ANB_OK;
}

int anb_get_stream(anb_net* net, void** cuda_stream) {
  if (!net || !cuda_stream) return fail(ANB_ERR_ARG, "NULL argument");
  int rc = ensure_device(net);
  if (rc) return rc;
  *cuda_stream = (void*)net->stream;
  return ANB_OK;
}

int anb_array_create(anb_net* net, const char* name, size_t bytes) {
  if (!net || !name || !*name) return fail(ANB_ERR_ARG, "NULL argument");
  int rc = ensure_device(net);
  if (rc) return rc;
  return create_array(net, name, bytes);
}

int anb_array_free(anb_net* net, const char* name) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  Array* a = find(net, name);
  if (!a) return fail(ANB_ERR_ARG, std::string("unknown array ") + (name ? name : "(null)"));
  int rc = ensure_device(net);
  if (rc) return rc;
  ANB_CUDA(cudaStreamSynchronize(net->stream));
  cudaFree(a->ptr);
  net->arrays.erase(name);
  net->bindings_dirty = true;
  return ANB_OK;
}

int anb_array_write(anb_net* net, const char* name, size_t offset, const void* src, size_t bytes) {
  if (!net || (!src && bytes)) return fail(ANB_ERR_ARG, "NULL argument");
  Array* a = find(net, name);
  if (!a) return fail(ANB_ERR_ARG, std::string("unknown array ") + (name ? name : "(null)"));
  if (offset > a->bytes || bytes > a->bytes - offset)
    return fail(ANB_ERR_ARG, std::string("write beyond the end of ") + name);
  if (!bytes) return ANB_OK;
  int rc = ensure_device(net);
  if (rc) return rc;
  ANB_CUDA(cudaMemcpyAsync((char*)a->ptr + offset, src, bytes, cudaMemcpyHostToDevice, net->stream));
  ANB_CUDA(cudaStreamSynchronize(net->stream));
  return ANB_OK;
}

int anb_array_read(anb_net* net, const char* name, size_t offset, void* dst, size_t bytes) {
  if (!net || (!dst && bytes)) return fail(ANB_ERR_ARG, "NULL argument");
  Array* a = find(net, name);
  if (!a) return fail(ANB_ERR_ARG, std::string("unknown array ") + (name ? name : "(null)"));
  if (offset > a->bytes || bytes > a->bytes - offset)
    return fail(ANB_ERR_ARG, std::string("read beyond the end of ") + name);
  if (!bytes) return ANB_OK;
  int rc = ensure_device(net);
  if (rc) return rc;
  return read_staged(net, (const char*)a->ptr + offset, dst, bytes);
}

int anb_array_fill_zero(anb_net* net, const char* name) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  Array* a = find(net, name);
  if (!a) return fail(ANB_ERR_ARG, std::string("unknown array ") + (name ? name : "(null)"));
  int rc = ensure_device(net);
  if (rc) return rc;
  if (a->bytes) ANB_CUDA(cudaMemsetAsync(a->ptr, 0, a->bytes, net->stream));
  ANB_CUDA(cudaStreamSynchronize(net->stream));
  return ANB_OK;
}

int anb_array_info(anb_net* net, const char* name, void** device_ptr, size_t* bytes) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  Array* a = find(net, name);
  if (!a) return fail(ANB_ERR_ARG, std::string("unknown array ") + (name ? name : "(null)"));
  if (device_ptr) *device_ptr = a->ptr;
  if (bytes) *bytes = a->bytes;
  return ANB_OK;
}

int anb_module_load(anb_net* net, const char* source, const char* options) {
  if (!net || !source) return fail(ANB_ERR_ARG, "NULL argument");
  int rc = ensure_device(net);
  if (rc) return rc;
  std::vector<std::string> opts = {"--gpu-architecture=sm_100a", "-std=c++17", "-default-device",
                                   "-lineinfo"};
  if (options) {
    std::string s(options), cur;
    for (char c : s) {
      if (c == '\n') {
        if (!cur.empty()) opts.push_back(cur);
        cur.clear();
      } else {
        cur.push_back(c);
      }
    }
    if (!cur.empty()) opts.push_back(cur);
  }
  std::vector<const char*> copts;
  for (auto& o : opts) copts.push_back(o.c_str());

  nvrtcProgram prog;
  if (nvrtcCreateProgram(&prog, source, "anb_network.cu", 0, nullptr, nullptr) != NVRTC_SUCCESS)
    return fail(ANB_ERR_COMPILE, "nvrtcCreateProgram failed");
  nvrtcResult cr = nvrtcCompileProgram(prog, (int)copts.size(), copts.data());
  size_t log_size = 0;
  nvrtcGetProgramLogSize(prog, &log_size);
  std::string log(log_size, '\0');
  if (log_size) nvrtcGetProgramLog(prog, &log[0]);
  if (cr != NVRTC_SUCCESS) {
    nvrtcDestroyProgram(&prog);
    return fail(ANB_ERR_COMPILE, std::string("NVRTC: ") + nvrtcGetErrorString(cr) + "\n" + log);
  }
  size_t cubin_size = 0;
  if (nvrtcGetCUBINSize(prog, &cubin_size) != NVRTC_SUCCESS || cubin_size == 0) {
    nvrtcDestroyProgram(&prog);
    return fail(ANB_ERR_COMPILE, "NVRTC produced no cubin");
  }
  std::vector<char> cubin(cubin_size);
  nvrtcGetCUBIN(prog, cubin.data());
  nvrtcDestroyProgram(&prog);

  ANB_CUDA(cudaStreamSynchronize(net->stream));
  drop_graph(net);
  net->plan.clear();
  net->packs.clear();
  net->stops.clear();
  net->has_local = false;
  if (net->module) {
    g_drv.moduleUnload(net->module);
    net->module = nullptr;
  }
  ANB_CU(g_drv.moduleLoadData(&net->module, cubin.data()));
  net->bindings_dirty = true;
  return bind(net);
}

// ---- entry points shaped like the reference module's set_seed,
// estimate_record_size and proj<k>_wrapper.init_from_lil ----------------------------

int anb_set_seed(anb_net* net, uint64_t seed, int num_sources, int use_seed_seq) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  if (num_sources < 0) return fail(ANB_ERR_ARG, "num_sources < 0");
  (void)use_seed_seq;
  const uint32_t key[2] = {(uint32_t)(seed & 0xffffffffull), (uint32_t)(seed >> 32)};
  Array* a = find(net, "rng_seed");
  if (a && a->bytes != sizeof(key)) return fail(ANB_ERR_ARG, "rng_seed has an unexpected size");
  if (!a) {
    int rc = anb_array_create(net, "rng_seed", sizeof(key));
    if (rc) return rc;
  }
  return anb_array_write(net, "rng_seed", 0, key, sizeof(key));
}

int anb_record_declare(anb_net* net, const char* ring, int64_t values_per_record, int value_bytes,
                       int64_t period_steps) {
  if (!net || !ring) return fail(ANB_ERR_ARG, "NULL argument");
  if (values_per_record < 0 || value_bytes <= 0 || period_steps <= 0)
    return fail(ANB_ERR_ARG, "record sizes and period must be positive");
  for (auto& r : net->records)
    if (r.ring == ring) {
      r.values = values_per_record;
      r.value_bytes = value_bytes;
      r.period = period_steps;
      return ANB_OK;
    }
  anb_net::Record r;
  r.ring = ring;
  r.values = values_per_record;
  r.value_bytes = value_bytes;
  r.period = period_steps;
  net->records.push_back(r);
  return ANB_OK;
}

int anb_estimate_record_size(anb_net* net, int64_t nsteps, size_t* mib) {
  if (!net || !mib) return fail(ANB_ERR_ARG, "NULL argument");
  if (nsteps < 0) return fail(ANB_ERR_ARG, "nsteps < 0");
  unsigned long long bytes = 0;
  for (const auto& r : net->records)
    bytes += (unsigned long long)(nsteps / r.period) * (unsigned long long)r.values *
             (unsigned long long)r.value_bytes;
  *mib = (size_t)(bytes >> 20);
  return ANB_OK;
}

namespace {
uint16_t to_bf16_rne(float f) {
  uint32_t u;
  std::memcpy(&u, &f, 4);
  if ((u & 0x7f800000u) == 0x7f800000u && (u & 0x007fffffu)) return (uint16_t)((u >> 16) | 0x40u);
  const uint32_t lsb = (u >> 16) & 1u;
  return (uint16_t)((u + 0x7fffu + lsb) >> 16);
}
}  // namespace

int anb_init_from_lil(anb_net* net, const char* prefix, int n_rows, const int* post_ranks,
                      const int64_t* row_begin, const int* pre_ranks, const double* w,
                      const int* delays, int requires_sorting, int weight_bytes, int64_t* nnz_out) {
  if (!net || !prefix || n_rows < 0 || (n_rows > 0 && (!post_ranks || !row_begin)))
    return fail(ANB_ERR_ARG, "NULL argument or negative row count");
  if (weight_bytes != 8 && weight_bytes != 4 && weight_bytes != 2)
    return fail(ANB_ERR_ARG, "weight_bytes must be 8, 4 or 2");
  const int64_t nnz = n_rows ? row_begin[n_rows] : 0;
  if (n_rows && row_begin[0] != 0) return fail(ANB_ERR_ARG, "row_begin[0] must be 0");
  for (int r = 0; r < n_rows; ++r) {
    if (row_begin[r + 1] < row_begin[r]) return fail(ANB_ERR_ARG, "row_begin is not ascending");
    if (post_ranks[r] < 0) return fail(ANB_ERR_ARG, "negative post rank");
  }
  if (nnz > 0 && (!pre_ranks || !w)) return fail(ANB_ERR_ARG, "pre_ranks or w is NULL");
  if (nnz >= (1ll << 31)) return fail(ANB_ERR_ARG, "more than 2^31 - 1 synapses");
  for (int64_t j = 0; j < nnz; ++j)
    if (pre_ranks[j] < 0) return fail(ANB_ERR_ARG, "negative pre rank");
  // dendrites in ascending post rank when the caller asks for sorting (the
  // reference's pairsort of init_matrix_from_lil), else in the given order
  std::vector<int> order(n_rows);
  for (int r = 0; r < n_rows; ++r) order[r] = r;
  if (requires_sorting)
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return post_ranks[a] < post_ranks[b]; });
  std::vector<int> post(n_rows), row_ptr(n_rows + 1), col(nnz), dly;
  std::vector<unsigned char> wv((size_t)nnz * weight_bytes);
  bool uniform_delay = true;
  if (delays)
    for (int64_t j = 1; j < nnz; ++j)
      if (delays[j] != delays[0]) uniform_delay = false;
  if (delays && !uniform_delay) dly.resize(nnz);
  int64_t k = 0;
  for (int i = 0; i < n_rows; ++i) {
    const int r = order[i];
    post[i] = post_ranks[r];
    row_ptr[i] = (int)k;
    for (int64_t j = row_begin[r]; j < row_begin[r + 1]; ++j, ++k) {
      col[k] = pre_ranks[j];
      if (weight_bytes == 8) {
        std::memcpy(&wv[k * 8], &w[j], 8);
      } else if (weight_bytes == 4) {
        const float f = (float)w[j];
        std::memcpy(&wv[k * 4], &f, 4);
      } else {
        const uint16_t h = to_bf16_rne((float)w[j]);
        std::memcpy(&wv[k * 2], &h, 2);
      }
      if (!dly.empty()) dly[k] = delays[j];
    }
  }
  row_ptr[n_rows] = (int)k;
  const std::string p(prefix);
  int rc = anb_array_create(net, (p + "__post_rank").c_str(), sizeof(int) * (size_t)n_rows);
  if (!rc) rc = anb_array_write(net, (p + "__post_rank").c_str(), 0, post.data(), sizeof(int) * post.size());
  if (!rc) rc = anb_array_create(net, (p + "__row_ptr").c_str(), sizeof(int) * row_ptr.size());
  if (!rc) rc = anb_array_write(net, (p + "__row_ptr").c_str(), 0, row_ptr.data(), sizeof(int) * row_ptr.size());
  if (!rc) rc = anb_array_create(net, (p + "__col").c_str(), sizeof(int) * (size_t)nnz);
  if (!rc) rc = anb_array_write(net, (p + "__col").c_str(), 0, col.data(), sizeof(int) * col.size());
  if (!rc) rc = anb_array_create(net, (p + "__w").c_str(), wv.size());
  if (!rc) rc = anb_array_write(net, (p + "__w").c_str(), 0, wv.data(), wv.size());
  if (!rc && !dly.empty()) {
    rc = anb_array_create(net, (p + "__dly").c_str(), sizeof(int) * dly.size());
    if (!rc) rc = anb_array_write(net, (p + "__dly").c_str(), 0, dly.data(), sizeof(int) * dly.size());
  }
  if (rc) return rc;
  if (nnz_out) *nnz_out = nnz;
  return ANB_OK;
}

int anb_module_set_constant(anb_net* net, const char* name, double value) {
  if (!net || !name) return fail(ANB_ERR_ARG, "NULL argument");
  if (!net->module) return fail(ANB_ERR_STATE, "no module loaded");
  int rc = ensure_device(net);
  if (rc) return rc;
  CUdeviceptr dptr = 0;
  size_t sz = 0;
  CUresult r = g_drv.moduleGetGlobal(&dptr, &sz, net->module, name);
  if (r == CUDA_ERROR_NOT_FOUND) return ANB_OK;  // declared but used by no kernel: removed
  if (r != CUDA_SUCCESS) return fail(ANB_ERR_ARG, std::string("constant ") + name + " not accessible");
  if (sz == 8) {
    ANB_CUDA(cudaMemcpyAsync((void*)dptr, &value, 8, cudaMemcpyHostToDevice, net->stream));
  } else if (sz == 4) {
    const float f = (float)value;
    ANB_CUDA(cudaMemcpyAsync((void*)dptr, &f, 4, cudaMemcpyHostToDevice, net->stream));
  } else {
    return fail(ANB_ERR_ARG, std::string(name) + " is not a float or double constant");
  }
  ANB_CUDA(cudaStreamSynchronize(net->stream));
  return ANB_OK;
}

int anb_nvrtc_compile(const char* source, const char* options, char* log, size_t log_len,
                      size_t* cubin_bytes) {
  if (!source) return fail(ANB_ERR_ARG, "source is NULL");
  std::vector<std::string> opts = {"--gpu-architecture=sm_100a", "-std=c++17", "-default-device",
                                   "-lineinfo"};
  if (options) {
    std::string s(options), cur;
    for (char c : s) {
      if (c == '\n') {
        if (!cur.empty()) opts.push_back(cur);
        cur.clear();
      } else {
        cur.push_back(c);
      }
    }
    if (!cur.empty()) opts.push_back(cur);
  }
  std::vector<const char*> copts;
  for (auto& o : opts) copts.push_back(o.c_str());
  nvrtcProgram prog;
  if (nvrtcCreateProgram(&prog, source, "anb_network.cu", 0, nullptr, nullptr) != NVRTC_SUCCESS)
    return fail(ANB_ERR_COMPILE, "nvrtcCreateProgram failed");
  nvrtcResult cr = nvrtcCompileProgram(prog, (int)copts.size(), copts.data());
  size_t log_size = 0;
  nvrtcGetProgramLogSize(prog, &log_size);
  std::string text(log_size, '\0');
  if (log_size) nvrtcGetProgramLog(prog, &text[0]);
  if (log && log_len) {
    std::strncpy(log, text.c_str(), log_len - 1);
    log[log_len - 1] = '\0';
  }
  size_t sz = 0;
  if (cr == NVRTC_SUCCESS) nvrtcGetCUBINSize(prog, &sz);
  nvrtcDestroyProgram(&prog);
  if (cubin_bytes) *cubin_bytes = sz;
  if (cr != NVRTC_SUCCESS)
    return fail(ANB_ERR_COMPILE, std::string("NVRTC: ") + nvrtcGetErrorString(cr) + "\n" + text);
  return ANB_OK;
}

namespace {
// Spike-ring decoding on the device. The ring's words are cut into slots
// [first[i], first[i + 1]) (one, or one per instance of a batch); row r =
// slot * steps + step, one warp per row, so the pairs come out by slot, step
// and rank.
__device__ __forceinline__ unsigned anb_dec_word(const uint32_t* row, int64_t w, int64_t n) {
  const int64_t valid = n - 32 * w;                 // bits of this word that are neurons
  unsigned m = row[w];
  if (valid <= 0) return 0u;
  if (valid < 32) m &= (1u << valid) - 1u;
  return m;
}

__global__ void anb_dec_count(const uint32_t* __restrict__ ring, int64_t steps, int64_t words,
                              int64_t n, int64_t rows, const long long* __restrict__ first,
                              long long* __restrict__ counts) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += nw) {
    const int64_t slot = r / steps;
    const uint32_t* row = ring + (r - slot * steps) * words;
    const int64_t w1 = first[slot + 1];
    int c = 0;
    for (int64_t w = first[slot] + lane; w < w1; w += 32) c += __popc(anb_dec_word(row, w, n));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) counts[r] = c;
  }
}

// Exclusive prefix sum of counts[0..steps) in place, total in counts[steps]
// (one CTA of 1024 threads, chunk by chunk with a carry).
__global__ void anb_dec_scan(long long* __restrict__ counts, int64_t steps) {
  __shared__ long long sums[32];
  __shared__ long long carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t base = 0; base < steps; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const long long x = i < steps ? counts[i] : 0;
    long long incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      long long s = lane < (int)(blockDim.x >> 5) ? sums[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const long long v = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += v;
      }
      sums[lane] = s;
    }
    __syncthreads();
    const long long before = carry + (warp ? sums[warp - 1] : 0);
    if (i < steps) counts[i] = before + incl - x;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = before + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) counts[steps] = carry;
}

// Pairs in order: out[2k] = step, out[2k+1] = rank within the slot.
__global__ void anb_dec_emit(const uint32_t* __restrict__ ring, int64_t steps, int64_t words,
                             int64_t n, int64_t rows, const long long* __restrict__ first,
                             const long long* __restrict__ offsets, int* __restrict__ out,
                             int64_t capacity) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += nw) {
    const int64_t slot = r / steps, step = r - slot * steps;
    const uint32_t* row = ring + step * words;
    const int64_t wb = first[slot], we = first[slot + 1];
    int64_t base = offsets[r];
    for (int64_t w0 = wb; w0 < we; w0 += 32) {
      const int64_t w = w0 + lane;
      unsigned m = w < we ? anb_dec_word(row, w, n) : 0u;
      const int c = __popc(m);
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      int64_t k = base + incl - c;
      while (m) {
        const int b = __ffs(m) - 1;
        m &= m - 1;
        if (k < capacity) {
          out[2 * k] = (int)step;
          out[2 * k + 1] = (int)((w - wb) * 32 + b);
        }
        ++k;
      }
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
}
}  // namespace

int anb_monitor_decode_slots(anb_net* net, const char* array, int64_t steps, int64_t words_per_step,
                             int64_t n, int64_t n_slots, const int64_t* first_word, int64_t* offsets) {
  if (!net || !array || !offsets || !first_word || steps < 0 || words_per_step < 0 || n_slots < 1)
    return fail(ANB_ERR_ARG, "bad argument");
  Array* a = find(net, array);
  if (!a) return fail(ANB_ERR_ARG, std::string("unknown array ") + array);
  if ((size_t)(steps * words_per_step) * 4 > a->bytes)
    return fail(ANB_ERR_ARG, "more rows requested than the array holds");
  if (steps >= ((int64_t)1 << 31) || words_per_step * 32 >= ((int64_t)1 << 31))
    return fail(ANB_ERR_ARG, "ring too large for 32-bit steps and ranks");
  for (int64_t i = 0; i < n_slots; ++i)
    if (first_word[i] < 0 || first_word[i + 1] < first_word[i] || first_word[i + 1] > words_per_step)
      return fail(ANB_ERR_ARG, "slots must be ascending ranges of the ring's words");
  int rc = ensure_device(net);
  if (rc) return rc;
  std::lock_guard<std::recursive_mutex> lock(net->stage_mutex);
  net->dec_last = net->dec_ready = 0;
  for (int64_t i = 0; i <= n_slots; ++i) offsets[i] = 0;
  if (steps == 0) return ANB_OK;
  const int64_t rows = steps * n_slots;
  if (net->dec_rows_cap < rows + 1) {
    if (net->dec_rows) cudaFree(net->dec_rows);
    net->dec_rows = nullptr;
    net->dec_rows_cap = 0;
    ANB_CUDA(cudaMalloc(&net->dec_rows, (size_t)(rows + 1) * sizeof(long long)));
    net->dec_rows_cap = rows + 1;
  }
  if (net->dec_first_cap < n_slots + 1) {
    if (net->dec_first) cudaFree(net->dec_first);
    net->dec_first = nullptr;
    net->dec_first_cap = 0;
    ANB_CUDA(cudaMalloc(&net->dec_first, (size_t)(n_slots + 1) * sizeof(long long)));
    net->dec_first_cap = n_slots + 1;
  }
  ANB_CUDA(cudaMemcpyAsync(net->dec_first, first_word, (size_t)(n_slots + 1) * sizeof(long long),
                           cudaMemcpyHostToDevice, net->stream));
  // few spikes are decoded and copied with one wait: pairs up to dec_guess
  // come along with the counts (a first buffer of 64 KB: larger allocations
  // take milliseconds)
  const int64_t stage_pairs = (int64_t)(kStage / (2 * sizeof(int)));
  if (!net->dec_out) {
    net->dec_out_cap = 0;
    ANB_CUDA(cudaMalloc(&net->dec_out, 8192 * 2 * sizeof(int)));
    net->dec_out_cap = 8192;
  }
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, net->device);
  const uint32_t* ring = static_cast<const uint32_t*>(a->ptr);
  const long long* first = net->dec_first;
  anb_dec_count<<<sms * 4, 256, 0, net->stream>>>(ring, steps, words_per_step, n, rows, first, net->dec_rows);
  anb_dec_scan<<<1, 1024, 0, net->stream>>>(net->dec_rows, rows);
  anb_dec_emit<<<sms * 4, 256, 0, net->stream>>>(ring, steps, words_per_step, n, rows, first, net->dec_rows,
                                                 net->dec_out, net->dec_out_cap);
  ANB_CUDA(cudaGetLastError());
  // the counts before every slot's first row, and the total
  const size_t off_bytes = (size_t)(n_slots + 1) * 8;
  void* off_dst = off_bytes <= kStage ? (void*)net->stage : (void*)offsets;
  ANB_CUDA(cudaMemcpy2DAsync(off_dst, 8, net->dec_rows, (size_t)steps * 8, 8, (size_t)n_slots + 1,
                             cudaMemcpyDeviceToHost, net->stream));
  const int64_t guess = std::min(std::min(stage_pairs, net->dec_out_cap), net->dec_guess);
  if (guess > 0)
    ANB_CUDA(cudaMemcpyAsync(net->stage + kStage, net->dec_out, (size_t)guess * 2 * sizeof(int),
                             cudaMemcpyDeviceToHost, net->stream));
  ANB_CUDA(cudaStreamSynchronize(net->stream));
  if (off_dst != (void*)offsets) std::memcpy(offsets, off_dst, off_bytes);
  const int64_t total = offsets[n_slots];
  net->dec_last = total;
  net->dec_ready = std::min(guess, total);
  net->dec_guess = total + total / 4 + 512;
  if (total > net->dec_out_cap) {
    // more than fitted: emit them again into a larger buffer
    cudaFree(net->dec_out);
    net->dec_out = nullptr;
    net->dec_out_cap = 0;
    const int64_t cap = total + total / 4;
    ANB_CUDA(cudaMalloc(&net->dec_out, (size_t)cap * 2 * sizeof(int)));
    net->dec_out_cap = cap;
    anb_dec_emit<<<sms * 4, 256, 0, net->stream>>>(ring, steps, words_per_step, n, rows, first,
                                                   net->dec_rows, net->dec_out, net->dec_out_cap);
    ANB_CUDA(cudaGetLastError());
  }
  return ANB_OK;
}

int anb_monitor_fetch(anb_net* net, int64_t first_step, int64_t* out_steps, int64_t* out_ranks,
                      int64_t count) {
  if (!net || count < 0 || (count > 0 && (!out_steps || !out_ranks)))
    return fail(ANB_ERR_ARG, "bad argument");
  std::lock_guard<std::recursive_mutex> lock(net->stage_mutex);
  if (count > net->dec_last) return fail(ANB_ERR_ARG, "more spikes requested than were decoded");
  int rc = ensure_device(net);
  if (rc) return rc;
  const int* p = reinterpret_cast<const int*>(net->stage + kStage);
  std::vector<int> rest;
  if (count > net->dec_ready) {
    rest.resize((size_t)count * 2);
    rc = read_staged(net, net->dec_out, rest.data(), (size_t)count * 2 * sizeof(int));
    if (rc) return rc;
    p = rest.data();
  }
  for (int64_t i = 0; i < count; ++i) {
    out_steps[i] = first_step + p[2 * i];
    out_ranks[i] = p[2 * i + 1];
  }
  net->dec_last = net->dec_ready = 0;
  return ANB_OK;
}

int anb_monitor_decode(anb_net* net, const char* array, int64_t steps, int64_t words_per_step,
                       int64_t n, int32_t* out_steps, int32_t* out_ranks, int64_t capacity,
                       int64_t* count) {
  if (!net || !array || !count || capacity < 0) return fail(ANB_ERR_ARG, "bad argument");
  if (capacity > 0 && (!out_steps || !out_ranks)) return fail(ANB_ERR_ARG, "output is NULL");
  const int64_t first[2] = {0, words_per_step};
  int64_t off[2] = {0, 0};
  *count = 0;
  std::lock_guard<std::recursive_mutex> lock(net->stage_mutex);
  int rc = anb_monitor_decode_slots(net, array, steps, words_per_step, n, 1, first, off);
  if (rc) return rc;
  *count = off[1];
  const int64_t k = off[1] < capacity ? off[1] : capacity;
  std::vector<int64_t> s((size_t)k), r((size_t)k);
  rc = anb_monitor_fetch(net, 0, s.data(), r.data(), k);
  if (rc) return rc;
  for (int64_t i = 0; i < k; ++i) {
    out_steps[i] = (int32_t)s[i];
    out_ranks[i] = (int32_t)r[i];
  }
  return ANB_OK;
}

int anb_bank_interleave(const int64_t* row_ptr, int64_t n_rows, const int32_t* post, int64_t* perm) {
  if (n_rows < 0 || (n_rows > 0 && (!row_ptr || !post || !perm)))
    return fail(ANB_ERR_ARG, "anb_bank_interleave: invalid arguments");
  for (int64_t r = 0; r < n_rows; ++r)
    if (row_ptr[r + 1] < row_ptr[r]) return fail(ANB_ERR_ARG, "anb_bank_interleave: row pointers decrease");
  std::vector<int64_t> by_bank, slots;
  for (int64_t r = 0; r < n_rows; ++r) {
    const int64_t b = row_ptr[r], e = row_ptr[r + 1];
    const int64_t n = e - b;
    if (n == 0) continue;
    // the row's synapses by bank (post rank mod 32), stable within a bank
    int64_t start[33] = {0};
    for (int64_t q = b; q < e; ++q) ++start[(post[q] & 31) + 1];
    for (int k = 0; k < 32; ++k) start[k + 1] += start[k];
    by_bank.assign((size_t)n, 0);
    for (int64_t q = b; q < e; ++q) by_bank[(size_t)start[post[q] & 31]++] = q;
    // positions in the order lane, block, component: one aligned group of 4
    // positions per lane, 32 lanes per 128-position block; the positions of
    // one block with the same component are one warp's atomic instruction
    slots.clear();
    const int64_t base = b & ~(int64_t)3;
    const int64_t blocks = (e - base + 127) / 128;
    for (int64_t l = 0; l < 32; ++l)
      for (int64_t blk = 0; blk < blocks; ++blk)
        for (int64_t c = 0; c < 4; ++c) {
          const int64_t q = base + blk * 128 + 4 * l + c;
          if (q >= b && q < e) slots.push_back(q);
        }
    for (int64_t j = 0; j < n; ++j) perm[slots[(size_t)j] - row_ptr[0]] = by_bank[(size_t)j];
  }
  return ANB_OK;
}

int64_t anb_bitmap_decode(const uint32_t* words, int64_t steps, int64_t words_per_step,
                          int64_t n, int64_t* out_steps, int64_t* out_ranks, int64_t capacity) {
  int64_t k = 0;
  for (int64_t s = 0; s < steps; ++s) {
    const uint32_t* row = words + s * words_per_step;
    int64_t w = 0;
    // two words at a time: most words of a raster are zero
    for (; w + 1 < words_per_step; w += 2) {
      uint64_t m = (uint64_t)row[w] | ((uint64_t)row[w + 1] << 32);
      while (m) {
        const int b = __builtin_ctzll(m);
        m &= m - 1;
        const int64_t rank = w * 32 + b;
        if (rank >= n) continue;
        if (k < capacity) {
          out_steps[k] = s;
          out_ranks[k] = rank;
        }
        ++k;
      }
    }
    if (w < words_per_step) {
      uint32_t m = row[w];
      while (m) {
        const int b = __builtin_ctz(m);
        m &= m - 1;
        const int64_t rank = w * 32 + b;
        if (rank >= n) continue;
        if (k < capacity) {
          out_steps[k] = s;
          out_ranks[k] = rank;
        }
        ++k;
      }
    }
  }
  return k;
}

int anb_plan_clear(anb_net* net) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  drop_graph(net);
  net->plan.clear();
  net->packs.clear();
  return ANB_OK;
}

static int resolve(anb_net* net, const char* kernel, unsigned grid, unsigned block, unsigned smem,
                   Launch* out) {
  if (!net || !kernel) return fail(ANB_ERR_ARG, "NULL argument");
  if (!net->module) return fail(ANB_ERR_STATE, "no module loaded");
  if (grid == 0 || block == 0 || block > 1024) return fail(ANB_ERR_ARG, "bad launch shape");
  Launch l;
  l.name = kernel;
  l.grid = grid;
  l.block = block;
  l.smem = smem;
  CUresult r = g_drv.moduleGetFunction(&l.fn, net->module, kernel);
  if (r != CUDA_SUCCESS) return fail(ANB_ERR_ARG, std::string("kernel not found: ") + kernel);
  // the 48 KB default covers static and dynamic shared memory together:
  // opt in whenever the dynamic part comes near it
  if (smem > 32 * 1024)
    ANB_CU(g_drv.funcSetAttribute(l.fn, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, (int)smem));
  *out = l;
  return ANB_OK;
}

int anb_plan_add(anb_net* net, const char* kernel, unsigned grid, unsigned block,
                 unsigned shared_bytes) {
  return anb_plan_add_concurrent(net, kernel, grid, block, shared_bytes, 0);
}

int anb_plan_add_concurrent(anb_net* net, const char* kernel, unsigned grid, unsigned block,
                            unsigned shared_bytes, int group) {
  Launch l;
  int rc = resolve(net, kernel, grid, block, shared_bytes, &l);
  if (rc) return rc;
  if (group < 0) return fail(ANB_ERR_ARG, "group must be >= 0");
  l.group = group;
  drop_graph(net);
  net->plan.push_back(l);
  return ANB_OK;
}

int anb_set_local_kernel_cooperative(anb_net* net, const char* kernel, unsigned block,
                                     unsigned shared_bytes, unsigned* grid_out) {
  if (!net || !kernel) return fail(ANB_ERR_ARG, "NULL argument");
  Launch l;
  int rc = resolve(net, kernel, 1, block, shared_bytes, &l);
  if (rc) return rc;
  int per_sm = 0, sms = 0;
  ANB_CU(g_drv.maxActiveBlocks(&per_sm, l.fn, (int)block, (size_t)shared_bytes));
  ANB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, net->device));
  if (per_sm < 1) return fail(ANB_ERR_ARG, std::string(kernel) + ": no CTA fits on an SM");
  l.grid = (unsigned)(per_sm * sms);
  l.cooperative = true;
  net->local = l;
  net->has_local = true;
  if (grid_out) *grid_out = l.grid;
  return ANB_OK;
}

int anb_plan_add_bsr_tc(anb_net* net, const char* prefix, const char* x_array,
                        const char* y_array, int n_block_rows, int batch, int n_pre, int n_post,
                        int group) {
  if (!net || !prefix || !x_array || !y_array) return fail(ANB_ERR_ARG, "NULL argument");
  if (batch < 16 || batch > 256 || batch % 16)
    return fail(ANB_ERR_ARG, "batch must be a multiple of 16 between 16 and 256");
  if (n_block_rows < 0 || n_pre <= 0 || n_post <= 0 || n_block_rows * 64 < n_post)
    return fail(ANB_ERR_ARG, "inconsistent block-sparse sizes");
  if (group < 0) return fail(ANB_ERR_ARG, "group must be >= 0");
  Launch l;
  l.name = std::string(prefix) + "_bsr_tc";
  l.op = kOpBsrTc;
  l.group = group;
  const std::string p(prefix);
  const std::string names[6] = {p + "__brow", p + "__bcol", p + "__tiles", x_array, p + "__xt",
                                y_array};
  const size_t n_bcols = (size_t)(n_pre + 63) / 64;
  for (int i = 0; i < 6; ++i) {
    Array* a = find(net, names[i].c_str());
    if (!a) return fail(ANB_ERR_ARG, "unknown array " + names[i]);
    l.arr[i] = names[i];
  }
  if (find(net, names[3].c_str())->bytes < sizeof(float) * (size_t)batch * n_pre)
    return fail(ANB_ERR_ARG, names[3] + " holds fewer than batch x n_pre floats");
  if (find(net, names[5].c_str())->bytes < sizeof(float) * (size_t)batch * n_post)
    return fail(ANB_ERR_ARG, names[5] + " holds fewer than batch x n_post floats");
  if (find(net, names[4].c_str())->bytes < 2 * n_bcols * (size_t)batch * 64)
    return fail(ANB_ERR_ARG, names[4] + " is too small for the packed rates");
  l.iarg[0] = n_block_rows;
  l.iarg[1] = batch;
  l.iarg[2] = n_pre;
  l.iarg[3] = n_post;
  drop_graph(net);
  net->plan.push_back(l);
  return ANB_OK;
}

int anb_plan_add_bsr_shared(anb_net* net, const char* prefix, const char* tiles_array,
                            const char* y_array, int n_block_rows, int parts, int batch, int n_post) {
  if (!net || !prefix || !tiles_array || !y_array) return fail(ANB_ERR_ARG, "NULL argument");
  if (batch < 16 || batch > 256 || batch % 16)
    return fail(ANB_ERR_ARG, "batch must be a multiple of 16 between 16 and 256");
  if (n_block_rows < 0 || parts < 1 || n_post <= 0 || n_block_rows * 64 < n_post)
    return fail(ANB_ERR_ARG, "inconsistent block-sparse sizes");
  Launch l;
  const std::string p(prefix);
  l.name = p + "_bsr_tc";
  l.op = kOpBsrShared;
  const std::string names[6] = {p + "__brow", p + "__bcol", p + "__tiles", "", tiles_array, y_array};
  for (int i = 0; i < 6; ++i) {
    if (i != 3 && !find(net, names[i].c_str())) return fail(ANB_ERR_ARG, "unknown array " + names[i]);
    l.arr[i] = names[i];
  }
  if (find(net, names[0].c_str())->bytes < 4 * ((size_t)n_block_rows * parts + 1))
    return fail(ANB_ERR_ARG, names[0] + " holds too few runs of blocks");
  if (find(net, y_array)->bytes < sizeof(float) * (size_t)batch * n_post)
    return fail(ANB_ERR_ARG, std::string(y_array) + " holds fewer than batch x n_post floats");
  l.iarg[0] = n_block_rows;
  l.iarg[1] = batch;
  l.iarg[2] = parts;
  l.iarg[3] = n_post;
  drop_graph(net);
  net->plan.push_back(l);
  return ANB_OK;
}

int anb_plan_pack(anb_net* net, const char* x_array, const char* tiles_array, int batch, int n_pre,
                  int first_block) {
  if (!net || !x_array || !tiles_array) return fail(ANB_ERR_ARG, "NULL argument");
  if (batch < 16 || batch > 256 || batch % 16 || n_pre <= 0 || first_block < 0)
    return fail(ANB_ERR_ARG, "inconsistent sizes");
  Array* x = find(net, x_array);
  Array* t = find(net, tiles_array);
  if (!x || !t) return fail(ANB_ERR_ARG, std::string("unknown array ") + (x ? tiles_array : x_array));
  if (x->bytes < sizeof(float) * (size_t)batch * n_pre ||
      t->bytes < 2 * ((size_t)first_block + (n_pre + 63) / 64) * batch * 64)
    return fail(ANB_ERR_ARG, "the arrays are too small for the rates and their tiles");
  anb_net::Pack p;
  p.x = x_array;
  p.tiles = tiles_array;
  p.batch = batch;
  p.n_pre = n_pre;
  p.first_block = first_block;
  net->packs.push_back(p);
  return ANB_OK;
}

int anb_set_local_kernel(anb_net* net, const char* kernel, unsigned grid, unsigned block,
                         unsigned shared_bytes) {
  Launch l;
  int rc = resolve(net, kernel, grid, block, shared_bytes, &l);
  if (rc) return rc;
  net->local = l;
  net->has_local = true;
  return ANB_OK;
}

int anb_set_local_kernel_ex(anb_net* net, const char* kernel, unsigned grid, unsigned block,
                            unsigned shared_bytes, unsigned cluster) {
  if (cluster == 0 || cluster > 16 || grid % cluster != 0)
    return fail(ANB_ERR_ARG, "cluster size must divide the grid and be at most 16");
  Launch l;
  int rc = resolve(net, kernel, grid, block, shared_bytes, &l);
  if (rc) return rc;
  l.cluster = cluster;
  if (cluster > 1) {
    if (cluster > 8)
      ANB_CU(g_drv.funcSetAttribute(l.fn, CU_FUNC_ATTRIBUTE_NON_PORTABLE_CLUSTER_SIZE_ALLOWED, 1));
    CUlaunchAttribute attr;
    std::memset(&attr, 0, sizeof(attr));
    attr.id = CU_LAUNCH_ATTRIBUTE_CLUSTER_DIMENSION;
    attr.value.clusterDim.x = cluster;
    attr.value.clusterDim.y = 1;
    attr.value.clusterDim.z = 1;
    CUlaunchConfig cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDimX = grid;
    cfg.gridDimY = 1;
    cfg.gridDimZ = 1;
    cfg.blockDimX = block;
    cfg.blockDimY = 1;
    cfg.blockDimZ = 1;
    cfg.sharedMemBytes = shared_bytes;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    ANB_CU(g_drv.maxActiveClusters(&clusters, l.fn, &cfg));
    if (clusters < 1)
      return fail(ANB_ERR_ARG, "a cluster of " + std::to_string(cluster) + " CTAs with " +
                                   std::to_string(shared_bytes) +
                                   " bytes of shared memory each cannot be scheduled");
  }
  net->local = l;
  net->has_local = true;
  return ANB_OK;
}

int anb_set_pdl(anb_net* net, int on) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  drop_graph(net);
  net->pdl = on != 0;
  net->pdl_prev = false;
  return ANB_OK;
}

int anb_set_graph_steps(anb_net* net, int steps) {
  if (!net || steps < 0) return fail(ANB_ERR_ARG, "bad argument");
  drop_graph(net);
  net->graph_steps = steps;
  return ANB_OK;
}

int anb_run(anb_net* net, int64_t nsteps) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  if (nsteps < 0) return fail(ANB_ERR_ARG, "negative step count");
  if (nsteps == 0) return ANB_OK;
  if (!net->module) return fail(ANB_ERR_STATE, "no module loaded");
  int rc = ensure_device(net);
  if (rc) return rc;
  rc = bind(net);
  if (rc) return rc;
  if (net->has_local) {
    if (net->local.cooperative) {
      // the grid barrier's counters start at zero (a run that gave up may
      // have left a partial count)
      Array* gb = find(net, "gbar");
      if (gb) ANB_CUDA(cudaMemsetAsync(gb->ptr, 0, gb->bytes, net->stream));
    }
    int64_t done = 0;
    while (done < nsteps) {
      long long t0 = (long long)(net->t + done);
      int n = (int)((nsteps - done) > (1 << 30) ? (1 << 30) : (nsteps - done));
      void* params[] = {&t0, &n};
      rc = net->timing ? timed_launch(net, net->local, params) : launch(net, net->local, params);
      if (rc) return rc;
      done += n;
    }
    net->t += nsteps;
    return ANB_OK;
  }
  for (const auto& p : net->packs) {
    Array* x = find(net, p.x.c_str());
    Array* tl = find(net, p.tiles.c_str());
    if (!x || !tl) return fail(ANB_ERR_STATE, p.x + " or " + p.tiles + " is missing");
    if (anb_bsr_tc_pack_x((const float*)x->ptr, p.batch, p.n_pre,
                          (uint16_t*)tl->ptr + (size_t)p.first_block * p.batch * 64, net->stream) != 0)
      return fail(ANB_ERR_CUDA, "packing of " + p.x + " failed");
    net->pdl_prev = false;
  }
  int64_t remaining = nsteps;
  if (!net->timing && net->graph_steps > 1 && nsteps >= net->graph_steps) {
    rc = build_graph(net);
    if (rc) return rc;
    while (remaining >= net->graph_steps) {
      ANB_CUDA(cudaGraphLaunch(net->graph, net->stream));
      remaining -= net->graph_steps;
    }
  }
  // (what kernels read before they wait for their predecessor may have been
  // written by the copies or kernels before this run)
  net->pdl_prev = false;
  for (int64_t s = 0; s < remaining; ++s) {
    rc = run_plan_once(net);
    if (rc) return rc;
  }
  net->t += nsteps;
  return ANB_OK;
}

int anb_step(anb_net* net) { return anb_run(net, 1); }

int anb_set_stop_kernel(anb_net* net, int pop, const char* kernel, unsigned grid, unsigned block,
                        int all_mode) {
  Launch l;
  int rc = resolve(net, kernel, grid, block, 0, &l);
  if (rc) return rc;
  if (pop < 0) return fail(ANB_ERR_ARG, "negative population id");
  Array* f = find(net, "stop_flags");
  if (!f || f->bytes < (size_t)(pop + 1) * 8) return fail(ANB_ERR_STATE, "stop_flags array missing or short");
  for (auto& st : net->stops)
    if (st.pop == pop) {
      st.l = l;
      st.all = all_mode ? 1 : 0;
      return ANB_OK;
    }
  net->stops.push_back({pop, l, all_mode ? 1 : 0});
  return ANB_OK;
}

int anb_run_until(anb_net* net, int64_t steps, const int* populations, int n_populations, int or_and,
                  int64_t* done, int* stopped) {
  if (!net || !done || !stopped || (n_populations > 0 && !populations))
    return fail(ANB_ERR_ARG, "NULL argument");
  if (steps < 0 || n_populations < 0) return fail(ANB_ERR_ARG, "negative count");
  *done = 0;
  *stopped = 0;
  if (net->stops.empty()) {                // no stop condition in the network: plain run
    int rc = anb_run(net, steps);
    if (rc) return rc;
    *done = steps;
    return ANB_OK;
  }
  if (net->has_local) return fail(ANB_ERR_STATE, "stop conditions need the grid engine");
  Array* f = find(net, "stop_flags");
  if (!f) return fail(ANB_ERR_STATE, "stop_flags array missing");
  std::vector<const anb_net::Stop*> checked;
  for (int i = 0; i < n_populations; ++i)
    for (const auto& st : net->stops)
      if (st.pop == populations[i]) checked.push_back(&st);
  std::vector<long long> flags(f->bytes / 8);
  for (int64_t n = 0; n < steps; ++n) {
    int rc = anb_run(net, 1);
    if (rc) return rc;
    ++*done;
    bool stop = or_and != 0;
    if (!checked.empty()) {
      for (const auto* st : checked) {
        rc = launch(net, st->l, nullptr);
        if (rc) return rc;
      }
      ANB_CUDA(cudaMemcpyAsync(flags.data(), f->ptr, flags.size() * 8, cudaMemcpyDeviceToHost,
                               net->stream));
      ANB_CUDA(cudaStreamSynchronize(net->stream));
      for (const auto* st : checked) {
        const bool marked = flags[st->pop] == (long long)net->t;
        const bool cond = st->all ? !marked : marked;
        stop = or_and ? (stop && cond) : (stop || cond);
      }
    }
    // as in the reference, a list of populations without any stop condition
    // ends an "and" run after one step
    if (stop && n_populations > 0) {
      *stopped = 1;
      break;
    }
  }
  return ANB_OK;
}

int anb_synchronize(anb_net* net) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  int rc = ensure_device(net);
  if (rc) return rc;
  int code = 0;
  rc = anb_device_error(net, &code);   // waits for the stream
  if (rc) return rc;
  if (net->timing) {
    rc = collect_times(net);
    if (rc) return rc;
  }
  switch (code) {
    case 0:
      return ANB_OK;
    case 1:  // ANB_DEVERR_BARRIER_TIMEOUT
      return fail(ANB_ERR_TIMEOUT, "a bounded device-side wait gave up (barrier timeout, "
                                   "device error code 1); clear it with anb_clear_device_error");
    case 2:  // ANB_DEVERR_INDEX
      return fail(ANB_ERR_STATE, "a kernel met an index out of range (device error code 2)");
    case 3:  // ANB_DEVERR_MONITOR_OVERFLOW
      return fail(ANB_ERR_STATE, "a monitor's device ring was full (device error code 3)");
    default:
      return fail(ANB_ERR_STATE, "device-side error code " + std::to_string(code));
  }
}

int anb_device_error(anb_net* net, int* code) {
  if (!net || !code) return fail(ANB_ERR_ARG, "NULL argument");
  Array* a = find(net, "err");
  int v[4] = {0, 0, 0, 0};
  int rc = read_staged(net, a->ptr, v, sizeof(v));
  if (rc) return rc;
  *code = v[0];
  return ANB_OK;
}

int anb_clear_device_error(anb_net* net) { return anb_array_fill_zero(net, "err"); }

namespace {
// Reads the flush buffer (twice the L2 size) so that L2 holds only clean lines
// of it afterwards: the next kernel starts with a cold cache and no dirty
// lines to write back. The sink is written only if the sum of the buffer
// equals an impossible value, which keeps the reads alive.
__global__ void anb_flush_read(const uint4* __restrict__ p, size_t n, unsigned* sink) {
  unsigned acc = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const uint4 v = p[i];
    acc ^= v.x ^ v.y ^ v.z ^ v.w;
  }
  if (acc == 0x9e3779b9u) *sink = acc;
}
}  // namespace

// Streaming read of n 16-byte words, four loads in flight per thread, no
// reuse (evict-first loads): the cold-read floor of a kernel that must read
// that many bytes once.
__global__ void anb_stream_read_kernel(const uint4* __restrict__ p, size_t n, unsigned* sink) {
  unsigned acc = 0;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n; i += 4 * stride) {
    const uint4 a = __ldcs(p + i), b = __ldcs(p + i + stride), c = __ldcs(p + i + 2 * stride),
                d = __ldcs(p + i + 3 * stride);
    acc ^= a.x ^ b.y ^ c.z ^ d.w;
  }
  for (; i < n; i += stride) acc ^= __ldcs(p + i).x;
  if (acc == 0x9e3779b9u) *sink = acc;
}

int anb_flush_l2(anb_net* net) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  int rc = ensure_device(net);
  if (rc) return rc;
  if (!net->flush_buf) {
    int dev = 0, l2 = 0;
    ANB_CUDA(cudaGetDevice(&dev));
    ANB_CUDA(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev));
    net->flush_bytes = (size_t)(l2 > 0 ? l2 : (128 << 20)) * 2;
    cudaError_t e = cudaMalloc(&net->flush_buf, net->flush_bytes + 256);
    if (e != cudaSuccess) {
      net->flush_buf = nullptr;
      return fail(ANB_ERR_ALLOC, "L2 flush buffer");
    }
    ANB_CUDA(cudaMemsetAsync(net->flush_buf, 0x5a, net->flush_bytes + 256, net->stream));
  }
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, net->device);
  anb_flush_read<<<sms * 4, 512, 0, net->stream>>>(
      reinterpret_cast<const uint4*>(net->flush_buf), net->flush_bytes / 16,
      reinterpret_cast<unsigned*>(static_cast<char*>(net->flush_buf) + net->flush_bytes));
  ANB_CUDA(cudaGetLastError());
  return ANB_OK;
}

int anb_stream_read(anb_net* net, size_t bytes, int reps, double* ms_median) {
  if (!net || !ms_median || bytes < 16 || reps < 1 || reps > 64) return fail(ANB_ERR_ARG, "bad arguments");
  int rc = ensure_device(net);
  if (rc) return rc;
  void* buf = nullptr;
  const size_t n = bytes / 16;
  if (cudaMalloc(&buf, n * 16 + 16) != cudaSuccess) return fail(ANB_ERR_ALLOC, "stream buffer");
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  std::vector<float> ts;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, net->device);
  cudaError_t e = cudaMemsetAsync(buf, 0x33, n * 16 + 16, net->stream);
  if (e == cudaSuccess) e = cudaEventCreate(&e0);
  if (e == cudaSuccess) e = cudaEventCreate(&e1);
  for (int r = 0; r < reps && e == cudaSuccess; ++r) {
    rc = anb_flush_l2(net);
    if (rc) break;
    cudaEventRecord(e0, net->stream);
    anb_stream_read_kernel<<<sms * 8, 256, 0, net->stream>>>(
        reinterpret_cast<const uint4*>(buf), n, reinterpret_cast<unsigned*>(static_cast<char*>(buf) + n * 16));
    cudaEventRecord(e1, net->stream);
    e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    ts.push_back(ms);
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaFree(buf);
  if (rc) return rc;
  if (e != cudaSuccess) return fail(ANB_ERR_CUDA, std::string("stream read: ") + cudaGetErrorString(e));
  std::sort(ts.begin(), ts.end());
  *ms_median = ts[ts.size() / 2];
  return ANB_OK;
}

// Tile-fill floor: every CTA streams its share of `copies` tiles of
// `tile_bytes`, picked pseudo-randomly from `n_tiles` tiles of an L2-resident
// buffer, into `stages` shared-memory stages with bulk copies completing on
// one mbarrier per stage. Lane 0 of warp w issues the copies of stage w (one
// thread's bulk copies are served one after another, so every stage has its
// own issuing thread): the floor of a kernel that stages such tiles from L2
// through shared memory. Every wait is bounded; a timeout is reported in
// `err`.
__global__ void anb_tile_fill_kernel(const unsigned char* __restrict__ src, int n_tiles,
                                     unsigned tile_bytes, int copies, int stages, int* err,
                                     unsigned* sink) {
  extern __shared__ __align__(128) unsigned char anb_tf_smem[];
  __shared__ __align__(8) unsigned long long full[16];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) != 0 || w >= stages) return;
  const unsigned mb = (unsigned)__cvta_generic_to_shared(&full[w]);
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  auto wait = [&](unsigned parity) {
    unsigned done = 0;
    for (int it = 0; it < (1 << 24) && !done; ++it)
      asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                   : "=r"(done) : "r"(mb), "r"(parity) : "memory");
    if (!done) atomicExch(err, 1);
    return done != 0;
  };
  unsigned char* dst = anb_tf_smem + (size_t)w * tile_bytes;
  unsigned acc = 0;
  int k = 0;                                   // uses of this stage
  for (long long i = blockIdx.x + (long long)w * gridDim.x; i < copies;
       i += (long long)stages * gridDim.x, ++k) {
    if (k > 0) {
      if (!wait((unsigned)(k - 1) & 1u)) return;
      acc += dst[0];
    }
    const unsigned t = (unsigned)(((unsigned long long)i * 2654435761ull) % (unsigned)n_tiles);
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }"
                 ::"r"(mb), "r"(tile_bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src + (size_t)t * tile_bytes),
                 "r"(tile_bytes), "r"(mb)
                 : "memory");
  }
  if (k > 0) {
    if (!wait((unsigned)(k - 1) & 1u)) return;
    acc += dst[0];
  }
  if (acc == 0x9e3779b9u) *sink = acc;
}

int anb_tile_fill(anb_net* net, int n_tiles, int tile_bytes, int copies, int ctas_per_sm, int stages,
                  int reps, double* ms_median) {
  if (!net || !ms_median || n_tiles < 1 || tile_bytes < 16 || tile_bytes % 16 || tile_bytes > (64 << 10) ||
      copies < 1 || ctas_per_sm < 1 || ctas_per_sm > 8 || stages < 1 || stages > 16 || reps < 1 || reps > 64 ||
      (size_t)stages * tile_bytes > (200u << 10))
    return fail(ANB_ERR_ARG, "bad arguments");
  int rc = ensure_device(net);
  if (rc) return rc;
  const size_t bytes = (size_t)n_tiles * tile_bytes;
  void* buf = nullptr;
  if (cudaMalloc(&buf, bytes + 64) != cudaSuccess) return fail(ANB_ERR_ALLOC, "tile buffer");
  int* err = reinterpret_cast<int*>(static_cast<char*>(buf) + bytes);
  unsigned* sink = reinterpret_cast<unsigned*>(static_cast<char*>(buf) + bytes + 16);
  const size_t smem = (size_t)stages * tile_bytes;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, net->device);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  std::vector<float> ts;
  cudaError_t e = cudaMemsetAsync(buf, 0x33, bytes + 64, net->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, 4, net->stream);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(anb_tile_fill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaEventCreate(&e0);
  if (e == cudaSuccess) e = cudaEventCreate(&e1);
  const int grid = sms * ctas_per_sm;
  // one untimed pass brings the tiles into L2
  for (int r = 0; r <= reps && e == cudaSuccess; ++r) {
    cudaEventRecord(e0, net->stream);
    anb_tile_fill_kernel<<<grid, 32 * stages, smem, net->stream>>>(static_cast<const unsigned char*>(buf), n_tiles,
                                                         (unsigned)tile_bytes, copies, stages, err, sink);
    cudaEventRecord(e1, net->stream);
    e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    if (r > 0) ts.push_back(ms);
  }
  int h_err = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&h_err, err, 4, cudaMemcpyDeviceToHost);
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaFree(buf);
  if (e != cudaSuccess) return fail(ANB_ERR_CUDA, std::string("tile fill: ") + cudaGetErrorString(e));
  if (h_err) return fail(ANB_ERR_TIMEOUT, "tile fill: a bulk-copy wait timed out");
  std::sort(ts.begin(), ts.end());
  *ms_median = ts[ts.size() / 2];
  return ANB_OK;
}

int anb_kernel_timing(anb_net* net, int enable) {
  if (!net) return fail(ANB_ERR_ARG, "net is NULL");
  int rc = ensure_device(net);
  if (rc) return rc;
  ANB_CUDA(cudaStreamSynchronize(net->stream));
  rc = collect_times(net);
  if (rc) return rc;
  net->timing = enable != 0;
  if (enable) {
    net->times.clear();
    net->time_index.clear();
  }
  return ANB_OK;
}

int anb_kernel_time_count(anb_net* net, int* count) {
  if (!net || !count) return fail(ANB_ERR_ARG, "NULL argument");
  *count = (int)net->times.size();
  return ANB_OK;
}

int anb_kernel_time_get(anb_net* net, int index, char* name, size_t name_len, double* total_ms,
                        int64_t* launches) {
  if (!net || index < 0 || index >= (int)net->times.size())
    return fail(ANB_ERR_ARG, "bad kernel index");
  const KernelTime& k = net->times[index];
  if (name && name_len) {
    std::strncpy(name, k.name.c_str(), name_len - 1);
    name[name_len - 1] = '\0';
  }
  if (total_ms) *total_ms = k.total_ms;
  if (launches) *launches = k.launches;
  return ANB_OK;
}

}  // extern "C"

// device-side connectivity construction (uses the helpers above)
#include "connect.cuh"
