// Recording and replaying a training step.  The executor's node loop costs the host 5-9 us per operator call (Python,
// ctypes, launch), which is what bounds every graph whose kernels are shorter than that: a 52-launch MLP step took 0.54 ms
// of which the GPU worked 0.1, Inception-v3 at batch 2 (1289 launches) 8.8 ms.  Here one step's launches are collected once
// into a CUDA graph (with the programmatic launch edges of launch_dep) and replayed with one call.
//
// The graph is built node by node in the launch functions, a chain in the order of the calls; nothing of the step executes
// meanwhile.  It is not captured from a stream: while any stream is captured, a wait for the whole device is an error in every
// thread, in code that knows nothing of this library too, and ends the capture.  What has to differ from an ordinary call is
// listed at the declarations in common.h.  A replay leaves the library's books as the step itself would: every tensor the
// step writes gets a new write version, the packs it overwrites in the plans no longer count as what an ordinary call left
// there, the launches are counted, and the maxima of the parameters stay known.
#include "common.h"
#include <algorithm>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace tf {

thread_local StepGraph* t_recording = nullptr;
static std::atomic<uint64_t> g_layout_epoch{1};
void bump_layout_epoch() { g_layout_epoch.fetch_add(1, std::memory_order_relaxed); }
int tensor_path_error();
int launch_waiting();
void drop_held();
void tc_recording_begins();
bool dp_active();

constexpr int kZeroedWords = 12288;       // maxima of a step's tensors: one word per tracked write (Inception-v4: about 900)
constexpr int kSeedWords = 1022;          // dropout calls of a step
constexpr int kCarries = 1024;            // parameters whose maximum crosses steps

struct StepGraph {
  cudaStream_t stream = nullptr;          // the calls of the recording name it (name_stream)
  cudaGraph_t graph = nullptr;
  cudaGraphNode_t last = nullptr;         // the node every next one waits for
  bool last_is_kernel = false;
  cudaGraphExec_t exec = nullptr;
  uint32_t* words = nullptr;              // [zeroed words][c1, c2][seeds]
  int used = 0;
  const char* refused = nullptr;          // why the step cannot be recorded
  std::vector<unsigned> seeds;            // of the recorded step, in call order
  bool has_adam = false;
  float c1 = 0.f, c2 = 0.f;
  std::unordered_map<size_t, std::vector<void*>> free_blocks;
  std::vector<std::pair<void*, std::vector<char>>> owned;      // tables that its kernels read, and the memory they were uploaded from
  std::vector<const void*> written;
  std::vector<const void**> made;         // sources of the packs and indices in plans that the graph writes
  std::vector<AmaxCarry> carries;
  long long launches = 0;
  uint64_t epoch = 0;
  uint64_t id = 0;
  cudaStream_t home = nullptr;            // where it is replayed, and whose scratch its kernels use
};
static std::atomic<uint64_t> g_recordings{0};
uint64_t recording_id() { return t_recording ? t_recording->id : 0; }

void* recording_own(std::vector<char>& bytes) {
  StepGraph* g = t_recording;
  t_recording = nullptr;                  // not a block that was freed in the recording: its kernels still write those
  void* p = pool_alloc(bytes.size());
  t_recording = g;
  if (!p) return nullptr;
  g->owned.emplace_back(p, std::move(bytes));
  const std::vector<char>& kept = g->owned.back().second;
  if (cudaMemcpyAsync(p, kept.data(), kept.size(), cudaMemcpyHostToDevice, g->home) != cudaSuccess) { cudaGetLastError(); return nullptr; }
  return p;
}
void recording_refuse(const char* why) { if (!t_recording->refused) t_recording->refused = why; }
uint32_t* recording_word() {
  StepGraph* g = t_recording;
  if (g->used >= kZeroedWords) { recording_refuse("more tracked tensors than a recording has words for"); return g->words; }
  return g->words + g->used++;
}
void* recording_take_block(size_t bytes) {
  auto it = t_recording->free_blocks.find(bytes);
  if (it == t_recording->free_blocks.end() || it->second.empty()) return nullptr;
  void* p = it->second.back();
  it->second.pop_back();
  return p;
}
void recording_keep_block(void* p, size_t bytes) { t_recording->free_blocks[bytes].push_back(p); }
const uint32_t* recording_seed(unsigned seed) {
  StepGraph* g = t_recording;
  if ((int)g->seeds.size() >= kSeedWords) { recording_refuse("more dropout calls than a recording has seeds for"); return g->words; }
  g->seeds.push_back(seed);
  return g->words + kZeroedWords + 2 + g->seeds.size() - 1;
}
const float* recording_adam_corrections(float c1, float c2) {
  StepGraph* g = t_recording;
  if (g->has_adam && (g->c1 != c1 || g->c2 != c2)) recording_refuse("two pairs of Adam's bias corrections in one step");
  g->has_adam = true; g->c1 = c1; g->c2 = c2;
  return reinterpret_cast<const float*>(g->words + kZeroedWords);
}
void recording_note_launches(int n) { t_recording->launches += n; }
void recording_note_write(const void* p) { t_recording->written.push_back(p); }
void recording_note_made(const void** source) { t_recording->made.push_back(source); }
cudaStream_t recording_home() { return t_recording->home; }
cudaStream_t recording_stream() { return t_recording->stream; }

// ---- nodes --------------------------------------------------------------------------------------
static cudaError_t recorded(cudaError_t e, cudaGraphNode_t node, bool kernel, bool dependent) {
  StepGraph* g = t_recording;
  if (e == cudaSuccess && g->last) {
    cudaGraphEdgeData edge;
    memset(&edge, 0, sizeof(edge));
    if (dependent && g->last_is_kernel) { edge.type = cudaGraphDependencyTypeProgrammatic; edge.from_port = cudaGraphKernelNodePortProgrammatic; }
    e = cudaGraphAddDependencies_v2(g->graph, &g->last, &node, &edge, 1);
  }
  if (e != cudaSuccess) { recording_refuse(cudaGetErrorString(e)); return e; }
  g->last = node; g->last_is_kernel = kernel;
  return cudaSuccess;
}
static bool recorded_stream(cudaStream_t s) {
  if (s == t_recording->stream) return true;
  recording_refuse("an operator was called on another stream than the recording's");
  return false;
}
cudaError_t recording_add_kernel(const void* kernel, const LaunchShape& l, void** args, cudaStream_t s) {
  if (!recorded_stream(s)) return cudaErrorInvalidResourceHandle;
  cudaKernelNodeParams p;
  memset(&p, 0, sizeof(p));
  p.func = (void*)kernel; p.gridDim = l.grid; p.blockDim = l.block; p.sharedMemBytes = (unsigned)l.smem; p.kernelParams = args;
  cudaGraphNode_t node = nullptr;
  cudaError_t e = cudaGraphAddKernelNode(&node, t_recording->graph, nullptr, 0, &p);
  if (e == cudaSuccess && l.cluster > 0) {
    cudaLaunchAttributeValue v;
    memset(&v, 0, sizeof(v));
    v.clusterDim.x = l.cluster; v.clusterDim.y = 1; v.clusterDim.z = 1;
    e = cudaGraphKernelNodeSetAttribute(node, cudaLaunchAttributeClusterDimension, &v);
  }
  return recorded(e, node, true, l.dependent);
}
cudaError_t clear_on_stream(void* ptr, size_t bytes, cudaStream_t s) {
  if (!t_recording) return cudaMemsetAsync(ptr, 0, bytes, s);
  if (!recorded_stream(s)) return cudaErrorInvalidResourceHandle;
  cudaMemsetParams p;
  memset(&p, 0, sizeof(p));
  p.dst = ptr; p.elementSize = bytes % 4 == 0 ? 4 : 1; p.width = bytes / p.elementSize; p.height = 1;
  cudaGraphNode_t node = nullptr;
  const cudaError_t e = cudaGraphAddMemsetNode(&node, t_recording->graph, nullptr, 0, &p);
  return recorded(e, node, false, false);
}
cudaError_t copy_on_stream(void* to, const void* from, size_t bytes, cudaStream_t s) {
  if (!t_recording) return cudaMemcpyAsync(to, from, bytes, cudaMemcpyDeviceToDevice, s);
  if (!recorded_stream(s)) return cudaErrorInvalidResourceHandle;
  cudaGraphNode_t node = nullptr;
  const cudaError_t e = cudaGraphAddMemcpyNode1D(&node, t_recording->graph, nullptr, 0, to, from, bytes, cudaMemcpyDeviceToDevice);
  return recorded(e, node, false, false);
}

// Values of this replay (bias corrections, seeds) into the words the recorded kernels read; up to 960 per launch by value.
constexpr int kValuesPerLaunch = 960;
struct StepValues { uint32_t v[kValuesPerLaunch]; };
__global__ void __launch_bounds__(256) step_values_kernel(const __grid_constant__ StepValues vals, uint32_t* __restrict__ dst, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = vals.v[i];
}
// End of a recorded step: the maxima of the parameters just written, for the packs of the next step.
struct CarryList { const uint32_t* from[kCarries]; uint32_t* to[kCarries]; };
__global__ void __launch_bounds__(256) step_carry_kernel(const __grid_constant__ CarryList list, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) *list.to[i] = *list.from[i];
}
void amax_of_array(const float* src, int64_t n, uint32_t* word, cudaStream_t s);

// Finished recordings.  The lock is held while one is replayed, freed or made to give up its memory.
static std::mutex g_graphs_mu;
static std::vector<StepGraph*> g_graphs;
// A finished recording writes the data that a plan keeps beside *source.
bool recordings_use(const void* const* source) {
  std::lock_guard<std::mutex> lk(g_graphs_mu);
  for (const StepGraph* g : g_graphs) if (std::binary_search(g->made.begin(), g->made.end(), (const void**)source)) return true;
  return false;
}
static void step_graph_release(StepGraph* g) {
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  if (g->words) pool_free(g->words);
  for (auto& kv : g->free_blocks) for (void* p : kv.second) pool_free(p);
  for (auto& o : g->owned) pool_free(o.first);
  g->owned.clear();
  g->exec = nullptr; g->graph = nullptr; g->words = nullptr;
  g->free_blocks.clear();
  cudaGetLastError();
}
static void step_graph_free(StepGraph* g) {
  {
    std::lock_guard<std::mutex> lk(g_graphs_mu);
    g_graphs.erase(std::remove(g_graphs.begin(), g_graphs.end(), g), g_graphs.end());
  }
  step_graph_release(g);
  delete g;
}
bool recordings_give_up_memory() {
  if (t_recording) return false;         // the blocks would go to that recording
  std::lock_guard<std::mutex> lk(g_graphs_mu);
  if (g_graphs.empty()) return false;
  if (cudaDeviceSynchronize() != cudaSuccess) { cudaGetLastError(); return false; }      // no replay is in flight
  for (StepGraph* g : g_graphs) step_graph_release(g);
  g_graphs.clear();
  return true;
}

// The stream that recorded calls name: one per device, so that a recording neither creates nor destroys one.  Nothing runs on it.
static cudaStream_t name_stream() {
  static std::mutex mu;
  static cudaStream_t streams[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return nullptr; }
  std::lock_guard<std::mutex> lk(mu);
  if (!streams[dev] && cudaStreamCreateWithFlags(&streams[dev], cudaStreamNonBlocking) != cudaSuccess) { cudaGetLastError(); streams[dev] = nullptr; }
  return streams[dev];
}

}  // namespace tf
using namespace tf;

extern "C" {

// Starts recording the calls this thread makes from now on; *graph receives the recording and *stream_cell the stream the
// calls have to be given; the step will be replayed on *replay_stream.  0 = recording, 1 = not possible now (timing on,
// data-parallel exchange active), -1 = error.
int TfStepRecordBegin(void** graph, void** stream_cell, void** replay_stream) {
  TF_REQUIRE(graph && stream_cell && replay_stream && !t_recording, "TfStepRecordBegin: bad arguments, or this thread is recording already");
  flush_deferred();
  if (launch_waiting()) return -1;       // called before, and not for the recording's stream
  if (g_timing_level > 0 || g_sync_every_op || dp_active() || tensor_path_error() != 0) return 1;
  StepGraph* g = new StepGraph;
  g->words = (uint32_t*)pool_alloc(sizeof(uint32_t) * (kZeroedWords + 2 + kSeedWords));
  if (!g->words) { delete g; return 1; }
  g->stream = name_stream();
  if (!g->stream || cudaGraphCreate(&g->graph, 0) != cudaSuccess) {
    step_graph_free(g);
    TF_FAIL("TfStepRecordBegin: no stream or graph could be created");
  }
  g->home = *(cudaStream_t*)replay_stream;
  g->epoch = g_layout_epoch.load();
  g->id = g_recordings.fetch_add(1) + 1;
  t_recording = g;
  tc_recording_begins();
  *graph = g;
  *stream_cell = (void*)g->stream;
  clear_on_stream(g->words, sizeof(uint32_t) * kZeroedWords, g->stream);
  return 0;
}

// Ends the recording.  keep = 0 abandons it.  Returns 0 when *graph can be replayed; 1 when the step could not be recorded
// (the graph is gone and every cached operand counts as out of date: run the step with ordinary calls).
int TfStepRecordEnd(void** graph, int keep) {
  TF_REQUIRE(graph && *graph && t_recording == (StepGraph*)*graph, "TfStepRecordEnd: this thread is not recording that step");
  StepGraph* g = t_recording;
  flush_deferred();
  if (!keep) drop_held();
  else if (launch_held(g->stream)) recording_refuse("the filter gradients that were held back could not be launched");
  bool ok = keep != 0 && !g->refused;
  if (ok) {
    g->carries.resize(kCarries);
    int n = 0;
    ok = amax_take_carries(g->id, g->carries.data(), kCarries, &n);
    if (!ok) recording_refuse("more parameters with a tracked maximum than a recording carries");
    g->carries.resize(n);
    CarryList list;
    int m = 0;
    for (const AmaxCarry& c : g->carries) if (c.from) { list.from[m] = c.from; list.to[m] = c.carry; ++m; }
    if (ok && m) { launch_plain(step_carry_kernel, dim3(1), dim3(256), 0, g->stream, list, m); g->launches += 1; }
  }
  ok = ok && !g->refused;
  if (ok) {
    const cudaError_t e = cudaGraphInstantiate(&g->exec, g->graph, 0);
    if (e != cudaSuccess) { ok = false; recording_refuse(cudaGetErrorString(e)); }
  }
  cudaGraphDestroy(g->graph);
  g->graph = nullptr;
  if (ok && g->epoch != g_layout_epoch.load()) { ok = false; recording_refuse("packed operands moved while the step was recorded"); }
  t_recording = nullptr;
  if (!ok) {
    cudaGetLastError();
    if (keep) set_error("the step cannot be recorded: %s", g->refused);       // an abandoned recording keeps the error that stopped it
    invalidate_all_versions();       // calls of the recording marked operands as packed; nothing ran
    step_graph_free(g);
    *graph = nullptr;
    return 1;
  }
  std::sort(g->written.begin(), g->written.end());
  g->written.erase(std::unique(g->written.begin(), g->written.end()), g->written.end());
  std::sort(g->made.begin(), g->made.end());
  g->made.erase(std::unique(g->made.begin(), g->made.end()), g->made.end());
  std::lock_guard<std::mutex> lk(g_graphs_mu);
  g_graphs.push_back(g);
  return 0;
}

// Replays a recorded step on the stream: nseeds dropout seeds in call order, Adam's beta powers of this step.
// 0 = enqueued, 1 = out of date (record it again), 2 = not possible now (use ordinary calls), -1 = error.
// `params` are the arrays the step updates in place: a carried maximum that is out of date is taken from them.
int TfStepReplay(void* graph, const unsigned* seeds, int nseeds, float b1t, float b2t, const DLArrayHandle* params, int nparams, void** cudaStream) {
  StepGraph* g = (StepGraph*)graph;
  TF_REQUIRE(g && !t_recording, "TfStepReplay: nothing to replay");
  flush_deferred();
  StreamLease lease(g->home);            // no operator of another thread between its launches
  std::lock_guard<std::mutex> lk(g_graphs_mu);
  if (!g->exec) return 1;                // gave up its memory
  if (g->epoch != g_layout_epoch.load()) return 1;
  if (g_timing_level > 0 || g_sync_every_op || dp_active()) return 2;
  TF_REQUIRE(tensor_path_error() == 0, "TfStepReplay: an earlier tensor-core kernel timed out on a barrier; refusing to launch");
  TF_REQUIRE(nseeds == (int)g->seeds.size(), "TfStepReplay: %d seeds for %d dropout calls", nseeds, (int)g->seeds.size());
  cudaStream_t s = stream_of(cudaStream);
  TF_REQUIRE(s == g->home, "TfStepReplay: not the stream the step was recorded for");
  note_compute_stream(s);
  // maxima that no replay of this step left behind: the tensor was written by something else since
  for (const AmaxCarry& c : g->carries) {
    if (amax_carry_valid(c.data)) continue;
    if (const uint32_t* w = amax_tracked(c.data)) {
      TF_CUDA(cudaMemcpyAsync(c.carry, w, 4, cudaMemcpyDeviceToDevice, s));
    } else {
      int64_t n = 0;
      for (int i = 0; i < nparams; ++i) if (params[i] && params[i]->data == c.data) n = numel(params[i]);
      if (!n) return 1;
      TF_CUDA(cudaMemsetAsync(c.carry, 0, 4, s));
      amax_of_array((const float*)c.data, n, c.carry, s);
      TF_AFTER(s, "TfStepReplay");
    }
    amax_set_carry_valid(c.data);
  }
  if (g->has_adam || nseeds > 0) {
    const int total = 2 + nseeds;
    StepValues vals;
    for (int at = 0; at < total; at += kValuesPerLaunch) {
      const int n = std::min(kValuesPerLaunch, total - at);
      for (int i = 0; i < n; ++i) {
        const int k = at + i;
        const float c = k == 0 ? 1.f - b1t : 1.f - b2t;
        if (k < 2) memcpy(&vals.v[i], &c, 4); else vals.v[i] = seeds[k - 2];
      }
      launch_plain(step_values_kernel, dim3(1), dim3(256), 0, s, vals, g->words + kZeroedWords + at, n);
      TF_AFTER(s, "TfStepReplay");
    }
  }
  TF_CUDA(cudaGraphLaunch(g->exec, s));
  g_launches.fetch_add(g->launches, std::memory_order_relaxed);
  bump_versions(g->written.data(), g->written.size());
  for (const void** source : g->made) *source = nullptr;
  for (const AmaxCarry& c : g->carries) if (c.from) amax_set_carry_valid(c.data);
  return 0;
}

int TfStepGraphFree(void* graph) {
  if (graph) step_graph_free((StepGraph*)graph);
  return 0;
}

}  // extern "C"
