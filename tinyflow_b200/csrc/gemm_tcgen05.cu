// Tensor-core path of the dense contractions: a persistent, warp-specialised 3xFP16 GEMM on the
// Blackwell tcgen05 pipeline (TMA -> shared memory -> tcgen05.mma -> TMEM -> registers -> HBM).
//
// 3xFP16.  Every fp32 operand tensor is scaled by a power of two s chosen from its largest magnitude
// (max|a|*s in [2^14, 2^15)), and every element is split once into hi = fp16(a*s) and lo = fp16(a*s - hi)
// by a packing kernel: 22 mantissa bits, the same as a tf32 hi/lo pair, and elements down to 2^-18 of the
// tensor's maximum keep all of them (smaller ones lose absolute precision below 2^-40 of the maximum).
// The GEMM accumulates hi*hi + lo*hi + hi*lo in fp32 TMEM (the dropped lo*lo term is below 2^-22
// relative) and the epilogue multiplies by 1/(s_A*s_B), exact.  fp16 inputs run the tensor pipe at twice
// the tf32 rate and halve the operand bytes.  Packed operands are plain 2-D row-major
// matrices [rows][cols] (cols contiguous) so that one kernel serves every contraction:
//
//   matmul            A, B packed as they lie; the operand's "major" (K contiguous or M/N contiguous)
//                     is a run-time flag that only changes the TMA box shape and the UMMA descriptor.
//   conv forward      activations packed pixel-major [N * frame_h * frame_w][C] with the zero halo
//                     materialised, filters packed [Cout][tap][C]; a filter tap is then a constant
//                     row shift of the activation matrix.  The K loop takes 64 channels at a time and
//                     walks the taps for them: one 2-D TMA box of up to 192 activation rows serves
//                     every tap whose shift lies inside it, and a tap's filter tile is a box of its own.
//                     Outputs computed for halo anchors are discarded by the epilogue.
//   conv backward-data  same kernel on the packed output gradient with the flipped filter
//                     [Cin][tap'][Cout]; a strided 1x1 scatters into a zeroed dx.
//   conv backward-filter  dW[k][c][tap] = sum_rows dy[row][k] * x[row + shift(tap)][c]: both operands
//                     are M/N-major, the reduction runs over pixel rows.
//
// A last wave that is not full, and products of few tiles, cut their reductions over CTAs: raw partial sums, added in a fixed
// order through a workspace or a cluster's shared memory.  No atomics on sums: the same bits on every run.
//
// Kernel roles (384 threads): warps 0 and 11 = TMA producers of A and B, warp 1 = TMEM owner and issuer of the wide MMAs, warp
// 10 = issuer of the narrow ones, warps 2-9 = epilogue (two per TMEM lane quarter, half the columns each).  Shared memory holds
// a ring of A blocks and a ring of B tiles (hi and lo, 128-byte swizzle, 64 halves of K per stage); TMEM holds two accumulator
// sets so that promoting one group of stages to registers overlaps the MMAs of the next.  Every mbarrier wait is bounded: on
// time-out the CTA raises an error flag the host reads, drains its outstanding copies, frees its TMEM and returns.
#include "common.h"
#include <cfloat>
#include <cuda.h>
#include <cuda_fp16.h>
#include <algorithm>
#include <mutex>
#include <type_traits>
#include <unordered_map>
#include <vector>

namespace tf {

// ------------------------------------------------------------------------------------------------
// write versions: lets cached packs detect that their source tensor changed
// ------------------------------------------------------------------------------------------------
static std::mutex g_ver_mu;
static std::unordered_map<const void*, uint64_t> g_versions;
static uint64_t g_ver_counter = 1;
static uint64_t version_locked(const void* p) {
  auto it = g_versions.find(p);
  if (it == g_versions.end()) { g_versions[p] = ++g_ver_counter; return g_ver_counter; }
  return it->second;
}
void note_write(const void* p) {
  if (t_recording) recording_note_write(p);
  std::lock_guard<std::mutex> lk(g_ver_mu);
  g_versions[p] = ++g_ver_counter;
}
uint64_t version_of(const void* p) {
  std::lock_guard<std::mutex> lk(g_ver_mu);
  return version_locked(p);
}
void bump_versions(const void* const* ptrs, size_t n) {
  std::lock_guard<std::mutex> lk(g_ver_mu);
  for (size_t i = 0; i < n; ++i) g_versions[ptrs[i]] = ++g_ver_counter;
}
void invalidate_all_versions() {
  std::lock_guard<std::mutex> lk(g_ver_mu);
  for (auto& kv : g_versions) kv.second = ++g_ver_counter;
}

// producer-tracked maxima: two device words per tensor, handed out from zero-filled chunks.  A third word per tensor
// carries the maximum from one replay of a recorded step to the next, and `rec_*` is the word of the recording that is
// being made (valid inside it only).
struct AmaxSlot {
  uint32_t* words = nullptr; unsigned uses = 0; uint64_t version = 0; int cur = 0;
  uint32_t* carry = nullptr; uint64_t carry_version = 0;
  uint64_t rec = 0; uint32_t* rec_word = nullptr; uint64_t rec_version = 0; bool rec_wants_carry = false;
};
static std::unordered_map<const void*, AmaxSlot> g_amax;
// A key is an array's address, or an odd address in its first word (bound_key): such a word is as old as the array, whoever writes that.
static uint64_t array_version_locked(const void* key) { return version_locked(reinterpret_cast<const void*>(reinterpret_cast<uintptr_t>(key) & ~uintptr_t(3))); }
static uint32_t* g_amax_chunk = nullptr;
static int g_amax_left = 0;
static uint32_t* amax_chunk_words(int n) {
  if (g_amax_left < n) {
    const int kWords = 16384;
    uint32_t* chunk = nullptr;
    if (cudaMalloc((void**)&chunk, kWords * sizeof(uint32_t)) != cudaSuccess || clear_now(chunk, kWords * sizeof(uint32_t)) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    g_amax_chunk = chunk; g_amax_left = kWords;
  }
  uint32_t* w = g_amax_chunk;
  g_amax_chunk += n; g_amax_left -= n;
  return w;
}
static void amax_enter_recording(AmaxSlot& sl) {
  if (sl.rec != recording_id()) { sl.rec = recording_id(); sl.rec_word = nullptr; sl.rec_version = 0; sl.rec_wants_carry = false; }
}
AmaxOut amax_track_begin(const void* data) {
  std::lock_guard<std::mutex> lk(g_ver_mu);
  AmaxSlot& sl = g_amax[data];
  if (t_recording) {
    amax_enter_recording(sl);
    sl.rec_word = recording_word();
    sl.rec_version = array_version_locked(data);
    return AmaxOut{sl.rec_word, nullptr};
  }
  if (!sl.words && !(sl.words = amax_chunk_words(2))) return AmaxOut{};
  const int k = (int)(sl.uses++ & 1u);
  sl.cur = k;
  sl.version = array_version_locked(data);
  return AmaxOut{sl.words + k, sl.words + (k ^ 1)};
}
const uint32_t* amax_tracked(const void* data) {
  std::lock_guard<std::mutex> lk(g_ver_mu);
  auto it = g_amax.find(data);
  if (it == g_amax.end()) return nullptr;
  AmaxSlot& sl = it->second;
  const uint64_t v = array_version_locked(data);
  if (t_recording && sl.rec == recording_id() && sl.rec_word && sl.rec_version == v) return sl.rec_word;
  const uint32_t* found = sl.words && sl.version == v ? sl.words + sl.cur : (sl.carry && sl.carry_version == v ? sl.carry : nullptr);
  if (!t_recording || !found) return found;
  // read before the recorded step has written it: at a replay the value has to come from the step before
  if (!sl.carry && !(sl.carry = amax_chunk_words(1))) return nullptr;
  amax_enter_recording(sl);
  sl.rec_wants_carry = true;
  return sl.carry;
}
bool amax_take_carries(uint64_t recording, AmaxCarry* out, int max, int* count) {
  std::lock_guard<std::mutex> lk(g_ver_mu);
  *count = 0;
  for (auto& kv : g_amax) {
    AmaxSlot& sl = kv.second;
    if (sl.rec != recording) continue;
    if (sl.rec_wants_carry) {
      if (*count >= max) return false;
      const bool rewritten = sl.rec_word && sl.rec_version == array_version_locked(kv.first);     // by a kernel that tracks its maximum, last
      out[(*count)++] = AmaxCarry{kv.first, sl.carry, rewritten ? sl.rec_word : nullptr};
    }
    sl.rec = 0;
  }
  return true;
}
bool amax_carry_valid(const void* data) {
  std::lock_guard<std::mutex> lk(g_ver_mu);
  auto it = g_amax.find(data);
  return it != g_amax.end() && it->second.carry && it->second.carry_version == array_version_locked(data);
}
void amax_set_carry_valid(const void* data) {
  std::lock_guard<std::mutex> lk(g_ver_mu);
  g_amax[data].carry_version = array_version_locked(data);
}

// ------------------------------------------------------------------------------------------------
// device-side primitives (inline PTX)
// ------------------------------------------------------------------------------------------------
constexpr int BM = 128;            // UMMA M (TMEM lanes)
constexpr int kThreads = 320;
constexpr int kNarrowWarp = 10, kBWarp = 11, kGemmThreads = 384;     // one-CTA kernel: two more warps issue
// The two arithmetic modes differ only in the element type of the packed operands.  A stage always holds one
// 128-byte swizzle row of K per tile row (K-major) or 128 bytes of M/N per K row (M/N-major), and is consumed by four
// MMAs; the tile byte sizes are therefore the same in both modes and only the element counts change.
enum { kArithF16 = 0, kArithTF32 = 1 };
template <int AR> struct Arith;
template <> struct Arith<kArithF16> {
  typedef __half Elem;
  static constexpr int kBK = 64;            // elements of K per stage (128 B)
  static constexpr int kGW = 64;            // M/N-major operands: elements of M/N per 128-byte group row
  static constexpr uint32_t kFormat = 0;    // instruction-descriptor operand format: f16
  // M/N-major shared-memory descriptor: 128-byte swizzle with 16-byte atoms (layout type 2), 8-row K groups 1024 B apart
  static constexpr uint32_t kMnLayout = 2, kMnSbo = 1024;
};
template <> struct Arith<kArithTF32> {
  typedef float Elem;
  static constexpr int kBK = 32;
  static constexpr int kGW = 32;
  static constexpr uint32_t kFormat = 2;    // tf32
  // 32-bit M/N-major operands exist only with the 128-byte swizzle of 32-byte atoms (layout type 1): 4-row K groups
  // 512 B apart; the tensor map of such an operand asks for the same swizzle
  static constexpr uint32_t kMnLayout = 1, kMnSbo = 512;
};
static inline int bk_of(int ar) { return ar == kArithTF32 ? 32 : 64; }
static inline int gw_of(int ar) { return ar == kArithTF32 ? 32 : 64; }
static inline int elem_of(int ar) { return ar == kArithTF32 ? 4 : 2; }
constexpr int kGroupIters = 4;     // stages accumulated in TMEM before the epilogue promotes them to registers
// A product of two data tensors (post-ReLU activations times their sparse gradients) is a sum a few large terms dominate,
// so the accumulator is as large as sum|a||b| itself and every truncating tensor-core accumulation into it costs half an
// ulp of THAT: 16 accumulations per group showed up to 16 ulp (3-4 ulp rms) on Inception-v3's filter gradients against
// 3 (0.8) for fp32 FMA.  Such launches promote after every stage (4 accumulations).  Sums with a weight operand have many
// comparable terms of both signs and stay below the fp32 FMA error at 4 stages per group.
constexpr int kGroupItersDataByData = 1;
// kind::tf32 consumes 8 elements of K per instruction, half of kind::f16's 16, and its stages hold half as many: the same
// count of truncating accumulations covers a quarter of the reduction, and the 128-channel 1x1 layers of ResNet-50 (one
// group of 16) came out at 1.05 ulp rms against 0.47 for fp32 FMA.  Two stages per group keep it under twice the FMA error.
constexpr int kGroupItersTF32 = 2;
constexpr long long kWaitCycles = 3000000000ll;   // ~1.5 s at 2 GHz: far beyond any legitimate wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait.  Returns false (and raises *abort_flag) if the barrier does not flip in time or another
// role already aborted.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, long long limit_cycles = kWaitCycles) {
  if (mbar_try_wait(bar, parity)) return true;
  long long t0 = clock64();
  for (;;) {
    for (int i = 0; i < 64; ++i) if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > limit_cycles) { *abort_flag = 1; return false; }
  }
}
// One lane of a converged warp.  tcgen05.mma and the bulk copies take their operands from uniform registers: under a branch the
// compiler knows to be taken by one elected lane of a converged warp it moves them there directly, under `lane == 0` it
// serialises over the (possibly) active lanes first.
__device__ __forceinline__ bool elect_one() {
  uint32_t yes;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(yes));
  return yes != 0;
}
// The same for the warps that issue copies and MMAs.  Nothing their loops do may branch on the outcome: as long as all control
// flow is uniform the compiler keeps stage counters, descriptors and coordinates in uniform registers, where these
// instructions take them from.  So a wait that gives up only marks the role as `bad`, which then issues nothing more and runs
// through the rest of its loop.
__device__ __forceinline__ void mbar_wait_mark(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int& bad) {
  if (!bad && !mbar_wait(bar, parity, abort_flag)) bad = 1;
}
// Non-blocking look at a phase; true: complete (and the data it guards visible to this lane)
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ void tensormap_prefetch(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tcgen05_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
template <int AR>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if (AR == kArithF16) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
  }
}
// The same with descriptors in two words each: only the low word (the address) differs from one MMA to the next
template <int AR>
__device__ __forceinline__ void umma_at(uint32_t tmem_d, uint32_t a_low, uint32_t a_high, uint32_t b_low, uint32_t b_high, uint32_t idesc, uint32_t accumulate) {
  umma<AR>(tmem_d, (uint64_t)a_low | (uint64_t)a_high << 32, (uint64_t)b_low | (uint64_t)b_high << 32, idesc, accumulate);
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ---- CTA pairs (cta_group::2): two CTAs of a cluster on neighbouring SMs compute one 256-row tile; each loads its own 128
// rows of A and HALF of the B tile, and the tensor cores of both SMs read both halves.  All of the pair's loads report to
// the barrier of the pair's first CTA (rank 0), whose MMA warp issues for both.
__device__ __forceinline__ uint32_t cluster_ctarank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of the same shared-memory object in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t smem_of_cta(uint32_t local_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_at(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// tiled load into this CTA's shared memory whose bytes are counted by the barrier at `bar_cluster_addr` (any CTA of the pair)
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar_cluster_addr) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar_cluster_addr) : "memory");
}
// arrives, once the MMAs issued so far have completed, on the barrier at this shared-memory offset in BOTH CTAs of the
// pair: one commit per CTA, each naming that CTA's barrier by its cluster address
__device__ __forceinline__ void tcgen05_commit_pair(uint64_t* bar) {
  const uint32_t local = smem_u32(bar);
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_of_cta(local, 0)) : "memory");
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_of_cta(local, 1)) : "memory");
}
template <int AR>
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if (AR == kArithF16) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
  }
}

// Shared-memory matrix descriptor, descriptor version 1 (Blackwell), 128-byte swizzle:
//   K-major operand : rows of 128 B (64 halves / 32 floats of K), 16-byte atoms (layout type 2), 8-row groups 1024 B
//                     apart (SBO); LBO unused (= 16 B); one MMA advances the start address by 32 B.
//   MN-major operand: [K rows of one stage][128 B of M/N] per column group, column groups one stage of K rows apart
//                     (LBO).  fp16: 16-byte atoms (layout type 2), 8-row K groups 1024 B apart (SBO), one MMA (K = 16)
//                     advances the start address by 2048 B.  tf32: 32-byte atoms (layout type 1), 4-row K groups 512 B
//                     apart, one MMA (K = 8) advances it by 1024 B.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t layout_type) {
  return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)(lbo_bytes >> 4) << 16) | ((uint64_t)(sbo_bytes >> 4) << 32) |
         (1ull << 46) | ((uint64_t)layout_type << 61);
}

// ------------------------------------------------------------------------------------------------
// kernel parameters
// ------------------------------------------------------------------------------------------------
enum { kModeGemm = 0, kModeConv = 1, kModeWgrad = 2 };
enum { kEpiRowMajor = 0, kEpiNchw = 1, kEpiWgrad = 2 };
enum { kAccPair = 0, kAccThree = 1 };
constexpr int kMaxTaps = 49;

struct alignas(128) GemmParams {
  CUtensorMap a_hi, a_lo, b_hi, b_lo;
  int mode, a_mn, b_mn, epi;
  int M, N;                       // valid extents of the output tile grid
  int m_tiles, n_tiles, tap_tiles;
  int k_total;                    // stages of one output tile's whole reduction
  // Schedule.  Tiles [0, full_tiles) are computed whole, round robin over the CTAs (whole waves).  The remaining
  // tail_tiles tiles - a partial wave - either run whole as well (tail_share == 0) or have their
  // tail_tiles * k_total stages cut into one contiguous range of tail_share stages per CTA, so that every SM does the
  // same amount of work; a range may cover pieces of several tiles.  Each piece leaves its raw partial sums in a
  // workspace slot and reduce_partials_kernel adds the pieces of a tile in a fixed order (no atomics: results are
  // bit-identical from run to run).
  int full_tiles, tail_tiles, tail_share, slots_per_cta;
  // tail_pieces > 0 instead: every tail tile is cut at the same stages into this many pieces; a CTA takes tail_run of one tile in
  // a row, and the CTAs of one range of stages lie side by side.
  int tail_pieces, tail_run;
  float* workspace;               // [slot][BN columns][128 rows] fp32
  int chunks_per_tap;             // kModeConv: K stages per tap
  int b_tap_pitch;                // kModeConv: columns per tap in the packed filter
  int ntaps;
  float* out;
  uint32_t *amax, *amax_clear;    // where the epilogue leaves max|out| (null: nobody asked), and the word the next write of `out` will use
  const float* a_scale; const float* b_scale;   // device words: the power-of-two scales the packs were made with
  long long ldc;                  // kEpiRowMajor
  // kEpiNchw: row m -> (image, i, j) in a frame of frame_h x frame_w, stored at output pixel
  // (oi, oj) = (i*out_sh + out_off_h, j*out_sw + out_off_w) of channel plane c: ((image*out_c + c)*out_h + oi)*out_w + oj;
  // rows with i >= valid_h, j >= valid_w or (oi, oj) outside the plane are dropped
  int frame_h, frame_w, valid_h, valid_w, out_c, out_h, out_w, out_sh, out_sw, out_off_h, out_off_w;
  int* err;                       // device-visible error word (mapped host memory)
  // kModeWgrad: M-tile rows are taps_per_tile slots of `slot` input channels of one filter tap each.  slots_per_tap > 1: a tap takes that
  // many slots in a row, and m_tiles is 1
  int slot, taps_per_tile, slots_per_tap;
  double operand_bytes;           // of A and B together (host side)
  int group_iters;                // stages accumulated in TMEM before the epilogue promotes them to registers
  int group_limit;                // most stages of a group, 0: no limit of the launch's own (host side)
  int data_by_data;               // both operands are activations / gradients (filter gradients, X^T dY): host-side hint for group_iters
  // Shared memory: a ring of A blocks and a ring of B tiles.  A filter's taps read the same rows of the activation matrix
  // at different shifts, so in kModeConv an A block holds a_rows >= 128 rows, fetched once, and serves every tap of a run (taps
  // whose shifts lie within a_rows - 128 of one another); a tap's operand is the block's start address plus shift * 128 bytes.
  // Everywhere else a block serves one stage.  b_resident: one B tile per CTA for the whole launch, all its stages kept.
  int a_rows, a_slots, b_slots, b_resident;
  int one_ring;                   // A and B of a stage share slot number and barriers (every block serves one stage)
  const void *pack_a, *pack_b;    // host side: the packs that the operands are (filter gradients)
  int sum_run;                    // pieces that reduce_partials_kernel adds in one run (see reduce_tile)
  int hold;                       // host side: the product may wait for others (a filter gradient; see hold_products)
  int acc_mode;                   // where the accumulators sit in TMEM: kAccPair or kAccThree (see the MMA issuer)
  int cross_groups;               // kAccThree: groups whose cross terms accumulate before they are promoted
  int cluster;                    // > 1: the reduction of every tile is cut over the CTAs of a cluster and added up in shared memory
  // kModeConv, taps in the order they are walked for every chunk of channels (runs one after the other):
  uint32_t tap_word[kMaxTaps];    // row shift inside the run's block | first tap of its run << 8 | last << 9
  int tap_off[kMaxTaps];          // row shift of the run's first tap, applied to A (filter gradients, pair kernel: of the tap itself)
  short tap_col[kMaxTaps];        // first column of the tap's channels in A (space-to-depth packs keep one phase per column block)
  short tap_b[kMaxTaps];          // which tap block of the packed filter the tap multiplies
  short pair_shift[kMaxTaps];     // pair kernel: the tap's own row shift is tap_off + pair_shift
};
constexpr int kMaxASlots = 4, kMaxBSlots = 16, kMaxCluster = 8;
constexpr int kSmemBarriers = 512;
constexpr int kSmemLimit = 232448 - 1024;            // 227 KiB less the slack to align to 1024
static inline int gemm_smem_bytes(const GemmParams& p, int bn) { return p.a_slots * p.a_rows * 256 + p.b_slots * bn * 256 + kSmemBarriers + 1024; }

// One unit of a CTA's work: `kcount` stages of tile `tile` starting at stage k0.  slot < 0: the item is the tile's
// whole reduction and its epilogue stores to the output; otherwise its partial sums go to that workspace slot.
struct WorkItem { int tile, k0, kcount, slot; };
__device__ __forceinline__ int piece_start(const GemmParams& p, int piece) { return (int)((long long)p.k_total * piece / p.tail_pieces); }
// The sequence of items of this CTA; the three warp roles walk it independently and must see the same sequence.
struct WorkIter {
  int tile, u, u1, first_tail_tile;
  __device__ __forceinline__ explicit WorkIter(const GemmParams& p) {
    tile = blockIdx.x;
    u = u1 = first_tail_tile = 0;
    if (p.cluster > 1) return;
    if (p.tail_pieces > 0) {
      const int range = blockIdx.x / p.tail_tiles;
      first_tail_tile = blockIdx.x - range * p.tail_tiles;
      u = range * p.tail_run; u1 = min(u + p.tail_run, p.tail_pieces);
    } else if (p.tail_share > 0) {
      u = blockIdx.x * p.tail_share;
      u1 = min(u + p.tail_share, p.tail_tiles * p.k_total);
      first_tail_tile = u / p.k_total;
    }
  }
  __device__ __forceinline__ bool next(const GemmParams& p, WorkItem& w) {
    if (p.cluster > 1) {                  // one item per CTA: its share of the cluster's tile
      if (tile < 0) return false;
      const int rank = tile % p.cluster;
      w.tile = tile / p.cluster; w.slot = -1;
      w.k0 = (int)((long long)p.k_total * rank / p.cluster);
      w.kcount = (int)((long long)p.k_total * (rank + 1) / p.cluster) - w.k0;
      tile = -1;
      return true;
    }
    const int whole = p.tail_share > 0 ? p.full_tiles : p.full_tiles + p.tail_tiles;
    if (tile < whole) {
      w.tile = tile; w.k0 = 0; w.kcount = p.k_total; w.slot = -1;
      tile += gridDim.x;
      return true;
    }
    if (p.tail_pieces > 0) {
      if (u >= u1) return false;
      w.tile = p.full_tiles + first_tail_tile; w.slot = u * p.tail_tiles + first_tail_tile;
      w.k0 = piece_start(p, u);
      w.kcount = piece_start(p, ++u) - w.k0;
      return true;
    }
    if (u < u1) {
      const int t = u / p.k_total, k0 = u - t * p.k_total;
      const int len = min(p.k_total - k0, u1 - u);
      w.tile = p.full_tiles + t; w.k0 = k0; w.kcount = len;
      w.slot = blockIdx.x * p.slots_per_cta + (t - first_tail_tile);
      u += len;
      return true;
    }
    return false;
  }
};
// tile index -> coordinates; n fastest so consecutive CTAs share the A tile through L2
__device__ __forceinline__ void decode_tile(const GemmParams& p, int tile, int& mt, int& nt, int& tap) {
  nt = tile % p.n_tiles; tile /= p.n_tiles;
  tap = tile % p.tap_tiles;
  mt = tile / p.tap_tiles;
}
// Where row `row_in_tile` of tile (mt, tap) lands in the output: everything of the address but the column term.
struct RowAddr { bool ok; long long base; uint32_t col_stride; };
__device__ __forceinline__ RowAddr row_address(const GemmParams& p, int mt, int tap, int row_in_tile) {
  const long long m = (long long)mt * BM + row_in_tile;
  RowAddr r;
  r.ok = m < p.M; r.base = 0; r.col_stride = 1;
  if (p.epi == kEpiRowMajor) {
    r.base = m * p.ldc;
  } else if (p.epi == kEpiNchw) {
    const int per_img = p.frame_h * p.frame_w;
    const int img = (int)(m / per_img);
    const int rem = (int)(m - (long long)img * per_img), i = rem / p.frame_w, j = rem - i * p.frame_w;
    const int oi = i * p.out_sh + p.out_off_h, oj = j * p.out_sw + p.out_off_w;
    r.ok = r.ok && i < p.valid_h && j < p.valid_w && oi >= 0 && oi < p.out_h && oj >= 0 && oj < p.out_w;
    r.col_stride = (uint32_t)(p.out_h * p.out_w);
    r.base = ((long long)img * p.out_c) * r.col_stride + (long long)oi * p.out_w + oj;
  } else {   // kEpiWgrad: tile row -> (tap slot, input channel c), column n = output channel: out[(n * C + c) * ntaps + tap]
    const int sl = row_in_tile / p.slot, u = tap * p.taps_per_tile + sl, t = u / p.slots_per_tap;
    const int c = (mt + u - t * p.slots_per_tap) * p.slot + row_in_tile - sl * p.slot;
    r.ok = t < p.ntaps && c < p.M;
    r.base = (long long)c * p.ntaps + t;
    r.col_stride = (uint32_t)(p.M * p.ntaps);
  }
  return r;
}

// Per-tap values of a convolution, spread over the lanes of a warp: a look-up by a counter that every lane knows is one
// reduction, where an indexed read of the parameter space is a chain of constant-cache loads in front of every stage.  (A
// reduction and not a shuffle: its result is known to be the same in all lanes, so what is computed from it can stay in
// uniform registers.)
struct TapTable {
  uint32_t v0, v1;
  int lane;
  template <class F> __device__ __forceinline__ TapTable(int n, int lane_, F&& f) : lane(lane_) {
    v0 = lane < n ? f(lane) : 0u;
    v1 = lane + 32 < n ? f(lane + 32) : 0u;
  }
  __device__ __forceinline__ uint32_t at(int i) const { return __reduce_or_sync(0xffffffffu, lane == (i & 31) ? (i < 32 ? v0 : v1) : 0u); }
};
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
// 32 (16) columns of BLOCKS accumulator blocks, block_cols columns apart, of this thread's row, added
template <int NC, int BLOCKS> __device__ __forceinline__ void load_sum(uint32_t taddr, uint32_t block_cols, float2* v) {
  float2 b[BLOCKS > 1 ? BLOCKS - 1 : 1][NC / 2];
  if (NC == 32) {
    tmem_ld32(taddr, reinterpret_cast<float*>(v));
#pragma unroll
    for (int i = 1; i < BLOCKS; ++i) tmem_ld32(taddr + i * block_cols, reinterpret_cast<float*>(b[i - 1]));
  } else {
    tmem_ld16(taddr, reinterpret_cast<float*>(v));
#pragma unroll
    for (int i = 1; i < BLOCKS; ++i) tmem_ld16(taddr + i * block_cols, reinterpret_cast<float*>(b[i - 1]));
  }
  tmem_ld_wait();
#pragma unroll
  for (int i = 1; i < BLOCKS; ++i)
#pragma unroll
    for (int q = 0; q < NC / 2; ++q) v[q] = __fadd2_rn(v[q], b[i - 1][q]);
}

// What bounds it.  A K step of 16 is 192 tensor cycles at BN = 128 (N = 2*BN and N = BN).  Its operands are read from shared
// memory at 128 bytes per cycle: 12 KB for the wide and 8 KB for the narrow instruction, 160 cycles; TMA writes another 64 KB per
// stage of four K steps, 512 cycles, so with one block per stage shared memory alone takes 1152 cycles against 768 of the
// tensor pipe, and that is what long reductions ran at (1160 measured).  Runs of taps fetch the activation rows once for up to 9
// stages (36 KB a stage for a 3x3 window of a 28-wide image) and filters of one tile that fit stay in shared memory: with
// 512 channels, 28 x 28, 3x3, batch 64 the product went from 625 to 548 us, with 64 channels, 224 x 224, from 1128 to 886.
// Short reductions are bound by start and epilogue: 4000 cycles to the first MMA, 2500-4000 from the last to the end.
template <int BN, int AR>
__global__ void __launch_bounds__(kGemmThreads, 1) gemm3x_kernel(const __grid_constant__ GemmParams p) {
  using T = Arith<AR>;
  constexpr int BK = T::kBK;
  constexpr uint32_t kGroupStride = BK * 128;               // M/N-major operands: bytes between 128-byte-wide column groups
  constexpr int kTmemCols = 512;                            // all of it: one CTA per SM
  constexpr bool kSets3 = BN == 64;                         // room for two complete sets of three accumulator blocks
  constexpr int kSetCols = kSets3 ? 3 * BN : 2 * BN;
  constexpr int kBTile = BN * 128, kBSlot = 2 * kBTile;     // the hi and the lo tile, in the order the accumulators ask for
  const bool three = !kSets3 && p.acc_mode == kAccThree;
  // Main plus first cross term and the second cross term accumulate into different blocks (unless kAccPair puts them into
  // one), so two warps issue them, each at its own pace.
  const int issuers = kSets3 || three ? 2 : 1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int a_half = p.a_rows * 128, a_slot_bytes = 2 * a_half;       // hi rows, then lo rows
  uint8_t* const b_smem = smem + p.a_slots * a_slot_bytes;
  uint64_t* a_full = reinterpret_cast<uint64_t*>(b_smem + p.b_slots * kBSlot);
  uint64_t* a_empty = a_full + kMaxASlots;
  uint64_t* b_full = a_empty + kMaxASlots;
  uint64_t* b_empty = b_full + kMaxBSlots;
  uint64_t* acc_full = b_empty + kMaxBSlots;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* cross_empty = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(cross_empty + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (warp == 0) {         // the whole warp: one thread took 500 cycles over it
    constexpr int kBars = 2 * kMaxASlots + 2 * kMaxBSlots + 5;
    for (int i = lane; i < kBars; i += 32) {
      const int k = i - 2 * kMaxASlots, j = k - 2 * kMaxBSlots;
      const int count = k < 0 ? (i < kMaxASlots ? 1 : issuers) : j < 0 ? (k < kMaxBSlots ? (p.one_ring ? 2 : 1) : issuers) : j < 2 ? issuers : 8;
      mbar_init(&a_full[i], count);
    }
    if (lane == 0) *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  // Everything up to grid_dep_sync() in the roles below (barriers, TMEM, tap tables) overlaps the tail of the kernel in front.

  if (warp == 0 || warp == kBWarp) {
    // ===================== TMA producer =====================
    // the whole warp walks the work and waits; one elected lane issues the copies
    {
      int as = 0, bs = 0;
      uint32_t aph = 0, bph = 0;
      uint32_t armed_a = 0, armed_b = 0, phase_a = 0, phase_b = 0;         // per slot: filled at least once, phase of the last fill
      int bad = 0;
      const bool do_a = warp == 0, do_b = !do_a;
      bool b_loaded = false;
      int group = 0;                      // as the MMA issuer counts them: the parity decides the order of the B tiles
      const bool conv = p.mode == kModeConv;
      const int period = conv ? p.ntaps : 1;
      const TapTable words(conv ? p.ntaps : 0, lane, [&](int t) { return p.tap_word[t]; });
      const TapTable offs(conv ? p.ntaps : 0, lane, [&](int t) { return (uint32_t)p.tap_off[t]; });
      const TapTable cols(conv ? p.ntaps : 0, lane, [&](int t) { return (uint32_t)(uint16_t)p.tap_col[t] | (uint32_t)p.tap_b[t] << 16; });
      if (elect_one()) {
        tensormap_prefetch(do_a ? &p.a_hi : &p.b_hi);
        tensormap_prefetch(do_a ? &p.a_lo : &p.b_lo);
      }
      grid_dep_sync();
      WorkIter iter(p);
      WorkItem w;
      while (iter.next(p, w)) {
        int mt, nt, tap;
        decode_tile(p, w.tile, mt, nt, tap);
        const int m0 = mt * BM, n0 = nt * BN;
        int ch = w.k0 / period, ti = w.k0 - ch * period;
        int left = p.group_iters;         // stages to the next accumulator group
        int slot_off[2] = {0, 0}, slot_grp[2] = {0, 0};       // kModeWgrad: row shift and column group of the tile's slots
        if (p.mode == kModeWgrad && do_a) {
#pragma unroll
          for (int sl = 0; sl < 2; ++sl) {
            const int u = tap * p.taps_per_tile + sl, t = u / p.slots_per_tap, cb = mt + u - t * p.slots_per_tap;
            slot_off[sl] = t < p.ntaps ? p.tap_off[t] : 0x40000000;
            slot_grp[sl] = (cb * p.slot + (t < p.ntaps ? p.tap_col[t] : 0)) / T::kGW;
          }
        }
        for (int it = 0; it < w.kcount; ++it) {
          const int git = w.k0 + it;                  // stage index within the tile's reduction
          const uint32_t word = conv ? words.at(ti) : 0x300u, tc = conv ? cols.at(ti) : 0u;
          const int off = conv ? (int)offs.at(ti) : 0;
          const bool fetch_a = it == 0 || (word & 0x100u);
          if (p.one_ring) {
            mbar_wait_mark(&b_empty[bs], bph ^ 1, abort_flag, bad);
            armed_b |= 1u << bs; phase_b = (phase_b & ~(1u << bs)) | (bph << bs);
          }
          if (do_a && fetch_a) {
            if (!p.one_ring) {
              mbar_wait_mark(&a_empty[as], aph ^ 1, abort_flag, bad);
              armed_a |= 1u << as; phase_a = (phase_a & ~(1u << as)) | (aph << as);
            }
            uint8_t *a_hi = smem + as * a_slot_bytes, *a_lo = a_hi + a_half;
            uint64_t* bar = p.one_ring ? &b_full[bs] : &a_full[as];
            if (elect_one() && !bad) {
              mbar_expect_tx(bar, a_slot_bytes);
              if (conv) {
                const int col = (int)(short)(tc & 0xffffu) + ch * BK, row = m0 + off;
                tma_load_2d(a_hi, &p.a_hi, col, row, bar);
                tma_load_2d(a_lo, &p.a_lo, col, row, bar);
              } else if (p.mode == kModeWgrad) {
                // M/N-major operands come through a 3-D view {group width, rows, column groups}: one copy lands
                // [groups][BK rows][128 B], the layout the M/N-major descriptor expects.  One copy per tap slot; a slot past
                // the last tap reads rows beyond the pack (the copy still completes with its full byte count and fills zeros).
                const int gps = p.slot / T::kGW;
#pragma unroll
                for (int sl = 0; sl < 2; ++sl) {
                  if (sl == p.taps_per_tile) break;
                  const int row = slot_off[sl] < 0x40000000 ? git * BK + slot_off[sl] : 0x40000000;
                  tma_load_3d(a_hi + sl * gps * kGroupStride, &p.a_hi, 0, row, slot_grp[sl], bar);
                  tma_load_3d(a_lo + sl * gps * kGroupStride, &p.a_lo, 0, row, slot_grp[sl], bar);
                }
              } else if (p.a_mn) {
                tma_load_3d(a_hi, &p.a_hi, 0, git * BK, m0 / T::kGW, bar);
                tma_load_3d(a_lo, &p.a_lo, 0, git * BK, m0 / T::kGW, bar);
              } else {
                tma_load_2d(a_hi, &p.a_hi, git * BK, m0, bar);
                tma_load_2d(a_lo, &p.a_lo, git * BK, m0, bar);
              }
            }
            if (++as == p.a_slots) { as = 0; aph ^= 1; }
          }
          if (p.one_ring && !do_b && ++bs == p.b_slots) { bs = 0; bph ^= 1; }
          if (do_b && !b_loaded) {
            if (!p.one_ring) {
              if (!p.b_resident) mbar_wait_mark(&b_empty[bs], bph ^ 1, abort_flag, bad);
              armed_b |= 1u << bs; phase_b = (phase_b & ~(1u << bs)) | (bph << bs);
            }
            const bool hi_first = three && (group & 1) == 0;
            uint8_t *b_lo = b_smem + bs * kBSlot + (hi_first ? kBTile : 0), *b_hi = b_smem + bs * kBSlot + (hi_first ? 0 : kBTile);
            if (elect_one() && !bad) {
              mbar_expect_tx(&b_full[bs], kBSlot);
              if (conv) {
                const int col = (int)(tc >> 16) * p.b_tap_pitch + ch * BK;
                tma_load_2d(b_lo, &p.b_lo, col, n0, &b_full[bs]);
                tma_load_2d(b_hi, &p.b_hi, col, n0, &b_full[bs]);
              } else if (p.b_mn) {
                tma_load_3d(b_lo, &p.b_lo, 0, git * BK, n0 / T::kGW, &b_full[bs]);
                tma_load_3d(b_hi, &p.b_hi, 0, git * BK, n0 / T::kGW, &b_full[bs]);
              } else {
                tma_load_2d(b_lo, &p.b_lo, git * BK, n0, &b_full[bs]);
                tma_load_2d(b_hi, &p.b_hi, git * BK, n0, &b_full[bs]);
              }
            }
            if (++bs == p.b_slots) { bs = 0; bph ^= 1; }
          }
          if (++ti == period) { ti = 0; ++ch; }
          if (--left == 0) { left = p.group_iters; ++group; }
        }
        if (left != p.group_iters) ++group;
        if (p.b_resident) b_loaded = true;
      }
      if (*abort_flag) {
        // let copies that are still in flight land before the CTA gives its shared memory back
        for (int s = 0; s < kMaxASlots + kMaxBSlots; ++s) {
          const bool is_a = s < kMaxASlots;
          const int i = is_a ? s : s - kMaxASlots;
          if (!(((is_a ? armed_a : armed_b) >> i) & 1)) continue;
          long long t0 = clock64();
          while (!mbar_try_wait(is_a ? &a_full[i] : &b_full[i], ((is_a ? phase_a : phase_b) >> i) & 1) && clock64() - t0 < 100000000ll) {}
        }
      }
    }
  } else if (warp == 1 || warp == kNarrowWarp) {
    // ===================== MMA issuer =====================
    {
      // Three products per K step: A_hi*B_hi (main) and the cross terms A_hi*B_lo, A_lo*B_hi.  The two B tiles lie back to back
      // in their slot, so ONE instruction with N = 2*BN computes main and the first cross term into neighbouring TMEM blocks.
      // Every accumulation into TMEM truncates the sum, an error proportional to the accumulator's magnitude; the cross
      // terms are 2^-11 of the main one and have blocks of their own, so the large accumulator sees one truncation per K step.
      // Where the blocks lie, and who issues.  One warp issues 8 MMAs, 1-3 commits and the bookkeeping of a stage in some 1250
      // cycles, where the tensor pipe needs 768 (BN = 128) or 448 (BN = 64).  MMAs into different blocks need no order among
      // them, so where the two cross terms have blocks of their own two warps issue, one the wide instructions and one the
      // narrow ones, each at its own pace (512 channels, 28 x 28, 3x3, batch 64: 603 -> 548 us; 64 channels, 224 x 224: 985 -> 886):
      //   BN = 64           two sets of {cross, main, cross'}: 384 columns;
      //   kAccThree         main0, cross, main1, cross' (4*BN columns): main alternates between its two blocks from group to group,
      //                     the cross terms accumulate for cross_groups groups before the epilogue takes them.  The wide
      //                     instruction goes to (main0, cross) or (cross, main1), hence the order of the B tiles;
      //   kAccPair          two sets of {cross, main} and one issuer: short reductions, where the next tile must not wait for the
      //                     epilogue to read the cross terms, and short groups of one stage (see launch_gemm).
      // instruction descriptor: D = f32 (bits 4-5 = 1), A format at bit 7, B format at bit 10, majors at bits 15 / 16,
      // N >> 3 at bit 17, M >> 4 at bit 24
      const uint32_t idesc_base = (1u << 4) | (T::kFormat << 7) | (T::kFormat << 10) | ((uint32_t)p.a_mn << 15) | ((uint32_t)p.b_mn << 16) |
                                  ((uint32_t)(BM >> 4) << 24);
      const uint32_t idesc_wide = idesc_base | ((uint32_t)((2 * BN) >> 3) << 17), idesc_narrow = idesc_base | ((uint32_t)(BN >> 3) << 17);
      // K-major: one MMA advances 32 bytes along the 128-byte row; M/N-major: one MMA covers K rows of 128 bytes each
      // (16 rows of fp16, 8 of tf32), column groups kGroupStride apart
      const uint32_t a_lbo = p.a_mn ? kGroupStride : 16u, b_lbo = p.b_mn ? kGroupStride : 16u;
      const uint32_t a_kstep = p.a_mn ? kGroupStride / 4 : 32u, b_kstep = p.b_mn ? kGroupStride / 4 : 32u;
      const uint32_t a_sbo = p.a_mn ? T::kMnSbo : 1024u, b_sbo = p.b_mn ? T::kMnSbo : 1024u;
      const uint32_t a_lt = p.a_mn ? T::kMnLayout : 2u, b_lt = p.b_mn ? T::kMnLayout : 2u;
      // Only the low word of a descriptor changes: its address field (16-byte units, no carry out of it below 256 KB)
      const uint64_t a_desc = umma_desc(smem_u32(smem), a_lbo, a_sbo, a_lt), b_desc = umma_desc(smem_u32(b_smem), b_lbo, b_sbo, b_lt);
      const uint32_t a_word = (uint32_t)a_desc, a_high = (uint32_t)(a_desc >> 32), b_word = (uint32_t)b_desc, b_high = (uint32_t)(b_desc >> 32);
      const uint32_t a_step = a_kstep >> 4, b_step = b_kstep >> 4, a_slot16 = (uint32_t)a_slot_bytes >> 4, a_half16 = (uint32_t)a_half >> 4;
      constexpr uint32_t kBSlot16 = kBSlot >> 4, kBTile16 = kBTile >> 4;
      const bool conv = p.mode == kModeConv, one_ring = p.one_ring, resident = p.b_resident;
      const int period = conv ? p.ntaps : 1, group_iters = p.group_iters, a_slots = p.a_slots, b_slots = p.b_slots, cross_groups = p.cross_groups;
      const TapTable words(conv ? p.ntaps : 0, lane, [&](int t) { return p.tap_word[t]; });
      auto issue = [&](auto role_of) {
        constexpr int kRole = decltype(role_of)::value;     // 1: the wide instructions, 2: the narrow ones, 3: both
        int as = 0, bs = 0;
        uint32_t aph = 0, bph = 0;
        int group = 0;            // accumulator groups issued so far (alternating TMEM buffers)
        int epoch = 0;            // kAccThree: times the cross terms started afresh
        int bad = 0;
        bool ready = false;       // the next stage's operands were seen to have arrived
        uint32_t word = 0x300u;
        WorkIter iter(p);
        WorkItem w;
        while (iter.next(p, w)) {
          int ti = 0;
          if (conv) { ti = w.k0 % period; word = words.at(ti); }
          if (resident) { bs = 0; bph = 0; }           // the slots were filled once: their first phase stays complete
          bool first = true;
          int in_epoch = 0;                            // groups since the cross terms started afresh
          for (int it0 = 0; it0 < w.kcount; it0 += group_iters, ++group) {
            const int acc = group & 1;
            mbar_wait_mark(&acc_empty[acc], ((group >> 1) & 1) ^ 1, abort_flag, bad);
            if (three && in_epoch == 0) {
              mbar_wait_mark(cross_empty, (epoch & 1) ^ 1, abort_flag, bad);
              ++epoch;
            }
            const uint32_t d_wide = tmem_base + acc * (three ? BN : kSetCols);
            const uint32_t d_narrow = three ? tmem_base + 3 * BN : d_wide + (kSets3 ? 2 * BN : 0);
            const bool hi_first = three && acc == 0;
            const uint32_t hi_at = hi_first ? 0u : kBTile16, lo_at = kBTile16 - hi_at;
            const int it1 = min(it0 + group_iters, w.kcount);
            for (int it = it0; it < it1; ++it) {
              if (first && !one_ring) mbar_wait_mark(&a_full[as], aph, abort_flag, bad);
              if (!ready) mbar_wait_mark(&b_full[bs], bph, abort_flag, bad);
              tcgen05_fence_after();
              const bool last = (word & 0x200u) != 0 || it == w.kcount - 1;
              const uint32_t ah = a_word + as * a_slot16 + (word & 0xffu) * 8u, al = ah + a_half16;
              const uint32_t bw = b_word + bs * kBSlot16, bh = bw + hi_at;                  // bw: N = 2*BN runs on into the second B tile
              const uint32_t keep_main = it > it0 ? 1u : 0u, keep_cross = three ? (it > it0 || in_epoch > 0 ? 1u : 0u) : keep_main;
              uint64_t* const b_done = &b_empty[bs];
              uint64_t* const a_done = &a_empty[as];
              if (++bs == b_slots) { bs = 0; if (!resident) bph ^= 1; }
              if (last && ++as == a_slots) { as = 0; aph ^= 1; }
              ready = mbar_test(&b_full[bs], bph);
              if (conv) { if (++ti == period) ti = 0; word = words.at(ti); }
              first = (word & 0x100u) != 0;
              if (elect_one() && !bad) {
                if (kRole & 1) {
                  if (three && !keep_main && keep_cross) {      // main starts afresh, the cross terms go on
                    umma_at<AR>(hi_first ? d_wide : d_wide + BN, ah, a_high, bh, b_high, idesc_narrow, 0u);
                    umma_at<AR>(hi_first ? d_wide + BN : d_wide, ah, a_high, bw + lo_at, b_high, idesc_narrow, 1u);
                  } else {
                    umma_at<AR>(d_wide, ah, a_high, bw, b_high, idesc_wide, keep_main);
                  }
                }
                if (kRole & 2) umma_at<AR>(d_narrow, al, a_high, bh, b_high, idesc_narrow, three || kSets3 ? keep_cross : 1u);
#pragma unroll
                for (int q = 1; q < 4; ++q) {
                  if (kRole & 1) umma_at<AR>(d_wide, ah + q * a_step, a_high, bw + q * b_step, b_high, idesc_wide, 1u);
                  if (kRole & 2) umma_at<AR>(d_narrow, al + q * a_step, a_high, bh + q * b_step, b_high, idesc_narrow, 1u);
                }
                // the commits free the slots once the MMAs above have read them
                if (!resident) tcgen05_commit(b_done);
                if (last && !one_ring) tcgen05_commit(a_done);
                if (it == it1 - 1) tcgen05_commit(&acc_full[acc]);
              }
            }
            if (++in_epoch == cross_groups) in_epoch = 0;
          }
        }
      };
      if (issuers == 1) { if (warp == 1) issue(std::integral_constant<int, 3>()); }
      else if (warp == 1) issue(std::integral_constant<int, 1>());
      else issue(std::integral_constant<int, 2>());
    }
  } else {
    // ===================== epilogue: warps 2..9 =====================
    // A warp may only read the TMEM lane quarter (warp % 4); two warps share each quarter and take one half of
    // the tile's columns each, so that every scheduler has two epilogue warps to alternate between.
    grid_dep_sync();
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    constexpr int HC = BN / 2;                  // columns per epilogue warp
    constexpr int NC = HC % 32 == 0 ? 32 : 16;  // columns per TMEM load
    const int row_in_tile = quarter * 32 + lane;
    const float inv_scale = (1.f / __ldg(p.a_scale)) * (1.f / __ldg(p.b_scale));     // powers of two: exact
    const float2 scale2 = make_float2(inv_scale, inv_scale);
    int group = 0;
    uint32_t top = 0;         // largest |value| this thread stored; one atomic per warp and launch
    bool ok = true;
    WorkIter iter(p);
    WorkItem w;
    while (ok && iter.next(p, w)) {
      int mt, nt, tap;
      decode_tile(p, w.tile, mt, nt, tap);
      const int kcount = w.kcount;
      const int n0 = nt * BN + half * HC;
      const RowAddr ra = row_address(p, mt, tap, row_in_tile);
      const bool row_ok = ra.ok;
      const uint32_t col_bytes = ra.col_stride * 4u;
      char* const row_out = reinterpret_cast<char*>(p.out + ra.base + (long long)n0 * ra.col_stride);
      const int ncols = max(0, min(HC, p.N - n0));
      const bool vec_ok = p.epi == kEpiRowMajor && ((ra.base + n0) & 3) == 0;

      auto wait_group = [&](int acc_buf, int grp) -> bool {   // lane 0 polls, the warp follows (keeps .sync.aligned loads converged)
        int got = lane == 0 ? (int)mbar_wait(&acc_full[acc_buf], (grp >> 1) & 1, abort_flag) : 1;
        return __shfl_sync(0xffffffffu, got, 0) != 0;
      };
      // NC values of this thread's row at columns c0.. of the warp's half; offsets of 32 bits (BN planes are far below 2^32 elements):
      // 64-bit ones cost 1-2 us of 70 in stores alone
      auto store_cols = [&](const float2* v2, int c0) {
        const float* v = reinterpret_cast<const float*>(v2);
        if (!row_ok || c0 >= ncols) return;
        if (p.amax) {
#pragma unroll
          for (int q = 0; q < NC; ++q) top = max(top, amax_bits(v[q]));
        }
        char* dst = row_out + (uint64_t)col_bytes * (uint32_t)c0;
        if (vec_ok && c0 + NC <= ncols) {
#pragma unroll
          for (int q = 0; q < NC / 4; ++q) reinterpret_cast<float4*>(dst)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        } else if (c0 + NC <= ncols) {
#pragma unroll
          for (int q = 0; q < NC; ++q) reinterpret_cast<float*>(dst)[(size_t)((uint32_t)q * ra.col_stride)] = v[q];
        } else {
#pragma unroll
          for (int q = 0; q < NC; ++q)
            if (c0 + q < ncols) reinterpret_cast<float*>(dst)[(size_t)((uint32_t)q * ra.col_stride)] = v[q];
        }
      };
      const uint32_t t_lane = tmem_base + half * HC + ((uint32_t)(quarter * 32) << 16);

      if (w.slot < 0 && kcount <= p.group_iters && p.cluster <= 1 && !three) {
        // One accumulator group: stream TMEM straight to memory.
        const int acc = group & 1;
        if (!wait_group(acc, group)) { ok = false; break; }
        ++group;
        tcgen05_fence_after();
#pragma unroll 1
        for (int c0 = 0; c0 < HC; c0 += NC) {
          float2 v[NC / 2];
          load_sum<NC, kSets3 ? 3 : 2>(t_lane + acc * kSetCols + c0, BN, v);
          if (c0 + NC >= HC) {     // last chunk read: the accumulator can be reused while we store
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc]);
          }
#pragma unroll
          for (int q = 0; q < NC / 2; ++q) v[q] = __fmul2_rn(v[q], scale2);
          store_cols(v, c0);
        }
        continue;
      }

      // The tensor core accumulates with truncation, so a long chain of MMAs into one TMEM accumulator
      // drifts; each group of group_iters stages is therefore accumulated in TMEM on its own and promoted
      // here into fp32 registers with round-to-nearest adds.
      float2 accv[HC / 2];
#pragma unroll
      for (int q = 0; q < HC / 2; ++q) accv[q] = make_float2(0.f, 0.f);
      int in_epoch = 0;
      for (int it0 = 0; it0 < kcount && ok; it0 += p.group_iters, ++group) {
        const int acc = group & 1;
        if (!wait_group(acc, group)) { ok = false; break; }
        tcgen05_fence_after();
        if (three) {
#pragma unroll
          for (int c0 = 0; c0 < HC; c0 += NC) {
            float2 v[NC / 2];
            load_sum<NC, 1>(t_lane + acc * 2 * BN + c0, 0, v);
#pragma unroll
            for (int q = 0; q < NC / 2; ++q) accv[c0 / 2 + q] = __fadd2_rn(accv[c0 / 2 + q], v[q]);
          }
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[acc]);
          if (++in_epoch < p.cross_groups && it0 + p.group_iters < kcount) continue;
          in_epoch = 0;
#pragma unroll
          for (int c0 = 0; c0 < HC; c0 += NC) {
            float2 v[NC / 2];
            load_sum<NC, 2>(t_lane + BN + c0, 2 * BN, v);
#pragma unroll
            for (int q = 0; q < NC / 2; ++q) accv[c0 / 2 + q] = __fadd2_rn(accv[c0 / 2 + q], v[q]);
          }
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(cross_empty);
        } else {
#pragma unroll
          for (int c0 = 0; c0 < HC; c0 += NC) {
            float2 v[NC / 2];
            load_sum<NC, kSets3 ? 3 : 2>(t_lane + acc * kSetCols + c0, BN, v);
#pragma unroll
            for (int q = 0; q < NC / 2; ++q) accv[c0 / 2 + q] = __fadd2_rn(accv[c0 / 2 + q], v[q]);
          }
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[acc]);
        }
      }
      if (!ok) break;
      if (w.slot >= 0 || p.cluster > 1) {
        // a piece of a tile: raw partial sums, [column][row] so that a warp's 32 rows coalesce - to the workspace (split tail), or
        // to this CTA's own shared memory, whose operands have all been read by now (cluster)
        float* ws = (p.cluster > 1 ? reinterpret_cast<float*>(smem) : p.workspace + (size_t)w.slot * BN * BM) + half * HC * BM + row_in_tile;
#pragma unroll
        for (int q = 0; q < HC / 2; ++q) { ws[(size_t)(2 * q) * BM] = accv[q].x; ws[(size_t)(2 * q + 1) * BM] = accv[q].y; }
        continue;
      }
#pragma unroll
      for (int c0 = 0; c0 < HC; c0 += NC) {
#pragma unroll
        for (int q = 0; q < NC / 2; ++q) accv[c0 / 2 + q] = __fmul2_rn(accv[c0 / 2 + q], scale2);
        store_cols(accv + c0 / 2, c0);
      }
    }
    if (p.amax) {
      top = __reduce_max_sync(0xffffffffu, top);
      if (lane == 0 && top) atomicMax(p.amax, top);
      if (blockIdx.x == 0 && threadIdx.x == 64 && p.amax_clear) *p.amax_clear = 0u;
    }
  }

  if (p.cluster > 1) {
    // Every CTA of the cluster adds up its share of the tile's columns, in rank order (bit-reproducible).  kUnroll columns of all
    // pieces are in flight at once.  The traffic between the SMs bounds it (some 15 cycles per 128-byte load: 8000 cycles for 6
    // pieces of 128 x 96); bulk copies between the CTAs took as long.
    constexpr int kUnroll = 4, kLanes = kGemmThreads / BM;
    const int rank = blockIdx.x % p.cluster, tile = blockIdx.x / p.cluster;
    int mt, nt, tap;
    decode_tile(p, tile, mt, nt, tap);
    const int row = threadIdx.x & (BM - 1);
    const RowAddr ra = row_address(p, mt, tap, row);
    const float inv_scale = (1.f / __ldg(p.a_scale)) * (1.f / __ldg(p.b_scale));
    const int c1 = min(BN * (rank + 1) / p.cluster, p.N - nt * BN);
    uint32_t top = 0;
    __syncwarp();
    cluster_sync_all();
    if (!*abort_flag) {
      for (int c0 = BN * rank / p.cluster + (int)threadIdx.x / BM; c0 < c1; c0 += kUnroll * kLanes) {
        float sum[kUnroll] = {0.f, 0.f, 0.f, 0.f}, rest[kUnroll] = {0.f, 0.f, 0.f, 0.f};
        float v[kMaxCluster][kUnroll];
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r)
          if (r < p.cluster) {
            const uint32_t piece = smem_of_cta(smem_u32(smem), r) + row * 4u;
#pragma unroll
            for (int j = 0; j < kUnroll; ++j) v[r][j] = ld_cluster(piece + (uint32_t)min(c0 + j * kLanes, c1 - 1) * (BM * 4u));
          }
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r)
          if (r < p.cluster) {
#pragma unroll
            for (int j = 0; j < kUnroll; ++j) (r < kMaxCluster / 2 ? sum : rest)[j] += v[r][j];
          }
#pragma unroll
        for (int j = 0; j < kUnroll; ++j) {
          sum[j] += rest[j];                  // runs of kSumChunk, as reduce_tile adds them
          const int c = c0 + j * kLanes;
          if (ra.ok && c < c1) {
            p.out[ra.base + (long long)(nt * BN + c) * ra.col_stride] = sum[j] * inv_scale;
            top = max(top, amax_bits(sum[j] * inv_scale));
          }
        }
      }
    }
    if (p.amax) {
      top = __reduce_max_sync(0xffffffffu, top);
      if (lane == 0 && top) atomicMax(p.amax, top);
    }
    __syncwarp();
    cluster_sync_all();        // nobody leaves while its shared memory is still read
  }

  // ===================== teardown =====================
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
  if (threadIdx.x == 0 && *abort_flag && p.err) atomicExch(p.err, 1);
}

// ------------------------------------------------------------------------------------------------
// Many small filter gradients in one launch.  A product of 3-30 stages a CTA spends 4000 cycles up to its first MMA, 2500 from its
// last to its end, and most of these have fewer tiles than SMs, so they cut their reductions over all of them and add the pieces
// up in a cluster's shared memory or a second kernel.  Nothing reads a filter gradient before the parameters are updated, so the
// executor lets the library hold them back (hold_product), and one launch works through the tiles of several, dealt to the CTAs so
// that all finish together: whole tiles where the reduction is short, their pieces where it is long.
//
// The bits are those of the separate launches: a tile kept whole (or one of its chunks of kSumChunk pieces, see reduce_tile) is
// still added up piece by piece, in the order of the pieces, with the same accumulator blocks; the second set of sums just fits the
// 168 registers a thread can have.  Roles: warps 0 and 3 copy A and B,
// 1 and 2 issue, 4-11 epilogue.  Both operands M/N-major, groups of one stage.
// A step of Inception-v3 at batch 2 has 94 of them, 1.1 ms in separate launches and 0.22 in two: 4495 -> 3702 us
// (chunks instead of whole tiles 0.06 more, see reduce_tile).  ResNet-50 at batch 19
// 4453 -> 3938, DenseNet-121 at batch 32 14.58 -> 13.39 ms.
// ------------------------------------------------------------------------------------------------
constexpr int kSumChunk = 4;      // pieces added in order before their sum goes to the tile's
static_assert(2 * kSumChunk == kMaxCluster, "the sum over a cluster takes two runs");
struct GroupTable {
  const GemmParams* problems;
  const int4* items;              // {problem, tile, pieces or -1: all of the tile's, the workspace slot of their sum}; pieces: the first + (their number << 16)
  const int* first;               // CTA -> its first item; one more than CTAs
  const int4* sums;               // tiles that were dealt out: {problem, tile, their first slot, from one to the next; negative: each holds a chunk, not a piece}
  float* workspace;
  int* err;
};
// number of pieces that tile `tile` of a held-back product is added up from
__host__ __device__ inline int tile_pieces(const GemmParams& p, int tile) { return p.cluster > 1 ? p.cluster : p.tail_pieces > 0 && tile >= p.full_tiles ? p.tail_pieces : 1; }
struct GroupIter {
  int at, end, piece, last;
  int4 item, next_item;
  int k_total, pieces;
  const GemmParams* q;
  __device__ __forceinline__ explicit GroupIter(const GroupTable& t) : at(__ldg(t.first + blockIdx.x)), end(__ldg(t.first + blockIdx.x + 1)), piece(0), last(-1) {
    if (at < end) next_item = __ldg(t.items + at);
  }
  // The next run of stages.  `fresh`: of another tile than the one before; `done`: its last
  __device__ __forceinline__ bool next(const GroupTable& t, int& k0, int& kcount, bool& fresh, bool& done) {
    fresh = piece > last;
    if (fresh) {
      if (at == end) return false;
      item = next_item;
      if (++at < end) next_item = __ldg(t.items + at);       // a memory round trip ahead
      q = t.problems + item.x;
      k_total = q->k_total;
      pieces = tile_pieces(*q, item.y);
      piece = item.z < 0 ? 0 : item.z & 0xffff;
      last = item.z < 0 ? pieces - 1 : piece + (item.z >> 16) - 1;
    }
    k0 = (int)((long long)k_total * piece / pieces);
    kcount = (int)((long long)k_total * (piece + 1) / pieces) - k0;
    done = piece++ == last;
    return true;
  }
};
__device__ __forceinline__ void tensormap_acquire(const CUtensorMap* map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
template <int BN> constexpr int kGroupStages = BN == 64 ? 4 : 3;
template <int BN> constexpr int kGroupSmem = kGroupStages<BN> * (BM + BN) * 256 + kSmemBarriers + 1024;

template <int BN, int AR>
__global__ void __launch_bounds__(kGemmThreads, 1) gemm3x_group_kernel(const __grid_constant__ GroupTable t) {
  using T = Arith<AR>;
  constexpr int BK = T::kBK, kStages = kGroupStages<BN>;
  constexpr uint32_t kGroupStride = BK * 128;
  constexpr int kTmemCols = 512;
  constexpr bool kSets3 = BN == 64;                         // accumulator sets as in gemm3x_kernel: {cross, main, cross'} or {cross, main}
  constexpr int kSetCols = kSets3 ? 3 * BN : 2 * BN, kIssuers = kSets3 ? 2 : 1;
  constexpr int kAHalf = BM * 128, kBTile = BN * 128, kStageBytes = 2 * kAHalf + 2 * kBTile;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
  uint64_t* empty = full + kStages;
  uint64_t* acc_full = empty + kStages;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (warp == 0) {
    if (lane < 2 * kStages + 4) mbar_init(&full[lane], lane < kStages ? 2 : lane < 2 * kStages + 2 ? kIssuers : 8);       // both copying warps; the issuers; the epilogue's warps
    if (lane == 0) *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  grid_dep_sync();

  if (warp < 4) {
    if (warp == 0 || warp == 3) {
      // ===================== TMA producers: A (warp 0) and B (warp 3) =====================
      const bool do_a = warp == 0;
      int slot = 0, bad = 0;
      uint32_t ph = 0, armed = 0, phase = 0;                // per slot: filled at least once, phase of the last fill
      int k0, kcount;
      bool fresh, done;
      GroupIter iter(t);
      int row0[2] = {0, 0}, grp[2] = {0, 0}, slots = 1, gps = 0;
      while (iter.next(t, k0, kcount, fresh, done)) {
        const GemmParams& q = *iter.q;
        const CUtensorMap *map_hi = do_a ? &q.a_hi : &q.b_hi, *map_lo = do_a ? &q.a_lo : &q.b_lo;
        if (fresh) {
          if (elect_one()) { tensormap_acquire(map_hi); tensormap_acquire(map_lo); }
          __syncwarp();
          int mt, nt, tap;
          decode_tile(q, iter.item.y, mt, nt, tap);
          if (!do_a) {
            grp[0] = nt * BN / T::kGW;
          } else if (q.mode == kModeWgrad) {                // a copy for each tap slot of the tile, at its row shift
            slots = q.taps_per_tile; gps = q.slot / T::kGW;
#pragma unroll
            for (int sl = 0; sl < 2; ++sl) {
              const int u = tap * q.taps_per_tile + sl, tp = u / q.slots_per_tap, cb = mt + u - tp * q.slots_per_tap;
              row0[sl] = tp < q.ntaps ? q.tap_off[tp] : 0x40000000;
              grp[sl] = (cb * q.slot + (tp < q.ntaps ? q.tap_col[tp] : 0)) / T::kGW;
            }
          } else {
            slots = 1; row0[0] = 0; grp[0] = mt * BM / T::kGW;
          }
        }
        for (int it = 0; it < kcount; ++it) {
          mbar_wait_mark(&empty[slot], ph ^ 1, abort_flag, bad);
          armed |= 1u << slot; phase = (phase & ~(1u << slot)) | (ph << slot);
          uint8_t* const a = smem + slot * kStageBytes + (do_a ? 0 : 2 * kAHalf);
          uint64_t* const bar = &full[slot];
          const int row = (k0 + it) * BK;
          if (elect_one() && !bad) {
            if (do_a) {
              mbar_expect_tx(bar, 2 * kAHalf);
#pragma unroll
              for (int sl = 0; sl < 2; ++sl) {
                if (sl == slots) break;
                const int r = row0[sl] < 0x40000000 ? row + row0[sl] : 0x40000000;      // past the last tap: rows beyond the pack, zeros
                tma_load_3d(a + sl * gps * kGroupStride, map_hi, 0, r, grp[sl], bar);
                tma_load_3d(a + kAHalf + sl * gps * kGroupStride, map_lo, 0, r, grp[sl], bar);
              }
            } else {
              mbar_expect_tx(bar, 2 * kBTile);
              tma_load_3d(a, map_lo, 0, row, grp[0], bar);
              tma_load_3d(a + kBTile, map_hi, 0, row, grp[0], bar);
            }
          }
          if (++slot == kStages) { slot = 0; ph ^= 1; }
        }
      }
      if (*abort_flag) {
        // let copies that are still in flight land before the CTA gives its shared memory back
        for (int i = 0; i < kStages; ++i) {
          if (!((armed >> i) & 1)) continue;
          long long t0 = clock64();
          while (!mbar_try_wait(&full[i], (phase >> i) & 1) && clock64() - t0 < 100000000ll) {}
        }
      }
    } else if (warp == 1 || kIssuers == 2) {
      // ===================== MMA issuers: warp 1 the wide instructions (BN = 128: the narrow ones too), warp 2 the narrow ones =====================
      constexpr uint32_t idesc_base = (1u << 4) | (T::kFormat << 7) | (T::kFormat << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(BM >> 4) << 24);
      constexpr uint32_t idesc_wide = idesc_base | ((uint32_t)((2 * BN) >> 3) << 17), idesc_narrow = idesc_base | ((uint32_t)(BN >> 3) << 17);
      constexpr uint32_t kStep16 = kGroupStride / 4 >> 4, kStage16 = kStageBytes >> 4, kAHalf16 = kAHalf >> 4, kBTile16 = kBTile >> 4;
      const uint64_t desc = umma_desc(smem_u32(smem), kGroupStride, T::kMnSbo, T::kMnLayout);
      const uint32_t low = (uint32_t)desc, high = (uint32_t)(desc >> 32);
      const bool wide = warp == 1, narrow = kIssuers == 1 || warp == 2;
      int slot = 0, bad = 0, group = 0;
      uint32_t ph = 0;
      int k0, kcount;
      bool fresh, done;
      GroupIter iter(t);
      while (iter.next(t, k0, kcount, fresh, done)) {
        for (int it = 0; it < kcount; ++it, ++group) {
          const int acc = group & 1;
          mbar_wait_mark(&acc_empty[acc], ((group >> 1) & 1) ^ 1, abort_flag, bad);
          mbar_wait_mark(&full[slot], ph, abort_flag, bad);
          tcgen05_fence_after();
          const uint32_t ah = low + slot * kStage16, al = ah + kAHalf16, bw = ah + 2 * kAHalf16, bh = bw + kBTile16;       // bw: N = 2*BN runs on into the hi tile
          const uint32_t d_wide = tmem_base + acc * kSetCols, d_narrow = d_wide + (kSets3 ? 2 * BN : 0);
          uint64_t* const freed = &empty[slot];
          if (++slot == kStages) { slot = 0; ph ^= 1; }
          if (elect_one() && !bad) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if (wide) umma_at<AR>(d_wide, ah + k * kStep16, high, bw + k * kStep16, high, idesc_wide, k > 0);
              if (narrow) umma_at<AR>(d_narrow, al + k * kStep16, high, bh + k * kStep16, high, idesc_narrow, kSets3 ? k > 0 : 1u);
            }
            tcgen05_commit(freed);
            tcgen05_commit(&acc_full[acc]);
          }
        }
      }
    }
  } else {
    // ===================== epilogue: warps 4..11 =====================
    const int quarter = warp & 3, half = (warp - 4) >> 2;
    constexpr int HC = BN / 2, NC = 16;         // columns per warp, and per TMEM load
    const int row_in_tile = quarter * 32 + lane;
    const uint32_t t_lane = tmem_base + half * HC + ((uint32_t)(quarter * 32) << 16);
    int group = 0;
    bool ok = true;
    int k0, kcount;
    bool fresh, done;
    float2 total[HC / 2];
    GroupIter iter(t);
    while (ok && iter.next(t, k0, kcount, fresh, done)) {
      if (fresh) {
#pragma unroll
        for (int q = 0; q < HC / 2; ++q) total[q] = make_float2(0.f, 0.f);
      }
      float2 accv[HC / 2];
#pragma unroll
      for (int q = 0; q < HC / 2; ++q) accv[q] = make_float2(0.f, 0.f);
      for (int it = 0; it < kcount; ++it, ++group) {
        const int acc = group & 1;
        int got = lane == 0 ? (int)mbar_wait(&acc_full[acc], (group >> 1) & 1, abort_flag) : 1;
        if (__shfl_sync(0xffffffffu, got, 0) == 0) { ok = false; break; }
        tcgen05_fence_after();
#pragma unroll
        for (int c0 = 0; c0 < HC; c0 += NC) {
          float2 v[NC / 2];
          load_sum<NC, kSets3 ? 3 : 2>(t_lane + acc * kSetCols + c0, BN, v);
#pragma unroll
          for (int q = 0; q < NC / 2; ++q) accv[c0 / 2 + q] = __fadd2_rn(accv[c0 / 2 + q], v[q]);
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[acc]);
      }
      if (!ok) break;
#pragma unroll
      for (int q = 0; q < HC / 2; ++q) total[q] = __fadd2_rn(total[q], accv[q]);
      if (!done) continue;
      if (iter.item.z >= 0) {                   // not the whole tile: raw sums for reduce_group_kernel
        float* ws = t.workspace + (size_t)iter.item.w * BN * BM + half * HC * BM + row_in_tile;
#pragma unroll
        for (int q = 0; q < HC / 2; ++q) { ws[(size_t)(2 * q) * BM] = total[q].x; ws[(size_t)(2 * q + 1) * BM] = total[q].y; }
        continue;
      }
      const GemmParams& q = *iter.q;
      int mt, nt, tap;
      decode_tile(q, iter.item.y, mt, nt, tap);
      const RowAddr ra = row_address(q, mt, tap, row_in_tile);
      const int n0 = nt * BN + half * HC, ncols = ra.ok ? max(0, min(HC, q.N - n0)) : 0;
      const float inv_scale = (1.f / __ldg(q.a_scale)) * (1.f / __ldg(q.b_scale));     // powers of two: exact
      const float2 scale2 = make_float2(inv_scale, inv_scale);
      float* const dst = q.out + ra.base + (long long)n0 * ra.col_stride;
#pragma unroll
      for (int c = 0; c < HC / 2; ++c) total[c] = __fmul2_rn(total[c], scale2);
      if (q.epi == kEpiRowMajor && ((ra.base + n0) & 3) == 0 && ncols == HC) {
#pragma unroll
        for (int c = 0; c < HC / 4; ++c) reinterpret_cast<float4*>(dst)[c] = make_float4(total[2 * c].x, total[2 * c].y, total[2 * c + 1].x, total[2 * c + 1].y);
      } else {
#pragma unroll
        for (int c = 0; c < HC; ++c)
          if (c < ncols) dst[(size_t)((uint32_t)c * ra.col_stride)] = c & 1 ? total[c / 2].y : total[c / 2].x;
      }
    }
  }

  // ===================== teardown =====================
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
  if (threadIdx.x == 0 && *abort_flag && t.err) atomicExch(t.err, 1);
}

// ------------------------------------------------------------------------------------------------
// The same product on CTA pairs.  A cluster of two CTAs owns one 256 x 128 tile: CTA r loads rows [128 r, 128 r + 128)
// of A and rows [64 r, 64 r + 64) of the B tile (hi and lo each), so a stage is 48 KB per CTA instead of 64 KB - the
// operand traffic from L2, which is what bounds the one-CTA kernel, drops to three quarters per multiply - and four
// stages fit.  Rank 0's MMA warp issues three instructions of M = 256, N = 128 per K step for both SMs (A_hi B_hi into
// block 1; A_hi B_lo and A_lo B_hi into block 0: the N = 2 BN trick of the one-CTA kernel does not carry over, because
// a pair instruction takes the first half of its N columns from rank 0's shared memory and the second from rank 1's,
// which would interleave the blocks).  Each CTA's epilogue warps read their own 128 TMEM lanes.  K-major operands,
// whole tiles only (no split tail); every wait is bounded as in the one-CTA kernel, and both CTAs meet at a cluster
// barrier before either gives its shared memory and TMEM back.
// ------------------------------------------------------------------------------------------------
struct PairLayout {
  static constexpr int kBN = 128, kHalfN = 64, kStages = 4;
  static constexpr int kABytes = BM * 128, kBBytes = kHalfN * 128;
  static constexpr int kStageBytes = 2 * kABytes + 2 * kBBytes;      // per CTA: 48 KiB
  static constexpr int kBarrierBytes = 256;
  static constexpr int kTotal = kStages * kStageBytes + kBarrierBytes + 1024;
};

template <int AR>
__global__ void __launch_bounds__(kThreads, 1) gemm3x_pair_kernel(const __grid_constant__ GemmParams p) {
  using T = Arith<AR>;
  using L = PairLayout;
  constexpr int BN = L::kBN;
  constexpr int BK = T::kBK;
  constexpr int kTmemCols = 512;                            // two accumulator sets of 2*BN fp32 columns
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kStages * L::kStageBytes);      // used in rank 0 only
  uint64_t* empty = full + L::kStages;
  uint64_t* acc_full = empty + L::kStages;
  uint64_t* acc_empty = acc_full + 2;                                                    // used in rank 0 only
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int pair_m_tiles = (p.m_tiles + 1) >> 1;
  const int pair_tiles = pair_m_tiles * p.n_tiles * p.tap_tiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < L::kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 16); }    // 8 epilogue warps of each CTA
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {   // one warp of each CTA, same destination offset: the allocation spans both SMs
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();       // the peer's barriers exist before anything is sent to them
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dep_sync();

  auto decode = [&](int tile, int& mt, int& nt, int& tap) {
    nt = tile % p.n_tiles; tile /= p.n_tiles;
    tap = tile % p.tap_tiles;
    mt = 2 * (tile / p.tap_tiles) + (int)rank;
  };

  if (warp == 0) {
    // ===================== TMA producer (both CTAs) =====================
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      int issued = 0;
      for (int tile = pair; ok && tile < pair_tiles; tile += npairs) {
        int mt, nt, tap;
        decode(tile, mt, nt, tap);
        const int m0 = mt * BM, n0 = nt * BN + (int)rank * L::kHalfN;
        for (int it = 0; it < p.k_total; ++it) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) { ok = false; break; }
          uint8_t* st = smem + stage * L::kStageBytes;
          uint8_t *a_hi = st, *a_lo = st + L::kABytes, *b_hi = st + 2 * L::kABytes, *b_lo = b_hi + L::kBBytes;
          if (rank == 0) mbar_expect_tx(&full[stage], 2 * L::kStageBytes);      // this CTA's bytes and the peer's
          const uint32_t bar = smem_of_cta(smem_u32(&full[stage]), 0);
          int a_col, a_row, b_col;
          if (p.mode == kModeConv) {
            const int t = it / p.chunks_per_tap, ch = it - t * p.chunks_per_tap;
            a_col = p.tap_col[t] + ch * BK; a_row = m0 + p.tap_off[t] + p.pair_shift[t];
            b_col = p.tap_b[t] * p.b_tap_pitch + ch * BK;
          } else {
            a_col = it * BK; a_row = m0; b_col = it * BK;
          }
          tma_load_2d_pair(a_hi, &p.a_hi, a_col, a_row, bar);
          tma_load_2d_pair(a_lo, &p.a_lo, a_col, a_row, bar);
          tma_load_2d_pair(b_hi, &p.b_hi, b_col, n0, bar);
          tma_load_2d_pair(b_lo, &p.b_lo, b_col, n0, bar);
          ++issued;
          if (++stage == L::kStages) { stage = 0; phase ^= 1; }
        }
      }
      // Rank 0's MMA warp releases stages with arrivals that are sent to both CTAs.  Stay until every stage this CTA
      // filled has been released, so that no arrival is still on its way when the CTA gives its shared memory back.
      for (int s = 0; ok && s < L::kStages && s < issued; ++s) {
        if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) { ok = false; break; }
        if (++stage == L::kStages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (rank 0 for both SMs) =====================
    if (lane == 0 && rank == 0) {
      // instruction descriptor: D = f32, A / B formats, K-major both, N = BN, M = 256 (both CTAs' 128 rows)
      const uint32_t idesc = (1u << 4) | (T::kFormat << 7) | (T::kFormat << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((2 * BM) >> 4) << 24);
      int stage = 0; uint32_t phase = 0;
      int group = 0;
      bool ok = true;
      for (int tile = pair; ok && tile < pair_tiles; tile += npairs) {
        for (int it0 = 0; it0 < p.k_total && ok; it0 += p.group_iters, ++group) {
          const int acc = group & 1;
          if (!mbar_wait(&acc_empty[acc], ((group >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
          tcgen05_fence_after();
          const uint32_t d_cross = tmem_base + acc * 2 * BN, d_main = d_cross + BN;
          const int it1 = min(it0 + p.group_iters, p.k_total);
          for (int it = it0; it < it1; ++it) {
            if (!mbar_wait(&full[stage], phase, abort_flag)) { ok = false; break; }
            tcgen05_fence_after();
            const uint32_t st = smem_u32(smem + stage * L::kStageBytes);
            const uint32_t a_hi = st, a_lo = st + L::kABytes, b_hi = st + 2 * L::kABytes, b_lo = b_hi + L::kBBytes;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint64_t ah = umma_desc(a_hi + k * 32, 16, 1024, 2), al = umma_desc(a_lo + k * 32, 16, 1024, 2);
              const uint64_t bh = umma_desc(b_hi + k * 32, 16, 1024, 2), bl = umma_desc(b_lo + k * 32, 16, 1024, 2);
              const uint32_t accum = (it > it0 || k > 0) ? 1u : 0u;
              umma_pair<AR>(d_cross, ah, bl, idesc, accum);
              umma_pair<AR>(d_main, ah, bh, idesc, accum);
              umma_pair<AR>(d_cross, al, bh, idesc, 1u);
            }
            tcgen05_commit_pair(&empty[stage]);      // frees the stage in both CTAs
            if (++stage == L::kStages) { stage = 0; phase ^= 1; }
          }
          if (ok) tcgen05_commit_pair(&acc_full[acc]);
        }
      }
    }
  } else {
    // ===================== epilogue: warps 2..9 of both CTAs, each CTA its own 128 rows =====================
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    constexpr int HC = BN / 2;
    const int row_in_tile = quarter * 32 + lane;
    const float inv_scale = (1.f / __ldg(p.a_scale)) * (1.f / __ldg(p.b_scale));
    const uint32_t acc_empty_rank0 = smem_of_cta(smem_u32(&acc_empty[0]), 0);      // + 8 bytes for set 1
    int group = 0;
    bool ok = true;
    for (int tile = pair; ok && tile < pair_tiles; tile += npairs) {
      int mt, nt, tap;
      decode(tile, mt, nt, tap);
      const int n0 = nt * BN + half * HC;
      const RowAddr ra = row_address(p, mt, tap, row_in_tile);
      const bool row_ok = ra.ok && mt < p.m_tiles;
      const uint32_t col_stride = ra.col_stride;
      float* const row_out = p.out + ra.base + (long long)n0 * col_stride;
      const int ncols = max(0, min(HC, p.N - n0));
      const bool vec_ok = p.epi == kEpiRowMajor && ((ra.base + n0) & 3) == 0;
      float accv[HC];
#pragma unroll
      for (int q = 0; q < HC; ++q) accv[q] = 0.f;
      for (int it0 = 0; it0 < p.k_total && ok; it0 += p.group_iters, ++group) {
        const int acc = group & 1;
        int got = lane == 0 ? (int)mbar_wait(&acc_full[acc], (group >> 1) & 1, abort_flag) : 1;
        if (__shfl_sync(0xffffffffu, got, 0) == 0) { ok = false; break; }
        tcgen05_fence_after();
        const uint32_t t_base = tmem_base + acc * 2 * BN + half * HC + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
        for (int c0 = 0; c0 < HC; c0 += 16) {
          float v1[16], v2[16];
          tmem_ld16(t_base + c0, v1);
          tmem_ld16(t_base + BN + c0, v2);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 16; ++q) accv[c0 + q] += v1[q] + v2[q];
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_at(acc_empty_rank0 + 8u * acc);
      }
      if (!ok) break;
      if (!row_ok) continue;
      if (vec_ok && ncols == HC) {
        float4* dst = reinterpret_cast<float4*>(row_out);
#pragma unroll
        for (int q = 0; q < HC / 4; ++q) dst[q] = make_float4(accv[4 * q] * inv_scale, accv[4 * q + 1] * inv_scale, accv[4 * q + 2] * inv_scale, accv[4 * q + 3] * inv_scale);
      } else {
#pragma unroll
        for (int q = 0; q < HC; ++q)
          if (q < ncols) row_out[(size_t)((uint32_t)q * col_stride)] = accv[q] * inv_scale;
      }
    }
  }

  // ===================== teardown =====================
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();       // neither CTA's MMAs, commits or remote arrivals are outstanding past this point
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
  if (threadIdx.x == 0 && *abort_flag && p.err) atomicExch(p.err, 1);
}

// Adds up the pieces of every split tile in piece order and writes the result where the GEMM's own epilogue would have: the order
// in which the grouped kernel adds them where it keeps a tile to itself, so both give the same bits.  Every `chunk`
// pieces (one where no grouped kernel adds them, else kSumChunk) their sum goes to the tile's, whose rounding errors are carried along
// (two-sum): with 49 pieces in one run the error of a filter gradient is 20 % larger.  Bound by latency.
//   MANY = false (tiles of few pieces; the blocks' starts are what counts): grid (tiles, BN / 8), 256 threads, a thread has 4 columns
//     of 4 pieces in flight.
//   MANY = true (few tiles of many pieces): grid (tiles, BN / 8, 4), 16 warps take three pieces of 8 columns x 32 rows each to shared
//     memory, so that 48 pieces cost one memory round trip, and 8 of them add one column each.  With 16 pieces of a column in flight
//     in one thread instead ResNet-50 at batch 19 took 4524 us a step, with this 4389 (4434 with 4 row groups).
constexpr int kReduceCols = 8;
template <bool MANY> constexpr int kReduceThreads = MANY ? 512 : 256;
template <int BN, bool MANY, class Piece>
__device__ __forceinline__ void reduce_tile(const GemmParams& p, int tile, int pieces, int chunk, Piece&& piece) {
  int mt, nt, tap;
  decode_tile(p, tile, mt, nt, tap);
  constexpr int COLS = MANY ? 1 : 4;
  const int row = MANY ? blockIdx.z * 32 + (threadIdx.x & 31) : threadIdx.x & (BM - 1);
  const int c0 = blockIdx.y * kReduceCols + (MANY ? threadIdx.x / 32 : threadIdx.x / BM * COLS);
  float sum[COLS], run[COLS], lost[COLS];
#pragma unroll
  for (int q = 0; q < COLS; ++q) sum[q] = run[q] = lost[q] = 0.f;
  auto close_run = [&](int q) {
    const float s = __fadd_rn(sum[q], run[q]), b = __fsub_rn(s, sum[q]);
    lost[q] = __fadd_rn(lost[q], __fadd_rn(__fsub_rn(sum[q], __fsub_rn(s, b)), __fsub_rn(run[q], b)));
    sum[q] = s;
    run[q] = 0.f;
  };
  if (MANY) {
    constexpr int kEach = 3, kAtOnce = 16 * kEach;
    __shared__ float held[kAtOnce][kReduceCols][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int g0 = 0; g0 < pieces; g0 += kAtOnce) {
      float v[kEach][kReduceCols];
#pragma unroll
      for (int e = 0; e < kEach; ++e) {
        const int g = g0 + e * 16 + warp;
        if (g < pieces) {
          const float* ws = piece(g) + (size_t)blockIdx.y * kReduceCols * BM + row;
#pragma unroll
          for (int q = 0; q < kReduceCols; ++q) v[e][q] = __ldcg(ws + (size_t)q * BM);
        }
      }
      if (g0) __syncthreads();
#pragma unroll
      for (int e = 0; e < kEach; ++e)
#pragma unroll
        for (int q = 0; q < kReduceCols; ++q) held[e * 16 + warp][q][lane] = v[e][q];
      __syncthreads();
      const int n = min(kAtOnce, pieces - g0);
      if (warp < kReduceCols)
        for (int i = 0; i < n; ++i) {
          run[0] = __fadd_rn(run[0], held[i][warp][lane]);
          if (((i + 1) & (chunk - 1)) == 0) close_run(0);
        }
    }
    if (warp >= kReduceCols) return;
  } else {
    constexpr int DEPTH = 4;
    for (int g = 0; g < pieces; g += DEPTH) {
      float v[DEPTH][COLS];
#pragma unroll
      for (int d = 0; d < DEPTH; ++d) {
        if (g + d < pieces) {
          const float* ws = piece(g + d) + (size_t)c0 * BM + row;
#pragma unroll
          for (int q = 0; q < COLS; ++q) v[d][q] = __ldcg(ws + (size_t)q * BM);
        }
      }
#pragma unroll
      for (int d = 0; d < DEPTH; ++d)
        if (g + d < pieces) {
#pragma unroll
          for (int q = 0; q < COLS; ++q) {
            run[q] = __fadd_rn(run[q], v[d][q]);
            if (((g + d + 1) & (chunk - 1)) == 0) close_run(q);
          }
        }
    }
  }
#pragma unroll
  for (int q = 0; q < COLS; ++q) {
    close_run(q);
    // infinities and NaN as a plain sum has them
    if (fabsf(sum[q]) <= FLT_MAX) sum[q] = __fadd_rn(sum[q], lost[q]);
  }
  const RowAddr ra = row_address(p, mt, tap, row);
  const float inv_scale = (1.f / __ldg(p.a_scale)) * (1.f / __ldg(p.b_scale));
  uint32_t top = 0;
#pragma unroll
  for (int q = 0; q < COLS; ++q) {
    const int n = nt * BN + c0 + q;
    if (ra.ok && n < p.N) {
      p.out[ra.base + (long long)n * ra.col_stride] = sum[q] * inv_scale;
      top = max(top, amax_bits(sum[q] * inv_scale));
    }
  }
  if (!p.amax) return;
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0 && top) atomicMax(p.amax, top);
}
template <int BN, bool MANY>
__global__ void __launch_bounds__(kReduceThreads<MANY>) reduce_partials_kernel(const __grid_constant__ GemmParams p) {
  grid_dep_sync();
  const int t = blockIdx.x;                            // tail tile
  // Cut at common stages: piece g sits in slot g * tail_tiles + t.  Otherwise CTA g of the GEMM covered stages
  // [g * share, (g + 1) * share) of the tail; its first piece belongs to tail tile (g * share) / k_total and its pieces sit in
  // consecutive slots
  const bool aligned = p.tail_pieces > 0;
  const int first = aligned ? 0 : (int)(((long long)t * p.k_total) / p.tail_share);
  const int last = aligned ? p.tail_pieces - 1 : (int)((((long long)t + 1) * p.k_total - 1) / p.tail_share);
  reduce_tile<BN, MANY>(p, p.full_tiles + t, last - first + 1, p.sum_run, [&](int i) -> const float* {
    const int g = first + i;
    const int slot = aligned ? g * p.tail_tiles + t : g * p.slots_per_cta + (t - (int)(((long long)g * p.tail_share) / p.k_total));
    return p.workspace + (size_t)slot * BN * BM;
  });
}

template <int BN, bool MANY>
__global__ void __launch_bounds__(kReduceThreads<MANY>) reduce_group_kernel(const __grid_constant__ GroupTable t) {
  grid_dep_sync();
  const int4 e = __ldg(t.sums + blockIdx.x);
  const GemmParams& p = t.problems[e.x];
  const int pieces = tile_pieces(p, e.y), between = abs(e.w);
  reduce_tile<BN, MANY>(p, e.y, e.w < 0 ? (pieces + kSumChunk - 1) / kSumChunk : pieces, e.w < 0 ? 1 : kSumChunk,
                        [&](int g) -> const float* { return t.workspace + (size_t)(e.z + g * between) * BN * BM; });
}

// Exercises the bounded wait on its own: one thread waits, with a short limit, on a barrier that nothing arms; the wait
// gives up, raises the CTA's abort flag and the kernel reports it through the error word exactly as the GEMM does.
__global__ void barrier_timeout_probe_kernel(long long limit_cycles, int* err) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const bool flipped = mbar_wait(&bar, 0, &abort_flag, limit_cycles);
    if (!flipped && abort_flag && err) atomicExch(err, 1);
  }
}

// ------------------------------------------------------------------------------------------------
// packing kernels (fp32 -> power-of-two scale + hi / lo fp16 pair)
// ------------------------------------------------------------------------------------------------
// Largest magnitude of a tensor, as the bit pattern of a non-negative float (unsigned order = float order).
__global__ void __launch_bounds__(256) amax_kernel(const float* __restrict__ src, long long n, uint32_t* __restrict__ amax) {
  grid_dep_sync();
  uint32_t m = 0;
  const long long stride = (long long)gridDim.x * blockDim.x, tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  auto fold = [&](float4 v) {
    m = max(max(m, __float_as_uint(fabsf(v.x))), max(__float_as_uint(fabsf(v.y)), max(__float_as_uint(fabsf(v.z)), __float_as_uint(fabsf(v.w)))));
  };
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const float4* s4 = reinterpret_cast<const float4*>(src);
    const long long n4 = n / 4;
    long long i = tid;
    for (; i + 3 * stride < n4; i += 4 * stride) {       // four independent 16-byte loads in flight per thread
      float4 a = __ldg(s4 + i), b = __ldg(s4 + i + stride), c = __ldg(s4 + i + 2 * stride), d = __ldg(s4 + i + 3 * stride);
      fold(a); fold(b); fold(c); fold(d);
    }
    for (; i < n4; i += stride) fold(__ldg(s4 + i));
    for (long long k = n4 * 4 + tid; k < n; k += stride) m = max(m, __float_as_uint(fabsf(__ldg(src + k))));
  } else {
    for (long long i = tid; i < n; i += stride) m = max(m, __float_as_uint(fabsf(__ldg(src + i))));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m) atomicMax(amax, m);
}
// Scale words of one pack: amax[0..1] alternate between uses (the pack kernel of use k reads amax[k & 1] and clears
// amax[(k + 1) & 1] for the next use, so no separate clearing launch is needed), scale = the power of two in force.
// keep: where the maximum in force is left for other packs of the same tensor.
struct ScaleRef { const uint32_t* amax_cur; uint32_t* amax_next; float* scale; uint32_t* keep; };
// s = 2^(14 - floor(log2 amax)): amax * s lies in [2^14, 2^15), below the fp16 maximum 65504 after rounding
__device__ __forceinline__ float scale_from_amax(uint32_t bits) {
  int e = (int)((bits >> 23) & 0xff);
  if (bits == 0 || e == 0xff) return 1.f;             // all zero, or Inf/NaN inside (the results are meaningless then)
  if (e == 0) e = 1;
  int se = 14 - (e - 127);
  se = se > 120 ? 120 : (se < -120 ? -120 : se);
  return __uint_as_float((uint32_t)(se + 127) << 23);
}
// A tf32 pack is not scaled: its ScaleRef has no amax word and the scale in force is 1.
__device__ __forceinline__ float pack_scale(const ScaleRef& r, bool first_thread) {
  const float s = r.amax_cur ? scale_from_amax(__ldg(r.amax_cur)) : 1.f;
  if (first_thread) { *r.scale = s; if (r.amax_next) *r.amax_next = 0; if (r.keep) *r.keep = __ldg(r.amax_cur); }
  return s;
}
// hi / lo pair of one value: fp16 (22 mantissa bits together) or tf32 (round to nearest, low 13 bits zero)
__device__ __forceinline__ void split_pair(float a, __half& hi, __half& lo) {
  hi = __float2half_rn(a);
  lo = __float2half_rn(a - __half2float(hi));
}
__device__ __forceinline__ float tf32_rn(float a) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(a));
  return __uint_as_float(r);
}
__device__ __forceinline__ void split_pair(float a, float& hi, float& lo) {
  hi = tf32_rn(a);
  lo = tf32_rn(a - hi);
}
// eight consecutive values -> eight hi and eight lo elements at hi + o, lo + o (o a multiple of 8): 16-byte stores
__device__ __forceinline__ void store8(__half* hi, __half* lo, long long o, const float* v) {
  __align__(16) __half2 h[4];
  __align__(16) __half2 l[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    h[e] = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
    const float2 hf = __half22float2(h[e]);
    l[e] = __floats2half2_rn(v[2 * e] - hf.x, v[2 * e + 1] - hf.y);
  }
  *reinterpret_cast<uint4*>(hi + o) = *reinterpret_cast<const uint4*>(h);
  *reinterpret_cast<uint4*>(lo + o) = *reinterpret_cast<const uint4*>(l);
}
__device__ __forceinline__ void store8(float* hi, float* lo, long long o, const float* v) {
  float h[8], l[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) split_pair(v[e], h[e], l[e]);
  float4* hp = reinterpret_cast<float4*>(hi + o);
  float4* lp = reinterpret_cast<float4*>(lo + o);
  hp[0] = make_float4(h[0], h[1], h[2], h[3]); hp[1] = make_float4(h[4], h[5], h[6], h[7]);
  lp[0] = make_float4(l[0], l[1], l[2], l[3]); lp[1] = make_float4(l[4], l[5], l[6], l[7]);
}

// rows x cols row-major (pitch src_ld) -> hi/lo with pitch dst_ld.  VEC8: eight consecutive columns per thread
// (two 16-byte loads, one 16-byte store each of hi and lo); needs cols and src_ld multiples of 8 and a 16-byte
// aligned source (the packs' pitch is a multiple of 64).
template <bool VEC8, class E>
__global__ void __launch_bounds__(256) pack_matrix_kernel(const float* __restrict__ src, long long src_ld, E* __restrict__ hi, E* __restrict__ lo,
                                                          long long dst_ld, long long rows, long long cols, ScaleRef sr) {
  grid_dep_sync();
  const float sc = pack_scale(sr, blockIdx.x == 0 && threadIdx.x == 0);
  const long long stride = (long long)gridDim.x * blockDim.x;
  if (VEC8) {
    const long long cols8 = cols >> 3, total = rows * cols8;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
      const long long r = i / cols8, c = (i - r * cols8) << 3;
      const float4 a = __ldg(reinterpret_cast<const float4*>(src + r * src_ld + c));
      const float4 b = __ldg(reinterpret_cast<const float4*>(src + r * src_ld + c) + 1);
      const float v[8] = {a.x * sc, a.y * sc, a.z * sc, a.w * sc, b.x * sc, b.y * sc, b.z * sc, b.w * sc};
      store8(hi, lo, r * dst_ld + c, v);
    }
  } else {
    const long long total = rows * cols;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
      long long r = i / cols, c = i - r * cols;
      E h, l;
      split_pair(src[r * src_ld + c] * sc, h, l);
      hi[r * dst_ld + c] = h;
      lo[r * dst_ld + c] = l;
    }
  }
}

// NCHW activations -> pixel-major frame [N][frame_h][frame_w][pitch]:
//   dst(n, i, j, dst_c0 + c) = src(n, c, i * sh - off_h, j * sw - off_w) when that sample exists, else 0
// (off > 0 places the source behind a zero halo; off <= 0 with sh > 1 selects one phase of a strided sampling).
// Channels c < c_limit are written (zeros past C).  One block moves 32 frame columns x TC channels of one frame
// row through shared memory: reads run along w (TC/8 independent loads per thread in flight), writes along c as
// 16-byte vectors (8 halves) of hi and of lo.
struct PackGeom { int N, C, H, W, frame_h, frame_w, off_h, off_w, sh, sw, pitch, dst_c0, c_limit; };
// kPackRelu: the source is the input of a ReLU; the kernel applies it, writes the fp32 result to y_out (same layout as the
// source), records max|y| like the stand-alone ReLU kernel does, and packs y.  The pack's scale then comes from max|x|, an
// upper bound of max|y| that is known before the pass starts.  kPackReluBwd: the same for the ReLU's backward, y = mask > 0 ? x : 0.
// HBM-bound: 16 and 20 bytes an element where the two kernels one after the other move 20 and 24.
enum { kPackPlain = 0, kPackRelu = 1, kPackReluBwd = 2 };
template <int TC, class E, int MODE>
__global__ void __launch_bounds__(256) pack_nchw_kernel(const float* __restrict__ src, E* __restrict__ hi, E* __restrict__ lo, PackGeom g, ScaleRef sr,
                                                        const float* __restrict__ mask, float* __restrict__ y_out, AmaxOut am) {
  grid_dep_sync();
  // tile[c][f ^ (c / 8)]: the XOR keeps both phases free of bank conflicts (stores: 32 lanes = 32 frame positions
  // of one channel; loads: lanes = 8-channel groups of a few positions that are TC/8 apart)
  __shared__ float tile[TC][32];
  const float sc = pack_scale(sr, blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0);
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;      // 32 x 8
  const int fsize = g.frame_h * g.frame_w;
  const int f0 = blockIdx.y * 32;                              // 32 consecutive frame positions (row-major over the frame)
  const int cblocks = (g.c_limit + TC - 1) / TC;               // blocks cover every column that has to be defined
  const int n = blockIdx.x / cblocks, c0 = (blockIdx.x % cblocks) * TC;
  {
    const int f = f0 + tx, i = f / g.frame_w, j = f - i * g.frame_w;
    const int si = i * g.sh - g.off_h, sj = j * g.sw - g.off_w;
    const bool ok = f < fsize && si >= 0 && si < g.H && sj >= 0 && sj < g.W;
    const long long plane = (long long)g.H * g.W;
    // one 64-bit address per thread, advanced by eight planes per load; the range checks are hoisted out of the
    // unrolled loads (a block whose channels all exist and a thread whose position has a source take the plain path)
    const float* sp = src + ((long long)n * g.C + c0 + ty) * plane + (long long)si * g.W + sj;
    const long long step = 8 * plane;
    const int avail = g.C - c0 - ty;                  // channels at or after this thread's first one
    float v[TC / 8];
    if (ok && c0 + TC <= g.C) {
#pragma unroll
      for (int k = 0; k < TC / 8; ++k) { v[k] = __ldg(sp); sp += step; }
    } else if (ok) {
#pragma unroll
      for (int k = 0; k < TC / 8; ++k) { v[k] = 8 * k < avail ? __ldg(sp) : 0.f; sp += step; }
    } else {
#pragma unroll
      for (int k = 0; k < TC / 8; ++k) v[k] = 0.f;
    }
    if (MODE != kPackPlain) {
      uint32_t m = 0;
      if (ok) {
        const long long at = (sp - src) - (long long)(TC / 8) * step;       // the element the first load read
        float* yp = y_out + at;
        if (MODE == kPackReluBwd) {
          const float* mp = mask + at;
          float u[TC / 8];
#pragma unroll
          for (int k = 0; k < TC / 8; ++k) { u[k] = 8 * k < avail ? __ldg(mp) : 0.f; mp += step; }
#pragma unroll
          for (int k = 0; k < TC / 8; ++k) v[k] = u[k] > 0.f ? v[k] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < TC / 8; ++k) {
          const float x = v[k];
          if (MODE == kPackRelu) v[k] = x > 0.f ? x : (x != x ? x : 0.f);    // NaN propagates
          if (8 * k < avail) { *yp = v[k]; m = max(m, amax_bits(v[k])); }
          yp += step;
        }
      }
      amax_commit(am, m);
    }
    float* trow = &tile[ty][0];
#pragma unroll
    for (int k = 0; k < TC / 8; ++k) trow[k * 8 * 32 + (tx ^ k)] = v[k] * sc;       // channel ty + 8k, column tx ^ ((ty + 8k) >> 3)
  }
  __syncthreads();
  {
    // a warp pass writes 32 / LPP whole pixels: lane -> (pixel slot, 8-channel group); 16-byte stores of hi and of lo
    constexpr int LPP = TC / 8;                       // lanes per pixel
    const int grp = tx % LPP, px = tx / LPP, cl = grp * 8, c = c0 + cl;
    for (int jb = ty; jb < LPP; jb += 8) {
      const int ff = jb + px * LPP, f = f0 + ff;
      if (f < fsize && c < g.c_limit) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = tile[cl + e][ff ^ grp];
        store8(hi, lo, ((long long)n * fsize + f) * g.pitch + g.dst_c0 + c, v);
      }
    }
  }
}

// NCHW activations -> explicit patch matrix [N*P*Q][pitch], column (c*R + r)*S + s = the filter's own flat index
// within one output channel, so the convolution becomes a 1x1 one over C*R*S "channels".  Used where the
// channel count is too small to fill a 64-wide reduction chunk per tap (first layers, C = 3).
// A block makes the patches of `span` outputs of one output row: the C*R input rows they read go to shared memory, scaled and with
// their zeros, once; a thread keeps to one group of 8 columns, whose offsets stay in its registers, and writes 16 bytes of hi and of lo
// per output.  Columns past the last group are left as they are: the forward product's tensor map ends at the last column, and in
// the filter gradient they reach only outputs that are not stored.  Bound by HBM writes; with two columns a lane, gathered from
// global memory, instructions bound it (3x3 of 3 channels, 224 x 224, batch 64: 715 us, now 137; 7x7 stride 2: 255, now 203, where the gathered reads meet in banks).
struct PatchGeom { int C, H, W, R, S, P, Q, sh, sw, pad_h, pad_w, cols, pitch, span, groups; };
constexpr int kPatchFloats = 8192;            // input rows of a block
template <class E>
__global__ void __launch_bounds__(256) pack_patches_kernel(const float* __restrict__ src, E* __restrict__ hi, E* __restrict__ lo, const __grid_constant__ PatchGeom g, ScaleRef sr) {
  extern __shared__ float patch_rows[];
  grid_dep_sync();
  const float sc = pack_scale(sr, blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0);
  const int n = blockIdx.x / g.P, p = blockIdx.x - n * g.P, q0 = blockIdx.y * g.span, count = min(g.span, g.Q - q0);
  const int width = (g.span - 1) * g.sw + g.S, i0 = p * g.sh - g.pad_h, j0 = q0 * g.sw - g.pad_w;
  for (int row = threadIdx.x >> 5; row < g.C * g.R; row += 8) {            // a warp a row
    const int c = row / g.R, i = i0 + row - c * g.R;
    const bool inside = i >= 0 && i < g.H;
    const float* const from = src + (((long long)n * g.C + c) * g.H + (inside ? i : 0)) * g.W;
#pragma unroll 4
    for (int x = threadIdx.x & 31; x < width; x += 32) {
      const int j = j0 + x;
      patch_rows[row * width + x] = inside && j >= 0 && j < g.W ? __ldg(from + j) * sc : 0.f;
    }
  }
  __syncthreads();
  const int per = blockDim.x / g.groups, lane = threadIdx.x / g.groups, group = threadIdx.x - lane * g.groups;
  if (lane >= per) return;
  int off[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int col = group * 8 + e, row = col / g.S;
    off[e] = col < g.cols ? row * width + col - row * g.S : -1;
  }
  const long long first = (long long)blockIdx.x * g.Q + q0;
  for (int q = lane; q < count; q += per) {
    const float* const at = patch_rows + q * g.sw;
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = off[e] >= 0 ? at[off[e]] : 0.f;
    store8(hi, lo, (first + q) * g.pitch + group * 8, v);
  }
}

// Filters [K][C][taps] -> the forward layout [K][tap][C up to pad_f] and / or the backward-data layout [C][flipped tap][K up to
// pad_d].  One launch packs any number of filters: a step's 50-150 filters, packed when their convolution came up, were as
// many launches of 5 us for 1-2 us of traffic.  A block moves 32 x 32 filters through shared memory, so that the fp32 words are
// read in order and both layouts are written in rows of 64 bytes; read straight from the filter, the backward-data layout took a
// sector per element.  Where a launch packs many filters the instructions bound it before HBM (12 bytes an element) does: rows that lie in
// one run are read 16 bytes at a time without a division, both layouts are written 16 bytes a thread, and a block of a 1x1 filter
// takes 288 channels (Inception-v3, 24 million: 126 -> 68 us, 4.2 TB/s; VGG-16 at 15 million 63 -> 37).  Where it packs one (an ordinary step
// packs each filter when its convolution comes up), by the latency of a block's loads: it takes up to 9 taps, 36 loads a thread
// one behind the other, unless `tap_step` spreads the taps over more blocks, which read the same sectors again from L2.
struct FilterJob {
  const float* w;
  void *hi_f, *lo_f, *hi_d, *lo_d;       // a layout that is not wanted: null
  const uint32_t* amax; uint32_t* amax_next;
  float *scale_f, *scale_d;
  int K, C, taps, pad_f, pad_d, k_blocks, c_blocks, first_block;
};
// MAX is 1 or kFilterJobs: the table travels as a kernel parameter, and 13 KB of it cost a launch of one filter 10 us.
constexpr int kFilterJobs = 128, kFilterTaps = 9, kFilterTile = 32;
template <int MAX> struct FilterJobs { int n, tap_step; FilterJob job[MAX]; };
template <class E, int MAX>
__global__ void __launch_bounds__(256) pack_filters_kernel(const __grid_constant__ FilterJobs<MAX> jobs) {
  grid_dep_sync();
  __shared__ float tile[kFilterTile][kFilterTile * kFilterTaps + 1];
  int lo = 0, hi = jobs.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs.job[mid].first_block <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const FilterJob& j = jobs.job[lo];
  const int block = blockIdx.x - j.first_block, kc = block / j.k_blocks;
  const int wide = j.taps == 1 ? jobs.tap_step : 1;            // a 1x1 filter: as many blocks of 32 channels as others have taps
  const int k0 = (block - kc * j.k_blocks) * kFilterTile, c0 = kc % j.c_blocks * kFilterTile * wide, t0 = kc / j.c_blocks * jobs.tap_step;
  const float sc = j.amax ? scale_from_amax(__ldg(j.amax)) : 1.f;
  if (block == 0 && threadIdx.x == 0) {
    if (j.scale_f) *j.scale_f = sc;
    if (j.scale_d) *j.scale_d = sc;
    if (j.amax_next) *j.amax_next = 0u;
  }
  const int taps = j.taps, K = j.K, C = j.C, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  E *const hi_f = (E*)j.hi_f, *const lo_f = (E*)j.lo_f, *const hi_d = (E*)j.hi_d, *const lo_d = (E*)j.lo_d;
  const int nt = min(jobs.tap_step, taps - t0), row = kFilterTile * wide * nt;
  const int there = min(kFilterTile * wide, C - c0) * taps;           // floats of a row of the tile when it holds all taps
  if (nt == taps && ((uintptr_t)j.w & 15) == 0 && (C * taps & 3) == 0) {        // then they lie in one run, beginning at a multiple of 16 bytes
    for (int r = warp; r < kFilterTile; r += 8) {
      const float* src = j.w + ((long long)(k0 + r) * C + c0) * taps;
      const int n = k0 + r < K ? there : 0;
#pragma unroll
      for (int i = 0; i < (kFilterTile * kFilterTaps + 127) / 128; ++i) {
        const int e = 4 * (lane + 32 * i);
        if (e >= row) break;
        const float4 v = e < n ? __ldg(reinterpret_cast<const float4*>(src + e)) : make_float4(0.f, 0.f, 0.f, 0.f);
        tile[r][e] = v.x * sc; tile[r][e + 1] = v.y * sc; tile[r][e + 2] = v.z * sc; tile[r][e + 3] = v.w * sc;
      }
    }
  } else {
    for (int r = warp; r < kFilterTile; r += 8) {
      const float* src = j.w + ((long long)(k0 + r) * C + c0) * taps + t0;
      for (int e = lane; e < row; e += 32) {
        const int c = e / nt, t = e - c * nt;
        tile[r][e] = k0 + r < K && c0 + c < C ? __ldg(src + (long long)c * taps + t) * sc : 0.f;
      }
    }
  }
  __syncthreads();
  // eight values along the packed dimension a thread: 4 lanes write 64 bytes of a row, lanes of a warp read different banks
  const int eight = (threadIdx.x & 3) * 8;
  const int per_row = nt * wide;
  for (int line = threadIdx.x >> 2; line < row; line += 64) {
    float v[8];
    if (hi_f) {
      const int r = line / per_row, u = line - r * per_row, t = wide > 1 ? 0 : u, c = (wide > 1 ? u * kFilterTile : 0) + eight;
      if (k0 + r < K && c0 + c < j.pad_f) {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = tile[r][(c + e) * nt + t];
        store8(hi_f, lo_f, ((long long)(k0 + r) * taps + t0 + t) * j.pad_f + c0 + c, v);
      }
    }
    const int r = line / nt, t = line - r * nt;
    if (hi_d && c0 + r < C && k0 + eight < j.pad_d) {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = tile[eight + e][r * nt + t];
      store8(hi_d, lo_d, ((long long)(c0 + r) * taps + taps - 1 - t0 - t) * j.pad_d + k0 + eight, v);
    }
  }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
    return (EncodeTiledFn)p;
  }();
  return fn;
}
static inline CUtensorMapDataType map_type(int ar) { return ar == kArithTF32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16; }

// 2-D row-major [rows][cols] with `pitch` elements per row; box = one 128-byte row of K x box_rows rows, 128-byte swizzle.
static int make_map(CUtensorMap* m, int ar, const void* base, long long rows, long long cols, long long pitch, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  TF_REQUIRE(fn, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)pitch * elem_of(ar)};
  cuuint32_t box[2] = {(cuuint32_t)bk_of(ar), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, map_type(ar), 2, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TF_REQUIRE(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed with %d (rows %lld cols %lld pitch %lld)", (int)r, rows, cols, pitch);
  return 0;
}
// M/N-major operand: 3-D view {group width, rows, pitch / group width column groups} (a group is 128 bytes of M/N) with
// a box of `tile_cols` columns x one stage of K rows.  The pack's pitch is a multiple of 64 elements, so every group lies
// inside the allocation; columns past the logical width only reach output rows / columns that the epilogue masks.
static int make_map_mn(CUtensorMap* m, int ar, const void* base, long long rows, long long pitch, int tile_cols) {
  EncodeTiledFn fn = encode_fn();
  TF_REQUIRE(fn, "cuTensorMapEncodeTiled is not available from this driver");
  const int gw = gw_of(ar);
  TF_REQUIRE(pitch % gw == 0 && tile_cols % gw == 0, "M/N-major operand: pitch %lld / tile width %d are not multiples of %d", pitch, tile_cols, gw);
  cuuint64_t dims[3] = {(cuuint64_t)gw, (cuuint64_t)rows, (cuuint64_t)(pitch / gw)};
  cuuint64_t strides[2] = {(cuuint64_t)pitch * elem_of(ar), 128};
  cuuint32_t box[3] = {(cuuint32_t)gw, (cuuint32_t)bk_of(ar), (cuuint32_t)(tile_cols / gw)};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(m, map_type(ar), 3, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  ar == kArithTF32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TF_REQUIRE(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled (3-D) failed with %d (rows %lld pitch %lld tile %d)", (int)r, rows, pitch, tile_cols);
  return 0;
}

static std::mutex g_tc_mu;      // guards the lazily created process-wide state below
static int* error_word() {      // mapped pinned word: the kernels raise it, the host polls it for free
  static int* host = nullptr;
  static int* dev = nullptr;
  std::lock_guard<std::mutex> lk(g_tc_mu);
  if (!host) {
    if (cudaHostAlloc((void**)&host, sizeof(int), cudaHostAllocMapped) != cudaSuccess) { cudaGetLastError(); host = nullptr; return nullptr; }
    *host = 0;
    if (cudaHostGetDevicePointer((void**)&dev, host, 0) != cudaSuccess) { cudaGetLastError(); dev = nullptr; }
  }
  return dev;
}
static int* error_word_host() {
  static std::atomic<int*> host{nullptr};
  int* h = host.load(std::memory_order_acquire);
  if (!h) {
    int* dev = error_word();
    if (!dev) return nullptr;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, dev) == cudaSuccess) { h = (int*)at.hostPointer; host.store(h, std::memory_order_release); }
  }
  return h;
}
int tensor_path_error() { int* h = error_word_host(); return h ? *(volatile int*)h : 0; }
void tensor_path_error_clear() { int* h = error_word_host(); if (h) *(volatile int*)h = 0; }

int tensor_path_timeout_probe(long long limit_cycles, cudaStream_t s) {
  int* err = error_word();
  TF_REQUIRE(err, "the error word could not be mapped");
  TF_REQUIRE(limit_cycles > 0 && limit_cycles <= 2000000000ll, "limit must be between 1 and 2e9 cycles");
  barrier_timeout_probe_kernel<<<1, 32, 0, s>>>(limit_cycles, err);
  return after_launch(s, "barrier_timeout_probe", 1);
}

// Arithmetic of the tensor path: 0 = 3xFP16 (scaled fp16 hi/lo pairs, kind::f16), 1 = 3xTF32 (tf32 hi/lo pairs, kind::tf32).
static std::atomic<int> g_arith{[] { const char* e = getenv("TINYFLOW_ARITH"); return (e && (!strcmp(e, "3xtf32") || !strcmp(e, "1"))) ? 1 : 0; }()};
int tensor_arithmetic() { return g_arith.load(std::memory_order_relaxed); }
void set_tensor_arithmetic(int a) { if (g_arith.exchange(a, std::memory_order_relaxed) != a) bump_layout_epoch(); }

// ---- schedule: whole waves of tiles, then the partial wave cut into equal per-CTA ranges of stages -------------------
// Costs are in units of one stage of one tile.  Splitting the tail pays a fixed price per CTA (the partial sums make a
// round trip through the workspace and a second kernel adds them), so it is taken only when the tail is clearly
// unbalanced and its reductions are long enough to share.
static float g_tail_gain = [] { const char* e = getenv("TINYFLOW_TAIL_GAIN"); return e ? (float)atof(e) : 0.9f; }();
static float g_tail_cost = [] { const char* e = getenv("TINYFLOW_TAIL_COST"); return e ? (float)atof(e) : 12.f; }();     // workspace round trip + second kernel, in stages
// A reduction over few tiles is cut over clusters of 2-8 CTAs instead (sum in shared memory, no workspace and no second
// kernel); `max_clusters(c)` says how many clusters of c the device runs at once.  The sum costs about 6 stages whatever
// the cluster (768 -> 192 channels, 17 x 17, 1x1, batch 2: 17.0 -> 15.3 us in clusters of 6).  Against it the workspace costs
// 4 stages and 0.15 per tile (its traffic): 70 tiles of 36 stages 34.0 us split and 29.7 in clusters of 2, 40 of 72
// stages 33.8 and 32.5 in clusters of 3, but 12 of 72 stages 19.2 and 23 in clusters of 8.
// How the partial wave is cut.  With a contiguous range of stages per CTA all SMs work, but the ranges of different tiles begin at
// different stages: a filter gradient, whose tiles all read both operands along K, then fetches them from HBM once per CTA when
// L2 cannot hold them (256 -> 256 channels, 57 x 57 frames, batch 64, 36 tiles: 990 us, 7.5 TB/s of operands), and most CTAs
// leave two partial sums.  Cut at the same stages into as many pieces as there are CTAs for, the CTAs of a range share what they
// fetch (736 us; with two issuers 672), and each leaves one sum (768 -> 192 channels, 17 x 17, 1x1, batch 32: 33.0 -> 28.0 us).  The price is idle
// CTAs where sms / tiles is not whole: up to 10 % where operands are read once, 25 % for filter gradients, 50 % beyond L2.
static constexpr double kL2Holds = 64e6;
// Stages that one running sum takes before it is put down: a sum's rounding grows with its length, and another 64 KB per 384 stages
// (300 us) cost nothing.
static constexpr int kLongestSum = 384;
template <class MaxClusters> static size_t plan_schedule(GemmParams& g, int bn, MaxClusters max_clusters) {       // bytes of workspace
  const int sms = device_sm_count();
  const int tiles = g.m_tiles * g.n_tiles * g.tap_tiles;
  g.full_tiles = tiles; g.tail_tiles = 0; g.tail_share = 0; g.slots_per_cta = 0; g.tail_pieces = g.tail_run = 0; g.workspace = nullptr; g.cluster = 1;
  const int rem = tiles % sms;
  static const bool no_split = getenv("TINYFLOW_NO_TAIL_SPLIT") != nullptr;
  if (rem == 0 || no_split) return 0;
  const double whole = g.k_total + 8.0;
  const double limit = g_tail_gain * whole;
  double best = limit;
  if (tiles < sms) {
    for (int c = 2; c <= kMaxCluster && c <= g.k_total && tiles * c <= sms; ++c) {
      const double cost = (g.k_total + c - 1) / c + 8.0 + 6.0;
      if (cost < best && tiles <= max_clusters(c)) { best = cost; g.cluster = c; }
    }
  }
  if (g.k_total < 8) return 0;
  const long long units = (long long)rem * g.k_total;
  int share = (int)((units + sms - 1) / sms);
  if (share < 4) share = 4;                                   // shorter pieces are all overhead
  if (share + 8.0 + g_tail_cost >= limit || (g.cluster > 1 && share + 8.0 + 4.0 + 0.15 * rem >= best)) return 0;
  g.cluster = 1;
  g.full_tiles = tiles - rem; g.tail_tiles = rem; g.tail_share = share;
  g.slots_per_cta = (share - 1 + g.k_total - 1) / g.k_total + 1;       // tiles a range of `share` stages can touch
  int ctas = (int)((units + share - 1) / share);
  // All tiles cut at the same stages, one piece a CTA, wherever that leaves few CTAs idle.
  const int pieces = std::min(sms / rem, g.k_total / 2);          // two stages at least
  if (pieces >= 2) {
    const int even = (g.k_total + pieces - 1) / pieces;
    const double slack = !(g.a_mn && g.b_mn) ? 1.1 : g.operand_bytes > kL2Holds ? 1.5 : 1.25;
    if (even <= share * slack) {
      g.tail_run = (even + kLongestSum - 1) / kLongestSum;
      g.tail_pieces = pieces * g.tail_run; g.tail_share = even; g.slots_per_cta = g.tail_run; ctas = rem * pieces;
    }
  }
  return (size_t)ctas * g.slots_per_cta * bn * BM * sizeof(float);
}
// How shared memory is dealt to the two rings, and whether the B tile of a CTA stays there: with all of a CTA's tiles in one
// column of the grid (its size a multiple of n_tiles) and room for every stage of B beside two A blocks.
static int plan_smem(GemmParams& g, int bn, int grid) {
  const int limit = kSmemLimit - kSmemBarriers, a = g.a_rows * 256, b = bn * 256;
  const int tiles = g.full_tiles + g.tail_tiles;
  g.b_resident = g.one_ring = 0;
  if (g.acc_mode == kAccPair && g.mode != kModeWgrad && g.tail_share == 0 && g.cluster == 1 && tiles > grid && g.n_tiles <= 4 && g.k_total <= kMaxBSlots && g.k_total * b + 2 * a <= limit) {
    g.b_resident = 1;
    g.b_slots = g.k_total;
    g.a_slots = std::min(kMaxASlots, (limit - g.k_total * b) / a);
    return grid / g.n_tiles * g.n_tiles;
  }
  if (g.a_rows > BM) {
    g.a_slots = 2;
    g.b_slots = std::min(kMaxBSlots, (limit - 2 * a) / b);
  } else {
    g.a_slots = g.b_slots = std::min(kMaxASlots, limit / (a + b));
    g.one_ring = 1;
  }
  return grid;
}

// The kernel may use all shared memory: asked for ahead of its first launch and of the first question how many clusters of it fit
template <int BN, int AR> static cudaError_t gemm_kernel_ready() {
  static const cudaError_t attr = cudaFuncSetAttribute(gemm3x_kernel<BN, AR>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit + 1024);
  return attr;
}
template <int BN, int AR> static int max_clusters_of(int c) {
  static std::atomic<int> known[9];
  int n = known[c].load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(c); cfg.blockDim = dim3(kGemmThreads); cfg.dynamicSmemBytes = kSmemLimit + 1024;
    cudaLaunchAttribute attr;
    memset(&attr, 0, sizeof(attr));
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = c; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, gemm3x_kernel<BN, AR>, &cfg) != cudaSuccess || n <= 0) { cudaGetLastError(); n = -1; }
    known[c].store(n, std::memory_order_relaxed);
  }
  return n;
}
// stages that a CTA works through for one tile
static int longest_run(const GemmParams& p) { return p.tail_share > 0 && p.full_tiles == 0 ? p.tail_share : p.k_total / p.cluster; }
// The form of the summing kernel for tiles of about that many pieces
template <int BN, class F> static cudaError_t launch_reduce(int tiles, int pieces, F&& launch) {
  const dim3 grid(tiles, BN / kReduceCols);
  if (pieces >= 12 && tiles * (BN / kReduceCols) <= 2 * device_sm_count()) return launch(std::true_type(), dim3(grid.x, grid.y, BM / 32), dim3(kReduceThreads<true>));
  return launch(std::false_type(), grid, dim3(kReduceThreads<false>));
}
// Stages per CTA from which a product is launched on its own: at 128 columns those that take two issuers (groups hold products of one
// layout of the accumulators); at 64 columns 102 still gain (DenseNet-121 13.76 -> 13.50 ms against a limit of 24).
template <int BN> constexpr int kHeldRun = BN == 64 ? 160 : 24;
// By its schedule the product could wait for others (see held_back)
template <int BN> static bool could_wait(const GemmParams& p) {
  return BN != 96 && p.group_iters == 1 && p.acc_mode == kAccPair && longest_run(p) < kHeldRun<BN> && (p.tail_share == 0 || p.tail_pieces > 0);
}
// Schedule, stages per accumulator group and accumulator blocks of a launch: what decides the bits of its result
template <int BN, int AR> static size_t plan_launch(GemmParams& p) {
  const size_t bytes = plan_schedule(p, BN, max_clusters_of<BN, AR>);
  static const int group_iters = getenv("TINYFLOW_GROUP_ITERS") ? atoi(getenv("TINYFLOW_GROUP_ITERS")) : 0;
  p.group_iters = group_iters > 0 ? group_iters : (p.data_by_data ? kGroupItersDataByData : (AR == kArithTF32 ? kGroupItersTF32 : kGroupIters));
  if (p.group_limit) p.group_iters = std::min(p.group_iters, p.group_limit);
  // cross terms promoted every 64 stages: 256 accumulations into a sum 2^-12 of the whole truncate less than 2^-28 of it
  p.cross_groups = 64 / p.group_iters;
  // Two issuers gain from 8 stages per CTA on (equal at 18 of 128 columns, 1 us of 65 at 36); at 96 columns the narrow MMAs
  // are short enough for one warp (12 stages: 19.2 against 21.2 us).
  // Groups of one stage begin the main sum anew with two instructions instead of a wide one: equal at 22 stages, 4 % faster
  // at 55, 9 % at 841 (512 -> 512 channels, 28 x 28, 3x3, batch 64: 750 -> 673 us).
  p.acc_mode = BN != 64 && p.k_total > p.group_iters && longest_run(p) >= (BN == 128 && p.group_iters > 1 ? 8 : 24) ? kAccThree : kAccPair;
  p.sum_run = could_wait<BN>(p) ? kSumChunk : 1;
  return bytes;
}
template <int BN, int AR> static bool held_back(const GemmParams& p, size_t workspace_bytes, cudaStream_t s, double flops);
template <int BN, int AR> static int launch_planned(GemmParams& p, size_t workspace_bytes, bool may_wait, cudaStream_t s, double flops, const char* what, int* oom);
template <int BN, int AR> static int launch_gemm(GemmParams& p, cudaStream_t s, double flops, const char* what, int* oom) {
  TF_CUDA((gemm_kernel_ready<BN, AR>()));
  TF_REQUIRE(tensor_path_error() == 0, "%s: an earlier tensor-core kernel timed out on a barrier; refusing to launch", what);
  const size_t bytes = plan_launch<BN, AR>(p);
  return launch_planned<BN, AR>(p, bytes, p.hold != 0, s, flops, what, oom);
}
template <int BN, int AR> static int launch_planned(GemmParams& p, size_t bytes, bool may_wait, cudaStream_t s, double flops, const char* what, int* oom) {
  StreamLease lease(s);
  // (one that waits has the workspace of a launch of its own, too: a shortage is reported by the call that meets it, see launch_some)
  if (bytes && !(p.workspace = (float*)lease.scratch(kScratchTiles, bytes))) {
    if (oom) *oom = bytes > 0x7fffffffu ? 0x7fffffff : (int)bytes;
    return 1;
  }
  if (may_wait && held_back<BN, AR>(p, bytes, s, flops)) return 0;
  const int sms = device_sm_count();
  const int tiles = p.full_tiles + p.tail_tiles;
  int grid = tiles < sms ? tiles : sms;
  if (p.tail_share > 0) {
    const int ctas = p.tail_pieces > 0 ? p.tail_tiles * (p.tail_pieces / p.tail_run) : (int)(((long long)p.tail_tiles * p.k_total + p.tail_share - 1) / p.tail_share);
    grid = p.full_tiles > 0 ? sms : ctas;
  }
  if (p.cluster > 1) grid = tiles * p.cluster;
  grid = plan_smem(p, BN, grid);
  TF_REQUIRE(p.cluster == 1 || BM * BN * 4 <= p.a_slots * p.a_rows * 256 + p.b_slots * BN * 256, "%s: a piece of a tile does not fit where its operands were", what);
  note_compute_stream(s);
  static const bool detail = getenv("TINYFLOW_TIMING_DETAIL") != nullptr;    // one timing row per distinct problem shape
  char name[192];
  if (detail) snprintf(name, sizeof(name), "gemm3x%s mode%d M%d N%d ktotal%d taps%d bn%d tiles%d tail%d share%d cl%d p%d a%dx%d b%d%s %s", AR == kArithTF32 ? "tf32" : "f16", p.mode, p.M,
                       p.N, p.k_total, p.tap_tiles, BN, tiles, p.tail_tiles, p.tail_share, p.cluster, p.tail_pieces, p.a_slots, p.a_rows, p.b_slots, p.b_resident ? "r" : "", what + 5);
  KernelTimer kt(detail ? name : (AR == kArithTF32 ? "gemm3xtf32_tcgen05" : "gemm3xf16_tcgen05"), s, flops, 0, 1);
  if (p.cluster > 1) {
    TF_CUDA(launch_cluster(gemm3x_kernel<BN, AR>, p.cluster, dim3(grid), dim3(kGemmThreads), (size_t)gemm_smem_bytes(p, BN), s, p));
  } else {
    TF_CUDA(launch_dep(gemm3x_kernel<BN, AR>, dim3(grid), dim3(kGemmThreads), (size_t)gemm_smem_bytes(p, BN), s, p));
  }
  TF_AFTER(s, what);
  if (p.tail_share > 0) {
    const int pieces = p.tail_pieces > 0 ? p.tail_pieces : p.k_total / p.tail_share + 1;
    launch_reduce<BN>(p.tail_tiles, pieces, [&](auto many, dim3 grid, dim3 block) { return launch_dep(reduce_partials_kernel<BN, decltype(many)::value>, grid, block, 0, s, p); });
    TF_AFTER(s, what);
  }
  return 0;
}
// ---- filter gradients that wait for others -------------------------------------------------------------------------
// Between TfHoldProducts(1) and (0) the caller says that nothing but TfLaunchHeld() stands between a filter gradient and its readers
// (the executor: only the parameter updates at the end of the step read it), and that what the product reads, the packs of its
// plan, is not packed anew before (release_held() looks after that; the kernels of the other files read the arrays themselves).  Products whose CTAs have many stages to do are launched
// at once: they gain nothing, and their operands are in L2 now.
struct HeldProduct { GemmParams g; int bn, ar; size_t workspace_bytes; double flops; };
static thread_local bool t_hold = false;
static thread_local std::vector<HeldProduct> t_held;
static thread_local double t_held_work = 0;           // tiles x stages
constexpr int kHeldWork = 1024;                       // stages per SM that are launched together at the latest (64: ResNet-50 b19 4096 us, 256: 3999, 512 and all: 3976)
int launch_held_simt(cudaStream_t s);       // gemm_simt.cu: weight gradients of dense layers
void drop_held_simt();
int launch_held_sums(cudaStream_t s);       // ops_basic.cu: bias gradients
void drop_held_sums();
int launch_held_direct(cudaStream_t s);     // conv_direct.cu: filter gradients of layers of few channels
void drop_held_direct();
// Whatever a thread holds was called on one stream, and is launched there.
static thread_local bool t_waiting = false;           // something is held, on t_waiting_stream
static thread_local cudaStream_t t_waiting_stream = nullptr;
void hold_products(bool on) { t_hold = on; }
static void forget_held() { t_held.clear(); t_held_work = 0; t_waiting = false; drop_held_simt(); drop_held_sums(); drop_held_direct(); }
void drop_held() { forget_held(); t_hold = false; }
static bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &capture) == cudaSuccess) return capture != cudaStreamCaptureStatusNone;
  cudaGetLastError();
  return true;
}
// The call may wait: its caller says so, nothing that waits was called on another stream, and no graph of the caller's own is being
// captured (it would copy from a table that is gone).  True: the caller holds it now.
bool may_hold(cudaStream_t s) {
  if (!t_hold || (t_waiting && s != t_waiting_stream) || capturing(t_recording ? recording_home() : s)) return false;
  t_waiting = true; t_waiting_stream = s;
  return true;
}

constexpr size_t kStagedCopy = 1 << 16;
// Partial sums that the products of one launch may have between them: the largest of the benchmark's graphs has 345 MB (DenseNet-121 at
// batch 56), one product on its own 10 MB at most.
constexpr size_t kGroupBytes = size_t(512) << 20;
// 0: launched, -1: error, 1: too many at once, no memory for the table or the partial sums, or a graph of the caller's own is being captured
// (its copy of the table would read host memory that is gone at a replay); nothing was launched
template <int BN, int AR> static int launch_group(HeldProduct* const* products, int n, cudaStream_t s) {
  static const cudaError_t attr = cudaFuncSetAttribute(gemm3x_group_kernel<BN, AR>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGroupSmem<BN>);
  TF_CUDA(attr);
  if (!t_recording && capturing(s)) return 1;
  const int sms = device_sm_count();
  // Whole tiles, or chunks of their pieces, up to half of a CTA's share (a fifth: 0.3 % slower); longer reductions as their pieces.  Longest first, to the CTA that is free first.
  constexpr int kItemCost = 4;                        // an item's start and end, in stages
  struct Item { int4 what; int stages; };
  std::vector<Item> items;
  std::vector<int4> sums;
  std::vector<const GemmParams*> held;
  double work = 0, flops = 0;
  for (int i = 0; i < n; ++i) { held.push_back(&products[i]->g); flops += products[i]->flops; }
  for (const GemmParams* g : held) work += (double)g->m_tiles * g->n_tiles * g->tap_tiles * (g->k_total + kItemCost);
  const int whole = std::max(8, (int)(work / sms / 2));
  int slots = 0, most_pieces = 0;
  for (int i = 0; i < (int)held.size(); ++i) {
    const GemmParams& g = *held[i];
    const int tiles = g.m_tiles * g.n_tiles * g.tap_tiles;
    const int width = g.k_total <= whole ? kSumChunk : 1;
    for (int part = 0, more = 1; more; ++part) {        // the parts of one range of stages side by side
      more = 0;
      for (int tile = 0; tile < tiles; ++tile) {
        const int n = tile_pieces(g, tile), parts = (n + width - 1) / width;
        if (parts == 1) {
          if (part == 0) items.push_back({make_int4(i, tile, -1, 0), g.k_total});
          continue;
        }
        if (part >= parts) continue;
        const int split = tiles - (g.cluster > 1 ? 0 : g.full_tiles), t = tile - (tiles - split);
        const int first = part * width, end = std::min(n, first + width);
        if (part == 0) { sums.push_back(make_int4(i, tile, slots + t, width > 1 ? -split : split)); most_pieces = std::max(most_pieces, parts); }
        items.push_back({make_int4(i, tile, first + ((end - first) << 16), slots + part * split + t), (int)((long long)g.k_total * end / n - (long long)g.k_total * first / n)});
        if (part + 1 < parts) more = 1;
        else if (tile + 1 == tiles) slots += parts * split;
      }
    }
  }
  const int count = (int)items.size(), grid = std::min(sms, count);
  std::vector<int> order(count), cta(count), first(grid + 1, 0);
  {
    int longest = 0;
    for (const Item& it : items) longest = std::max(longest, it.stages);
    std::vector<int> at(longest + 2, 0);
    for (const Item& it : items) ++at[longest - it.stages + 1];
    for (int k = 0; k <= longest; ++k) at[k + 1] += at[k];
    for (int i = 0; i < count; ++i) order[at[longest - items[i].stages]++] = i;
  }
  std::vector<long long> heap(grid);                   // load * 65536 + CTA, the least first
  for (int c = 0; c < grid; ++c) heap[c] = c;
  for (int i : order) {
    cta[i] = (int)(heap[0] & 0xffff);
    ++first[cta[i] + 1];
    const long long now = heap[0] + (long long)(items[i].stages + kItemCost) * 65536;
    int at = 0;
    for (int below; (below = 2 * at + 1) < grid; at = below) {
      if (below + 1 < grid && heap[below + 1] < heap[below]) ++below;
      if (heap[below] >= now) break;
      heap[at] = heap[below];
    }
    heap[at] = now;
  }
  for (int c = 0; c < grid; ++c) first[c + 1] += first[c];
  // one table on the device: the problems, the items of every CTA, the sums
  const size_t at_items = held.size() * sizeof(GemmParams), at_sums = at_items + items.size() * sizeof(int4), at_first = at_sums + sums.size() * sizeof(int4);
  std::vector<char> table(at_first + (grid + 1) * sizeof(int));
  for (size_t i = 0; i < held.size(); ++i) memcpy(table.data() + i * sizeof(GemmParams), held[i], sizeof(GemmParams));
  memcpy(table.data() + at_first, first.data(), (grid + 1) * sizeof(int));
  for (int i : order) memcpy(table.data() + at_items + sizeof(int4) * first[cta[i]]++, &items[i].what, sizeof(int4));
  if (!sums.empty()) memcpy(table.data() + at_sums, sums.data(), sums.size() * sizeof(int4));
  StreamLease lease(s);
  GroupTable t;
  t.err = error_word();
  t.workspace = nullptr;
  const size_t bytes = (size_t)slots * BN * BM * sizeof(float);
  if (n > 1 && bytes > kGroupBytes) return 1;
  if (bytes && !(t.workspace = (float*)lease.scratch(kScratchTiles, bytes))) return 1;
  char* dev;
  if (t_recording) {
    dev = (char*)recording_own(table);                // lives and is uploaded with the recording
  } else {
    dev = (char*)lease.scratch(kScratchGroup, table.size());
    // pageable: staged before the call returns, without waiting for the stream up to 64 KB a copy
    for (size_t at = 0; dev && at < table.size(); at += kStagedCopy)
      TF_CUDA(cudaMemcpyAsync(dev + at, table.data() + at, std::min(kStagedCopy, table.size() - at), cudaMemcpyHostToDevice, s));
  }
  if (!dev) return 1;
  t.problems = (const GemmParams*)dev; t.items = (const int4*)(dev + at_items); t.sums = (const int4*)(dev + at_sums); t.first = (const int*)(dev + at_first);
  note_compute_stream(s);
  KernelTimer kt(AR == kArithTF32 ? "gemm3xtf32_tcgen05" : "gemm3xf16_tcgen05", s, flops, 0, 1);
  TF_CUDA(launch_dep(gemm3x_group_kernel<BN, AR>, dim3(grid), dim3(kGemmThreads), (size_t)kGroupSmem<BN>, s, t));
  TF_AFTER(s, "filter gradients");
  if (!sums.empty()) {
    launch_reduce<BN>((int)sums.size(), most_pieces, [&](auto many, dim3 g, dim3 block) { return launch_dep(reduce_group_kernel<BN, decltype(many)::value>, g, block, 0, s, t); });
    TF_AFTER(s, "filter gradients");
  }
  return 0;
}
// As many together as there is memory for: on a full device a group gives way to its halves, and one product to the launch of its own whose
// workspace its call has seen to.  The bits are the same either way.
template <int BN, int AR> static int launch_some(HeldProduct* const* products, int n, cudaStream_t s) {
  const int rc = launch_group<BN, AR>(products, n, s);
  if (rc != 1) return rc;
  if (n > 1) {
    if (const int first = launch_some<BN, AR>(products, n / 2, s)) return first;
    return launch_some<BN, AR>(products + n / 2, n - n / 2, s);
  }
  int oom = 0;
  HeldProduct& h = *products[0];
  if (launch_planned<BN, AR>(h.g, h.workspace_bytes, false, s, h.flops, "DLGpuConvolutionBackwardFilter", &oom) == 0) return 0;
  TF_REQUIRE(!oom, "filter gradients: the device is out of memory, %d bytes of partial sums short", oom);
  return -1;
}
static int launch_held_filters(cudaStream_t s) try {
  if (t_held.empty()) return 0;
  std::vector<HeldProduct> all;
  all.swap(t_held);
  t_held_work = 0;
  TF_REQUIRE(tensor_path_error() == 0, "filter gradients: an earlier tensor-core kernel timed out on a barrier; refusing to launch");
  for (int ar : {kArithF16, kArithTF32})
    for (int bn : {64, 128}) {
      std::vector<HeldProduct*> some;
      for (HeldProduct& h : all)
        if (h.bn == bn && h.ar == ar) some.push_back(&h);
      if (some.empty()) continue;
      const int n = (int)some.size();
      const int rc = ar == kArithTF32 ? (bn == 64 ? launch_some<64, kArithTF32>(some.data(), n, s) : launch_some<128, kArithTF32>(some.data(), n, s))
                                      : (bn == 64 ? launch_some<64, kArithF16>(some.data(), n, s) : launch_some<128, kArithF16>(some.data(), n, s));
      if (rc) return rc;
    }
  return 0;
} catch (const std::bad_alloc&) { TF_FAIL("filter gradients: out of host memory"); }
// All that waits, on its own stream; after an error nothing waits any more
int launch_waiting() try {
  if (!t_waiting) return 0;
  const cudaStream_t s = t_waiting_stream;
  t_waiting = false;
  int rc = launch_held_filters(s);
  if (!rc) rc = launch_held_direct(s);
  if (!rc) rc = launch_held_simt(s);
  if (!rc) rc = launch_held_sums(s);
  if (rc) forget_held();
  return rc;
} catch (const std::bad_alloc&) { forget_held(); TF_FAIL("gradients that waited: out of host memory"); }
// What waits if it was called on this stream
int launch_held(cudaStream_t s) { return t_waiting && s == t_waiting_stream ? launch_waiting() : 0; }
// Before the pack at `hi` is written again, on stream s: what still has to read it goes first.  (While s is captured nothing is written;
// the order of what the caller makes of the capture is the caller's.)
static bool held_reads(const void* hi) {
  for (const HeldProduct& h : t_held) if (h.g.pack_a == hi || h.g.pack_b == hi) return true;
  return false;
}
static int release_held(const void* hi, cudaStream_t s) {
  if (held_reads(hi)) {
    if (int rc = launch_held_filters(t_waiting_stream)) return rc;
    if (s == t_waiting_stream || capturing(s)) return 0;
    cudaEvent_t read;
    TF_CUDA(cudaEventCreateWithFlags(&read, cudaEventDisableTiming));
    cudaError_t e = cudaEventRecord(read, t_waiting_stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s, read, 0);
    cudaEventDestroy(read);
    TF_CUDA(e);
    return 0;
  }
  return 0;
}
// Takes the product if it may wait
template <int BN, int AR> static bool held_back(const GemmParams& p, size_t workspace_bytes, cudaStream_t s, double flops) {
  if (!could_wait<BN>(p) || p.amax) return false;
  if (!may_hold(s) || !held(t_held, HeldProduct{p, BN, AR, workspace_bytes, flops})) return false;
  t_held_work += (double)p.m_tiles * p.n_tiles * p.tap_tiles * p.k_total;
  return true;
}
// CTA-pair launch: 74 clusters of two CTAs, programmatic dependent launch as everywhere else.
static bool g_pair_attr_done[2] = {false, false};
template <int AR> static int launch_gemm_pair(const GemmParams& p, cudaStream_t s, double flops, const char* what) {
  using L = PairLayout;
  {
    std::lock_guard<std::mutex> lk(g_tc_mu);
    if (!g_pair_attr_done[AR]) {
      TF_CUDA(cudaFuncSetAttribute(gemm3x_pair_kernel<AR>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal));
      g_pair_attr_done[AR] = true;
    }
  }
  TF_REQUIRE(tensor_path_error() == 0, "%s: an earlier tensor-core kernel timed out on a barrier; refusing to launch", what);
  static const int group_iters = getenv("TINYFLOW_GROUP_ITERS") ? atoi(getenv("TINYFLOW_GROUP_ITERS")) : 0;
  const_cast<GemmParams&>(p).group_iters = group_iters > 0 ? group_iters : (p.data_by_data ? kGroupItersDataByData : (AR == kArithTF32 ? kGroupItersTF32 : kGroupIters));
  const int pair_tiles = ((p.m_tiles + 1) / 2) * p.n_tiles * p.tap_tiles;
  const int pairs = std::min(device_sm_count() / 2, pair_tiles);
  note_compute_stream(s);
  static const bool detail = getenv("TINYFLOW_TIMING_DETAIL") != nullptr;
  char name[192];
  if (detail) snprintf(name, sizeof(name), "gemm3x%s pairs mode%d M%d N%d ktotal%d pairtiles%d %s", AR == kArithTF32 ? "tf32" : "f16", p.mode, p.M, p.N, p.k_total, pair_tiles, what + 5);
  KernelTimer kt(detail ? name : (AR == kArithTF32 ? "gemm3xtf32_tcgen05" : "gemm3xf16_tcgen05"), s, flops, 0, 1);
  TF_CUDA(launch_cluster(gemm3x_pair_kernel<AR>, 2, dim3(2 * pairs), dim3(kThreads), (size_t)L::kTotal, s, p));
  TF_AFTER(s, what);
  return 0;
}
// Pairs pay where the one-CTA kernel waits for operands: K-major operands, 128-column tiles, reductions of at least 8
// stages, and enough 256-row tiles to occupy the 74 pairs.
static int g_pairs_mode = [] { const char* e = getenv("TINYFLOW_PAIRS"); return e ? atoi(e) : 0; }();
static bool pairs_wanted(int bn, int m_tiles, int n_tiles, int k_total) {
  if (g_pairs_mode == 0 || bn != 128) return false;
  if (g_pairs_mode >= 2) return true;                   // 2: wherever the kernel can run (tests)
  return k_total >= 8 && ((m_tiles + 1) / 2) * n_tiles >= 60;
}
template <int AR> static int launch_gemm_ar(int bn, GemmParams& p, cudaStream_t s, double flops, const char* what, int* oom) {
  return bn == 64 ? launch_gemm<64, AR>(p, s, flops, what, oom) : bn == 96 ? launch_gemm<96, AR>(p, s, flops, what, oom) : launch_gemm<128, AR>(p, s, flops, what, oom);
}
// Plans the schedule (which may need workspace) and launches.  Returns 0 on success, -1 on error, 1 when the workspace
// could not be allocated (*oom holds the byte count).
static int launch_gemm_bn(int bn, int ar, GemmParams& p, cudaStream_t s, double flops, const char* what, int* oom) {
  if (p.a_rows == 0) p.a_rows = BM;
  return ar == kArithTF32 ? launch_gemm_ar<kArithTF32>(bn, p, s, flops, what, oom) : launch_gemm_ar<kArithF16>(bn, p, s, flops, what, oom);
}
// N-tile width.  M/N-major B operands come in 64-column groups, so they take 64 or 128; K-major ones may also take
// 96, which wastes less on widths such as 96, 160, 192 or 288.
static inline int pick_bn(long long n, bool b_k_major = false) {
  if (n <= 64) return 64;
  if (!b_k_major) return 128;
  long long w128 = (n + 127) / 128 * 128, w96 = (n + 95) / 96 * 96;
  return w96 < w128 ? 96 : 128;
}
static inline long long round_up(long long a, long long b) { return (a + b - 1) / b * b; }

struct Pack {           // a packed operand living in pooled device memory
  void* hi = nullptr; void* lo = nullptr;
  uint32_t* words = nullptr;       // device: amax[0], amax[1] (alternating between uses), scale (float), spare
  unsigned uses = 0;
  int arith = kArithF16;           // element type of hi / lo
  long long rows = 0, cols = 0, pitch = 0;
  const void* src = nullptr; uint64_t version = 0; int tag = 0;   // cache key
  uint64_t recording = 0;          // the recording whose graph fills the pack, 0: an ordinary call did
  void made_from(const void* s, uint64_t ver, int t) { src = s; version = ver; tag = t; recording = recording_id(); if (t_recording) recording_note_made(&src); }
  size_t bytes() const { return (size_t)rows * pitch * elem_of(arith); }
  const float* scale() const { return reinterpret_cast<const float*>(words + 2); }
};
// A pack for one call, in the stream's scratch: hi, lo and (outside a recording, whose words are cleared at every replay) the words.
static int pack_in_scratch(Pack& pk, StreamLease& lease, int slot, int ar, long long rows, long long cols, cudaStream_t s, int* oom) {
  pk.rows = rows; pk.cols = cols; pk.pitch = round_up(cols, 64); pk.arith = ar;
  char* const base = (char*)lease.scratch(slot, 2 * pk.bytes() + 16);          // bytes() is a multiple of 128
  if (!base) { if (oom) *oom = pk.bytes() > 0x3ffffff0u ? 0x7fffffff : (int)(2 * pk.bytes() + 16); return 1; }
  pk.hi = base; pk.lo = base + pk.bytes();
  if (t_recording) {
    for (int i = 0; i < 4; ++i) { uint32_t* w = recording_word(); if (!i) pk.words = w; }       // consecutive
    return 0;
  }
  pk.words = (uint32_t*)(base + 2 * pk.bytes());
  TF_CUDA(cudaMemsetAsync(pk.words, 0, 16, s));
  return 0;
}
static int pack_alloc(Pack& pk, int ar, long long rows, long long cols, cudaStream_t s, int* oom) {
  const long long pitch = round_up(cols, 64);
  if (!pk.words) {
    if (t_recording) TF_FAIL("a packed operand of a recorded step has never been packed before");    // its words could not be cleared now
    pk.words = (uint32_t*)pool_alloc(16);
    if (!pk.words || cudaMemsetAsync(pk.words, 0, 16, s) != cudaSuccess) { if (oom) *oom = 16; return 1; }
    pk.uses = 0;
  }
  if (pk.hi && pk.rows == rows && pk.pitch == pitch && pk.arith == ar) { pk.cols = cols; return 0; }
  if (pk.hi) { pool_free(pk.hi); pool_free(pk.lo); pk.hi = pk.lo = nullptr; bump_layout_epoch(); }
  pk.rows = rows; pk.cols = cols; pk.pitch = pitch; pk.src = nullptr; pk.arith = ar;
  pk.hi = pool_alloc(pk.bytes());
  pk.lo = pk.hi ? pool_alloc(pk.bytes()) : nullptr;
  if (!pk.lo) {
    if (pk.hi) pool_free(pk.hi);
    pk.hi = nullptr;
    if (oom) *oom = pk.bytes() > 0x7fffffffu ? 0x7fffffff : (int)pk.bytes();
    return 1;
  }
  return 0;
}
static void pack_release(Pack& pk) {
  if (pk.hi) { pool_free(pk.hi); pool_free(pk.lo); pk.hi = pk.lo = nullptr; }
  if (pk.words) pool_free(pk.words);
  pk.words = nullptr;
}
// Starts one use of the pack: reduces max|src| over n contiguous floats into this use's amax word and returns the
// references the pack kernel needs.  Several pack launches of the same use (stride phases) share one ScaleRef.
// A tf32 pack needs no maximum: its scale is 1.  `bound`: take the scale from this word instead.
static ScaleRef begin_pack(Pack& pk, const float* src, long long n, cudaStream_t s, const uint32_t* bound = nullptr) {
  ScaleRef r{nullptr, nullptr, reinterpret_cast<float*>(pk.words + 2), nullptr};
  if (pk.arith == kArithTF32) return r;
  uint32_t* fresh;                      // zero when the amax kernel below adds to it
  if (t_recording) {
    fresh = recording_word();
  } else {
    const unsigned k = pk.uses++ & 1;
    fresh = pk.words + k;
    r.amax_next = pk.words + (k ^ 1);
  }
  r.amax_cur = bound ? bound : fresh;
  if (bound) return r;
  static const bool no_track = getenv("TINYFLOW_NO_AMAX_TRACKING") != nullptr;
  if (const uint32_t* tracked = no_track ? nullptr : amax_tracked(src)) {
    r.amax_cur = tracked;               // the producer of src already reduced max|src| in its own pass
    return r;
  }
  KernelTimer kt("amax", s, 0, 4.0 * n);
  launch_dep(amax_kernel, dim3(grid_for(n, 256, 32)), dim3(256), 0, s, src, n, fresh);
  return r;
}
// *word (zero, or a maximum to add to) becomes the largest magnitude of n contiguous floats
void amax_of_array(const float* src, int64_t n, uint32_t* word, cudaStream_t s) {
  launch_dep(amax_kernel, dim3(grid_for(n, 256, 32)), dim3(256), 0, s, src, (long long)n, word);
}
// Calls `fn(hi, lo)` with the pack's buffers typed by its element type.
template <class F> static void with_elems(const Pack& pk, F&& fn) {
  if (pk.arith == kArithTF32) fn((float*)pk.hi, (float*)pk.lo);
  else fn((__half*)pk.hi, (__half*)pk.lo);
}

static int run_pack_matrix(const float* src, long long ld, Pack& pk, cudaStream_t s) {
  long long total = pk.rows * pk.cols;
  ScaleRef sr = begin_pack(pk, src, total, s);          // callers pass ld == cols: the matrix is contiguous
  KernelTimer kt("pack_matrix", s, 0, 4.0 * total + 2.0 * elem_of(pk.arith) * total);
  const bool vec = pk.cols % 8 == 0 && ld % 8 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  with_elems(pk, [&](auto* hi, auto* lo) {
    using E = std::remove_pointer_t<decltype(hi)>;
    if (vec) launch_dep(pack_matrix_kernel<true, E>, dim3(grid_for(total / 8, 256, 2)), dim3(256), 0, s, src, ld, hi, lo, pk.pitch, pk.rows, pk.cols, sr);
    else launch_dep(pack_matrix_kernel<false, E>, dim3(grid_for(total, 256, 4)), dim3(256), 0, s, src, ld, hi, lo, pk.pitch, pk.rows, pk.cols, sr);
  });
  TF_AFTER(s, "pack_matrix");
  return 0;
}

// ---- matmul ---------------------------------------------------------------------------------------
int tc_matmul(const float* A, bool tA, const float* B, bool tB, float* C, int64_t M, int64_t N, int64_t K, cudaStream_t s, int* oom) {
  // Two packs, their maxima, the product and the sum of its split tiles cost about 20 us before the first multiply-add counts:
  // below 0.3 GFLOP the CUDA-core kernel is through sooner (figures at its pick of tiles).  Forced (path 2): whatever fits.
  if (M < 16 || N < 16 || K < 64 || (double)M * N * K < (contraction_path() == 2 ? 4e6 : 1.5e8)) return 0;
  if (!encode_fn()) return 0;
  const int ar = tensor_arithmetic(), bk = bk_of(ar);
  // A is stored [M][K] (K-major) or, transposed, [K][M] (M-major); B is stored [K][N] (N-major) or [N][K] (K-major)
  Pack pa, pb;
  StreamLease lease(s);
  long long a_rows = tA ? K : M, a_cols = tA ? M : K, b_rows = tB ? N : K, b_cols = tB ? K : N;
  int rc = pack_in_scratch(pa, lease, kScratchPackA, ar, a_rows, a_cols, s, oom);
  if (!rc) rc = pack_in_scratch(pb, lease, kScratchPackB, ar, b_rows, b_cols, s, oom);
  if (rc) return rc < 0 ? -1 : 0;
  rc = run_pack_matrix(A, a_cols, pa, s);
  if (!rc) rc = run_pack_matrix(B, b_cols, pb, s);
  GemmParams p;
  memset(&p, 0, sizeof(p));
  const int bn = pick_bn(N, tB);
  p.mode = kModeGemm; p.a_mn = tA ? 1 : 0; p.b_mn = tB ? 0 : 1; p.epi = kEpiRowMajor;
  p.data_by_data = tA ? 1 : 0;     // A^T B is how a dense layer's weight gradient (X^T dY) arrives
  if (!rc) rc = p.a_mn ? make_map_mn(&p.a_hi, ar, pa.hi, pa.rows, pa.pitch, BM) : make_map(&p.a_hi, ar, pa.hi, pa.rows, pa.cols, pa.pitch, BM);
  if (!rc) rc = p.a_mn ? make_map_mn(&p.a_lo, ar, pa.lo, pa.rows, pa.pitch, BM) : make_map(&p.a_lo, ar, pa.lo, pa.rows, pa.cols, pa.pitch, BM);
  if (!rc) rc = p.b_mn ? make_map_mn(&p.b_hi, ar, pb.hi, pb.rows, pb.pitch, bn) : make_map(&p.b_hi, ar, pb.hi, pb.rows, pb.cols, pb.pitch, bn);
  if (!rc) rc = p.b_mn ? make_map_mn(&p.b_lo, ar, pb.lo, pb.rows, pb.pitch, bn) : make_map(&p.b_lo, ar, pb.lo, pb.rows, pb.cols, pb.pitch, bn);
  if (!rc) {
    p.M = (int)M; p.N = (int)N;
    p.m_tiles = (int)((M + BM - 1) / BM); p.n_tiles = (int)((N + bn - 1) / bn); p.tap_tiles = 1;
    p.k_total = (int)((K + bk - 1) / bk);
    p.out = C; p.ldc = N; p.err = error_word();
    p.a_scale = pa.scale(); p.b_scale = pb.scale();
    rc = launch_gemm_bn(bn, ar, p, s, 2.0 * M * N * K, "DLGpuMatrixMultiply", oom);
  }
  return rc < 0 ? -1 : (rc > 0 ? 0 : 1);    // a missing workspace sends the call to the CUDA-core kernel
}

// ---- convolution -------------------------------------------------------------------------------------
// Shapes the tensor path takes (everything else returns 0 and runs on the CUDA cores):
//   class A: 1x1 window, no padding, any stride (frame = the P x Q output grid, x sampled with the stride);
//   class B: stride 1, padding <= window - 1 on each axis, any window: frame = (H + R - 1) x (W + S - 1); x sits at
//            offset (pad_h, pad_w), dy at (R - 1 - pad_h, S - 1 - pad_w), which gives each the zero halo its role
//            needs (forward padding for x, "full" correlation for dy);
//   class D: strided windows: space-to-depth phases (see conv_state);
//   class C: too few input channels for a per-tap reduction chunk: x is expanded into patches (C*R*S columns) and
//            the problem runs as class A over C*R*S channels; forward and filter gradient only.
struct ConvTc {
  int cls = 0;                 // 0 unsupported, 1 class A, 2 class B, 3 class C, 4 class D
  int frame_h = 0, frame_w = 0;                          // frame geometry shared by the x and dy packs
  int x_off_h = 0, x_off_w = 0, dy_off_h = 0, dy_off_w = 0;
  int eC = 0, eR = 1, eS = 1;                            // reduction channels and window of the problem as the GEMM sees it
  int cp = 0;                                            // class D: columns per stride phase (C rounded up to 64)
  bool dgrad_seen = false;                               // backward-data has run on this plan: forward also packs its filter layout
  bool track_y = false, track_dx = false;                // a ReLU asked for max|y| / max|dx|: the epilogue leaves it
  bool y_made = false, dx_made = false;                  // ... and so does the first call, before anybody can have asked
  static bool tracks(bool asked, bool* made, int ar) { const bool t = asked || !*made; if (ar == kArithF16) *made = true; return t; }
  Pack x, dy, wf, wd;
  ConvTc* x_owner = this;                                // whose x pack the plan reads: another plan's of the same recorded step, or its own
  std::mutex mu;
  const Pack& x_pack() const { return x_owner->x; }
};
static ConvTc* conv_state(ConvPlan* p) {
  if (!p->tc_state) {
    ConvTc* st = new ConvTc;
    st->eC = p->C; st->eR = p->R; st->eS = p->S;
    bool base = p->dataformat == 0 && p->K >= 16 && p->K % 4 == 0 && p->R * p->S <= kMaxTaps;
    bool ok = base && p->C >= 16 && p->C % 4 == 0;
    if (ok && p->R == 1 && p->S == 1 && p->pad_h == 0 && p->pad_w == 0) {
      st->cls = 1; st->frame_h = p->P; st->frame_w = p->Q;
    } else if (ok && p->stride_h == 1 && p->stride_w == 1 && p->pad_h <= p->R - 1 && p->pad_w <= p->S - 1) {
      st->cls = 2;
      static const bool shared_halo = [] { const char* e = getenv("TINYFLOW_SHARED_HALO"); return e ? atoi(e) != 0 : true; }();
      if (shared_halo) {
        // x and dy both sit at the frame's origin and the frame is only max(pad, window-1-pad) wider / taller than the
        // input: a tap that reaches left of column 0 lands in the zero gap that ends the previous frame row (right of
        // the last column: the gap of its own row), above row 0 in the zero rows that end the previous image (or before
        // the pack: zero fill).  The gap is shared by both sides, so the frame has (H+g)(W+g) positions instead of
        // (H+R-1)(W+S-1): 1.31x the outputs instead of 1.65x at 7x7 with a 3x3 window.
        const int gh = std::max(p->pad_h, p->R - 1 - p->pad_h), gw = std::max(p->pad_w, p->S - 1 - p->pad_w);
        st->frame_h = p->H + gh; st->frame_w = p->W + gw;
      } else {
        st->frame_h = p->H + p->R - 1; st->frame_w = p->W + p->S - 1;
        st->x_off_h = p->pad_h; st->x_off_w = p->pad_w; st->dy_off_h = p->R - 1 - p->pad_h; st->dy_off_w = p->S - 1 - p->pad_w;
      }
    } else if (ok && p->stride_h * p->stride_w <= 16 && p->pad_h <= p->R - 1 && p->pad_w <= p->S - 1 &&
               (long long)p->stride_h * p->stride_w * round_up(p->C, 64) < 32768) {
      // strided window: x is split into stride_h*stride_w phases (space to depth), each tap reads one phase at a
      // stride-1 shift; dy sits behind a halo of (R-1)/stride_h, (S-1)/stride_w for the backward-data pass
      st->cls = 4; st->cp = (int)round_up(p->C, 64);
      st->dy_off_h = (p->R - 1) / p->stride_h; st->dy_off_w = (p->S - 1) / p->stride_w;
      int uh = (p->H - 1 + p->pad_h) / p->stride_h + 1, uw = (p->W - 1 + p->pad_w) / p->stride_w + 1;
      st->frame_h = (uh > p->P ? uh : p->P) + st->dy_off_h; st->frame_w = (uw > p->Q ? uw : p->Q) + st->dy_off_w;
    } else if (base && p->C < 16 && p->C * p->R * p->S <= 1024) {
      st->cls = 3; st->frame_h = p->P; st->frame_w = p->Q;
      st->eC = p->C * p->R * p->S; st->eR = st->eS = 1;
    }
    // small problems are launch-bound: leave them to the CUDA-core kernel
    double flops = 2.0 * p->N * p->K * p->P * p->Q * p->C * p->R * p->S;
    if (flops < 2e7) st->cls = 0;
    p->tc_state = st;
  }
  return (ConvTc*)p->tc_state;
}

// The state itself stays: notes of producers may name it.  So do packs that a recording writes.  A product of this thread that waits reads
// its packs first (if its launch fails it is forgotten, and the error is the thread's last one).
void tc_release(void* tc_state) {
  ConvTc* st = (ConvTc*)tc_state;
  if (!st) return;
  std::lock_guard<std::mutex> lk(st->mu);
  for (Pack* pk : {&st->x, &st->dy, &st->wf, &st->wd}) {
    if (recordings_use(&pk->src)) continue;
    if (pk->hi && held_reads(pk->hi)) launch_held_filters(t_waiting_stream);
    pack_release(*pk);
    pk->src = nullptr;
  }
}

// One launch of the frame pack: `chans` channels of an NCHW tensor (spatial dims H x W) into columns dst_c0 .. dst_c0 + cover
// of pk (zeros past `chans`)
static int launch_pack_nchw(Pack& pk, const ScaleRef& sr, const float* src, int N, int chans, int H, int W, int frame_h, int frame_w, int off_h, int off_w,
                            int sh, int sw, int dst_c0, int cover, cudaStream_t s, float* relu_out = nullptr, AmaxOut relu_am = AmaxOut{}, const float* mask = nullptr) {
  PackGeom g{N, chans, H, W, frame_h, frame_w, off_h, off_w, sh, sw, (int)pk.pitch, dst_c0, cover};
  // The widest channel block, as long as that makes four blocks an SM (16 of tf32, whose blocks move twice the bytes): a small frame in
  // wide blocks is one wave of long chains.  Inception-v4 b16 3xTF32 19.41 -> 18.83 ms a step (four: 19.11), VGG-16 b7 1323 -> 1301 us; with
  // 16 blocks of fp16 DenseNet-121 b32 12.50 -> 12.65 ms.
  int tc = cover > 64 ? 128 : cover > 32 ? 64 : 32;
  const int enough = (pk.arith == kArithTF32 ? 16 : 4) * device_sm_count();
  while (tc > 32 && (long long)N * ((cover + tc - 1) / tc) * ((frame_h * frame_w + 31) / 32) < enough) tc /= 2;
  dim3 grid(N * ((cover + tc - 1) / tc), (frame_h * frame_w + 31) / 32);
  TF_REQUIRE(grid.y <= 65535, "pack: frame of %d x %d positions is too large", frame_h, frame_w);
  const char* what = mask ? "relu_bwd_pack" : relu_out ? "relu_pack" : "pack_nchw";
  KernelTimer kt(what, s, 0, (mask ? 12.0 : relu_out ? 8.0 : 4.0) * N * chans * H * W / (sh * sw) + 2.0 * elem_of(pk.arith) * pk.rows * cover);
  with_elems(pk, [&](auto* hi, auto* lo) {
    using E = std::remove_pointer_t<decltype(hi)>;
    auto launch = [&](auto mode) {
      constexpr int MODE = decltype(mode)::value;
      if (tc == 128) launch_dep(pack_nchw_kernel<128, E, MODE>, grid, dim3(256), 0, s, src, hi, lo, g, sr, mask, relu_out, relu_am);
      else if (tc == 64) launch_dep(pack_nchw_kernel<64, E, MODE>, grid, dim3(256), 0, s, src, hi, lo, g, sr, mask, relu_out, relu_am);
      else launch_dep(pack_nchw_kernel<32, E, MODE>, grid, dim3(256), 0, s, src, hi, lo, g, sr, mask, relu_out, relu_am);
    };
    if (mask) launch(std::integral_constant<int, kPackReluBwd>());
    else if (relu_out) launch(std::integral_constant<int, kPackRelu>());
    else launch(std::integral_constant<int, kPackPlain>());
  });
  TF_AFTER(s, what);
  return 0;
}
// A pack counts only where it was made: a recorded step reads none that was there before (the caller may rewrite its source
// between replays, and nothing of the step would pack it again), an ordinary call none that a recording has only announced.
static bool pack_valid(const Pack& pk, int ar, const void* src, uint64_t ver, int tag, long long rows, long long cols) {
  return pk.hi && pk.arith == ar && pk.src == src && pk.version == ver && pk.tag == tag && pk.rows == rows && pk.cols == cols &&
         pk.recording == recording_id();
}
// ---- producers that write a consumer's pack ---------------------------------------------------------------------------
// The graph calls BN -> ReLU -> convolution as separate entry points, and the convolution then re-reads the ReLU's output
// to pack it.  Every ReLU call that comes with a descriptor (one per graph node, stable from step to step) leaves a note
// "this address was written by that node"; when a frame pack of x is made, the node that wrote x is looked up and the
// plan is remembered under the node.  From the next step on that node's ReLU packs its output for the plan in the same
// pass (relu_pack), whatever address the executor hands it, and the convolution finds the pack valid.  A wrong guess
// costs one unused pack.
//
// The fused kernel takes the pack's scale from max|x|, the bound of max|y| that is known when it starts.  A step's bits may not depend on
// what earlier steps taught the plans, so the same scale goes into every pack of y that a ReLU could have written: the plain ReLU, too,
// leaves the bound of its input behind (tc_relu_bound, under a key beside y's address), and pack_x takes it.  For the same reason the first call of a
// convolution tracks its output's maximum whether somebody asked or not.  (While first steps scaled by max|y|, 5 of 150 of them, of graphs of
// any size, differed from the second in the last bits of their smallest operands: up to 4e-8 of Adam's moments after one step.)
struct PackTarget { ConvTc* st; int N, C, H, W; };
static std::atomic<long long> g_fused_relu_packs{0};
static std::mutex g_targets_mu;
struct ReluNote { const void* node; uint64_t version; const void* x; uint64_t x_version; bool bound; };
static std::unordered_map<const void*, ReluNote> g_relu_writer;             // output address -> the ReLU node that wrote it, and the write version it left
static std::unordered_map<const void*, PackTarget> g_pack_targets;          // ReLU descriptor -> plan that packs its output
static bool fuse_relu_packs() {
  static const bool on = [] { const char* e = getenv("TINYFLOW_FUSE_RELU_PACK"); return e ? atoi(e) != 0 : true; }();
  return on;
}
static const void* bound_key(const void* y) { return (const char*)y + 1; }
// Before y = relu(x) runs on its own, after the version bump: the word that bounds max|x|, if there is one, and the word that the kernel copies it to.
ReluBound tc_relu_bound(const float* x, const float* y) {
  if (!fuse_relu_packs() || x == y || tensor_arithmetic() != kArithF16) return ReluBound{};
  const uint32_t* from = amax_tracked(x);
  return from ? ReluBound{from, amax_track_begin(bound_key(y)).word} : ReluBound{};
}
void tc_note_relu_output(const void* node, const void* y, const void* x, bool bound) {     // call after the output's write version was bumped
  if (!node) return;
  const uint64_t ver = version_of(y), x_ver = version_of(x);
  std::lock_guard<std::mutex> lk(g_targets_mu);
  g_relu_writer[y] = ReluNote{node, ver, x, x_ver, bound};
}
// A convolution's output is what a ReLU reads, forward and backward; its maximum, folded into the epilogue, is the bound that
// lets the ReLU write the next pack too.  Only outputs that a ReLU has asked about are tracked (behind a batch
// norm nobody needs it, and ResNet-50 lost 0.5 % with all of them tracked).
struct ConvNote { bool* wanted; uint64_t version; };
static std::unordered_map<const void*, ConvNote> g_conv_writer;
static void note_conv_output(const float* out, bool* wanted) {      // call after the output's write version was bumped
  const uint64_t ver = version_of(out);
  std::lock_guard<std::mutex> lk(g_targets_mu);
  g_conv_writer[out] = ConvNote{wanted, ver};
}
static void ask_for_maximum_locked(const void* x, uint64_t ver) {
  auto it = g_conv_writer.find(x);
  if (it != g_conv_writer.end() && it->second.version == ver) *it->second.wanted = true;
}
static const uint32_t* bound_of(const float* x) {
  const uint64_t ver = version_of(x);
  {
    std::lock_guard<std::mutex> lk(g_targets_mu);
    ask_for_maximum_locked(x, ver);
  }
  return amax_tracked(x);
}
// The bound that the ReLU which wrote x scales the pack with when it writes it itself; null: no ReLU did, or it does not write packs
static const uint32_t* relu_bound_of(const float* x, uint64_t ver) {
  {
    std::lock_guard<std::mutex> lk(g_targets_mu);
    auto it = g_relu_writer.find(x);
    if (it == g_relu_writer.end() || it->second.version != ver || !it->second.bound) return nullptr;
  }
  return amax_tracked((const float*)bound_key(x));
}
static void remember_pack_target(const void* x, uint64_t ver, ConvTc* st, const ConvPlan* p) {
  std::lock_guard<std::mutex> lk(g_targets_mu);
  auto it = g_relu_writer.find(x);
  if (it == g_relu_writer.end() || it->second.version != ver) return;
  g_pack_targets[it->second.node] = PackTarget{st, p->N, p->C, p->H, p->W};
  ask_for_maximum_locked(it->second.x, it->second.x_version);
}

// Inside a recorded step the branches of a module read one pack of their common input: convolutions whose frames agree (1x1 windows
// of any filter count, equal windows) find the pack an earlier one has made.  Only inside one recording: its launches
// run in one order on one stream, so a pack that was valid when it was recorded is valid at every replay, and plans of a step are
// not used by two threads at once.  (A pack written by a ReLU is not offered: its scale comes from a bound, and a replayed step
// keeps the bits of the ordinary one.)
struct SharedPack { const float* x; ConvTc* st; int N, C, H, W, sh, sw; };
static thread_local std::vector<SharedPack> t_shared_packs;
void tc_recording_begins() { t_shared_packs.clear(); }
static void offer_pack(const float* x, ConvTc* st, int N, int C, int H, int W, int sh, int sw) {
  if (t_recording) t_shared_packs.push_back(SharedPack{x, st, N, C, H, W, sh, sw});
}
static ConvTc* find_shared_pack(const ConvTc* st, int ar, const ConvPlan* p, const float* x, uint64_t ver, long long rows, long long cols) {
  if (!t_recording) return nullptr;
  for (const SharedPack& e : t_shared_packs) {
    ConvTc* o = e.st;
    if (e.x != x || o == st || e.N != p->N || e.C != p->C || e.H != p->H || e.W != p->W || e.sh != p->stride_h || e.sw != p->stride_w) continue;
    if (o->cls != st->cls || o->frame_h != st->frame_h || o->frame_w != st->frame_w || o->x_off_h != st->x_off_h || o->x_off_w != st->x_off_w || !o->mu.try_lock()) continue;
    const bool ok = pack_valid(o->x, ar, x, ver, o->cls, rows, cols);
    o->mu.unlock();
    if (ok) return o;
  }
  return nullptr;
}

// the x operand of a plan: frame pack (classes A, B), patch matrix (class C) or one frame per stride phase (class D)
static int pack_x(ConvTc* st, int ar, const ConvPlan* p, const float* x, cudaStream_t s, int* oom) {
  Pack& pk = st->x;
  st->x_owner = st;
  const uint64_t ver = version_of(x);
  const long long n_src = (long long)p->N * p->C * p->H * p->W;
  if (st->cls == 3) {
    long long rows = (long long)p->N * p->P * p->Q;
    if (pack_valid(pk, ar, x, ver, 3, rows, st->eC)) return 0;
    if (release_held(pk.hi, s)) return -1;
    if (pack_alloc(pk, ar, rows, st->eC, s, oom)) return 1;
    ScaleRef sr = begin_pack(pk, x, n_src, s);
    PatchGeom g{p->C, p->H, p->W, p->R, p->S, p->P, p->Q, p->stride_h, p->stride_w, p->pad_h, p->pad_w, st->eC, (int)pk.pitch, p->Q, (st->eC + 7) / 8};
    auto floats = [&] { return p->C * p->R * ((g.span - 1) * p->stride_w + p->S); };
    while (floats() > kPatchFloats && g.span > 1) g.span = (g.span + 1) / 2;          // a span of one has a patch's 1024 floats at most
    KernelTimer kt("pack_patches", s, 0, 2.0 * elem_of(ar) * rows * 8 * g.groups);
    TF_REQUIRE((long long)p->N * p->P < 1ll << 31 && (p->Q + g.span - 1) / g.span <= 65535, "pack: %d x %d x %d outputs are too many", p->N, p->P, p->Q);
    with_elems(pk, [&](auto* hi, auto* lo) {
      using E = std::remove_pointer_t<decltype(hi)>;
      launch_dep(pack_patches_kernel<E>, dim3(p->N * p->P, (p->Q + g.span - 1) / g.span), dim3(256), floats() * sizeof(float), s, x, hi, lo, g, sr);
    });
    TF_AFTER(s, "pack_patches");
    pk.made_from(x, ver, 3);
    return 0;
  }
  const long long rows = (long long)p->N * st->frame_h * st->frame_w;
  const int phases = st->cls == 4 ? p->stride_h * p->stride_w : 1;
  const long long cols = st->cls == 4 ? (long long)phases * st->cp : p->C;
  if (pack_valid(pk, ar, x, ver, st->cls, rows, cols)) return 0;
  if (st->cls == 1 || st->cls == 2)
    if (ConvTc* o = find_shared_pack(st, ar, p, x, ver, rows, cols)) { st->x_owner = o; return 0; }
  if (release_held(pk.hi, s)) return -1;
  if (pack_alloc(pk, ar, rows, cols, s, oom)) return 1;
  const bool relu_writes = (st->cls == 1 || st->cls == 2) && p->stride_h == 1 && p->stride_w == 1;      // the packs that a ReLU can write
  ScaleRef sr = begin_pack(pk, x, n_src, s, relu_writes && ar == kArithF16 ? relu_bound_of(x, ver) : nullptr);
  int rc = 0;
  if (st->cls == 4) {
    // phase (a, b) holds x_padded(sh*u + a, sw*v + b) = x(sh*u + a - pad_h, sw*v + b - pad_w) at frame position (u, v)
    for (int a = 0; a < p->stride_h && !rc; ++a)
      for (int b = 0; b < p->stride_w && !rc; ++b) {
        int ph = a * p->stride_w + b;
        rc = launch_pack_nchw(pk, sr, x, p->N, p->C, p->H, p->W, st->frame_h, st->frame_w, p->pad_h - a, p->pad_w - b, p->stride_h, p->stride_w, ph * st->cp, st->cp, s);
      }
  } else {
    rc = launch_pack_nchw(pk, sr, x, p->N, p->C, p->H, p->W, st->frame_h, st->frame_w, st->x_off_h, st->x_off_w, p->stride_h, p->stride_w, 0, (int)pk.pitch, s);
  }
  if (rc) return -1;
  pk.made_from(x, ver, st->cls);
  if (st->cls == 1 || st->cls == 2) offer_pack(x, st, p->N, p->C, p->H, p->W, p->stride_h, p->stride_w);
  if (relu_writes) remember_pack_target(x, ver, st, p);
  return 0;
}
static int pack_dy(ConvTc* st, int ar, const ConvPlan* p, const float* dy, cudaStream_t s, int* oom) {
  Pack& pk = st->dy;
  const uint64_t ver = version_of(dy);
  const long long rows = (long long)p->N * st->frame_h * st->frame_w;
  if (pack_valid(pk, ar, dy, ver, 2, rows, p->K)) return 0;
  if (release_held(pk.hi, s)) return -1;
  if (pack_alloc(pk, ar, rows, p->K, s, oom)) return 1;
  ScaleRef sr = begin_pack(pk, dy, (long long)p->N * p->K * p->P * p->Q, s);
  if (launch_pack_nchw(pk, sr, dy, p->N, p->K, p->P, p->Q, st->frame_h, st->frame_w, st->dy_off_h, st->dy_off_w, 1, 1, 0, (int)pk.pitch, s)) return -1;
  pk.made_from(dy, ver, 2);
  return 0;
}
// Filter packs are keyed like the activation packs (pointer, write version): an optimiser step bumps the version.
// filter_job() prepares the pack of one filter (layouts: 1 forward, 2 backward-data) and stamps it as made; 0 on success.
static int filter_job(ConvTc* st, int ar, const float* w, const ConvPlan* p, int layouts, cudaStream_t s, int* oom, FilterJob* job) {
  const int taps = st->eR * st->eS;
  memset(job, 0, sizeof(*job));
  job->w = w; job->K = p->K; job->C = st->eC; job->taps = taps;
  const uint64_t ver = version_of(w);
  Pack* first = nullptr;
  for (int d = 0; d < 2; ++d) {
    if (!(layouts >> d & 1)) continue;
    Pack& pk = d ? st->wd : st->wf;
    const int rows = d ? st->eC : p->K, pad = (int)round_up(d ? p->K : st->eC, 64);
    if (pack_alloc(pk, ar, rows, (long long)taps * pad, s, oom)) return 1;
    (d ? job->hi_d : job->hi_f) = pk.hi; (d ? job->lo_d : job->lo_f) = pk.lo; (d ? job->pad_d : job->pad_f) = pad;
    (d ? job->scale_d : job->scale_f) = reinterpret_cast<float*>(pk.words + 2);
    if (!first) first = &pk;
    pk.made_from(w, ver, 10 + d);
  }
  const ScaleRef sr = begin_pack(*first, w, (long long)p->K * p->C * p->R * p->S, s);
  job->amax = sr.amax_cur; job->amax_next = sr.amax_next;
  return 0;
}
template <int MAX> static int launch_filter_jobs(FilterJobs<MAX>& jobs, int ar, cudaStream_t s) {
  double elems = 0;
  for (int i = 0; i < jobs.n; ++i) {
    FilterJob& j = jobs.job[i];
    j.k_blocks = (std::max(j.K, j.pad_d) + kFilterTile - 1) / kFilterTile;
    elems += (double)j.K * j.C * j.taps;
  }
  // As many taps (1x1: blocks of channels) a block as still give two blocks an SM.
  int blocks = 0;
  for (int step : {kFilterTaps, 3, 1}) {
    jobs.tap_step = step;
    blocks = 0;
    for (int i = 0; i < jobs.n; ++i) {
      FilterJob& j = jobs.job[i];
      const int channels = kFilterTile * (j.taps == 1 ? step : 1);
      j.c_blocks = (std::max(j.C, j.pad_f) + channels - 1) / channels;
      j.first_block = blocks;
      blocks += j.k_blocks * j.c_blocks * ((j.taps + step - 1) / step);
    }
    if (blocks >= 2 * device_sm_count()) break;
  }
  KernelTimer kt("pack_filters", s, 0, elems * (4.0 + 4.0 * elem_of(ar)));
  TF_CUDA(ar == kArithTF32 ? launch_dep(pack_filters_kernel<float, MAX>, dim3(blocks), dim3(256), 0, s, jobs) : launch_dep(pack_filters_kernel<__half, MAX>, dim3(blocks), dim3(256), 0, s, jobs));
  TF_AFTER(s, "pack_filters");
  return 0;
}
static bool filter_packed(const ConvTc* st, int ar, const float* w, const ConvPlan* p, int flip) {
  const int rows = flip ? st->eC : p->K, pad = (int)round_up(flip ? p->K : st->eC, 64);
  return pack_valid(flip ? st->wd : st->wf, ar, w, version_of(w), 10 + flip, rows, (long long)st->eR * st->eS * pad);
}
// `with_other` makes the forward call produce the backward-data pack in the same launch.
static int pack_filter(ConvTc* st, int ar, const float* w, const ConvPlan* p, int flip, bool with_other, cudaStream_t s, int* oom) {
  if (filter_packed(st, ar, w, p, flip)) return 0;
  FilterJobs<1> one;
  one.n = 1;
  if (int rc = filter_job(st, ar, w, p, flip ? 2 : with_other ? 3 : 1, s, oom, &one.job[0])) return rc;
  return launch_filter_jobs(one, ar, s);
}
// The filters that a step's convolutions read, each for its plan: those that are not packed already, in one launch ahead of the
// convolutions that find them packed.  What it leaves out the convolution packs when it comes up.
int tc_pack_filters(ConvPlan* const* plans, const float* const* filters, const int64_t* sizes, int n, cudaStream_t s) {
  if (contraction_path_is_cuda_cores() || !encode_fn()) return 0;
  const int ar = tensor_arithmetic();
  FilterJobs<kFilterJobs> jobs;
  jobs.n = 0;
  for (int i = 0; i < n; ++i) {
    const ConvPlan* p = plans[i];
    ConvTc* st = (ConvTc*)p->tc_state;
    if (!st || !st->cls || sizes[i] != (int64_t)p->K * p->C * p->R * p->S) continue;
    std::lock_guard<std::mutex> lk(st->mu);
    if (!st->wf.hi || st->wf.arith != ar || (ar == kArithF16 && !amax_tracked(filters[i]))) continue;
    if (filter_packed(st, ar, filters[i], p, 0) && (!st->dgrad_seen || filter_packed(st, ar, filters[i], p, 1))) continue;
    int oom = 0;
    if (filter_job(st, ar, filters[i], p, st->dgrad_seen ? 3 : 1, s, &oom, &jobs.job[jobs.n])) continue;
    if (++jobs.n < kFilterJobs) continue;
    if (launch_filter_jobs(jobs, ar, s)) return -1;
    jobs.n = 0;
  }
  return jobs.n ? launch_filter_jobs(jobs, ar, s) : 0;
}

// forward and backward-data share one launcher: out[pixel][ch_out] = sum_{tap, ch_in} act[pixel + off(tap)][col(tap) + ch_in] * filt[ch_out][b(tap)][ch_in]
struct TapList { int n = 0; int off[kMaxTaps]; int col[kMaxTaps]; int b[kMaxTaps]; void add(int o, int c, int bb) { off[n] = o; col[n] = c; b[n] = bb; ++n; } };
struct OutGeom { int valid_h, valid_w, out_h, out_w, out_sh, out_sw, out_off_h, out_off_w; };
// returns 0 on success, -1 on error, 1 when scratch memory was short (*oom set)
// Orders the taps into runs that share one block of activation rows: same columns, shifts at most `span` apart.  The
// span (up to 64 rows, a block of 192) is the one that fetches the fewest bytes per stage: runs of whole windows on narrow
// images, of window rows on wide ones.
static void plan_runs(GemmParams& g, const TapList& taps, int bn) {
  int order[kMaxTaps];
  for (int t = 0; t < taps.n; ++t) order[t] = t;
  std::sort(order, order + taps.n, [&](int a, int b) { return taps.col[a] != taps.col[b] ? taps.col[a] < taps.col[b] : taps.off[a] < taps.off[b]; });
  auto group = [&](int span, GemmParams* out) -> double {            // bytes of A and B per stage
    int runs = 0, widest = 0, t0 = 0;
    for (int i = 0; i < taps.n; ++i) {
      const int t = order[i], f = order[t0];
      const bool fresh = i == 0 || taps.col[t] != taps.col[f] || taps.off[t] - taps.off[f] > span;
      if (fresh) { t0 = i; ++runs; }
      const int shift = taps.off[t] - taps.off[order[t0]];
      widest = std::max(widest, shift);
      if (out) {
        if (fresh && i) out->tap_word[i - 1] |= 0x200u;
        out->tap_word[i] = (uint32_t)shift | (fresh ? 0x100u : 0u) | (i == taps.n - 1 ? 0x200u : 0u);
        out->tap_off[i] = taps.off[order[t0]]; out->pair_shift[i] = (short)shift;
        out->tap_col[i] = (short)taps.col[t];
        out->tap_b[i] = (short)taps.b[t];
      }
    }
    const int rows = BM + (widest + 7) / 8 * 8;
    if (out) out->a_rows = rows;
    return (double)runs * rows * 256 / taps.n + bn * 256;
  };
  int best = 0;
  double least = group(0, nullptr);
  for (int span = 1; span <= 64; ++span) {
    const double bytes = group(span, nullptr);
    if (bytes < least) { least = bytes; best = span; }
  }
  group(best, &g);
}
constexpr int kNarrowTiles = 64, kNarrowStages = 32;
static int conv_like(const Pack& act, const Pack& filt, int ch_in, int ch_out, int frame_h, int frame_w, float* out, const TapList& taps,
                     const OutGeom& og, double flops, cudaStream_t s, const char* what, int* oom, AmaxOut* track) {
  GemmParams g;
  memset(&g, 0, sizeof(g));
  const int ar = act.arith, bk = bk_of(ar);
  int bn = pick_bn(ch_out, true);
  // Few tiles of a short reduction: 64 columns, so that nearly twice the CTAs each do a stage of two thirds the time.  Up to 64 tiles
  // and 32 stages: Inception-v3 b2 3616 -> 3490 us a step, DenseNet-121 b32 12.60 -> 12.50 ms (longer reductions fill the SMs by being
  // cut, and a wide tile costs less a stage: all of up to 148 tiles, VGG-16 b7 1331 -> 1356 us).  Where fewer pieces are left, more stages
  // gather in an accumulator; a promotion after every second one keeps the error where it was: rms against float64 over twelve layers, in
  // 2^-24 of the result's, forward / input gradient, 4.28 / 4.37 with wide tiles and 3.27 / 3.40 so.  3xTF32 promotes after every
  // second stage anyway, 3.10 / 3.36 with wide tiles and 3.06 / 3.31 so.
  if (bn > 64) {
    const long long mt = (act.rows + BM - 1) / BM;
    if (mt * ((ch_out + bn - 1) / bn) <= kNarrowTiles && mt * ((ch_out + 63) / 64) <= device_sm_count() && taps.n * ((ch_in + bk - 1) / bk) <= kNarrowStages) {
      bn = 64; g.group_limit = 2;
    }
  }
  g.mode = kModeConv; g.epi = kEpiNchw;
  g.M = (int)act.rows; g.N = ch_out;
  g.m_tiles = (int)((act.rows + BM - 1) / BM); g.n_tiles = (ch_out + bn - 1) / bn; g.tap_tiles = 1;
  g.ntaps = taps.n;
  g.chunks_per_tap = (ch_in + bk - 1) / bk;
  g.b_tap_pitch = (int)round_up(ch_in, 64);
  g.k_total = g.ntaps * g.chunks_per_tap;
  plan_runs(g, taps, bn);
  const bool pairs = pairs_wanted(bn, g.m_tiles, g.n_tiles, g.k_total);
  if (pairs) g.a_rows = BM;
  int rc = make_map(&g.a_hi, ar, act.hi, act.rows, act.cols, act.pitch, g.a_rows);
  if (!rc) rc = make_map(&g.a_lo, ar, act.lo, act.rows, act.cols, act.pitch, g.a_rows);
  if (!rc) rc = make_map(&g.b_hi, ar, filt.hi, filt.rows, filt.cols, filt.pitch, pairs ? bn / 2 : bn);      // a pair's CTAs load half a B tile each
  if (!rc) rc = make_map(&g.b_lo, ar, filt.lo, filt.rows, filt.cols, filt.pitch, pairs ? bn / 2 : bn);
  if (rc) return -1;
  g.out = out; g.err = error_word();
  g.a_scale = act.scale(); g.b_scale = filt.scale();
  g.frame_h = frame_h; g.frame_w = frame_w; g.valid_h = og.valid_h; g.valid_w = og.valid_w;
  g.out_c = ch_out; g.out_h = og.out_h; g.out_w = og.out_w; g.out_sh = og.out_sh; g.out_sw = og.out_sw; g.out_off_h = og.out_off_h; g.out_off_w = og.out_off_w;
  if (track && ar == kArithF16 && g_pairs_mode == 0) {        // launches that write one output share the word
    if (!track->word) *track = amax_track_begin(out);
    g.amax = track->word; g.amax_clear = track->clear;
  }
  if (pairs) return ar == kArithTF32 ? launch_gemm_pair<kArithTF32>(g, s, flops, what) : launch_gemm_pair<kArithF16>(g, s, flops, what);
  return launch_gemm_bn(bn, ar, g, s, flops, what, oom);
}
static double conv_flops(const ConvPlan* p) { return 2.0 * p->N * p->K * p->P * p->Q * p->C * p->R * p->S; }
// result of a tensor-path entry point from the launcher's code
static inline int tc_result(int rc) { return rc < 0 ? -1 : (rc > 0 ? 1 : 1); }

// ReLU forward (graph node `node`: the address of its descriptor) whose output the tensor path is expected to pack next:
// y = relu(x) and the consumer plan's frame pack of y in one pass.  Returns 1 when it did that, 0 when the caller should run the plain ReLU (no known consumer, or in the
// fp16 arithmetic no recorded max|x| to bound the scale with), -1 on error.
int tc_fused_relu_pack(const void* node, const float* x, float* y, int64_t n, cudaStream_t s) {
  if (!fuse_relu_packs() || !node || contraction_path_is_cuda_cores()) return 0;
  PackTarget t;
  {
    std::lock_guard<std::mutex> lk(g_targets_mu);
    auto it = g_pack_targets.find(node);
    if (it == g_pack_targets.end()) return 0;
    t = it->second;
  }
  if ((int64_t)t.N * t.C * t.H * t.W != n || x == y) return 0;
  const int ar = tensor_arithmetic();
  ConvTc* st = t.st;
  const uint32_t* bound = ar == kArithF16 ? bound_of(x) : nullptr;
  if (ar == kArithF16 && !bound) return 0;
  std::lock_guard<std::mutex> lk(st->mu);
  Pack& pk = st->x;
  int oom = 0;
  const long long rows = (long long)t.N * st->frame_h * st->frame_w;
  if (release_held(pk.hi, s)) return -1;
  if (pack_alloc(pk, ar, rows, t.C, s, &oom)) return 0;
  note_write(y);
  AmaxOut am = amax_track_begin(y);
  uint32_t* const keep = bound ? amax_track_begin(bound_key(y)).word : nullptr;
  ScaleRef sr{bound, nullptr, reinterpret_cast<float*>(pk.words + 2), keep};       // scale from max|x| >= max|relu(x)|; tf32: no scale
  note_compute_stream(s);
  if (launch_pack_nchw(pk, sr, x, t.N, t.C, t.H, t.W, st->frame_h, st->frame_w, st->x_off_h, st->x_off_w, 1, 1, 0, (int)pk.pitch, s, y, am)) return -1;
  pk.made_from(y, version_of(y), st->cls);
  tc_note_relu_output(node, y, x, keep != nullptr);
  g_fused_relu_packs.fetch_add(1, std::memory_order_relaxed);
  return 1;
}
// ReLU backward (held back by its entry point) whose output is the dy of a convolution's backward call: out = mask > 0 ? dy : 0
// and the plan's pack of it in one pass.  1 when it did that, 0 when the caller should run the ReLU on its own.  The scale comes from max|dy|: where
// that lies 2^r above max|out|, because the mask takes the largest values away, the pack keeps out to 2^(r-39) of max|out| and better: half an fp32
// ulp of it, 2^-25, up to r = 14.
int tc_fused_relu_bwd_pack(ConvPlan* p, const float* mask, const float* dy, float* out, cudaStream_t s) {
  ConvTc* st = conv_state(p);
  // (a layer of few channels goes through here as patches, unless the direct kernels take it: they have up to 32 filters at stride 1)
  const bool taken = p->C >= 16 || (st->cls == 3 && (p->K > 32 || p->stride_h > 1 || p->stride_w > 1));
  if (!fuse_relu_packs() || !st->cls || p->K < 16 || !taken || !encode_fn() || out == mask || out == dy) return 0;
  const int ar = tensor_arithmetic();
  const uint32_t* bound = ar == kArithF16 ? bound_of(dy) : nullptr;       // max|dy| >= max|out|
  if (ar == kArithF16 && !bound) return 0;
  std::lock_guard<std::mutex> lk(st->mu);
  Pack& pk = st->dy;
  int oom = 0;
  if (release_held(pk.hi, s)) return -1;
  if (pack_alloc(pk, ar, (long long)p->N * st->frame_h * st->frame_w, p->K, s, &oom)) return 0;
  note_write(out);
  const AmaxOut am = amax_track_begin(out);
  note_compute_stream(s);
  ScaleRef sr{bound, nullptr, reinterpret_cast<float*>(pk.words + 2), nullptr};
  if (launch_pack_nchw(pk, sr, dy, p->N, p->K, p->P, p->Q, st->frame_h, st->frame_w, st->dy_off_h, st->dy_off_w, 1, 1, 0, (int)pk.pitch, s, out, am, mask)) return -1;
  pk.made_from(out, version_of(out), 2);
  return 1;
}
long long fused_relu_pack_count() { return g_fused_relu_packs.load(std::memory_order_relaxed); }

int tc_conv_fwd(ConvPlan* p, const float* x, const float* w, float* y, cudaStream_t s, int* oom) {
  ConvTc* st = conv_state(p);
  if (!st->cls || !encode_fn()) return 0;
  const int ar = tensor_arithmetic();
  std::lock_guard<std::mutex> lk(st->mu);
  if (pack_x(st, ar, p, x, s, oom)) return *oom ? 1 : -1;
  if (pack_filter(st, ar, w, p, 0, st->dgrad_seen, s, oom)) return *oom ? 1 : -1;
  TapList taps;
  for (int r = 0; r < st->eR; ++r)
    for (int q = 0; q < st->eS; ++q) {
      if (st->cls == 4) taps.add((r / p->stride_h) * st->frame_w + q / p->stride_w, ((r % p->stride_h) * p->stride_w + q % p->stride_w) * st->cp, r * st->eS + q);
      else if (st->cls == 2) taps.add((r - p->pad_h + st->x_off_h) * st->frame_w + (q - p->pad_w + st->x_off_w), 0, r * st->eS + q);   // output (p, q) is anchored at frame position (p, q)
      else taps.add(r * st->frame_w + q, 0, r * st->eS + q);
    }
  OutGeom og{p->P, p->Q, p->P, p->Q, 1, 1, 0, 0};
  AmaxOut track;
  note_conv_output(y, &st->track_y);
  const bool tracks = ConvTc::tracks(st->track_y, &st->y_made, ar);
  return tc_result(conv_like(st->x_pack(), st->wf, st->eC, p->K, st->frame_h, st->frame_w, y, taps, og, conv_flops(p), s, "DLGpuConvolution2DForward", oom, tracks ? &track : nullptr));
}

int tc_conv_dgrad(ConvPlan* p, const float* dy, const float* w, float* dx, cudaStream_t s, int* oom) {
  ConvTc* st = conv_state(p);
  if (!st->cls || st->cls == 3 || !encode_fn()) return 0;
  const int ar = tensor_arithmetic();
  std::lock_guard<std::mutex> lk(st->mu);
  if (pack_dy(st, ar, p, dy, s, oom)) return *oom ? 1 : -1;
  st->dgrad_seen = true;                                           // from now on forward packs both layouts in one launch
  if (pack_filter(st, ar, w, p, 1, false, s, oom)) return *oom ? 1 : -1;     // [C][flipped tap][K]; a no-op when forward made it
  const int ntap = p->R * p->S;
  int rc = 0;
  AmaxOut track;
  note_conv_output(dx, &st->track_dx);
  const bool tracks = ConvTc::tracks(st->track_dx, &st->dx_made, ar);
  if (st->cls == 1) {
    // a strided 1x1 window reaches only every stride-th input position: the rest of dx is zero
    bool strided = p->stride_h > 1 || p->stride_w > 1;
    if (strided && clear_on_stream(dx, sizeof(float) * (size_t)p->N * p->C * p->H * p->W, s) != cudaSuccess) return -1;
    TapList taps; taps.add(0, 0, 0);
    OutGeom og{p->P, p->Q, p->H, p->W, p->stride_h, p->stride_w, 0, 0};
    rc = conv_like(st->dy, st->wd, p->K, p->C, st->frame_h, st->frame_w, dx, taps, og, conv_flops(p), s, "DLGpuConvolutionBackwardData", oom, tracks ? &track : nullptr);
  } else if (st->cls == 2) {
    TapList taps;
    // dx(h, w), anchored at frame position (h, w), reads dy(h - lo_h + r, w - lo_w + s) with lo = window - 1 - pad
    for (int r = 0; r < p->R; ++r)
      for (int q = 0; q < p->S; ++q)
        taps.add((r - (p->R - 1 - p->pad_h) + st->dy_off_h) * st->frame_w + (q - (p->S - 1 - p->pad_w) + st->dy_off_w), 0, r * p->S + q);
    OutGeom og{p->H, p->W, p->H, p->W, 1, 1, 0, 0};
    rc = conv_like(st->dy, st->wd, p->K, p->C, st->frame_h, st->frame_w, dx, taps, og, conv_flops(p), s, "DLGpuConvolutionBackwardData", oom, tracks ? &track : nullptr);
  } else {
    // One launch per stride phase (a, b): dx_padded(sh*u + a, sw*v + b) = sum over the taps r = sh*r' + a, s = sw*s' + b of
    // dy(u - r', v - s') * w(r, s); dy sits at frame offset (hh, hw), so the shift is (hh - r') rows and (hw - s') columns.
    // The phases write disjoint positions of dx; positions no phase reaches stay zero.
    if (clear_on_stream(dx, sizeof(float) * (size_t)p->N * p->C * p->H * p->W, s) != cudaSuccess) return -1;
    for (int a = 0; a < p->stride_h && !rc; ++a)
      for (int b = 0; b < p->stride_w && !rc; ++b) {
        TapList taps;
        for (int r = a; r < p->R; r += p->stride_h)
          for (int q = b; q < p->S; q += p->stride_w)
            taps.add((st->dy_off_h - r / p->stride_h) * st->frame_w + (st->dy_off_w - q / p->stride_w), 0, ntap - 1 - (r * p->S + q));
        if (!taps.n) continue;      // no tap lands on this phase: it stays zero
        OutGeom og{st->frame_h, st->frame_w, p->H, p->W, p->stride_h, p->stride_w, a - p->pad_h, b - p->pad_w};
        rc = conv_like(st->dy, st->wd, p->K, p->C, st->frame_h, st->frame_w, dx, taps, og, conv_flops(p) * taps.n / ntap, s, "DLGpuConvolutionBackwardData", oom, tracks ? &track : nullptr);
      }
  }
  return tc_result(rc);
}

static int launch_wgrad(const ConvTc* st, int bn, int ar, GemmParams& g, cudaStream_t s, double flops, int* oom) {
  g.operand_bytes = 2.0 * st->dy.bytes() + 2.0 * st->x_pack().bytes();
  g.hold = 1; g.pack_a = st->x_pack().hi; g.pack_b = st->dy.hi;
  const int rc = launch_gemm_bn(bn, ar, g, s, flops, "DLGpuConvolutionBackwardFilter", oom);
  // what has gathered goes when it fills the SMs
  if (rc == 0 && t_held_work >= (double)kHeldWork * device_sm_count() && launch_held_filters(t_waiting_stream)) return -1;
  return tc_result(rc);
}
int tc_conv_wgrad(ConvPlan* p, const float* x, const float* dy, float* dw, cudaStream_t s, int* oom) {
  ConvTc* st = conv_state(p);
  if (!st->cls || !encode_fn()) return 0;
  const int ar = tensor_arithmetic(), bk = bk_of(ar);
  std::lock_guard<std::mutex> lk(st->mu);
  if (pack_x(st, ar, p, x, s, oom)) return *oom ? 1 : -1;
  if (pack_dy(st, ar, p, dy, s, oom)) return *oom ? 1 : -1;
  GemmParams g;
  memset(&g, 0, sizeof(g));
  g.err = error_word(); g.out = dw; g.data_by_data = 1;
  const int kit = (int)((st->dy.rows + bk - 1) / bk);       // the reduction runs over the frame's pixel rows
  if (st->eR * st->eS == 1 && st->dy_off_h == 0 && st->dy_off_w == 0) {
    // One tap: dW[k][c] = dy^T x is a plain GEMM over the two packs, and either operand may take the M side.
    // Take the orientation whose padded tile grid is smaller (64 input channels would fill half of a 128-row tile).
    auto padded = [](long long m, long long n) { int b = pick_bn(n); return ((m + BM - 1) / BM * BM) * ((n + b - 1) / b * b); };
    const long long slot_rows = st->eC > 64 ? (st->eC + BM - 1) / BM * BM : BM;
    const int bn_x = pick_bn(p->K);
    const long long as_is = slot_rows * ((p->K + bn_x - 1) / bn_x * bn_x);
    if (padded(p->K, st->eC) < as_is) {
      const int bn = pick_bn(st->eC);
      g.mode = kModeGemm; g.a_mn = 1; g.b_mn = 1; g.epi = kEpiRowMajor;
      int rc = make_map_mn(&g.a_hi, ar, st->dy.hi, st->dy.rows, st->dy.pitch, BM);
      if (!rc) rc = make_map_mn(&g.a_lo, ar, st->dy.lo, st->dy.rows, st->dy.pitch, BM);
      if (!rc) rc = make_map_mn(&g.b_hi, ar, st->x_pack().hi, st->x_pack().rows, st->x_pack().pitch, bn);
      if (!rc) rc = make_map_mn(&g.b_lo, ar, st->x_pack().lo, st->x_pack().rows, st->x_pack().pitch, bn);
      if (rc) return -1;
      g.a_scale = st->dy.scale(); g.b_scale = st->x_pack().scale();
      g.M = p->K; g.N = st->eC; g.ldc = st->eC;
      g.m_tiles = (p->K + BM - 1) / BM; g.n_tiles = (st->eC + bn - 1) / bn; g.tap_tiles = 1; g.ntaps = 1;
      g.k_total = kit;
      return launch_wgrad(st, bn, ar, g, s, conv_flops(p), oom);
    }
  }
  // A = x (M = tap slots x input channels), B = dy (N = output channels); both M/N-major, reduction over pixel rows.
  const int bn = pick_bn(p->K);
  g.mode = kModeWgrad; g.a_mn = 1; g.b_mn = 1; g.epi = kEpiWgrad;
  g.M = st->eC; g.N = p->K; g.ntaps = st->eR * st->eS;
  // Few input channels: two filter taps share one 128-row tile (slots of 64 channels), so that the tensor core's
  // M dimension is full and dy is read once for both.
  // So do an odd number of 64-channel blocks of a filter with several taps: 160 channels in 7 taps are 21 blocks in 11 tiles, where
  // whole tiles per tap are 14.
  const int blocks64 = (st->eC + 63) / 64;
  g.slot = blocks64 % 2 == 0 || (blocks64 > 1 && g.ntaps == 1) ? BM : 64;
  g.taps_per_tile = BM / g.slot;
  g.slots_per_tap = g.slot == BM ? 1 : blocks64;
  int rc = make_map_mn(&g.a_hi, ar, st->x_pack().hi, st->x_pack().rows, st->x_pack().pitch, g.slot);
  if (!rc) rc = make_map_mn(&g.a_lo, ar, st->x_pack().lo, st->x_pack().rows, st->x_pack().pitch, g.slot);
  if (!rc) rc = make_map_mn(&g.b_hi, ar, st->dy.hi, st->dy.rows, st->dy.pitch, bn);
  if (!rc) rc = make_map_mn(&g.b_lo, ar, st->dy.lo, st->dy.rows, st->dy.pitch, bn);
  if (rc) return -1;
  g.a_scale = st->x_pack().scale(); g.b_scale = st->dy.scale();
  g.m_tiles = g.slots_per_tap > 1 ? 1 : (st->eC + g.slot - 1) / g.slot;
  g.tap_tiles = (g.ntaps * g.slots_per_tap + g.taps_per_tile - 1) / g.taps_per_tile;
  g.n_tiles = (p->K + bn - 1) / bn;
  // dy row m' holds output pixel (p, q) at frame position (p + dy_off_h, q + dy_off_w); tap (r, s) needs the padded
  // input at (p + r, q + s), which sits at frame row m' + (r - dy_off_h) * frame_w + (s - dy_off_w)
  for (int r = 0; r < st->eR; ++r)
    for (int q = 0; q < st->eS; ++q) {
      int t = r * st->eS + q;
      if (st->cls == 4) {
        g.tap_off[t] = (r / p->stride_h - st->dy_off_h) * st->frame_w + (q / p->stride_w - st->dy_off_w);
        g.tap_col[t] = (short)(((r % p->stride_h) * p->stride_w + q % p->stride_w) * st->cp);
      } else {
        const int ph = st->cls == 2 ? p->pad_h : st->x_off_h, pw = st->cls == 2 ? p->pad_w : st->x_off_w;    // classes A / C: no padding, offsets 0
        g.tap_off[t] = (r - ph + st->x_off_h - st->dy_off_h) * st->frame_w + (q - pw + st->x_off_w - st->dy_off_w);
      }
    }
  g.k_total = kit;
  return launch_wgrad(st, bn, ar, g, s, conv_flops(p), oom);
}

}  // namespace tf
