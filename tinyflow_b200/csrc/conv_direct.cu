// Convolutions of small images with few channels (LeNet's layers), stride 1, exact fp32.  As a matrix product such a layer
// has 6-16 rows: a 64-wide tile multiplies mostly padding and spends its time turning flat indices into addresses
// (the 16 -> 6 channel input gradient at 14x14, batch 256: 283 us for 0.24 GFLOP).  Here a block keeps one image (zero halo
// included) and all filters in shared memory, so an operand costs one shared-memory read and no index arithmetic:
//   forward / input gradient   a thread owns 4 neighbouring outputs of 2-4 channels: per input channel and filter row two or
//                              three 16-byte reads of the image row and S of the filters feed 8*S to 16*S multiply-adds.  Images of few outputs leave most of an SM
//                              idle, so neighbouring lanes share the input channels of one such item and add up their sums.
//   filter gradient            a thread owns one (output channel, input channel, filter row) and slides along the image row
//                              with S accumulators: two reads feed S multiply-adds.  Bound by shared-memory reads; images are
//                              dealt to the blocks, whose partial sums are added in block order (bit-reproducible).
// Filling shared memory is a chain of load latencies unless everything is in flight at once: asynchronous copies, zeros for the halo.
// LeNet at batch 256, us in the step: forward 12.5 -> 8.3 and 13.7 -> 9.6, input gradient of 16 -> 6 channels 39.1 -> 12.1, filter
// gradients 16.7 -> 10.0 and 12.4 -> 6.1.
#include "common.h"
#include <algorithm>
#include <vector>

namespace tf {

__device__ __forceinline__ void copy_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async16(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_arrived() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// Division of indices below 2^16 by a divisor below 2^16: a runtime division takes 20 instructions, and filling shared memory has two an element
struct FastDiv {
  uint32_t m;
  FastDiv(int d = 1) : m(d > 1 ? (uint32_t)((0x100000000ull + d - 1) / d) : 0u) {}
  __device__ __forceinline__ int operator()(int i) const { return m ? (int)__umulhi((uint32_t)i, m) : i; }
};
// planes of h x w into planes of hp x wp, the first element behind pad_h rows and pad_w columns of zeros, zeros all around
struct HaloImage { int planes, h, w, hp, wp, pad_h, pad_w, plane; FastDiv by_h, by_w; };       // plane: floats from one to the next
__device__ __forceinline__ void clear_halo(float* dst, const HaloImage& g) {
  for (int i = 4 * threadIdx.x; i < g.planes * g.plane; i += 4 * blockDim.x) *reinterpret_cast<float4*>(dst + i) = make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void copy_image(float* dst, const float* src, const HaloImage& g) {
  for (int i = threadIdx.x; i < g.planes * g.h * g.w; i += blockDim.x) {
    const int row = g.by_w(i), x = i - row * g.w, c = g.by_h(row), y = row - c * g.h;
    copy_async4(dst + c * g.plane + (y + g.pad_h) * g.wp + x + g.pad_w, src + i);
  }
}

struct DirectConv {
  const float* in; const float* w; float* out;
  int N, Ci, Co, Ho, Wo, R, S;
  int flip;                   // input gradient: w is [in][out][R][S], read back to front
  HaloImage image;            // the input as a block keeps it, its size rounded up to 4
  int w_at;                   // where the filters begin behind it
  int groups, items;          // 4-output groups per row, work items of one image
  int split;                  // neighbouring lanes (1, 2 or 4) that share an item's input channels
  FastDiv by_inner, by_taps, by_groups, by_rows;
};
constexpr int kDirectThreads = 512;
// filters of a thread's channels lie side by side, 4 floats of which 3 are used for CH = 3
template <int CH> constexpr int kChPitch = CH == 3 ? 4 : CH;

template <int S, int CH>
__global__ void __launch_bounds__(kDirectThreads) direct_conv_kernel(const DirectConv p, AmaxOut am) {
  extern __shared__ __align__(16) float direct_smem[];
  float* xs = direct_smem;                                     // [Ci][hp][wp]
  float* ws = direct_smem + p.w_at;                            // [set of channels][Ci][R][S][kPitch]
  const int plane = p.image.plane, wpitch = p.image.wp;
  clear_halo(xs, p.image);
  __syncthreads();
  grid_dep_sync();
  constexpr int kPitch = kChPitch<CH>;
  const int n = blockIdx.x, sets = (p.Co + CH - 1) / CH, rs = p.R * S;
  copy_image(xs, p.in + (long long)n * p.Ci * p.image.h * p.image.w, p.image);
  // the filters in the order they lie in
  const int inner = (p.flip ? p.Co : p.Ci) * rs, total = p.Co * p.Ci * rs;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int outer = p.by_inner(i), rem = i - outer * inner, ch = p.by_taps(rem), t = rem - ch * rs;
    const int o = p.flip ? ch : outer, ci = p.flip ? outer : ch;
    copy_async4(ws + ((o / CH * p.Ci + ci) * rs + (p.flip ? rs - 1 - t : t)) * kPitch + o % CH, p.w + i);
  }
  for (int ch = p.Co - (sets - 1) * CH; ch < CH; ++ch)         // channels that the last set lacks
    for (int i = threadIdx.x; i < p.Ci * rs; i += blockDim.x) ws[((sets - 1) * p.Ci * rs + i) * kPitch + ch] = 0.f;
  copies_arrived();
  __syncthreads();
  uint32_t big = 0;
  const int part = threadIdx.x & (p.split - 1), per_block = blockDim.x / p.split;
  for (int base = blockIdx.y * per_block; base < p.items; base += gridDim.y * per_block) {
    const int mine = base + threadIdx.x / p.split;
    const bool live = mine < p.items;
    const int item = live ? mine : 0, gr = p.by_groups(item), g = item - gr * p.groups, set = p.by_rows(gr), row = gr - set * p.Ho;
    float acc[CH][4];
#pragma unroll
    for (int a = 0; a < CH; ++a)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[a][q] = 0.f;
    for (int ci = part; live && ci < p.Ci; ci += p.split) {
      const float* xr = xs + ci * plane + row * wpitch + 4 * g;
      const float* wp = ws + (set * p.Ci + ci) * rs * kPitch;
      for (int r = 0; r < p.R; ++r, xr += wpitch, wp += S * kPitch) {
        constexpr int kVec = (S + 3 + 3) / 4;
        float x[4 * kVec];
#pragma unroll
        for (int v = 0; v < kVec; ++v) *reinterpret_cast<float4*>(x + 4 * v) = *reinterpret_cast<const float4*>(xr + 4 * v);
#pragma unroll
        for (int s = 0; s < S; ++s) {
          float f[4];
          if (CH == 2) *reinterpret_cast<float2*>(f) = *reinterpret_cast<const float2*>(wp + s * kPitch);
          else *reinterpret_cast<float4*>(f) = *reinterpret_cast<const float4*>(wp + s * kPitch);
#pragma unroll
          for (int a = 0; a < CH; ++a)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[a][q] = fmaf(x[s + q], f[a], acc[a][q]);
        }
      }
    }
    for (int step = 1; step < p.split; step *= 2) {
#pragma unroll
      for (int a = 0; a < CH; ++a)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[a][q] += __shfl_xor_sync(0xffffffffu, acc[a][q], step);
    }
    if (!live || part) continue;
#pragma unroll
    for (int a = 0; a < CH; ++a) {
      const int o = set * CH + a;
      if (o >= p.Co) continue;
      float* dst = p.out + (((long long)n * p.Co + o) * p.Ho + row) * p.Wo + 4 * g;
#pragma unroll
      for (int q = 0; q < 4; ++q) if (4 * g + q < p.Wo) { dst[q] = acc[a][q]; big = max(big, amax_bits(acc[a][q])); }
    }
  }
  amax_commit(am, big);
}

struct DirectWgrad {
  const float* x; const float* dy; float* part;
  int N, C, K, P, Q, R;
  HaloImage image;
  int items, slices, rows_per_slice;
  int dy_at, dy_vec;          // dy behind x in shared memory, 16-byte copies of it
};
constexpr int kWgradThreads = 512, kWgradItems = 4;

// Share `block` of `blocks` of the images of a layer; every block of the launch calls it with the same shared memory
template <int S, int IT>
__device__ __forceinline__ void direct_wgrad(const DirectWgrad& p, int block, int blocks) {
  extern __shared__ __align__(16) float direct_smem[];
  float* xs = direct_smem;                          // [C][hp][wp]
  float* ds = direct_smem + p.dy_at;                // [K][P][Q]
  const int plane = p.image.plane, wp = p.image.wp;
  clear_halo(xs, p.image);
  const int slice = IT == 1 ? threadIdx.x / p.items : 0, first = IT == 1 ? threadIdx.x - slice * p.items : threadIdx.x;
  const bool live = slice < p.slices;
  float acc[IT][S];
#pragma unroll
  for (int i = 0; i < IT; ++i)
#pragma unroll
    for (int s = 0; s < S; ++s) acc[i][s] = 0.f;
  for (int n = block; n < p.N; n += blocks) {
    __syncthreads();
    const float* dsrc = p.dy + (long long)n * p.K * p.P * p.Q;
    copy_image(xs, p.x + (long long)n * p.C * p.image.h * p.image.w, p.image);
    const int count = p.K * p.P * p.Q;
    if (p.dy_vec) {
      for (int i = 4 * threadIdx.x; i < count; i += 4 * kWgradThreads) copy_async16(ds + i, dsrc + i);
    } else {
      for (int i = threadIdx.x; i < count; i += kWgradThreads) copy_async4(ds + i, dsrc + i);
    }
    copies_arrived();
    __syncthreads();
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int item = first + it * kWgradThreads;
      if (!live || item >= p.items) continue;
      const int r = item % p.R, c = (item / p.R) % p.C, k = item / (p.R * p.C);
      const int p0 = slice * p.rows_per_slice, p1 = min(p.P, p0 + p.rows_per_slice);
      for (int pp = p0; pp < p1; ++pp) {
        const float* xr = xs + c * plane + (pp + r) * wp;
        const float* dr = ds + (k * p.P + pp) * p.Q;
        float win[S + 3];
#pragma unroll
        for (int s = 0; s < S - 1; ++s) win[s] = xr[s];
        int q = 0;
        for (; q + 4 <= p.Q; q += 4) {              // four positions a trip: the window moves once for 4*S multiply-adds
          float d[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) { win[S - 1 + j] = xr[q + S - 1 + j]; d[j] = dr[q + j]; }
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int s = 0; s < S; ++s) acc[it][s] = fmaf(win[s + j], d[j], acc[it][s]);
#pragma unroll
          for (int s = 0; s < S - 1; ++s) win[s] = win[s + 4];
        }
        for (; q < p.Q; ++q) {
          win[S - 1] = xr[q + S - 1];
          const float d = dr[q];
#pragma unroll
          for (int s = 0; s < S; ++s) acc[it][s] = fmaf(win[s], d, acc[it][s]);
#pragma unroll
          for (int s = 0; s < S - 1; ++s) win[s] = win[s + 1];
        }
      }
    }
  }
  float* out = p.part + (long long)block * p.items * S;
  if (IT > 1 || p.slices == 1) {
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int item = first + it * kWgradThreads;
      if (!live || item >= p.items) continue;
#pragma unroll
      for (int s = 0; s < S; ++s) out[item * S + s] = acc[it][s];
    }
    return;
  }
  __syncthreads();
  if (live) {
#pragma unroll
    for (int s = 0; s < S; ++s) direct_smem[(slice * p.items + first) * S + s] = acc[0][s];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < p.items * S; i += blockDim.x) {
    float t = 0.f;
    for (int z = 0; z < p.slices; ++z) t += direct_smem[z * p.items * S + i];
    out[i] = t;
  }
}
template <int S, int IT>
__global__ void __launch_bounds__(kWgradThreads) direct_wgrad_kernel(const DirectWgrad p) {
  grid_dep_sync();
  direct_wgrad<S, IT>(p, blockIdx.x, gridDim.x);
}
// out[c] = sum over the blocks' partial filters, in block order within each of 32 warps
__device__ __forceinline__ void direct_wgrad_sum(const float* __restrict__ part, float* __restrict__ out, int rows, int cols, int block) {
  __shared__ float sm[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, c = block * 32 + tx;
  float acc = 0.f;
  if (c < cols) {
#pragma unroll 10
    for (int r = ty; r < rows; r += 32) acc += part[(long long)r * cols + c];
  }
  sm[ty][tx] = acc;
  __syncthreads();
  if (ty == 0 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) t += sm[j][tx];
    out[c] = t;
  }
}

__global__ void __launch_bounds__(1024) direct_wgrad_sum_kernel(const float* __restrict__ part, float* __restrict__ out, int rows, int cols) {
  grid_dep_sync();
  direct_wgrad_sum(part, out, rows, cols, blockIdx.x);
}
// Layers whose gradients may wait (see hold_products in gemm_tcgen05.cu) share both launches: the two of LeNet at batch 256 took 24 us one after
// the other, 20 together.  Blocks and order of the sums are those of the separate launches.
constexpr int kWgradJobs = 8;
struct DirectJob { DirectWgrad d; float* out; int blocks, cols, first, first_sum; };
struct DirectJobs { int n; DirectJob job[kWgradJobs]; };
template <int S>
__global__ void __launch_bounds__(kWgradThreads) direct_wgrad_group_kernel(const __grid_constant__ DirectJobs jobs) {
  grid_dep_sync();
  int k = 0;
  while (k + 1 < jobs.n && jobs.job[k + 1].first <= (int)blockIdx.x) ++k;
  const DirectJob& j = jobs.job[k];
  direct_wgrad<S, 1>(j.d, (int)blockIdx.x - j.first, j.blocks);
}
__global__ void __launch_bounds__(1024) direct_wgrad_group_sum_kernel(const __grid_constant__ DirectJobs jobs) {
  grid_dep_sync();
  int k = 0;
  while (k + 1 < jobs.n && jobs.job[k + 1].first_sum <= (int)blockIdx.x) ++k;
  const DirectJob& j = jobs.job[k];
  direct_wgrad_sum(j.d.part, j.out, j.blocks, j.cols, (int)blockIdx.x - j.first_sum);
}

constexpr size_t kDirectSmem = 96 * 1024;
// The layers taken: stride 1, windows 3, 5 or 7 wide, an image that fits in shared memory together with the filters, and few
// enough channels that the tensor path would multiply padding (it takes 16 channels and more, in multiples of 4; its first
// layers of three channels have large images and many filters and stay there).
static bool direct_shape(const ConvPlan* p) {
  return p->dataformat == 0 && p->stride_h == 1 && p->stride_w == 1 && (p->S == 3 || p->S == 5 || p->S == 7) && p->R <= 7 && p->pad_h <= p->R - 1 && p->pad_w <= p->S - 1 &&
         p->K <= 32 && p->C <= 32 && (p->C < 16 || p->K < 16) && (long long)p->K * p->C * p->R * p->S <= 8192 && p->P == p->H + 2 * p->pad_h - p->R + 1 && p->Q == p->W + 2 * p->pad_w - p->S + 1;
}
template <int CH> static int launch_direct_of(DirectConv d, cudaStream_t s, double flops, const char* what) {
  HaloImage& g = d.image;
  d.groups = (d.Wo + 3) / 4;
  g.planes = d.Ci;
  g.hp = d.Ho + d.R - 1;
  g.wp = (4 * d.groups + d.S + 2) / 4 * 4;           // every 16-byte read of the last group stays inside the row
  g.by_h = FastDiv(g.h); g.by_w = FastDiv(g.w);
  d.items = (d.Co + CH - 1) / CH * d.Ho * d.groups;
  if (d.items >= 1 << 16) return 0;
  // Threads: all items of an image at once where they fit; lanes share items while the device has room for more threads.
  d.split = 1;
  while (d.split < 4 && d.Ci >= 2 * d.split && d.items * 2 * d.split <= kDirectThreads && (long long)d.N * d.items * d.split < 1024ll * device_sm_count()) d.split *= 2;
  // the planes that neighbouring lanes read begin 32 / split banks apart
  g.plane = g.hp * g.wp;
  if (d.split > 1) while (g.plane % 32 != 32 / d.split) g.plane += 4;
  d.w_at = d.Ci * g.plane;                           // a multiple of 4
  const size_t smem = sizeof(float) * ((size_t)d.w_at + (size_t)(d.Co + CH - 1) / CH * kChPitch<CH> * d.Ci * d.R * d.S);
  if (smem > kDirectSmem) return 0;
  d.by_inner = FastDiv((d.flip ? d.Co : d.Ci) * d.R * d.S); d.by_taps = FastDiv(d.R * d.S); d.by_groups = FastDiv(d.groups); d.by_rows = FastDiv(d.Ho);
  const int lanes = d.items * d.split, threads = std::min(kDirectThreads, (lanes + 31) / 32 * 32);
  // one block per image unless that leaves SMs idle
  int gy = (lanes + threads - 1) / threads;
  while (gy > 1 && (long long)d.N * (gy - 1) >= 4 * device_sm_count()) --gy;
  if (gy > 65535) gy = 65535;
  note_compute_stream(s);
  KernelTimer kt("direct_conv", s, flops, 0, 1);
  auto kernel = d.S == 3 ? direct_conv_kernel<3, CH> : d.S == 5 ? direct_conv_kernel<5, CH> : direct_conv_kernel<7, CH>;
  TF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDirectSmem));
  TF_CUDA(launch_dep(kernel, dim3(d.N, gy), dim3(threads), smem, s, d, amax_track_begin(d.out)));
  TF_AFTER(s, what);
  return 1;
}
// Channels of a thread: the more the fewer reads of the image feed a multiply-add (shared memory is the bound), as long as they divide up.
static int launch_direct(const DirectConv& d, cudaStream_t s, double flops, const char* what) {
  if (d.Co % 4 == 0) return launch_direct_of<4>(d, s, flops, what);
  if (d.Co % 3 == 0) return launch_direct_of<3>(d, s, flops, what);
  return launch_direct_of<2>(d, s, flops, what);
}
// Each returns 1 when it took the call, 0 when the shape is not one of its own, -1 on error.
int direct_conv_fwd(const ConvPlan* p, const float* x, const float* w, float* y, cudaStream_t s) {
  if (!direct_shape(p)) return 0;
  DirectConv d{x, w, y, p->N, p->C, p->K, p->P, p->Q, p->R, p->S, 0, HaloImage{0, p->H, p->W, 0, 0, p->pad_h, p->pad_w}};
  return launch_direct(d, s, 2.0 * p->N * p->K * p->P * p->Q * p->C * p->R * p->S, "DLGpuConvolution2DForward");
}
int direct_conv_dgrad(const ConvPlan* p, const float* dy, const float* w, float* dx, cudaStream_t s) {
  if (!direct_shape(p)) return 0;
  DirectConv d{dy, w, dx, p->N, p->K, p->C, p->H, p->W, p->R, p->S, 1, HaloImage{0, p->P, p->Q, 0, 0, p->R - 1 - p->pad_h, p->S - 1 - p->pad_w}};
  return launch_direct(d, s, 2.0 * p->N * p->K * p->P * p->Q * p->C * p->R * p->S, "DLGpuConvolutionBackwardData");
}
template <int S> static int launch_wgrad(const DirectWgrad& d, int grid, size_t smem, cudaStream_t s) {
  const int per = (d.items + kWgradThreads - 1) / kWgradThreads;
  auto kernel = per <= 1 ? direct_wgrad_kernel<S, 1> : per <= 2 ? direct_wgrad_kernel<S, 2> : direct_wgrad_kernel<S, kWgradItems>;
  TF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDirectSmem));
  TF_CUDA(launch_dep(kernel, dim3(grid), dim3(kWgradThreads), smem, s, d));
  return 0;
}
struct HeldDirect { DirectJob job; int S; size_t smem; double flops; };
static thread_local std::vector<HeldDirect> t_held_direct;
void drop_held_direct() { t_held_direct.clear(); }
template <int S> static int launch_direct_group(const DirectJobs& jobs, int blocks, size_t smem, cudaStream_t s) {
  TF_CUDA(cudaFuncSetAttribute(direct_wgrad_group_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDirectSmem));
  TF_CUDA(launch_dep(direct_wgrad_group_kernel<S>, dim3(blocks), dim3(kWgradThreads), smem, s, jobs));
  return 0;
}
int launch_held_direct(cudaStream_t s) {
  std::vector<HeldDirect> all;
  all.swap(t_held_direct);
  for (int S : {3, 5, 7}) {
    size_t at = 0;
    int most = kWgradJobs;
    while (true) {
      DirectJobs jobs;
      jobs.n = 0;
      int blocks = 0, sums = 0;
      size_t smem = 0, floats = 0;
      double flops = 0;
      const size_t begin = at;
      for (; at < all.size() && jobs.n < most; ++at) {
        if (all[at].S != S) continue;
        DirectJob& j = jobs.job[jobs.n++] = all[at].job;
        j.first = blocks; blocks += j.blocks;
        j.first_sum = sums; sums += (j.cols + 31) / 32;
        smem = std::max(smem, all[at].smem); floats += (size_t)j.blocks * j.cols; flops += all[at].flops;
      }
      if (!jobs.n) break;
      StreamLease lease(s);
      float* part = (float*)lease.scratch(kScratchContract, sizeof(float) * floats);
      if (!part && jobs.n > 1) { most = jobs.n / 2; at = begin; continue; }        // a full device: fewer together (the call of each has seen to its own)
      TF_REQUIRE(part, "filter gradients: the device is out of memory, %zu bytes of partial sums short", sizeof(float) * floats);
      for (int i = 0; i < jobs.n; ++i) { jobs.job[i].d.part = part; part += (size_t)jobs.job[i].blocks * jobs.job[i].cols; }
      note_compute_stream(s);
      KernelTimer kt("direct_conv", s, flops, 0, 1);
      if ((S == 3 ? launch_direct_group<3>(jobs, blocks, smem, s) : S == 5 ? launch_direct_group<5>(jobs, blocks, smem, s) : launch_direct_group<7>(jobs, blocks, smem, s)) != 0) return -1;
      TF_AFTER(s, "filter gradients");
      TF_CUDA(launch_dep(direct_wgrad_group_sum_kernel, dim3(sums), dim3(1024), 0, s, jobs));
      TF_AFTER(s, "filter gradients");
    }
  }
  return 0;
}
int direct_conv_wgrad(const ConvPlan* p, const float* x, const float* dy, float* dw, cudaStream_t s) {
  if (!direct_shape(p) || p->K * p->C * p->R > kWgradThreads * kWgradItems) return 0;
  DirectWgrad d{x, dy, nullptr, p->N, p->C, p->K, p->P, p->Q, p->R, HaloImage{p->C, p->H, p->W, p->P + p->R - 1, 0, p->pad_h, p->pad_w, 0, p->H, p->W}, p->K * p->C * p->R, 1, p->P};
  d.image.wp = (p->Q + p->S - 1) | 1;           // odd pitch: the filter rows of a warp fall in different banks
  d.image.plane = d.image.hp * d.image.wp;
  if (d.items <= kWgradThreads) {               // threads to spare: cut the image rows
    d.slices = kWgradThreads / d.items;
    if (d.slices > p->P) d.slices = p->P;
    d.rows_per_slice = (p->P + d.slices - 1) / d.slices;
  }
  d.dy_at = (p->C * d.image.plane + 3) / 4 * 4;
  d.dy_vec = p->K * p->P * p->Q % 4 == 0 && aligned16(dy);
  size_t floats = (size_t)d.dy_at + (size_t)p->K * p->P * p->Q;
  if (d.slices > 1 && floats < (size_t)d.slices * d.items * p->S) floats = (size_t)d.slices * d.items * p->S;
  if (floats * sizeof(float) > kDirectSmem) return 0;
  const int cols = d.items * p->S, grid = p->N < 2 * device_sm_count() ? p->N : 2 * device_sm_count();
  StreamLease lease(s);
  d.part = (float*)lease.scratch(kScratchContract, sizeof(float) * (size_t)grid * cols);
  if (!d.part) return 0;
  const HeldDirect call{DirectJob{d, dw, grid, cols, 0, 0}, p->S, floats * sizeof(float), 2.0 * p->N * p->K * p->P * p->Q * p->C * p->R * p->S};
  if (d.items <= kWgradThreads && may_hold(s) && held(t_held_direct, call)) return 1;
  note_compute_stream(s);
  KernelTimer kt("direct_conv", s, 2.0 * p->N * p->K * p->P * p->Q * p->C * p->R * p->S, 0, 1);
  if ((p->S == 3 ? launch_wgrad<3>(d, grid, floats * sizeof(float), s) : p->S == 5 ? launch_wgrad<5>(d, grid, floats * sizeof(float), s) : launch_wgrad<7>(d, grid, floats * sizeof(float), s)) != 0) return -1;
  TF_AFTER(s, "DLGpuConvolutionBackwardFilter");
  TF_CUDA(launch_dep(direct_wgrad_sum_kernel, dim3((cols + 31) / 32), dim3(1024), 0, s, (const float*)d.part, dw, grid, cols));
  TF_AFTER(s, "DLGpuConvolutionBackwardFilter");
  return 1;
}

}  // namespace tf
