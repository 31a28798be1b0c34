// Exact-fp32 matrix product for the sizes the tensor path is too long a road for: packing two operands, one tcgen05 launch
// and the sum over split tiles are six kernels, about 25 us whatever the size, and a 64 x 784 x 256 layer is 0.4 us of
// CUDA-core work.
//
// What bounds these products is latency (few tiles, long reductions) or, for a handful of rows, reading the weight matrix
// once.  So the reduction is cut over the CTAs of a thread-block cluster: each computes its share of K for the same tile,
// and the tile is added up through distributed shared memory, every CTA one slice of it, in rank order (bit-reproducible,
// no workspace, no second kernel).  The next K block is fetched into registers while the current one is multiplied.
//
// Measured against the kernel it replaced and against the tensor path: the table in simt_matmul(), where the tile is chosen.
#include "common.h"
#include <algorithm>
#include <vector>
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace tf {

struct SimtGemm {
  const float* A; const float* B; float* C;
  int M, N, K;
  long long lda, ldb, ldc;
  int k_per_cta;            // multiple of BK
  int a_vec, b_vec, c_vec;  // 16-byte accesses allowed
};

// One BMxBK (or BKxBN) block of an operand: `rows` index M (or N), `k` the reduction.  KFAST: k is contiguous in memory.
// A thread moves VPT groups of four elements along the contiguous direction.
template <int ROWS, int BK, int THREADS, bool KFAST> struct BlockLoader {
  static constexpr int kGroups = ROWS * BK / 4;
  static constexpr int VPT = (kGroups + THREADS - 1) / THREADS;
  float4 v[VPT];
  __device__ __forceinline__ void fetch(const float* __restrict__ p, long long ld, int row0, int rows, int k0, int k1, bool vec) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int g = threadIdx.x + i * THREADS;
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (kGroups % THREADS && g >= kGroups) continue;
      if (KFAST) {
        const int r = row0 + g / (BK / 4), k = k0 + (g % (BK / 4)) * 4;
        if (r >= rows || k >= k1) continue;
        const float* q = p + (long long)r * ld + k;
        if (vec && k + 4 <= k1) v[i] = __ldg(reinterpret_cast<const float4*>(q));
        else { v[i].x = __ldg(q); if (k + 1 < k1) v[i].y = __ldg(q + 1); if (k + 2 < k1) v[i].z = __ldg(q + 2); if (k + 3 < k1) v[i].w = __ldg(q + 3); }
      } else {
        const int k = k0 + g / (ROWS / 4), r = row0 + (g % (ROWS / 4)) * 4;
        if (r >= rows || k >= k1) continue;
        const float* q = p + (long long)k * ld + r;
        if (vec && r + 4 <= rows) v[i] = __ldg(reinterpret_cast<const float4*>(q));
        else { v[i].x = __ldg(q); if (r + 1 < rows) v[i].y = __ldg(q + 1); if (r + 2 < rows) v[i].z = __ldg(q + 2); if (r + 3 < rows) v[i].w = __ldg(q + 3); }
      }
    }
  }
  // into s[k][row], row pitch ROWS + 4: 16-byte aligned rows for the vector reads
  __device__ __forceinline__ void put(float (*s)[ROWS + 4]) const {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int g = threadIdx.x + i * THREADS;
      if (kGroups % THREADS && g >= kGroups) continue;
      if (KFAST) {
        const int r = g / (BK / 4), k = (g % (BK / 4)) * 4;
        s[k][r] = v[i].x; s[k + 1][r] = v[i].y; s[k + 2][r] = v[i].z; s[k + 3][r] = v[i].w;
      } else {
        *reinterpret_cast<float4*>(&s[g / (ROWS / 4)][(g % (ROWS / 4)) * 4]) = v[i];
      }
    }
  }
};

// One tile, or the share of it of CTA `rank` of `ranks` (the first of them is CTA `first` of the cluster)
template <int BM, int BN, int TM, int TN, int BK, bool A_KFAST, bool B_KFAST>
__device__ __forceinline__ void simt_tile(const SimtGemm& p, int m0, int n0, int rank, int ranks, int first) {
  constexpr int THREADS = (BM / TM) * (BN / TN);
  constexpr int kTile = 2 * BK * (BM + 4) + 2 * BK * (BN + 4);
  constexpr int kSmem = kTile > BM * BN ? kTile : BM * BN;
  __shared__ __align__(16) float smem[kSmem];
  float (*As)[BK][BM + 4] = reinterpret_cast<float (*)[BK][BM + 4]>(smem);
  float (*Bs)[BK][BN + 4] = reinterpret_cast<float (*)[BK][BN + 4]>(smem + 2 * BK * (BM + 4));
  cg::cluster_group cluster = cg::this_cluster();
  const int kbeg = rank * p.k_per_cta, kend = min(p.K, kbeg + p.k_per_cta);
  const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  BlockLoader<BM, BK, THREADS, A_KFAST> la;
  BlockLoader<BN, BK, THREADS, B_KFAST> lb;
  if (kbeg < kend) {
    la.fetch(p.A, p.lda, m0, p.M, kbeg, kend, p.a_vec);
    lb.fetch(p.B, p.ldb, n0, p.N, kbeg, kend, p.b_vec);
    la.put(As[0]); lb.put(Bs[0]);
  }
  __syncthreads();
  int buf = 0;
  for (int k = kbeg; k < kend; k += BK, buf ^= 1) {
    const bool more = k + BK < kend;
    if (more) {
      la.fetch(p.A, p.lda, m0, p.M, k + BK, kend, p.a_vec);
      lb.fetch(p.B, p.ldb, n0, p.N, k + BK, kend, p.b_vec);
    }
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[buf][kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Bs[buf][kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    if (more) { la.put(As[buf ^ 1]); lb.put(Bs[buf ^ 1]); }
    __syncthreads();
  }
  if (ranks == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int m = m0 + ty * TM + i;
      if (m >= p.M) continue;
      float* c = p.C + (long long)m * p.ldc + n0 + tx * TN;
      if (TN == 4 && p.c_vec && n0 + tx * TN + 4 <= p.N) {
        *reinterpret_cast<float4*>(c) = make_float4(acc[i][0], acc[i][TN > 1 ? 1 : 0], acc[i][TN > 2 ? 2 : 0], acc[i][TN > 3 ? 3 : 0]);
      } else {
#pragma unroll
        for (int j = 0; j < TN; ++j) if (n0 + tx * TN + j < p.N) c[j] = acc[i][j];
      }
    }
    return;
  }
  // the partial tile into shared memory (the operand blocks are done with), then one slice of the tile per CTA
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) smem[(ty * TM + i) * BN + tx * TN + j] = acc[i][j];
  cluster.sync();
  const float* part[16];
#pragma unroll
  for (int r = 0; r < 16; ++r) part[r] = r < ranks ? cluster.map_shared_rank(smem, first + r) : smem;
  const int slice = (BM * BN + ranks - 1) / ranks, end = min(BM * BN, (rank + 1) * slice);
  for (int e = rank * slice + threadIdx.x; e < end; e += THREADS) {
    float t = 0.f;
#pragma unroll
    for (int r = 0; r < 16; ++r) if (r < ranks) t += part[r][e];
    const int m = m0 + e / BN, n = n0 + e % BN;
    if (m < p.M && n < p.N) p.C[(long long)m * p.ldc + n] = t;
  }
  cluster.sync();           // nobody leaves while its shared memory is still read
}
template <int BM, int BN, int TM, int TN, int BK, bool A_KFAST, bool B_KFAST>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) simt_gemm_kernel(const SimtGemm p) {
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  grid_dep_sync();
  simt_tile<BM, BN, TM, TN, BK, A_KFAST, B_KFAST>(p, blockIdx.y * BM, (int)(blockIdx.x / ranks) * BN, rank, ranks, 0);      // the CTAs of a cluster are neighbours in x
}

// ---- weight gradients of dense layers that wait for others --------------------------------------------------------------
// As the filter gradients of convolutions (hold_products): nobody reads them before the parameters are updated, and a launch
// each is a chain of 3-5 us kernels.  Tiles, shares of K and order of the sums are those of the separate launches.  All
// clusters have the largest size that one of the products asks for; smaller ones share a cluster.
constexpr int kSimtJobs = 16, kHeldTile = 32, kHeldTiles = 1024;
struct SimtJob { SimtGemm p; int ranks, n_tiles, tiles, first_cluster; };
struct SimtJobs { int n; SimtJob job[kSimtJobs]; };
__global__ void __launch_bounds__(128) simt_group_kernel(const __grid_constant__ SimtJobs jobs) {
  cg::cluster_group cluster = cg::this_cluster();
  const int size = (int)cluster.num_blocks(), at = (int)cluster.block_rank(), id = blockIdx.x / size;
  grid_dep_sync();
  int k = 0;
  while (k + 1 < jobs.n && jobs.job[k + 1].first_cluster <= id) ++k;
  const SimtJob& j = jobs.job[k];
  const int sub = at / j.ranks, tile = (id - j.first_cluster) * (size / j.ranks) + sub;
  if (tile < j.tiles) simt_tile<32, 32, 4, 2, 32, false, false>(j.p, tile / j.n_tiles * kHeldTile, tile % j.n_tiles * kHeldTile, at - sub * j.ranks, j.ranks, sub * j.ranks);
  if (size > 1 && (tile >= j.tiles || j.ranks == 1)) { cluster.sync(); cluster.sync(); }        // those of the tiles that are cut
}

template <int BM, int BN, int TM, int TN, int BK, bool AK, bool BKF>
static cudaError_t launch_simt(const SimtGemm& p, int cluster, cudaStream_t s) {
  if (cluster > 8) {
    static const cudaError_t allowed = cudaFuncSetAttribute(simt_gemm_kernel<BM, BN, TM, TN, BK, AK, BKF>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (allowed != cudaSuccess) return allowed;
  }
  return launch_cluster(simt_gemm_kernel<BM, BN, TM, TN, BK, AK, BKF>, cluster, dim3((unsigned)cluster * ((p.N + BN - 1) / BN), (p.M + BM - 1) / BM), dim3((BM / TM) * (BN / TN)), 0, s, p);
}
template <int BM, int BN, int TM, int TN, int BK>
static cudaError_t launch_simt_layout(const SimtGemm& p, bool a_kfast, bool b_kfast, int cluster, cudaStream_t s) {
  if (a_kfast) return b_kfast ? launch_simt<BM, BN, TM, TN, BK, true, true>(p, cluster, s) : launch_simt<BM, BN, TM, TN, BK, true, false>(p, cluster, s);
  return b_kfast ? launch_simt<BM, BN, TM, TN, BK, false, true>(p, cluster, s) : launch_simt<BM, BN, TM, TN, BK, false, false>(p, cluster, s);
}

// ---- a handful of rows against large weights: dense layers on small batches -------------------------------------------------
// Reading (the weight gradient: writing) the weights once is the bound, and what it takes is enough 16-byte accesses in flight.  Three
// kernels, one per place of the weights; up to 16 rows stay in registers.  Sums are cut over warps, and over a cluster's CTAs, and added in
// a fixed order.  7 rows against 4608 x 4096 and 4096 x 4096 weights (11.6 and 10.3 us at the copy rate), each: product 22.5 us, gradient of
// the rows 33.7, gradient of the weights 16.3 (the tiles above: 30.5, 44.5 and 24.2).  The first two still wait for memory: 3.1 and 2.0 TB/s.
//
// C = A[M x K] B[K x N]: a lane owns 4 columns, a warp a run of K, 8 rows of B in flight; the rows of A lie in shared memory.
// (With 16 rows in flight a block took so many registers that an SM held one: 46 us.)
constexpr int kRowThreads = 256, kRowWarps = kRowThreads / 32, kRowCols = 128;
template <int MR>
__global__ void __launch_bounds__(kRowThreads) rows_nn_kernel(const SimtGemm p) {
  extern __shared__ __align__(16) float rows_smem[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kw = p.k_per_cta / kRowWarps, seg = p.k_per_cta;
  grid_dep_sync();
  const int kbeg = rank * seg, count = max(0, min(seg, p.K - kbeg));
  for (int m = warp; m < MR; m += kRowWarps)
    for (int k = lane; k < seg; k += 32) {
      const bool there = m < p.M && k < count;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(rows_smem + m * seg + k)),
                   "l"(p.A + (there ? (long long)m * p.lda + kbeg + k : 0)), "r"(there ? 4 : 0) : "memory");
    }
  const int n = (int)(blockIdx.x / ranks) * kRowCols + lane * 4, k1 = min((warp + 1) * kw, count);
  float4 w[8];
  auto fetch = [&](int k) {
    const float* const b = p.B + (long long)(kbeg + k) * p.ldb + n;
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = n < p.N && k + j < k1 ? __ldg(reinterpret_cast<const float4*>(b + j * p.ldb)) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  fetch(warp * kw);                      // the first rows of B come with those of A
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  float2 acc[MR][2];
#pragma unroll
  for (int m = 0; m < MR; ++m) acc[m][0] = acc[m][1] = make_float2(0.f, 0.f);
  for (int k = warp * kw; k < k1; k += 8) {
#pragma unroll
    for (int m = 0; m < MR; ++m) {
      const float4 x0 = *reinterpret_cast<const float4*>(rows_smem + m * seg + k), x1 = *reinterpret_cast<const float4*>(rows_smem + m * seg + k + 4);
      const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 xx = make_float2(x[j], x[j]);
        acc[m][0] = __ffma2_rn(xx, make_float2(w[j].x, w[j].y), acc[m][0]);
        acc[m][1] = __ffma2_rn(xx, make_float2(w[j].z, w[j].w), acc[m][1]);
      }
    }
    if (k + 8 < k1) fetch(k + 8);
  }
  __syncthreads();                       // the rows are done with
  float4* const part = reinterpret_cast<float4*>(rows_smem);               // [warp][MR][32 lanes]
#pragma unroll
  for (int m = 0; m < MR; ++m) part[(warp * MR + m) * 32 + lane] = make_float4(acc[m][0].x, acc[m][0].y, acc[m][1].x, acc[m][1].y);
  __syncthreads();
  auto add = [](float4& a, const float4 b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; };
  auto store = [&](int i, const float4 v) {
    const int m = i >> 5, c = (int)(blockIdx.x / ranks) * kRowCols + (i & 31) * 4;
    if (m >= p.M || c >= p.N) return;
    float* const dst = p.C + (long long)m * p.ldc + c;
    if (p.c_vec) *reinterpret_cast<float4*>(dst) = v;
    else { dst[0] = v.x; dst[1] = v.y; dst[2] = v.z; dst[3] = v.w; }
  };
  for (int i = threadIdx.x; i < MR * 32; i += kRowThreads) {
    float4 t = part[i];
#pragma unroll
    for (int w = 1; w < kRowWarps; ++w) add(t, part[w * MR * 32 + i]);
    if (ranks == 1) store(i, t); else part[i] = t;
  }
  if (ranks == 1) return;
  cluster.sync();
  for (int i = rank * kRowThreads + threadIdx.x; i < MR * 32; i += ranks * kRowThreads) {
    float4 t = *cluster.map_shared_rank(part + i, 0);
    for (int r = 1; r < ranks; ++r) add(t, *cluster.map_shared_rank(part + i, r));
    store(i, t);
  }
  cluster.sync();           // nobody leaves while its shared memory is still read
}

// C = A[M x K] B[N x K]^T: a warp owns two rows of B along a run of K, a lane 4 columns at a time; the rows of A come through L1.
// (Four rows a warp halve those reads and take registers: the same time.)
constexpr int kRowSet = 2;
template <int MR>
__global__ void __launch_bounds__(kRowThreads) rows_nt_kernel(const SimtGemm p) {
  constexpr int kSums = MR * kRowSet;
  __shared__ float part[kRowWarps][kSums];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, runs = (p.K + p.k_per_cta - 1) / p.k_per_cta;       // of K, neighbouring warps
  grid_dep_sync();
  const int set = ((int)blockIdx.x * kRowWarps + warp) / runs, run = warp % runs, n0 = set * kRowSet;
  const int kend = min(p.K, (run + 1) * p.k_per_cta);
  float2 acc[kSums];
#pragma unroll
  for (int i = 0; i < kSums; ++i) acc[i] = make_float2(0.f, 0.f);
  const float* const b0 = p.B + (long long)min(n0, p.N - 1) * p.ldb;
  const float* const b1 = p.B + (long long)min(n0 + 1, p.N - 1) * p.ldb;
#pragma unroll 4
  for (int k = run * p.k_per_cta + lane * 4; k < kend; k += 128) {
    const float4 w[kRowSet] = {__ldg(reinterpret_cast<const float4*>(b0 + k)), __ldg(reinterpret_cast<const float4*>(b1 + k))};
#pragma unroll
    for (int m = 0; m < MR; ++m) {
      const float4 x = __ldg(reinterpret_cast<const float4*>(p.A + (long long)min(m, p.M - 1) * p.lda + k));
#pragma unroll
      for (int r = 0; r < kRowSet; ++r) {
        float2& a = acc[m * kRowSet + r];
        a = __ffma2_rn(make_float2(x.z, x.w), make_float2(w[r].z, w[r].w), __ffma2_rn(make_float2(x.x, x.y), make_float2(w[r].x, w[r].y), a));
      }
    }
  }
  float sum[kSums];
#pragma unroll
  for (int i = 0; i < kSums; ++i) sum[i] = acc[i].x + acc[i].y;
  // kSums sums over 32 lanes: a step adds pairs of lanes and halves what each keeps, lane i ends up with sum i
  if (kSums == 16) {
#pragma unroll
    for (int i = 0; i < kSums; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 16);
  }
#pragma unroll
  for (int step = kSums / 2; step > 0; step /= 2)
#pragma unroll
    for (int i = 0; i < step; ++i) {
      const bool upper = lane & step;
      const float keep = upper ? sum[i + step] : sum[i], give = upper ? sum[i] : sum[i + step];
      sum[i] = keep + __shfl_xor_sync(0xffffffffu, give, step);
    }
  if (lane < kSums) part[warp][lane] = sum[0];
  __syncthreads();
  if (run != 0 || lane >= kSums) return;
  float t = part[warp][lane];
  for (int r = 1; r < runs; ++r) t += part[warp + r][lane];
  const int m = lane / kRowSet, n = n0 + lane % kRowSet;
  if (m < p.M && n < p.N) p.C[(long long)m * p.ldc + n] = t;
}

// C = A[K x M]^T B[K x N] of at most KR rows: a thread keeps its 4 columns of B and writes them times one row of A^T after the other.
constexpr int kOuterRows = 32;
template <int KR>
__global__ void __launch_bounds__(kRowThreads) rows_tn_kernel(const SimtGemm p) {
  grid_dep_sync();
  const int n = ((int)blockIdx.x * kRowThreads + threadIdx.x) * 4, m0 = blockIdx.y * kOuterRows;
  if (n >= p.N) return;
  float4 b[KR];
#pragma unroll
  for (int k = 0; k < KR; ++k) b[k] = k < p.K ? __ldg(reinterpret_cast<const float4*>(p.B + (long long)k * p.ldb + n)) : make_float4(0.f, 0.f, 0.f, 0.f);
  const int m1 = min(p.M, m0 + kOuterRows);
  for (int m = m0; m < m1; m += 4) {
    float4 out[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) out[j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      if (k >= p.K) break;
      const float4 a4 = __ldg(reinterpret_cast<const float4*>(p.A + (long long)k * p.lda + m));
      const float a[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        out[j].x = fmaf(a[j], b[k].x, out[j].x); out[j].y = fmaf(a[j], b[k].y, out[j].y);
        out[j].z = fmaf(a[j], b[k].z, out[j].z); out[j].w = fmaf(a[j], b[k].w, out[j].w);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(p.C + (long long)(m + j) * p.ldc + n) = out[j];
  }
}

// Takes the product if it is one of those: 1, 0 if not, -1 on error.  Below a million weights, or where these leave SMs without a block
// (2048 x 1000: 13.4 us against 9.3), the tiles are faster; rows that cannot be read 16 bytes at a time stay with them, too.
constexpr int kFewRows = 16;
constexpr size_t kRowSmem = 200 * 1024;
template <int MR> static int launch_rows_nn(SimtGemm p, cudaStream_t s) {
  const int sms = device_sm_count(), groups = (p.N + kRowCols - 1) / kRowCols;
  int cluster = 1;
  auto smem = [&] { return std::max((size_t)p.k_per_cta * MR, (size_t)kRowWarps * MR * kRowCols) * sizeof(float); };
  auto cut = [&] { p.k_per_cta = (int)(((long long)p.K + cluster * kRowWarps * 8 - 1) / (cluster * kRowWarps * 8)) * kRowWarps * 8; };        // a warp's run is a multiple of 8
  cut();
  while (cluster < 8 && (groups * cluster < 2 * sms || smem() > kRowSmem / 2) && p.K >= 64 * kRowWarps * cluster) { cluster *= 2; cut(); }
  if (smem() > kRowSmem || groups * cluster < sms) return 0;
  static const cudaError_t attr = cudaFuncSetAttribute(rows_nn_kernel<MR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowSmem);
  TF_CUDA(attr);
  KernelTimer kt("rows_gemm", s, 2.0 * (double)p.M * p.N * p.K, 0, 1);
  TF_CUDA(launch_cluster(rows_nn_kernel<MR>, cluster, dim3(groups * cluster), dim3(kRowThreads), smem(), s, p));
  return 1;
}
static int rows_matmul(const SimtGemm& p, bool tA, bool tB, cudaStream_t s) {
  const int sms = device_sm_count();
  if (!tA && p.M <= kFewRows && (double)p.K * p.N >= 1e6) {
    if (!tB && p.b_vec && p.N % 4 == 0) return p.M <= 8 ? launch_rows_nn<8>(p, s) : launch_rows_nn<16>(p, s);
    if (tB && p.a_vec && p.b_vec && p.K % 4 == 0) {
      const long long sets = (p.N + kRowSet - 1) / kRowSet;
      int runs = 1;
      while (runs < kRowWarps && sets * runs < 24ll * sms && p.K >= 256 * runs) runs *= 2;
      if (sets * runs < 8ll * sms) return 0;
      SimtGemm q = p;
      q.k_per_cta = (int)(((p.K + runs - 1) / runs + 127) / 128 * 128);
      runs = (p.K + q.k_per_cta - 1) / q.k_per_cta;
      while (kRowWarps % runs) { q.k_per_cta += 128; runs = (p.K + q.k_per_cta - 1) / q.k_per_cta; }       // whole sets in a block
      const dim3 grid((unsigned)((sets * runs + kRowWarps - 1) / kRowWarps));
      KernelTimer kt("rows_gemm", s, 2.0 * (double)p.M * p.N * p.K, 0, 1);
      TF_CUDA(p.M <= 8 ? launch_dep(rows_nt_kernel<8>, grid, dim3(kRowThreads), 0, s, q) : launch_dep(rows_nt_kernel<16>, grid, dim3(kRowThreads), 0, s, q));
      return 1;
    }
  }
  if (tA && !tB && p.K <= kFewRows && (double)p.M * p.N >= 1e6 && p.a_vec && p.b_vec && p.c_vec && p.M % 4 == 0 && p.N % 4 == 0 && (p.M + kOuterRows - 1) / kOuterRows <= 65535) {
    const dim3 grid((p.N + 4 * kRowThreads - 1) / (4 * kRowThreads), (p.M + kOuterRows - 1) / kOuterRows);
    KernelTimer kt("rows_gemm", s, 2.0 * (double)p.M * p.N * p.K, 0, 1);
    TF_CUDA(p.K <= 8 ? launch_dep(rows_tn_kernel<8>, grid, dim3(kRowThreads), 0, s, p) : launch_dep(rows_tn_kernel<16>, grid, dim3(kRowThreads), 0, s, p));
    return 1;
  }
  return 0;
}

static thread_local std::vector<SimtJob> t_held_simt;
void drop_held_simt() { t_held_simt.clear(); }
int launch_held_simt(cudaStream_t s) {
  std::vector<SimtJob> all;
  all.swap(t_held_simt);
  for (size_t from = 0; from < all.size(); from += kSimtJobs) {
    SimtJobs jobs;
    jobs.n = (int)std::min(all.size() - from, (size_t)kSimtJobs);
    int size = 1, clusters = 0;
    double flops = 0;
    for (int i = 0; i < jobs.n; ++i) size = std::max(size, all[from + i].ranks);
    for (int i = 0; i < jobs.n; ++i) {
      SimtJob& j = jobs.job[i] = all[from + i];
      j.first_cluster = clusters;
      clusters += (j.tiles * j.ranks + size - 1) / size;
      flops += 2.0 * j.p.M * j.p.N * j.p.K;
    }
    note_compute_stream(s);
    KernelTimer kt("simt_gemm", s, flops, 0, 1);
    TF_CUDA(launch_cluster(simt_group_kernel, size, dim3((unsigned)(clusters * size)), dim3(128), 0, s, jobs));
    TF_AFTER(s, "weight gradients");
  }
  return 0;
}

// C[M x N] = op(A) op(B), row-major, leading dimensions of the arrays as they are stored.
int simt_matmul(const float* A, bool tA, const float* B, bool tB, float* C, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldb, int64_t ldc, cudaStream_t s, const char* what) {
  if (M <= 0 || N <= 0) return 0;
  TF_REQUIRE(M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), "%s: extent too large", what);
  SimtGemm p{A, B, C, (int)M, (int)N, (int)K, lda, ldb, ldc, 0, lda % 4 == 0 && aligned16(A), ldb % 4 == 0 && aligned16(B), ldc % 4 == 0 && aligned16(C)};
  const int sms = device_sm_count();
  // Tile: 8 rows where there are no more (the rest of a taller tile would multiply nothing), 64 x 64 once those alone
  // give every SM one, else 32 x 32.  Cluster: the smallest power of two that occupies the SMs, with at least two K
  // blocks to each CTA, at most 8; the 8-row tile only streams the weights and wants several CTAs per SM, so it may
  // take the non-portable 16.
  //   M x K x N          this kernel   before      tensor path with its packs (us, back to back)
  //   64 x 784 x 256         6.4         20             19.0
  //   1000 x 256 x 100       6.7         22             15.6
  //   32 x 2048 x 2048      15.9        110             24.8
  //   1000 x 784 x 256      24.7         58             21.1
  const int cfg = M <= 8 ? 0 : ((M + 63) / 64) * ((N + 63) / 64) >= sms || M > 32 * 65535ll ? 2 : 1;
  const int bm = cfg == 0 ? 8 : cfg == 1 ? 32 : 64, bn = cfg == 1 ? 32 : 64, bk = cfg == 2 ? 16 : 32;
  const long long tiles = ((M + bm - 1) / bm) * ((N + bn - 1) / bn);
  TF_REQUIRE((M + bm - 1) / bm <= 65535, "%s: M too large for the CUDA-core path", what);
  const int want = cfg == 0 ? 6 * sms : cfg == 1 ? 3 * sms : sms;
  int cluster = 1;
  while (cluster < (cfg == 0 ? 16 : 8) && tiles * cluster < want && (K + bk - 1) / bk >= 4 * cluster) cluster *= 2;
  p.k_per_cta = (int)(((K + cluster - 1) / cluster + bk - 1) / bk * bk);
  if (cfg == 1 && tA && !tB && tiles <= kHeldTiles && may_hold(s) && held(t_held_simt, SimtJob{p, cluster, (int)((N + 31) / 32), (int)tiles, 0})) return 0;
  note_compute_stream(s);
  if (const int rc = rows_matmul(p, tA, tB, s)) {
    if (rc < 0) return -1;
    TF_AFTER(s, what);
    return 0;
  }
  KernelTimer kt("simt_gemm", s, 2.0 * (double)M * (double)N * (double)K, 0, 1);
  const cudaError_t e = cfg == 0 ? launch_simt_layout<8, 64, 8, 1, 32>(p, !tA, tB, cluster, s)
                      : cfg == 1 ? launch_simt_layout<32, 32, 4, 2, 32>(p, !tA, tB, cluster, s)
                                 : launch_simt_layout<64, 64, 4, 4, 16>(p, !tA, tB, cluster, s);
  TF_CUDA(e);
  TF_AFTER(s, what);
  return 0;
}

}  // namespace tf
