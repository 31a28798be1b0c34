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

template <int BM, int BN, int TM, int TN, int BK, bool A_KFAST, bool B_KFAST>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) simt_gemm_kernel(const SimtGemm p) {
  constexpr int THREADS = (BM / TM) * (BN / TN);
  constexpr int kTile = 2 * BK * (BM + 4) + 2 * BK * (BN + 4);
  constexpr int kSmem = kTile > BM * BN ? kTile : BM * BN;
  __shared__ __align__(16) float smem[kSmem];
  float (*As)[BK][BM + 4] = reinterpret_cast<float (*)[BK][BM + 4]>(smem);
  float (*Bs)[BK][BN + 4] = reinterpret_cast<float (*)[BK][BN + 4]>(smem + 2 * BK * (BM + 4));
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  grid_dep_sync();
  const int m0 = blockIdx.y * BM, n0 = (int)(blockIdx.x / ranks) * BN;      // the CTAs of a cluster are neighbours in x
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
  for (int r = 0; r < 16; ++r) part[r] = r < ranks ? cluster.map_shared_rank(smem, r) : smem;
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
  note_compute_stream(s);
  KernelTimer kt("simt_gemm", s, 2.0 * (double)M * (double)N * (double)K, 0, 1);
  const cudaError_t e = cfg == 0 ? launch_simt_layout<8, 64, 8, 1, 32>(p, !tA, tB, cluster, s)
                      : cfg == 1 ? launch_simt_layout<32, 32, 4, 2, 32>(p, !tA, tB, cluster, s)
                                 : launch_simt_layout<64, 64, 4, 4, 16>(p, !tA, tB, cluster, s);
  TF_CUDA(e);
  TF_AFTER(s, what);
  return 0;
}

}  // namespace tf
