// C[M, N] = A[M, K] * W[N, K]^T with float32 FMA accumulation on the CUDA cores.
// This is the matrix product of the true 32-bit path (no tensor cores, no TF32) and the plain
// twin of the tensor-core products.  Counterpart in the reference: cublasLtMatmul through
// tops/csrc/tops/tensorrt_llm/common/cublasMMWrapper.cpp:122-209.
//
// Float32: K is cut into eight parts of part_len(K) values (a multiple of 32; the last ones may be empty).  A part is the
// sum of two chains of FMAs in ascending k, of its even k and of its odd k (the two halves of fma.rn.f32x2 on the values as
// they lie in memory), and out = (((p0 + p1) + p2) + p3) + (((p4 + p5) + p6) + p7).
// All three kernels below keep to that order, so a row's result does not depend by a bit on M, on which other rows share
// the launch or on the kernel that was chosen.  (One chain over all of K, as before, leaves a product of few rows no
// parallelism along k, and its rounding error is larger.)
// bfloat16: every output element is accumulated by one thread over k = 0 .. K-1 in ascending order.
#include "common.cuh"

LMSF_DEFINE_LAST_ERROR(lmsf_gemm_simt)

namespace lmsf {

constexpr int BM = 64, BN = 64, BK = 16;

constexpr int kParts = 8;
__host__ __device__ constexpr int part_len(int K) { return ((K + kParts - 1) / kParts + 31) / 32 * 32; }

// Any sizes and alignments, one scalar load per value.
template <typename TA, typename TC>
__global__ void __launch_bounds__(256) gemm_tn_kernel(TC* __restrict__ C, const TA* __restrict__ A,
                                                      const TA* __restrict__ W, int M, int N, int K, long long lda,
                                                      long long ldw, long long ldc, long long batch_a,
                                                      long long batch_w, long long batch_c) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  A += (size_t)blockIdx.z * batch_a;   // one product per blockIdx.z (a head, for instance); all strides 0 for one product
  W += (size_t)blockIdx.z * batch_w;
  C += (size_t)blockIdx.z * batch_c;
  const int tx = tid % 16, ty = tid / 16;  // thread's 4x4 patch: rows ty*4.., cols tx*4..
  const int lr = tid / 4, lk = (tid % 4) * 4;  // loader: row lr of the tile, k offsets lk..lk+3

  float acc[4][4], odd[4][4], tot[4][4], half[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = odd[i][j] = tot[i][j] = half[i][j] = 0.f;
  const bool in_parts = sizeof(TA) == 4;   // float32: the sum of the parts
  const int L = part_len(K);

  for (int k0 = 0; k0 < K; k0 += BK) {
    if (in_parts && k0 > 0 && k0 % L == 0) {
      const bool to_half = k0 == kParts / 2 * L;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          tot[i][j] += acc[i][j] + odd[i][j];
          acc[i][j] = odd[i][j] = 0.f;
          if (to_half) { half[i][j] = tot[i][j]; tot[i][j] = 0.f; }
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = k0 + lk + e;
      const int m = m0 + lr, n = n0 + lr;
      As[lk + e][lr] = (m < M && k < K) ? to_f32(A[(size_t)m * lda + k]) : 0.f;
      Ws[lk + e][lr] = (n < N && k < K) ? to_f32(W[(size_t)n * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float& c = in_parts && (kk & 1) ? odd[i][j] : acc[i][j];
          c = fmaf(a[i], w[j], c);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) C[(size_t)m * ldc + n] = from_f32<TC>(in_parts ? half[i][j] + (tot[i][j] + (acc[i][j] + odd[i][j])) : acc[i][j]);
    }
  }
}

// ---- float32, rows that can be read 16 bytes at a time ------------------------------------------------------

struct F32Args {
  float* C; const float* A; const float* W;
  int M, N, K;
  long long lda, ldw, ldc, batch_a, batch_w, batch_c;
  int w_constant;        // no kernel of the step writes W: it may be read before the kernel ahead has ended
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool ok) {   // 16 bytes, zeros where there is nothing
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// d += a * b, both halves
__device__ __forceinline__ void fma2(float2& d, float ax, float ay, float bx, float by) {
  asm("{\n.reg .b64 a, b, c;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%0, %1};\nfma.rn.f32x2 c, a, b, c;\nmov.b64 {%0, %1}, c;\n}\n"
      : "+f"(d.x), "+f"(d.y) : "f"(ax), "f"(ay), "f"(bx), "f"(by));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Up to 16 rows of A: a stream over W.  A block takes 16 rows of W, its warp w the parts 2 w (lanes 0..15, a row of W
// each) and 2 w + 1 (lanes 16..31), through a ring of its own of cp.async stages of 32 k: 4 KB of W (chunks of 16 bytes
// swizzled by the row, so that eight lanes read eight different banks) and the matching x, which all lanes of a part read
// together.  Bound by the stream: with five stages (three at 16 rows) two blocks fit an SM and keep 128 KB of W asked for.  Where the caller
// says that W is a weight, its first stages are asked for before the kernel before this one has ended, and the kernel after this one
// may start as early.  Any other W may be what that kernel writes: then everything waits, as in plain stream order.  One launch after the
// other on different weights at 3 rows: 128,256 x 2,048 in 151 us (7.0 TB/s), 16,384 x 2,048 in 25 us (5.3), 2,048 x 8,192 in
// 14 us (4.8); 31 and 25 us for the last two with single FMAs and an address per copy.  (Prompts of 515 tokens and 12 decoded
// tokens for three requests, Llama-3.2-1B: 294 -> 50.8 ms with this kernel and the next.)
template <int NT, bool DEEP> constexpr int few_stages = (NT <= 4 ? 5 : (NT <= 8 ? 4 : 3)) * (DEEP ? 2 : 1);
template <int NT, bool DEEP>
__global__ void __launch_bounds__(128) f32_few_rows_kernel(F32Args a) {
  constexpr int kFewStages = few_stages<NT, DEEP>;
  constexpr int kStage = 4096 + 2 * NT * 128;
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = lane & 15, h = lane >> 4;
  const int n0 = blockIdx.x * 16;
  const float* A = a.A + (size_t)blockIdx.y * a.batch_a;
  const float* W = a.W + (size_t)blockIdx.y * a.batch_w;
  float* C = a.C + (size_t)blockIdx.y * a.batch_c;
  const int L = part_len(a.K), first = 2 * warp * L;
  const int n_st = first < a.K ? L / 32 : 0;          // the second part's values beyond K are zeros
  const uint32_t ring = smem_u32(smem) + warp * (kFewStages * kStage);

  // the lane's copies: chunk ch of rows r0, r0 + 4, ... of the first part, then of the second
  const int r0 = lane >> 3, ch = lane & 7;
  const float* w0 = W + (size_t)(n0 + r0) * a.ldw + first + ch * 4;
  const size_t w_step = (size_t)4 * a.ldw;
  const bool whole = n0 + 16 <= a.N && a.K == kParts * L;        // nothing to leave out
  auto issue_w = [&](int c) {
    const uint32_t st = ring + (c % kFewStages) * kStage;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = r0 + 4 * i;
      const uint32_t dst = st + row * 128 + ((ch ^ (row & 7)) << 4);
      const float* src = w0 + (i & 3) * w_step + (i >> 2) * L + c * 32;
      if (whole) {
        cp16(dst, src);
      } else {
        const bool ok = n0 + (row & 15) < a.N && first + (i >> 2) * L + c * 32 + ch * 4 < a.K;
        cp16(dst, ok ? src : W, ok);
      }
    }
  };
  auto issue_x = [&](int c) {
    const uint32_t st = ring + (c % kFewStages) * kStage + 4096;
#pragma unroll
    for (int i = 0; i < (NT * 16 + 31) / 32; ++i) {
      const int row = r0 + 4 * i;
      if (NT % 2 && row >= 2 * NT) break;
      const int k = first + (row / NT) * L + c * 32 + ch * 4, m = row % NT;
      const bool ok = m < a.M && k < a.K;
      cp16(st + row * 128 + (ch << 4), ok ? A + (size_t)m * a.lda + k : A, ok);
    }
  };
  if (a.w_constant) {
    pdl_launch_dependents();
    for (int s = 0; s < kFewStages - 1; ++s)
      if (s < n_st) issue_w(s);
  }
  pdl_wait();
  for (int s = 0; s < kFewStages - 1; ++s) {
    if (s < n_st) {
      if (!a.w_constant) issue_w(s);
      issue_x(s);
    }
    cp_commit();
  }

  float2 acc[NT];
#pragma unroll
  for (int m = 0; m < NT; ++m) acc[m] = make_float2(0.f, 0.f);
  for (int c = 0; c < n_st; ++c) {
    cp_wait<kFewStages - 2>();
    __syncwarp();
    if (c + kFewStages - 1 < n_st) { issue_w(c + kFewStages - 1); issue_x(c + kFewStages - 1); }
    cp_commit();
    const unsigned char* st = smem + warp * (kFewStages * kStage) + (c % kFewStages) * kStage;
    const unsigned char* xs = st + 4096 + h * (NT * 128);
#pragma unroll(NT <= 8 ? 8 : 2)
    for (int j = 0; j < 8; ++j) {
      const float4 w = *reinterpret_cast<const float4*>(st + lane * 128 + ((j ^ (r & 7)) << 4));
#pragma unroll
      for (int m = 0; m < NT; ++m) {
        const float4 x = *reinterpret_cast<const float4*>(xs + m * 128 + (j << 4));
        fma2(acc[m], x.x, x.y, w.x, w.y);
        fma2(acc[m], x.z, x.w, w.z, w.w);
      }
    }
  }
  cp_wait<0>();
  __syncthreads();
  float* part = reinterpret_cast<float*>(smem);       // [part][m][row]
#pragma unroll
  for (int m = 0; m < NT; ++m) part[((2 * warp + h) * NT + m) * 16 + r] = acc[m].x + acc[m].y;
  __syncthreads();
  for (int i = threadIdx.x; i < NT * 16; i += 128) {
    const int m = i / 16, n = n0 + i % 16;
    if (m >= a.M || n >= a.N) continue;
    float p[kParts];
#pragma unroll
    for (int q = 0; q < kParts; ++q) p[q] = part[q * NT * 16 + i];
    C[(size_t)m * a.ldc + n] = (((p[0] + p[1]) + p[2]) + p[3]) + (((p[4] + p[5]) + p[6]) + p[7]);
  }
}

// More rows: tiles of 64 rows of A and 128 of W by 128 threads with 8 x 8 results each (a row of A every 8 rows, a row of W
// every 16, so that the reads of four k of a warp's 4 x 8 lanes fall on different banks), cp.async stages of 32 k.  Bound by the
// FMA pipe; 128 fma.rn.f32x2 per 16 reads of 16 bytes (single FMAs stalled on their operands' register banks).  CS: blocks of a cluster that share a tile along k, where the tiles alone
// leave SMs idle: 2 (a half of the parts each) or 8 (a part each); their sums meet in shared memory.  At 515 rows
// 16,384 x 2,048 takes 0.87 ms (39.6 TFLOP/s), 2,048 x 8,192 0.45 ms, 2,048 x 2,048 0.122 ms; 0.99, 0.49 and 0.131 ms with
// single FMAs.
constexpr int TM = 64, TN = 128, TK = 32, kTileStages = 2, kTileRow = TK * 4 + 16, kTileStage = (TM + TN) * kTileRow;

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_remote(uint32_t addr, int rank) {
  uint32_t ra;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(ra) : "memory");
  return v;
}

template <int CS>
__global__ void __launch_bounds__(128, 2) f32_tile_kernel(F32Args a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = blockIdx.x % CS;                    // clusters lie along x
  const int m0 = blockIdx.x / CS * TM, n0 = blockIdx.y * TN;
  const int tx = (lane & 7) + 8 * (warp & 1), ty = (lane >> 3) + 4 * (warp >> 1);   // rows tx + 16 j of W, ty + 8 i of A
  const float* A = a.A + (size_t)blockIdx.z * a.batch_a;
  const float* W = a.W + (size_t)blockIdx.z * a.batch_w;
  float* C = a.C + (size_t)blockIdx.z * a.batch_c;
  const int L = part_len(a.K), first = rank * (kParts / CS) * L, st_part = L / TK;
  const int n_st = first < a.K ? min(kParts / CS * st_part, (a.K - first + TK - 1) / TK) : 0;
  const uint32_t base = smem_u32(smem);

  auto issue = [&](int s) {
    const uint32_t st = base + (s % kTileStages) * kTileStage;
    const int k0 = first + s * TK;
#pragma unroll
    for (int i = 0; i < (TM + TN) * 8 / 128; ++i) {
      const int idx = tid + 128 * i, row = idx >> 3, ch = idx & 7, k = k0 + ch * 4;
      const bool of_a = row < TM;                      // the same for all threads of a pass
      const int g = of_a ? m0 + row : n0 + row - TM;
      const bool ok = g < (of_a ? a.M : a.N) && k < a.K;
      const float* src = of_a ? A + (size_t)g * a.lda + k : W + (size_t)g * a.ldw + k;
      cp16(st + row * kTileRow + (ch << 4), ok ? src : a.A, ok);
    }
  };

  float2 acc[8][8];
  float* tot = reinterpret_cast<float*>(smem + kTileStages * kTileStage);   // [8 i + j][thread]: the parts of a half so far
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = make_float2(0.f, 0.f);
  for (int s = 0; s < kTileStages - 1; ++s) {
    if (s < n_st) issue(s);
    cp_commit();
  }
  bool parked = false;                                 // CS 1: the first four parts' sum waits in C
  int next_fold = st_part, parts_in_half = 0;
  for (int s = 0; s < n_st; ++s) {
    cp_wait<kTileStages - 2>();
    __syncthreads();
    if (s + kTileStages - 1 < n_st) issue(s + kTileStages - 1);
    cp_commit();
    const unsigned char* st = smem + (s % kTileStages) * kTileStage;
    const unsigned char* as = st + ty * kTileRow;
    const unsigned char* ws = st + (TM + tx) * kTileRow;
#pragma unroll
    for (int k4 = 0; k4 < TK / 4; ++k4) {
      float4 w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = *reinterpret_cast<const float4*>(ws + 16 * j * kTileRow + k4 * 16);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(as + 8 * i * kTileRow + k4 * 16);
#pragma unroll
        for (int j = 0; j < 8; ++j) fma2(acc[i][j], x.x, x.y, w[j].x, w[j].y);
#pragma unroll
        for (int j = 0; j < 8; ++j) fma2(acc[i][j], x.z, x.w, w[j].z, w[j].w);
      }
    }
    if (CS < kParts && (s + 1 == next_fold || s + 1 == n_st)) {
      next_fold += st_part;
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float* t = tot + (8 * i + j) * 128 + tid;
          const float p = acc[i][j].x + acc[i][j].y;
          *t = parts_in_half ? *t + p : p;
          acc[i][j] = make_float2(0.f, 0.f);
        }
      ++parts_in_half;
      if (CS == 1 && s + 1 == kParts / 2 * st_part && s + 1 < n_st) {
        parked = true;
        parts_in_half = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int m = m0 + ty + 8 * i, n = n0 + tx + 16 * j;
            if (m < a.M && n < a.N) C[(size_t)m * a.ldc + n] = tot[(8 * i + j) * 128 + tid];
          }
      }
    }
  }
  cp_wait<0>();
  if constexpr (CS == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int m = m0 + ty + 8 * i, n = n0 + tx + 16 * j;
        if (m < a.M && n < a.N) {
          float* c = C + (size_t)m * a.ldc + n;
          const float t = tot[(8 * i + j) * 128 + tid];
          *c = parked ? *c + t : t;
        }
      }
  } else {
    const uint32_t tot_addr = base + kTileStages * kTileStage;
    if (CS == kParts || parts_in_half == 0) {          // a part each, or a half that K does not reach (zeros)
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) tot[(8 * i + j) * 128 + tid] = acc[i][j].x + acc[i][j].y;
    }
    cluster_sync();
    if (CS == 2 && rank == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int m = m0 + ty + 8 * i, n = n0 + tx + 16 * j;
          const float v = tot[(8 * i + j) * 128 + tid] + ld_remote(tot_addr + ((8 * i + j) * 128 + tid) * 4, 1);
          if (m < a.M && n < a.N) C[(size_t)m * a.ldc + n] = v;
        }
    }
    if (CS == kParts) {                                // block `rank` adds up the rows ty + 8 rank of the tile
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float p[kParts];
#pragma unroll
        for (int q = 0; q < kParts; ++q) p[q] = ld_remote(tot_addr + ((8 * rank + j) * 128 + tid) * 4, q);
        const int m = m0 + ty + 8 * rank, n = n0 + tx + 16 * j;
        if (m < a.M && n < a.N)
          C[(size_t)m * a.ldc + n] = (((p[0] + p[1]) + p[2]) + p[3]) + (((p[4] + p[5]) + p[6]) + p[7]);
      }
    }
    cluster_sync();                                    // nobody leaves while its sums are being read
  }
}

static int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  }
  return n;
}

template <int NT, bool DEEP>
static int launch_few(const F32Args& a, int batch, cudaStream_t s) {
  constexpr int smem = 4 * few_stages<NT, DEEP> * (4096 + 2 * NT * 128);
  cudaError_t e = cudaFuncSetAttribute(f32_few_rows_kernel<NT, DEEP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  return launch_pdl(f32_few_rows_kernel<NT, DEEP>, dim3(ceil_div(a.N, 16), batch), dim3(128), smem, s, a);
}

// At most one block an SM and a long stream each (K of 4,096 and more): the ring takes all of the shared memory.
// Shorter streams leave room for the next product's blocks, whose first stages then overlap.  (Rings of both depths at 1, 3, 8 and 16
// rows: 2,048 x 8,192 15.1 -> 13.3, 18.1 -> 13.9, 29.4 -> 22.8 and 58.5 -> 49.6 us; 1,024 x 16,384 28.1 -> 23.2, 31.9 -> 24.5, 55.2 ->
// 42.5, 112 -> 97; 1,024 x 4,096 7.6 -> 6.6, 8.6 -> 7.0, 14.7 -> 11.6, 28.7 -> 25.0; 256 x 8,192 within 3 %.  Below the line, 2,048 x
// 2,048: 4.7 -> 4.8, 5.6 -> 5.0, 8.3 -> 7.2, 15.7 -> 13.5 of a product alone after others like it.)
template <int NT>
static int launch_few_rows(const F32Args& a, int batch, cudaStream_t s) {
  const bool deep = (long long)ceil_div(a.N, 16) * batch <= sm_count() && a.K >= 4096;
  return deep ? launch_few<NT, true>(a, batch, s) : launch_few<NT, false>(a, batch, s);
}

template <int CS>
static int launch_tile(const F32Args& a, int batch, cudaStream_t s) {
  constexpr int smem = kTileStages * kTileStage + 64 * 128 * 4;
  cudaError_t e = cudaFuncSetAttribute(f32_tile_kernel<CS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ceil_div(a.M, TM) * CS, ceil_div(a.N, TN), batch);
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, f32_tile_kernel<CS>, a);
}

// Few rows: a build takes as many rows as its number says or fewer, and pays for all of them (FMAs, and reads of x from shared
// memory): 16,384 x 2,048 takes 22.5, 22.4, 23.4, 27.1, 27.3, 34.4 and 61.2 us in the builds of 1, 2, 3, 4, 6, 8 and 16, to a few percent
// whatever the rows.  So up to 8 rows the builds lie close together, and 5 and 7 rows, which lose little (27.4 and 34.8), go with
// the next; between 8 and 16 none has been tried.  17 rows by tiles: 123 us.
static int launch_f32(const F32Args& a, int batch, cudaStream_t s) {
  if (a.M <= 1) return launch_few_rows<1>(a, batch, s);
  if (a.M <= 2) return launch_few_rows<2>(a, batch, s);
  if (a.M == 3) return launch_few_rows<3>(a, batch, s);
  if (a.M <= 4) return launch_few_rows<4>(a, batch, s);
  if (a.M <= 6) return launch_few_rows<6>(a, batch, s);
  if (a.M <= 8) return launch_few_rows<8>(a, batch, s);
  if (a.M <= 16) return launch_few_rows<16>(a, batch, s);
  // Two blocks fit an SM: the tiles alone where they fill the device, shared by two along k where that fills it, else by eight.  (Alone,
  // by two, by eight at K = 2,048: 16 tiles 136, 76 and 35 us, 64 tiles 139, 76 and 66, 144 tiles 140, 125 and 133, 216 tiles
  // 238, 180 and 194, 256 tiles 237, 232 and 226, 1,152 tiles 874, 875 and 960.  Just above a line the sharing below it is still
  // the better one, because the last wave is nearly empty: 80 tiles 139, 124 and 80, 320 tiles 346, 286 and 279.)
  const long long tiles = (long long)ceil_div(a.M, TM) * ceil_div(a.N, TN) * batch;
  if (tiles >= 2 * sm_count()) return launch_tile<1>(a, batch, s);
  if (2 * tiles >= sm_count()) return launch_tile<2>(a, batch, s);
  return launch_tile<8>(a, batch, s);
}

}  // namespace lmsf

// `batch` products in one launch: product b reads A + b * batch_a and W + b * batch_w and writes C + b * batch_c
// (elements).  The heads of one activation matrix are such a batch: batch_a = head size, lda = the row stride.
// in_dtype: type of A and W; out_dtype: type of C.  Leading dimensions in elements.  w_constant: W is a weight, which no kernel
// of the step writes; 0: W may have been written by the launch just before this one.
LMSF_API int lmsf_gemm_tn_simt_batched(void* C, const void* A, const void* W, int M, int N, int K, long long lda,
                                       long long ldw, long long ldc, int batch, long long batch_a, long long batch_w,
                                       long long batch_c, int in_dtype, int out_dtype, int w_constant, void* stream) {
  using namespace lmsf;
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (K <= 0) LMSF_REFUSE("gemm: K=%d must be positive", K);
  if (lda < K || ldw < K || ldc < N) LMSF_REFUSE("gemm: a leading dimension is smaller than its row");
  if (batch > 65535) LMSF_REFUSE("gemm: more than 65535 products in one launch");
  dim3 grid(ceil_div(N, BN), ceil_div(M, BM), batch);
  if (grid.y > 65535) LMSF_REFUSE("gemm: M=%d is too large for one launch", M);
  cudaStream_t s = (cudaStream_t)stream;
  const bool wide = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && batch_a % 4 == 0 && batch_w % 4 == 0 &&
                    (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
  if (in_dtype == LMSF_F32 && out_dtype == LMSF_F32 && wide && ceil_div(N, TN) <= 65535)
    return launch_f32(F32Args{(float*)C, (const float*)A, (const float*)W, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c,
                              w_constant ? 1 : 0}, batch, s);
  if (in_dtype == LMSF_F32 && out_dtype == LMSF_F32)
    gemm_tn_kernel<float, float><<<grid, 256, 0, s>>>((float*)C, (const float*)A, (const float*)W, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c);
  else if (in_dtype == LMSF_BF16 && out_dtype == LMSF_BF16)
    gemm_tn_kernel<bf16, bf16><<<grid, 256, 0, s>>>((bf16*)C, (const bf16*)A, (const bf16*)W, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c);
  else if (in_dtype == LMSF_BF16 && out_dtype == LMSF_F32)
    gemm_tn_kernel<bf16, float><<<grid, 256, 0, s>>>((float*)C, (const bf16*)A, (const bf16*)W, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c);
  else
    LMSF_REFUSE("gemm: unsupported dtype pair (in %d, out %d)", in_dtype, out_dtype);
  return LMSF_LAUNCH_STATUS();
}

LMSF_API int lmsf_gemm_tn_simt(void* C, const void* A, const void* W, int M, int N, int K, long long lda,
                               long long ldw, long long ldc, int in_dtype, int out_dtype, int w_constant, void* stream) {
  return lmsf_gemm_tn_simt_batched(C, A, W, M, N, K, lda, ldw, ldc, 1, 0, 0, 0, in_dtype, out_dtype, w_constant, stream);
}
