// out[T, I] = act(x Wg^T) * (x Wu^T) for many rows (bfloat16, float32 sums), W = [Wg; Wu] stacked along its rows: the gate and up
// products of a prompt and their activation in one kernel on the 5th-generation tensor cores.
//
// What bounds it: the tensor cores.  The product followed by an activation of its own writes gate and up to memory, reads them
// and writes their product: at 2,048 x 14,336 that is 37 us at 4.8 TB/s behind 323 us of product.
//
// Shape: a pair of CTAs (a cluster, cta_group::2) computes 256 rows x 128 features, that is an accumulator of 256 x 256: one CTA holds
// 128 rows of x; of W one CTA brings the 128 gate rows, the other the 128 up rows of the same features, so that a thread of
// the epilogue finds a row's gate and up values in its own lane of tensor memory.  K is walked in
// steps of 64 through a ring of stages (16 KB of x and 16 KB of W per CTA, tensor-map copies, 128-byte swizzle) whose barriers
// lie in the leading CTA; both halves of tensor memory (256 columns each) hold an accumulator, so that the epilogue of a tile runs
// beside the products of the next one.  The launch has one pair per two SMs, each taking tiles in turn; the tiles of up to 16
// blocks of rows follow one another over the features, so that the rows of x stay in L2 and a block of W is read by its
// neighbours at the same time.
//   warps 0-7  epilogue: a row a thread, each of two threads half of its columns (with four warps and expf it took longer than the
//              products at K = 2,048: 2,048 x 8,192 116 us, now 91)
//   warp 8     producer of this CTA's copies
//   warp 9     issues the products (the leading CTA's alone)
// Measured, cold weights, product and activation apart -> this kernel, by the power that is left to the device: K 4,096, I 14,336: 512
// rows 108 to 121 -> 95 to 109 us, 1,024 204 to 231 -> 165 to 188, 2,048 361 to 417 -> 302 to 351, 8,192 1,408 to 1,434 -> 1,163 to 1,354 (up
// to 1.65 PFLOP/s); K 2,048, I 8,192: 512 rows 37 to 39 -> 30 to 32, 2,048 131 to 144 -> 89 to 96, 8,192 464 to 512 -> 355.  At 2,048 x 14,336 the
// tensor cores are busy in 97 % of the cycles in which an SM works and in 87 % of the launch (the waves are 0.93 full).
// Every wait is bounded; a block that gives up raises error code 4.
#include "tc_common.cuh"

LMSF_DEFINE_LAST_ERROR(lmsf_gemm_gated_tc)

namespace lmsf {
namespace pairs {
using namespace tc;

constexpr int BM = 128, BF = 128, BK = 64;          // per CTA: rows of x and of W; k per stage
constexpr int kStages = 6;
constexpr int kSlab = BM * BK * 2;                  // 16 KB: x, and W
constexpr int kStageBytes = 2 * kSlab;
constexpr int kSmemBytes = kStages * kStageBytes + 1024;
constexpr int kEpilogue = 8;                        // warps of the epilogue: four rows' quarters x two halves of the columns
constexpr int kThreads = 32 * (kEpilogue + 2);
constexpr int kRaster = 16;                         // blocks of 256 tokens whose tiles follow one another

struct Args {
  bf16* out; long long ldo;
  int T, I, K, act;                                 // I: columns of out
  int m_tiles, f_tiles;
  int* error_flag;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t leader_addr(uint32_t local) {      // the same place in the leading CTA's shared memory
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(local));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void load_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t leader_bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(leader_bar) : "memory");
}
__device__ __forceinline__ void umma_pair(bool leader, uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nsetp.ne.b32 q, %5, 0;\n@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"((uint32_t)leader) : "memory");
}
__device__ __forceinline__ void commit_pair(bool leader, uint32_t bar) {      // arrives at this place in both CTAs
  asm volatile("{\n.reg .pred q;\n.reg .b16 m;\nmov.b16 m, 3;\nsetp.ne.b32 q, %1, 0;\n"
               "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n}\n"
               ::"r"(bar), "r"((uint32_t)leader) : "memory");
}
__device__ __forceinline__ void arrive_leader(uint32_t leader_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_bar) : "memory");
}
// as mbar_wait_f, for phases that another CTA of the cluster completes
__device__ __forceinline__ bool wait_cluster(uint32_t bar, uint32_t parity, volatile int* failed) {
  uint32_t done = 0;
  for (int it = 0; it < kWaitLimit && !done; ++it) {
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\nselp.b32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (!done && *failed) return false;
  }
  if (!done) *failed = 1;
  return done != 0;
}

// silu by the special-function unit's 2^x and 1/x: within a few 2^-23 times (1 + |g|) of the value for g above -87.3, which is rounded to
// bfloat16 next (gate and up are not rounded before, as they are where the activation is a kernel of its own); below, where 1 + e^-g
// passes 2^126 and its reciprocal is flushed, it is 0 for a value of at most 9e-37 in size
__device__ __forceinline__ float act_apply(float g, int act) {
  if (act == 0) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(g * -1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return g * r;
  }
  const float k = 0.7978845608028654f;
  return 0.5f * g * (1.0f + tanhf(k * (g + 0.044715f * g * g * g)));
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gated_kernel(const Args a, const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * kStages + 4];
  __shared__ uint32_t tmem_base_mem;
  __shared__ volatile int failed_mem;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank();
  const uint32_t smem = (smem_addr(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar0 = smem_addr(&bars[0]);
  auto full = [&](int s) { return bar0 + 8u * s; };                         // the leader's: 64 KB of both CTAs' copies
  auto empty = [&](int s) { return bar0 + 8u * (kStages + s); };            // in each CTA: the products that read the stage are done
  auto acc_full = [&](int b) { return bar0 + 8u * (2 * kStages + b); };     // in each CTA
  auto acc_empty = [&](int b) { return bar0 + 8u * (2 * kStages + 2 + b); };// the leader's: the epilogue's warps of both CTAs
  volatile int* failed = &failed_mem;
  pdl_launch_dependents();
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 2 * kEpilogue); }
    failed_mem = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kEpilogue + 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_mem)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                               // both CTAs' barriers are set up
  tc_fence_after();
  const uint32_t tmem = tmem_base_mem;
  const int k_steps = (a.K + BK - 1) / BK;
  const int n_tiles = a.m_tiles * a.f_tiles, n_pairs = gridDim.x >> 1, pair = blockIdx.x >> 1;
  // tile t: bands of kRaster blocks of tokens; inside a band the blocks of tokens run fastest
  auto place = [&](int t, int& m, int& f) {
    const int per_band = kRaster * a.f_tiles, band = t / per_band, in = t - band * per_band;
    const int wide = min(kRaster, a.m_tiles - band * kRaster);
    f = in / wide;
    m = band * kRaster + in - f * wide;
  };
  pdl_wait();

  if (warp == kEpilogue) {
    // ---------------------------------------------------------------- copies
    const bool one = elect_one();
    int slot = 0, round = 0, issued = 0;
    bool ok = true;
    for (int t = pair; t < n_tiles && ok; t += n_pairs) {
      int m, f;
      place(t, m, f);
      const int row = m * 2 * BM + rank * BM, w_row = (rank ? a.I : 0) + f * BF;
      for (int ks = 0; ks < k_steps; ++ks) {
        if (round > 0 && !wait_cluster(empty(slot), (round - 1) & 1, failed)) { ok = false; break; }
        if (one) {
          const uint32_t st = smem + slot * kStageBytes, bar = leader_addr(full(slot));
          if (rank == 0) mbar_arrive_expect_tx(full(slot), 2 * kStageBytes);
          load_pair(st, &x_map, ks * BK, row, bar);
          load_pair(st + kSlab, &w_map, ks * BK, w_row, bar);
        }
        ++issued;
        if (++slot == kStages) { slot = 0; ++round; }
      }
    }
    // The ring once more: the products' arrivals on this CTA's `empty` barriers for the last stages.  The leader's tensor core sends
    // them here on its own, so neither the last accumulator's arrival nor the cluster's barrier says that they have come, and a CTA
    // that ends before they do leaves shared memory that is still written.
    for (int k = max(0, issued - kStages); k < issued && ok; ++k) ok = wait_cluster(empty(k % kStages), (uint32_t)((k / kStages) & 1), failed);
    // after a failure: this CTA's copies land before it ends (the leader's barriers count both CTAs'; the peer's are let land by
    // the wait at the cluster's last barrier, which the leader reaches behind this)
    __syncwarp();
    if (*failed && rank == 0)
      for (int k = max(0, issued - kStages); k < issued; ++k) mbar_wait_drain(full(k % kStages), (uint32_t)((k / kStages) & 1));
  } else if (warp == kEpilogue + 1) {
    // ---------------------------------------------------------------- products
    if (rank == 0) {
      constexpr uint32_t idesc = instr_desc(2 * BM, 2 * BF, 0);
      const bool leader = elect_one();
      int slot = 0, round = 0, n = 0;
      bool ok = true;
      for (int t = pair; t < n_tiles && ok; t += n_pairs, ++n) {
        const int b = n & 1;
        if (n >= 2 && !wait_cluster(acc_empty(b), ((n >> 1) - 1) & 1, failed)) break;
        tc_fence_after();
        for (int ks = 0; ks < k_steps; ++ks) {
          if (!wait_cluster(full(slot), round & 1, failed)) { ok = false; break; }
          tc_fence_after();
          const uint32_t st = smem + slot * kStageBytes;
          const uint64_t da = smem_desc(st, 16, 1024), dw = smem_desc(st + kSlab, 16, 1024);
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            umma_pair(leader, tmem + b * 256, da + (uint64_t)((kk * 32) >> 4), dw + (uint64_t)((kk * 32) >> 4), idesc, (ks > 0 || kk > 0) ? 1u : 0u);
          commit_pair(leader, empty(slot));
          if (++slot == kStages) { slot = 0; ++round; }
        }
        if (ok) commit_pair(leader, acc_full(b));
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int quarter = warp & 3, half = warp >> 2;  // a warp reads the lanes of its quarter of tensor memory
    int n = 0;
    for (int t = pair; t < n_tiles; t += n_pairs, ++n) {
      const int b = n & 1;
      if (!wait_cluster(acc_full(b), (n >> 1) & 1, failed)) break;
      tc_fence_after();
      int m, f;
      place(t, m, f);
      const int row = m * 2 * BM + rank * BM + quarter * 32 + lane;
      const bool live = row < a.T;
      const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + b * 256;
      auto free_accumulator = [&]() {               // everything is in registers: the accumulator may be written again
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_leader(leader_addr(acc_empty(b)));
      };
      const int f0 = f * BF;
      bf16* dst = a.out + (size_t)row * a.ldo + f0;
#pragma unroll
      for (int cc = 0; cc < BF / 2; cc += 32) {
        const int c = half * (BF / 2) + cc;
        __syncwarp();
        float g[32], u[32];
        tmem_ld32_issue(acc + c, g);
        tmem_ld32_issue(acc + BF + c, u);
        tmem_wait_ld();
        if (cc == BF / 2 - 32) free_accumulator();
        if (!live) continue;
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          if (f0 + c + j < a.I) {                 // I is a multiple of 8
            uint32_t v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int i = j + 2 * e;
              v[e] = pack2(act_apply(g[i], a.act) * u[i], act_apply(g[i + 1], a.act) * u[i + 1]);
            }
            *reinterpret_cast<uint4*>(dst + c + j) = make_uint4(v[0], v[1], v[2], v[3]);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                               // neither CTA's shared or tensor memory is used any more
  tc_fence_after();
  if (*failed && tid == 0 && a.error_flag) atomicExch(a.error_flag, 4);
  if (warp == kEpilogue + 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// a [rows][K] matrix for the copy engine, boxes of 64 x 128; made for every call: nothing is kept by an address
static bool make_map(CUtensorMap* m, const void* p, long long rows, int K, long long ld) {
  EncodeTiledFn encode = encode_tiled_fn();
  if (!encode) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {BK, BM};
  const cuuint32_t elem_strides[2] = {1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace pairs
}  // namespace lmsf

// x: [T][ldx], W: [2 I][K] (gate rows, then up rows), out: [T][ldo]; act 0 silu, 1 gelu (tanh form).
LMSF_API int lmsf_gemm_gated_tc(void* out, long long ldo, const void* x, long long ldx, const void* W, int T, int I, int K, int act,
                                int* error_flag, void* stream) {
  using namespace lmsf;
  using namespace lmsf::pairs;
  if (T <= 0) return 0;
  if (K < 8 || K % 8 || I < 8 || I % 8 || ldx % 8 || ldx < K || ldo % 8 || ldo < I || ((uintptr_t)out | (uintptr_t)x | (uintptr_t)W) % 16)
    LMSF_REFUSE("gemm_gated_tc: K=%d, I=%d and the strides must be multiples of 8 and the operands 16-byte aligned", K, I);
  if (act != 0 && act != 1) LMSF_REFUSE("gemm_gated_tc: unknown activation code %d", act);
  Args a{(bf16*)out, ldo, T, I, K, act, ceil_div(T, 2 * BM), ceil_div(I, BF), error_flag};
  if ((long long)a.m_tiles * a.f_tiles > (1 << 30)) LMSF_REFUSE("gemm_gated_tc: %d rows are too many", T);
  CUtensorMap xm, wm;
  if (!make_map(&xm, x, T, K, ldx) || !make_map(&wm, W, 2ll * I, K, K)) LMSF_REFUSE("gemm_gated_tc: cuTensorMapEncodeTiled refused the operands' geometry");
  // asked and set for every call: both belong to the current device, of which a process may use several
  int dev = 0, n_sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n_sms < 2)
    LMSF_REFUSE("gemm_gated_tc: the device's number of SMs cannot be read");
  const cudaError_t e = cudaFuncSetAttribute(gated_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  if (e != cudaSuccess) return (int)e;
  const int tiles = a.m_tiles * a.f_tiles, pairs = tiles < n_sms / 2 ? tiles : n_sms / 2;
  return launch_pdl(gated_kernel, dim3(2 * pairs), dim3(kThreads), kSmemBytes, (cudaStream_t)stream, a, xm, wm);
}
