// attn_decode.cu — one kernel for the attention block of a decode step.
//
// For one new token per row it does, per (row, kv head), what the reference spreads over
// reshape/transpose, optional per-head RMSNorm (catgrad-llm/src/models/qwen3.rs:187-217),
// apply_rope_embedding (catgrad-llm/src/helpers.rs:202-221), repeat_kv (helpers.rs:147-161),
// the masked softmax(q k^T / sqrt(d)) v of catgrad-llm/src/models/llama.rs:97-108 and the
// cache append of catgrad-llm/src/legacy/models/utils.rs:210-228:
//
//   1. request this CTA's slice of cached keys and values (TMA, a tile of each per warp)
//      before anything else, then, while they fly, split the f32 qkv row, normalise / rotate
//      q and the new k, round them to bf16 (the cache precision) and append k, v to the cache;
//   2. the query heads that share the kv head are the rows of one 16-row MMA tile, so
//      q k^T and p v for 32 keys are a few mma.sync instructions per warp instead of
//      thousands of scalar FMAs; online softmax per head;
//   3. the slices of one (row, kv head) form a thread-block cluster: each pushes its partials
//      (max, sum, weighted values) to the CTA that finishes them, which merges them out of its own shared
//      memory into the bf16 output that the output projection reads.  No scratch in HBM, no second kernel.
//
// The whole block is latency-bound (a few MB per layer), so the design minimises dependent
// round trips and instruction count rather than bytes.

#include "attn_decode.cuh"
#include "kernels.h"
#include "mma.cuh"

namespace cg {

namespace {

constexpr int MAX_REP = ATTN_MAX_REP;

// one CTA per item; the slices of one (row, kv head) are one thread-block cluster
template <bool ROWS>
struct KernelEnv {
  __device__ __forceinline__ int tid() const { return threadIdx.x; }
  __device__ __forceinline__ void sync_cta() const { __syncthreads(); }
  __device__ __forceinline__ void sync_group() const {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  __device__ __forceinline__ uint32_t cluster_rank(int s) const { return (uint32_t)s; }
  // one item per CTA: partials are pushed into the finishing CTA's landing area
  static constexpr bool kPush = true;
  float* land;
  const CUtensorMap *map_k, *map_v;
  __device__ __forceinline__ float* landing() const { return land; }
  static constexpr bool kRows = ROWS;
  // The position is first + *step, or first alone.  (Held by value: no address of a kernel parameter is taken, whatever space
  // the parameters lie in.)
  const int64_t* step;
  int64_t first;
  __device__ __forceinline__ int64_t position() const { return first + (step ? *(const volatile int64_t*)step : 0); }
  // the projected row, and the position when it lives on the device, belong to the stream order
  __device__ __forceinline__ int64_t settle(int64_t) const {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return position();
  }
};

// What is reached by the tables and the counter on the device, before and behind the wait, and why it is in range: slot and
// pos0 have an entry per row, blockIdx.y < rows of them; a slot whose cache would end past cache_rows and a settled position outside
// [0, Tmax) raise the error word, are replaced by ones in range and append nothing; the early position is clamped.  Angles
// are [Tmax][rot_dims / 2] (rows) or [Tmax][D / 2], temperatures [Tmax], by position; biases [nh][ld_bias], read for live
// keys only, whose distance is 0 to the position.  A tile begins at a key below the position or the new one, so inside the cache; what
// of it lies past the cache's end reads as zeros, past the row's end is masked.  Landing areas: attn_dec_landing_bytes.
// (Four CTAs per SM leave 128 registers a thread: all that head sizes 128 and 256 use; the row form at 256 spills 8 bytes.)
template <int D, bool ROWS>
__global__ void __launch_bounds__(128, 4)
k_attn_dec(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, AttnDecArgs a, float scale) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = (uint32_t)__cvta_generic_to_shared(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  KernelEnv<ROWS> env;
  env.map_k = &map_k;
  env.map_v = &map_v;
  env.land = (float*)(smem + attn_dec_smem_bytes<D>());
  // Before the dependency wait: the first tiles of cached keys and values can be on the way
  // while the projection GEMM still runs.  What makes that sound: every writer of the device-side
  // position (the one-thread state kernel, in plain stream order; the arg-max kernel, after its
  // own dependency wait) stores a value v only after every kernel that wrote cache rows below v
  // has completed, so whatever value is visible here, the rows below it are complete.  The value
  // may be a step old; it is re-read after the wait and a changed value repeats the request.
  // (Row tables are copied in plain stream order before any kernel that reads them.)
  if constexpr (ROWS) {
    env.step = a.rows.step;
    env.first = a.rows.pos0[blockIdx.y];
  } else {
    env.step = a.pos_dev;
    env.first = a.pos_dev ? 0 : a.pos0;
  }
  int64_t pos_early = env.position();
  pos_early = pos_early < 0 ? 0 : (pos_early >= a.Tmax ? a.Tmax - 1 : pos_early);
  attn_dec_item<D>(a, scale, (int)blockIdx.x, (int64_t)blockIdx.y, (int)blockIdx.z, pos_early, smem, env);
}

template <int D, bool ROWS>
int launch(cg_ctx* c, const AttnDecArgs& args) {
  AttnDecArgs a = args;
  a.err = c->core->dev_err;
  CUtensorMap mk, mv;
  CG_TRY(tc::make_map(c, &mk, a.k_cache, a.cache_rows, D, D, attn_dec_keys(D)));
  CG_TRY(tc::make_map(c, &mv, a.v_cache, a.cache_rows, D, D, attn_dec_keys(D)));
  const size_t smem = 1024 + attn_dec_smem_bytes<D>() + (a.splits > 1 ? attn_dec_landing_bytes(a.nh / a.nkv, D, a.splits) : 0);
  static PerDeviceFlag configured_on;
  bool& configured = configured_on.at(c->core->device);
  if (!configured) {
    CG_CUDA(c, cudaFuncSetAttribute(k_attn_dec<D, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(1024 + attn_dec_smem_bytes<D>() + attn_dec_landing_bytes(MAX_REP, D, 16))));
    configured = true;
  }
  static PerDeviceFlag wide_on;
  bool& wide = wide_on.at(c->core->device);
  if (!wide && a.splits > 8) {
    CG_CUDA(c, cudaFuncSetAttribute(k_attn_dec<D, ROWS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    wide = true;
  }
  dim3 grid((unsigned)a.nkv, (unsigned)a.B, (unsigned)a.splits);
  const float scale = a.scale > 0.f ? a.scale : 1.0f / sqrtf((float)D);
  CG_CUDA(c, launch_kernel(c, k_attn_dec<D, ROWS>, grid, dim3(128), smem, a.splits, mk, mv, a, scale));
  CG_LAUNCHED(c);
  return CG_OK;
}

}  // namespace

// Context slices per (row, kv head): a power of two up to 16 (one cluster; above 8 is the non-portable size this GPU
// supports).  A slice keeps at least 128 keys at full context, one chunk per warp, and all CTAs together
// stay within two per SM: beyond that a CTA's fixed part (query preparation, merges) costs more than the
// shorter loop gives, unless a slice would have more than 256 keys; then three to four per SM, as many as fit, will do.
// But a cluster of 16 has to fit into one GPC, where head sizes above 64 leave two or three CTAs per SM: with more than some 20
// rows and kv heads (24 at head size 64) such clusters wait for one another.  Us per step of four layers with 8 / 16 slices, 2048 keys of
// 4200: 32 x 64 124 / 144; 24 x 128 201 / 223; 24 x 256 178 / 197; 20 x 128 142 / 146; 20 x 256 173 / 170; 24 x 64, 4096 keys 116 / 112.
// Ms per pass with 1 / 2 / 4 / 8 / 16 slices (the rule's choice in brackets):
//   8 rows x 8 kv heads, 640 keys, d 64 (128 steps of 16 layers)    106.2  102.0 [100.1] 101.9  119.0
//   32 x 8, 558 keys, d 128 (48 steps of 4 layers)                   66.1 [64.3]   65.2   67.6   74.3
//   1 x 8, 8200 keys, d 128 (8 steps of 4 layers)                    22.7   20.7   20.2   20.5  [20.1]
//   4 x 4, 2113 keys, d 256 (64 steps of 4 layers)                   42.0   36.6   33.7   32.5  [32.4]
//   8 x 4, 1073 keys, d 128, 8 heads each (48 steps of 4 layers)     38.6   37.9   37.5  [37.5]  38.4
int attn_dec_splits(int64_t Tmax, int64_t pairs, int d) {
  constexpr int64_t SMS = 148;
  int s = 1;
  const bool fits = pairs <= (d == 64 ? 24 : 20);  // in clusters of 16
  while (s < 16 && (int64_t)s * 128 < Tmax &&
         (pairs * s * 2 <= 2 * SMS || ((int64_t)s * 256 < Tmax && pairs * s * 2 <= 4 * SMS && (s < 8 || fits))))
    s *= 2;
  return s;
}

int k_launch_attn_dec(cg_ctx* c, const AttnDecArgs& a) {
  if (a.nkv <= 0 || a.nh % a.nkv || a.nh / a.nkv > MAX_REP)
    return fail(c, CG_ERR_UNSUPPORTED, "attention decode: query heads per kv head must be 1..8");
  if (a.d != 64 && a.d != 128 && a.d != 256) return fail(c, CG_ERR_UNSUPPORTED, "attention: head_dim must be 64, 128 or 256");
  if (a.B > 65535) return fail(c, CG_ERR_UNSUPPORTED, "attention: too many rows");
  if (!a.rows.rows && !a.pos_dev && a.pos0 >= a.Tmax) return fail(c, CG_ERR_SHAPE, "attention: KV cache capacity exceeded");
  if (a.B == 0) return CG_OK;
  if (a.cache_rows <= 0 || a.cache_rows > 2147483647ll) return fail(c, CG_ERR_UNSUPPORTED, "attention: more cache rows than a tile coordinate holds");
  if (!a.rows.rows && a.B * a.nkv * a.Tmax > a.cache_rows) return fail(c, CG_ERR_SHAPE, "attention: more rows than the KV cache holds");
  if (a.rows.rows) {
    switch (a.d) {
      case 64: return launch<64, true>(c, a);
      case 128: return launch<128, true>(c, a);
      default: return launch<256, true>(c, a);
    }
  }
  switch (a.d) {
    case 64: return launch<64, false>(c, a);
    case 128: return launch<128, false>(c, a);
    default: return launch<256, false>(c, a);
  }
}

}  // namespace cg
