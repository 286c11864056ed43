// What surrounds the expert gathers of a mixture-of-experts layer: the router's choices turned into
// slots, and the activation between the two gathers. Both are small; what they cost is launches (a
// dozen elementwise, sort and scan kernels before), so each is one.
#include "common.cuh"

namespace bn {
namespace {

constexpr int ROUTE_THREADS = 1024;
constexpr int64_t ROUTE_EXPERTS = 48 * 1024;  // counters of this many experts fit shared memory; more are counted in seg

// Slot g = choice g of the router, in token order: its expert (int32), input row g / k and its own
// number; with seg, the slots grouped by expert besides: expert e's are order[seg[e] .. seg[e + 1])
// (in no particular order: a slot's output does not depend on its neighbours). Ids outside 0 ..
// E - 1 are in no group. One block.
__global__ void __launch_bounds__(ROUTE_THREADS) route_kernel(const void *__restrict__ ids, int wide, int64_t G, int64_t k, int64_t E, uint32_t *__restrict__ ei, uint32_t *__restrict__ xi, uint32_t *__restrict__ iota, uint32_t *__restrict__ seg, uint32_t *__restrict__ order) {
  extern __shared__ uint32_t shared_counts[];
  const bool in_seg = E > ROUTE_EXPERTS;
  uint32_t *const counts = in_seg ? seg + 1 : shared_counts;  // [E], then running places: in the end, in seg, where the next expert's slots start
  __shared__ uint32_t warp_sum[32], carry;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  auto id = [&](int64_t g) { return wide ? (uint32_t)reinterpret_cast<const int64_t *>(ids)[g] : reinterpret_cast<const uint32_t *>(ids)[g]; };
  if (seg) {
    for (int64_t e = threadIdx.x; e < E; e += ROUTE_THREADS) counts[e] = 0;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
  }
  for (int64_t g = threadIdx.x; g < G; g += ROUTE_THREADS) {
    const uint32_t e = id(g);
    if (ei) ei[g] = e;
    if (xi) xi[g] = (uint32_t)(g / k);
    if (iota) iota[g] = (uint32_t)g;
    if (seg && e < E) atomicAdd(counts + e, 1u);
  }
  if (!seg) return;
  __syncthreads();
  for (int64_t e0 = 0; e0 < E; e0 += ROUTE_THREADS) {  // exclusive prefix sum
    const int64_t e = e0 + threadIdx.x;
    const uint32_t own = e < E ? counts[e] : 0u;
    uint32_t upto = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t n = __shfl_up_sync(BN_FULL, upto, d);
      if (lane >= (uint32_t)d) upto += n;
    }
    if (lane == 31) warp_sum[warp] = upto;
    __syncthreads();
    uint32_t before = carry;
    for (uint32_t w = 0; w < warp; w++) before += warp_sum[w];
    if (e < E) {
      counts[e] = before + upto - own;
      if (!in_seg) seg[e] = counts[e];
    }
    __syncthreads();
    if (threadIdx.x == ROUTE_THREADS - 1) carry = before + upto;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    if (in_seg) seg[0] = 0;
    else seg[E] = carry;
  }
  for (int64_t g = threadIdx.x; g < G; g += ROUTE_THREADS) {
    const uint32_t e = id(g);
    if (e < E) order[atomicAdd(counts + e, 1u)] = (uint32_t)g;
  }
}

__device__ __forceinline__ float silu_times(float g, float u) { return g / (1.0f + expf(-g)) * u; }

// h = silu(gate) * up, in fp32, one rounding to BF16. Two values a thread.
__global__ void __launch_bounds__(256) swiglu_kernel(const uint16_t *__restrict__ gate, const uint16_t *__restrict__ up, int64_t n, uint16_t *__restrict__ h, bool pairs) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the gather that made gate and up
  const int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 2;
  auto wide = [](uint32_t b) { return __uint_as_float(b << 16); };
  if (pairs && i + 1 < n) {
    const uint32_t g = *reinterpret_cast<const uint32_t *>(gate + i), u = *reinterpret_cast<const uint32_t *>(up + i);
    const uint32_t lo = f32_to_bf16_bits(silu_times(wide(g & 0xFFFFu), wide(u & 0xFFFFu))), hi = f32_to_bf16_bits(silu_times(wide(g >> 16), wide(u >> 16)));
    *reinterpret_cast<uint32_t *>(h + i) = lo | (hi << 16);
  } else {
    for (int64_t j = i; j < i + 2 && j < n; j++) h[j] = f32_to_bf16_bits(silu_times(wide(gate[j]), wide(up[j])));
  }
}

}  // namespace
}  // namespace bn

extern "C" int bn_moe_route(const void *ids, int ids64, int64_t G, int64_t k, int64_t E, uint32_t *ei, uint32_t *xi, uint32_t *iota, uint32_t *seg, uint32_t *order, void *stream) {
  if (G < 0 || k < 1 || E < 0 || (G && !ids) || (seg && G && !order)) return bn::fail(BN_ERR_ARG, "bn_moe_route: null pointer or bad size");
  if (G == 0 && !seg) return BN_OK;
  const size_t smem = seg && E <= bn::ROUTE_EXPERTS ? (size_t)E * 4 : 0;
  BN_CUDA(bn::allow_smem(bn::route_kernel, bn::ROUTE_EXPERTS * 4));
  bn::route_kernel<<<1, bn::ROUTE_THREADS, smem, (cudaStream_t)stream>>>(ids, ids64, G, k, E, ei, xi, iota, seg, order);
  return bn::launched("route_kernel");
}

extern "C" int bn_swiglu(const uint16_t *gate, const uint16_t *up, int64_t n, uint16_t *h, void *stream) {
  if (n < 0 || (n && (!gate || !up || !h))) return bn::fail(BN_ERR_ARG, "bn_swiglu: null pointer or negative size");
  if (n == 0) return BN_OK;
  const bool pairs = !((reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(up) | reinterpret_cast<uintptr_t>(h)) & 3);
  const int64_t blocks = (n + 511) / 512;
  if (blocks > 0x7FFFFFFF) return bn::fail(BN_ERR_ARG, "bn_swiglu: too many values");
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks), cfg.blockDim = dim3(256), cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = 1;
  BN_CUDA(cudaLaunchKernelEx(&cfg, bn::swiglu_kernel, gate, up, n, h, pairs));
  return bn::launched("swiglu_kernel");
}
