// hs_kernels.cu -- the per-groom kernels: step, init, layout transposes.
#include <algorithm>
#include <type_traits>

#include "hs_internal.h"
#include "hs_lanes.cuh"
#include "hs_step.cuh"
#include "hs_stream.cuh"
#include "hs_tmem.cuh"

namespace hs {

namespace {

constexpr int kStepBlock = 64;

// Overlapped frames (programmatic dependent launch). A groom's frames are
// back-to-back kernels on one stream; launched by launch_overlapped, a
// frame's blocks may become resident while the previous kernel's last
// blocks still run: each block signals at its start that the next kernel
// may be scheduled (frame_release), does the set-up that touches no
// simulation state (spheres into shared memory, tensor-memory allocation),
// then waits in frame_acquire until the previous kernel has completed and
// its writes are visible, before its first load of the state. Launched
// the ordinary way, both are no-ops.
__device__ __forceinline__ void frame_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void frame_acquire() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... Params, typename... Args>
cudaError_t launch_overlapped(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                              Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Copies the groom's spheres and overlap masks from the kernel parameters
// into shared memory (constant indices only, so the parameter block is
// never copied to local memory). Ends with a barrier.
__device__ __forceinline__ SphereSet stage_spheres(const FrameConst& fc, float4* s_c, float* s_r2, uint32_t* s_adj) {
#pragma unroll
  for (int k = 0; k < HS_MAX_SPHERES; ++k) {
    if (threadIdx.x == k && k < fc.nspheres) {
      s_c[k] = fc.spheres[k];
      s_r2[k] = fc.r2[k];
      s_adj[k] = fc.adj[k];
    }
  }
  __syncthreads();
  return SphereSet{s_c, s_r2, s_adj, fc.nspheres};
}

// Velocity slots of the plain step: registers up to 16 points per strand,
// shared memory above (keeps the register file for the positions).
template <int CAP>
struct PlainVsmem {
  static constexpr bool value = CAP > 16;
};

// FAST (every kernel below): the groom's FAST contract, a kernel of its own
// (no code of the other contract in it).
// Reference mode is held to 80 registers (the frame's constants of 8 points
// spill 88 bytes), so that 11 blocks fit an SM rather than 10: 100,003
// strands x 8 alone 26.5 -> 21.2 us (their 1,563 blocks are then one wave),
// three such grooms in turn 14.9 -> 14.4 us.
// MANY: the DFTL push-out among many spheres (strand_frame_regs_dftl).
template <int CAP, bool REF, bool FAST, bool MANY>
__global__ void __launch_bounds__(kStepBlock, REF ? 11 : 0) k_step(GroomView g, FrameConst fc) {
  extern __shared__ float4 s_vel[];  // per-thread velocity rows, when in shared memory
  __shared__ float4 s_c[HS_MAX_SPHERES];
  __shared__ float s_r2[HS_MAX_SPHERES];
  __shared__ uint32_t s_adj[HS_MAX_SPHERES];
  frame_release();
  const SphereSet S = stage_spheres(fc, s_c, s_r2, s_adj);
  frame_acquire();
  const uint32_t s = blockIdx.x * kStepBlock + threadIdx.x;
  if constexpr (REF) strand_frame_ref<CAP, PlainVsmem<CAP>::value>(fc, S, g, s, s < g.nstrands, s_vel, threadIdx.x);
  else
    strand_frame_regs_dftl<CAP, PlainVsmem<CAP>::value, FAST, MANY>(fc, S, g, s, s < g.nstrands, s_vel, threadIdx.x);
}

template <int CAP, bool REF, bool FAST, bool MANY = false>
cudaError_t launch_step_cap(const GroomView& g, const FrameConst& fc, cudaStream_t st) {
  const unsigned grid = (g.nstrands + kStepBlock - 1) / kStepBlock;
  const size_t smem = PlainVsmem<CAP>::value ? vslot_bytes<CAP>(kStepBlock) : 0;
  return launch_overlapped(k_step<CAP, REF, FAST, MANY>, grid, kStepBlock, smem, st, g, fc);
}

bool fast_frame(const FrameConst& fc) { return fc.mode == HS_MODE_DFTL && fc.contract == HS_CONTRACT_FAST; }

template <int CAP>
cudaError_t launch_step_mode(const GroomView& g, const FrameConst& fc, cudaStream_t st) {
  if (fc.mode == HS_MODE_REFERENCE) return launch_step_cap<CAP, true, false>(g, fc, st);
  if (fc.nspheres > kFewSpheres)
    return fast_frame(fc) ? launch_step_cap<CAP, false, true, true>(g, fc, st)
                          : launch_step_cap<CAP, false, false, true>(g, fc, st);
  return fast_frame(fc) ? launch_step_cap<CAP, false, true>(g, fc, st) : launch_step_cap<CAP, false, false>(g, fc, st);
}

// Streaming form (hs_stream.cuh): state in shared memory, one runtime loop
// per pass, any point count. One warp per block: the shared state is what
// bounds residency, and single-warp blocks pack it tightest.
constexpr int kStreamBlock = 32;

template <bool REF, bool FAST>
__global__ void __launch_bounds__(kStreamBlock) k_step_stream(GroomView g, FrameConst fc) {
  extern __shared__ float4 s_state[];  // X then V, each [npoints][kStreamBlock]
  __shared__ float4 s_c[HS_MAX_SPHERES];
  __shared__ float s_r2[HS_MAX_SPHERES];
  __shared__ uint32_t s_adj[HS_MAX_SPHERES];
  frame_release();
  const SphereSet S = stage_spheres(fc, s_c, s_r2, s_adj);
  frame_acquire();
  const uint32_t s = blockIdx.x * kStreamBlock + threadIdx.x;
  float4* Xs = s_state + threadIdx.x;
  float4* Vs = s_state + g.npoints * kStreamBlock + threadIdx.x;
  strand_frame_stream<REF, XShared4, VShared, kCachedSpheres, false, false, FAST>(
      fc, S, g, s, s < g.nstrands, XShared4{Xs, kStreamBlock}, VShared{Vs, kStreamBlock});
}

// Streaming form with the velocities in tensor memory (hs_tmem.cuh): a
// block is 4 warps, one per TMEM lane quadrant; shared memory holds the
// positions only, 12 bytes a point (the rest lengths ride in the w of the
// TMEM velocity slots).
constexpr int kTmemBlock = 128;

// MANY: the push-out's form for grooms among many spheres (push_seg). P:
// pairs of substeps at once (step_pairs, WavePass).
template <bool REF, bool MANY, int P, bool FAST>
__global__ void __launch_bounds__(kTmemBlock, P == 2 ? 2 : 4) k_step_stream_tmem(GroomView g, FrameConst fc) {
  extern __shared__ float4 s_pos[];  // positions, compact: float2 (x, y) then float z, each [npoints][kTmemBlock]
  __shared__ float4 s_c[HS_MAX_SPHERES];
  __shared__ float s_r2[HS_MAX_SPHERES];
  __shared__ uint32_t s_adj[HS_MAX_SPHERES];
  __shared__ uint32_t s_taddr;
  frame_release();
  const SphereSet S = stage_spheres(fc, s_c, s_r2, s_adj);
  const uint32_t warp = threadIdx.x / 32;
  const uint32_t ncols = tmem::cols_for(g.npoints);
  if (warp == 0) {
    tmem::alloc(&s_taddr, ncols);
    tmem::relinquish();
  }
  tmem::fence_before_sync();
  __syncthreads();
  tmem::fence_after_sync();
  frame_acquire();
  const uint32_t base = s_taddr;
  const VTmem V{base + ((warp * 32u) << 16)};
  const uint32_t s = blockIdx.x * kTmemBlock + threadIdx.x;
  float2* xy = reinterpret_cast<float2*>(s_pos);
  float* z = reinterpret_cast<float*>(xy + g.npoints * kTmemBlock);
  const XShared3 X{xy + threadIdx.x, z + threadIdx.x, kTmemBlock};
  strand_frame_stream<REF, XShared3, VTmem, 8, true, MANY, FAST, P, P == 1 ? 4 : 8>(fc, S, g, s, s < g.nstrands, X, V);
  tmem::fence_before_sync();
  __syncthreads();
  tmem::fence_after_sync();
  if (warp == 0) tmem::dealloc(base, ncols);
}

// Blocks of the tensor-memory step resident on one SM are bounded by its
// 512 TMEM columns as well as by shared memory: the dynamic shared memory
// is padded so that shared memory is the tighter bound, and no block waits
// in its allocation.
size_t tmem_step_smem(uint32_t npoints) {
  const int sm_smem = device_attribute(cudaDevAttrMaxSharedMemoryPerMultiprocessor, 228 * 1024);
  const size_t need = (sizeof(float2) + sizeof(float)) * npoints * kTmemBlock;
  const size_t blocks_by_tmem = 512 / tmem::cols_for(npoints);
  const size_t per_block = static_cast<size_t>(sm_smem) / blocks_by_tmem + 1;  // one more block would not fit
  const size_t fixed = 1024 + 3 * 1024;  // reserved + static (spheres, masks, TMEM slot), rounded up
  return std::max(need, per_block > fixed ? per_block - fixed : need);
}

// Pairs of substeps a DFTL groom runs at once. They pay where schedulers wait
// on chain links, and where sphere tests run two-wide: less than a wave of
// warps (16 an SM, 8 for more than 32 points), longer strands, more spheres.
// Among more than 8 spheres one substep at a time goes through flagged spheres
// only (push_seg), which pairs do not: among 11 to 16 that is the faster form
// up to 32 points; further on pairs pay again, more and more. An odd substep
// is left over and changes form: it takes the gain away but for the most
// spheres. Grooms in turn on streams of their own share the SMs, one alone
// does not: the lines lie where both gain, or one gains and the other loses
// less. Single pass against one pair / two pairs, us a frame, 8 substeps
// unless S is given (EXACT; three grooms in turn, hair settled among the
// spheres):
//   half a wave       23,347 x 24 among 7 spheres 31.8 / 29.6 (FAST 27.6 /
//                     27.0), x 28 (S 5) 33.1 / 27.5; among 12 33.1 / 38.0,
//                     among 24 84.7 / 62.0; x 16 among 32 70.8 / 47.6
//   a wave            76,267 x 24 among 7 48.9 / 50.1, among 24 82.2 / 94.0;
//                     x 28 (S 5) among 7 40.7 / 49.8, among 16 47.4 / 70.3; x
//                     32 among 32 217 / 165, S 5 126 / 128; 50,585 x 23 among
//                     7 (S 5) 33.0 / 32.7
//   more than 32      25,292 x 36 among 4 33.1 / 31.9 / 32.1, x 64 59.6 / 55.2
//     points          / 53.6; 11,673 x 64 among 12 (S 5) 45.5 / 63.2 / 51.9;
//                     116,736 x 36 among 4 123 / 123 / 129, among 16 166 / 195
//                     / 164, among 24 (S 5) 192 / 256 / 215; x 64 among 4 (S
//                     5) 151 / 154 / 160, among 32 717 / 687 / 567, S 5 461 /
//                     481 / 423
//   one sphere        x 64 315 / 275 / 282 (a head: every strand is near it);
//                     50,585 x 32 53.7 / 53.1
//   none              x 64 176 / 169 / 158; 25,292 x 36 22.6 / 24.3 / 23.5
int step_pairs(const GroomView& g, const FrameConst& fc) {
  if (fc.iterations != 1 || fc.substeps < 2) return 0;
  const uint32_t sms = static_cast<uint32_t>(device_attribute(cudaDevAttrMultiProcessorCount, 152));
  const uint32_t tiles = (g.nstrands + 31) / 32;
  const int spheres = fc.nspheres;
  const bool even = fc.substeps % 2 == 0;
  const bool half = tiles <= 8u * sms;  // half a wave up to 32 points, a wave above
  if (g.npoints > 32) {
    if (spheres == 0) return g.npoints > 48 ? 2 : 0;
    if (spheres == 1) return 1;
    if (spheres <= kFewSpheres) return half ? 1 : (even && g.npoints > 48 ? 2 : 0);
    return even || spheres <= 12 || spheres > 24 || g.npoints > 48 ? 2 : 0;
  }
  const bool most = tiles <= 12u * sms, wave = tiles <= 16u * sms, fast = fast_frame(fc);
  if (!even) return spheres > 24 && most && g.npoints >= (half ? 12u : 16u) ? 1 : 0;
  if (spheres > 24) return wave && g.npoints >= 12 ? 1 : 0;
  if (spheres > 20) return most && g.npoints >= 16 ? 1 : 0;
  if (g.npoints < 20 || !(fast ? half : most)) return 0;
  if (spheres > 16) return half && !fast ? 1 : 0;
  return spheres >= (fast ? 6 : 4) && spheres <= 10 ? 1 : 0;
}

using StepKernel = void (*)(GroomView, FrameConst);
template <bool FAST>
StepKernel dftl_step_tmem(bool many, int pairs) {
  if (pairs == 2) return k_step_stream_tmem<false, false, 2, FAST>;
  if (pairs == 1) return k_step_stream_tmem<false, false, 1, FAST>;
  return many ? k_step_stream_tmem<false, true, 0, FAST> : k_step_stream_tmem<false, false, 0, FAST>;
}
StepKernel dftl_step_tmem(bool many, int pairs, bool fast) {
  return fast ? dftl_step_tmem<true>(many, pairs) : dftl_step_tmem<false>(many, pairs);
}

cudaError_t launch_step_stream_tmem(const GroomView& g, const FrameConst& fc, cudaStream_t st) {
  const unsigned grid = (g.nstrands + kTmemBlock - 1) / kTmemBlock;
  const size_t smem = tmem_step_smem(g.npoints);
  static std::atomic<uint64_t> optin{0};
  once_per_device(optin, [] {
    const int bytes = 200 * 1024;
    for (const bool fast : {false, true})
      for (const bool many : {false, true})
        for (const int pairs : {0, 1, 2})
          cudaFuncSetAttribute(dftl_step_tmem(many, pairs, fast), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    cudaFuncSetAttribute(k_step_stream_tmem<true, false, 0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  });
  if (fc.mode == HS_MODE_REFERENCE)
    return launch_overlapped(k_step_stream_tmem<true, false, 0, false>, grid, kTmemBlock, smem, st, g, fc);
  return launch_overlapped(dftl_step_tmem(fc.nspheres > kFewSpheres, step_pairs(g, fc), fast_frame(fc)), grid, kTmemBlock,
                           smem, st, g, fc);
}

// Lane groups (hs_lanes.cuh): a block of K warps per 32-strand tile, the
// tile's starting state in shared memory ([npoints][32] positions, then
// velocities). Register cap 128 (16 warps a SM). MANY: the push-out's form
// for grooms among many spheres (push_seg), where a strand reaches a dozen of
// them: us a frame without -> with, 8 substeps, EXACT, 2,858 x 41 among 18
// 25.1 -> 15.7, 4,096 x 64 among 32 59 -> 39, 8,192 x 24 among 32 37 -> 35.
template <int K, bool FAST, bool MANY>
__global__ void __launch_bounds__(K * 32, 16 / K) k_step_lanes(GroomView g, FrameConst fc) {
  extern __shared__ float4 s_state[];
  __shared__ float4 s_c[HS_MAX_SPHERES];
  __shared__ float s_r2[HS_MAX_SPHERES];
  __shared__ uint32_t s_adj[HS_MAX_SPHERES];
  __shared__ TileStats s_ts[32];
  frame_release();
  const SphereSet S = stage_spheres(fc, s_c, s_r2, s_adj);
  frame_acquire();
  tile_frame_lanes<K, FAST, MANY>(fc, S, g, blockIdx.x, s_state, s_state + g.npoints * 32, s_ts);
}

template <int K>
cudaError_t launch_step_lanes_k(const GroomView& g, const FrameConst& fc, cudaStream_t st) {
  const unsigned grid = (g.nstrands + 31) / 32;
  const size_t smem = 2 * sizeof(float4) * 32 * g.npoints;
  static const StepKernel kernels[2][2] = {{k_step_lanes<K, false, false>, k_step_lanes<K, false, true>},
                                         {k_step_lanes<K, true, false>, k_step_lanes<K, true, true>}};
  static std::atomic<uint64_t> optin{0};
  once_per_device(optin, [] {
    const int bytes = 2 * static_cast<int>(sizeof(float4)) * 32 * HS_MAX_POINTS_PER_STRAND;
    for (const auto& contract : kernels)
      for (const StepKernel k : contract) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  });
  const StepKernel k = kernels[fast_frame(fc) ? 1 : 0][fc.nspheres > kFewSpheres ? 1 : 0];
  return launch_overlapped(k, grid, K * 32, smem, st, g, fc);
}

cudaError_t launch_step_lanes(const GroomView& g, const FrameConst& fc, cudaStream_t st) {
  switch (lane_group(fc.mode, fc.substeps, fc.iterations)) {
    case 2: return launch_step_lanes_k<2>(g, fc, st);
    case 4: return launch_step_lanes_k<4>(g, fc, st);
    case 8: return launch_step_lanes_k<8>(g, fc, st);
    case 16: return launch_step_lanes_k<16>(g, fc, st);
    default: return cudaErrorNotSupported;
  }
}

// Point counts the plain step runs with its velocities in tensor memory
// (all that take the streaming form).
bool plain_uses_tmem(const GroomView& g) { return g.npoints > 8 && g.npoints <= HS_MAX_POINTS_PER_STRAND; }

cudaError_t launch_step_stream(const GroomView& g, const FrameConst& fc, cudaStream_t st) {
  if (plain_uses_tmem(g)) return launch_step_stream_tmem(g, fc, st);
  const unsigned grid = (g.nstrands + kStreamBlock - 1) / kStreamBlock;
  const size_t smem = 2 * sizeof(float4) * g.npoints * kStreamBlock;
  // 64 points x 32 threads x 2 arrays = 64 KB: above the default 48 KB.
  static std::atomic<uint64_t> optin{0};
  once_per_device(optin, [] {
    const int bytes = 2 * static_cast<int>(sizeof(float4)) * HS_MAX_POINTS_PER_STRAND * kStreamBlock;
    cudaFuncSetAttribute(k_step_stream<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    cudaFuncSetAttribute(k_step_stream<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    cudaFuncSetAttribute(k_step_stream<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  });
  if (fc.mode == HS_MODE_REFERENCE) {
    return launch_overlapped(k_step_stream<true, false>, grid, kStreamBlock, smem, st, g, fc);
  } else if (fast_frame(fc)) {
    return launch_overlapped(k_step_stream<false, true>, grid, kStreamBlock, smem, st, g, fc);
  } else {
    return launch_overlapped(k_step_stream<false, false>, grid, kStreamBlock, smem, st, g, fc);
  }
}

}  // namespace

namespace {

// Hair::init_simulation (src/fx/hair.cc:262-288), one thread per strand.
__global__ void k_init(GroomView g, InitArgs a, float4* root_rest) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= g.nstrands) return;
  const V3 r = v3(a.roots[3 * s], a.roots[3 * s + 1], a.roots[3 * s + 2]);
  const V3 nrm = v3(a.normals[3 * s], a.normals[3 * s + 1], a.normals[3 * s + 2]);
  const float u = hash_u01(a.length_key, a.strand_base + g.order[s]);  // the caller's index
  // rv = 1 + jitter * (1 - 2u)   (src/fx/hair.cc:268-270)
  const float rv = __fadd_rn(1.0f, __fmul_rn(a.length_jitter, __fsub_rn(1.0f, __fmul_rn(2.0f, u))));
  const int n = static_cast<int>(g.npoints);
  if (a.length_rule == HS_LENGTH_REFERENCE) {
    const float scale_offset = __fdiv_rn(a.max_length, static_cast<float>(n));
    float last = 0.0f;
    for (int i = 0; i < n; ++i) {
      const float offset = __fmul_rn(__fmul_rn(static_cast<float>(i), scale_offset), rv);
      const V3 q = add(r, mul(offset, nrm));
      g.pos[static_cast<size_t>(i) * g.stride + s] = make_float4(q.x, q.y, q.z, __fsub_rn(offset, last));
      g.vel[static_cast<size_t>(i) * g.stride + s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      last = offset;
    }
  } else {
    const float L = a.lengths ? a.lengths[s] : __fmul_rn(a.max_length, rv);
    const float seg = __fdiv_rn(L, static_cast<float>(n - 1));
    for (int i = 0; i < n; ++i) {
      const float offset = __fmul_rn(static_cast<float>(i), seg);
      const V3 q = add(r, mul(offset, nrm));
      g.pos[static_cast<size_t>(i) * g.stride + s] = make_float4(q.x, q.y, q.z, i == 0 ? 0.0f : seg);
      g.vel[static_cast<size_t>(i) * g.stride + s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }
  if (root_rest) root_rest[s] = make_float4(r.x, r.y, r.z, 0.0f);
}

// Transposes between strand-major (s*N + i) and [point][strand] (i*stride + s).
// A block moves 32 strands: their N float4 are contiguous in strand-major
// order, and each point row of 32 strands is 512 contiguous bytes.
// `order` (the caller's index of each stored strand) places stored strand s
// at strand-major row order[s]: the outside sees the caller's order.
constexpr int kTileStrands = 32;

// C: floats a point in `out`: 4, or 3 for (x, y, z) alone. Bound by memory
// latency (a block is one round of loads, a barrier, one of stores), so the
// strands' places are loaded with their points, not after the barrier; no
// index is divided by N, and tile rows are an odd number of float4, so that
// the eight strands of a 128-bit store phase fall in different banks. A warp
// writes `per` strands at a time (a power of two; one above 16 points).
// Before (places after the barrier, t / N per point, rows of N + 1): 50,021
// strands x 23 10.5 -> 7.9 us, 65,536 x 16 8.3 -> 7.4, 262,144 x 32 58 -> 52
// (268 MB moved, 40 us at the copy bandwidth). Blocks of 4 warps up to 12
// points a strand, of 8 above (4 against 8 warps, 100,003 x 9: 6.3 against
// 8.3 us; 50,021 x 23: 8.3 against 7.7; 20,000 x 64: 9.4 against 8.4). Rows handed to the copy engine: 47 us for 262,144 x 32, but 8.3 for
// 50,021 x 23 and 5.3 against 4.2 for 4,096 x 16.
template <int C>
__global__ void __launch_bounds__(256) k_to_strand_major(const float4* __restrict__ soa, float* __restrict__ out,
                                                         const uint32_t* __restrict__ order, uint32_t nstrands,
                                                         uint32_t npoints, uint32_t stride, uint32_t row, uint32_t per) {
  extern __shared__ float4 tile[];  // [kTileStrands][row]
  using Elem = typename std::conditional<C == 4, float4, float>::type;
  const uint32_t s0 = blockIdx.x * kTileStrands, lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const uint32_t ns = min(static_cast<uint32_t>(kTileStrands), nstrands - s0);
  const uint32_t place = lane < ns ? order[s0 + lane] : 0u;
  if (lane < ns) {
    const float4* const from = soa + s0 + lane;
#pragma unroll 4
    for (uint32_t i = warp; i < npoints; i += blockDim.x / 32) tile[lane * row + i] = from[static_cast<size_t>(i) * stride];
  }
  __syncthreads();
  const uint32_t elems = C == 4 ? npoints : 3 * npoints, warps = blockDim.x / 32;
  const auto put = [&](uint32_t sl, uint32_t to, uint32_t e) {
    const float4* const r = tile + sl * row;
    Elem* const o = reinterpret_cast<Elem*>(out) + static_cast<size_t>(to) * elems;
    if constexpr (C == 4) o[e] = r[e];
    else o[e] = reinterpret_cast<const float*>(r)[e + e / 3];
  };
  if (per == 1) {
#pragma unroll 2
    for (uint32_t sl = warp; sl < ns; sl += warps) {
      const uint32_t to = __shfl_sync(0xffffffffu, place, sl);
      for (uint32_t e = lane; e < elems; e += 32) put(sl, to, e);
    }
  } else {  // elems <= 32 / per
    const uint32_t width = 32 / per, e = lane % width;
#pragma unroll 2
    for (uint32_t b = warp * per; b < kTileStrands; b += warps * per) {
      const uint32_t sl = b + lane / width;
      const uint32_t to = __shfl_sync(0xffffffffu, place, sl);
      if (sl < ns && e < elems) put(sl, to, e);
    }
  }
}

template <int C>
cudaError_t launch_strand_major(const float4* soa, float* out, const uint32_t* order, uint32_t nstrands,
                                uint32_t npoints, uint32_t stride, cudaStream_t st) {
  if (nstrands == 0) return cudaSuccess;
  const uint32_t row = npoints | 1u, elems = C == 4 ? npoints : 3 * npoints;
  uint32_t per = 1;
  while (per < 32 && 2 * per * elems <= 32) per *= 2;
  k_to_strand_major<C><<<(nstrands + kTileStrands - 1) / kTileStrands, npoints <= 12 ? 128 : 256,
                         sizeof(float4) * kTileStrands * row, st>>>(soa, out, order, nstrands, npoints, stride, row, per);
  return cudaGetLastError();
}

// Tile rows are padded by one float4 so that the 32 strands of a point
// (one row each) fall in different shared-memory banks.
__global__ void k_from_strand_major(const float4* __restrict__ in, float4* __restrict__ soa,
                                    const uint32_t* __restrict__ order, uint32_t nstrands, uint32_t npoints,
                                    uint32_t stride) {
  __shared__ float4 tile[kTileStrands * (HS_MAX_POINTS_PER_STRAND + 1)];
  const uint32_t s0 = blockIdx.x * kTileStrands;
  const uint32_t ns = min(static_cast<uint32_t>(kTileStrands), nstrands - s0);
  const uint32_t total = ns * npoints;
  const uint32_t row = npoints + 1;
  for (uint32_t t = threadIdx.x; t < total; t += blockDim.x) {
    const uint32_t sl = t / npoints, i = t % npoints;
    tile[sl * row + i] = in[static_cast<size_t>(order[s0 + sl]) * npoints + i];
  }
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < kTileStrands * npoints; t += blockDim.x) {
    const uint32_t i = t / kTileStrands, sl = t % kTileStrands;
    if (sl < ns) soa[static_cast<size_t>(i) * stride + s0 + sl] = tile[sl * row + i];
  }
}

// [point][stride] -> [point][nstrands] in the caller's strand order.
__global__ void k_to_point_major(const float4* __restrict__ soa, float4* __restrict__ out,
                                 const uint32_t* __restrict__ order, uint32_t nstrands, uint32_t npoints,
                                 uint32_t stride) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nstrands) return;
  const uint32_t c = order[s];
  for (uint32_t i = 0; i < npoints; ++i)
    out[static_cast<size_t>(i) * nstrands + c] = soa[static_cast<size_t>(i) * stride + s];
}

__global__ void k_copy_roots(const float4* __restrict__ soa, float4* __restrict__ root_rest, uint32_t nstrands) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < nstrands) {
    const float4 p = soa[s];
    root_rest[s] = make_float4(p.x, p.y, p.z, 0.0f);
  }
}

}  // namespace

int step_capacity(uint32_t npoints) {
  if (npoints < HS_MIN_POINTS_PER_STRAND) return 0;
  if (npoints <= 4) return 4;
  if (npoints <= 8) return 8;
  if (npoints <= 16) return 16;
  if (npoints <= 24) return 24;
  if (npoints <= 32) return 32;
  if (npoints <= HS_MAX_POINTS_PER_STRAND) return 64;
  return 0;
}

int plain_mapping(const GroomView& g, const FrameConst& fc, int mapping) {
  const int K = lane_group(fc.mode, fc.substeps, fc.iterations);
  if (mapping == HS_MAPPING_LANES || K == 0) return mapping == HS_MAPPING_LANES ? HS_MAPPING_LANES : HS_MAPPING_THREAD;
  if (mapping == HS_MAPPING_THREAD) return HS_MAPPING_THREAD;
  // AUTO: lane groups while they make at most `limit` warps per SM (32-strand
  // tiles x K). Their time grows with those warps times the wavefront's N + 2 S
  // steps; a thread per strand takes S N chain links whatever the warps, until
  // these fill the SMs. So the two meet at a multiple of S N / (N + 2 S), the
  // larger the more sphere tests a thread runs in turn. Measured multiples
  // (2 - 16 substeps, 4 - 64 points): 2.5 - 4 without spheres (5 up to 8
  // points, where a thread per strand is the register form), 4.3 - 6.5 at one,
  // 6.5 - 9.5 at 3 - 7, 7.2 - 13 at 10 - 32. Lanes / thread, us a frame (EXACT):
  // 20,000 x 16, S 4, 7 spheres (16.4 warps) 8.2 / 11.0, 50,000 x 64 (41.1)
  // 65.4 / 45.0, 54,476 x 32 without spheres (44.8) 31.0 / 17.4. A group of
  // two holds few warps of long strands in shared memory, and gains only while
  // they are resident together (22,431 x 64, S 2: 27.3 / 19.7).
  // The multiples lie between those of one groom alone (3.5, 6.5, 9.5 and 13 by
  // the same classes) and of three in turn on streams of their own, which share
  // the SMs (1.9, 3.3, 4.3 and 6.4): 12,000 x 16 among 2, S 5, FAST, takes 18.6
  // / 22.8 alone, 13.6 / 9.2 in turn.
  const uint32_t N = g.npoints, S = static_cast<uint32_t>(fc.substeps);
  const float multiple = fc.nspheres > 8 ? 8.5f : fc.nspheres > 1 ? 7.0f : fc.nspheres == 1 || N <= 8 ? 5.0f : 3.0f;
  float limit = multiple * static_cast<float>(S * N) / static_cast<float>(N + 2 * S);
  if (K == 2) limit = std::min(limit, 2.0f * static_cast<float>(227u / N));  // blocks of 1 KB a point
  const int sms = device_attribute(cudaDevAttrMultiProcessorCount, 152);
  const float warps = static_cast<float>((static_cast<uint64_t>(g.nstrands) + 31) / 32 * static_cast<uint64_t>(K));
  return warps <= limit * static_cast<float>(sms) ? HS_MAPPING_LANES : HS_MAPPING_THREAD;
}

cudaError_t launch_step(const GroomView& g, const FrameConst& fc, int mapping, cudaStream_t st) {
  if (g.nstrands == 0) return cudaSuccess;
  if (plain_mapping(g, fc, mapping) == HS_MAPPING_LANES) return launch_step_lanes(g, fc, st);
  // Short strands: everything in registers. Longer: the streaming form.
  if (g.npoints > 8) return launch_step_stream(g, fc, st);
  switch (step_capacity(g.npoints)) {
    case 4: return launch_step_mode<4>(g, fc, st);
    case 8: return launch_step_mode<8>(g, fc, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_init(const GroomView& g, const InitArgs& a, float4* root_rest, cudaStream_t st) {
  if (g.nstrands == 0) return cudaSuccess;
  k_init<<<(g.nstrands + 127) / 128, 128, 0, st>>>(g, a, root_rest);
  return cudaGetLastError();
}

cudaError_t launch_to_strand_major(const float4* soa, float4* out, const uint32_t* order, uint32_t nstrands,
                                   uint32_t npoints, uint32_t stride, cudaStream_t st) {
  return launch_strand_major<4>(soa, reinterpret_cast<float*>(out), order, nstrands, npoints, stride, st);
}

cudaError_t launch_to_strand_major_xyz(const float4* soa, float* out, const uint32_t* order, uint32_t nstrands,
                                       uint32_t npoints, uint32_t stride, cudaStream_t st) {
  return launch_strand_major<3>(soa, out, order, nstrands, npoints, stride, st);
}

cudaError_t launch_from_strand_major(const float4* in, float4* soa, const uint32_t* order, uint32_t nstrands,
                                     uint32_t npoints, uint32_t stride, cudaStream_t st) {
  if (nstrands == 0) return cudaSuccess;
  k_from_strand_major<<<(nstrands + kTileStrands - 1) / kTileStrands, 256, 0, st>>>(in, soa, order, nstrands,
                                                                                      npoints, stride);
  return cudaGetLastError();
}

cudaError_t launch_to_point_major(const float4* soa, float4* out, const uint32_t* order, uint32_t nstrands,
                                  uint32_t npoints, uint32_t stride, cudaStream_t st) {
  if (nstrands == 0) return cudaSuccess;
  k_to_point_major<<<(nstrands + 255) / 256, 256, 0, st>>>(soa, out, order, nstrands, npoints, stride);
  return cudaGetLastError();
}

cudaError_t launch_copy_roots(const float4* soa, float4* root_rest, uint32_t nstrands, cudaStream_t st) {
  if (nstrands == 0) return cudaSuccess;
  k_copy_roots<<<(nstrands + 255) / 256, 256, 0, st>>>(soa, root_rest, nstrands);
  return cudaGetLastError();
}

// A few attributes per device are asked for; each slot caches one as a
// single 64-bit word (attribute + 1 in the high half, 0 = empty; the value
// in the low half), so that a reader sees a pair or nothing.
int device_attribute(cudaDeviceAttr attr, int fallback) {
  static std::atomic<uint64_t> cache[kMaxDevices][4];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return fallback;
  }
  const uint64_t key = static_cast<uint64_t>(static_cast<uint32_t>(attr) + 1u) << 32;
  for (std::atomic<uint64_t>& slot : cache[dev]) {
    uint64_t w = slot.load(std::memory_order_acquire);
    if ((w & ~uint64_t{0xffffffffu}) == key) return static_cast<int>(static_cast<uint32_t>(w));
    if (w != 0) continue;
    int v = 0;
    if (cudaDeviceGetAttribute(&v, attr, dev) != cudaSuccess) {
      cudaGetLastError();
      return fallback;
    }
    const uint64_t entry = key | static_cast<uint32_t>(v);
    if (slot.compare_exchange_strong(w, entry, std::memory_order_acq_rel) || w == entry) return v;
  }
  int v = 0;
  if (cudaDeviceGetAttribute(&v, attr, dev) != cudaSuccess) {
    cudaGetLastError();
    return fallback;
  }
  return v;
}

}  // namespace hs
