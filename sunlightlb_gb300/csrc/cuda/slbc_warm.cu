// Tensor-core kernels of the learned warm start (BF16 inputs, FP32
// accumulation in TMEM, tcgen05.mma issued by one thread, operands staged by
// TMA through a 4-stage mbarrier pipeline).
//
// slbc_tc_gemm: D[M x N] (FP32, row-major, leading dimension ldd) =
// A[M x K] * B[N x K]^T with A and B BF16, row-major (K contiguous).  The
// weight gradients of the network's convolutions are this product.
#include <algorithm>
#include <cstring>
#include <mutex>

#include "slbc_internal.cuh"
#include "slbc_tc.cuh"

#include <cuda_bf16.h>

namespace {

using namespace slbc;

constexpr int kBM = 128, kBN = 128, kBK = 64, kStages = 4;
constexpr int kTileA = kBM * kBK * 2;  // bytes of one A stage (128 rows x 128 B)
constexpr int kTileB = kBN * kBK * 2;
constexpr int kGemmSmem = kStages * (kTileA + kTileB) + 1024;
constexpr uint32_t kWaitLimit = 1u << 20;  // polls before a wait gives up
constexpr int kConvSms = 152;              // blocks of a persistent convolution, one per SM

// error flag of the tensor-core kernels, one per device
int *g_tc_err[64];
std::mutex g_tc_lock;

int *tc_err_flag() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> guard(g_tc_lock);
  if (!g_tc_err[dev]) {
    if (cudaMalloc(&g_tc_err[dev], sizeof(int)) != cudaSuccess) return nullptr;
    if (cudaMemset(g_tc_err[dev], 0, sizeof(int)) != cudaSuccess) return nullptr;
  }
  return g_tc_err[dev];
}

// Opt a kernel into `bytes` of dynamic shared memory on the current device;
// the attribute is per device, so `done` keeps one bit per device index.
cudaError_t smem_opt_in(const void *fn, int bytes, unsigned long long &done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> guard(g_tc_lock);
  if (done >> dev & 1ull) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done |= 1ull << dev;
  return e;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point
typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
  static EncodeTiled fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiled)p;
  });
  return fn;
}

// 2-D BF16 row-major matrix (rows x cols, cols contiguous), box of
// box_rows x 64 elements (128 bytes, 128-byte swizzle)
bool make_map_2d(CUtensorMap *map, const void *ptr, long long rows, long long cols, int box_rows) {
  EncodeTiled enc = encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// One 128 x 128 output tile per block of 128 threads: thread 0 loads (TMA),
// thread 32 issues the MMAs, all four warps read the accumulator back.
__global__ void __launch_bounds__(128, 1)
k_gemm_bf16(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, float *D, int ldd,
            int K, int *err) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u;
  uint8_t *tA = smem_raw + pad;
  uint8_t *tB = tA + kStages * kTileA;
  __shared__ uint64_t full[kStages], empty[kStages], done;
  __shared__ uint32_t tmem_base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
  const int nk = K / kBK;
  if (warp == 0) {
    tc::tmem_alloc(&tmem_base, kBN);
    tc::tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < kStages; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(&done, 1);
    tc::fence_mbar_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  bool ok = true;
  int issued = 0;
  if (warp == 0 && tc::elect_one()) {
    for (int kt = 0; kt < nk; kt++) {
      const int s = kt % kStages;
      if (kt >= kStages && !tc::mbar_wait(&empty[s], ((kt / kStages) - 1) & 1, kWaitLimit)) {
        ok = false;
        break;
      }
      tc::mbar_expect_tx(&full[s], kTileA + kTileB);
      tc::tma_load_2d(tA + s * kTileA, &ta, &full[s], kt * kBK, m0);
      tc::tma_load_2d(tB + s * kTileB, &tb, &full[s], kt * kBK, n0);
      issued = kt + 1;
    }
  } else if (warp == 1 && tc::elect_one()) {
    constexpr uint32_t idesc = tc::idesc_bf16(kBM, kBN);
    for (int kt = 0; kt < nk; kt++) {
      const int s = kt % kStages;
      if (!tc::mbar_wait(&full[s], (kt / kStages) & 1, kWaitLimit)) {
        ok = false;
        break;
      }
      tc::fence_after_sync();
      const uint64_t ad = tc::smem_desc(tA + s * kTileA, tc::kSwizzle128, 128);
      const uint64_t bd = tc::smem_desc(tB + s * kTileB, tc::kSwizzle128, 128);
#pragma unroll
      for (int kk = 0; kk < kBK / 16; kk++)  // 16 BF16 = 32 bytes = 2 descriptor units
        tc::mma_bf16(tmem, ad + 2 * kk, bd + 2 * kk, idesc, (kt | kk) != 0);
      tc::mma_commit(&empty[s]);
    }
    tc::mma_commit(&done);
  }
  __syncwarp();
  const bool okd = __all_sync(0xffffffffu, tc::mbar_wait(&done, 0, kWaitLimit));
  tc::fence_after_sync();
  if (okd) {
    const int row = m0 + warp * 32 + lane;
#pragma unroll 1
    for (int c = 0; c < kBN; c += 8) {
      float v[8];
      tc::tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
      float4 *dst = (float4 *)(D + (long long)row * ldd + n0 + c);
      dst[0] = make_float4(v[0], v[1], v[2], v[3]);
      dst[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
  }
  if (!ok || !okd) atomicExch(err, 1);
  if (warp == 0 && tc::elect_one()) {
    // the loads this thread issued have all landed before the block ends
    for (int kt = issued > kStages ? issued - kStages : 0; kt < issued; kt++)
      if (!tc::mbar_wait(&full[kt % kStages], (kt / kStages) & 1, kWaitLimit)) atomicExch(err, 2);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, kBN);
}

bool aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

// ---- periodic 3x3x3 convolution as an implicit GEMM ---------------------------
// Activations are channels-last BF16 with a one-voxel periodic halo:
// buf[n][z + 1][y + 1][x + 1][c] for z < D, y < H, x < W (the halo holds the
// wrapped neighbours, slbc_tc_halo).  Output tile: 128 voxels (a box of
// wbox x hbox x dbox) x all cout channels.  K runs over the 27 taps x the
// 32-channel chunks of the input: per step one TMA box of the input
// (32 channels x the tile shifted by the tap) and the tap's weights
// (cout x 32), two MMAs of K = 16.  Weights: w[tap][chunk][cout][32].
struct ConvArgs {
  int D, H, W;
  int cin, cout;
  int in_coff;
  int out_ctot, out_coff;
  int wbox, hbox, dbox;
  int relu;
  int tmem_cols;
  const float *bias;         // cout values or null
  const __nv_bfloat16 *mask; // or null: output *= (mask > 0), same layout as out
  __nv_bfloat16 *out;
  float *out_f32;            // or null: FP32 output (same layout) instead of out
};

constexpr int kConvTileA = 128 * 64;       // 128 voxels x 32 channels x 2 B

// Pipeline depth by output width: a stage is one A tile and one B tile of
// cout rows x 64 B, and every depth below keeps the stages within 96 KB, so
// two CTAs share an SM.
__host__ __device__ constexpr int conv_stages(int cout) { return cout <= 64 ? 8 : (cout <= 128 ? 6 : 4); }
__host__ __device__ constexpr int conv_smem(int nst, int cout) { return nst * (kConvTileA + cout * 64) + 1024; }
constexpr int kConvSmemMax = conv_smem(8, 64);
static_assert(conv_smem(6, 128) <= kConvSmemMax && conv_smem(4, 256) <= kConvSmemMax, "stage budget");

// The producer and the MMA issuer step through (tap, channel chunk, stage,
// round) with counters instead of divisions: for the narrow layers an MMA pair
// takes a few tens of cycles, so the single-thread loops set the pace.  On
// coarse grids, whose 128-voxel tiles are far fewer than the SMs, the output
// channels are split over the blocks of gridDim.z (a.cout each): the K loop of
// 27 taps x cin is the same length but its stages are smaller and deeper.
template <int NST>
__global__ void __launch_bounds__(128, 2)
k_conv_fwd(const __grid_constant__ CUtensorMap tx, const __grid_constant__ CUtensorMap tw, ConvArgs a, int *err) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u;
  uint8_t *tA = smem_raw + pad;
  const uint32_t tile_b = (uint32_t)a.cout * 64u;  // of this block's output channels
  const int co0 = (int)blockIdx.z * a.cout;
  uint8_t *tB = tA + NST * kConvTileA;
  __shared__ uint64_t full[NST], empty[NST], done;
  __shared__ uint32_t tmem_base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.y;
  const int tiles_x = a.W / a.wbox, tiles_y = a.H / a.hbox;
  const int m = blockIdx.x;
  const int x0 = (m % tiles_x) * a.wbox, y0 = ((m / tiles_x) % tiles_y) * a.hbox, z0 = (m / (tiles_x * tiles_y)) * a.dbox;
  const int nck = a.cin / 32;
  const int nk = 27 * nck;
  const uint32_t bytes_b = (uint32_t)a.cout * 64u;
  if (warp == 0) {
    tc::tmem_alloc(&tmem_base, (uint32_t)a.tmem_cols);
    tc::tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < NST; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(&done, 1);
    tc::fence_mbar_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  bool ok = true;
  int issued = 0;
  if (warp == 0 && tc::elect_one()) {
    int s = 0, round = 0, ck = 0, dx = 0, dy = 0, dz = 0;
    int c = a.in_coff, wrow = co0;
    for (int kt = 0; kt < nk; kt++) {
      if (round > 0 && !tc::mbar_wait(&empty[s], (uint32_t)(round - 1) & 1u, kWaitLimit)) {
        ok = false;
        break;
      }
      tc::mbar_expect_tx(&full[s], (uint32_t)kConvTileA + bytes_b);
      tc::tma_load_5d(tA + s * kConvTileA, &tx, &full[s], c, x0 + dx, y0 + dy, z0 + dz, n);
      tc::tma_load_2d(tB + s * tile_b, &tw, &full[s], 0, wrow);
      issued = kt + 1;
      wrow += a.cout * (int)gridDim.z;
      c += 32;
      if (++ck == nck) {
        ck = 0;
        c = a.in_coff;
        if (++dx == 3) {
          dx = 0;
          if (++dy == 3) {
            dy = 0;
            ++dz;
          }
        }
      }
      if (++s == NST) {
        s = 0;
        ++round;
      }
    }
  } else if (warp == 1 && tc::elect_one()) {
    const uint32_t idesc = tc::idesc_bf16(128, a.cout);
    const uint64_t ad0 = tc::smem_desc(tA, tc::kSwizzle64, 64);
    const uint64_t bd0 = tc::smem_desc(tB, tc::kSwizzle64, 64);
    int s = 0, round = 0;
    for (int kt = 0; kt < nk; kt++) {
      if (!tc::mbar_wait(&full[s], (uint32_t)round & 1u, kWaitLimit)) {
        ok = false;
        break;
      }
      tc::fence_after_sync();
      // the start-address field counts 16-byte units
      const uint64_t ad = ad0 + (uint64_t)(s * (kConvTileA >> 4));
      const uint64_t bd = bd0 + (uint64_t)(s * (tile_b >> 4));
      tc::mma_bf16(tmem, ad, bd, idesc, kt != 0);
      tc::mma_bf16(tmem, ad + 2, bd + 2, idesc, 1);
      tc::mma_commit(&empty[s]);
      if (++s == NST) {
        s = 0;
        ++round;
      }
    }
    tc::mma_commit(&done);
  }
  __syncwarp();
  const bool okd = __all_sync(0xffffffffu, tc::mbar_wait(&done, 0, kWaitLimit));
  tc::fence_after_sync();
  if (okd) {
    const int r = warp * 32 + lane;
    const int vx = x0 + r % a.wbox, vy = y0 + (r / a.wbox) % a.hbox, vz = z0 + r / (a.wbox * a.hbox);
    const long long vox = (((long long)n * (a.D + 2) + vz + 1) * (a.H + 2) + vy + 1) * (a.W + 2) + vx + 1;
    __nv_bfloat16 *dst = a.out + vox * a.out_ctot + a.out_coff + co0;
    const __nv_bfloat16 *msk = a.mask ? a.mask + vox * a.out_ctot + a.out_coff + co0 : nullptr;
#pragma unroll 1
    for (int c = 0; c < a.cout; c += 8) {
      float v[8];
      tc::tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
      if (a.bias) {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] += a.bias[co0 + c + i];
      }
      if (a.relu) {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = fmaxf(v[i], 0.0f);
      }
      if (msk) {
        const uint4 mv = *(const uint4 *)(msk + c);
        const __nv_bfloat16 *mb = (const __nv_bfloat16 *)&mv;
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __bfloat162float(mb[i]) > 0.0f ? v[i] : 0.0f;
      }
      if (a.out_f32) {
        float4 *fd = (float4 *)(a.out_f32 + vox * a.out_ctot + a.out_coff + co0 + c);
        fd[0] = make_float4(v[0], v[1], v[2], v[3]);
        fd[1] = make_float4(v[4], v[5], v[6], v[7]);
      } else {
        uint4 o;
        __nv_bfloat162 *ob = (__nv_bfloat162 *)&o;
#pragma unroll
        for (int i = 0; i < 4; i++) ob[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        *(uint4 *)(dst + c) = o;
      }
    }
  }
  if (!ok || !okd) atomicExch(err, 1);
  if (warp == 0 && tc::elect_one()) {
    for (int kt = issued > NST ? issued - NST : 0; kt < issued; kt++)
      if (!tc::mbar_wait(&full[kt % NST], (kt / NST) & 1, kWaitLimit)) atomicExch(err, 2);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, (uint32_t)a.tmem_cols);
}

// One accumulator row per lane (COUT columns from TMEM address acc) to the
// voxel at element `at` of the output: bias, ReLU, mask, conversion.
template <int COUT>
__device__ __forceinline__ void conv_rows_out(const ConvArgs &a, uint32_t acc, long long at, const float *bias) {
#pragma unroll 1
  for (int c = 0; c < COUT; c += 16) {
    float v[16];
    tc::tmem_ld16(acc + (uint32_t)c, v);
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] += bias[c + i];
    if (a.relu) {
#pragma unroll
      for (int i = 0; i < 16; i++) v[i] = fmaxf(v[i], 0.0f);
    }
    if (a.mask) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uint4 mv = *(const uint4 *)(a.mask + at + c + 8 * h);
        const __nv_bfloat16 *mb = (const __nv_bfloat16 *)&mv;
#pragma unroll
        for (int i = 0; i < 8; i++) v[8 * h + i] = __bfloat162float(mb[i]) > 0.0f ? v[8 * h + i] : 0.0f;
      }
    }
    if (a.out_f32) {
      float4 *fd = (float4 *)(a.out_f32 + at + c);
#pragma unroll
      for (int h = 0; h < 4; h++) fd[h] = make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
    } else {
      uint4 o[2];
      __nv_bfloat162 *ob = (__nv_bfloat162 *)o;
#pragma unroll
      for (int i = 0; i < 8; i++) ob[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      uint4 *dst = (uint4 *)(a.out + at + c);
      dst[0] = o[0];
      dst[1] = o[1];
    }
  }
}

// Convolution of 32, 64 and, as two parts of 64, 128 output channels (and of 32
// to 96), one persistent block per SM, every
// input voxel staged once per 32-channel chunk.  An output item is 8 (x) x 16
// (y) x up to S (z) voxels; input planes of 10 x 18 voxels (64-byte rows, x
// fastest, halo included) go through a ring in shared memory, one TMA box
// each.  The 128 rows of an MMA are the 16 y-lines of 8 voxels: groups of 8
// rows at a pitch of 10 rows, so the tap (dx, dy) only moves the start by
// 10 dy + dx rows (the swizzle is a function of the address, not of the row).
// Weights come per (chunk, dx); with one chunk they stay for all items.
//
// An MMA of 128 x N x 16 takes max(32 + N / 4, N / 2) cycles: its A rows and
// weights come from shared memory at 128 bytes per cycle.  Input plane zi
// serves the output slices zi - 2, zi - 1 and zi (dz = 2, 1, 0), whose
// accumulators are neighbours in TMEM, so the weights of the three dz lie
// stacked in that order and one MMA of 128 x 3 cout does all three from one
// read of A.  Every accumulator receives its products in the order chunk, dx,
// dz, dy.  A plane leaves the ring in the last dx of its chunk, plane by
// plane, while the next item's come in; two accumulator sets alternate between
// items, so four warps write item i while the MMAs of item i + 1 run.
//
// Bound: the MMAs (75% of the peak for 32 output channels by the formula).
// Measured at 128^3: 32 -> 32 channels 136 -> 95 us (854 -> 1220 TFLOP/s), 96
// -> 32 1300 TFLOP/s; 64^3: 64 -> 64 channels 60 -> 44 us (1320 TFLOP/s); before,
// a stage held the input block of one x-shift (three times the copies), the
// issuing thread was slower than the tensor core, and a tile had 2 or 4 slices.
// 128 channels in two parts: the six layers on 4 x 16^3 of a training iteration
// 190 -> 125 us (64 tiles of two slices were less than half of the SMs).
// 32 -> 96 at 4 x 64^3: 280 -> 116 us (k_conv_fwd before, whose order of
// products, dz, dy, dx, it keeps).
template <int COUT>
struct ConvR {
  static constexpr int kS = 256 / COUT;                // slices of an item, at most
  static constexpr int kPlane = 23 * 512;              // 180 rows of 64 B
  static constexpr int kPlanes = COUT == 32 ? 14 : COUT == 64 ? 12 : 5;
  static constexpr int kTileB = 9 * COUT * 64;
  static constexpr int kStagesB = COUT == 64 ? 2 : 3;
  static constexpr int kSmem = kPlanes * kPlane + kStagesB * kTileB + 1024;
  static constexpr int kSet = kS * COUT;               // TMEM columns of one accumulator set
  static_assert(kSmem <= 227 * 1024 - 2048 && 2 * kSet <= 512 && kS + 2 <= kPlanes, "budget");
};

// The MMAs of one 32-channel chunk of an item, issued by one thread.  The
// loop over the planes is unrolled for each run length, so that next to the
// ring position everything is a constant: a plane's six MMAs take some 300
// cycles of the tensor core, and what the thread does between them must take
// less (computed with run-time lengths: 350 cycles per plane; the five
// 32-channel layers of a 128^3 grid 706 us).
template <int COUT>
struct ConvRIssue {
  using C = ConvR<COUT>;
  uint32_t a_ring, b_ring, d0;    // low descriptor words (16-byte units); accumulator set
  uint64_t *full_b, *empty_b, *full_p, *empty_p;
  uint32_t limit = kWaitLimit;    // of a wait; 0 once one has run out
  int slot = 0, sb = 0;           // ring slot of the chunk's first plane, next weight stage
  uint32_t phase_p = 0, phase_b = 0;
  bool keep_b, with_b;

  __device__ __forceinline__ void wait(uint64_t *bar, uint32_t phase) {
    if (!tc::mbar_wait(bar, phase, limit)) limit = 0;
  }

  __device__ __forceinline__ static void mma(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t accumulate) {
    tc::mma_bf16(d, tc::desc_of(a, tc::kSwizzle64, 10 * 64), tc::desc_of(b, tc::kSwizzle64, 8 * 64), idesc, accumulate);
  }

  // The one chunk of 32 input channels with all weights in shared memory: each
  // plane is finished, in the order dz, dy, dx, before it leaves the ring.
  template <int LEN>
  __device__ __forceinline__ void whole() {
    if constexpr (LEN <= C::kS) {
      constexpr uint32_t tap = COUT * 64 >> 4, plane = C::kPlane >> 4, stage = C::kTileB >> 4;
      if (with_b)
        for (int dx = 0; dx < 3; dx++) wait(&full_b[dx], 0);
#pragma unroll
      for (int zi = 0; zi < LEN + 2; zi++) {
        wait(&full_p[slot], phase_p);
        tc::fence_after_sync();
        const int lo = zi > LEN - 1 ? zi - (LEN - 1) : 0, hi = zi < 2 ? zi : 2;  // dz of the slices this plane serves
        const uint32_t d = d0 + (uint32_t)((zi - hi) * COUT), id = tc::idesc_bf16(128, (hi - lo + 1) * COUT);
        const uint32_t az = a_ring + (uint32_t)slot * plane, bz = b_ring + (uint32_t)(2 - hi) * tap;
#pragma unroll
        for (int t = 0; t < 18; t++) {
          const int dy = t / 6, dx = t / 2 % 3, kk = t % 2;
          const uint32_t at = az + (uint32_t)(dy * 40 + dx * 4 + 2 * kk);
          const uint32_t bt = bz + (uint32_t)(dx * stage + dy * 3 * tap + 2 * kk);
          if (t == 0 && lo == 0) {
            // the first product of the last of these slices (dz = 0) overwrites it
            if (hi > 0) mma(d, at, bt, tc::idesc_bf16(128, hi * COUT), 1);
            mma(d + (uint32_t)(hi * COUT), at, bt + hi * tap, tc::idesc_bf16(128, COUT), 0);
          } else {
            mma(d, at, bt, id, 1);
          }
        }
        tc::mma_commit(&empty_p[slot]);
        if (++slot == C::kPlanes) {
          slot = 0;
          phase_p ^= 1u;
        }
      }
    }
  }

  template <int LEN>
  __device__ __forceinline__ void chunk(uint32_t more) {
    if constexpr (LEN <= C::kS) {
      constexpr uint32_t tap = COUT * 64 >> 4, plane = C::kPlane >> 4;
      int sp = slot;
      uint32_t ph = phase_p;
#pragma unroll 1
      for (int dx = 0; dx < 3; dx++) {
        if (with_b) {
          wait(&full_b[sb], phase_b);
          tc::fence_after_sync();
        }
        const uint32_t bx = b_ring + (uint32_t)sb * (C::kTileB >> 4), acc = more | (dx > 0);
        sp = slot;
        ph = phase_p;
#pragma unroll
        for (int zi = 0; zi < LEN + 2; zi++) {
          if (dx == 0) {
            wait(&full_p[sp], ph);
            tc::fence_after_sync();
          }
          // dz of the slices this plane serves
          const int lo = zi > LEN - 1 ? zi - (LEN - 1) : 0, hi = zi < 2 ? zi : 2;
          const uint32_t d = d0 + (uint32_t)((zi - hi) * COUT), id = tc::idesc_bf16(128, (hi - lo + 1) * COUT);
          const uint32_t az = a_ring + (uint32_t)sp * plane + (uint32_t)dx * 4u, bz = bx + (uint32_t)(2 - hi) * tap;
          if (lo == 0 && hi > 0 && !acc) {
            // the first product of the last of these slices (dz = 0) overwrites it
            mma(d, az, bz, tc::idesc_bf16(128, hi * COUT), 1);
            mma(d + (uint32_t)(hi * COUT), az, bz + hi * tap, tc::idesc_bf16(128, COUT), 0);
          } else {
            mma(d, az, bz, id, lo == 0 && hi == 0 ? acc : 1);
          }
          mma(d, az + 2, bz + 2, id, 1);
          mma(d, az + 40, bz + 3 * tap, id, 1);
          mma(d, az + 42, bz + 3 * tap + 2, id, 1);
          mma(d, az + 80, bz + 6 * tap, id, 1);
          mma(d, az + 82, bz + 6 * tap + 2, id, 1);
          if (dx == 2) tc::mma_commit(&empty_p[sp]);
          if (++sp == C::kPlanes) {
            sp = 0;
            ph ^= 1u;
          }
        }
        if (with_b && !keep_b) tc::mma_commit(&empty_b[sb]);
        if (++sb == C::kStagesB) {
          sb = 0;
          phase_b ^= 1u;
        }
      }
      slot = sp;
      phase_p = ph;
    }
  }
};

template <int COUT>
__global__ void __launch_bounds__(192, 1)
k_conv_r(const __grid_constant__ CUtensorMap tx, const __grid_constant__ CUtensorMap tw, ConvArgs a, int runs,
         int items, int parts, int *err) {
  after_previous();
  using C = ConvR<COUT>;
  constexpr int NB = C::kStagesB, NP = C::kPlanes;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u;
  constexpr uint32_t tap_b = COUT * 64;  // one tap's weights
  uint8_t *const tB = smem_raw + pad, *const tA = tB + NB * C::kTileB;
  __shared__ uint64_t full_b[NB], empty_b[NB], full_p[NP], empty_p[NP], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base;
  __shared__ float bias[128];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_x = a.W / 8, tiles_y = a.H / 16, cols = tiles_x * tiles_y;
  const int nck = a.cin / 32;
  const bool keep_b = nck == 1 && NB >= 3;  // all weights fit: loaded for the first item only
  if (warp == 0) {
    tc::tmem_alloc(&tmem_base, 512);
    tc::tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < NB; s++) {
      tc::mbar_init(&full_b[s], 1);
      tc::mbar_init(&empty_b[s], 1);
    }
    for (int s = 0; s < NP; s++) {
      tc::mbar_init(&full_p[s], 1);
      tc::mbar_init(&empty_p[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], 4);
    }
    tc::fence_mbar_init();
  }
  for (int c = threadIdx.x; c < a.cout; c += 192) bias[c] = a.bias ? a.bias[c] : 0.0f;
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  bool ok = true;
  // an item is a part of the output channels of a tile; first slice and number
  // of slices of a tile: a column is cut into `runs` almost equal runs
  const auto slices = [&](int item, int &z0) {
    const int run = (item / cols) % runs;
    z0 = run * a.D / runs;
    return (run + 1) * a.D / runs - z0;
  };
  if (warp == 0 && tc::elect_one()) {  // copies
    int nb = 0, np = 0;    // weight stages and planes issued
    const auto load_b = [&](int ck, int dx, int part) {
      const int s = nb % NB;
      if (nb >= NB && !tc::mbar_wait(&empty_b[s], (uint32_t)(nb / NB - 1) & 1u, kWaitLimit)) return false;
      tc::mbar_expect_tx(&full_b[s], (uint32_t)C::kTileB);
      for (int dy = 0; dy < 3; dy++)
        for (int dz = 0; dz < 3; dz++)
          tc::tma_load_2d(tB + s * C::kTileB + (dy * 3 + 2 - dz) * tap_b, &tw, &full_b[s], 0,
                          ((dz * 9 + dy * 3 + dx) * nck + ck) * a.cout + part * COUT);
      nb++;
      return true;
    };
    for (int work = blockIdx.x; work < items * parts && ok; work += gridDim.x) {
      const int item = work / parts, part = work - item * parts;
      const int x0 = (item % tiles_x) * 8, y0 = ((item / tiles_x) % tiles_y) * 16, n = item / (cols * runs);
      int z0;
      const int len = slices(item, z0);
      const bool with_b = !keep_b || work == (int)blockIdx.x;
      for (int ck = 0; ck < nck && ok; ck++) {
        if (with_b) ok = load_b(ck, 0, part);
        for (int zi = 0; zi < len + 2 && ok; zi++) {
          const int s = np % NP;
          if (np >= NP && !tc::mbar_wait(&empty_p[s], (uint32_t)(np / NP - 1) & 1u, kWaitLimit)) {
            ok = false;
            break;
          }
          tc::mbar_expect_tx(&full_p[s], 180 * 64);
          // padded coordinates: interior voxel v is v + 1, the halo before it v
          tc::tma_load_5d(tA + s * C::kPlane, &tx, &full_p[s], a.in_coff + ck * 32, x0, y0, z0 + zi, n);
          np++;
        }
        if (with_b && ok) ok = load_b(ck, 1, part);
        if (with_b && ok) ok = load_b(ck, 2, part);
      }
    }
    // the copies issued have landed before the block ends
    for (int i = nb > NB ? nb - NB : 0; i < nb; i++)
      if (!tc::mbar_wait(&full_b[i % NB], (uint32_t)(i / NB) & 1u, kWaitLimit)) atomicExch(err, 2);
    for (int i = np > NP ? np - NP : 0; i < np; i++)
      if (!tc::mbar_wait(&full_p[i % NP], (uint32_t)(i / NP) & 1u, kWaitLimit)) atomicExch(err, 2);
  } else if (warp == 1 && tc::elect_one()) {  // MMAs
    ConvRIssue<COUT> m;
    m.a_ring = (uint32_t)tc::smem_desc(tA, tc::kSwizzle64, 64, 10 * 64);
    m.b_ring = (uint32_t)tc::smem_desc(tB, tc::kSwizzle64, 64);
    m.full_b = full_b; m.empty_b = empty_b; m.full_p = full_p; m.empty_p = empty_p;
    m.keep_b = keep_b;
    int g = 0;
    for (int work = blockIdx.x; work < items * parts && m.limit; work += gridDim.x, g++) {
      const int set = g & 1;
      int z0;
      const int len = slices(work / parts, z0);
      m.with_b = !keep_b || g == 0;
      if (g >= 2) m.wait(&acc_empty[set], (uint32_t)((g >> 1) - 1) & 1u);
      tc::fence_after_sync();
      m.d0 = tmem + (uint32_t)(set * C::kSet);
      if constexpr (COUT > 64) {
        if (len == 1) m.template whole<1>();
        else m.template whole<2>();
      } else {
        for (int ck = 0; ck < nck; ck++) {
          const uint32_t more = ck > 0;
          switch (len) {
            case 1: m.template chunk<1>(more); break;
            case 2: m.template chunk<2>(more); break;
            case 3: m.template chunk<3>(more); break;
            case 4: m.template chunk<4>(more); break;
            case 5: m.template chunk<5>(more); break;
            case 6: m.template chunk<6>(more); break;
            case 7: m.template chunk<7>(more); break;
            default: m.template chunk<8>(more); break;
          }
        }
      }
      tc::mma_commit(&acc_full[set]);
    }
    ok = m.limit != 0;
  } else if (warp >= 2) {  // accumulators to memory
    const int quarter = warp & 3, row = quarter * 32 + lane;
    int g = 0;
    for (int work = blockIdx.x; work < items * parts; work += gridDim.x, g++) {
      const int set = g & 1, item = work / parts, co0 = (work - item * parts) * COUT;
      int z0;
      const int len = slices(item, z0);
      ok = __all_sync(0xffffffffu, tc::mbar_wait(&acc_full[set], (uint32_t)(g >> 1) & 1u, kWaitLimit));
      if (!ok) break;
      tc::fence_after_sync();
      const int vx = (item % tiles_x) * 8 + row % 8, vy = ((item / tiles_x) % tiles_y) * 16 + row / 8;
      const int n = item / (cols * runs);
#pragma unroll 1
      for (int sl = 0; sl < len; sl++) {
        const long long vox = (((long long)n * (a.D + 2) + z0 + sl + 1) * (a.H + 2) + vy + 1) * (a.W + 2) + vx + 1;
        conv_rows_out<COUT>(a, tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(set * C::kSet + sl * COUT),
                            vox * a.out_ctot + a.out_coff + co0, bias + co0);
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acc_empty[set]);
    }
  }
  if (!ok) atomicExch(err, 1);
  tc::fence_before_sync();
  __syncthreads();
  __syncwarp();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

// Convolution of 32, 64 or 128 output channels on grids 8 high (y), where
// k_conv_r's tiles do not fit, in its order of products; one persistent block
// per SM.  An output tile is 16 (x) x 8 (y) x 2 (z) voxels.  For each 32-channel chunk and each x-shift dx, one 5-D TMA
// box brings the input block x0+dx .. x0+dx+15, y0-1 .. y0+8, z0-1 .. z0+2
// (rows of 64 B, x fastest) into shared memory, with the weights of the nine
// taps of that dx.  The 128 rows of input plane zi shifted by dy start at row
// (zi * 10 + dy) * 16.  Two accumulator sets alternate between tiles, so four
// warps convert and write tile t while the copies and MMAs of tile t + 1 run.
// Bound: operand staging.
template <int COUT>
struct ConvZ {
  static constexpr int S = 2;
  static constexpr int kTileA = (S + 2) * 160 * 64;
  static constexpr int kTileB = 9 * COUT * 64;
  static constexpr int kStages = COUT == 32 ? 3 : 2;
  static constexpr int kSmem = kStages * (kTileA + kTileB) + 1024;
  static constexpr bool kStack = 3 * COUT <= 256;
  static constexpr int kSet = S * COUT;  // TMEM columns of one accumulator set
  static_assert(kSmem <= 227 * 1024 - 2048 && 2 * kSet <= 512, "stage budget");
};

template <int COUT>
__global__ void __launch_bounds__(192, 1)
k_conv_z(const __grid_constant__ CUtensorMap tx, const __grid_constant__ CUtensorMap tw, ConvArgs a, int items,
         int *err) {
  after_previous();
  using C = ConvZ<COUT>;
  constexpr int NST = C::kStages, S = C::S;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u;
  uint8_t *tA = smem_raw + pad;
  constexpr uint32_t tap_b = COUT * 64;  // one tap's weights
  uint8_t *tB = tA + NST * C::kTileA;
  __shared__ uint64_t full[NST], empty[NST], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base;
  __shared__ float bias[COUT];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_x = a.W / 16, tiles_y = a.H / 8, tiles_z = a.D / S;
  const int nck = a.cin / 32;
  const int nk = 3 * nck;  // stages of a tile: (chunk, dx)
  if (warp == 0) {
    tc::tmem_alloc(&tmem_base, 2 * C::kSet);
    tc::tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < NST; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], 4);
    }
    tc::fence_mbar_init();
  }
  for (int c = threadIdx.x; c < COUT; c += 192) bias[c] = a.bias ? a.bias[c] : 0.0f;
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  bool ok = true;
  if (warp == 0 && tc::elect_one()) {  // copies
    int s = 0, round = 0;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      const int x0 = (item % tiles_x) * 16, y0 = ((item / tiles_x) % tiles_y) * 8,
                z0 = ((item / (tiles_x * tiles_y)) % tiles_z) * S, n = item / (tiles_x * tiles_y * tiles_z);
      for (int ck = 0; ck < nck && ok; ck++)
        for (int dx = 0; dx < 3; dx++) {
          if (round > 0 && !tc::mbar_wait(&empty[s], (uint32_t)(round - 1) & 1u, kWaitLimit)) {
            ok = false;
            break;
          }
          tc::mbar_expect_tx(&full[s], (uint32_t)(C::kTileA + C::kTileB));
          // padded coordinates: interior voxel v is v + 1, so x0 + dx is x0 + dx - 1 inside
          tc::tma_load_5d(tA + s * C::kTileA, &tx, &full[s], a.in_coff + ck * 32, x0 + dx, y0, z0, n);
          uint8_t *bs = tB + s * C::kTileB;
          for (int dy = 0; dy < 3; dy++)
            for (int dz = 0; dz < 3; dz++)
              tc::tma_load_2d(bs + (dy * 3 + 2 - dz) * tap_b, &tw, &full[s], 0, ((dz * 9 + dy * 3 + dx) * nck + ck) * COUT);
          if (++s == NST) { s = 0; ++round; }
        }
    }
    // the copies issued have landed before the block ends
    const int issued = round * NST + s;
    for (int kt = issued > NST ? issued - NST : 0; kt < issued; kt++)
      if (!tc::mbar_wait(&full[kt % NST], (kt / NST) & 1, kWaitLimit)) atomicExch(err, 2);
  } else if (warp == 1 && tc::elect_one()) {  // MMAs
    int s = 0, round = 0, g = 0;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x, g++) {
      const int set = g & 1;
      if (g >= 2 && !tc::mbar_wait(&acc_empty[set], (uint32_t)((g >> 1) - 1) & 1u, kWaitLimit)) {
        ok = false;
        break;
      }
      tc::fence_after_sync();
      const uint32_t d0 = tmem + (uint32_t)(set * C::kSet);
      for (int kt = 0; kt < nk; kt++) {
        if (!tc::mbar_wait(&full[s], (uint32_t)round & 1u, kWaitLimit)) {
          ok = false;
          break;
        }
        tc::fence_after_sync();
        const uint64_t a0 = tc::smem_desc(tA + s * C::kTileA, tc::kSwizzle64, 64);
        const uint64_t b0 = tc::smem_desc(tB + s * C::kTileB, tc::kSwizzle64, 64);
#pragma unroll
        for (int zi = 0; zi < S + 2; zi++) {
          constexpr int kLast = S - 1;
          const int lo = zi > kLast ? zi - kLast : 0, hi = zi < 2 ? zi : 2;  // dz of the slices this plane serves
#pragma unroll
          for (int dy = 0; dy < 3; dy++) {
            // start-address fields count 16-byte units; rows of 64 B
            const uint64_t ad = a0 + (uint64_t)((zi * 10 + dy) * 16 * 4);
            const uint64_t bd = b0 + (uint64_t)(dy * 3 * (tap_b >> 4));
            auto mma = [&](int dz_lo, int dz_hi, int kk, uint32_t acc) {
              tc::mma_bf16(d0 + (uint32_t)((zi - dz_hi) * COUT), ad + 2 * kk,
                           bd + (uint64_t)((2 - dz_hi) * (tap_b >> 4)) + 2 * kk,
                           tc::idesc_bf16(128, (dz_hi - dz_lo + 1) * COUT), acc);
            };
            for (int kk = 0; kk < 2; kk++) {
              // the first product of an accumulator (dz = 0, dy = 0) overwrites it
              const bool fresh = kt == 0 && dy == 0 && kk == 0 && lo == 0;
              if (!C::kStack) {
                for (int dz = lo; dz <= hi; dz++) mma(dz, dz, kk, !(fresh && dz == 0));
              } else if (fresh) {
                if (hi > 0) mma(1, hi, kk, 1);
                mma(0, 0, kk, 0);
              } else {
                mma(lo, hi, kk, 1);
              }
            }
          }
        }
        tc::mma_commit(&empty[s]);
        if (++s == NST) { s = 0; ++round; }
      }
      tc::mma_commit(&acc_full[set]);
    }
  } else if (warp >= 2) {  // accumulators to memory
    const int quarter = warp & 3, row = quarter * 32 + lane;
    int g = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x, g++) {
      const int set = g & 1;
      ok = __all_sync(0xffffffffu, tc::mbar_wait(&acc_full[set], (uint32_t)(g >> 1) & 1u, kWaitLimit));
      if (!ok) break;
      tc::fence_after_sync();
      const int vx = (item % tiles_x) * 16 + row % 16, vy = ((item / tiles_x) % tiles_y) * 8 + row / 16;
      const int z0 = ((item / (tiles_x * tiles_y)) % tiles_z) * S, n = item / (tiles_x * tiles_y * tiles_z);
#pragma unroll 1
      for (int sl = 0; sl < S; sl++) {
        const long long vox = (((long long)n * (a.D + 2) + z0 + sl + 1) * (a.H + 2) + vy + 1) * (a.W + 2) + vx + 1;
        const long long at = vox * a.out_ctot + a.out_coff;
        conv_rows_out<COUT>(a, tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(set * C::kSet + sl * COUT), at, bias);
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acc_empty[set]);
    }
  }
  if (!ok) atomicExch(err, 1);
  tc::fence_before_sync();
  __syncthreads();
  __syncwarp();
  if (warp == 0) tc::tmem_dealloc(tmem, 2 * C::kSet);
}

// Periodic halo of channels [coff, coff + nch) (nch a multiple of 8): every
// halo voxel gets its wrapped interior voxel.  The halo voxels of a sample
// are enumerated face by face: the planes z = 0 and z = D + 1 whole, then
// for interior z the rows y = 0 and y = H + 1, then for interior z, y the
// columns x = 0 and x = W + 1.
// I: 32-bit unless the vectors of all halo voxels do not fit it (64-bit
// divisions took 4.5 us of a launch where the copies take 2).
template <typename I>
__global__ void __launch_bounds__(256) k_halo(__nv_bfloat16 *buf, int B, int D, int H, int W, int ctot, int coff, int nch) {
  after_previous();
  const I row = (I)(W + 2), face = (I)(H + 2) * row, side = (I)D * row, wall = (I)D * (I)H;
  const I per = 2 * (face + side + wall), nv = (I)(nch / 8), total = (I)B * per * nv;
  for (I e = (I)blockIdx.x * 256 + threadIdx.x; e < total; e += (I)gridDim.x * 256) {
    const I h = e / nv;
    const int cv = (int)(e - h * nv), n = (int)(h / per);
    I r = h - (I)n * per;
    int x, y, z;
    if (r < 2 * face) {
      z = r < face ? 0 : D + 1;
      if (r >= face) r -= face;
      y = (int)(r / row);
      x = (int)(r - (I)y * row);
    } else if ((r -= 2 * face) < 2 * side) {
      y = r < side ? 0 : H + 1;
      if (r >= side) r -= side;
      z = (int)(r / row);
      x = (int)(r - (I)z * row);
      z++;
    } else {
      r -= 2 * side;
      x = r < wall ? 0 : W + 1;
      if (r >= wall) r -= wall;
      z = (int)(r / (I)H);
      y = 1 + (int)(r - (I)z * (I)H);
      z++;
    }
    const int sx = x == 0 ? W : (x == W + 1 ? 1 : x);
    const int sy = y == 0 ? H : (y == H + 1 ? 1 : y);
    const int sz = z == 0 ? D : (z == D + 1 ? 1 : z);
    const long long src = (((long long)n * (D + 2) + sz) * (H + 2) + sy) * (W + 2) + sx;
    const long long dst = (((long long)n * (D + 2) + z) * (H + 2) + y) * (W + 2) + x;
    *(uint4 *)(buf + dst * ctot + coff + 8 * cv) = *(const uint4 *)(buf + src * ctot + coff + 8 * cv);
  }
}

// 5-D map of a padded channels-last buffer: box of 32 channels x wbox x
// hbox x dbox x 1 (64-byte rows, 64-byte swizzle)
bool make_map_act(CUtensorMap *map, const void *ptr, int B, int D, int H, int W, int ctot, int wbox, int hbox,
                  int dbox) {
  EncodeTiled enc = encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[5] = {(cuuint64_t)ctot, (cuuint64_t)W + 2, (cuuint64_t)H + 2, (cuuint64_t)D + 2,
                              (cuuint64_t)B};
  const cuuint64_t s1 = (cuuint64_t)ctot * 2;
  const cuuint64_t strides[4] = {s1, s1 * (W + 2), s1 * (W + 2) * (H + 2), s1 * (W + 2) * (H + 2) * (D + 2)};
  const cuuint32_t box[5] = {32, (cuuint32_t)wbox, (cuuint32_t)hbox, (cuuint32_t)dbox, 1};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void *>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// 2-D map of rows of 32 BF16 (64 bytes), box of box_rows rows, 64-byte swizzle
bool make_map_rows32(CUtensorMap *map, const void *ptr, long long rows, int box_rows) {
  EncodeTiled enc = encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[2] = {32, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {64};
  const cuuint32_t box[2] = {32, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ---- weight gradients ------------------------------------------------------------
// dW[tap][co][ci] = sum_u dY[u - off(tap)][co] * X[u][ci] over all voxels u
// of all samples.  Both operands are channel-major with K = voxels flattened
// over the padded volume: row pitch Wp (a multiple of 8, >= W + 2), plane
// (H + 2) * Wp, sample stride pstride (a multiple of 64).  X's copy has a
// zero halo, so halo positions add nothing; dY's three copies S_dx (dx =
// 0, 1, 2) carry the periodic halo and the x part of the tap offset, so the
// y and z parts are aligned flat shifts of the TMA box.  Taps are stacked
// along M (128 rows = taps x output channels); K is split over blocks into
// FP32 partial sums, added in a fixed order afterwards.
struct WgradArgs {
  int cin, cout, co_rows, taps_per_tile, co_tiles;
  int ntile;
  int Wp;
  int plane;
  long long k_tiles;
  int splits;
  int tmem_cols;
  float *partial;  // [splits][27][cout][cin]
};

constexpr int kWgTileA = 128 * 128;  // 128 rows x 64 K x 2 B
constexpr int kWgTileB = 256 * 128;  // up to 256 rows
constexpr int kWgSmem = kStages * (kWgTileA + kWgTileB) + 1024;

// B stages hold ntile rows of 128 bytes (the dynamic shared memory is sized
// by ntile), so layers with up to 64 input channels fit two blocks per SM.
__global__ void __launch_bounds__(128, 2)
k_wgrad(const __grid_constant__ CUtensorMap a0, const __grid_constant__ CUtensorMap a1,
        const __grid_constant__ CUtensorMap a2, const __grid_constant__ CUtensorMap tb, WgradArgs w, int *err) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u;
  uint8_t *tA = smem_raw + pad;
  uint8_t *tB = tA + kStages * kWgTileA;
  const int tile_b = w.ntile * 128;  // bytes of one B stage (a multiple of 2048)
  __shared__ uint64_t full[kStages], empty[kStages], done;
  __shared__ uint32_t tmem_base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = blockIdx.x / w.co_tiles, cot = blockIdx.x % w.co_tiles;
  const int tap0 = group * w.taps_per_tile, co0 = cot * w.co_rows, ci0 = blockIdx.y * w.ntile;
  // K tiles z, z + splits, z + 2 splits, ... (z = blockIdx.z): the blocks
  // of one launch work through one run of consecutive tiles at a time, so
  // the windows that other taps read again (up to a plane further on) are
  // still in L2
  const long long kz = blockIdx.z;
  const int nk = kz < w.k_tiles ? (int)((w.k_tiles - kz + w.splits - 1) / w.splits) : 0;
  const uint32_t bytes_a = 128u * 128u, bytes_b = (uint32_t)w.ntile * 128u;
  if (warp == 0) {
    tc::tmem_alloc(&tmem_base, (uint32_t)w.tmem_cols);
    tc::tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < kStages; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(&done, 1);
    tc::fence_mbar_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  bool ok = true;
  int issued = 0;
  if (warp == 0 && tc::elect_one()) {
    for (int kt = 0; kt < nk; kt++) {
      const int s = kt % kStages;
      if (kt >= kStages && !tc::mbar_wait(&empty[s], ((kt / kStages) - 1) & 1, kWaitLimit)) {
        ok = false;
        break;
      }
      const int k0 = (int)((kz + (long long)kt * w.splits) * 64);
      tc::mbar_expect_tx(&full[s], bytes_a + bytes_b);
      for (int tl = 0; tl < w.taps_per_tile; tl++) {
        const int tap = tap0 + tl < 27 ? tap0 + tl : 26;  // rows past tap 26 are discarded
        const int dz = tap / 9, dy = (tap / 3) % 3, dx = tap % 3;
        const int x = k0 - (dy - 1) * w.Wp - (dz - 1) * w.plane;
        const CUtensorMap *am = dx == 0 ? &a0 : (dx == 1 ? &a1 : &a2);
        tc::tma_load_2d(tA + s * kWgTileA + tl * w.co_rows * 128, am, &full[s], x, co0);
      }
      tc::tma_load_2d(tB + s * tile_b, &tb, &full[s], k0, ci0);
      issued = kt + 1;
    }
  } else if (warp == 1 && tc::elect_one()) {
    const uint32_t idesc = tc::idesc_bf16(128, w.ntile);
    for (int kt = 0; kt < nk; kt++) {
      const int s = kt % kStages;
      if (!tc::mbar_wait(&full[s], (kt / kStages) & 1, kWaitLimit)) {
        ok = false;
        break;
      }
      tc::fence_after_sync();
      const uint64_t ad = tc::smem_desc(tA + s * kWgTileA, tc::kSwizzle128, 128);
      const uint64_t bd = tc::smem_desc(tB + s * tile_b, tc::kSwizzle128, 128);
#pragma unroll
      for (int kk = 0; kk < 4; kk++) tc::mma_bf16(tmem, ad + 2 * kk, bd + 2 * kk, idesc, (kt | kk) != 0);
      tc::mma_commit(&empty[s]);
    }
    tc::mma_commit(&done);
  }
  __syncwarp();
  const bool okd = __all_sync(0xffffffffu, tc::mbar_wait(&done, 0, kWaitLimit));
  tc::fence_after_sync();
  if (okd) {
    const int r = warp * 32 + lane;
    const int tap = tap0 + r / w.co_rows, co = co0 + r % w.co_rows;
    float *dst = w.partial + (((long long)blockIdx.z * 27 + tap) * w.cout + co) * w.cin + ci0;
#pragma unroll 1
    for (int c = 0; c < w.ntile; c += 8) {
      float v[8];
      tc::tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
      if (nk == 0) {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = 0.0f;
      }
      if (tap < 27) {
        ((float4 *)(dst + c))[0] = make_float4(v[0], v[1], v[2], v[3]);
        ((float4 *)(dst + c))[1] = make_float4(v[4], v[5], v[6], v[7]);
      }
    }
  }
  if (!ok || !okd) atomicExch(err, 1);
  if (warp == 0 && tc::elect_one()) {
    for (int kt = issued > kStages ? issued - kStages : 0; kt < issued; kt++)
      if (!tc::mbar_wait(&full[kt % kStages], (kt / kStages) & 1, kWaitLimit)) atomicExch(err, 2);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, (uint32_t)w.tmem_cols);
}

// ---- weight gradients, taps stacked along N ----------------------------------
// The same sum with the y/z part of the tap offset moved to the input:
// dW[tap][co][ci] = sum_v S_dx[v][co] * X[v + s][ci], s = (dy - 1) * Wp +
// (dz - 1) * plane (v = u - s; X is zero outside its interior and TMA fills
// zeros outside the array, so the terms are the same).  Per K tile of 64
// flat positions a block then loads the three dY copies once (M: dx blocks
// of cout rows, 128 rows = up to 3 copies, a 4th block of 32 rows for cout =
// 32 is never loaded and its accumulator rows are dropped) and the input
// window at nt shifts s (N: nt taps x cc input channels, up to 288 rows in
// two MMAs), instead of 27 shifted dY tiles against one input tile: the
// operand bytes staged per FLOP drop 2.7x for 32 channels, and every MMA
// is 128 x 144 instead of 128 x 32.
struct WgradNArgs {
  int cin, cout;
  int dpm;        // dx copies per M tile
  int nt;         // (dy, dz) taps per block
  int groups;     // tap groups: ceil(9 / nt)
  int cc;         // input channels per block (cin, or a divisor of it)
  int ci_chunks;  // cin / cc
  int n_rows;     // nt * cc: accumulator columns
  int n_mma;      // columns per MMA (n_rows split into equal parts of <= 256)
  int Wp, plane;
  long long k_tiles;
  int splits;
  int tmem_cols;
  float *partial;  // [splits][27][cout][cin]
  // one TMA box per stage and operand where the layout allows it: the dpm
  // dY copies as one 3-D box (copies equally spaced in memory), the nt
  // input windows as one 4-D box (nt = 9: dy, dz = 0..2; nt = 3: dy =
  // 0..2 at one dz) of a view with strides Wp and plane along dy and dz;
  // the 4-D box is used where all its windows lie inside the array
  int a3, b4;
  long long b4_dim0;  // first-axis extent of the window view
  // dY copies in K-tile blocks [tile][3][cout][64] (slbc_tc_cmajor_tiles):
  // a0 boxes dpm * cout rows of a tile, a1 boxes cout rows
  int a_tiles;
};

constexpr int kWgnMaxRows = 288;
constexpr int kWgnSmem = kStages * (kWgTileA + kWgnMaxRows * 128) + 1024;

// Block decomposition of k_wgrad_n and k_wgrad_f for (cin, cout); false when it
// does not apply (cout not 32, 64 or 128).  Channels per block come in multiples
// of `step` (k_wgrad_f: 32, the channels of its boxes).
bool wgrad_n_plan(int cin, int cout, WgradNArgs &w, int step = 16) {
  if (!(cout == 32 || cout == 64 || cout == 128) || cin < 16 || cin % 16) return false;
  w.cin = cin;
  w.cout = cout;
  w.dpm = std::min(128 / cout, 3);
  int cc = cin;
  if (cc > 256) {
    cc = 0;
    for (int c = 256; c >= step; c -= step)
      if (cin % c == 0) { cc = c; break; }
    if (!cc) return false;
  }
  int groups = (9 * cc + kWgnMaxRows - 1) / kWgnMaxRows, nt = (9 + groups - 1) / groups;
  while (nt * cc > kWgnMaxRows) {
    groups++;
    nt = (9 + groups - 1) / groups;
  }
  w.cc = cc;
  w.ci_chunks = cin / cc;
  w.nt = nt;
  w.groups = groups;
  w.n_rows = nt * cc;
  const int parts = (w.n_rows + 255) / 256;
  if (w.n_rows % (16 * parts)) return false;
  w.n_mma = w.n_rows / parts;
  w.tmem_cols = 32;
  while (w.tmem_cols < w.n_rows) w.tmem_cols *= 2;
  return true;
}

int wgrad_n_ctas(const WgradNArgs &w) { return ((3 + w.dpm - 1) / w.dpm) * w.groups * w.ci_chunks; }

__global__ void __launch_bounds__(128, 1)
k_wgrad_n(const __grid_constant__ CUtensorMap a0, const __grid_constant__ CUtensorMap a1,
          const __grid_constant__ CUtensorMap a2, const __grid_constant__ CUtensorMap tb,
          const __grid_constant__ CUtensorMap a_all, const __grid_constant__ CUtensorMap b_win, WgradNArgs w,
          int *err) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u;
  uint8_t *tA = smem_raw + pad;
  uint8_t *tB = tA + kStages * kWgTileA;
  const int tile_b = w.n_rows * 128;  // bytes of one B stage (a multiple of 2048)
  __shared__ uint64_t full[kStages], empty[kStages], done;
  __shared__ uint32_t tmem_base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunk = blockIdx.x % w.ci_chunks;
  const int g = (blockIdx.x / w.ci_chunks) % w.groups;
  const int mt = blockIdx.x / (w.ci_chunks * w.groups);
  const int ci0 = chunk * w.cc;
  // K tiles z, z + splits, z + 2 splits, ... (z = blockIdx.z): the blocks
  // of one launch work through one run of consecutive tiles at a time, so
  // the windows that other taps read again (up to a plane further on) are
  // still in L2
  const long long kz = blockIdx.z;
  const int nk = kz < w.k_tiles ? (int)((w.k_tiles - kz + w.splits - 1) / w.splits) : 0;
  // bytes landing per stage: the dY copies and input windows actually loaded
  int a_blocks = 0, b_taps = 0;
  for (int d = 0; d < w.dpm; d++) a_blocks += mt * w.dpm + d < 3;
  for (int t = 0; t < w.nt; t++) b_taps += g * w.nt + t < 9;
  const uint32_t bytes = (uint32_t)(a_blocks * w.cout * 128 + b_taps * w.cc * 128);
  if (warp == 0) {
    tc::tmem_alloc(&tmem_base, (uint32_t)w.tmem_cols);
    tc::tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < kStages; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(&done, 1);
    tc::fence_mbar_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  bool ok = true;
  int issued = 0;
  if (warp == 0 && tc::elect_one()) {
    for (int kt = 0; kt < nk; kt++) {
      const int s = kt % kStages;
      if (kt >= kStages && !tc::mbar_wait(&empty[s], ((kt / kStages) - 1) & 1, kWaitLimit)) {
        ok = false;
        break;
      }
      const int k0 = (int)((kz + (long long)kt * w.splits) * 64);
      tc::mbar_expect_tx(&full[s], bytes);
      if (w.a_tiles) {
        if (a_blocks == w.dpm) {
          tc::tma_load_3d(tA + s * kWgTileA, &a0, &full[s], 0, mt * w.dpm * w.cout, k0 >> 6);
        } else {
          for (int d = 0; d < a_blocks; d++)
            tc::tma_load_3d(tA + s * kWgTileA + d * w.cout * 128, &a1, &full[s], 0, (mt * w.dpm + d) * w.cout, k0 >> 6);
        }
      } else if (w.a3 && a_blocks == w.dpm) {
        tc::tma_load_3d(tA + s * kWgTileA, &a_all, &full[s], k0, 0, mt * w.dpm);
      } else {
        for (int d = 0; d < w.dpm; d++) {
          const int dx = mt * w.dpm + d;
          if (dx >= 3) break;
          const CUtensorMap *am = dx == 0 ? &a0 : (dx == 1 ? &a1 : &a2);
          tc::tma_load_2d(tA + s * kWgTileA + d * w.cout * 128, am, &full[s], k0, 0);
        }
      }
      // first window of the group: dy = 0 at the group's first dz
      const long long xw = (long long)k0 - w.Wp + ((g * w.nt) / 3 - 1) * (long long)w.plane;
      if (w.b4 && b_taps == w.nt && xw >= 0 && xw + 64 <= w.b4_dim0) {
        tc::tma_load_4d(tB + s * tile_b, &b_win, &full[s], (int)xw, ci0, 0, 0);
      } else {
        for (int t = 0; t < w.nt; t++) {
          const int yz = g * w.nt + t;
          if (yz >= 9) break;
          const int dy = yz % 3, dz = yz / 3;
          // may start before 0 or end past the array: TMA fills zeros there
          const int x = k0 + (dy - 1) * w.Wp + (dz - 1) * w.plane;
          tc::tma_load_2d(tB + s * tile_b + t * w.cc * 128, &tb, &full[s], x, ci0);
        }
      }
      issued = kt + 1;
    }
  } else if (warp == 1 && tc::elect_one()) {
    const uint32_t idesc = tc::idesc_bf16(128, w.n_mma);
    const int parts = w.n_rows / w.n_mma;
    for (int kt = 0; kt < nk; kt++) {
      const int s = kt % kStages;
      if (!tc::mbar_wait(&full[s], (kt / kStages) & 1, kWaitLimit)) {
        ok = false;
        break;
      }
      tc::fence_after_sync();
      const uint64_t ad = tc::smem_desc(tA + s * kWgTileA, tc::kSwizzle128, 128);
      for (int j = 0; j < parts; j++) {
        const uint64_t bd = tc::smem_desc(tB + s * tile_b + j * w.n_mma * 128, tc::kSwizzle128, 128);
#pragma unroll
        for (int kk = 0; kk < 4; kk++)
          tc::mma_bf16(tmem + (uint32_t)(j * w.n_mma), ad + 2 * kk, bd + 2 * kk, idesc, (kt | kk) != 0);
      }
      tc::mma_commit(&empty[s]);
    }
    tc::mma_commit(&done);
  }
  __syncwarp();
  const bool okd = __all_sync(0xffffffffu, tc::mbar_wait(&done, 0, kWaitLimit));
  tc::fence_after_sync();
  if (okd) {
    const int r = warp * 32 + lane;
    const int d = r / w.cout, co = r % w.cout;
    const int dx = mt * w.dpm + d;
    const bool row_ok = d < w.dpm && dx < 3;
#pragma unroll 1
    for (int c = 0; c < w.n_rows; c += 8) {
      float v[8];
      tc::tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);  // whole warp
      if (nk == 0) {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = 0.0f;
      }
      const int t = c / w.cc, yz = g * w.nt + t;
      if (row_ok && yz < 9) {
        const int tap = (yz / 3) * 9 + (yz % 3) * 3 + dx;
        float *dst = w.partial + (((long long)blockIdx.z * 27 + tap) * w.cout + co) * w.cin + ci0 + c % w.cc;
        ((float4 *)dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
        ((float4 *)dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
      }
    }
  }
  if (!ok || !okd) atomicExch(err, 1);
  if (warp == 0 && tc::elect_one()) {
    for (int kt = issued > kStages ? issued - kStages : 0; kt < issued; kt++)
      if (!tc::mbar_wait(&full[kt % kStages], (kt / kStages) & 1, kWaitLimit)) atomicExch(err, 2);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, (uint32_t)w.tmem_cols);
}

// The same sums, tile by tile and in the same order, from flat copies that keep
// the channels last (k_flat): position f = (z * (H + 2) + y) * Wp + x of a sample
// is a row of `ctot` channels.  K is then the row index of the staged tiles (MN-
// major operands), so a tile of 64 positions is 64 rows of 64 or 128 bytes and
// the three x-shifted views of dY are one tile of 72 rows read from three
// starting rows: M block i of the operand begins i rows further on and holds tap
// dx = 2 - i.  The input's nt windows are boxes of 64 rows x 32 channels.
//
// Against k_wgrad_n it stages 40 instead of 48 KB per K tile at 32 channels, and
// the copies are one pass each without a transpose, one of dY instead of three.
// Bound: the tensor pipe (71-83% active at 32 output channels on 4 x 64^3, with
// L2 at 69% and shared memory at 67-78%; 61% at 64 on 4 x 32^3).  Measured, the
// 13 layers of a training iteration of 4 x 64^3: 1228 -> 735 us, their copies 835
// -> 451 us.
constexpr int kWgfTileA = 72 * 128 * 2;
constexpr int kWgfSmem = kStages * (kWgfTileA + kWgnMaxRows * 128) + 1024;

__global__ void __launch_bounds__(128, 1)
k_wgrad_f(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
          const __grid_constant__ CUtensorMap b_win, WgradNArgs w, int *err) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u;
  uint8_t *tA = smem_raw + pad;
  uint8_t *tB = tA + kStages * kWgfTileA;
  const int tile_b = w.n_rows * 128;  // bytes of one B stage (a multiple of 4096)
  __shared__ uint64_t full[kStages], empty[kStages], done;
  __shared__ uint32_t tmem_base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunk = blockIdx.x % w.ci_chunks;
  const int g = (blockIdx.x / w.ci_chunks) % w.groups;
  const int mt = blockIdx.x / (w.ci_chunks * w.groups);
  const int ci0 = chunk * w.cc;
  const long long kz = blockIdx.z;  // K tiles kz, kz + splits, ...
  const int nk = kz < w.k_tiles ? (int)((w.k_tiles - kz + w.splits - 1) / w.splits) : 0;
  int b_taps = 0;
  for (int t = 0; t < w.nt; t++) b_taps += g * w.nt + t < 9;
  const int row_a = w.cout == 32 ? 64 : 128;  // bytes of an A row: 32 or 64 channels
  const uint32_t bytes = (uint32_t)(72 * w.cout * 2 + b_taps * w.cc * 128);
  if (warp == 0) {
    tc::tmem_alloc(&tmem_base, (uint32_t)w.tmem_cols);
    tc::tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < kStages; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(&done, 1);
    tc::fence_mbar_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  bool ok = true;
  if (warp == 0 && tc::elect_one()) {
    int issued = 0;
    for (int kt = 0; kt < nk; kt++) {
      const int s = kt % kStages;
      if (kt >= kStages && !tc::mbar_wait(&empty[s], ((kt / kStages) - 1) & 1, kWaitLimit)) {
        ok = false;
        break;
      }
      const int k0 = (int)((kz + (long long)kt * w.splits) * 64);
      tc::mbar_expect_tx(&full[s], bytes);
      // rows before 0 and past the end are zero
      tc::tma_load_3d(tA + s * kWgfTileA, &ta, &full[s], 0, k0 - 1, 0);
      // first window of the group: dy = 0 at the group's first dz
      const long long xw = (long long)k0 - w.Wp + ((g * w.nt) / 3 - 1) * (long long)w.plane;
      if (w.b4 && b_taps == w.nt && xw >= 0 && xw + 64 <= w.b4_dim0) {
        tc::tma_load_5d(tB + s * tile_b, &b_win, &full[s], 0, (int)xw, ci0 / 32, 0, 0);
      } else {
        for (int t = 0; t < b_taps; t++) {
          const int yz = g * w.nt + t, dy = yz % 3, dz = yz / 3;
          tc::tma_load_3d(tB + s * tile_b + t * w.cc * 128, &tb, &full[s], 0, k0 + (dy - 1) * w.Wp + (dz - 1) * w.plane,
                          ci0 / 32);
        }
      }
      issued = kt + 1;
    }
    for (int kt = issued > kStages ? issued - kStages : 0; kt < issued; kt++)
      if (!tc::mbar_wait(&full[kt % kStages], (kt / kStages) & 1, kWaitLimit)) atomicExch(err, 2);
  } else if (warp == 1 && tc::elect_one()) {
    // columns in one MMA or two, whole blocks of 32 each
    const int n1 = w.n_rows <= 256 ? w.n_rows : (w.n_rows / 64 + 1) / 2 * 64 > 256 ? 256 : (w.n_rows / 64 + 1) / 2 * 64;
    const int n2 = w.n_rows - n1;
    const uint32_t id1 = tc::idesc_bf16_mn(128, n1), id2 = tc::idesc_bf16_mn(128, n2);
    // the M blocks: one row further on for the next dx, or (128 output
    // channels) the other 64 channels
    const uint32_t mn = w.cout == 128 ? 72 * 128 : row_a;
    const uint64_t a0 = tc::smem_desc_mn(tA, w.cout == 32 ? tc::kSwizzle64 : tc::kSwizzle128, row_a, mn) +
                        (uint64_t)(mt * w.dpm * (row_a >> 4));
    const uint64_t b0 = tc::smem_desc_mn(tB, tc::kSwizzle64, 64, 64 * 64);
    for (int kt = 0; kt < nk; kt++) {
      const int s = kt % kStages;
      if (!tc::mbar_wait(&full[s], (kt / kStages) & 1, kWaitLimit)) {
        ok = false;
        break;
      }
      tc::fence_after_sync();
      const uint64_t ad = a0 + (uint64_t)(s * (kWgfTileA >> 4)), bd = b0 + (uint64_t)(s * (tile_b >> 4));
#pragma unroll
      for (int kk = 0; kk < 4; kk++)
        tc::mma_bf16(tmem, ad + (uint64_t)(kk * row_a), bd + (uint64_t)(kk * 64), id1, (kt | kk) != 0);
      if (n2) {
        const uint64_t be = bd + (uint64_t)(n1 / 32 * (64 * 64 >> 4));
#pragma unroll
        for (int kk = 0; kk < 4; kk++)
          tc::mma_bf16(tmem + (uint32_t)n1, ad + (uint64_t)(kk * row_a), be + (uint64_t)(kk * 64), id2, (kt | kk) != 0);
      }
      tc::mma_commit(&empty[s]);
    }
    tc::mma_commit(&done);
  }
  __syncwarp();
  const bool okd = __all_sync(0xffffffffu, tc::mbar_wait(&done, 0, kWaitLimit));
  tc::fence_after_sync();
  if (okd) {
    const int r = warp * 32 + lane, d = r / w.cout, co = r % w.cout, off = mt * w.dpm + d;
    const bool row_ok = d < w.dpm && off < 3;
#pragma unroll 1
    for (int c = 0; c < w.n_rows; c += 8) {
      float v[8];
      tc::tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);  // whole warp
      if (nk == 0) {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = 0.0f;
      }
      const int yz = g * w.nt + c / w.cc;
      if (row_ok && yz < 9) {
        const int tap = yz / 3 * 9 + yz % 3 * 3 + 2 - off;
        float *dst = w.partial + (((long long)blockIdx.z * 27 + tap) * w.cout + co) * w.cin + ci0 + c % w.cc;
        ((float4 *)dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
        ((float4 *)dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
      }
    }
  }
  if (!ok || !okd) atomicExch(err, 1);
  tc::fence_before_sync();
  __syncthreads();
  __syncwarp();
  if (warp == 0) tc::tmem_dealloc(tmem, (uint32_t)w.tmem_cols);
}

// Flat copies of channels [coff, coff + nch) with the row pitch Wp:
// dst[n * pstride + (z * (H + 2) + y) * Wp + x][c] = src[n][z][y][x][coff + c], 0
// beyond x = W + 1 (zero_halo: interior voxels only).  A warp takes a row of
// positions at a time (the last `row` of a sample: what is left of its stride).
// Bound: HBM.
__global__ void __launch_bounds__(256) k_flat(const __nv_bfloat16 *src, int B, int D, int H, int W, int ctot, int coff,
                                              int nch, int Wp, int pstride, int zero_halo, __nv_bfloat16 *dst) {
  after_previous();
  const int rows = (D + 2) * (H + 2), nv = nch / 8, tail = pstride - rows * Wp;
  const int lane = threadIdx.x & 31, step = (int)gridDim.x * 8;
  for (int q = (int)blockIdx.x * 8 + (int)(threadIdx.x >> 5); q < B * (rows + 1); q += step) {
    const int n = q / (rows + 1), row = q - n * (rows + 1), z = row / (H + 2), y = row - z * (H + 2);
    const bool in = row < rows && (!zero_halo || (z >= 1 && z <= D && y >= 1 && y <= H));
    const int len = (row < rows ? Wp : tail) * nv, lo = zero_halo ? 1 : 0, hi = zero_halo ? W : W + 1;
    const __nv_bfloat16 *from = src + ((long long)n * rows + row) * (W + 2) * ctot + coff;
    uint4 *to = (uint4 *)(dst + ((long long)n * pstride + (long long)row * Wp) * nch);
#pragma unroll 4
    for (int i = lane; i < len; i += 32) {
      const int x = (int)((unsigned)i / (unsigned)nv), cv = i - x * nv;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (in && x >= lo && x <= hi) v = *(const uint4 *)(from + (long long)x * ctot + 8 * cv);
      to[i] = v;
    }
  }
}

// dw[i] = sum over splits of partial[s][i], in split order
__global__ void k_sum_splits(const float *partial, long long n, int splits, float *dw) {
  after_previous();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float v = 0.0f;
    for (int s = 0; s < splits; s++) v += partial[(long long)s * n + i];
    dw[i] = v;
  }
}

// Channel-major flat copies of channels [coff, coff + nch) of a padded
// channels-last buffer: dst[c][n * pstride + (z * (H + 2) + y) * Wp + x] =
// src[n][z][y][x - shift][coff + c] for 0 <= x - shift <= W + 1 (0 beyond;
// zero_halo: interior voxels only, every halo position 0), copy_stride
// elements apart for the NC copies at shift, shift + 1, ...; with ncopy > 0
// the 64-position rows go to K-tile blocks instead, dst[t][copy + i][c][64]
// for t = flat position / 64 (the three x-shifted copies of an output
// gradient side by side per tile: one contiguous 12 KB block of DRAM per
// 32-channel tile for the weight gradient's A operand).
//
// A block moves 256 consecutive flat positions x 32 channels: the voxels
// (and one to either side for the shifted copies) come into shared memory as
// channel rows, 16 bytes per access, and leave through transposing matrix
// loads whose row addresses carry the shift, so the source is read once for
// all copies; four lanes exchange their pieces so that each writes 16 bytes
// of one channel.  Each position's voxel is worked out once per block in
// 32-bit arithmetic.  Bound: HBM (the copies written).  Before, one copy per
// launch with 64-bit divisions per access and 2-byte shared stores: 2.75 ms
// of a training iteration of 4 x 64^3.
constexpr int kCmPos = 256, kCmPitch = 80;  // bytes per row of 32 channels: 8 rows hit 8 different bank groups

//
// I: 32-bit voxels and positions of a sample, and blocks of work, where they
// fit it, else 64-bit.
template <int NC, typename I>
__global__ void __launch_bounds__(256) k_cmajor(const __nv_bfloat16 *src, int B, int D, int H, int W, int ctot, int coff,
                                                int nch, int Wp, long long pstride, int shift, int zero_halo, int copy,
                                                int ncopy, long long copy_stride, __nv_bfloat16 *dst) {
  after_previous();
  __shared__ __align__(16) unsigned char rows[(kCmPos + 3) * kCmPitch];  // positions -1 .. 256, and a row of zeros
  __shared__ I voxel[kCmPos + 2];
  __shared__ int xs[kCmPos + 2];
  constexpr int kZero = kCmPos + 2;
  const I plane = (I)(H + 2) * Wp, per_sample = (I)(D + 2) * plane;
  const long long total = (long long)B * pstride;
  const I nck = (nch + 31) / 32, works = (I)((total + kCmPos - 1) / kCmPos) * nck;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < kCmPitch / 4) ((unsigned *)(rows + kZero * kCmPitch))[threadIdx.x] = 0u;
  for (I work = blockIdx.x; work < works; work += gridDim.x) {
    const I blk = work / nck;
    const int c0 = (int)(work - blk * nck) * 32, cw = min(32, nch - c0);
    const long long e0 = (long long)blk * kCmPos;
    __syncthreads();
    for (int i = threadIdx.x; i < kCmPos + 2; i += 256) {
      const long long e = e0 + i - 1;
      I v = -1;
      int x = -0x4000;  // no voxel there
      if (e >= 0 && e < total) {
        const I n = (I)(e / pstride), f = (I)(e - n * pstride);
        if (f < per_sample) {
          const I z = f / plane, r = f - z * plane, y = r / Wp;
          x = (int)(r - y * Wp);
          bool in = x <= W + 1;
          if (zero_halo) in = in && x >= 1 && x <= W && y >= 1 && y <= H && z >= 1 && z <= D;
          if (in) v = ((n * (D + 2) + z) * (H + 2) + y) * (W + 2) + x;
        }
      }
      voxel[i] = v;
      xs[i] = x;
    }
    __syncthreads();
    for (int a = threadIdx.x; a < (kCmPos + 2) * 4; a += 256) {
      const int i = a >> 2, cv = a & 3;
      const I v = voxel[i];
      uint4 u = make_uint4(0, 0, 0, 0);
      if (v >= 0 && 8 * cv < cw) u = *(const uint4 *)(src + (long long)v * ctot + coff + c0 + 8 * cv);
      *(uint4 *)(rows + i * kCmPitch + 16 * cv) = u;
    }
    __syncthreads();
    // warp w transposes positions [32 w, 32 w + 32), 8 channels at a time
#pragma unroll
    for (int i = 0; i < NC; i++) {
      const int s = shift + i;
      // this lane's row address: position 32 w + lane, moved by the shift
      const int p = 32 * warp + lane, xsrc = xs[p + 1] - s;
      const int row = xsrc >= 0 && xsrc <= W + 1 ? p + 1 - s : kZero;
      const uint32_t at = tc::smem_u32(rows + row * kCmPitch);
      for (int cv = 0; 8 * cv < cw; cv++) {
        unsigned r0, r1, r2, r3;
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                     : "r"(at + 16 * cv));
        // lane 4 c + q holds positions 8 j + 2 q, + 1 of channel c in r_j:
        // exchange so that it holds positions 8 q .. 8 q + 7
        const bool q1 = lane & 1, q2 = lane & 2;
        unsigned a = __shfl_xor_sync(0xffffffffu, q1 ? r0 : r1, 1), b = __shfl_xor_sync(0xffffffffu, q1 ? r2 : r3, 1);
        if (q1) { r0 = a; r2 = b; } else { r1 = a; r3 = b; }
        a = __shfl_xor_sync(0xffffffffu, q2 ? r0 : r2, 2);
        b = __shfl_xor_sync(0xffffffffu, q2 ? r1 : r3, 2);
        if (q2) { r0 = a; r1 = b; } else { r2 = a; r3 = b; }
        const int c = c0 + 8 * cv + (lane >> 2);
        const long long e = e0 + 32 * warp + 8 * (lane & 3);
        if (e < total) {
          const long long o = ncopy ? (((e >> 6) * ncopy + copy + i) * nch + c) * 64 + (e & 63)
                                    : (long long)i * copy_stride + (long long)c * total + e;
          *(uint4 *)(dst + o) = make_uint4(r0, r1, r2, r3);
        }
      }
    }
  }
}

// 2-D map: rows x cols BF16 (cols contiguous), box 64 x box_rows (128-byte swizzle)
bool make_map_k64(CUtensorMap *map, const void *ptr, long long rows, long long cols, int box_rows) {
  return make_map_2d(map, ptr, rows, cols, box_rows);
}

// 3 equally spaced copies (copy_bytes apart) of rows x cols BF16: box of 64
// columns x rows x ncopy copies
bool make_map_copies(CUtensorMap *map, const void *ptr, long long rows, long long cols, long long copy_bytes,
                     int ncopy) {
  EncodeTiled enc = encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, 3};
  const cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)copy_bytes};
  const cuuint32_t box[3] = {64, (cuuint32_t)rows, (cuuint32_t)ncopy};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// K-tile blocks [ntiles][rows][64] BF16: box of 64 x box_rows x 1
bool make_map_tiles(CUtensorMap *map, const void *ptr, long long rows, long long ntiles, int box_rows) {
  EncodeTiled enc = encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)ntiles};
  const cuuint64_t strides[2] = {128, (cuuint64_t)rows * 128};
  const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Shifted windows of rows x cols BF16 (row-major, channel rows): element
// (x, c, dy, dz) = ptr[c * cols + x + dy * Wp + dz * plane]; the first axis
// ends (ny - 1) * Wp + (nz - 1) * plane short of cols, so no window reaches
// past its row.  Box: 64 x box_rows x ny x nz.
bool make_map_windows(CUtensorMap *map, const void *ptr, long long rows, long long cols, int Wp, long long plane,
                      int box_rows, int ny, int nz, long long &dim0) {
  EncodeTiled enc = encode_fn();
  if (!enc) return false;
  dim0 = cols - (ny - 1) * (long long)Wp - (nz - 1) * plane;
  if (dim0 < 64) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)dim0, (cuuint64_t)rows, (cuuint64_t)ny, (cuuint64_t)nz};
  const cuuint64_t strides[3] = {(cuuint64_t)cols * 2, (cuuint64_t)Wp * 2, (cuuint64_t)plane * 2};
  const cuuint32_t box[4] = {64, (cuuint32_t)box_rows, (cuuint32_t)ny, (cuuint32_t)nz};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Flat channels-last copies of `rows` positions x nch channels: boxes of box_ch
// (32 or 64) channels x box_rows positions x box_chunks, and (ny, nz > 1) the
// windows of such boxes Wp and plane positions apart.
bool make_map_flat(CUtensorMap *map, const void *ptr, long long rows, int nch, int box_ch, int box_rows, int box_chunks) {
  EncodeTiled enc = encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)box_ch, (cuuint64_t)rows, (cuuint64_t)(nch / box_ch)};
  const cuuint64_t strides[2] = {(cuuint64_t)nch * 2, (cuuint64_t)box_ch * 2};
  const cuuint32_t box[3] = {(cuuint32_t)box_ch, (cuuint32_t)box_rows, (cuuint32_t)box_chunks};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, box_ch == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool make_map_flat_windows(CUtensorMap *map, const void *ptr, long long rows, int nch, int box_chunks, int Wp,
                           long long plane, int ny, int nz, long long &dim0) {
  EncodeTiled enc = encode_fn();
  if (!enc) return false;
  dim0 = rows - (ny - 1) * (long long)Wp - (nz - 1) * plane;
  if (dim0 < 64) return false;
  const cuuint64_t pos = (cuuint64_t)nch * 2;
  const cuuint64_t dims[5] = {32, (cuuint64_t)dim0, (cuuint64_t)(nch / 32), (cuuint64_t)ny, (cuuint64_t)nz};
  const cuuint64_t strides[4] = {pos, 64, pos * Wp, pos * (cuuint64_t)plane};
  const cuuint32_t box[5] = {32, 64, (cuuint32_t)box_chunks, (cuuint32_t)ny, (cuuint32_t)nz};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void *>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// M tile of 128 voxels for a D x H x W grid: false when the grid does not
// tile (sides powers of two with W * H * D >= 128 do)
bool tile_shape(int D, int H, int W, int &wbox, int &hbox, int &dbox) {
  wbox = W < 128 ? W : 128;
  hbox = H < 128 / wbox ? H : 128 / wbox;
  dbox = 128 / (wbox * hbox);
  return wbox * hbox * dbox == 128 && W % wbox == 0 && H % hbox == 0 && D % dbox == 0 && wbox <= 256 &&
         hbox <= 256 && dbox <= 256;
}

// nc copies (1 or 3) at shift, shift + 1, ...
int cmajor_launch(const char *who, const void *src, int B, int D, int H, int W, int ctot, int coff, int nch, int Wp,
                  long long pstride, int shift, int nc, int zero_halo, int copy, int ncopy, long long copy_stride,
                  void *dst, void *stream) {
  if (B < 1 || nch < 1 || coff < 0 || coff + nch > ctot || Wp < W + 2 || Wp % 8 || pstride % 64 ||
      pstride < (long long)(D + 2) * (H + 2) * Wp || shift < -1 || shift + nc - 1 > 1)
    return slbc::set_error(std::string(who) + ": bad geometry"), 1;
  if (nch % 8 || coff % 8 || ctot % 8 || !aligned16(src) || !aligned16(dst))
    return slbc::set_error(std::string(who) + ": channels in multiples of 8, 16-byte aligned buffers"), 1;
  const long long work = ((long long)B * pstride + kCmPos - 1) / kCmPos * ((nch + 31) / 32);
  const int blocks = (int)std::min<long long>(work, 152LL * 8);
  const auto go = [&](auto kernel) {
    launch_pdl(kernel, blocks, 256, 0, (cudaStream_t)stream, (const __nv_bfloat16 *)src, B, D, H, W, ctot, coff, nch,
               Wp, pstride, shift, zero_halo, copy, ncopy, copy_stride, (__nv_bfloat16 *)dst);
  };
  // below 2^30: the walk over the work adds the grid without a wrap
  const bool fits = std::max({pstride, (long long)B * (D + 2) * (H + 2) * (W + 2), work}) < 1LL << 30;
  if (nc == 3) fits ? go(k_cmajor<3, int>) : go(k_cmajor<3, long long>);
  else fits ? go(k_cmajor<1, int>) : go(k_cmajor<1, long long>);
  slbc::count_launch();
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return slbc::set_error(std::string(who) + ": " + cudaGetErrorString(e)), 1;
  return 0;
}

// Both weight-gradient entry points: dY as three channel-major copies (dy0,
// dy1, dy2) or, with dyt, as K-tile blocks of the three copies.
int wgrad_launch(const char *who, const void *dy0, const void *dy1, const void *dy2, const void *dyt, const void *xt,
                 int B, int D, int H, int W, int Wp, long long pstride, int cin, int cout, float *partial,
                 long long partial_floats, int splits, float *dw, void *stream) {
  const std::string me(who);
  WgradArgs w;
  if (cout < 32 || (cout > 128 && cout % 128) || (cout <= 128 && 128 % cout) || cin < 16 || cin % 16)
    return slbc::set_error(me + ": cout must be 32, 64, 128 or a multiple of 128; cin a multiple of 16"), 1;
  if (Wp < W + 2 || Wp % 8 || pstride % 64 || pstride < (long long)(D + 2) * (H + 2) * Wp || splits < 1)
    return slbc::set_error(me + ": bad geometry"), 1;
  if (partial_floats < (long long)splits * 27 * cout * cin)
    return slbc::set_error(me + ": partial buffer too small"), 1;
  if (dyt) dy0 = dy1 = dy2 = dyt;
  if (!aligned16(dy0) || !aligned16(dy1) || !aligned16(dy2) || !aligned16(xt) || !aligned16(partial) ||
      !aligned16(dw))
    return slbc::set_error(me + ": buffers must be 16-byte aligned"), 1;
  const long long cols = (long long)B * pstride;
  WgradNArgs wn;
  const bool plan_n = wgrad_n_plan(cin, cout, wn);
  if (dyt && !plan_n) return slbc::set_error(me + ": K-tile blocks need cout 32, 64 or 128"), 1;
  if (plan_n) {  // taps stacked along N
    wn.Wp = Wp;
    wn.plane = (H + 2) * Wp;
    wn.k_tiles = cols / 64;
    wn.splits = splits;
    wn.partial = partial;
    int *err = tc_err_flag();
    if (!err) return slbc::set_error(me + ": no device error flag"), 1;
    CUtensorMap m0, m1, m2, mb;
    wn.a_tiles = dyt != nullptr;
    if (wn.a_tiles) {
      if (!make_map_tiles(&m0, dyt, 3LL * cout, wn.k_tiles, wn.dpm * cout) ||
          !make_map_tiles(&m1, dyt, 3LL * cout, wn.k_tiles, cout) || !make_map_k64(&mb, xt, cin, cols, wn.cc))
        return slbc::set_error(me + ": tensor map encoding failed"), 1;
      m2 = m0;
    } else if (!make_map_k64(&m0, dy0, cout, cols, cout) || !make_map_k64(&m1, dy1, cout, cols, cout) ||
               !make_map_k64(&m2, dy2, cout, cols, cout) || !make_map_k64(&mb, xt, cin, cols, wn.cc)) {
      return slbc::set_error(me + ": tensor map encoding failed"), 1;
    }
    // single-box forms (each falls back to the per-copy / per-tap boxes
    // when its map cannot be made)
    CUtensorMap ma = m0, mw = mb;
    const long long cstride = (const char *)dy1 - (const char *)dy0;
    wn.a3 = !wn.a_tiles && wn.dpm > 1 && cstride >= (long long)cout * cols * 2 && cstride % 16 == 0 &&
            (const char *)dy2 - (const char *)dy1 == cstride && make_map_copies(&ma, dy0, cout, cols, cstride, wn.dpm);
    wn.b4_dim0 = 0;
    wn.b4 = (wn.nt == 9 || wn.nt == 3) &&
            make_map_windows(&mw, xt, cin, cols, Wp, wn.plane, wn.cc, 3, wn.nt / 3, wn.b4_dim0);
    if (!wn.a3) ma = m0;
    if (!wn.b4) mw = mb;
    static unsigned long long attr_n_done = 0;
    cudaError_t e = smem_opt_in((const void *)k_wgrad_n, kWgnSmem, attr_n_done);
    if (e != cudaSuccess) return slbc::set_error(me + ": " + cudaGetErrorString(e)), 1;
    const dim3 grid((unsigned)wgrad_n_ctas(wn), 1, (unsigned)splits);
    const int smem = kStages * (kWgTileA + wn.n_rows * 128) + 1024;
    launch_pdl(k_wgrad_n, grid, 128, smem, (cudaStream_t)stream, m0, m1, m2, mb, ma, mw, wn, err);
    slbc::count_launch();
    e = cudaGetLastError();
    if (e != cudaSuccess) return slbc::set_error(me + ": " + cudaGetErrorString(e)), 1;
    const long long n = 27LL * cout * cin;
    launch_pdl(k_sum_splits, (int)std::min<long long>((n + 255) / 256, 152LL * 8), 256, 0, (cudaStream_t)stream,
               partial, n, splits, dw);
    slbc::count_launch();
    e = cudaGetLastError();
    if (e != cudaSuccess) return slbc::set_error(me + ": " + cudaGetErrorString(e)), 1;
    return 0;
  }
  w.cin = cin; w.cout = cout;
  w.co_rows = cout < 128 ? cout : 128;
  w.taps_per_tile = 128 / w.co_rows;
  w.co_tiles = cout / w.co_rows;
  w.ntile = cin;
  while (w.ntile > 256) w.ntile /= 2;
  if (cin % w.ntile || w.ntile % 16) return slbc::set_error(me + ": cin does not split into N tiles"), 1;
  w.Wp = Wp;
  w.plane = (H + 2) * Wp;
  w.k_tiles = (long long)B * pstride / 64;
  w.splits = splits;
  w.tmem_cols = 32;
  while (w.tmem_cols < w.ntile) w.tmem_cols *= 2;
  w.partial = partial;
  int *err = tc_err_flag();
  if (!err) return slbc::set_error(me + ": no device error flag"), 1;
  CUtensorMap m0, m1, m2, mb;
  if (!make_map_k64(&m0, dy0, cout, cols, w.co_rows) || !make_map_k64(&m1, dy1, cout, cols, w.co_rows) ||
      !make_map_k64(&m2, dy2, cout, cols, w.co_rows) || !make_map_k64(&mb, xt, cin, cols, w.ntile))
    return slbc::set_error(me + ": tensor map encoding failed"), 1;
  static unsigned long long attr_done = 0;
  cudaError_t e = smem_opt_in((const void *)k_wgrad, kWgSmem, attr_done);
  if (e != cudaSuccess) return slbc::set_error(me + ": " + cudaGetErrorString(e)), 1;
  const dim3 grid((unsigned)(((27 + w.taps_per_tile - 1) / w.taps_per_tile) * w.co_tiles), (unsigned)(cin / w.ntile),
                  (unsigned)splits);
  const int smem = kStages * (kWgTileA + w.ntile * 128) + 1024;
  launch_pdl(k_wgrad, grid, 128, smem, (cudaStream_t)stream, m0, m1, m2, mb, w, err);
  slbc::count_launch();
  e = cudaGetLastError();
  if (e != cudaSuccess) return slbc::set_error(me + ": " + cudaGetErrorString(e)), 1;
  const long long n = 27LL * cout * cin;
  launch_pdl(k_sum_splits, (int)std::min<long long>((n + 255) / 256, 152LL * 8), 256, 0, (cudaStream_t)stream, partial,
             n, splits, dw);
  slbc::count_launch();
  e = cudaGetLastError();
  if (e != cudaSuccess) return slbc::set_error(me + ": " + cudaGetErrorString(e)), 1;
  return 0;
}

}  // namespace

extern "C" {

int slbc_tc_gemm(const void *A, const void *B, float *D, int M, int N, int K, int ldd, void *stream) {
  if (M <= 0 || N <= 0 || K <= 0 || M % kBM || N % kBN || K % kBK)
    return slbc::set_error("slbc_tc_gemm: M and N must be multiples of 128 and K of 64"), 1;
  if (ldd < N || ldd % 4) return slbc::set_error("slbc_tc_gemm: ldd must be >= N and a multiple of 4"), 1;
  if (!aligned16(A) || !aligned16(B) || !aligned16(D))
    return slbc::set_error("slbc_tc_gemm: A, B and D must be 16-byte aligned"), 1;
  int *err = tc_err_flag();
  if (!err) return slbc::set_error("slbc_tc_gemm: no device error flag"), 1;
  CUtensorMap ta, tb;
  if (!make_map_2d(&ta, A, M, K, kBM) || !make_map_2d(&tb, B, N, K, kBN))
    return slbc::set_error("slbc_tc_gemm: tensor map encoding failed"), 1;
  static unsigned long long attr_done = 0;
  cudaError_t e = smem_opt_in((const void *)k_gemm_bf16, kGemmSmem, attr_done);
  if (e != cudaSuccess) return slbc::set_error(std::string("slbc_tc_gemm: ") + cudaGetErrorString(e)), 1;
  launch_pdl(k_gemm_bf16, dim3(N / kBN, M / kBM), 128, kGemmSmem, (cudaStream_t)stream, ta, tb, D, ldd, K, err);
  slbc::count_launch();
  e = cudaGetLastError();
  if (e != cudaSuccess) return slbc::set_error(std::string("slbc_tc_gemm: ") + cudaGetErrorString(e)), 1;
  return 0;
}

static int conv3d(const void *in, int B, int D, int H, int W, int in_ctot, int in_coff, int cin, const void *wgt,
                  const float *bias, int cout, void *out, float *out_f32, int out_ctot, int out_coff, int relu,
                  const void *mask, void *stream) {
  ConvArgs a;
  if (!out == !out_f32) return slbc::set_error("slbc_tc_conv3d: exactly one output buffer"), 1;
  if (out_f32 && out_ctot % 4) return slbc::set_error("slbc_tc_conv3d_f32: out_ctot must be a multiple of 4"), 1;
  if (!out) out = out_f32;  // alignment checks below
  if (B < 1 || cin < 32 || cin % 32 || cout < 16 || cout > 256 || cout % 16)
    return slbc::set_error("slbc_tc_conv3d: cin must be a multiple of 32, cout a multiple of 16 up to 256"), 1;
  if (in_ctot % 8 || in_coff % 8 || in_coff + cin > in_ctot || out_ctot % 8 || out_coff % 8 ||
      out_coff + cout > out_ctot)
    return slbc::set_error("slbc_tc_conv3d: channel counts and offsets must be multiples of 8 and fit"), 1;
  if (!tile_shape(D, H, W, a.wbox, a.hbox, a.dbox))
    return slbc::set_error("slbc_tc_conv3d: the grid does not tile into 128-voxel boxes"), 1;
  if (!aligned16(in) || !aligned16(wgt) || !aligned16(out) || (mask && !aligned16(mask)))
    return slbc::set_error("slbc_tc_conv3d: buffers must be 16-byte aligned"), 1;
  int *err = tc_err_flag();
  if (!err) return slbc::set_error("slbc_tc_conv3d: no device error flag"), 1;
  CUtensorMap tx, tw;
  if (!make_map_act(&tx, in, B, D, H, W, in_ctot, a.wbox, a.hbox, a.dbox) ||
      !make_map_rows32(&tw, wgt, 27LL * (cin / 32) * cout, cout))
    return slbc::set_error("slbc_tc_conv3d: tensor map encoding failed"), 1;
  a.D = D; a.H = H; a.W = W;
  a.cin = cin; a.cout = cout; a.in_coff = in_coff;
  a.out_ctot = out_ctot; a.out_coff = out_coff;
  a.relu = relu;
  a.tmem_cols = 32;
  while (a.tmem_cols < cout) a.tmem_cols *= 2;
  a.bias = bias;
  a.mask = (const __nv_bfloat16 *)mask;
  a.out = out_f32 ? nullptr : (__nv_bfloat16 *)out;
  a.out_f32 = out_f32;
  if ((cout == 32 || cout == 64 || cout == 128 || (cout == 96 && cin == 32)) && W % 8 == 0 && H % 16 == 0) {
    // A column of 8 x 16 voxels is cut into runs along z.  Fewer, longer runs
    // read fewer halo planes; the count is the one whose busiest block has the
    // least work, in MMA cycles per chunk and tap pair: 32 per input plane (its
    // A rows) and cout / 4 per slice and dz (the weights).
    const int parts = cout == 128 ? 2 : 1, co = cout / parts;  // output channels in parts of `co`
    const int cols = (W / 8) * (H / 16), most = 256 / co;
    int runs = (D + most - 1) / most;
    double best = 0.0;
    for (int k = runs; k <= D; k++) {
      const double len = (double)D / k;
      const long long rounds = ((long long)cols * k * B * parts + kConvSms - 1) / kConvSms;
      const double work = (double)rounds * (32.0 * (len + 2.0) + 0.75 * co * len);
      if (k == runs || work < best) {
        best = work;
        runs = k;
      }
    }
    CUtensorMap th;
    if (!make_map_act(&th, in, B, D, H, W, in_ctot, 10, 18, 1) ||
        !make_map_rows32(&tw, wgt, 27LL * (cin / 32) * cout, co))
      return slbc::set_error("slbc_tc_conv3d: tensor map encoding failed"), 1;
    const int items = cols * runs * B;
    static unsigned long long attr_r[3] = {0, 0, 0};
    const auto go = [&](auto kernel, int smem, int slot) {
      cudaError_t e = smem_opt_in((const void *)kernel, smem, attr_r[slot]);
      if (e != cudaSuccess) return e;
      launch_pdl(kernel, std::min(items * parts, kConvSms), 192, smem, (cudaStream_t)stream, th, tw, a, runs, items,
                 parts, err);
      slbc::count_launch();
      return cudaGetLastError();
    };
    const cudaError_t e = co == 32   ? go(k_conv_r<32>, ConvR<32>::kSmem, 0)
                          : co == 64 ? go(k_conv_r<64>, ConvR<64>::kSmem, 1)
                                     : go(k_conv_r<96>, ConvR<96>::kSmem, 2);
    if (e != cudaSuccess) return slbc::set_error(std::string("slbc_tc_conv3d: ") + cudaGetErrorString(e)), 1;
    return 0;
  }
  if ((cout == 32 || cout == 64 || cout == 128) && W % 16 == 0 && H % 8 == 0 && D % 2 == 0) {
    CUtensorMap th;
    if (!make_map_act(&th, in, B, D, H, W, in_ctot, 16, 10, 4))
      return slbc::set_error("slbc_tc_conv3d: tensor map encoding failed"), 1;
    const int items = (int)((long long)(W / 16) * (H / 8) * (D / 2) * B);
    static unsigned long long attr_z[3] = {0, 0, 0};
    const auto go = [&](auto kernel, int smem, int slot) {
      cudaError_t e = smem_opt_in((const void *)kernel, smem, attr_z[slot]);
      if (e != cudaSuccess) return e;
      launch_pdl(kernel, std::min(items, kConvSms), 192, smem, (cudaStream_t)stream, th, tw, a, items, err);
      slbc::count_launch();
      return cudaGetLastError();
    };
    cudaError_t e;
    if (cout == 128) e = go(k_conv_z<128>, ConvZ<128>::kSmem, 0);
    else if (cout == 64) e = go(k_conv_z<64>, ConvZ<64>::kSmem, 1);
    else e = go(k_conv_z<32>, ConvZ<32>::kSmem, 2);
    if (e != cudaSuccess) return slbc::set_error(std::string("slbc_tc_conv3d: ") + cudaGetErrorString(e)), 1;
    return 0;
  }
  // as many parts of the output channels as fit one wave, at least 32 each
  const long long tiles = (long long)D * H * W / 128 * B;
  int parts = 1;
  while (cout % (32 * parts) == 0 && cout / (2 * parts) >= 32 && tiles * 2 * parts <= kConvSms) parts *= 2;
  if (parts > 1) {
    a.cout = cout / parts;
    if (!make_map_rows32(&tw, wgt, 27LL * (cin / 32) * cout, a.cout))
      return slbc::set_error("slbc_tc_conv3d: tensor map encoding failed"), 1;
    a.tmem_cols = 32;
    while (a.tmem_cols < a.cout) a.tmem_cols *= 2;
  }
  static unsigned long long attr_done[3] = {0, 0, 0};
  const int nst = conv_stages(a.cout), smem = conv_smem(nst, a.cout);
  const void *fn = nst == 8 ? (const void *)k_conv_fwd<8> : (nst == 6 ? (const void *)k_conv_fwd<6> : (const void *)k_conv_fwd<4>);
  cudaError_t e = smem_opt_in(fn, kConvSmemMax, attr_done[nst == 8 ? 0 : (nst == 6 ? 1 : 2)]);
  if (e != cudaSuccess) return slbc::set_error(std::string("slbc_tc_conv3d: ") + cudaGetErrorString(e)), 1;
  const dim3 grid((unsigned)((long long)D * H * W / 128), (unsigned)B, (unsigned)parts);
  if (nst == 8)
    launch_pdl(k_conv_fwd<8>, grid, 128, smem, (cudaStream_t)stream, tx, tw, a, err);
  else if (nst == 6)
    launch_pdl(k_conv_fwd<6>, grid, 128, smem, (cudaStream_t)stream, tx, tw, a, err);
  else
    launch_pdl(k_conv_fwd<4>, grid, 128, smem, (cudaStream_t)stream, tx, tw, a, err);
  slbc::count_launch();
  e = cudaGetLastError();
  if (e != cudaSuccess) return slbc::set_error(std::string("slbc_tc_conv3d: ") + cudaGetErrorString(e)), 1;
  return 0;
}

int slbc_tc_conv3d(const void *in, int B, int D, int H, int W, int in_ctot, int in_coff, int cin, const void *wgt,
                   const float *bias, int cout, void *out, int out_ctot, int out_coff, int relu, const void *mask,
                   void *stream) {
  return conv3d(in, B, D, H, W, in_ctot, in_coff, cin, wgt, bias, cout, out, nullptr, out_ctot, out_coff, relu, mask,
                stream);
}

int slbc_tc_conv3d_f32(const void *in, int B, int D, int H, int W, int in_ctot, int in_coff, int cin,
                       const void *wgt, const float *bias, int cout, float *out, int out_ctot, int out_coff,
                       void *stream) {
  return conv3d(in, B, D, H, W, in_ctot, in_coff, cin, wgt, bias, cout, nullptr, out, out_ctot, out_coff, 0, nullptr,
                stream);
}

int slbc_tc_halo(void *buf, int B, int D, int H, int W, int ctot, int coff, int nch, void *stream) {
  if (B < 1 || D < 1 || H < 1 || W < 1 || ctot % 8 || coff % 8 || nch % 8 || nch < 8 || coff + nch > ctot)
    return slbc::set_error("slbc_tc_halo: channel counts and offsets must be multiples of 8 and fit"), 1;
  if (!aligned16(buf)) return slbc::set_error("slbc_tc_halo: buffer must be 16-byte aligned"), 1;
  const long long per = 2LL * (H + 2) * (W + 2) + 2LL * D * (W + 2) + 2LL * D * H;
  const long long total = (long long)B * per * (nch / 8);
  const int blocks = (int)std::min<long long>((total + 255) / 256, 152LL * 16);
  const auto go = [&](auto kernel) {
    launch_pdl(kernel, blocks, 256, 0, (cudaStream_t)stream, (__nv_bfloat16 *)buf, B, D, H, W, ctot, coff, nch);
  };
  if (total < (1LL << 31)) go(k_halo<unsigned>);  // the grid's stride may go past the end
  else go(k_halo<unsigned long long>);
  slbc::count_launch();
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return slbc::set_error(std::string("slbc_tc_halo: ") + cudaGetErrorString(e)), 1;
  return 0;
}

int slbc_tc_cmajor(const void *src, int B, int D, int H, int W, int ctot, int coff, int nch, int Wp,
                   long long pstride, int shift, int zero_halo, void *dst, void *stream) {
  return cmajor_launch("slbc_tc_cmajor", src, B, D, H, W, ctot, coff, nch, Wp, pstride, shift, 1, zero_halo, 0, 0, 0,
                       dst, stream);
}

int slbc_tc_cmajor_tiles(const void *src, int B, int D, int H, int W, int ctot, int coff, int nch, int Wp,
                         long long pstride, int shift, int copy, int ncopy, void *dst, void *stream) {
  if (ncopy < 1 || copy < 0 || copy >= ncopy)
    return slbc::set_error("slbc_tc_cmajor_tiles: copy must lie in [0, ncopy)"), 1;
  return cmajor_launch("slbc_tc_cmajor_tiles", src, B, D, H, W, ctot, coff, nch, Wp, pstride, shift, 1, 0, copy, ncopy,
                       0, dst, stream);
}

int slbc_tc_cmajor_shifts(const void *src, int B, int D, int H, int W, int ctot, int coff, int nch, int Wp,
                          long long pstride, int tiles, void *dst, void *stream) {
  return cmajor_launch("slbc_tc_cmajor_shifts", src, B, D, H, W, ctot, coff, nch, Wp, pstride, -1, 3, 0, 0, tiles ? 3 : 0,
                       (long long)nch * B * pstride, dst, stream);
}

int slbc_tc_flat(const void *src, int B, int D, int H, int W, int ctot, int coff, int nch, int Wp, long long pstride,
                 int zero_halo, void *dst, void *stream) {
  if (B < 1 || nch < 8 || coff < 0 || coff + nch > ctot || Wp < W + 2 || Wp % 8 || pstride % 64 ||
      pstride < (long long)(D + 2) * (H + 2) * Wp || (long long)B * ((long long)(D + 2) * (H + 2) + 1) >= 1LL << 30 ||
      pstride >= 1LL << 31)
    return slbc::set_error("slbc_tc_flat: bad geometry"), 1;
  if (nch % 8 || coff % 8 || ctot % 8 || !aligned16(src) || !aligned16(dst))
    return slbc::set_error("slbc_tc_flat: channels must be multiples of 8 and buffers 16-byte aligned"), 1;
  const long long warps = (long long)B * ((long long)(D + 2) * (H + 2) + 1);
  launch_pdl(k_flat, (int)std::min<long long>((warps + 7) / 8, 152LL * 8), 256, 0, (cudaStream_t)stream,
             (const __nv_bfloat16 *)src, B, D, H, W, ctot, coff, nch, Wp, (int)pstride, zero_halo, (__nv_bfloat16 *)dst);
  slbc::count_launch();
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return slbc::set_error(std::string("slbc_tc_flat: ") + cudaGetErrorString(e)), 1;
  return 0;
}

int slbc_tc_wgrad_flat(const void *dyf, const void *xf, int B, int D, int H, int W, int Wp, long long pstride, int cin,
                       int cout, float *partial, long long partial_floats, int splits, float *dw, void *stream) {
  const std::string me = "slbc_tc_wgrad_flat";
  WgradNArgs w;
  if (cin % 32 || !wgrad_n_plan(cin, cout, w, 32))
    return slbc::set_error(me + ": cout must be 32, 64 or 128, cin a multiple of 32"), 1;
  const long long rows = (long long)B * pstride;
  if (B < 1 || Wp < W + 2 || Wp % 8 || pstride % 64 || pstride < (long long)(D + 2) * (H + 2) * Wp || splits < 1 ||
      rows >= 1LL << 31)
    return slbc::set_error(me + ": bad geometry"), 1;
  const long long n = 27LL * cout * cin;
  if (partial_floats < splits * n) return slbc::set_error(me + ": partial buffer too small"), 1;
  if (!aligned16(dyf) || !aligned16(xf) || !aligned16(partial) || !aligned16(dw))
    return slbc::set_error(me + ": buffers must be 16-byte aligned"), 1;
  int *err = tc_err_flag();
  if (!err) return slbc::set_error(me + ": no device error flag"), 1;
  w.Wp = Wp;
  w.plane = (H + 2) * Wp;
  w.k_tiles = rows / 64;
  w.splits = splits;
  w.partial = partial;
  w.a3 = w.a_tiles = 0;
  CUtensorMap ta, tb, win;
  const int ch = cout == 32 ? 32 : 64;
  if (!make_map_flat(&ta, dyf, rows, cout, ch, 72, cout / ch) || !make_map_flat(&tb, xf, rows, cin, 32, 64, w.cc / 32))
    return slbc::set_error(me + ": tensor map encoding failed"), 1;
  w.b4_dim0 = 0;
  w.b4 = (w.nt == 9 || w.nt == 3) &&
         make_map_flat_windows(&win, xf, rows, cin, w.cc / 32, Wp, w.plane, 3, w.nt / 3, w.b4_dim0);
  if (!w.b4) win = tb;
  static unsigned long long attr_done = 0;
  cudaError_t e = smem_opt_in((const void *)k_wgrad_f, kWgfSmem, attr_done);
  if (e != cudaSuccess) return slbc::set_error(me + ": " + cudaGetErrorString(e)), 1;
  const int smem = kStages * (kWgfTileA + w.n_rows * 128) + 1024;
  launch_pdl(k_wgrad_f, dim3((unsigned)wgrad_n_ctas(w), 1, (unsigned)splits), 128, smem, (cudaStream_t)stream, ta, tb, win,
             w, err);
  slbc::count_launch();
  e = cudaGetLastError();
  if (e != cudaSuccess) return slbc::set_error(me + ": " + cudaGetErrorString(e)), 1;
  launch_pdl(k_sum_splits, (int)std::min<long long>((n + 255) / 256, 152LL * 8), 256, 0, (cudaStream_t)stream, partial, n,
             splits, dw);
  slbc::count_launch();
  e = cudaGetLastError();
  if (e != cudaSuccess) return slbc::set_error(me + ": " + cudaGetErrorString(e)), 1;
  return 0;
}

int slbc_tc_wgrad_splits(int cin, int cout, long long k_tiles, long long max_splits) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    sms = 152;
  WgradNArgs wn;
  long long want;
  // as many splits as fill the SMs in one wave: a block left over for a
  // second wave would take as long as the whole first one
  if (wgrad_n_plan(cin, cout, wn)) {
    const int ctas = wgrad_n_ctas(wn);  // one block per SM
    want = sms / ctas;
  } else {  // two blocks per SM
    const int co_rows = cout < 128 ? cout : 128;
    int ntile = cin;
    while (ntile > 256) ntile /= 2;
    const int blocks = ((27 + 128 / co_rows - 1) / (128 / co_rows)) * (cout / co_rows) * (cin / ntile);
    want = 2 * sms / blocks;
  }
  want = std::min(want, std::max(1LL, k_tiles / 8));
  want = std::min(want, max_splits);
  return (int)std::max(1LL, want);
}

int slbc_tc_wgrad(const void *dy0, const void *dy1, const void *dy2, const void *xt, int B, int D, int H, int W,
                  int Wp, long long pstride, int cin, int cout, float *partial, long long partial_floats, int splits,
                  float *dw, void *stream) {
  return wgrad_launch("slbc_tc_wgrad", dy0, dy1, dy2, nullptr, xt, B, D, H, W, Wp, pstride, cin, cout, partial,
                      partial_floats, splits, dw, stream);
}

int slbc_tc_wgrad_tiles(const void *dyt, const void *xt, int B, int D, int H, int W, int Wp, long long pstride,
                        int cin, int cout, float *partial, long long partial_floats, int splits, float *dw,
                        void *stream) {
  if (!dyt) return slbc::set_error("slbc_tc_wgrad_tiles: no dY blocks"), 1;
  return wgrad_launch("slbc_tc_wgrad_tiles", nullptr, nullptr, nullptr, dyt, xt, B, D, H, W, Wp, pstride, cin, cout,
                      partial, partial_floats, splits, dw, stream);
}

// Synchronises the device and returns (and clears) the tensor-core kernels'
// error flag: 0 fine, 1 a pipeline wait gave up, 2 a load never landed.
int slbc_tc_status(void) {
  int *err = tc_err_flag();
  if (!err) return -1;
  if (cudaDeviceSynchronize() != cudaSuccess) return -1;
  int v = 0;
  if (cudaMemcpy(&v, err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  if (v) cudaMemset(err, 0, sizeof(int));
  return v;
}

}  // extern "C"
