// Glue kernels of the learned warm start's network: pooling and
// upsampling between resolution levels (with their gradients, the ReLU masks
// and the skip-connection sums fused in), bias gradients, weight layouts for
// the tensor-core convolutions, Adam, the loss and the input encoding.
//
// Activation buffers are channels-last BF16 with a one-voxel periodic halo,
// buf[n][z + 1][y + 1][x + 1][c], total channels ctot, and a kernel works on
// a channel slice [coff, coff + C); C and coff multiples of 8 (16-byte
// vectors of 8 channels).
#include <cuda_bf16.h>

#include <algorithm>
#include <string>

#include "slbc_internal.cuh"

namespace {

using slbc::after_previous;
using slbc::launch_pdl;
using slbc::row_of;
using slbc::rows_grid;

typedef __nv_bfloat16 bf16;

struct Slice {
  bf16 *p;
  int ctot, coff;
};

__device__ __forceinline__ long long vox(int n, int z, int y, int x, int D, int H, int W) {
  return (((long long)n * (D + 2) + z + 1) * (H + 2) + y + 1) * (W + 2) + x + 1;
}

__device__ __forceinline__ void load8(const bf16 *p, float (&v)[8]) {
  const uint4 u = *(const uint4 *)p;
  const __nv_bfloat162 *h = (const __nv_bfloat162 *)&u;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

__device__ __forceinline__ void store8(bf16 *p, const float (&v)[8]) {
  uint4 u;
  __nv_bfloat162 *h = (__nv_bfloat162 *)&u;
#pragma unroll
  for (int i = 0; i < 4; i++) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  *(uint4 *)p = u;
}

int grid_for(long long n) { return (int)std::min<long long>((n + 255) / 256, 152LL * 32); }

// A row walk and its row counts in 32 bits where the rows fit it (64-bit
// divisions per vector bounded these kernels at a third to a fifth of the
// memory rate), else in 64: go(I()) launches the kernel for that index type.
template <typename F>
void for_rows(long long rows, F go) {
  if (rows < (1LL << 31)) go(0u);
  else go(0ull);
}

template <typename I>
__device__ __forceinline__ slbc::RowTurns<I> walk(I rows, int rowlen) {
  return slbc::row_turns<I>(blockIdx.x, gridDim.x, threadIdx.x, rows, (unsigned)rowlen);
}

// 2x2x2 average of the fine interior (D, H, W) into the coarse interior
template <typename I>
__global__ void __launch_bounds__(256) k_pool(Slice in, Slice out, int B, int D, int H, int W, int C) {
  after_previous();
  const int Dc = D / 2, Hc = H / 2, Wc = W / 2, nv = C / 8, len = Wc * nv;
  const auto w = walk<I>((I)B * (I)Dc * (I)Hc, len);
  for (I turn = w.first; turn < w.turns; turn += w.step) {
    const auto part = w.piece(turn);
    int n, z, y;
    row_of(part.row, Dc, Hc, n, z, y);
    const bf16 *src = in.p + vox(n, 2 * z, 2 * y, 0, D, H, W) * in.ctot + in.coff;
    bf16 *dst = out.p + vox(n, z, y, 0, Dc, Hc, Wc) * out.ctot + out.coff;
    const long long py = (long long)(W + 2) * in.ctot, pz = (H + 2) * py;
    for (unsigned e = part.e; e < part.end; e += 256) {
      const int x = (int)(e / (unsigned)nv), cv = (int)e - x * nv;
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int c = 0; c < 8; c++) {
        float v[8];
        load8(src + (c >> 2) * pz + ((c >> 1) & 1) * py + (2LL * x + (c & 1)) * in.ctot + 8 * cv, v);
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i] += v[i];
      }
#pragma unroll
      for (int i = 0; i < 8; i++) acc[i] *= 0.125f;
      store8(dst + (long long)x * out.ctot + 8 * cv, acc);
    }
  }
}

// gradient of k_pool: dfine = (dcoarse / 8 + add) * (mask > 0); add and mask
// optional (null pointers)
template <typename I>
__global__ void __launch_bounds__(256) k_pool_bwd(Slice dcoarse, Slice dfine, Slice add, Slice mask, int B, int D,
                                                  int H, int W, int C) {
  after_previous();
  const int nv = C / 8, len = W * nv;
  const auto w = walk<I>((I)B * (I)D * (I)H, len);
  for (I turn = w.first; turn < w.turns; turn += w.step) {
    const auto part = w.piece(turn);
    int n, z, y;
    row_of(part.row, D, H, n, z, y);
    const bf16 *src = dcoarse.p + vox(n, z / 2, y / 2, 0, D / 2, H / 2, W / 2) * dcoarse.ctot + dcoarse.coff;
    const long long v0 = vox(n, z, y, 0, D, H, W);
    for (unsigned e = part.e; e < part.end; e += 256) {
      const int x = (int)(e / (unsigned)nv), cv = (int)e - x * nv;
      float g[8];
      load8(src + (long long)(x / 2) * dcoarse.ctot + 8 * cv, g);
#pragma unroll
      for (int i = 0; i < 8; i++) g[i] *= 0.125f;
      const long long v = v0 + x;
      if (add.p) {
        float a[8];
        load8(add.p + v * add.ctot + add.coff + 8 * cv, a);
#pragma unroll
        for (int i = 0; i < 8; i++) g[i] += a[i];
      }
      if (mask.p) {
        float m[8];
        load8(mask.p + v * mask.ctot + mask.coff + 8 * cv, m);
#pragma unroll
        for (int i = 0; i < 8; i++) g[i] = m[i] > 0.0f ? g[i] : 0.0f;
      }
      store8(dfine.p + v * dfine.ctot + dfine.coff + 8 * cv, g);
    }
  }
}

// nearest upsampling: fine (D, H, W) interior = coarse parent; a thread
// reads its vector of the parent once and writes the eight children
template <typename I>
__global__ void __launch_bounds__(256) k_up(Slice in, Slice out, int B, int D, int H, int W, int C) {
  after_previous();
  const int Dc = D / 2, Hc = H / 2, Wc = W / 2, nv = C / 8, len = Wc * nv;
  const auto w = walk<I>((I)B * (I)Dc * (I)Hc, len);
  for (I turn = w.first; turn < w.turns; turn += w.step) {
    const auto part = w.piece(turn);
    int n, z, y;
    row_of(part.row, Dc, Hc, n, z, y);
    const bf16 *src = in.p + vox(n, z, y, 0, Dc, Hc, Wc) * in.ctot + in.coff;
    bf16 *dst = out.p + vox(n, 2 * z, 2 * y, 0, D, H, W) * out.ctot + out.coff;
    const long long py = (long long)(W + 2) * out.ctot, pz = (H + 2) * py;
    for (unsigned e = part.e; e < part.end; e += 256) {
      const int x = (int)(e / (unsigned)nv), cv = (int)e - x * nv;
      const uint4 v = *(const uint4 *)(src + (long long)x * in.ctot + 8 * cv);
#pragma unroll
      for (int c = 0; c < 8; c++)
        *(uint4 *)(dst + (c >> 2) * pz + ((c >> 1) & 1) * py + (2LL * x + (c & 1)) * out.ctot + 8 * cv) = v;
    }
  }
}

// gradient of k_up: dcoarse = sum of the 8 children * (mask > 0) (coarse mask)
template <typename I>
__global__ void __launch_bounds__(256) k_up_bwd(Slice dfine, Slice dcoarse, Slice mask, int B, int D, int H, int W, int C) {
  after_previous();
  const int Dc = D / 2, Hc = H / 2, Wc = W / 2, nv = C / 8, len = Wc * nv;
  const auto w = walk<I>((I)B * (I)Dc * (I)Hc, len);
  for (I turn = w.first; turn < w.turns; turn += w.step) {
    const auto part = w.piece(turn);
    int n, z, y;
    row_of(part.row, Dc, Hc, n, z, y);
    const bf16 *src = dfine.p + vox(n, 2 * z, 2 * y, 0, D, H, W) * dfine.ctot + dfine.coff;
    const long long py = (long long)(W + 2) * dfine.ctot, pz = (H + 2) * py;
    const long long v0 = vox(n, z, y, 0, Dc, Hc, Wc);
    for (unsigned e = part.e; e < part.end; e += 256) {
      const int x = (int)(e / (unsigned)nv), cv = (int)e - x * nv;
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int c = 0; c < 8; c++) {
        float v[8];
        load8(src + (c >> 2) * pz + ((c >> 1) & 1) * py + (2LL * x + (c & 1)) * dfine.ctot + 8 * cv, v);
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i] += v[i];
      }
      const long long v = v0 + x;
      if (mask.p) {
        float m[8];
        load8(mask.p + v * mask.ctot + mask.coff + 8 * cv, m);
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i] = m[i] > 0.0f ? acc[i] : 0.0f;
      }
      store8(dcoarse.p + v * dcoarse.ctot + dcoarse.coff + 8 * cv, acc);
    }
  }
}

// db[c] += sum over interior voxels of g.  The grid stride is a multiple of
// C / 8, so a thread always handles the same 8 channels: it sums in
// registers and adds to the block's shared sums once.  I: 32-bit voxel indices
// where they suffice (64-bit divisions per vector bounded it: 304 -> 245 us for
// the 15 layers of a training iteration of 4 x 64^3).
template <typename I>
__global__ void __launch_bounds__(256) k_bias_grad(Slice g, int B, int D, int H, int W, int C, float *db) {
  after_previous();
  extern __shared__ float sh[];
  for (int c = threadIdx.x; c < C; c += 256) sh[c] = 0.0f;
  __syncthreads();
  const int nv = C / 8, cv = threadIdx.x % nv;
  const I voxels = (I)B * (I)D * (I)H * (I)W, step = (I)gridDim.x * (I)(256 / nv);
  const bf16 *src = g.p + g.coff + 8 * cv;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
  for (I e = (I)blockIdx.x * (I)(256 / nv) + threadIdx.x / nv; e < voxels; e += step) {
    const I row = e / (I)W, t = row / (I)H;
    const int x = (int)(e - row * (I)W), y = (int)(row - t * (I)H), n = (int)(t / (I)D), z = (int)(t - (I)n * (I)D);
    float v[8];
    load8(src + vox(n, z, y, x, D, H, W) * g.ctot, v);
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i] += v[i];
  }
#pragma unroll
  for (int i = 0; i < 8; i++) atomicAdd(&sh[8 * cv + i], acc[i]);
  __syncthreads();
  for (int c = threadIdx.x; c < C; c += 256) atomicAdd(&db[c], sh[c]);
}

// The optimiser's kernels take lists of tensors: a network has 30 of them, most
// so small that a launch each (4.2 us) was most of their time.  A block takes
// `block` elements of one tensor and finds it in the table of first blocks,
// which comes with the launch: kListBlock of them, or 256 where the blocks of the
// whole list then fit the GPU at once (Adam on 27,648 elements: 4.0 us, 4.8 in
// blocks of 2048).  Bound: HBM for the large tensors.  Measured on the default
// network: Adam 126 -> 47 us, squares 120 -> 33 us, layouts about 125 -> 37 us,
// scaling 30 launches -> 1 of 2.8 us.
constexpr int kListMax = 48, kListBlock = 2048;

struct TensorList {
  float *p[4][kListMax];
  long long n[kListMax];
  unsigned first[kListMax];  // first block of each tensor
  int count, block;
};

// Block decomposition of `count` (<= kListMax) element counts; the blocks in all.
// Where blocks end in a sum (most: blocks it should not exceed, 0 for none), large
// lists take more elements per block: 30 M squares 152 -> 116 us.
unsigned list_blocks(int count, const long long *n, unsigned *first, int &block, long long most = 0) {
  const auto cut = [&](long long elements) {
    long long blocks = 0;
    for (int t = 0; t < count; t++) blocks += (n[t] + elements - 1) / elements;
    return blocks;
  };
  const long long blocks = cut(kListBlock);
  block = kListBlock;
  if (cut(256) <= 152 * 8) block = 256;
  else if (most > 0 && blocks > most) block = (int)std::min<long long>((blocks + most - 1) / most, 1024) * kListBlock;
  unsigned at = 0;
  for (int t = 0; t < count; t++) {
    first[t] = at;
    at += (unsigned)((n[t] + block - 1) / block);
  }
  return at;
}

__device__ __forceinline__ int list_tensor(const unsigned *first, int count) {
  int t = 0;
  while (t + 1 < count && first[t + 1] <= blockIdx.x) t++;
  return t;
}

// f(i) for the elements of this block of its tensor
template <typename F>
__device__ __forceinline__ void list_elements(unsigned first, long long n, int block, F f) {
  const long long i0 = (long long)(blockIdx.x - first) * block + threadIdx.x;
  for (int k0 = 0; k0 < block; k0 += kListBlock) {
#pragma unroll
    for (int k = 0; k < kListBlock; k += 256) {
      const long long i = i0 + k0 + k;
      if (k0 + k < block && i < n) f(i);
    }
  }
}

// Tensor-core layouts of master weights m[tap][cout][cin].  Forward: w[tap]
// [cin/32][cout][32].  dgrad for input channels [ci0, ci0 + nci): the forward
// kernel with these weights maps dY (cout channels) to dX: w[t][cout/32][nci]
// [32] = m[26 - t][32 ck + j][ci0 + ci].
struct LayoutList {
  const float *m[kListMax];
  bf16 *w[kListMax];
  int cout[kListMax], cin[kListMax], ci0[kListMax], nci[kListMax];  // nci 0: forward
  unsigned first[kListMax];
  int count, block;
};

__global__ void __launch_bounds__(256) k_layouts(const __grid_constant__ LayoutList L) {
  after_previous();
  const int t = list_tensor(L.first, L.count);
  const float *m = L.m[t];
  bf16 *w = L.w[t];
  const unsigned cout = L.cout[t], cin = L.cin[t], ci0 = L.ci0[t], nci = L.nci[t];
  list_elements(L.first[t], 27LL * cout * (nci ? nci : cin), L.block, [&](long long e) {
    const unsigned j = (unsigned)e & 31u;
    unsigned r = (unsigned)(e >> 5);
    const unsigned c = r % (nci ? nci : cout);
    r /= nci ? nci : cout;
    const unsigned nck = (nci ? cout : cin) / 32u, ck = r % nck, tap = r / nck;
    const long long row = nci ? ((long long)(26u - tap) * cout + ck * 32u + j) : (long long)tap * cout + c;
    w[e] = __float2bfloat16(m[row * cin + (nci ? ci0 + c : ck * 32u + j)]);
  });
}

__global__ void __launch_bounds__(256) k_adam(const __grid_constant__ TensorList L, float lr, float b1, float b2,
                                              float eps, float c1, float c2) {
  after_previous();
  const int t = list_tensor(L.first, L.count);
  float *p = L.p[0][t], *m = L.p[2][t], *v = L.p[3][t];
  const float *g = L.p[1][t];
  list_elements(L.first[t], L.n[t], L.block, [&](long long i) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  });
}

// Gradient-norm clipping against a running norm, all on the device (no
// host round trip per iteration).  state[0]: sum of squares of every
// gradient tensor (k_sqsum adds to it, k_clip_scale resets it); state[1]:
// running norm (0 before the first call); state[2]: the scale to apply.
__global__ void __launch_bounds__(256) k_sqsum(const __grid_constant__ TensorList L, double *state) {
  after_previous();
  __shared__ double sh[256];
  const int t = list_tensor(L.first, L.count);
  const float *g = L.p[0][t];
  double s = 0.0;
  list_elements(L.first[t], L.n[t], L.block, [&](long long i) { s += (double)g[i] * g[i]; });
  sh[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x < 32) {  // one warp adds for all: the FP64 pipe is what this kernel waits for
    for (int i = 32; i < 256; i += 32) s += sh[threadIdx.x + i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) atomicAdd(state, s);
  }
}

// scale = min(1, factor * running / norm); running <- decay * running +
// (1 - decay) * norm * scale.  A non-finite norm gives scale 0 (the
// gradients are zeroed) and leaves the running norm as it was.
__global__ void k_clip_scale(double *state, float factor, float decay) {
  after_previous();
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const double nrm = sqrt(state[0]);
  state[0] = 0.0;
  const double run = state[1] > 0.0 ? state[1] : nrm;
  if (!isfinite(nrm)) {
    state[2] = 0.0;
    return;
  }
  const double sc = nrm > (double)factor * run ? (double)factor * run / nrm : 1.0;
  state[1] = (double)decay * run + (1.0 - (double)decay) * nrm * sc;
  state[2] = sc;
}

__global__ void __launch_bounds__(256) k_scale(const __grid_constant__ TensorList L, const double *state) {
  after_previous();
  const float sc = (float)state[2];
  if (sc == 1.0f) return;
  const int t = list_tensor(L.first, L.count);
  float *g = L.p[0][t];
  list_elements(L.first[t], L.n[t], L.block, [&](long long i) { g[i] = sc == 0.0f ? 0.0f : g[i] * sc; });
}

// loss = mean over voxels and the nch components of (pred - label)^2, pred
// in FP32 channels 0..nch-1 of a padded buffer (ctot_p channels), label
// [n][D][H][W][nch] FP32; grad (BF16, gctot channels, padded) = d loss /
// d pred in channels 0..nch-1, 0 in the others.  loss[0] += the sum / count (inv:
// 1 / count).  Bound: the FP64 sums, so no thread divides in FP64 and the blocks
// are few (a division per thread and twice the blocks: 67 us on 4 x 64^3, 55 so).
template <typename I>
__global__ void __launch_bounds__(256) k_mse(const float *pred, int ctot_p, const float *label, int nch,
                                             const float *sample_w, int B, int D, int H, int W, bf16 *grad, int gctot,
                                             double *loss, double inv) {
  after_previous();
  __shared__ double sh[256];
  double acc = 0.0;
  const auto w = walk<I>((I)B * (I)D * (I)H, W);
  for (I turn = w.first; turn < w.turns; turn += w.step) {
    const auto part = w.piece(turn);
    int n, z, y;
    row_of(part.row, D, H, n, z, y);
    const long long v0 = vox(n, z, y, 0, D, H, W), e0 = (long long)part.row * W;
    const float sw = sample_w ? sample_w[n] : 1.0f;
    for (unsigned e = part.e; e < part.end; e += 256) {
      const int x = (int)e;
      const long long v = v0 + x;
      bf16 *gp = grad + v * gctot;
      for (int c = 0; c < gctot; c += 8) *(uint4 *)(gp + c) = make_uint4(0, 0, 0, 0);
      for (int c = 0; c < nch; c++) {
        const float d = pred[v * ctot_p + c] - label[(e0 + x) * nch + c];
        acc += (double)sw * d * d;
        gp[c] = __float2bfloat16((float)(2.0 * inv) * sw * d);
      }
    }
  }
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, sh[0] * inv);
}

// Projection of the prediction error on the label, per sample n:
// s_n = <label_n, pred_n - label_n> / <label_n, label_n> over the interior
// voxels and channels [0, nch) (labels [n][D][H][W][lch]).  k_proj_dot adds <label_n, pred_n> into
// dot[n] (grid.y = sample); k_proj_grad adds the derivative of
// (weight / B) * sum_n s_n^2 to the BF16 gradient and the term to the loss.
__global__ void k_proj_dot(const float *pred, int ctot_p, const float *label, int lch, int nch, int D, int H, int W,
                           double *dot) {
  after_previous();
  __shared__ double sh[256];
  const int n = blockIdx.y;
  const long long per = (long long)D * H * W;
  double acc = 0.0;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < per; e += (long long)gridDim.x * blockDim.x) {
    long long r = e;
    const int x = (int)(r % W); r /= W;
    const int y = (int)(r % H);
    const int z = (int)(r / H);
    const long long v = vox(n, z, y, x, D, H, W);
    const float *lb = label + ((long long)n * per + e) * lch;
    for (int c = 0; c < nch; c++) acc += (double)pred[v * ctot_p + c] * (double)lb[c];
  }
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(dot + n, sh[0]);
}

__global__ void k_proj_grad(const float *label, int lch, int nch, const double *lab_sq, const double *dot, int B, int D,
                            int H, int W, float weight, bf16 *grad, int gctot, double *loss) {
  after_previous();
  const long long per = (long long)D * H * W, total = (long long)B * per;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    long long r = e;
    const int x = (int)(r % W); r /= W;
    const int y = (int)(r % H); r /= H;
    const int z = (int)(r % D);
    const int n = (int)(r / D);
    const double q = lab_sq[n];
    if (!(q > 0.0)) continue;
    const double sn = (dot[n] - q) / q;
    const float coef = (float)(2.0 * weight * sn / (q * B));
    bf16 *gp = grad + vox(n, z, y, x, D, H, W) * gctot;
    for (int c = 0; c < nch; c++) gp[c] = __float2bfloat16(__bfloat162float(gp[c]) + coef * label[e * lch + c]);
    if (e % per == 0) atomicAdd(loss, (double)weight * sn * sn / B);
  }
}

// input encoding: channel 0 = 1 on solid nodes, 0 on fluid; with
// features = 1, channel 1 = d / R and channel 2 = (d / R)^2 where d is the
// periodic distance from a fluid node to the nearest solid node, searched
// over a cube of half-width R = 5 (d = R when none is that close; 0 on
// solid nodes); with features = 2 the search reaches R = 12 (the pores of
// open packings are wider than 5) and channel 3 carries min(d, 5) / 5, the
// near-wall form of the first encoding; other channels zero (interior; the
// halo is filled afterwards)
constexpr int kDistR1 = 5, kDistR2 = 12;

// The squared distance min over the cube of dx^2 + dy^2 + dz^2 (solid
// nodes, capped at R^2 <= 144, so it fits a byte) separates into three
// one-axis passes (a minimum of sums is the nested minimum), each over
// 2R + 1 neighbours instead of (2R + 1)^3.  Values stay integers, so the
// result equals the cube search.
// Pass 1 (along x): nearest solid node on the row, searched outwards.
template <int R, typename I>
__global__ void __launch_bounds__(256) k_dist_x(const unsigned char *solid, I rows, int W, unsigned char *a) {
  after_previous();
  const auto w = walk<I>(rows, W);
  for (I turn = w.first; turn < w.turns; turn += w.step) {
    const auto part = w.piece(turn);
    const unsigned char *src = solid + (long long)part.row * W;
    unsigned char *dst = a + (long long)part.row * W;
    for (unsigned e = part.e; e < part.end; e += 256) {
      const int x = (int)e;
      int best = src[x] ? 0 : R * R;
      if (W >= R) {
        for (int d = 1; d < R && best == R * R; d++) {
          const int l = x - d < 0 ? x - d + W : x - d, r = x + d >= W ? x + d - W : x + d;
          if (src[l] | src[r]) best = d * d;
        }
      } else {
        for (int d = 1; d < R && best == R * R; d++)
          if (src[((x - d) % W + W) % W] | src[(x + d) % W]) best = d * d;
      }
      dst[x] = (unsigned char)best;
    }
  }
}

// Passes 2 and 3 (along y: n = H rows of `inner` = W bytes; along z: n = D
// planes of W H): b = min over |d| <= R of d^2 + a at the node d steps away.
// A thread takes kDistRun consecutive nodes p of the pass at one place of the
// line: 2R + kDistRun loads serve them all.  Where lines hold whole words it
// takes four neighbouring bytes (VEC 4) as two pairs of 16 bits, for which one
// instruction adds and takes the minimum.  Bound: those instructions.  Measured
// at 128^3, R = 12: 127 -> 14 us for both passes; before, 25 loads per output,
// byte-wise minima in some ten instructions each and, along z, one block per
// plane.
constexpr int kDistRun = 4;

template <int R, int VEC, typename I>
__global__ void __launch_bounds__(256) k_dist_min(const unsigned char *a, int outers, int n, long long inner,
                                                  unsigned char *b) {
  after_previous();
  const I len = (I)inner / VEC, groups = (I)(n + kDistRun - 1) / kDistRun;
  const I total = (I)outers * groups * len;
  for (I i = (I)blockIdx.x * 256u + threadIdx.x; i < total; i += (I)gridDim.x * 256u) {
    const I row = i / len, e = i - row * len, outer = row / groups;
    const int p0 = (int)(row - outer * groups) * kDistRun;
    const unsigned char *base = a + (long long)outer * n * inner + VEC * e;
    unsigned lo[kDistRun], hi[kDistRun];
#pragma unroll
    for (int t = 0; t < kDistRun; t++) lo[t] = hi[t] = (unsigned)(R * R) * 0x00010001u;
#pragma unroll
    for (int k = -R; k < R + kDistRun; k++) {
      int q = p0 + k;
      if (n >= R + kDistRun) q = q < 0 ? q + n : q >= n ? q - n : q;
      else q = (q % n + n) % n;
      const unsigned char *at = base + (long long)q * inner;
      const unsigned v = VEC == 4 ? *(const unsigned *)at : *at;
      const unsigned vl = VEC == 4 ? __byte_perm(v, 0, 0x4140) : v, vh = VEC == 4 ? __byte_perm(v, 0, 0x4342) : 0u;
#pragma unroll
      for (int t = 0; t < kDistRun; t++) {
        const int d = k - t;
        if (d < -R || d > R) continue;
        lo[t] = __viaddmin_u16x2(vl, (unsigned)(d * d) * 0x00010001u, lo[t]);
        if (VEC == 4) hi[t] = __viaddmin_u16x2(vh, (unsigned)(d * d) * 0x00010001u, hi[t]);
      }
    }
    unsigned char *out = b + ((long long)outer * n + p0) * inner + VEC * e;
#pragma unroll
    for (int t = 0; t < kDistRun; t++) {
      if (p0 + t >= n) break;
      if (VEC == 4) *(unsigned *)(out + (long long)t * inner) = __byte_perm(lo[t], hi[t], 0x6420);
      else out[(long long)t * inner] = (unsigned char)lo[t];
    }
  }
}

// dist2: the squared distances of the passes above (null without features),
// searched to radius R
template <typename I>
__global__ void __launch_bounds__(256) k_encode(const unsigned char *solid, const unsigned char *dist2, int R, int B,
                                                int D, int H, int W, bf16 *out, int ctot) {
  after_previous();
  const int nv = ctot / 8, len = W * nv;
  const auto w = walk<I>((I)B * (I)D * (I)H, len);
  for (I turn = w.first; turn < w.turns; turn += w.step) {
    const auto part = w.piece(turn);
    int n, z, y;
    row_of(part.row, D, H, n, z, y);
    bf16 *dst = out + vox(n, z, y, 0, D, H, W) * ctot;
    const long long e0 = (long long)part.row * W;
    for (unsigned e = part.e; e < part.end; e += 256) {
      const int x = (int)(e / (unsigned)nv), cv = (int)e - x * nv;
      uint4 u = make_uint4(0, 0, 0, 0);
      if (cv == 0) {
        bf16 *p = (bf16 *)&u;
        const bool s = solid[e0 + x] != 0;
        p[0] = __float2bfloat16(s ? 1.0f : 0.0f);
        if (dist2 && !s) {
          const float dist = sqrtf((float)dist2[e0 + x]);
          const float d = dist * (1.0f / (float)R);
          p[1] = __float2bfloat16(d);
          p[2] = __float2bfloat16(d * d);
          if (R != kDistR1) p[3] = __float2bfloat16(fminf(dist, (float)kDistR1) * (1.0f / kDistR1));
        }
      }
      *(uint4 *)(dst + (long long)x * ctot + 8 * cv) = u;
    }
  }
}

// prediction (FP32 channels 0..2 of a padded buffer) * scale on fluid
// nodes into three FP32 arrays u[c * N + e] (0 on solid nodes), the layout
// of lbsetveldev; shift_x is subtracted from u_x on fluid nodes.  With
// drho, channel 3 * drho_scale into drho[e] (0 on solid nodes).
template <typename I>
__global__ void __launch_bounds__(256) k_decode(const float *pred, int ctot_p, const unsigned char *solid, int D, int H,
                                                int W, float scale, float shift_x, float *u, float drho_scale,
                                                float *drho) {
  after_previous();
  const long long total = (long long)D * H * W;
  const auto w = walk<I>((I)D * (I)H, W);
  for (I turn = w.first; turn < w.turns; turn += w.step) {
    const auto part = w.piece(turn);
    int n, z, y;
    row_of(part.row, D, H, n, z, y);
    const float *src = pred + vox(0, z, y, 0, D, H, W) * ctot_p;
    for (unsigned turn_e = part.e; turn_e < part.end; turn_e += 256) {
      const int x = (int)turn_e;
      const long long e = (long long)part.row * W + x;
      const float *v = src + (long long)x * ctot_p;
      const bool s = solid[e] != 0;
#pragma unroll
      for (int c = 0; c < 3; c++) u[c * total + e] = s ? 0.0f : scale * v[c] - (c == 0 ? shift_x : 0.0f);
      if (drho) drho[e] = s ? 0.0f : drho_scale * v[3];
    }
  }
}

// Uniform plane flux of a decoded state (u: 3 x D*H*W, x = the slowest
// index; the flux of x through plane i is q[i] = sum over the plane of u_x).
// k_plane_sum: one block per plane, a fixed summation order.
__global__ void __launch_bounds__(256) k_plane_sum(const float *u, int D, long long plane, double *q) {
  after_previous();
  __shared__ double sh[256];
  const int i = blockIdx.x;
  double acc = 0.0;
  for (long long e = threadIdx.x; e < plane; e += blockDim.x) acc += (double)u[(long long)i * plane + e];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) q[i] = sh[0];
}

// One block: the harmonic mean qh of the plane fluxes, the scale qh / q[i]
// of every plane and the pressure p[i] = sum over the planes before i of
// force (1 - qh / q) (midpoint rule, zero mean), both times gain; work =
// [q | scale | p | spread].  Any plane flux <= 0 leaves the planes as they
// are (scale = gain, p 0).  Thread t takes a run of consecutive planes; the
// runs' sums are scanned in thread order (one thread alone spent 127 us on
// the divisions of 128 planes).
__global__ void __launch_bounds__(256) k_plane_fix(int D, float force, float gain, double *work) {
  after_previous();
  __shared__ double sa[256], sb[256], lo[256], hi[256];
  __shared__ int all_ok;
  const double *q = work;
  double *scale = work + D, *p = work + 2 * D;
  const int t = threadIdx.x, run = (D + 255) / 256;
  const int i0 = min(D, t * run), i1 = min(D, i0 + run);
  if (t == 0) all_ok = 1;
  __syncthreads();
  double inv = 0.0, qsum = 0.0, qmin = q[min(i0, D - 1)], qmax = qmin;
  bool ok = true;
  for (int i = i0; i < i1; i++) {
    ok = ok && q[i] > 0.0;
    inv += 1.0 / q[i];
    qmin = fmin(qmin, q[i]);
    qmax = fmax(qmax, q[i]);
    qsum += q[i];
  }
  if (!ok) all_ok = 0;
  sa[t] = inv;
  sb[t] = qsum;
  lo[t] = qmin;
  hi[t] = qmax;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (t < o) {
      sa[t] += sa[t + o];
      sb[t] += sb[t + o];
      lo[t] = fmin(lo[t], lo[t + o]);
      hi[t] = fmax(hi[t], hi[t + o]);
    }
    __syncthreads();
  }
  ok = all_ok != 0;
  const double qh = D / sa[0];
  if (t == 0) work[3 * D] = ok ? (hi[0] - lo[0]) / (sb[0] / D) : -1.0;
  __syncthreads();
  double mine = 0.0;
  for (int i = i0; i < i1; i++) {
    scale[i] = (ok ? qh / q[i] : 1.0) * gain;
    mine += ok ? (double)force * (1.0 - qh / q[i]) : 0.0;
  }
  sa[t] = mine;
  __syncthreads();
  for (int o = 1; o < 256; o <<= 1) {  // inclusive scan of the runs
    const double add = t >= o ? sa[t - o] : 0.0;
    __syncthreads();
    sa[t] += add;
    __syncthreads();
  }
  double acc = t > 0 ? sa[t - 1] : 0.0, mean = 0.0;
  for (int i = i0; i < i1; i++) {
    const double g = ok ? (double)force * (1.0 - qh / q[i]) : 0.0;
    p[i] = acc + 0.5 * g;
    acc += g;
    mean += p[i];
  }
  sb[t] = mean;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (t < o) sb[t] += sb[t + o];
    __syncthreads();
  }
  mean = sb[0] / D;
  for (int i = i0; i < i1; i++) p[i] = (p[i] - mean) * gain;
}

// u[c][x] *= scale[i]; drho[x] = gain drho[x] + 3 p[i] on fluid nodes (p = rho / 3)
__global__ void k_plane_apply(float *u, float *drho, const unsigned char *solid, int D, long long plane,
                              float gain, const double *work) {
  after_previous();
  const long long total = (long long)D * plane;
  const double *scale = work + D, *p = work + 2 * D;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / plane);
    const float s = (float)scale[i];
    u[e] *= s;
    u[total + e] *= s;
    u[2 * total + e] *= s;
    if (drho) drho[e] = gain * drho[e] + (solid[e] ? 0.0f : (float)(3.0 * p[i]));
  }
}

// Uniform cross fluxes: the flux of u_y through every y plane (and of u_z
// through every z plane) made equal to its mean, as mass conservation
// requires of a steady periodic flow, by adding delta(plane) * |u| to the
// component (|u| taken before: zero at walls and in solids, so no slip is
// made).  u: 3 x D*H*W, x the slowest index, z the fastest.  work: q[H + W]
// (plane fluxes, y planes then z planes), m[H + W] (plane sums of |u|),
// delta[H + W].  One block per plane, a fixed summation order.
__global__ void __launch_bounds__(256) k_cross_sum(const float *u, int D, int H, int W, double *work) {
  after_previous();
  __shared__ double sq[256], sm[256];
  const int b = blockIdx.x;
  const bool ydir = b < H;
  const int c = ydir ? b : b - H;
  const long long total = (long long)D * H * W;
  const long long n = ydir ? (long long)D * W : (long long)D * H;
  double aq = 0.0, am = 0.0;
  for (long long t = threadIdx.x; t < n; t += blockDim.x) {
    long long e;
    if (ydir) e = ((t / W) * H + c) * W + t % W;  // t = i * W + k
    else e = t * W + c;                           // t = i * H + j
    const float ux = u[e], uy = u[total + e], uz = u[2 * total + e];
    aq += (double)(ydir ? uy : uz);
    am += sqrt((double)ux * ux + (double)uy * uy + (double)uz * uz);
  }
  sq[threadIdx.x] = aq;
  sm[threadIdx.x] = am;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      sq[threadIdx.x] += sq[threadIdx.x + o];
      sm[threadIdx.x] += sm[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    work[b] = sq[0];
    work[H + W + b] = sm[0];
  }
}

__global__ void k_cross_fix(int H, int W, double *work) {
  after_previous();
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const double *q = work, *m = work + H + W;
  double *delta = work + 2 * (H + W);
  double my = 0.0, mz = 0.0;
  for (int j = 0; j < H; j++) my += q[j];
  for (int k = 0; k < W; k++) mz += q[H + k];
  my /= H;
  mz /= W;
  for (int b = 0; b < H + W; b++) delta[b] = m[b] > 0.0 ? ((b < H ? my : mz) - q[b]) / m[b] : 0.0;
}

__global__ void k_cross_apply(float *u, int D, int H, int W, const double *work) {
  after_previous();
  const long long total = (long long)D * H * W;
  const double *delta = work + 2 * (H + W);
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(e % W), j = (int)((e / W) % H);
    const float ux = u[e], uy = u[total + e], uz = u[2 * total + e];
    const double sp = sqrt((double)ux * ux + (double)uy * uy + (double)uz * uz);
    u[total + e] = (float)(uy + delta[j] * sp);
    u[2 * total + e] = (float)(uz + delta[H + k] * sp);
  }
}

bool ok8(int ctot, int coff, int C) { return ctot % 8 == 0 && coff % 8 == 0 && C % 8 == 0 && C > 0 && coff + C <= ctot; }

bool empty(int B, int D, int H, int W) { return B < 1 || D < 1 || H < 1 || W < 1; }

int launched(const char *what) {
  slbc::count_launch();
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    slbc::set_error(std::string(what) + ": " + cudaGetErrorString(e));
    return 1;
  }
  return 0;
}

int bad(const char *msg) {
  slbc::set_error(msg);
  return 1;
}

// `arrays` pointer arrays of `count` tensors each, in launches of kListMax:
// go(list, blocks)
template <typename F>
int tensor_lists(const char *who, int count, const long long *n, int arrays, const void *const *const *ptrs, F go,
                 long long most = 0) {
  for (int t = 0; t < count; t++)
    if (n[t] <= 0) return bad((std::string(who) + ": empty tensor").c_str());
  for (int t0 = 0; t0 < count; t0 += kListMax) {
    TensorList L;
    L.count = std::min(kListMax, count - t0);
    for (int t = 0; t < L.count; t++) {
      for (int a = 0; a < arrays; a++) L.p[a][t] = (float *)ptrs[a][t0 + t];
      L.n[t] = n[t0 + t];
    }
    const unsigned blocks = list_blocks(L.count, L.n, L.first, L.block, most);
    go(L, blocks);
    if (launched(who)) return 1;
  }
  return 0;
}

}  // namespace

extern "C" {

int slbc_nn_pool(const void *in, int in_ctot, int in_coff, void *out, int out_ctot, int out_coff, int B, int D, int H,
                 int W, int C, void *stream) {
  if (!ok8(in_ctot, in_coff, C) || !ok8(out_ctot, out_coff, C) || D % 2 || H % 2 || W % 2)
    return bad("slbc_nn_pool: channel slices must be multiples of 8 and the grid even");
  if (empty(B, D, H, W)) return bad("slbc_nn_pool: empty grid");
  const long long rows = (long long)B * (D / 2) * (H / 2);
  for_rows(rows, [&](auto i) {
    launch_pdl(k_pool<decltype(i)>, rows_grid(rows, (long long)(W / 2) * (C / 8)), 256, 0, (cudaStream_t)stream,
               Slice{(bf16 *)in, in_ctot, in_coff}, Slice{(bf16 *)out, out_ctot, out_coff}, B, D, H, W, C);
  });
  return launched("slbc_nn_pool");
}

int slbc_nn_pool_bwd(const void *dcoarse, int dc_ctot, int dc_coff, void *dfine, int df_ctot, int df_coff,
                     const void *add, int a_ctot, int a_coff, const void *mask, int m_ctot, int m_coff, int B, int D,
                     int H, int W, int C, void *stream) {
  if (!ok8(dc_ctot, dc_coff, C) || !ok8(df_ctot, df_coff, C) || (add && !ok8(a_ctot, a_coff, C)) ||
      (mask && !ok8(m_ctot, m_coff, C)) || D % 2 || H % 2 || W % 2)
    return bad("slbc_nn_pool_bwd: channel slices must be multiples of 8 and the grid even");
  if (empty(B, D, H, W)) return bad("slbc_nn_pool_bwd: empty grid");
  const long long rows = (long long)B * D * H;
  for_rows(rows, [&](auto i) {
    launch_pdl(k_pool_bwd<decltype(i)>, rows_grid(rows, (long long)W * (C / 8)), 256, 0, (cudaStream_t)stream,
               Slice{(bf16 *)dcoarse, dc_ctot, dc_coff}, Slice{(bf16 *)dfine, df_ctot, df_coff},
               Slice{(bf16 *)add, a_ctot, a_coff}, Slice{(bf16 *)mask, m_ctot, m_coff}, B, D, H, W, C);
  });
  return launched("slbc_nn_pool_bwd");
}

int slbc_nn_up(const void *in, int in_ctot, int in_coff, void *out, int out_ctot, int out_coff, int B, int D, int H,
               int W, int C, void *stream) {
  if (!ok8(in_ctot, in_coff, C) || !ok8(out_ctot, out_coff, C) || D % 2 || H % 2 || W % 2)
    return bad("slbc_nn_up: channel slices must be multiples of 8 and the grid even");
  if (empty(B, D, H, W)) return bad("slbc_nn_up: empty grid");
  const long long rows = (long long)B * (D / 2) * (H / 2);
  for_rows(rows, [&](auto i) {
    launch_pdl(k_up<decltype(i)>, rows_grid(rows, (long long)(W / 2) * (C / 8)), 256, 0, (cudaStream_t)stream,
               Slice{(bf16 *)in, in_ctot, in_coff}, Slice{(bf16 *)out, out_ctot, out_coff}, B, D, H, W, C);
  });
  return launched("slbc_nn_up");
}

int slbc_nn_up_bwd(const void *dfine, int df_ctot, int df_coff, void *dcoarse, int dc_ctot, int dc_coff,
                   const void *mask, int m_ctot, int m_coff, int B, int D, int H, int W, int C, void *stream) {
  if (!ok8(df_ctot, df_coff, C) || !ok8(dc_ctot, dc_coff, C) || (mask && !ok8(m_ctot, m_coff, C)) || D % 2 ||
      H % 2 || W % 2)
    return bad("slbc_nn_up_bwd: channel slices must be multiples of 8 and the grid even");
  if (empty(B, D, H, W)) return bad("slbc_nn_up_bwd: empty grid");
  const long long rows = (long long)B * (D / 2) * (H / 2);
  for_rows(rows, [&](auto i) {
    launch_pdl(k_up_bwd<decltype(i)>, rows_grid(rows, (long long)(W / 2) * (C / 8)), 256, 0, (cudaStream_t)stream,
               Slice{(bf16 *)dfine, df_ctot, df_coff}, Slice{(bf16 *)dcoarse, dc_ctot, dc_coff},
               Slice{(bf16 *)mask, m_ctot, m_coff}, B, D, H, W, C);
  });
  return launched("slbc_nn_up_bwd");
}

int slbc_nn_bias_grad(const void *g, int ctot, int coff, int B, int D, int H, int W, int C, float *db, void *stream) {
  if (!ok8(ctot, coff, C) || C > 1024 || 256 % (C / 8)) return bad("slbc_nn_bias_grad: bad channel slice");
  const long long voxels = (long long)B * D * H * W;
  const auto go = [&](auto kernel) {
    launch_pdl(kernel, std::min(grid_for(voxels * (C / 8)), 152 * 4), 256, C * sizeof(float), (cudaStream_t)stream,
               Slice{(bf16 *)g, ctot, coff}, B, D, H, W, C, db);
  };
  if (voxels < (1LL << 31)) go(k_bias_grad<unsigned>);  // the grid's stride may go past the end
  else go(k_bias_grad<unsigned long long>);
  return launched("slbc_nn_bias_grad");
}

int slbc_nn_layouts(int count, const float *const *master, const int *cout, const int *cin, const int *ci0,
                    const int *nci, void *const *w, void *stream) {
  for (int t = 0; t < count; t++) {
    if (nci[t] ? cout[t] < 32 || cout[t] % 32 || ci0[t] < 0 || nci[t] < 1 || ci0[t] + nci[t] > cin[t]
               : cin[t] < 32 || cin[t] % 32 || cout[t] < 1)
      return bad("slbc_nn_layouts: bad channel counts");
  }
  for (int t0 = 0; t0 < count; t0 += kListMax) {
    LayoutList L;
    long long n[kListMax];
    L.count = std::min(kListMax, count - t0);
    for (int t = 0; t < L.count; t++) {
      L.m[t] = master[t0 + t];
      L.w[t] = (bf16 *)w[t0 + t];
      L.cout[t] = cout[t0 + t];
      L.cin[t] = cin[t0 + t];
      L.ci0[t] = ci0[t0 + t];
      L.nci[t] = nci[t0 + t];
      n[t] = 27LL * L.cout[t] * (L.nci[t] ? L.nci[t] : L.cin[t]);
    }
    const unsigned blocks = list_blocks(L.count, n, L.first, L.block);
    launch_pdl(k_layouts, blocks, 256, 0, (cudaStream_t)stream, L);
    if (launched("slbc_nn_layouts")) return 1;
  }
  return 0;
}

int slbc_nn_wfwd(const float *master, int cout, int cin, void *w, void *stream) {
  if (cin % 32 || cin < 32 || cout < 1) return bad("slbc_nn_wfwd: cin must be a multiple of 32");
  const int zero = 0;
  return slbc_nn_layouts(1, &master, &cout, &cin, &zero, &zero, &w, stream);
}

int slbc_nn_wdgrad(const float *master, int cout, int cin, int ci0, int nci, void *w, void *stream) {
  if (cout % 32 || cout < 32 || ci0 < 0 || nci < 1 || ci0 + nci > cin) return bad("slbc_nn_wdgrad: bad channel range");
  return slbc_nn_layouts(1, &master, &cout, &cin, &ci0, &nci, &w, stream);
}

int slbc_nn_adam_list(int count, float *const *p, const float *const *g, float *const *m, float *const *v,
                      const long long *n, float lr, float b1, float b2, float eps, int t, void *stream) {
  if (t < 1) return bad("slbc_nn_adam: step count starts at 1");
  const float c1 = 1.0f - powf(b1, (float)t), c2 = 1.0f - powf(b2, (float)t);
  const void *const *ptrs[4] = {(const void *const *)p, (const void *const *)g, (const void *const *)m,
                                (const void *const *)v};
  return tensor_lists("slbc_nn_adam", count, n, 4, ptrs, [&](const TensorList &L, unsigned blocks) {
    launch_pdl(k_adam, blocks, 256, 0, (cudaStream_t)stream, L, lr, b1, b2, eps, c1, c2);
  });
}

int slbc_nn_adam(float *p, const float *g, float *m, float *v, long long n, float lr, float b1, float b2, float eps,
                 int t, void *stream) {
  return slbc_nn_adam_list(1, &p, &g, &m, &v, &n, lr, b1, b2, eps, t, stream);
}

int slbc_nn_sqsum_list(int count, const float *const *g, const long long *n, double *state, void *stream) {
  const void *const *ptrs[1] = {(const void *const *)g};
  return tensor_lists("slbc_nn_sqsum", count, n, 1, ptrs, [&](const TensorList &L, unsigned blocks) {
    launch_pdl(k_sqsum, blocks, 256, 0, (cudaStream_t)stream, L, state);
  }, 152 * 32);
}

int slbc_nn_sqsum(const float *g, long long n, double *state, void *stream) {
  return slbc_nn_sqsum_list(1, &g, &n, state, stream);
}

int slbc_nn_clip(double *state, float factor, float decay, void *stream) {
  if (!(factor > 0.0f) || !(decay >= 0.0f && decay < 1.0f)) return bad("slbc_nn_clip: factor > 0, 0 <= decay < 1");
  launch_pdl(k_clip_scale, 1, 32, 0, (cudaStream_t)stream, state, factor, decay);
  return launched("slbc_nn_clip");
}

int slbc_nn_scale_list(int count, float *const *g, const long long *n, const double *state, void *stream) {
  const void *const *ptrs[1] = {(const void *const *)g};
  return tensor_lists("slbc_nn_scale", count, n, 1, ptrs, [&](const TensorList &L, unsigned blocks) {
    launch_pdl(k_scale, blocks, 256, 0, (cudaStream_t)stream, L, state);
  });
}

int slbc_nn_scale(float *g, long long n, const double *state, void *stream) {
  return slbc_nn_scale_list(1, &g, &n, state, stream);
}

int slbc_nn_mse(const float *pred, int ctot_p, const float *label, int nch, const float *sample_w, int B, int D, int H,
                int W, void *grad, int gctot, double *loss, void *stream) {
  if (nch < 1 || ctot_p < nch || gctot % 8 || gctot < 8 || gctot < nch) return bad("slbc_nn_mse: bad channel counts");
  if (empty(B, D, H, W)) return bad("slbc_nn_mse: empty grid");
  const long long rows = (long long)B * D * H;
  const double inv = 1.0 / ((double)nch * ((double)B * D * H * W));
  for_rows(rows, [&](auto i) {
    launch_pdl(k_mse<decltype(i)>, std::min(rows_grid(rows, W), 152 * 4), 256, 0, (cudaStream_t)stream, pred, ctot_p,
               label, nch, sample_w, B, D, H, W, (bf16 *)grad, gctot, loss, inv);
  });
  return launched("slbc_nn_mse");
}

int slbc_nn_proj(const float *pred, int ctot_p, const float *label, int lch, int nch, const double *lab_sq, int B, int D,
                 int H, int W, float weight, void *grad, int gctot, double *dot, double *loss, void *stream) {
  if (nch < 1 || lch < nch || ctot_p < nch || gctot % 8 || gctot < nch || B < 1 || B > 65535)
    return bad("slbc_nn_proj: bad arguments");
  const cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemsetAsync(dot, 0, sizeof(double) * B, st) != cudaSuccess) return bad("slbc_nn_proj: memset");
  const long long per = (long long)D * H * W;
  const dim3 g1((unsigned)std::min<long long>((per + 255) / 256, 152), (unsigned)B);
  launch_pdl(k_proj_dot, g1, 256, 0, st, pred, ctot_p, label, lch, nch, D, H, W, dot);
  if (launched("slbc_nn_proj")) return 1;
  launch_pdl(k_proj_grad, std::min(grid_for((long long)B * per), 152 * 4), 256, 0, st, label, lch, nch, lab_sq, dot, B,
             D, H, W, weight, (bf16 *)grad, gctot, loss);
  return launched("slbc_nn_proj");
}

int slbc_nn_encode(const unsigned char *solid, int B, int D, int H, int W, void *out, int ctot, int features,
                   void *stream) {
  if (ctot % 8 || ctot < 8) return bad("slbc_nn_encode: bad channel count");
  if (empty(B, D, H, W)) return bad("slbc_nn_encode: empty grid");
  const long long rows = (long long)B * D * H, total = rows * W;
  const cudaStream_t st = (cudaStream_t)stream;
  unsigned char *a = nullptr;
  if (features) {
    // two stream-ordered scratch masks of one byte per voxel, the second on a
    // word boundary
    const long long mask = (total + 255) / 256 * 256;
    const cudaError_t e = cudaMallocAsync((void **)&a, 2 * mask, st);
    if (e != cudaSuccess) return bad((std::string("slbc_nn_encode scratch: ") + cudaGetErrorString(e)).c_str());
    unsigned char *b = a + mask;
    for_rows(rows, [&](auto i) {
      using I = decltype(i);
      const auto go = [&](auto kernel) {
        launch_pdl(kernel, rows_grid(rows, W), 256, 0, st, solid, (I)rows, W, a);
      };
      if (features == 2) go(k_dist_x<kDistR2, I>);
      else go(k_dist_x<kDistR1, I>);
    });
    // whole words along x where W holds them
    const int vec = W % 4 == 0 ? 4 : 1;
    const auto pass = [&](const unsigned char *from, int outers, int n, long long inner, unsigned char *to) {
      const long long runs = (long long)outers * ((n + kDistRun - 1) / kDistRun) * (inner / vec);
      for_rows(runs, [&](auto i) {
        using I = decltype(i);
        const auto go = [&](auto kernel) { launch_pdl(kernel, grid_for(runs), 256, 0, st, from, outers, n, inner, to); };
        if (features == 2 && vec == 4) go(k_dist_min<kDistR2, 4, I>);
        else if (features == 2) go(k_dist_min<kDistR2, 1, I>);
        else if (vec == 4) go(k_dist_min<kDistR1, 4, I>);
        else go(k_dist_min<kDistR1, 1, I>);
      });
    };
    pass(a, B * D, H, W, b);
    pass(b, B, D, (long long)W * H, a);
    slbc::count_launch(3);
  }
  for_rows(rows, [&](auto i) {
    launch_pdl(k_encode<decltype(i)>, rows_grid(rows, (long long)W * (ctot / 8)), 256, 0, st, solid, a,
               features == 2 ? kDistR2 : kDistR1, B, D, H, W, (bf16 *)out, ctot);
  });
  const int rc = launched("slbc_nn_encode");
  if (a) {
    const cudaError_t e = cudaFreeAsync(a, st);
    if (e != cudaSuccess && rc == 0) return bad((std::string("slbc_nn_encode scratch: ") + cudaGetErrorString(e)).c_str());
  }
  return rc;
}

int slbc_nn_plane_flux(float *u, float *drho, const unsigned char *solid, int D, int H, int W, float force,
                       float gain, double *work, void *stream) {
  if (D < 1 || H < 1 || W < 1 || D > 65535 || !u || !solid || !work) return bad("slbc_nn_plane_flux: bad arguments");
  const cudaStream_t st = (cudaStream_t)stream;
  const long long plane = (long long)H * W;
  launch_pdl(k_plane_sum, D, 256, 0, st, u, D, plane, work);
  if (launched("slbc_nn_plane_flux")) return 1;
  launch_pdl(k_plane_fix, 1, 256, 0, st, D, force, gain, work);
  if (launched("slbc_nn_plane_flux")) return 1;
  launch_pdl(k_plane_apply, grid_for((long long)D * plane), 256, 0, st, u, drho, solid, D, plane, gain, work);
  return launched("slbc_nn_plane_flux");
}

int slbc_nn_cross_flux(float *u, int D, int H, int W, double *work, void *stream) {
  if (D < 1 || H < 1 || W < 1 || H + W > 65535 || !u || !work) return bad("slbc_nn_cross_flux: bad arguments");
  const cudaStream_t st = (cudaStream_t)stream;
  launch_pdl(k_cross_sum, H + W, 256, 0, st, u, D, H, W, work);
  if (launched("slbc_nn_cross_flux")) return 1;
  launch_pdl(k_cross_fix, 1, 32, 0, st, H, W, work);
  if (launched("slbc_nn_cross_flux")) return 1;
  launch_pdl(k_cross_apply, grid_for((long long)D * H * W), 256, 0, st, u, D, H, W, work);
  return launched("slbc_nn_cross_flux");
}

int slbc_nn_decode(const float *pred, int ctot_p, const unsigned char *solid, int D, int H, int W, float scale,
                   float shift_x, float *u, float drho_scale, float *drho, void *stream) {
  if (ctot_p < (drho ? 4 : 3)) return bad("slbc_nn_decode: bad channel count");
  if (empty(1, D, H, W)) return bad("slbc_nn_decode: empty grid");
  const long long rows = (long long)D * H;
  for_rows(rows, [&](auto i) {
    launch_pdl(k_decode<decltype(i)>, rows_grid(rows, W), 256, 0, (cudaStream_t)stream, pred, ctot_p, solid, D, H, W,
               scale, shift_x, u, drho_scale, drho);
  });
  return launched("slbc_nn_decode");
}

}  // extern "C"
