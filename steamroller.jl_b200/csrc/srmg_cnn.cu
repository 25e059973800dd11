// srmg_cnn.cu -- the learned warm start: a small BF16 convolutional network that maps
// (previous potential, change of the right-hand side) on one block tile (16 x 16 cells
// plus the 2-cell ghost halo) to a guess of the new potential on the block's 16 x 16
// cells.  No reference counterpart: the reference starts every solve from the previous
// potential held in the field (src/streamer.jl:322-334).
//
// Network (per 20 x 20 tile, zero padding at the tile edge, ReLU after layers 1-5):
//   conv3x3  2 -> 32, conv3x3 32 -> 32 (x4), conv3x3 32 -> 1; output = centre 16 x 16.
// Parameters (FP32 master vector, layer by layer): W_l [9 taps][co][ci], then b_l [co].
// Every convolution is an implicit GEMM on the tensor cores (mma.sync m16n8k16, BF16
// operands, FP32 accumulation): M = 16 output pixels, N = 8 output channels, K = 16
// input channels of one tap.  Tiles and weights live in shared memory with 64-byte rows
// (a pixel's or an output channel's 32 channels) and an XOR swizzle of the 16-byte chunks.
//
// Training kernels: forward (storing every layer's activations and ReLU signs), loss and
// output gradient, the chain of input gradients of all layers (the same convolution with
// the transposed, flipped weights, times the ReLU mask), the weight gradients of all layers
// (per-CTA partial sums over pixels on the tensor cores, then a fixed-order reduction), and
// Adam.
#include <cmath>
#include <cstring>
#include <vector>

#include <cuda_bf16.h>

#include "srmg_ctx.h"
#include "srmg_internal.h"

using namespace srmg;

#define CK(call)                                              \
  do {                                                        \
    int _rc = cuda_check(ctx, (call), #call);                 \
    if (_rc) return _rc;                                      \
  } while (0)
#define RC(call)               \
  do {                         \
    int _rc = (call);          \
    if (_rc) return _rc;       \
  } while (0)

namespace cnn {

constexpr int kL = 6;          // layers
constexpr int kC = 32;         // hidden channels
constexpr int kT = 20;         // tile side (16 cells + 2 ghosts each side)
constexpr int kNP = kT * kT;   // pixels per tile
// A tile in shared memory: rows of 21 pixels, pixel (y, x) at (y + 1) * 21 + x + 1, so that
// one zero pixel serves as the right ring of its row and the left ring of the next; 64
// bytes (32 channels) a pixel, the four 16-byte chunks XOR-swizzled by (pixel / 2) % 4.
constexpr int kRP = kT + 1;
constexpr int kTilePix = (kT + 2) * kRP + 1;  // the last tap of the last pixel included
constexpr int kTileBytes = kTilePix * kC * 2;
constexpr int kTiles = kNP / 16;         // M tiles of 16 pixels
constexpr int kWMat = kC * kC;           // one tap's 32 x 32 weight matrix (bf16)
constexpr int kWElems = kL * 9 * kWMat;  // packed weights of all layers
__host__ __device__ constexpr int cin(int l) { return l == 0 ? 2 : kC; }
__host__ __device__ constexpr int cout(int l) { return l == kL - 1 ? 1 : kC; }

// Offsets of W_l and b_l in the FP32 master vector.
__host__ __device__ inline int woff(int l) {
  int o = 0;
  for (int k = 0; k < l; ++k) o += 9 * cout(k) * cin(k) + cout(k);
  return o;
}
__host__ __device__ inline int boff(int l) { return woff(l) + 9 * cout(l) * cin(l); }
constexpr int nparams() {
  int o = 0;
  for (int k = 0; k < kL; ++k) o += 9 * cout(k) * cin(k) + cout(k);
  return o;
}

// Byte offset of element (row r, column c) in a 32 x 32 bf16 matrix with 64-byte rows
// and the 16-byte chunks XOR-swizzled by (r / 2) % 4.
__host__ __device__ inline int swz(int r, int c) {
  return r * 64 + ((((c >> 3) ^ (r >> 1)) & 3) << 4) + (c & 7) * 2;
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldsm4(uint32_t a, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(a));
}
__device__ __forceinline__ void ldsm4t(uint32_t a, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(a));
}
__device__ __forceinline__ void ldsm2t(uint32_t a, uint32_t &r0, uint32_t &r1) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(a));
}
__device__ __forceinline__ void ldsm2(uint32_t a, uint32_t &r0, uint32_t &r1) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(a));
}
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t *>(&v);
}

// First tap's tile pixel of output pixel p; tap (dy, dx) reads dy * kRP + dx further on.
__device__ __forceinline__ int tap0(int p) { return (p / kT) * kRP + p % kT; }
// Byte offset of 16-byte chunk c (8 channels) of tile pixel q.
__device__ __forceinline__ uint32_t tile_off(int q, int c) {
  return (uint32_t)(q * 64 + (((c ^ (q >> 1)) & 3) << 4));
}

__device__ __forceinline__ void group_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// A tile is convolved by a group of WPG warps, M tile mt by warp mt % WPG.  The group keeps
// the whole layer's output in registers (5 M tiles x 32 channels a warp with WPG = 5) and
// writes it over the input between two barriers, so a sample holds one 29 KB tile and
// three groups run in one CTA beside the packed weights of every layer.  A warp loads a
// tap's weights once for its 5 M tiles (0.35 ldmatrix per mma; one M tile at a time needs
// 0.75), and while one group waits at its barriers the others keep the tensor pipe
// busy.  WPG = 13 spreads one sample over the CTA where there is at most one per SM: 2 M tiles a
// warp, the shorter chain.
//
// mma.sync bounds it (m16n8k16 issues every ~8.7 cycles per SM sub-partition: 8550 of them per
// sample are 272 us for 4096 samples on 148 SMs).  Measured with 16 warps on one sample,
// one M tile at a time and two tiles in shared memory: 687 us.
constexpr int max_tiles(int wpg) { return (kTiles + wpg - 1) / wpg; }
constexpr int groups(int wpg) { return wpg == 5 ? 3 : 1; }
template <int WPG>
__device__ __forceinline__ bool has_tile(int wg, int i) { return kTiles % WPG == 0 || wg + i * WPG < kTiles; }

// acc[i] = bias + the convolution of M tile wg + i * WPG: for every output pixel and output
// channel co < 8 * NT the sum over taps and ci < 16 * KH in that order, W one 32 x 32
// swizzled matrix per tap at `w` (FLIP: the tap order reversed).
template <int WPG, int KH, int NT, bool FLIP>
__device__ __forceinline__ void conv_group(uint32_t tile, uint32_t w, int wg, const float *bias,
                                           float (&acc)[max_tiles(WPG)][4][4]) {
  constexpr int MT = max_tiles(WPG);
  const int lane = threadIdx.x & 31, t4 = lane & 3;
  int q0[MT];
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    // this lane's ldmatrix row: pixel (lane % 16) of the M tile, chunk lane / 16
    q0[i] = tap0((has_tile<WPG>(wg, i) ? wg + i * WPG : 0) * 16 + (lane & 15));
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const float b0 = bias ? bias[nt * 8 + 2 * t4] : 0.f, b1 = bias ? bias[nt * 8 + 2 * t4 + 1] : 0.f;
      acc[i][nt][0] = acc[i][nt][2] = b0;
      acc[i][nt][1] = acc[i][nt][3] = b1;
    }
  }
  // weight rows of this lane: NT = 4: (co lane/16 * 8 + lane%8, ci chunk (lane/8)%2), the
  // next two 8-row groups 1024 bytes on; NT = 1: co lane % 8
  const int br = (NT == 4 ? (lane >> 4) * 8 : 0) + (lane & 7);
  const uint32_t wl = w + swz(br, ((lane >> 3) & 1) * 8);
#pragma unroll 1
  for (int tap = 0; tap < 9; ++tap) {
    const uint32_t wb = wl + (uint32_t)((FLIP ? 8 - tap : tap) * kWMat * 2);
    const int qt = (tap / 3) * kRP + tap % 3;
#pragma unroll
    for (int kh = 0; kh < KH; ++kh) {
      uint32_t b[NT == 4 ? 8 : 2];
      if (NT == 4) {
        ldsm4(wb ^ (kh * 32), b[0], b[1], b[2], b[3]);
        ldsm4((wb + 1024) ^ (kh * 32), b[4], b[5], b[6], b[7]);
      } else {
        ldsm2(wb ^ (kh * 32), b[0], b[1]);
      }
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        if (!has_tile<WPG>(wg, i)) break;  // uniform per warp
        uint32_t a0, a1, a2, a3;
        ldsm4((tile + tile_off(q0[i] + qt, lane >> 4)) ^ (kh * 32), a0, a1, a2, a3);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) mma16816(acc[i][nt], a0, a1, a2, a3, b[2 * nt], b[2 * nt + 1]);
      }
    }
  }
}

// Shared memory of the forward and the input-gradient chain: packed weights, then (forward)
// the biases, then one tile per group.
constexpr int kFwdW = kWElems * 2, kBwdW = (kL - 1) * 9 * kWMat * 2;
constexpr int kBiasBytes = kL * kC * 4;
constexpr int fwd_smem(int wpg) { return kFwdW + kBiasBytes + groups(wpg) * kTileBytes; }
constexpr int bwd_smem(int wpg) { return kBwdW + groups(wpg) * kTileBytes; }
constexpr int cnn_threads(int wpg) { return groups(wpg) * wpg * 32; }

// Copies the 400 pixels (32 channels) of a tile to global [400][32], by `nthr` threads.
__device__ __forceinline__ void store_tile(const unsigned char *tile, __nv_bfloat16 *g, int t, int nthr) {
  for (int i = t; i < kNP * 4; i += nthr) {
    const int q = tap0(i >> 2) + kRP + 1;
    reinterpret_cast<uint4 *>(g)[i] = *reinterpret_cast<const uint4 *>(tile + tile_off(q, i & 3));
  }
}

// Forward pass over n samples.  x: [n][400][2] bf16 (tile pixel order y * 20 + x).
// y: [n][16][16] FP32 output (the tile's centre).  TRAIN keeps what the backward pass
// reads: xc [n][400][2], the input; acts [n][5][400][32] bf16, the inputs of layers 1..5; signs
// [n][5][400][4], their positive channels, byte (pixel, t4) bit 2 nt + j for channel
// 8 nt + 2 t4 + j.
template <int WPG, bool TRAIN>
__global__ void __launch_bounds__(cnn_threads(WPG), 1)
k_cnn_fwd(const __nv_bfloat16 *__restrict__ x, int n, const __nv_bfloat16 *__restrict__ wpk,
          const float *__restrict__ bias, float *__restrict__ y, uint32_t *__restrict__ xc,
          __nv_bfloat16 *__restrict__ acts, unsigned char *__restrict__ signs, const int *__restrict__ n_dev) {
  constexpr int MT = max_tiles(WPG), NTHR = WPG * 32, NX = (kNP + NTHR - 1) / NTHR;
  extern __shared__ __align__(128) unsigned char smraw[];
  float *sbias = reinterpret_cast<float *>(smraw + kFwdW);
  if (n_dev) n = min(n, *n_dev);  // sample count decided on the device
  {
    const uint4 *src = reinterpret_cast<const uint4 *>(wpk);
    uint4 *dst = reinterpret_cast<uint4 *>(smraw);
#pragma unroll 4
    for (int i = threadIdx.x; i < kFwdW / 16; i += blockDim.x) dst[i] = src[i];
    for (int i = threadIdx.x; i < kL * kC; i += blockDim.x) sbias[i] = bias[i];
    uint4 *z = reinterpret_cast<uint4 *>(smraw + kFwdW + kBiasBytes);  // the zero ring (and the rest)
    for (int i = threadIdx.x; i < groups(WPG) * kTileBytes / 16; i += blockDim.x) z[i] = make_uint4(0, 0, 0, 0);
  }
  __syncthreads();
  const int grp = threadIdx.x / NTHR, t = threadIdx.x % NTHR, wg = t >> 5;
  const int lane = t & 31, g = lane >> 2, t4 = lane & 3;
  unsigned char *tile = smraw + kFwdW + kBiasBytes + grp * kTileBytes;
  const uint32_t tile_s = smem_addr(tile), w_s = smem_addr(smraw);
  const uint32_t *x2 = reinterpret_cast<const uint32_t *>(x);
  uint32_t xv[NX];
  auto fetch = [&](int s) {
#pragma unroll
    for (int k = 0; k < NX; ++k)
      if (s < n && t + k * NTHR < kNP) xv[k] = x2[(int64_t)s * kNP + t + k * NTHR];
  };
  const int s0 = blockIdx.x + gridDim.x * grp, ds = gridDim.x * groups(WPG);
  fetch(s0);
  for (int s = s0; s < n; s += ds) {
    // input: channels 0, 1 from x, 2..15 zero (layer 0 reads channels 0..15)
#pragma unroll
    for (int k = 0; k < NX; ++k) {
      const int p = t + k * NTHR;
      if (p >= kNP) break;
      const int q = tap0(p) + kRP + 1;
      *reinterpret_cast<uint4 *>(tile + tile_off(q, 0)) = make_uint4(xv[k], 0, 0, 0);
      *reinterpret_cast<uint4 *>(tile + tile_off(q, 1)) = make_uint4(0, 0, 0, 0);
      if (TRAIN) xc[(int64_t)s * kNP + p] = xv[k];
    }
    group_sync(1 + grp, NTHR);
    float acc[MT][4][4];
#pragma unroll 1
    for (int l = 0; l < kL - 1; ++l) {
      const uint32_t w = w_s + (uint32_t)(l * 9 * kWMat * 2);
      if (l == 0) conv_group<WPG, 1, 4, false>(tile_s, w, wg, sbias, acc);
      else conv_group<WPG, 2, 4, false>(tile_s, w, wg, sbias + l * kC, acc);
      group_sync(1 + grp, NTHR);  // every warp has read the layer's input
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        if (!has_tile<WPG>(wg, i)) break;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int p = (wg + i * WPG) * 16 + g + 8 * r, q = tap0(p) + kRP + 1;
          uint32_t sg = 0;
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) {
            const uint32_t v = pack_bf16(fmaxf(acc[i][nt][2 * r], 0.f), fmaxf(acc[i][nt][2 * r + 1], 0.f));
            *reinterpret_cast<uint32_t *>(tile + tile_off(q, nt) + t4 * 4) = v;
            if (TRAIN) {
              // positive as stored: not zero, not NaN, no sign bit
              const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162 *>(&v);
              sg |= (__low2float(h) > 0.f ? 1u : 0u) << (2 * nt) | (__high2float(h) > 0.f ? 2u : 0u) << (2 * nt);
            }
          }
          if (TRAIN) signs[((int64_t)s * (kL - 1) + l) * (kNP * 4) + p * 4 + t4] = (unsigned char)sg;
        }
      }
      group_sync(1 + grp, NTHR);
      if (TRAIN) store_tile(tile, acts + ((int64_t)s * (kL - 1) + l) * kNP * kC, t, NTHR);
    }
    fetch(s + ds);
    conv_group<WPG, 2, 1, false>(tile_s, w_s + (uint32_t)((kL - 1) * 9 * kWMat * 2), wg, sbias + (kL - 1) * kC, acc);
    if (t4 == 0) {
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        if (!has_tile<WPG>(wg, i)) break;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int p = (wg + i * WPG) * 16 + g + 8 * r, yy = p / kT, xx = p % kT;
          if (yy >= 2 && yy < 18 && xx >= 2 && xx < 18) y[(int64_t)s * 256 + (yy - 2) * 16 + (xx - 2)] = acc[i][0][2 * r];
        }
      }
    }
    group_sync(1 + grp, NTHR);
  }
}

// Radial stencil weights of cell column qx (0..15) of a sample whose block starts at
// global r index ir0 (cylindrical: w- = (2i-2)/(2i-1), w+ = 2i/(2i-1), i = ir0+qx+1).
__device__ __forceinline__ void rweights(int geom, int ir0, int qx, float &wm, float &wp) {
  if (geom == 1) {
    const float i = (float)(ir0 + qx + 1);
    wm = (2.f * i - 2.f) / (2.f * i - 1.f);
    wp = (2.f * i) / (2.f * i - 1.f);
  } else {
    wm = 1.f;
    wp = 1.f;
  }
}

// Loss and output gradient.  Loss = mean_{n x 256} (y - t)^2 + lambda mean_{n x 196} rho^2,
// rho = L(y) + x1 on the 14 x 14 interior cells: the normalised residual of the guess, the
// discrete operator applied to the output plus the normalised right-hand-side change (both
// in units where the output scale is s_l |db|).  One sample per CTA pass, one thread per
// cell; rho is formed once per cell in shared memory (0 off the interior) and its gradient
// gathered from the neighbours whose stencil reads the cell.  Loss partials per CTA (fixed
// order) and dy[n][256] = dLoss/dy.
__global__ void __launch_bounds__(256)
k_cnn_loss(const float *__restrict__ y, const float *__restrict__ t, const __nv_bfloat16 *__restrict__ x,
           const int *__restrict__ ir0s, float lambda, int geom, int n, float *__restrict__ dy,
           double *__restrict__ loss_part) {
  __shared__ float sy[18][18], srho[18][18];  // a ring of zeros around the 16 x 16 cells
  __shared__ double sh[8];
  const double inv = 1.0 / (256.0 * (double)n), invr = 1.0 / (196.0 * (double)n);
  const int cy = threadIdx.x >> 4, cx = threadIdx.x & 15;
  const bool inner = cy >= 1 && cy <= 14 && cx >= 1 && cx <= 14;
  for (int i = threadIdx.x; i < 18 * 18; i += 256) srho[i / 18][i % 18] = sy[i / 18][i % 18] = 0.f;
  double acc = 0.0;
  for (int s = blockIdx.x; s < n; s += gridDim.x) {
    const int64_t k = (int64_t)s * 256 + threadIdx.x;
    const float yc = y[k], d = yc - t[k];
    acc += (double)d * (double)d * inv;
    float g = (float)(2.0 * inv) * d;
    if (lambda > 0.f) {
      const int ir0 = ir0s[s];
      float wm, wp;
      __syncthreads();
      sy[cy + 1][cx + 1] = yc;
      __syncthreads();
      if (inner) {
        rweights(geom, ir0, cx, wm, wp);
        const float L = wm * sy[cy + 1][cx] + wp * sy[cy + 1][cx + 2] + sy[cy][cx + 1] + sy[cy + 2][cx + 1] - 4.f * yc;
        const float rho = L + __bfloat162float(x[((int64_t)s * kNP + (cy + 2) * kT + cx + 2) * 2 + 1]);
        srho[cy + 1][cx + 1] = rho;
        acc += (double)lambda * (double)rho * (double)rho * invr;
      }
      __syncthreads();
      // this cell is the r- neighbour of (cy, cx + 1) and the r+ neighbour of (cy, cx - 1)
      float gr = -4.f * srho[cy + 1][cx + 1];
      rweights(geom, ir0, cx + 1, wm, wp);
      gr += wm * srho[cy + 1][cx + 2];
      rweights(geom, ir0, cx - 1, wm, wp);
      if (cx >= 2) gr += wp * srho[cy + 1][cx];
      gr += srho[cy + 2][cx + 1];
      gr += srho[cy][cx + 1];
      g += (float)(2.0 * invr) * lambda * gr;
    }
    dy[k] = g;
  }
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double c = 0.0;
    for (int w = 0; w < 8; ++w) c += sh[w];
    loss_part[blockIdx.x] = c;
  }
}

// The input gradients of layers 5..1, one chain per sample in its tile: dz_5 is dy (rounded
// to bf16) on the centre pixels of channel 0, and dz_{l-1} = (dz_l conv W_l^T flipped) *
// (A_l > 0), written to dz[n][5][400][32] for the weight gradients.  wt: transposed
// packed weights of layers 1..5 (rows = ci, columns = co); signs: the forward's.  One launch
// for the whole chain: a launch per layer read and wrote each dz and read each activation
// again (5 x 42 us at 1024 samples; the chain is bound by mma.sync as the forward is).
template <int WPG>
__global__ void __launch_bounds__(cnn_threads(WPG), 1)
k_cnn_dx(const float *__restrict__ dy, const __nv_bfloat16 *__restrict__ wt,
         const unsigned char *__restrict__ signs, __nv_bfloat16 *__restrict__ dz, int n) {
  constexpr int MT = max_tiles(WPG), NTHR = WPG * 32;
  extern __shared__ __align__(128) unsigned char smraw[];
  {
    const uint4 *src = reinterpret_cast<const uint4 *>(wt + 9 * kWMat);
    uint4 *dst = reinterpret_cast<uint4 *>(smraw);
#pragma unroll 4
    for (int i = threadIdx.x; i < kBwdW / 16; i += blockDim.x) dst[i] = src[i];
    uint4 *z = reinterpret_cast<uint4 *>(smraw + kBwdW);
    for (int i = threadIdx.x; i < groups(WPG) * kTileBytes / 16; i += blockDim.x) z[i] = make_uint4(0, 0, 0, 0);
  }
  __syncthreads();
  const int grp = threadIdx.x / NTHR, t = threadIdx.x % NTHR, wg = t >> 5;
  const int lane = t & 31, g = lane >> 2, t4 = lane & 3;
  unsigned char *tile = smraw + kBwdW + grp * kTileBytes;
  const uint32_t tile_s = smem_addr(tile), w_s = smem_addr(smraw);
  for (int s = blockIdx.x + gridDim.x * grp; s < n; s += gridDim.x * groups(WPG)) {
    for (int p = t; p < kNP; p += NTHR) {
      const int yy = p / kT, xx = p % kT, q = tap0(p) + kRP + 1;
      float v = 0.f;
      if (yy >= 2 && yy < 18 && xx >= 2 && xx < 18) v = dy[(int64_t)s * 256 + (yy - 2) * 16 + (xx - 2)];
      const __nv_bfloat16 h = __float2bfloat16_rn(v);
      *reinterpret_cast<uint4 *>(tile + tile_off(q, 0)) =
          make_uint4((uint32_t)*reinterpret_cast<const uint16_t *>(&h), 0, 0, 0);
      *reinterpret_cast<uint4 *>(tile + tile_off(q, 1)) = make_uint4(0, 0, 0, 0);
    }
    group_sync(1 + grp, NTHR);
    float acc[MT][4][4];
#pragma unroll 1
    for (int l = kL - 1; l >= 1; --l) {
      const uint32_t w = w_s + (uint32_t)((l - 1) * 9 * kWMat * 2);
      const unsigned char *sl = signs + ((int64_t)s * (kL - 1) + l - 1) * (kNP * 4) + t4;
      unsigned char sg[MT][2];
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int r = 0; r < 2; ++r)
          if (has_tile<WPG>(wg, i)) sg[i][r] = sl[((wg + i * WPG) * 16 + g + 8 * r) * 4];
      if (l == kL - 1) conv_group<WPG, 1, 4, true>(tile_s, w, wg, nullptr, acc);
      else conv_group<WPG, 2, 4, true>(tile_s, w, wg, nullptr, acc);
      group_sync(1 + grp, NTHR);
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        if (!has_tile<WPG>(wg, i)) break;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int q = tap0((wg + i * WPG) * 16 + g + 8 * r) + kRP + 1;
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) {
            const float m0 = (sg[i][r] >> (2 * nt)) & 1 ? acc[i][nt][2 * r] : 0.f;
            const float m1 = (sg[i][r] >> (2 * nt)) & 2 ? acc[i][nt][2 * r + 1] : 0.f;
            *reinterpret_cast<uint32_t *>(tile + tile_off(q, nt) + t4 * 4) = pack_bf16(m0, m1);
          }
        }
      }
      group_sync(1 + grp, NTHR);
      store_tile(tile, dz + ((int64_t)s * (kL - 1) + l - 1) * kNP * kC, t, NTHR);
    }
    group_sync(1 + grp, NTHR);
  }
}

// Weight gradients of all layers in one launch.  CTA b belongs to one layer l (the CTAs
// shared out by the layers' work, DwParts) and sums over its samples
//   dW[tap][co][ci] += sum_p dz_l[p][co] * A_l[p + off(tap)][ci],  db[co] += sum_p dz_l[p][co]
// into partials [cta][9][32][32] and [cta][32].  15 warps: warp = (fifth kg of the pixels, tap row
// dy), three taps x 32 co x 32 ci a warp, so that one dz fragment serves three taps and both
// of a tap's ci halves (8 ldmatrix per 24 mma; one warp per (tap, co half) took 3 per
// 4).  mma.sync truncates as it accumulates, and the error grows with the chain: a chain ends
// after kPart samples (kFlush in the first and last layer, whose registers have room for the
// sums beside) and goes to sums of rounded additions.  Sums of one sign over 6000 samples:
// dW_1..4 off by 5e-7 to 1.2e-6 of the sum and dW_5 by 1.6e-7, 2.0e-5 to 5.5e-5 with a chain
// over all of a CTA's samples (1024 samples: 5e-7 to 1.1e-6 and 2.0e-7, 1.9e-6 to 5.9e-6).  db
// is summed from the fragments by rounded additions, per sample and then over the samples
// (7.6e-8; by one more mma against ones 2e-5 to 7e-5).  The next sample's tiles arrive by
// cp.async while this one is summed.  mma.sync bounds it; a launch per layer without the
// copies in flight, with a serial db sum, took 6 x 55 us at 1024 samples.
constexpr int kDwThreads = 15 * 32;
constexpr int kFlush = 4, kPart = 16;
constexpr int kBwdSamples = 8192;
constexpr int kDwStage = kTileBytes + kNP * kC * 2;
constexpr int kDwSmem = 2 * kDwStage + 9 * kWMat * 4 + kC * 4;  // two stages and the CTA's sums
struct DwParts {
  int first[kL + 1];  // CTAs first[l] .. first[l + 1] - 1 work on layer l
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// MH: co halves with real channels; NT: ci columns / 8.
template <int MH, int NT>
__device__ __forceinline__ void dw_layer(unsigned char *sm, int l, int part, int nparts, const float *dy,
                                         const __nv_bfloat16 *dz, const uint32_t *xc, const __nv_bfloat16 *acts, int n,
                                         float *dw_part, float *db_part) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int kg = warp / 3, dyr = warp % 3;
  for (int i = threadIdx.x; i < kDwSmem / 16; i += blockDim.x)
    reinterpret_cast<uint4 *>(sm)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  const uint32_t sm_s = smem_addr(sm);
  auto load = [&](int s, int st) {
    const uint32_t a_s = sm_s + st * kDwStage, z_s = a_s + kTileBytes;
    if (NT == 1) {  // layer 0: the two input channels
      for (int p = threadIdx.x; p < kNP; p += blockDim.x)
        cp_async4(a_s + tile_off(tap0(p) + kRP + 1, 0), xc + (int64_t)s * kNP + p);
    } else {
      const __nv_bfloat16 *src = acts + ((int64_t)s * (kL - 1) + l - 1) * kNP * kC;
      for (int i = threadIdx.x; i < kNP * 4; i += blockDim.x)
        cp_async16(a_s + tile_off(tap0(i >> 2) + kRP + 1, i & 3), src + i * 8);
    }
    if (MH == 1) {  // layer 5: dz is dy on channel 0 of the centre pixels
      for (int k = threadIdx.x; k < 256; k += blockDim.x) {
        const __nv_bfloat16 h = __float2bfloat16_rn(dy[(int64_t)s * 256 + k]);
        const int p = ((k >> 4) + 2) * kT + (k & 15) + 2;
        *reinterpret_cast<__nv_bfloat16 *>(sm + st * kDwStage + kTileBytes + tile_off(p, 0)) = h;
      }
    } else {
      const __nv_bfloat16 *src = dz + ((int64_t)s * (kL - 1) + l) * kNP * kC;
      for (int i = threadIdx.x; i < kNP * 4; i += blockDim.x) cp_async16(z_s + tile_off(i >> 2, i & 3), src + i * 8);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  constexpr bool kShort = MH == 1 || NT == 1;  // the layers with fewer CTAs
  float acc[3][MH][NT][4], sum[kShort ? 3 : 1][MH][NT][4];
  float db[2] = {0.f, 0.f};  // co half dyr / 2 (dyr 1: none)
  float *red = reinterpret_cast<float *>(sm + 2 * kDwStage), *redb = red + 9 * kWMat;  // zero
  auto each = [&](auto fn) {  // over acc
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int m = 0; m < MH; ++m)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int j = 0; j < 4; ++j) fn(d, m, nt, j);
  };
  each([&](int d, int m, int nt, int j) {
    acc[d][m][nt][j] = 0.f;
    if (kShort) sum[d][m][nt][j] = 0.f;
  });
  int since = 0;
  auto flush = [&] {  // kShort: to the registers beside
    each([&](int d, int m, int nt, int j) {
      sum[d][m][nt][j] += acc[d][m][nt][j];
      acc[d][m][nt][j] = 0.f;
    });
  };
  auto put = [&] {  // to the CTA's sums, the five pixel fifths in order
    for (int k = 0; k < 5; ++k) {
      if (kg == k)
        each([&](int d, int m, int nt, int j) {
          red[(dyr * 3 + d) * kWMat + (m * 16 + g + (j >> 1) * 8) * kC + nt * 8 + 2 * t4 + (j & 1)] += acc[d][m][nt][j];
          acc[d][m][nt][j] = 0.f;
        });
      __syncthreads();
    }
  };
  const int mt = lane >> 3, r = lane & 7;
  int st = 0;
  if (part < n) load(part, 0);
  for (int s = part; s < n; s += nparts, st ^= 1) {
    if (s + nparts < n) {
      load(s + nparts, st ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const uint32_t a_s = sm_s + st * kDwStage, z_s = a_s + kTileBytes;
    float dbs[2] = {0.f, 0.f};  // this sample's
#pragma unroll 1
    for (int k0 = kg * 16; k0 < kNP; k0 += 80) {  // every fifth 16 pixels: no chain has only the rim
      // A operand (rows co, k = pixels) from dz [p][co] by transposed ldmatrix: matrices (co
      // 0-7, p 0-7), (co 8-15, p 0-7), (co 0-7, p 8-15), (co 8-15, p 8-15)
      uint32_t a[MH][4];
      const uint32_t ad = z_s + tile_off(k0 + r + (mt >> 1) * 8, mt & 1);
#pragma unroll
      for (int m = 0; m < MH; ++m) ldsm4t(ad ^ (m * 32), a[m][0], a[m][1], a[m][2], a[m][3]);
      // B operand (k = pixels, n = ci) from A_l [p + off][ci]: matrices (p 0-7, ci 0-7),
      // (p 8-15, ci 0-7), (p 0-7, ci 8-15), (p 8-15, ci 8-15)
      const int q = tap0(k0 + r + (mt & 1) * 8) + dyr * kRP;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const uint32_t bd = a_s + tile_off(q + d, NT == 1 ? 0 : mt >> 1);
        uint32_t b[NT == 1 ? 2 : 8];
        if (NT == 1) ldsm2t(bd, b[0], b[1]);
        else {
          ldsm4t(bd, b[0], b[1], b[2], b[3]);
          ldsm4t(bd ^ 32, b[4], b[5], b[6], b[7]);
        }
#pragma unroll
        for (int m = 0; m < MH; ++m)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
            mma16816(acc[d][m][nt], a[m][0], a[m][1], a[m][2], a[m][3], b[2 * nt], b[2 * nt + 1]);
      }
#pragma unroll
      for (int m = 0; m < MH; ++m)
        if (dyr == 2 * m) {
#pragma unroll
          for (int j = 0; j < 4; ++j)  // co g (j even) or g + 8, two pixels
            dbs[j & 1] += __uint_as_float(a[m][j] << 16) + __uint_as_float(a[m][j] & 0xffff0000u);
        }
    }
    db[0] += dbs[0];
    db[1] += dbs[1];
    ++since;
    if constexpr (kShort)
      if (since % kFlush == 0) flush();
    __syncthreads();  // the stage is free for the load after next
    if constexpr (!kShort)
      if (since % kPart == 0) put();
  }
  if constexpr (kShort) {
    flush();
    each([&](int d, int m, int nt, int j) { acc[d][m][nt][j] = sum[d][m][nt][j]; });
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) db[j] += __shfl_xor_sync(0xffffffffu, db[j], o);
  put();
  for (int k = 0; k < 5; ++k) {
#pragma unroll
    for (int m = 0; m < MH; ++m)
      if (kg == k && dyr == 2 * m && t4 == 0) {
        redb[m * 16 + g] += db[0];
        redb[m * 16 + g + 8] += db[1];
      }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < 9 * kWMat; i += blockDim.x)
    if ((MH == 2 || (i / kC) % kC < 16) && (NT == 4 || i % kC < 8)) dw_part[i] = red[i];
  if (threadIdx.x < MH * 16) db_part[threadIdx.x] = redb[threadIdx.x];
}

__global__ void __launch_bounds__(kDwThreads, 1)
k_cnn_dw(DwParts parts, const float *__restrict__ dy, const __nv_bfloat16 *__restrict__ dz,
         const uint32_t *__restrict__ xc, const __nv_bfloat16 *__restrict__ acts, int n, float *__restrict__ dw_part,
         float *__restrict__ db_part) {
  extern __shared__ __align__(128) unsigned char smraw[];
  int l = 0;
  while (l < kL - 1 && (int)blockIdx.x >= parts.first[l + 1]) ++l;
  const int part = blockIdx.x - parts.first[l], np = parts.first[l + 1] - parts.first[l];
  float *dw = dw_part + (int64_t)blockIdx.x * 9 * kWMat, *db = db_part + (int64_t)blockIdx.x * kC;
  if (l == 0) dw_layer<2, 1>(smraw, l, part, np, dy, dz, xc, acts, n, dw, db);
  else if (l < kL - 1) dw_layer<2, 4>(smraw, l, part, np, dy, dz, xc, acts, n, dw, db);
  else dw_layer<1, 4>(smraw, l, part, np, dy, dz, xc, acts, n, dw, db);
}

// Fixed-order sum of the per-CTA partials into the gradient (master layout), all layers in
// one launch, a thread per parameter (16 CTAs a layer were latency-bound: 6 x 37 us).
// add: to the gradient of the samples before.
__global__ void k_cnn_reduce(DwParts parts, const float *__restrict__ dw_part, const float *__restrict__ db_part,
                             float *__restrict__ grad, bool add) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nparams()) return;
  int l = 0;
  while (l < kL - 1 && i >= woff(l + 1)) ++l;
  const int co_n = cout(l), ci_n = cin(l), j = i - woff(l);
  const float *src;
  int stride;
  if (j < 9 * co_n * ci_n) {
    const int tap = j / (co_n * ci_n), rem = j % (co_n * ci_n);
    src = dw_part + tap * kWMat + (rem / ci_n) * kC + rem % ci_n;
    stride = 9 * kWMat;
  } else {
    src = db_part + (j - 9 * co_n * ci_n);
    stride = kC;
  }
  float s = 0.f;
#pragma unroll 8
  for (int k = parts.first[l]; k < parts.first[l + 1]; ++k) s += src[(int64_t)k * stride];
  grad[i] = add ? grad[i] + s : s;
}

#include "srmg_cnn_tc.cuh"

// Packed BF16 weights from the master vector: wpk (forward: rows co, columns ci) and
// wt (input gradient: rows ci, columns co), both [layer][tap][32 x 32 swizzled], zero
// where a layer has fewer channels; bias [layer][32].
__global__ void k_cnn_pack(const float *__restrict__ master, __nv_bfloat16 *__restrict__ wpk,
                           __nv_bfloat16 *__restrict__ wt, float *__restrict__ bias, unsigned char *__restrict__ wtc) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kL * 9 * kWMat; i += gridDim.x * blockDim.x) {
    const int l = i / (9 * kWMat), rem = i % (9 * kWMat), tap = rem / kWMat, r = (rem % kWMat) / kC,
              c = rem % kC;
    // forward: row co = r, column ci = c
    float vf = 0.f, vt = 0.f;
    if (r < cout(l) && c < cin(l)) vf = master[woff(l) + (tap * cout(l) + r) * cin(l) + c];
    // transposed: row ci = r, column co = c
    if (c < cout(l) && r < cin(l)) vt = master[woff(l) + (tap * cout(l) + c) * cin(l) + r];
    const int base = (l * 9 + tap) * kWMat * 2;
    *reinterpret_cast<__nv_bfloat16 *>(reinterpret_cast<char *>(wpk) + base + swz(r, c)) = __float2bfloat16_rn(vf);
    *reinterpret_cast<__nv_bfloat16 *>(reinterpret_cast<char *>(wt) + base + swz(r, c)) = __float2bfloat16_rn(vt);
    // tensor-core copy: canonical no-swizzle K-major, rows co, 16-byte chunks of ci
    *reinterpret_cast<__nv_bfloat16 *>(wtc + (l * 9 + tap) * 2048 + cm_off(r, c >> 3) + (c & 7) * 2) =
        __float2bfloat16_rn(vf);
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kL * kC; i += gridDim.x * blockDim.x) {
    const int l = i / kC, co = i % kC;
    bias[i] = co < cout(l) ? master[boff(l) + co] : 0.f;
  }
}

// Adam (Kingma & Ba 2015) on the FP32 master parameters.
__global__ void k_cnn_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                           float *__restrict__ v, int np, float lr, float b1, float b2, float eps, float c1,
                           float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// Samples of a tree: for leaf-holding block k (leaf[k] = {block, level}) the 20 x 20
// tile of (f * a, g * bsc), pixel order y * 20 + x, and the output scale
// s_level * |g| of the block.
__global__ void k_cnn_gather(const double *__restrict__ phi, const double *__restrict__ db, const int2 *__restrict__ leaf,
                             int nleaf, const double *__restrict__ norms, double s, __nv_bfloat16 *__restrict__ x,
                             double *__restrict__ scale, int *__restrict__ blk, const int *__restrict__ list = nullptr,
                             const int *__restrict__ count = nullptr) {
  // norms[0] = |phi|, norms[1] = |db| (leaf norms); 0 counts as 1.  With a list, sample
  // k is leaf block list[k], k < *count.
  const double a = norms[0] > 0 ? 1.0 / norms[0] : 1.0, bsc = norms[1] > 0 ? 1.0 / norms[1] : 1.0;
  const double dbrms = norms[1] > 0 ? norms[1] : 1.0;
  const int n = count ? min(nleaf, *count) : nleaf;
  const int64_t total = (int64_t)n * kNP;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int k = (int)(i / kNP), p = (int)(i % kNP);
    const int2 lb = leaf[list ? list[k] : k];
    const int64_t o = (int64_t)lb.x * kNP + p;
    reinterpret_cast<__nv_bfloat162 *>(x)[i] =
        __floats2bfloat162_rn((float)(phi[o] * a), (float)(db[o] * bsc));
    if (p == 0) {
      const double f = (double)((int64_t)1 << (lb.y - 1));
      scale[k] = s / (f * f) * dbrms;
      blk[k] = lb.x;
    }
  }
}

// Guess on the valid cells of every leaf-holding block: u = phi + y * scale.
__global__ void k_cnn_scatter(double *__restrict__ u, const double *__restrict__ phi, const float *__restrict__ y,
                              const double *__restrict__ scale, const int2 *__restrict__ leaf, int nleaf,
                              const int *__restrict__ list = nullptr, const int *__restrict__ count = nullptr) {
  const int n = count ? min(nleaf, *count) : nleaf;
  const int64_t total = (int64_t)n * 256;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int k = (int)(i >> 8), c = (int)(i & 255);
    const int64_t o = (int64_t)leaf[list ? list[k] : k].x * kNP + (2 + (c >> 4)) * kT + 2 + (c & 15);
    u[o] = phi[o] + (double)y[i] * scale[k];
  }
}

// d = ca a + cb b + cc c (b, c optional).
__global__ void k_lin_field(double *__restrict__ d, const double *__restrict__ a, double ca,
                            const double *__restrict__ b, double cb, const double *__restrict__ c, double cc,
                            int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double v = ca * a[i];
    if (b) v += cb * b[i];
    if (c) v += cc * c[i];
    d[i] = v;
  }
}

// Leaf-cell sums of squares of up to three fields over the leaf-holding blocks, one
// 256-thread block per tree block: part[k * 3 + j] = 4^-(l-1) sum over the block's leaf
// cells of f_j^2.  With `resid`, f_j is the residual -(b + L v_j / s_l) of candidate
// v_j instead of v_j itself.
__global__ void __launch_bounds__(256) k_leaf_sq3(const double *__restrict__ v0, const double *__restrict__ v1,
                                                  const double *__restrict__ v2, int nf, const double *__restrict__ b,
                                                  bool resid, double s, int op, double k2, int geom,
                                                  WTab<double> wt, const int2 *__restrict__ leaf,
                                                  const int4 *__restrict__ info, int nleaf,
                                                  double *__restrict__ part) {
  __shared__ double red[3][8];
  const int t = threadIdx.x;
  const int x = 2 + (t & 15), y = 2 + (t >> 4), o = x + kS * y;
  const int sub = ((x - 2) >> 3) + 2 * ((y - 2) >> 3);
  for (int k = blockIdx.x; k < nleaf; k += gridDim.x) {
    const int2 lb = leaf[k];
    const int4 bi = info[lb.x];
    const bool is_leaf = !(((bi.z & 15) >> sub) & 1);
    const double f = (double)((int64_t)1 << (lb.y - 1));
    const double sl = s / (f * f), wl = 1.0 / (f * f);
    const double centre = op == 1 ? -4.0 - sl * k2 : -4.0;
    const int64_t base = (int64_t)lb.x * kSS;
    const W5<double> w = weights<double>(wt, geom, bi.x, bi.y, x, y);
    double sq[3] = {0.0, 0.0, 0.0};
    const double *vs[3] = {v0, v1, v2};
    for (int j = 0; j < nf; ++j) {
      double val = vs[j][base + o];
      if (resid) val = -(b[base + o] + apply5<double>(vs[j] + base, x, y, w, centre) / sl);
      sq[j] = is_leaf ? val * val : 0.0;
    }
    for (int j = 0; j < 3; ++j) {
      double v = sq[j];
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if ((t & 31) == 0) red[j][t >> 5] = v;
    }
    __syncthreads();
    if (t < 3) {
      double c = 0.0;
      for (int q = 0; q < 8; ++q) c += red[t][q];
      part[(int64_t)k * 3 + t] = c * wl;
    }
    __syncthreads();
  }
}

// Fixed-order sums of the per-block partials: out[j] = sqrt(sum_k part[k * 3 + j]).
__global__ void __launch_bounds__(1024) k_leaf_sq3_reduce(const double *__restrict__ part, int nleaf, int nf,
                                                         double *__restrict__ out) {
  __shared__ double red[3][32];
  double v[3] = {0.0, 0.0, 0.0};
  for (int k = threadIdx.x; k < nleaf; k += blockDim.x)
    for (int j = 0; j < nf; ++j) v[j] += part[(int64_t)k * 3 + j];
  for (int j = 0; j < 3; ++j) {
    double a = v[j];
    for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
    if ((threadIdx.x & 31) == 0) red[j][threadIdx.x >> 5] = a;
  }
  __syncthreads();
  if (threadIdx.x < (unsigned)nf) {
    double c = 0.0;
    for (int q = 0; q < 32; ++q) c += red[threadIdx.x][q];
    out[threadIdx.x] = sqrt(c);
  }
}

// Active blocks: the leaf-holding blocks whose g energy (part[k * 3 + 1]) is at least
// theta times the largest, listed in leaf order (one CTA, fixed order).
__global__ void __launch_bounds__(1024) k_select_active(const double *__restrict__ part, int nleaf, double theta,
                                                       int *__restrict__ list, int *__restrict__ count) {
  __shared__ double smax[32];
  __shared__ int scnt[1024];
  double m = 0.0;
  for (int k = threadIdx.x; k < nleaf; k += blockDim.x) m = fmax(m, part[(int64_t)k * 3 + 1]);
  for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, off));
  if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double mm = 0.0;
    for (int q = 0; q < 32; ++q) mm = fmax(mm, smax[q]);
    smax[0] = mm;
  }
  __syncthreads();
  const double thr = theta * smax[0];
  const int chunk = (nleaf + blockDim.x - 1) / blockDim.x;
  const int k0 = threadIdx.x * chunk, k1 = min(nleaf, k0 + chunk);
  int c = 0;
  for (int k = k0; k < k1; ++k) c += part[(int64_t)k * 3 + 1] >= thr && part[(int64_t)k * 3 + 1] > 0.0;
  scnt[threadIdx.x] = c;
  __syncthreads();
  for (int off = 1; off < (int)blockDim.x; off <<= 1) {  // inclusive scan
    const int v = threadIdx.x >= (unsigned)off ? scnt[threadIdx.x - off] : 0;
    __syncthreads();
    scnt[threadIdx.x] += v;
    __syncthreads();
  }
  int w = scnt[threadIdx.x] - c;
  for (int k = k0; k < k1; ++k)
    if (part[(int64_t)k * 3 + 1] >= thr && part[(int64_t)k * 3 + 1] > 0.0) list[w++] = k;
  if (threadIdx.x == blockDim.x - 1) *count = scnt[threadIdx.x];
}

// f = u - phi2, g = b - 2 b1 + b2, ext = u + f, lrn = ext (every element).
__global__ void k_predict_prep(const double *__restrict__ u, const double *__restrict__ phi2,
                               const double *__restrict__ b, const double *__restrict__ b1,
                               const double *__restrict__ b2, double *__restrict__ f, double *__restrict__ g,
                               double *__restrict__ ext, double *__restrict__ lrn, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double ui = u[i], fi = ui - phi2[i];
    f[i] = fi;
    g[i] = b[i] - 2.0 * b1[i] + b2[i];
    ext[i] = ui + fi;
    lrn[i] = ui + fi;
  }
}

// Keep the candidate with the smallest residual norm (ties: the earlier one):
// r[0] previous potential (u itself), r[1] ext, r[2] lrn; copy it into u.
__global__ void k_predict_select(double *__restrict__ u, const double *__restrict__ ext,
                                 const double *__restrict__ lrn, const double *__restrict__ r, int *__restrict__ pick,
                                 int64_t n) {
  int p = 0;
  if (r[1] < r[0]) p = 1;
  if (r[2] < (p ? r[1] : r[0])) p = 2;
  if (blockIdx.x == 0 && threadIdx.x == 0) *pick = p;
  if (p == 0) return;
  const double *src = p == 1 ? ext : lrn;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    u[i] = src[i];
}

}  // namespace cnn

using namespace cnn;

struct srmg_cnn {
  int device = 0;
  cudaStream_t stream = nullptr;
  srmg_ctx *err_ctx = nullptr;  // error strings
  float *master = nullptr, *grad = nullptr, *adam_m = nullptr, *adam_v = nullptr;
  __nv_bfloat16 *wpk = nullptr, *wt = nullptr;
  float *bias = nullptr;
  unsigned char *wtc = nullptr;  // weights in the tcgen05 operand layout
  int *tc_err = nullptr;         // error word of the tcgen05 forward
  bool use_tc = false;           // the warm start's forward pass on tcgen05
  int adam_t = 0;
  int train_n = 0;  // samples of the last training forward
  DevBuf xc, acts, signs, dz, dy, dwp, dbp, lossp, y;
  int nsm = 0;
};

namespace {

int cnn_grid(srmg_cnn *net, int n) { return std::max(1, std::min(n, net->nsm)); }

int cnn_pack(srmg_cnn *net) {
  k_cnn_pack<<<64, 256, 0, net->stream>>>(net->master, net->wpk, net->wt, net->bias, net->wtc);
  return cuda_check(net->err_ctx, cudaGetLastError(), "k_cnn_pack");
}

int cnn_setup_attrs(srmg_cnn *net) {
  srmg_ctx *ctx = net->err_ctx;
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  CK(cudaFuncSetAttribute(k_cnn_fwd<5, false>, attr, fwd_smem(5)));
  CK(cudaFuncSetAttribute(k_cnn_fwd<5, true>, attr, fwd_smem(5)));
  CK(cudaFuncSetAttribute(k_cnn_fwd<13, false>, attr, fwd_smem(13)));
  CK(cudaFuncSetAttribute(k_cnn_fwd<13, true>, attr, fwd_smem(13)));
  CK(cudaFuncSetAttribute(k_cnn_dx<5>, attr, bwd_smem(5)));
  CK(cudaFuncSetAttribute(k_cnn_dx<13>, attr, bwd_smem(13)));
  CK(cudaFuncSetAttribute(k_cnn_dw, attr, kDwSmem));
  CK(cudaFuncSetAttribute(k_cnn_fwd_tc, attr, (int)sizeof(TcSmem)));
  return SRMG_OK;
}

// Launches the forward pass.  Up to one sample per SM the whole CTA works on one sample
// (13 warps), above that three samples share an SM (5 warps each).
template <bool TRAIN>
void launch_fwd(srmg_cnn *net, cudaStream_t stream, const __nv_bfloat16 *x, int n, float *y, const int *n_dev) {
  uint32_t *xc = (uint32_t *)net->xc.p;
  __nv_bfloat16 *acts = (__nv_bfloat16 *)net->acts.p;
  unsigned char *signs = (unsigned char *)net->signs.p;
  if (n <= net->nsm)
    k_cnn_fwd<13, TRAIN><<<n, cnn_threads(13), fwd_smem(13), stream>>>(x, n, net->wpk, net->bias, y, xc, acts, signs,
                                                                      n_dev);
  else
    k_cnn_fwd<5, TRAIN><<<net->nsm, cnn_threads(5), fwd_smem(5), stream>>>(x, n, net->wpk, net->bias, y, xc, acts,
                                                                          signs, n_dev);
}

// Forward pass keeping every layer's activations (training), outputs in net->y.
int cnn_fwd_train(srmg_cnn *net, const __nv_bfloat16 *x, int n) {
  srmg_ctx *ctx = net->err_ctx;
  const size_t layer = (size_t)n * kNP * kC * 2;  // one layer's activations or gradients
  RC(ensure(ctx, net->xc, (size_t)n * kNP * 4));
  RC(ensure(ctx, net->acts, (kL - 1) * layer));
  RC(ensure(ctx, net->signs, (size_t)(kL - 1) * n * kNP * 4));
  RC(ensure(ctx, net->dz, (size_t)std::min(n, kBwdSamples) * (kL - 1) * kNP * kC * 2));
  RC(ensure(ctx, net->y, (size_t)n * 256 * 4));
  RC(ensure(ctx, net->dy, (size_t)n * 256 * 4));
  RC(ensure(ctx, net->dwp, (size_t)net->nsm * 9 * kWMat * 4));
  RC(ensure(ctx, net->dbp, (size_t)net->nsm * kC * 4));
  RC(ensure(ctx, net->lossp, 1024 * 8));
  launch_fwd<true>(net, net->stream, x, n, (float *)net->y.p, nullptr);
  CK(cudaGetLastError());
  net->train_n = n;
  return SRMG_OK;
}

// The layers' shares of the weight-gradient CTAs: one CTA per SM, by the layers' work per
// sample (the first layer has 2 input channels, the last one output channel and its flushes:
// the backward pass at 1024 samples takes 331 us, with 0.6 instead of 0.7 17 us more).
DwParts dw_parts(int nsm, int n) {
  static const double work[kL] = {0.4, 1, 1, 1, 1, 0.7};
  DwParts p;
  p.first[0] = 0;
  double done = 0.0;
  for (int l = 0; l < kL; ++l) {
    done += work[l] / 5.1;
    const int to = l == kL - 1 ? nsm : (int)std::lround(done * nsm);
    p.first[l + 1] = p.first[l] + std::max(1, std::min(n, to - p.first[l]));
  }
  return p;
}

// Backward from the output gradient held in net->dy (n samples of the last forward), up to
// kBwdSamples at a time: their gradients of all five layers are in memory together (1 GB),
// and with those of a whole large batch a training step would need more than the 205 KB a
// sample that activations and two layers' gradients take (140 KB so).
int cnn_bwd(srmg_cnn *net, int n) {
  srmg_ctx *ctx = net->err_ctx;
  for (int s0 = 0; s0 < n; s0 += kBwdSamples) {
    const int m = std::min(n - s0, kBwdSamples);
    const float *dy = (const float *)net->dy.p + (int64_t)s0 * 256;
    const unsigned char *signs = (const unsigned char *)net->signs.p + (int64_t)s0 * (kL - 1) * kNP * 4;
    const __nv_bfloat16 *acts = (const __nv_bfloat16 *)net->acts.p + (int64_t)s0 * (kL - 1) * kNP * kC;
    const uint32_t *xc = (const uint32_t *)net->xc.p + (int64_t)s0 * kNP;
    __nv_bfloat16 *dz = (__nv_bfloat16 *)net->dz.p;
    if (m <= net->nsm) k_cnn_dx<13><<<m, cnn_threads(13), bwd_smem(13), net->stream>>>(dy, net->wt, signs, dz, m);
    else k_cnn_dx<5><<<net->nsm, cnn_threads(5), bwd_smem(5), net->stream>>>(dy, net->wt, signs, dz, m);
    const DwParts parts = dw_parts(net->nsm, m);
    k_cnn_dw<<<parts.first[kL], kDwThreads, kDwSmem, net->stream>>>(parts, dy, dz, xc, acts, m, (float *)net->dwp.p,
                                                                    (float *)net->dbp.p);
    k_cnn_reduce<<<(nparams() + 127) / 128, 128, 0, net->stream>>>(parts, (const float *)net->dwp.p,
                                                                  (const float *)net->dbp.p, net->grad, s0 > 0);
  }
  CK(cudaGetLastError());
  return SRMG_OK;
}

// Forward + loss + backward: gradient (master layout) in net->grad, loss partials.
int cnn_grad(srmg_cnn *net, const __nv_bfloat16 *x, const float *t, const int *ir0, float lambda, int geom, int n,
             double *loss) {
  srmg_ctx *ctx = net->err_ctx;
  RC(cnn_fwd_train(net, x, n));
  const int lg = std::min(1024, n);
  k_cnn_loss<<<lg, 256, 0, net->stream>>>((const float *)net->y.p, t, x, ir0, ir0 ? lambda : 0.f, geom, n,
                                          (float *)net->dy.p, (double *)net->lossp.p);
  RC(cnn_bwd(net, n));
  if (loss) {
    std::vector<double> lp(lg);
    CK(cudaMemcpyAsync(lp.data(), net->lossp.p, lg * sizeof(double), cudaMemcpyDeviceToHost, net->stream));
    CK(cudaStreamSynchronize(net->stream));
    double s = 0.0;
    for (double v : lp) s += v;
    *loss = s;
  }
  return SRMG_OK;
}

}  // namespace

extern "C" int srmg_cnn_nparams(void) { return nparams(); }

extern "C" int srmg_cnn_create(srmg_cnn **out, int device, uint64_t seed) {
  if (!out) return SRMG_ERR_BADARG;
  *out = nullptr;
  srmg_ctx *ctx = nullptr;
  int rc = srmg_create(&ctx, 2, 16, 2, device);
  if (rc) return rc;
  srmg_cnn *net = new srmg_cnn();
  net->device = device;
  net->err_ctx = ctx;
  net->stream = ctx->stream;
  cudaDeviceGetAttribute(&net->nsm, cudaDevAttrMultiProcessorCount, device);
  const int np = nparams();
  // He initialisation (normal, std sqrt(2 / fan_in)) from a splitmix64 stream, biases 0
  std::vector<float> h(np, 0.f);
  uint64_t st = seed ^ 0x9E3779B97F4A7C15ull;
  auto next = [&]() {
    uint64_t z = (st += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
  };
  for (int l = 0; l < kL; ++l) {
    const double sd = std::sqrt(2.0 / (9.0 * cin(l))) * (l == kL - 1 ? 0.1 : 1.0);
    for (int i = 0; i < 9 * cout(l) * cin(l); ++i) {
      const double u1 = std::max(next(), 1e-300), u2 = next();
      h[woff(l) + i] = (float)(sd * std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2));
    }
  }
  auto dalloc = [&](void **p, size_t b) { return cudaMalloc(p, b) == cudaSuccess; };
  if (!dalloc((void **)&net->master, np * 4) || !dalloc((void **)&net->grad, np * 4) ||
      !dalloc((void **)&net->adam_m, np * 4) || !dalloc((void **)&net->adam_v, np * 4) ||
      !dalloc((void **)&net->wpk, kWElems * 2) || !dalloc((void **)&net->wt, kWElems * 2) ||
      !dalloc((void **)&net->bias, kL * kC * 4) || !dalloc((void **)&net->wtc, kTcWBytes) ||
      !dalloc((void **)&net->tc_err, sizeof(int))) {
    srmg_cnn_destroy(net);
    return SRMG_ERR_NOMEM;
  }
  // Everything on the network's stream, in order: the stream is non-blocking, so
  // nothing orders it after work on the legacy default stream (a plain cudaMemset of
  // wtc could otherwise land after the pack below and wipe it).
  bool set = cudaMemcpyAsync(net->master, h.data(), np * 4, cudaMemcpyHostToDevice, net->stream) == cudaSuccess;
  for (auto [p, b] : {std::pair<void *, size_t>{net->adam_m, np * 4}, {net->adam_v, np * 4}, {net->grad, np * 4},
                      {net->wtc, (size_t)kTcWBytes}, {net->tc_err, sizeof(int)}})
    set = set && cudaMemsetAsync(p, 0, b, net->stream) == cudaSuccess;
  if (!set) {
    srmg_cnn_destroy(net);
    return SRMG_ERR_CUDA;
  }
  if ((rc = cnn_setup_attrs(net)) || (rc = cnn_pack(net))) {
    srmg_cnn_destroy(net);
    return rc;
  }
  cudaStreamSynchronize(net->stream);
  *out = net;
  return SRMG_OK;
}

extern "C" void srmg_cnn_destroy(srmg_cnn *net) {
  if (!net) return;
  cudaSetDevice(net->device);
  cudaStreamSynchronize(net->stream);
  for (void *p : {(void *)net->master, (void *)net->grad, (void *)net->adam_m, (void *)net->adam_v, (void *)net->wpk,
                  (void *)net->wt, (void *)net->bias, (void *)net->wtc, (void *)net->tc_err})
    if (p) cudaFree(p);
  for (DevBuf *b : {&net->xc, &net->acts, &net->signs, &net->dz, &net->dy, &net->dwp, &net->dbp, &net->lossp, &net->y})
    if (b->p) cudaFree(b->p);
  if (net->err_ctx) srmg_destroy(net->err_ctx);
  delete net;
}

extern "C" const char *srmg_cnn_last_error(const srmg_cnn *net) {
  return net ? srmg_last_error(net->err_ctx) : "null network";
}

extern "C" int srmg_cnn_get_params(srmg_cnn *net, float *host, int n) {
  if (!net || !host || n != nparams()) return SRMG_ERR_BADARG;
  cudaSetDevice(net->device);
  srmg_ctx *ctx = net->err_ctx;
  CK(cudaMemcpyAsync(host, net->master, n * 4, cudaMemcpyDeviceToHost, net->stream));
  CK(cudaStreamSynchronize(net->stream));
  return SRMG_OK;
}

extern "C" int srmg_cnn_set_params(srmg_cnn *net, const float *host, int n) {
  if (!net || !host || n != nparams()) return SRMG_ERR_BADARG;
  cudaSetDevice(net->device);
  srmg_ctx *ctx = net->err_ctx;
  CK(cudaMemcpyAsync(net->master, host, n * 4, cudaMemcpyHostToDevice, net->stream));
  CK(cudaMemsetAsync(net->adam_m, 0, n * 4, net->stream));
  CK(cudaMemsetAsync(net->adam_v, 0, n * 4, net->stream));
  net->adam_t = 0;
  RC(cnn_pack(net));
  CK(cudaStreamSynchronize(net->stream));
  return SRMG_OK;
}

extern "C" int srmg_cnn_forward(srmg_cnn *net, const uint16_t *x, float *y, int n) {
  if (!net || !x || !y || n < 0) return SRMG_ERR_BADARG;
  if (n == 0) return SRMG_OK;
  cudaSetDevice(net->device);
  srmg_ctx *ctx = net->err_ctx;
  launch_fwd<false>(net, net->stream, (const __nv_bfloat16 *)x, n, y, nullptr);
  CK(cudaGetLastError());
  return SRMG_OK;
}

extern "C" int srmg_cnn_forward_tc(srmg_cnn *net, const uint16_t *x, float *y, int n) {
  if (!net || !x || !y || n < 0) return SRMG_ERR_BADARG;
  if (n == 0) return SRMG_OK;
  cudaSetDevice(net->device);
  srmg_ctx *ctx = net->err_ctx;
  k_cnn_fwd_tc<<<cnn_grid(net, n), kTcThreads, sizeof(TcSmem), net->stream>>>((const __nv_bfloat16 *)x, n, net->wtc,
                                                                            net->bias, y, net->tc_err, nullptr);
  CK(cudaGetLastError());
  return SRMG_OK;
}

extern "C" int srmg_cnn_tc_status(srmg_cnn *net) {
  if (!net) return SRMG_ERR_BADARG;
  cudaSetDevice(net->device);
  srmg_ctx *ctx = net->err_ctx;
  int e = 0;
  CK(cudaStreamSynchronize(net->stream));
  CK(cudaMemcpy(&e, net->tc_err, sizeof(int), cudaMemcpyDeviceToHost));
  return e ? fail(ctx, SRMG_ERR_TIMEOUT, "tcgen05 forward: MMA completion wait timed out") : SRMG_OK;
}

extern "C" int srmg_cnn_use_tcgen05(srmg_cnn *net, int enable) {
  if (!net) return SRMG_ERR_BADARG;
  net->use_tc = enable != 0;
  return SRMG_OK;
}

extern "C" int srmg_cnn_gradients(srmg_cnn *net, const uint16_t *x, const float *t, const int *ir0, float lambda,
                                  int geom, int n, float *grad_host, double *loss) {
  if (!net || !x || !t || n <= 0 || lambda < 0 || geom < 0 || geom > 2) return SRMG_ERR_BADARG;
  cudaSetDevice(net->device);
  srmg_ctx *ctx = net->err_ctx;
  RC(cnn_grad(net, (const __nv_bfloat16 *)x, t, ir0, lambda, geom, n, loss));
  if (grad_host) {
    CK(cudaMemcpyAsync(grad_host, net->grad, nparams() * 4, cudaMemcpyDeviceToHost, net->stream));
    CK(cudaStreamSynchronize(net->stream));
  }
  return SRMG_OK;
}

static int cnn_adam_step(srmg_cnn *net, float lr) {
  net->adam_t++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - std::pow(b1, (float)net->adam_t), c2 = 1.f - std::pow(b2, (float)net->adam_t);
  k_cnn_adam<<<64, 256, 0, net->stream>>>(net->master, net->grad, net->adam_m, net->adam_v, nparams(), lr, b1, b2,
                                          1e-8f, c1, c2);
  return cnn_pack(net);
}

extern "C" int srmg_cnn_forward_train(srmg_cnn *net, const uint16_t *x, int n, float *y) {
  if (!net || !x || !y || n <= 0) return SRMG_ERR_BADARG;
  cudaSetDevice(net->device);
  srmg_ctx *ctx = net->err_ctx;
  RC(cnn_fwd_train(net, (const __nv_bfloat16 *)x, n));
  CK(cudaMemcpyAsync(y, net->y.p, (size_t)n * 256 * 4, cudaMemcpyDeviceToDevice, net->stream));
  CK(cudaStreamSynchronize(net->stream));
  return SRMG_OK;
}

extern "C" int srmg_cnn_backward_step(srmg_cnn *net, const float *dy, int n, float lr, float *grad_host) {
  if (!net || !dy || n <= 0 || n != net->train_n || lr < 0) return SRMG_ERR_BADARG;
  cudaSetDevice(net->device);
  srmg_ctx *ctx = net->err_ctx;
  // the caller's dy is its own to reuse: the backward kernels read a copy
  CK(cudaMemcpyAsync(net->dy.p, dy, (size_t)n * 256 * 4, cudaMemcpyDeviceToDevice, net->stream));
  RC(cnn_bwd(net, n));
  if (grad_host) {
    CK(cudaMemcpyAsync(grad_host, net->grad, nparams() * 4, cudaMemcpyDeviceToHost, net->stream));
    CK(cudaStreamSynchronize(net->stream));
  }
  if (lr > 0) RC(cnn_adam_step(net, lr));
  CK(cudaGetLastError());
  return SRMG_OK;
}

extern "C" int srmg_cnn_train_step(srmg_cnn *net, const uint16_t *x, const float *t, const int *ir0, float lambda,
                                   int geom, int n, float lr, double *loss) {
  if (!net || !x || !t || n <= 0 || !(lr > 0) || lambda < 0 || geom < 0 || geom > 2) return SRMG_ERR_BADARG;
  cudaSetDevice(net->device);
  srmg_ctx *ctx = net->err_ctx;
  RC(cnn_grad(net, (const __nv_bfloat16 *)x, t, ir0, lambda, geom, n, loss));
  RC(cnn_adam_step(net, lr));
  CK(cudaGetLastError());
  return SRMG_OK;
}

extern "C" int srmg_cnn_synchronize(srmg_cnn *net) {
  if (!net) return SRMG_ERR_BADARG;
  srmg_ctx *ctx = net->err_ctx;
  CK(cudaStreamSynchronize(net->stream));
  return SRMG_OK;
}

namespace {

int lin_field(srmg_ctx *ctx, double *d, const double *a, double ca, const double *b, double cb, const double *c,
              double cc, int64_t n) {
  k_lin_field<<<(int)std::min<int64_t>(4096, (n + 255) / 256), 256, 0, ctx->stream>>>(d, a, ca, b, cb, c, cc, n);
  return cuda_check(ctx, cudaGetLastError(), "k_lin_field");
}

// Leaf norms (sqrt of 4^-(l-1)-weighted sums over leaf cells) of up to three fields,
// or of their residuals, into out[0..nf) on the device.
int leaf_norms(srmg_ctx *ctx, const double *v0, const double *v1, const double *v2, int nf, const double *b,
               bool resid, double s, int op, double k2, int geom, double *part, double *out) {
  const int n = ctx->nleaf;
  if (n == 0) return cuda_check(ctx, cudaMemsetAsync(out, 0, nf * sizeof(double), ctx->stream), "memset");
  k_leaf_sq3<<<std::min(n, 148 * 8), 256, 0, ctx->stream>>>(v0, v1, v2, nf, b, resid, s, op, k2, geom,
                                                           WTab<double>{ctx->d_wm64, ctx->d_wp64}, ctx->d_leaf,
                                                           ctx->d_info, n, part);
  k_leaf_sq3_reduce<<<1, 1024, 0, ctx->stream>>>(part, n, nf, out);
  return cuda_check(ctx, cudaGetLastError(), "leaf norms");
}

// Samples of a tree from the input fields f (ghosts filled) and g (ghosts are filled
// here, on the copy gw unless gw == g): x, the per-sample output scale and block ids,
// with the input norms computed on the device (norms[0..1]).  No host synchronisation.
int cnn_pack_tree(srmg_ctx *ctx, const double *f, const double *g, double *gw, int64_t nblk_alloc, double s,
                  int op, double k2, int geom, const int8_t *bc, __nv_bfloat16 *x, double *scale, int *blk,
                  double *part, double *norms, int *list = nullptr, int *count = nullptr, double theta = 0.0) {
  const int64_t nval = nblk_alloc * (int64_t)kNP;
  if (gw != g) RC(lin_field(ctx, gw, g, 1.0, nullptr, 0.0, nullptr, 0.0, nval));
  const Signs sg = make_signs(bc);
  for (int l = 1; l <= ctx->nlev; l++) RC(L_fill_ghost<double>(ctx, gw, l, sg, 7));
  RC(leaf_norms(ctx, f, gw, nullptr, 2, nullptr, false, s, op, k2, geom, part, norms));
  const int n = ctx->nleaf;
  if (list) k_select_active<<<1, 1024, 0, ctx->stream>>>(part, n, theta, list, count);
  k_cnn_gather<<<(int)std::min<int64_t>(4096, ((int64_t)n * kNP + 255) / 256), 256, 0, ctx->stream>>>(
      f, gw, ctx->d_leaf, n, norms, s, x, scale, blk, list, count);
  CK(cudaGetLastError());
  return n;
}

}  // namespace

extern "C" int srmg_cnn_last_active(const srmg_ctx *ctx) { return ctx ? ctx->cnn_last_active : SRMG_ERR_BADARG; }

extern "C" int srmg_cnn_leaf_blocks(const srmg_ctx *ctx) {
  if (!ctx) return SRMG_ERR_BADARG;
  return ctx->has_tree ? ctx->nleaf : 0;
}

extern "C" int srmg_cnn_pack_dev(srmg_ctx *ctx, const double *f, const double *g, int64_t nblk_alloc, double s,
                                 int op, double k2, int geom, const int8_t bc[9], uint16_t *x, double *scale,
                                 int *blk, int max_samples) {
  RC(check_call(ctx, nblk_alloc, op, geom, bc));
  if (op == SRMG_OP_LAPLACIAN4)
    return fail(ctx, SRMG_ERR_UNSUPPORTED, "the learned warm start supports order-2 discretisations");
  if (!f || !g || !x || !scale || !blk) return fail(ctx, SRMG_ERR_BADARG, "srmg_cnn_pack_dev: null argument");
  if (max_samples < ctx->nleaf)
    return fail(ctx, SRMG_ERR_BADARG, "srmg_cnn_pack_dev: room for %d samples, the tree has %d", max_samples,
                ctx->nleaf);
  const int64_t nval = nblk_alloc * (int64_t)kNP;
  RC(ensure(ctx, ctx->cnn_work[0], nval * sizeof(double) + (3 * (size_t)ctx->nleaf + 8) * sizeof(double)));
  double *gw = (double *)ctx->cnn_work[0].p, *part = gw + nval, *norms = part + 3 * (size_t)ctx->nleaf;
  const int n = cnn_pack_tree(ctx, f, g, gw, nblk_alloc, s, op, k2, geom, bc, (__nv_bfloat16 *)x, scale, blk,
                              part, norms);
  if (n < 0) return n;
  CK(cudaStreamSynchronize(ctx->stream));
  return n;
}

extern "C" int srmg_cnn_predict_dev(srmg_ctx *ctx, srmg_cnn *net, double *u, const double *b, const double *b1,
                                    const double *phi2, const double *b2, int64_t nblk_alloc, double s, int op,
                                    double k2, int geom, const int8_t bc[9], int *which, double *resid) {
  RC(check_call(ctx, nblk_alloc, op, geom, bc));
  if (op == SRMG_OP_LAPLACIAN4)
    return fail(ctx, SRMG_ERR_UNSUPPORTED, "the learned warm start supports order-2 discretisations");
  if (!net || !u || !b || !b1 || !phi2 || !b2) return fail(ctx, SRMG_ERR_BADARG, "srmg_cnn_predict_dev: null argument");
  if (net->device != ctx->device) return fail(ctx, SRMG_ERR_BADARG, "network and context on different devices");
  const int n = ctx->nleaf;
  const int64_t nval = nblk_alloc * (int64_t)kNP;
  // work: f = u - phi2 (previous correction), g = b - 2 b1 + b2 (ghosts filled in place),
  // the extrapolated and the learned candidates, per-block partials and norms
  RC(ensure(ctx, ctx->cnn_work[1], (4 * (size_t)nval + 3 * (size_t)n + 16) * sizeof(double) + (n + 8) * sizeof(int)));
  double *f = (double *)ctx->cnn_work[1].p, *g = f + nval, *ext = g + nval, *lrn = ext + nval;
  double *part = lrn + nval, *norms = part + 3 * (size_t)n;  // norms[0..1] inputs, [2..4] residuals
  int *pick = (int *)(norms + 8), *count = pick + 1, *list = pick + 2;
  // x: [n][400][2] bf16; y: [n][256] float; scale: [n] double; blk: [n] int
  const size_t xb = (size_t)n * kNP * 2 * sizeof(__nv_bfloat16), yb = (size_t)n * 256 * sizeof(float),
               sb = (size_t)n * sizeof(double), bb = (size_t)n * sizeof(int);
  RC(ensure(ctx, ctx->cnn_work[2], xb + yb + sb + bb + 64));
  char *w = (char *)ctx->cnn_work[2].p;
  __nv_bfloat16 *x = (__nv_bfloat16 *)w;
  float *y = (float *)(w + ((xb + 15) & ~size_t(15)));
  double *scale = (double *)((char *)y + ((yb + 15) & ~size_t(15)));
  int *blk = (int *)((char *)scale + ((sb + 15) & ~size_t(15)));
  const int grid = (int)std::min<int64_t>(4096, (nval + 255) / 256);
  k_predict_prep<<<grid, 256, 0, ctx->stream>>>(u, phi2, b, b1, b2, f, g, ext, lrn, nval);
  CK(cudaGetLastError());
  // the network runs on the active blocks (g energy >= theta * the largest); the others
  // keep the extrapolation
  const double theta = ctx->cnn_active_ppm * 1e-6;
  const bool sel = ctx->cnn_active_ppm > 0;
  const int got = cnn_pack_tree(ctx, f, g, g, nblk_alloc, s, op, k2, geom, bc, x, scale, blk, part, norms,
                                sel ? list : nullptr, sel ? count : nullptr, theta);
  if (got < 0) return got;
  if (net->use_tc)
    k_cnn_fwd_tc<<<cnn_grid(net, n), kTcThreads, sizeof(TcSmem), ctx->stream>>>(x, n, net->wtc, net->bias, y,
                                                                                net->tc_err, sel ? count : nullptr);
  else
    launch_fwd<false>(net, ctx->stream, x, n, y, sel ? count : nullptr);
  CK(cudaGetLastError());
  k_cnn_scatter<<<(int)std::min<int64_t>(4096, ((int64_t)n * 256 + 255) / 256), 256, 0, ctx->stream>>>(
      lrn, ext, y, scale, ctx->d_leaf, n, sel ? list : nullptr, sel ? count : nullptr);
  // composite-grid functions of their leaves, ghosts filled
  const Signs sg = make_signs(bc);
  for (double *v : {ext, lrn}) {
    for (int l = ctx->nlev; l >= 2; l--) RC(L_restrict<double>(ctx, v, l));
    for (int l = 1; l <= ctx->nlev; l++) RC(L_fill_ghost<double>(ctx, v, l, sg, 7));
  }
  // residual norms of the three candidates; keep the smallest (device-side)
  RC(leaf_norms(ctx, u, ext, lrn, 3, b, true, s, op, k2, geom, part, norms + 2));
  k_predict_select<<<grid, 256, 0, ctx->stream>>>(u, ext, lrn, norms + 2, pick, nval);
  CK(cudaGetLastError());
  if (which || resid) {
    double h[3];
    int hp[2] = {0, n};
    CK(cudaMemcpyAsync(h, norms + 2, 3 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaMemcpyAsync(hp, pick, (sel ? 2 : 1) * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if (which) *which = hp[0];
    ctx->cnn_last_active = sel ? hp[1] : n;
    if (resid)
      for (int j = 0; j < 3; j++) resid[j] = h[j];
  }
  return SRMG_OK;
}
