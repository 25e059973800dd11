// srmg_stage.cu -- the stage preparation and post-processing around the field solve,
// on the device, so that a time step need not bring u, b or the charge through the
// host between the streamer update and the solve:
//   * netcharge! (src/streamer.jl:369-373) for the NetIonization chemistry;
//   * restrict_full! (src/restrict.jl:43-47) of a field over the whole tree;
//   * electric_field! (src/multigrid.jl:421-449) with a constant background field.
// For order-2 discretisations rhs_level! (src/multigrid.jl:363-388) is the identity,
// so the net charge itself is the solve's right-hand side.
#include <algorithm>
#include <cmath>

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

namespace {

// VectorBlockField{2, 16, 2} storage (src/blockfield.jl:84-95): (S+1) x (S+1) x 2 values
// per block, column-major, component d at offset d * (S+1)^2.
constexpr int kSV = kS + 1;
constexpr int kSSV = kSV * kSV;

// q = dot(n, (-1, +1)) = (-1 n_e) + (1 n_ion) on the valid cells of every block of the tree
// (used: the blocks' ids, null where they are 0..nblk-1): the products by +-1 are
// exact, so q is n_ion - n_e rounded once, as the reference computes it.  One launch for all
// levels, a thread per cell (V = double) or cell pair (V = double2, 16-byte aligned fields): a
// pure stream of 24 bytes a cell.  A launch per level with 8-byte accesses took 129 us
// on 51877 blocks (49 us of bytes).
template <typename V>
__global__ void __launch_bounds__(256) k_netcharge(double *__restrict__ q, const double *__restrict__ ne,
                                                   const double *__restrict__ nion, const int *__restrict__ used,
                                                   int nblk) {
  constexpr int W = sizeof(V) / sizeof(double), NR = kM / W;  // cells a thread, threads a row
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t k0 = t / (kM * NR);
  if (k0 >= nblk) return;
  const int64_t X = used ? used[k0] : k0;
  const int c = (int)(t % (kM * NR));
  const int64_t o = X * kSS + kS * (2 + c / NR) + 2 + W * (c % NR);
  V a = *reinterpret_cast<const V *>(ne + o), b = *reinterpret_cast<const V *>(nion + o);
  double *pa = reinterpret_cast<double *>(&a), *pb = reinterpret_cast<double *>(&b);
#pragma unroll
  for (int k = 0; k < W; ++k) pa[k] = __dadd_rn(-pa[k], pb[k]);
  *reinterpret_cast<V *>(q + o) = a;
}

// electric_field! on every block of the tree, a warp per pair of rows, a lane per valid cell.
// The face value f[I, d] = (u[I - e_d] - u[I]) / h_l + e0[d]: each lane forms its cell's lower
// faces; lanes 0..15 also the z faces above the upper row, lanes 16 and 17 the r faces at x =
// 18 (faces G+1 .. G+M+1 along d), and the upper faces of every cell come by shuffles --
// the division by h_l is most of the arithmetic (three a lane; four when each cell formed its
// upper faces too), and no warp waits for another.  |E| at the cell: sqrt((0 + s_1 s_1 / 4)
// + s_2 s_2 / 4), s_d = f[I, d] + f[I + e_d, d], every operation rounded on its own (no fused
// multiply-add; the quarter is exact either way), as in the reference.  One launch for
// all levels (info: block coordinates, child mask, level; used as in k_netcharge): a launch per
// level was 287 us on 51877 blocks, 650 MB of traffic (99 us).
// CTAs stream blocks through a ring of u tiles (cp.async, three blocks ahead).
constexpr int kEfRing = 4;
template <int CH>
__global__ void __launch_bounds__(256, 5) k_efield(double *__restrict__ e, double *__restrict__ eabs,
                                                   const double *__restrict__ u, const int4 *__restrict__ info,
                                                   const int *__restrict__ used, int nblk, double h1,
                                                   double rh1, double e0r, double e0z) {
  __shared__ __align__(16) double tile[kEfRing][kSS];
  const int lane = threadIdx.x & 31, cx = lane & 15, p = threadIdx.x >> 5;
  const int x = 2 + cx, y0 = 2 + 2 * p, y = y0 + (lane >> 4);
  const bool ez = lane < 16, er = lane == 16 || lane == 17;
  // the lane's extra face (any face of the tile where it has none)
  const int eo = ez ? x + kS * (y0 + 2) : 18 + kS * (y0 + (lane & 1)), el = eo - (ez ? kS : 1);
  auto fetch = [&](int j) {
    const int64_t k = blockIdx.x + (int64_t)j * gridDim.x;
    if (k < nblk) cp_tile<CH>(tile[j % kEfRing], u + (used ? used[k] : k) * kSS, kSS);
    cp_async_commit();
  };
  for (int j = 0; j < kEfRing - 1; ++j) fetch(j);
  for (int j = 0;; ++j) {
    const int64_t k = blockIdx.x + (int64_t)j * gridDim.x;
    if (k >= nblk) break;
    const int64_t X = used ? used[k] : k;
    const int level = info[X].w;
    cp_async_wait<kEfRing - 2>();
    __syncthreads();  // the tile is here, and no thread reads the last one's any more
    fetch(j + kEfRing - 1);
    const double *ub = tile[j % kEfRing];
    double *eb = e + X * (2 * kSSV);
    const double hl = __dmul_rn(h1, __hiloint2double((1024 - level) << 20, 0));   // h / 2^(level - 1)
    const double rh = __dmul_rn(rh1, __hiloint2double((1022 + level) << 20, 0));  // its reciprocal
    auto face = [&](double lo, double up, double e0) { return __dadd_rn(div_by(__dsub_rn(lo, up), hl, rh), e0); };
    const int o = x + kS * y;
    const double uc = ub[o];
    const double fr0 = face(ub[o - 1], uc, e0r), fz0 = face(ub[o - kS], uc, e0z);
    const double fx = face(ub[el], ub[eo], ez ? e0z : e0r);
    eb[x + kSV * y] = fr0;
    eb[kSSV + x + kSV * y] = fz0;
    if (er) eb[18 + kSV * (y0 + (lane & 1))] = fx;
    if (ez && p == 7) eb[kSSV + x + kSV * 18] = fx;
    const unsigned all = 0xffffffffu;
    const double nr = __shfl_down_sync(all, fr0, 1), xr = __shfl_sync(all, fx, 16 + (lane >> 4));
    const double nz = __shfl_down_sync(all, fz0, 16), xz = __shfl_sync(all, fx, cx);
    const double sr = __dadd_rn(fr0, cx == 15 ? xr : nr), sz = __dadd_rn(fz0, ez ? nz : xz);
    double f2 = __dadd_rn(0.0, __dmul_rn(__dmul_rn(sr, sr), 0.25));
    f2 = __dadd_rn(f2, __dmul_rn(__dmul_rn(sz, sz), 0.25));
    eabs[X * kSS + o] = __dsqrt_rn(f2);
  }
  cp_async_wait<0>();
}

}  // namespace

extern "C" int srmg_netcharge_dev(srmg_ctx *ctx, double *q, const double *ne, const double *nion,
                                  int64_t nblk_alloc) {
  RC(check_call(ctx, nblk_alloc, 0, 0, nullptr));
  if (!q || !ne || !nion) return fail(ctx, SRMG_ERR_BADARG, "srmg_netcharge: null field");
  const int64_t n = ctx->nused;
  if (n > 0) {
    const bool pairs = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(ne) |
                         reinterpret_cast<uintptr_t>(nion)) & 15) == 0;
    if (pairs) k_netcharge<double2><<<(unsigned)((n + 1) / 2), 256, 0, ctx->stream>>>(q, ne, nion, ctx->d_used, n);
    else k_netcharge<double><<<(unsigned)n, 256, 0, ctx->stream>>>(q, ne, nion, ctx->d_used, n);
    ctx->launches++;
  }
  CK(cudaGetLastError());
  return SRMG_OK;
}

extern "C" int srmg_restrict_full_dev(srmg_ctx *ctx, double *u, int64_t nblk_alloc) {
  RC(check_call(ctx, nblk_alloc, 0, 0, nullptr));
  if (!u) return fail(ctx, SRMG_ERR_BADARG, "srmg_restrict_full: null field");
  for (int l = ctx->nlev; l >= 2; l--) RC(srmg_restrict_level_dev(ctx, u, nblk_alloc, l));
  return SRMG_OK;
}

extern "C" int srmg_electric_field_dev(srmg_ctx *ctx, double *e, double *eabs, const double *u,
                                       int64_t nblk_alloc, double h, const double e0[2]) {
  RC(check_call(ctx, nblk_alloc, 0, 0, nullptr));
  if (!e || !eabs || !u || !e0) return fail(ctx, SRMG_ERR_BADARG, "srmg_electric_field: null argument");
  if (!(h > 0.0) || !std::isfinite(h)) return fail(ctx, SRMG_ERR_BADARG, "srmg_electric_field: h must be > 0");
  if (ctx->nused > 0) {
    const int grid = std::min(ctx->nused, 148 * 5);
    const auto kern = (reinterpret_cast<uintptr_t>(u) & 15) == 0 ? k_efield<16> : k_efield<8>;
    kern<<<grid, 256, 0, ctx->stream>>>(e, eabs, u, ctx->d_info, ctx->d_used, ctx->nused, h, recip_of(h), e0[0],
                                        e0[1]);
    ctx->launches++;
  }
  CK(cudaGetLastError());
  return SRMG_OK;
}

// Host-array variants (the ccall boundary): copies in, the device entry point, copies out.
extern "C" int srmg_netcharge(srmg_ctx *ctx, double *q, const double *ne, const double *nion, int64_t nblk_alloc) {
  RC(check_call(ctx, nblk_alloc, 0, 0, nullptr));
  if (!q || !ne || !nion) return fail(ctx, SRMG_ERR_BADARG, "srmg_netcharge: null field");
  double *dq, *dne, *dni;
  RC(stage_in(ctx, 0, q, nblk_alloc, &dq));
  RC(stage_in(ctx, 1, ne, nblk_alloc, &dne));
  RC(stage_in(ctx, 2, nion, nblk_alloc, &dni));
  RC(srmg_netcharge_dev(ctx, dq, dne, dni, nblk_alloc));
  RC(stage_out(ctx, q, dq, nblk_alloc));
  CK(cudaStreamSynchronize(ctx->stream));
  return SRMG_OK;
}

extern "C" int srmg_electric_field(srmg_ctx *ctx, double *e, double *eabs, const double *u, int64_t nblk_alloc,
                                   double h, const double e0[2]) {
  RC(check_call(ctx, nblk_alloc, 0, 0, nullptr));
  if (!e || !eabs || !u || !e0) return fail(ctx, SRMG_ERR_BADARG, "srmg_electric_field: null argument");
  double *du, *dabs;
  RC(stage_in(ctx, 0, u, nblk_alloc, &du));
  RC(stage_in(ctx, 1, eabs, nblk_alloc, &dabs));
  // the vector field (882 values per block) in the spare slot, copied in so that the
  // faces the reference does not write keep the caller's values
  const size_t vbytes = (size_t)nblk_alloc * 2 * kSSV * sizeof(double);
  RC(ensure(ctx, ctx->f64[2], vbytes));
  double *de = (double *)ctx->f64[2].p;
  CK(cudaMemcpyAsync(de, e, vbytes, cudaMemcpyHostToDevice, ctx->stream));
  RC(srmg_electric_field_dev(ctx, de, dabs, du, nblk_alloc, h, e0));
  CK(cudaMemcpyAsync(e, de, vbytes, cudaMemcpyDeviceToHost, ctx->stream));
  RC(stage_out(ctx, eabs, dabs, nblk_alloc));
  CK(cudaStreamSynchronize(ctx->stream));
  return SRMG_OK;
}
