// srmg_streamer.cu -- the electron transport and chemistry inside derivs!
// (src/streamer.jl:292-366) and the SSPRK3 stage combinations of step!
// (src/streamer.jl:386-425), on the device, for the streamer runs that generate the
// learned warm start's training pairs:
//   * flux! with the Koren scheme (src/fluid.jl:44-94): per leaf block and per face of
//     validindices(e, d), the upwind value n_u + koren_limited(n_u - n_u2, n_d - n_u)
//     (src/fluid.jl:265-280) times the drift velocity -mu E, plus the diffusion flux, and
//     the block's largest stable time step (CFL, diffusion, Maxwell relaxation);
//   * restrict_flux! (src/connectivity.jl:327-360): at every refinement boundary the
//     coarse block's face flux is the mean of the two fine face fluxes it covers;
//   * chemderivs! for NetIonization (src/chemistry.jl:29-82) with the MinimalTransportModel
//     (src/transport.jl:9-35): ionisation before the (empty) photoionization, attachment
//     after it, for both species (electrons and net positive ions);
//   * fluxderivs! (src/fluid.jl:8-30): the flux divergence with the geometry factors of
//     src/geometry.jl:27-29, accumulated face by face in the reference's order;
//   * the three SSPRK3 combinations n + dn1 dt, n + (dn1 dt/4 + dn2 dt/4),
//     n + ((dn1 dt/6 + dn2 dt/6) + dn3 2dt/3).
// Every operation is rounded on its own (no fused multiply-add), as in the reference,
// so fluxes, time steps and stage combinations are bit-exact against a restatement with
// IEEE double arithmetic; the chemistry calls exp(), which may differ in the last bit.
//
// The vector fields (e, flux) use the VectorBlockField{2, 16, 2} storage
// (src/blockfield.jl:84-95): 21 x 21 values per component, component d at offset 441 d,
// 882 values per block; face (x, y) of component d (0-based local indices) is the face
// between cell (x, y) - e_d and cell (x, y).
#include <algorithm>
#include <cmath>
#include <initializer_list>

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

constexpr int kSV = kS + 1;
constexpr int kSSV = kSV * kSV;

constexpr double kElemCharge = 1.6021766208e-19;  // src/constants.jl:55
constexpr double kEpsilon0 = 8.854187817620389e-12;  // src/constants.jl:56

__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dvd(double a, double b) { return __ddiv_rn(a, b); }

// Leaf blocks (no child in any subblock: isleaf, src/tree.jl:105-115) among the blocks
// holding a leaf cell.
__device__ __forceinline__ bool leaf_block(const int4 *info, int X) { return (info[X].z & 15) == 0; }

// Non-negative doubles order like their bit patterns as unsigned integers.
__device__ __forceinline__ void atomic_min_nonneg(double *addr, double v) {
  atomicMin(reinterpret_cast<unsigned long long *>(addr), (unsigned long long)__double_as_longlong(v));
}

// min(md, a / b) without the division where it cannot win: md > 0 and a > md b (1 + 8 eps)
// leave a / b above md.  (0 / 0 is NaN and ignored by fmin, as everywhere here.)
__device__ __forceinline__ double min_quotient(double md, double a, double b) {
  if (__double2hiint(md) > 0 && a > mul(mul(md, 1.0 + 8 * 2.220446049250313e-16), b)) return md;
  return fmin(md, dvd(a, b));
}

// Cell sizes of a level: h = h1 / 2^(l-1), its reciprocal and (h h / D) / 4.  Scaling by powers
// of two is exact, so the host forms the level-1 quotients once and the kernels need no
// division for them (dt1 < 0: some level's square or quotient could leave the normal range, and
// the limit is formed per block).
struct CellSize {
  double h1, rh1, dt1;
};
__device__ __forceinline__ double pow2(int k) { return __hiloint2double((1023 + k) << 20, 0); }

// The values a face of component d reads: E there, |E| on its two sides, n_e two cells either
// way along d.
struct FaceIn {
  double ed, e0, e1, n[4];
};
__device__ __forceinline__ FaceIn load_face(const double *eb, const double *ea, const double *n, int d, int x, int y) {
  const int st = d ? kS : 1, o = x + kS * y;
  FaceIn f;
  f.ed = eb[d * kSSV + x + kSV * y];
  f.e0 = ea[o];
  f.e1 = ea[o - st];
#pragma unroll
  for (int k = 0; k < 4; ++k) f.n[k] = n[o + (k - 2) * st];
  return f;
}

// The face's flux; md is lowered to its time-step limits h / |v| and the Maxwell time.
__device__ __forceinline__ double face_flux(const FaceIn &f, const srmg_transport &tr, double h, double rh, double r3,
                                            double r6, double &md) {
  const double eabs1 = mul(add(f.e0, f.e1), 0.5);  // exact either way
  const double v = mul(-f.ed, tr.mu);              // mobility / diffusion of the minimal model, theta = 1
  const bool neg = signbit(v);
  // downstream, upstream and twice-upstream cells along d
  const double nd = neg ? f.n[1] : f.n[2], nu = neg ? f.n[2] : f.n[1], nu2 = neg ? f.n[3] : f.n[0];
  const double a = sub(nu, nu2), b = sub(nd, nu);
  // koren_limited(a, b) = psi(a / b) b (src/fluid.jl:274-280)
  double lim = a;
  if (mul(a, b) < 0.0) lim = 0.0;
  else if (fabs(a) > fabs(mul(4.0, b))) lim = b;
  else if (fabs(mul(10.0, a)) > fabs(mul(4.0, b))) lim = add(div_by(b, 3.0, r3), div_by(a, 6.0, r6));
  double F = mul(v, add(nu, lim));
  const double maxwell = kEpsilon0 / kElemCharge;  // (co.epsilon_0 / co.elementary_charge)
  md = min_quotient(md, mul(maxwell, eabs1), fabs(F));
  md = min_quotient(md, h, fabs(v));
  return add(F, div_by(mul(tr.D, sub(f.n[1], f.n[2])), h, rh));
}

// The blocks a CTA streams: list entries blockIdx.x, + gridDim.x, ...; a ring of kRing tile
// sets in shared memory, the next kRing - 1 blocks' tiles in flight.
constexpr int kRing = 3;
constexpr int kTileSet = 2 * kSS + 2 * kSSV;  // n_e, |E| and a vector field, whole blocks
constexpr int kTileSetBytes = kTileSet * (int)sizeof(double);
constexpr int kFluxThreads = 288;             // 9 warps: 17 x 16 faces per dimension, one each a thread
constexpr int kFluxFaces = (kM + 1) * kM;

template <int CH>
__device__ __forceinline__ void load_set(double *sm, const double *a, const double *b, const double *vec, int X) {
  cp_tile<CH>(sm, a + (int64_t)X * kSS, kSS);
  cp_tile<CH>(sm + kSS, b + (int64_t)X * kSS, kSS);
  cp_tile<CH>(sm + 2 * kSS, vec + (int64_t)X * 2 * kSSV, 2 * kSSV);
}

// flux! (Koren) on the leaf blocks.  CTAs stream blocks: n_e, |E| and E tiles arrive by cp.async
// two blocks ahead, 272 threads take one face of each dimension.  A face is ~40 fp64
// operations (an fp64 instruction takes two issue slots) on 7 values: the divisions by h,
// 3 and 6 go through their reciprocals, and the time-step quotients are only formed where
// they can lower the minimum so far (over the thread's blocks; with BLK over the block, whose
// own minimum goes to maxdt_blk).  Bound by DRAM (740 MB on 51877 blocks, 113 us) and the
// fp64 pipe; 544 faces strided over 256 threads with eight divisions each, loads issued as
// needed and two barriers a block took 445 us.  ne needs 2 ghost layers, eabs 1.
template <bool BLK, int CH>
__global__ void __launch_bounds__(kFluxThreads, 4)
k_streamer_flux(double *__restrict__ flux, double *__restrict__ maxdt_blk, double *maxdt_min,
                const double *__restrict__ ne, const double *__restrict__ e, const double *__restrict__ eabs,
                const int2 *__restrict__ leaf, int nleaf, const int4 *__restrict__ info, CellSize cs,
                srmg_transport tr) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double s_min[kFluxThreads / 32];
  const int t = threadIdx.x, rx = 2 + t % (kM + 1), ry = 2 + t / (kM + 1), zx = 2 + (t & 15), zy = 2 + (t >> 4);
  const bool act = t < kFluxFaces;
  const double r3 = 1.0 / 3.0, r6 = 1.0 / 6.0;
  double md = INFINITY;
  auto fetch = [&](int j) {
    const int k = blockIdx.x + j * gridDim.x;
    if (k < nleaf) load_set<CH>(sm + (j % kRing) * kTileSet, ne, eabs, e, leaf[k].x);
    cp_async_commit();
  };
  for (int j = 0; j < kRing - 1; ++j) fetch(j);
  for (int j = 0;; ++j) {
    const int k = blockIdx.x + j * gridDim.x;
    if (k >= nleaf) break;
    const int2 lb = leaf[k];
    const int X = lb.x;
    const bool is_leaf = leaf_block(info, X);  // uniform per CTA
    cp_async_wait<kRing - 2>();
    __syncthreads();  // the block's tiles are here, and no thread reads the tiles of the last one any more
    fetch(j + kRing - 1);
    if (!is_leaf) continue;
    const double *n = sm + (j % kRing) * kTileSet, *ea = n + kSS, *eb = n + 2 * kSS;
    double *fb = flux + (int64_t)X * 2 * kSSV;
    const double h = mul(cs.h1, pow2(1 - lb.y)), rh = mul(cs.rh1, pow2(lb.y - 1));  // h /= 1 << (level - 1)
    const double dt = cs.dt1 >= 0.0 ? mul(cs.dt1, pow2(2 - 2 * lb.y)) : dvd(dvd(mul(h, h), tr.D), 4.0);
    md = BLK ? fmin(INFINITY, dt) : fmin(md, dt);
    if (act) {
      fb[rx + kSV * ry] = face_flux(load_face(eb, ea, n, 0, rx, ry), tr, h, rh, r3, r6, md);
      fb[kSSV + zx + kSV * zy] = face_flux(load_face(eb, ea, n, 1, zx, zy), tr, h, rh, r3, r6, md);
    }
    if (BLK) {
      double m = md;
      for (int off = 16; off > 0; off >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, off));
      if ((t & 31) == 0) s_min[t >> 5] = m;
      __syncthreads();
      if (t == 0) {
        for (int w = 1; w < kFluxThreads / 32; ++w) m = fmin(m, s_min[w]);
        maxdt_blk[X] = m;
        if (maxdt_min) atomic_min_nonneg(maxdt_min, m);
      }
    }
  }
  cp_async_wait<0>();
  if constexpr (!BLK) {
    if (!maxdt_min) return;
    for (int off = 16; off > 0; off >>= 1) md = fmin(md, __shfl_xor_sync(0xffffffffu, md, off));
    if ((t & 31) == 0 && md < INFINITY) atomic_min_nonneg(maxdt_min, md);
  }
}

// restrict_flux! over every refinement-boundary face of the tree in one launch (a face is
// next to either a coarser or a finer block, so no level's result feeds another's): thread
// (block, face, k) sets the coarse block's face k (0..7) of the half `subblock` covers to the
// mean of the two fine faces 2k, 2k + 1: f = ((0 + f_2k) + f_2k+1) / 2.
__global__ void k_restrict_flux(double *__restrict__ flux, const int4 *__restrict__ faceb,
                                const int *__restrict__ used, int nblk) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if ((t >> 5) >= nblk) return;
  const int64_t X = used ? used[t >> 5] : t >> 5;
  const int f = (int)(t >> 3) & 3, k = (int)(t & 7);
  const int4 fi = faceb[4 * X + f];
  if (fi.x != FACE_REFBND) return;
  const int d = f >> 1;  // the face's dimension: 0 for -r/+r, 1 for -z/+z
  const int fine_n = (f & 1) ? 2 + kM : 2, coarse_n = (f & 1) ? 2 : 2 + kM;  // normal face index
  const int sb = d == 0 ? fi.z >> 8 : fi.z & 255;  // the tangential half
  const int ct = 2 + 8 * (sb - 1) + k, ft = 2 + 2 * k;
  const double *src = flux + X * 2 * kSSV + d * kSSV;
  double *dst = flux + (int64_t)fi.y * 2 * kSSV + d * kSSV;
  auto at = [&](int nrm, int tan) { return d == 0 ? nrm + kSV * tan : tan + kSV * nrm; };
  const double s = add(add(0.0, src[at(fine_n, ft)]), src[at(fine_n, ft + 1)]);
  dst[at(coarse_n, ct)] = dvd(s, 2.0);
}

// chemderivs! (init, then add) and fluxderivs! on the valid cells of the leaf blocks:
// dni = pre + post; dne = (((pre + post) + lower-r) - upper-r) + lower-z) - upper-z,
// each face term (factor F) / h, factor = |1 + delta / (2 J - 1)| along the radial
// dimension (1 along the others and in Cartesian geometry).
// CTAs stream blocks as in k_streamer_flux, a thread a cell: grid-strided cells with ten
// divisions each, loads issued as needed, took 202 us on 51877 blocks (676 MB, 103 us); the
// factors' shared quotient and div_by leave three divisions and two exp, which the fp64
// pipe now shares the bound with.
template <int CH>
__global__ void __launch_bounds__(256, 4)
k_streamer_rates(double *__restrict__ dne, double *__restrict__ dni, const double *__restrict__ ne,
                 const double *__restrict__ eabs, const double *__restrict__ flux, const int2 *__restrict__ leaf,
                 int nleaf, const int4 *__restrict__ info, CellSize cs, int geom, srmg_transport tr) {
  extern __shared__ __align__(16) double sm[];
  const int x = 2 + (threadIdx.x & 15), y = 2 + (threadIdx.x >> 4), o = x + kS * y;
  auto fetch = [&](int j) {
    const int k = blockIdx.x + j * gridDim.x;
    if (k < nleaf) load_set<CH>(sm + (j % kRing) * kTileSet, ne, eabs, flux, leaf[k].x);
    cp_async_commit();
  };
  for (int j = 0; j < kRing - 1; ++j) fetch(j);
  for (int j = 0;; ++j) {
    const int k = blockIdx.x + j * gridDim.x;
    if (k >= nleaf) break;
    const int2 lb = leaf[k];
    const int64_t X = lb.x;
    const int4 bi = info[X];
    cp_async_wait<kRing - 2>();
    __syncthreads();  // as in k_streamer_flux
    fetch(j + kRing - 1);
    if ((bi.z & 15) != 0) continue;  // not a leaf block
    const double *s = sm + (j % kRing) * kTileSet, *fb = s + 2 * kSS;
    const double n1 = s[o], E = s[kSS + o];
    const double rl = fb[x + kSV * y], ru = fb[(x + 1) + kSV * y];
    const double zl = fb[kSSV + x + kSV * y], zu = fb[kSSV + x + kSV * (y + 1)];
    const double h = mul(cs.h1, pow2(1 - lb.y)), rh = mul(cs.rh1, pow2(lb.y - 1));
    // NetIonization, MinimalTransportModel: mobility mu, townsend ai exp(-Ei / E),
    // attachment aa exp(-Ea / E)
    const double pre = mul(mul(mul(tr.mu, E), n1), mul(tr.ai, exp(dvd(-tr.Ei, E))));
    const double post = mul(mul(mul(-tr.mu, E), n1), mul(tr.aa, exp(dvd(-tr.Ea, E))));
    const double chem = add(pre, post);
    dni[X * kSS + o] = chem;
    // factor(geom, J, +-e_dim) = |1 +- 1 / (2 J - 1)| along the radial dimension, else 1
    double lo = 1.0, up = 1.0;
    if (geom != 0) {
      const int64_t J = geom == 1 ? gidx(bi.x, x) : gidx(bi.y, y);
      const double q = dvd(1.0, (double)(2 * J - 1));
      lo = fabs(sub(1.0, q));
      up = fabs(add(1.0, q));
    }
    const bool r1 = geom == 1, r2 = geom == 2;
    double v = chem;
    v = add(v, div_by(r1 ? mul(lo, rl) : rl, h, rh));
    v = sub(v, div_by(r1 ? mul(up, ru) : ru, h, rh));
    v = add(v, div_by(r2 ? mul(lo, zl) : zl, h, rh));
    v = sub(v, div_by(r2 ? mul(up, zu) : zu, h, rh));
    dne[X * kSS + o] = v;
  }
  cp_async_wait<0>();
}

__global__ void k_init_min(double *m) { *m = INFINITY; }

// The SSPRK3 stage combinations of step! (src/streamer.jl:400-413), elementwise.
__global__ void k_ssprk3(double *__restrict__ out, const double *__restrict__ n, const double *__restrict__ d1,
                         const double *__restrict__ d2, const double *__restrict__ d3, int64_t count, double dt,
                         int stage) {
  const double dt1 = dvd(dt, 4.0), dt6 = dvd(dt, 6.0), dt23 = dvd(mul(2.0, dt), 3.0);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
    double inc;
    if (stage == 1) inc = mul(d1[i], dt);
    else if (stage == 2) inc = add(mul(d1[i], dt1), mul(d2[i], dt1));
    else inc = add(add(mul(d1[i], dt6), mul(d2[i], dt6)), mul(d3[i], dt23));
    out[i] = add(n[i], inc);
  }
}

int grid_of(int64_t work, int threads, int cap) {
  const int64_t g = (work + threads - 1) / threads;
  return (int)std::max<int64_t>(1, std::min<int64_t>(g, cap));
}

bool aligned16(std::initializer_list<const void *> ps) {
  uintptr_t v = 0;
  for (const void *p : ps) v |= reinterpret_cast<uintptr_t>(p);
  return (v & 15) == 0;
}

// Plain double operations, one rounding each (no contraction on the host side).
CellSize cell_size(double h, const srmg_transport &tr) {
  volatile double hh = h * h;
  volatile double q = hh / tr.D;
  auto safe = [](double v) { return v > 1e-200 && v < 1e200; };  // levels scale by 2^-58 at most
  return CellSize{h, recip_of(h), safe(hh) && safe(q) ? q / 4.0 : -1.0};
}

int check_transport(srmg_ctx *ctx, const srmg_transport *tr, const char *who) {
  if (!tr) return fail(ctx, SRMG_ERR_BADARG, "%s: null transport model", who);
  const double v[6] = {tr->mu, tr->D, tr->ai, tr->Ei, tr->aa, tr->Ea};
  for (double a : v)
    if (!std::isfinite(a)) return fail(ctx, SRMG_ERR_BADARG, "%s: transport values must be finite", who);
  if (!(tr->D > 0)) return fail(ctx, SRMG_ERR_BADARG, "%s: diffusion must be > 0", who);
  return SRMG_OK;
}

}  // namespace

extern "C" int srmg_streamer_flux_dev(srmg_ctx *ctx, double *flux, double *maxdt_blk, double *maxdt_min,
                                      const double *ne, const double *e, const double *eabs, int64_t nblk_alloc,
                                      double h, const srmg_transport *tr) {
  RC(check_call(ctx, nblk_alloc, 0, 0, nullptr));
  if (!flux || !ne || !e || !eabs) return fail(ctx, SRMG_ERR_BADARG, "srmg_streamer_flux_dev: null field");
  if (!(h > 0.0) || !std::isfinite(h)) return fail(ctx, SRMG_ERR_BADARG, "srmg_streamer_flux_dev: h must be > 0");
  RC(check_transport(ctx, tr, "srmg_streamer_flux_dev"));
  if (maxdt_min) {
    k_init_min<<<1, 1, 0, ctx->stream>>>(maxdt_min);
    ctx->launches++;
  }
  if (ctx->nleaf > 0) {
    const bool al = aligned16({flux, ne, e, eabs});
    const auto kern = maxdt_blk ? (al ? k_streamer_flux<true, 16> : k_streamer_flux<true, 8>)
                                : (al ? k_streamer_flux<false, 16> : k_streamer_flux<false, 8>);
    CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kRing * kTileSetBytes));
    kern<<<std::min(ctx->nleaf, 148 * 4), kFluxThreads, kRing * kTileSetBytes, ctx->stream>>>(
        flux, maxdt_blk, maxdt_min, ne, e, eabs, ctx->d_leaf, ctx->nleaf, ctx->d_info, cell_size(h, *tr), *tr);
    ctx->launches++;
  }
  if (ctx->refbnd_levels) {
    k_restrict_flux<<<(unsigned)(((int64_t)ctx->nused * 32 + 255) / 256), 256, 0, ctx->stream>>>(
        flux, ctx->d_faceb, ctx->d_used, ctx->nused);
    ctx->launches++;
  }
  CK(cudaGetLastError());
  return SRMG_OK;
}

extern "C" int srmg_streamer_rates_dev(srmg_ctx *ctx, double *dne, double *dni, const double *ne,
                                       const double *eabs, const double *flux, int64_t nblk_alloc, double h,
                                       int geom, const srmg_transport *tr) {
  RC(check_call(ctx, nblk_alloc, 0, 0, nullptr));
  if (!dne || !dni || !ne || !eabs || !flux) return fail(ctx, SRMG_ERR_BADARG, "srmg_streamer_rates_dev: null field");
  if (!(h > 0.0) || !std::isfinite(h)) return fail(ctx, SRMG_ERR_BADARG, "srmg_streamer_rates_dev: h must be > 0");
  if (geom < 0 || geom > 2) return fail(ctx, SRMG_ERR_BADARG, "srmg_streamer_rates_dev: geom must be 0, 1 or 2");
  RC(check_transport(ctx, tr, "srmg_streamer_rates_dev"));
  if (ctx->nleaf > 0) {
    const auto kern = aligned16({ne, eabs, flux}) ? k_streamer_rates<16> : k_streamer_rates<8>;
    CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kRing * kTileSetBytes));
    kern<<<std::min(ctx->nleaf, 148 * 4), 256, kRing * kTileSetBytes, ctx->stream>>>(
        dne, dni, ne, eabs, flux, ctx->d_leaf, ctx->nleaf, ctx->d_info, cell_size(h, *tr), geom, *tr);
    ctx->launches++;
  }
  CK(cudaGetLastError());
  return SRMG_OK;
}

extern "C" int srmg_ssprk3_stage_dev(srmg_ctx *ctx, double *out, const double *n, const double *dn1,
                                     const double *dn2, const double *dn3, int64_t count, double dt, int stage) {
  if (!ctx) return SRMG_ERR_BADARG;
  if (stage < 1 || stage > 3) return fail(ctx, SRMG_ERR_BADARG, "srmg_ssprk3_stage_dev: stage must be 1, 2 or 3");
  if (!out || !n || !dn1 || (stage >= 2 && !dn2) || (stage == 3 && !dn3) || count < 0)
    return fail(ctx, SRMG_ERR_BADARG, "srmg_ssprk3_stage_dev: bad arguments");
  if (!std::isfinite(dt)) return fail(ctx, SRMG_ERR_BADARG, "srmg_ssprk3_stage_dev: dt must be finite");
  CK(cudaSetDevice(ctx->device));
  if (count > 0) {
    k_ssprk3<<<grid_of(count, 256, 148 * 16), 256, 0, ctx->stream>>>(out, n, dn1, dn2, dn3, count, dt, stage);
    ctx->launches++;
  }
  CK(cudaGetLastError());
  return SRMG_OK;
}
