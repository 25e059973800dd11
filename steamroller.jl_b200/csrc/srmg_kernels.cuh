// srmg_kernels.cuh -- per-operation CUDA kernels for the FAS multigrid on a block tree.
//
// Block geometry is fixed at compile time: M = 16 valid cells per side, G = 2 ghost
// layers, S = 20, one block = S*S elements, dim 1 (r, "x") fastest.  All local indices
// here are 0-based: valid cells are x, y in [2, 17]; element (x, y) of block blk is at
// blk*400 + x + 20*y.  Block ids are 0-based on the device.
//
// Each kernel restates one reference routine and keeps its floating-point operation
// order where the result must be bit-exact (ghost copies, mirrors, linear
// interpolation, restriction, and the stencils of the smoother and the residual);
// __dadd_rn/__dmul_rn stop the compiler from contracting those into FMAs, and fma()
// stands where the reference calls muladd.  The same bodies run as separate kernels
// and inside the sequencer's single launch, with identical results.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include <initializer_list>

namespace srmg {

constexpr int kM = 16;
constexpr int kG = 2;
constexpr int kS = kM + 2 * kG;
constexpr int kSS = kS * kS;
// Per-item operator table of the persistent engine: s_l [32], stencil centre_l [32] and
// -(omega / diagonal)_l [32], indexed by level l.
constexpr int kParStride = 96;
// Blocks per norm chunk: the leaf norms are summed per chunk of up to this many
// consecutive blocks of one item and level, then per item over its chunks.
constexpr int kNormChunk = 4;
// Per-item result record of a device solve loop: {norm, |b|, initial norm, V-cycles run,
// defect-correction steps run (mixed mode; 0 in FP64 mode)}.
constexpr int kItemRec = 5;

// Top of a kernel launched by launch_pdl: lets the next kernel's blocks be scheduled, then
// waits for the previous kernel on the stream to complete.  fields: the kernel's pointers to
// memory that other kernels write.  The compiler may move an access through a __restrict__
// parameter above the wait (nothing else in the kernel, the wait included, can touch what it
// points to), and may read through one that is const by non-coherent loads, which are for
// memory that nothing writes while the kernel runs -- it runs here from before the wait.  So the
// pointers pass through an empty asm after it: what follows depends on that, and is coherent.
template <typename... P>
__device__ __forceinline__ void pdl_enter(P &...fields) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  (void)std::initializer_list<int>{([](auto &p) { asm volatile("" : "+l"(p)::"memory"); }(fields), 0)...};
}

// Face numbering (the four StarStencil directions): 0 = -r, 1 = +r, 2 = -z, 3 = +z.
enum FaceType : int { FACE_NONE = 0, FACE_NEIGHBOR = 1, FACE_BOUNDARY = 2, FACE_REFBND = 3 };

// Per-level device view of the tree.
struct LevelView {
  const int4 *blocks;   // [nblk] {blk, coord_r, coord_z, child_mask}; coords 1-based
  const int4 *faces;    // [nblk*4] {type, src_blk, sb_r, sb_z}
  const int4 *child;    // [nch] {fine_blk, coarse_blk, sb_r, sb_z} (fine at this level)
  int nblk;
  int nch;
  int level;
  // BoxStencil trees only (else null): [nblk*4] corner faces, corner q at direction
  // (2 (q & 1) - 1, 2 (q >> 1) - 1); {type, src_blk, a, b} with (a, b) the subblock of a
  // refinement corner or the boundary's bnd vector (components -1, 0, +1) of a
  // boundary corner.
  const int4 *cfaces;
};

// The reciprocal div_by takes for a divisor: 1 / d, or 0 (plain divisions) where d is so small
// or large that an intermediate result could leave the normal range.
__host__ __device__ inline double recip_of(double d) {
  const double m = d < 0 ? -d : d;
  return m > 1e-90 && m < 1e90 ? 1.0 / d : 0.0;
}

// a / d for a fixed d and its correctly rounded reciprocal rd: two corrections of the
// product a rd by the exact remainder.  The first makes q faithful (off by less than one
// unit in the last place), so that by Markstein's theorem (IBM J. Res. Dev. 34, 1990) the
// second gives the correctly rounded quotient, as long as nothing leaves the normal range;
// there, and for infinities and NaN, the division itself is called.
__device__ __forceinline__ double div_by(double a, double d, double rd) {
  // the exponent field: 2^-700 <= |a| < 2^670 (an integer test; the fp64 pipe is the bound),
  // and a reciprocal from recip_of.  A cell size passes recip_of on level 1 and is below 1e-90
  // by up to 2^-29 on the finest level: |a / d| < 2^(670 + 299 + 29) stays normal.
  if ((unsigned)((__double2hiint(a) & 0x7ff00000) - (323 << 20)) >= (1370u << 20) || __double2hiint(rd) == 0)
    return a == 0.0 && rd != 0.0 ? __dmul_rn(a, rd) : __ddiv_rn(a, d);
  double q = __dmul_rn(a, rd);
  q = fma(fma(-q, d, a), rd, q);
  return fma(fma(-q, d, a), rd, q);
}

// Operator parameters for one level.
template <typename T>
struct OpParams {
  int op;        // 0 Laplacian, 1 Helmholtz, 2 compact order-4 Laplacian
  int geom;      // 0 Cartesian, 1 cylindrical r = dim 1, 2 cylindrical r = dim 2
  T s;           // level scale s_l
  T centre;      // -4 or -4 - s_l*k2 (stencil centre, src/helmholtz.jl:43-45)
  T nwc;         // -(omega / diagelm)  (src/multigrid.jl:177)
  T omega;       // the relaxation factor itself (order 4 divides by a per-cell diagonal)
  T rs;          // 1 / s, correctly rounded
  const double *c4;  // order 4, cylindrical: kCoef4 coefficients per radial index, or null (formed per cell)
};
// Order-4 coefficients of one radial index: am, ap, em, cc, ep (coeffs9), the diagonal and its
// reciprocal (recip_of), as one 64-byte row.
constexpr int kCoef4 = 8;

// a / d with rd = 1 / d correctly rounded: div_by in double, the plain quotient in float.
__device__ __forceinline__ double quot(double a, double d, double rd) { return div_by(a, d, rd); }
__device__ __forceinline__ float quot(float a, float d, float) { return a / d; }

struct Signs { double v[9]; };  // boundary-condition table as doubles, column-major

// Radial weights (2i-2)/(2i-1), 2i/(2i-1) tabulated by 1-based global index
// (src/laplacian.jl:104-106).
template <typename T>
struct WTab { const T *wm; const T *wp; };

__device__ __forceinline__ int face_sign_index(int f) {
  // bnd == face for a star stencil; index (1 + bnd1) + 3 (1 + bnd2)
  return f == 0 ? 3 : f == 1 ? 5 : f == 2 ? 1 : 7;
}

template <typename T> __device__ __forceinline__ T dadd(T a, T b);
template <> __device__ __forceinline__ double dadd<double>(double a, double b) { return __dadd_rn(a, b); }
template <> __device__ __forceinline__ float dadd<float>(float a, float b) { return __fadd_rn(a, b); }
template <typename T> __device__ __forceinline__ T dmul(T a, T b);
template <> __device__ __forceinline__ double dmul<double>(double a, double b) { return __dmul_rn(a, b); }
template <> __device__ __forceinline__ float dmul<float>(float a, float b) { return __fmul_rn(a, b); }

// Whole-tile copies global -> shared by the CTA's threads (cp.async, CH = 16 or 8 bytes a
// copy: 16 needs 16-byte aligned fields), for kernels that stream blocks through a ring of
// tiles: a later block's tiles are in flight while one is worked on, without registers
// to hold them.  Every thread commits one group per ring step, empty or not, and waits
// with cp_async_wait<groups that may still be in flight>.
template <int CH>
__device__ __forceinline__ void cp_tile(double *dst, const double *src, int n) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  for (int i = threadIdx.x; i < n * 8 / CH; i += blockDim.x) {
    const char *s = reinterpret_cast<const char *>(src) + i * CH;
    if (CH == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + i * CH), "l"(s) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d + i * CH), "l"(s) : "memory");
  }
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Stencil weights of cell (x, y) of a block at 1-based coords (cr, cz).
template <typename T>
struct W5 { T zm, rm, rp, zp; };

template <typename T>
__device__ __forceinline__ W5<T> weights(const WTab<T> &wt, int geom, int cr, int cz, int x, int y) {
  W5<T> w{T(1), T(1), T(1), T(1)};
  if (geom == 1) {
    const int i = x - 1 + kM * (cr - 1);
    w.rm = wt.wm[i];
    w.rp = wt.wp[i];
  } else if (geom == 2) {
    const int j = y - 1 + kM * (cz - 1);
    w.zm = wt.wm[j];
    w.zp = wt.wp[j];
  }
  return w;
}

// applystencil, order 2 (src/laplacian.jl:25-49,78-118; src/helmholtz.jl:17-57):
// v = 0; v += c * u[I+S] over S = (0,-1), (-1,0), (0,0), (1,0), (0,1), each product and
// sum rounded on its own: the uncontracted reading of the reference's @fastmath
// stencil, and a rounding that does not depend on the context the body is inlined
// into (the compiler's choice of FMAs would).
template <typename T>
__device__ __forceinline__ T apply5(const T *ub, int x, int y, const W5<T> &w, T centre) {
  const int o = x + kS * y;
  T v = dadd<T>(T(0), dmul<T>(w.zm, ub[o - kS]));
  v = dadd<T>(v, dmul<T>(w.rm, ub[o - 1]));
  v = dadd<T>(v, dmul<T>(centre, ub[o]));
  v = dadd<T>(v, dmul<T>(w.rp, ub[o + 1]));
  v = dadd<T>(v, dmul<T>(w.zp, ub[o + kS]));
  return v;
}

// ---- compact order-4 Laplacian, LaplacianDiscretization{2,4} -------------------------
// applystencil (src/laplacian.jl:133-202): a 3x3 literal, rows along dimension 1 and
// columns along dimension 2, accumulated column-major (k = (d1 + 1) + 3 (d2 + 1),
// v = 0; v += c_k u) and divided by 6.  The cylindrical coefficients are integer
// polynomials of the radial 1-based global index i divided as doubles; every operation
// is rounded on its own (no contraction), so results are bit-exact against the oracle.
__device__ __forceinline__ void coeffs9(int geom, int64_t ir, int64_t iz, double c[9]) {
  if (geom == 0) {
    c[0] = 1; c[1] = 4; c[2] = 1; c[3] = 4; c[4] = -20; c[5] = 4; c[6] = 1; c[7] = 4; c[8] = 1;
    return;
  }
  const int64_t i = geom == 1 ? ir : iz;
  const int64_t q = 2 * i - 1;
  const double am = __ddiv_rn((double)(2 * (i - 1)), (double)q);
  const double ap = __ddiv_rn((double)(2 * i), (double)q);
  const double q3 = (double)(q * q * q);
  const double em = __ddiv_rn((double)(4 * (-2 + 9 * i - 16 * i * i + 8 * i * i * i)), q3);
  const double cc = __ddiv_rn((double)(-16 * (1 - 5 * i + 5 * i * i)), (double)((1 - 2 * i) * (1 - 2 * i)));
  const double ep = __ddiv_rn((double)(4 * (1 + i - 8 * i * i + 8 * i * i * i)), q3);
  if (geom == 1) {  // r = dimension 1 (src/laplacian.jl:156-164)
    c[0] = am; c[1] = 4; c[2] = ap; c[3] = em; c[4] = cc; c[5] = ep; c[6] = am; c[7] = 4; c[8] = ap;
  } else {          // r = dimension 2 (src/laplacian.jl:176-184)
    c[0] = am; c[1] = em; c[2] = am; c[3] = 4; c[4] = cc; c[5] = 4; c[6] = ap; c[7] = ep; c[8] = ap;
  }
}

// A row of the coefficient table, and the 9 coefficients it stands for.
struct Row4 {
  double am, ap, em, cc, ep, diag, rdiag;
  __device__ __forceinline__ Row4() {}
  __device__ __forceinline__ explicit Row4(const double *t) {
    const double2 *v = reinterpret_cast<const double2 *>(t);
    const double2 a = v[0], b = v[1], c = v[2], d = v[3];
    am = a.x, ap = a.y, em = b.x, cc = b.y, ep = c.x, diag = c.y, rdiag = d.x;
  }
};
__device__ __forceinline__ void spread9(const Row4 &r, int geom, double c[9]) {
  if (geom == 1) {
    c[0] = r.am; c[1] = 4; c[2] = r.ap; c[3] = r.em; c[4] = r.cc; c[5] = r.ep; c[6] = r.am; c[7] = 4; c[8] = r.ap;
  } else {
    c[0] = r.am; c[1] = r.em; c[2] = r.am; c[3] = 4; c[4] = r.cc; c[5] = 4; c[6] = r.ap; c[7] = r.ep; c[8] = r.ap;
  }
}

// The same from the table of this radial index (k_coef4, the same operations): forming the
// coefficients takes five divisions, more than the rest of a cell's update.
__device__ __forceinline__ void coeffs9(const double *c4, int geom, int64_t ir, int64_t iz, double c[9]) {
  if (!c4 || geom == 0) {
    coeffs9(geom, ir, iz, c);
    return;
  }
  spread9(Row4(c4 + kCoef4 * (geom == 1 ? ir : iz)), geom, c);
}

template <typename T>
__device__ __forceinline__ T apply9(const T *ub, int x, int y, int geom, int64_t ir, int64_t iz, const double *c4) {
  double c[9];
  coeffs9(c4, geom, ir, iz, c);
  T v = T(0);
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int d1 = k % 3 - 1, d2 = k / 3 - 1;
    v = dadd<T>(v, dmul<T>(T(c[k]), ub[(x + d1) + kS * (y + d2)]));
  }
  return quot(v, T(6), T(1) / T(6));  // exact: a sixth of a double is never halfway between two
}

// diagelm, order 4 (src/laplacian.jl:150-151, 205-209).
__device__ __forceinline__ double diagelm4(int geom, int64_t ir, int64_t iz) {
  if (geom == 0) return -20.0 / 6.0;
  const int64_t i = geom == 1 ? ir : iz;
  return __ddiv_rn(__ddiv_rn((double)(-16 * (1 - 5 * i + 5 * i * i)), (double)((1 - 2 * i) * (1 - 2 * i))), 6.0);
}

// The table of a tree: entry i for every radial 1-based global index i < n.
static __global__ void k_coef4(double *__restrict__ tab, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 1 || i >= n) return;
  double c[9];
  coeffs9(1, i, 0, c);
  double *t = tab + kCoef4 * i;
  t[0] = c[0];
  t[1] = c[2];
  t[2] = c[3];
  t[3] = c[4];
  t[4] = c[5];
  t[5] = diagelm4(1, i, 0);
  t[6] = recip_of(t[5]);
  t[7] = 0.0;
}

// 1-based global indices of local cell (x, y) of a block at 1-based coords (cr, cz)
// (global_first, src/mesh.jl:76-78).
__device__ __forceinline__ int64_t gidx(int c, int x) { return (int64_t)kM * (c - 1) + x - 1; }

// The left-hand side of any supported discretisation at cell (x, y).
template <typename T>
__device__ __forceinline__ T lhs_apply(const T *ub, int x, int y, const OpParams<T> &p, const WTab<T> &wt,
                                       int cr, int cz) {
  if (p.op == 2) return apply9<T>(ub, x, y, p.geom, gidx(cr, x), gidx(cz, y), p.c4);
  const W5<T> w = weights<T>(wt, p.geom, cr, cz, x, y);
  return apply5<T>(ub, x, y, w, p.centre);
}

// ---- ghost fill (src/connectivity.jl:155-258) --------------------------------------
// Tile X of a field: a block's values in a field in memory (srmg_coarse.cu has fields whose
// tiles lie in the shared memories of a cluster).
template <typename T>
__device__ __forceinline__ T *tile_of(T *u, int64_t X) { return u + X * kSS; }

template <typename T, class F>
__device__ __forceinline__ void fill_corner_cell(F u, const LevelView &lv, const Signs &sg, int phase, int64_t t);

// One warp per block, a lane one cell of each face: lane -> (layer g = lane/16, position
// k = lane%16).  The fill is a chain of dependent scattered loads (record, value, store), so
// it is bound by how many of them are in flight: the four faces' records are loaded
// together, then the four copied or mirrored values, before any is stored; refinement
// faces (three values each, few of them) follow on their own.  With a warp per (block, face)
// 36276 blocks took 72 us.  On a BoxStencil tree (lv.cfaces set) lanes 0..15 also fill the
// block's 16 corner cells (fill_corner_cell), in the order of fill_ghost!'s passes: the
// copy and boundary passes, a warp barrier, then interpolation -- a boundary corner mirrors
// its own block's refinement ghosts as they were before the fill, and no pass reads
// another block's ghosts of this level, so one launch does all three.
template <typename T, class F>
__device__ __forceinline__ void d_fill_ghost(F u, LevelView lv, Signs sg, int mask, int cta = blockIdx.x,
                                             int ctas = gridDim.x) {
  const int lane = threadIdx.x & 31;
  const int g = lane >> 4, k = lane & 15;
  const int stride = ctas * (blockDim.x >> 5);
  for (int bi = cta * (blockDim.x >> 5) + (threadIdx.x >> 5); bi < lv.nblk; bi += stride) {
    int type[4], src[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const int2 r = *reinterpret_cast<const int2 *>(lv.faces + 4 * bi + f);
      type[f] = r.x;
      src[f] = r.y;
    }
    T *ub = tile_of(u, lv.blocks[bi].x);
    T v[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const int x = f == 0 ? g : f == 1 ? 18 + g : 2 + k, y = f == 2 ? g : f == 3 ? 18 + g : 2 + k;  // the ghost
      if (type[f] == FACE_NEIGHBOR) {
        // _fill_ghost_copy! (src/connectivity.jl:184-198): ghost <- neighbour's valid
        // cell M positions away along the face normal.
        const int sx = f == 0 ? x + kM : f == 1 ? x - kM : x, sy = f == 2 ? y + kM : f == 3 ? y - kM : y;
        if (mask & 1) v[f] = tile_of(u, src[f])[sx + kS * sy];
      } else if (type[f] == FACE_BOUNDARY) {
        // fill_ghost_bnd! (src/connectivity.jl:217-231), mirrorghost (src/blockfield.jl:513-521)
        const int mx = f == 0 ? 2 * kG - 1 - x : f == 1 ? 2 * (kG + kM) - 1 - x : x;
        const int my = f == 2 ? 2 * kG - 1 - y : f == 3 ? 2 * (kG + kM) - 1 - y : y;
        if (mask & 2) v[f] = ub[mx + kS * my];
      }
    }
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const int x = f == 0 ? g : f == 1 ? 18 + g : 2 + k, y = f == 2 ? g : f == 3 ? 18 + g : 2 + k;
      if (type[f] == FACE_NEIGHBOR && (mask & 1)) ub[x + kS * y] = v[f];
      else if (type[f] == FACE_BOUNDARY && (mask & 2)) ub[x + kS * y] = dmul<T>(T(sg.v[face_sign_index(f)]), v[f]);
    }
    if (lv.cfaces) {
      if ((mask & 3) && lane < 16) fill_corner_cell<T>(u, lv, sg, mask & 3, (int64_t)bi * 16 + lane);
      __syncwarp();
    }
    if (mask & 4) {
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        if (type[f] != FACE_REFBND) continue;
        // fill_ghost_interp! (src/connectivity.jl:251-258) + interp! (src/interp.jl:24-63)
        // from the coarse block's subblockbnd(subblock, -face) (src/blockfield.jl:416-434):
        // the coarse source cell and the 0/1 child offsets per dimension.
        const int x = f == 0 ? g : f == 1 ? 18 + g : 2 + k, y = f == 2 ? g : f == 3 ? 18 + g : 2 + k;
        const int4 fi = lv.faces[4 * bi + f];
        const T *cb = tile_of(u, fi.y);
        const int sbr = fi.z, sbz = fi.w;
        const int jr = f == 0 ? 1 + 8 * sbr : f == 1 ? 2 + 8 * (sbr - 1) : 2 + 8 * (sbr - 1) + (k >> 1);
        const int jz = f == 2 ? 1 + 8 * sbz : f == 3 ? 2 + 8 * (sbz - 1) : 2 + 8 * (sbz - 1) + (k >> 1);
        const int ir = f <= 1 ? g : k & 1, iz = f <= 1 ? k & 1 : g, o = jr + kS * jz;
        T w = cb[o];
        if (!(mask & 8)) {  // else InterpCopy (src/interp.jl:66-85): the coarse cell's value itself
          const T wr = cb[o + (2 * ir - 1)], wz = cb[o + kS * (2 * iz - 1)];
          w = dmul<T>(T(0.5), w);
          w = dadd<T>(w, dmul<T>(T(0.25), wr));
          w = dadd<T>(w, dmul<T>(T(0.25), wz));
        }
        ub[x + kS * y] = w;
      }
    }
    if (lv.cfaces && (mask & 4) && lane < 16) fill_corner_cell<T>(u, lv, sg, 4, (int64_t)bi * 16 + lane);
  }
}

// ---- red-black Gauss-Seidel colour sweep (src/multigrid.jl:153-180, 238-243) ------
// Colour P updates valid cells with (x + y + 1) & 1 == P (0-based local indices).
// Ghost pushes of a colour sweep (2D trees, per-operation path): for every valid cell
// whose value a copy-and-boundary fill (fill_ghost! passes 1 and 2) writes into ghost
// cells, the list of those ghosts, CSR by (level-local block, cell): off[bi*256 + cell]
// .. off[bi*256 + cell + 1] index ent, ent = {ghost's index in the field, boundary-table
// entries of the mirrors on the way (low and high 4 bits, 15 = none)}.  The sweep that
// updates the cell writes them, so no fill launch has to follow it.  Built from the
// fill itself (srmg.cu, ensure_gs_push).  The boundary table reaches the sweep packed,
// two bits an entry (entry + 1: the pushes are used only where every entry is -1, 0 or 1).
struct PushView {
  const int *off;
  const int2 *ent;
  const int *cbi;  // [child edge] index of its fine block in the level's block list (2D trees)
};

template <typename T>
__device__ __forceinline__ void push_ghosts(T *__restrict__ u, const PushView &pv, unsigned sg, int bi, int x, int y,
                                            T v) {
  const int c = bi * 256 + (x - kG) + kM * (y - kG);
  const int e1 = pv.off[c + 1];
  for (int e = pv.off[c]; e < e1; ++e) {
    const int2 d = pv.ent[e];
    T w = v;
    // boundary-table entries are -1, 0 or 1: the products are exact in any order
    const int k1 = d.y & 15, k2 = d.y >> 4;
    if (k1 < 9) w = dmul<T>(T((int)((sg >> (2 * k1)) & 3u) - 1), w);
    if (k2 < 9) w = dmul<T>(T((int)((sg >> (2 * k2)) & 3u) - 1), w);
    u[d.x] = w;
  }
}

template <typename T>
__device__ __forceinline__ void d_gs_colour(T *__restrict__ u, const T *__restrict__ b, LevelView lv,
                                            OpParams<T> p, WTab<T> wt, int parity) {
  const int64_t total = (int64_t)lv.nblk * 128;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int bi = (int)(t >> 7), c = (int)(t & 127);
    const int y = 2 + (c >> 3);
    const int x = 2 + 2 * (c & 7) + ((parity ^ (y + 1)) & 1);
    const int4 bk = lv.blocks[bi];
    T *ub = u + (int64_t)bk.x * kSS;
    const W5<T> w = weights<T>(wt, p.geom, bk.y, bk.z, x, y);
    const T Lu = apply5<T>(ub, x, y, w, p.centre);
    const int o = x + kS * y;
    const T v = fma(p.s, b[(int64_t)bk.x * kSS + o], Lu);
    const T nv = fma(p.nwc, v, ub[o]);
    ub[o] = nv;
  }
}

// ---- residual (src/multigrid.jl:309-323, 349-354): r = -(b + Lu/s) ---------------
template <typename T>
__device__ __forceinline__ void d_residual(T *__restrict__ r, const T *__restrict__ u, const T *__restrict__ b,
                           LevelView lv, OpParams<T> p, WTab<T> wt) {
  const int64_t total = (int64_t)lv.nblk * 256;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int bi = (int)(t >> 8), c = (int)(t & 255);
    const int x = 2 + (c & 15), y = 2 + (c >> 4);
    const int4 bk = lv.blocks[bi];
    const int64_t base = (int64_t)bk.x * kSS;
    const int64_t o = base + x + kS * y;
    const T bo = b[o];  // in flight before the quotient's branch: 99 us otherwise on 36k blocks, 79 so
    const T Lu = lhs_apply<T>(u + base, x, y, p, wt, bk.y, bk.z);
    r[o] = -(bo + quot(Lu, p.s, p.rs));
  }
}

// ---- FAS coarse RHS (src/multigrid.jl:112-119, 331-344) ----------------------------
// For each Child edge of this level, on the coarse subblock: bf = -(r + L(u)/s_c).
template <typename T>
__device__ __forceinline__ void d_postrestrict(T *__restrict__ bf, const T *__restrict__ u, const T *__restrict__ r,
                               LevelView lv, const int2 *__restrict__ coord_of, OpParams<T> p,
                               WTab<T> wt) {
  const int64_t total = (int64_t)lv.nch * 64;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int e = (int)(t >> 6), c = (int)(t & 63);
    const int4 ch = lv.child[e];
    const int cblk = ch.y;
    const int x = 2 + 8 * (ch.z - 1) + (c & 7), y = 2 + 8 * (ch.w - 1) + (c >> 3);
    const int2 cc = coord_of[cblk];
    const int64_t base = (int64_t)cblk * kSS;
    const int64_t o = base + x + kS * y;
    const T ro = r[o];  // as in d_residual
    const T Lu = lhs_apply<T>(u + base, x, y, p, wt, cc.x, cc.y);
    bf[o] = -(ro + quot(Lu, p.s, p.rs));
  }
}

// ---- restriction (src/restrict.jl:5-37) --------------------------------------------
// coarse = ((((0 + f00) + f10) + f01) + f11) / 4 for each Child edge of this level.
template <typename T>
struct alignas(2 * sizeof(T)) Pair { T x, y; };

template <typename T>
__device__ __forceinline__ void d_restrict(T *__restrict__ u, LevelView lv) {
  const int64_t total = (int64_t)lv.nch * 64;
  const bool aligned = (reinterpret_cast<uintptr_t>(u) & (2 * sizeof(T) - 1)) == 0;  // uniform
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int e = (int)(t >> 6), c = (int)(t & 63);
    const int4 ch = lv.child[e];
    const int kx = c & 7, ky = c >> 3;
    const T *fb = u + (int64_t)ch.x * kSS + (2 + 2 * kx) + kS * (2 + 2 * ky);
    Pair<T> lo, hi;  // one load a row where the field allows it: half the load instructions
    if (aligned) {
      lo = *reinterpret_cast<const Pair<T> *>(fb);
      hi = *reinterpret_cast<const Pair<T> *>(fb + kS);
    } else {
      lo = Pair<T>{fb[0], fb[1]};
      hi = Pair<T>{fb[kS], fb[kS + 1]};
    }
    T f = dadd<T>(T(0), lo.x);
    f = dadd<T>(f, lo.y);
    f = dadd<T>(f, hi.x);
    f = dadd<T>(f, hi.y);
    u[(int64_t)ch.y * kSS + (2 + 8 * (ch.z - 1) + kx) + kS * (2 + 8 * (ch.w - 1) + ky)] =
        dmul<T>(f, T(0.25));
  }
}

// ---- prolongation-add (src/interp.jl:24-63, 107-115): u_f += P(u1_c) -------------
template <typename T>
__device__ __forceinline__ void d_interp_add(T *__restrict__ u, const T *__restrict__ u1, LevelView lv) {
  const int64_t total = (int64_t)lv.nch * 256;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int e = (int)(t >> 8), c = (int)(t & 255);
    const int4 ch = lv.child[e];
    const int dx = c & 15, dy = c >> 4;
    const int ir = dx & 1, iz = dy & 1;
    const int jr = 2 + 8 * (ch.z - 1) + (dx >> 1), jz = 2 + 8 * (ch.w - 1) + (dy >> 1);
    const T *cb = u1 + (int64_t)ch.y * kSS;
    const int o = jr + kS * jz;
    T v = dmul<T>(T(0.5), cb[o]);
    v = dadd<T>(v, dmul<T>(T(0.25), cb[o + (2 * ir - 1)]));
    v = dadd<T>(v, dmul<T>(T(0.25), cb[o + kS * (2 * iz - 1)]));
    T *d = u + (int64_t)ch.x * kSS + (2 + dx) + kS * (2 + dy);
    *d = dadd<T>(v, *d);
  }
}

// ---- whole-block copy / difference over a level (src/blockfield.jl:557-576) ------
template <typename T>
__device__ __forceinline__ void d_copy_level(T *__restrict__ dst, const T *__restrict__ src, LevelView lv) {
  const int64_t total = (int64_t)lv.nblk * kSS;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int bi = (int)(t / kSS), c = (int)(t % kSS);
    const int64_t o = (int64_t)lv.blocks[bi].x * kSS + c;
    dst[o] = src[o];
  }
}

template <typename T>
__device__ __forceinline__ void d_diff_level(T *__restrict__ dst, const T *__restrict__ a1, const T *a2,
                             LevelView lv) {
  const int64_t total = (int64_t)lv.nblk * kSS;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int bi = (int)(t / kSS), c = (int)(t % kSS);
    const int64_t o = (int64_t)lv.blocks[bi].x * kSS + c;
    dst[o] = a1[o] - a2[o];
  }
}

// ---- residual norm pieces -----------------------------------------------------------
// Sum over the level's LEAF cells (cells of subblocks without a child) of
// w_l * f(x)^2, with f = residual (mode 0) or the field itself (mode 1).  One partial
// per CTA, written to part[blockIdx.x]: deterministic for a fixed grid.
// This is the value resnorm! (src/multigrid.jl:391-417) obtains by squaring every
// cell and restricting the squares down to level 1: a leaf cell of level l ends up
// weighted by 4^-(l-1).
template <typename T, int NT>
__global__ void __launch_bounds__(NT) k_leafsq(double *__restrict__ part, const T *__restrict__ u,
                                               const T *__restrict__ b, LevelView lv,
                                               OpParams<T> p, WTab<T> wt, double wl, int mode) {
  pdl_enter(part, u, b);
  double acc = 0.0;
  const int64_t total = (int64_t)lv.nblk * 256;
  for (int64_t t = blockIdx.x * (int64_t)NT + threadIdx.x; t < total; t += (int64_t)gridDim.x * NT) {
    const int bi = (int)(t >> 8), c = (int)(t & 255);
    const int x = 2 + (c & 15), y = 2 + (c >> 4);
    const int4 bk = lv.blocks[bi];
    const int sub = ((x - 2) >> 3) + 2 * ((y - 2) >> 3);
    if ((bk.w >> sub) & 1) continue;  // covered by a child: not a leaf cell
    const int64_t base = (int64_t)bk.x * kSS;
    const int64_t o = base + x + kS * y;
    double v;
    if (mode == 0) {
      const T Lu = lhs_apply<T>(u + base, x, y, p, wt, bk.y, bk.z);
      v = (double)(-(b[o] + Lu / p.s));
    } else {
      v = (double)b[o];
    }
    acc = fma(v, v, acc);
  }
  __shared__ double sh[NT / 32];
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = (threadIdx.x < NT / 32) ? sh[threadIdx.x] : 0.0;
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (threadIdx.x == 0) part[blockIdx.x] = v * wl;
  }
}

// Final fixed-order reduction of n partials into out[0] (sqrt applied).
template <int NT>
__global__ void __launch_bounds__(NT) k_reduce_sqrt(double *out,
                                                    const double *part, int n) {
  pdl_enter(out, part);
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += NT) acc += part[i];
  __shared__ double sh[NT / 32];
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = (threadIdx.x < NT / 32) ? sh[threadIdx.x] : 0.0;
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (threadIdx.x == 0) out[0] = sqrt(v);
  }
}

// gauss_seidel!(..., FourColors{P1,P2}) (src/multigrid.jl:206-232): cells
// (2 + 2a + p1, 2 + 2b + p2), u -= omega (Lu + s b) / c, unfused.  row4: the cell's
// coefficient row in cylindrical geometry, from the table or (none built) formed here.
template <typename T>
__device__ __forceinline__ Row4 row4(const OpParams<T> &p, int64_t ir, int64_t iz) {
  if (p.c4) return Row4(p.c4 + kCoef4 * (p.geom == 1 ? ir : iz));
  Row4 r;
  double c[9];
  coeffs9(p.geom, ir, iz, c);
  r.am = c[0];
  r.ap = p.geom == 1 ? c[2] : c[6];
  r.em = p.geom == 1 ? c[3] : c[1];
  r.cc = c[4];
  r.ep = p.geom == 1 ? c[5] : c[7];
  r.diag = diagelm4(p.geom, ir, iz);
  r.rdiag = 0.0;
  return r;
}
// apply9 at the cell at uc in geometry GEOM, and the cell's update.
template <typename T, int GEOM>
__device__ __forceinline__ T sum9(const T *uc, const Row4 &r) {
  double c[9];
  if (GEOM == 0) coeffs9(0, 0, 0, c);
  else spread9(r, GEOM, c);
  T v = T(0);
#pragma unroll
  for (int k = 0; k < 9; ++k) v = dadd<T>(v, dmul<T>(T(c[k]), uc[(k % 3 - 1) + kS * (k / 3 - 1)]));
  return quot(v, T(6), T(1) / T(6));
}
template <typename T, int GEOM>
__device__ __forceinline__ T gs4_value(const T *uc, T bo, const OpParams<T> &p, const Row4 &r) {
  const T Lu = sum9<T, GEOM>(uc, r);
  const T w = dmul<T>(p.omega, dadd<T>(Lu, dmul<T>(p.s, bo)));
  const T upd = GEOM == 0 ? quot(w, T(-20.0 / 6.0), T(1.0 / (-20.0 / 6.0))) : quot(w, T(r.diag), T(r.rdiag));
  return uc[0] - upd;
}

template <typename T>
__device__ __forceinline__ void d_gs4(T *__restrict__ u, const T *__restrict__ b, LevelView lv, OpParams<T> p, int p1,
                                      int p2) {
  const int64_t total = (int64_t)lv.nblk * 64;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int bi = (int)(t >> 6), c = (int)(t & 63);
    const int x = 2 + 2 * (c & 7) + p1, y = 2 + 2 * (c >> 3) + p2;
    const int4 bk = lv.blocks[bi];
    T *ub = u + (int64_t)bk.x * kSS;
    const int o = x + kS * y;
    const Row4 r = p.geom ? row4(p, gidx(bk.y, x), gidx(bk.z, y)) : Row4();
    const T bo = b[(int64_t)bk.x * kSS + o];
    const T nv = p.geom == 1   ? gs4_value<T, 1>(ub + o, bo, p, r)
                 : p.geom == 2 ? gs4_value<T, 2>(ub + o, bo, p, r)
                               : gs4_value<T, 0>(ub + o, bo, p, r);
    ub[o] = nv;
  }
}

// rhs! over rhs_level! (src/multigrid.jl:363-388): q1 = R q on the valid cells.  Order
// 2: the identity (src/laplacian.jl:86-91,120-125).  Order 4: the literal
// (src/laplacian.jl:141-148,166-173,186-193) walked over its nonzero entries
// (0,-1), (-1,0), (0,0), (1,0), (0,1), then divided by 12.
template <typename T>
__global__ void k_rhs(T *__restrict__ q1, const T *__restrict__ q, LevelView lv, int op, int geom) {
  pdl_enter(q1, q);
  if (op != 2 && ((reinterpret_cast<uintptr_t>(q1) | reinterpret_cast<uintptr_t>(q)) & (2 * sizeof(T) - 1)) == 0) {
    // a copy: two cells a thread where the fields' alignment allows it
    const int64_t pairs = (int64_t)lv.nblk * 128;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < pairs; t += (int64_t)gridDim.x * blockDim.x) {
      const int64_t o = (int64_t)lv.blocks[t >> 7].x * kSS + 2 + 2 * (int)(t & 7) + kS * (2 + (int)((t >> 3) & 15));
      *reinterpret_cast<Pair<T> *>(q1 + o) = *reinterpret_cast<const Pair<T> *>(q + o);
    }
    return;
  }
  const int64_t total = (int64_t)lv.nblk * 256;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int bi = (int)(t >> 8), c = (int)(t & 255);
    const int x = 2 + (c & 15), y = 2 + (c >> 4);
    const int4 bk = lv.blocks[bi];
    const T *qb = q + (int64_t)bk.x * kSS;
    const int o = x + kS * y;
    if (op != 2) {
      q1[(int64_t)bk.x * kSS + o] = qb[o];
      continue;
    }
    T wzm = T(1), wrm = T(1), wrp = T(1), wzp = T(1);
    if (geom != 0) {
      const int64_t i = geom == 1 ? gidx(bk.y, x) : gidx(bk.z, y);
      const T wm = __ddiv_rn((double)(2 * i - 2), (double)(2 * i - 1));
      const T wp = __ddiv_rn((double)(2 * i), (double)(2 * i - 1));
      if (geom == 1) { wrm = wm; wrp = wp; } else { wzm = wm; wzp = wp; }
    }
    T v = T(0);
    v = dadd<T>(v, dmul<T>(wzm, qb[o - kS]));
    v = dadd<T>(v, dmul<T>(wrm, qb[o - 1]));
    v = dadd<T>(v, dmul<T>(T(8), qb[o]));
    v = dadd<T>(v, dmul<T>(wrp, qb[o + 1]));
    v = dadd<T>(v, dmul<T>(wzp, qb[o + kS]));
    q1[(int64_t)bk.x * kSS + o] = v / T(12);
  }
}

// Corner ghosts of a BoxStencil tree (src/connectivity.jl:155-258 with diagonal faces):
// 2 x 2 cells per corner, one thread (index t) per cell.  `mask` selects the passes:
// 1 = copy from the diagonal neighbour, 2 = boundary mirror, 4 = linear interpolation
// from the parent's subblockbnd cell (src/blockfield.jl:416-434, src/interp.jl:24-63).
// A boundary corner whose bnd is zero along one dimension mirrors the adjacent face's
// ghost cells, which fill_ghost! writes in an earlier pass.  fill_ghost! runs copy,
// boundary and interpolation in that order; here copy and boundary share one pass
// (mask 3): such a corner evaluates the face ghost it mirrors from that face's own
// source -- the neighbour's valid cell, or the mirrored valid cell -- with the same
// operations as the face pass, instead of reading it.  Interpolation (mask 4) follows: the
// boundary pass reads a refinement face's ghosts as they were before this fill.
template <typename T, class F>
__device__ __forceinline__ T face_ghost_value(F u, const T *ub, const LevelView &lv,
                                              const Signs &sg, int bi, int f, int x, int y) {
  const int4 ff = lv.faces[4 * bi + f];
  if (ff.x == FACE_NEIGHBOR) {  // as the copy pass of d_fill_ghost
    const T *src = tile_of(u, ff.y);
    int sx = x, sy = y;
    if (f == 0) sx = x + kM; else if (f == 1) sx = x - kM;
    else if (f == 2) sy = y + kM; else sy = y - kM;
    return src[sx + kS * sy];
  }
  if (ff.x == FACE_BOUNDARY) {  // as the boundary pass of d_fill_ghost
    int mx = x, my = y;
    if (f == 0) mx = 2 * kG - 1 - x; else if (f == 1) mx = 2 * (kG + kM) - 1 - x;
    else if (f == 2) my = 2 * kG - 1 - y; else my = 2 * (kG + kM) - 1 - y;
    return dmul<T>(T(sg.v[face_sign_index(f)]), ub[mx + kS * my]);
  }
  return ub[x + kS * y];  // a refinement face: not written by the copy and boundary passes
}

template <typename T, class F>
__device__ __forceinline__ void fill_corner_cell(F u, const LevelView &lv, const Signs &sg, int mask, int64_t t) {
  {
    const int bi = (int)(t >> 4), q = (int)((t >> 2) & 3), cell = (int)(t & 3);
    const int4 fi = lv.cfaces[4 * bi + q];
    const int type = fi.x;
    if (type == FACE_NONE) return;
    if ((type == FACE_NEIGHBOR && !(mask & 1)) || (type == FACE_BOUNDARY && !(mask & 2)) ||
        (type == FACE_REFBND && !(mask & 4)))
      return;
    const int fr = 2 * (q & 1) - 1, fz = 2 * (q >> 1) - 1;  // ghost direction
    const int ir = cell & 1, iz = cell >> 1;
    const int x = (fr < 0 ? 0 : kM + kG) + ir, y = (fz < 0 ? 0 : kM + kG) + iz;
    T *ub = tile_of(u, lv.blocks[bi].x);
    if (type == FACE_NEIGHBOR) {
      const T *src = tile_of(u, fi.y);
      ub[x + kS * y] = src[(x - kM * fr) + kS * (y - kM * fz)];
    } else if (type == FACE_BOUNDARY) {
      const int b0 = fi.z, b1 = fi.w;
      const int mx = b0 < 0 ? 2 * kG - 1 - x : b0 > 0 ? 2 * (kG + kM) - 1 - x : x;
      const int my = b1 < 0 ? 2 * kG - 1 - y : b1 > 0 ? 2 * (kG + kM) - 1 - y : y;
      const T a = T(sg.v[(1 + b0) + 3 * (1 + b1)]);
      T src;
      if ((mask & 1) && (b0 == 0) != (b1 == 0)) {
        // the mirror lands in the ghost cells of the face along the zero component,
        // which the copy part of this launch writes: evaluate that cell directly
        const int f = b0 == 0 ? (fr < 0 ? 0 : 1) : (fz < 0 ? 2 : 3);
        src = face_ghost_value<T>(u, ub, lv, sg, bi, f, mx, my);
      } else {
        src = ub[mx + kS * my];
      }
      ub[x + kS * y] = dmul<T>(a, src);
    } else {
      const T *cb = tile_of(u, fi.y);
      const int sbr = fi.z, sbz = fi.w;
      // subblockbnd(subblock, -face): the last cell of the subblock along a dimension
      // where the ghost lies below, the first where it lies above
      const int jr = fr < 0 ? 1 + 8 * sbr : 2 + 8 * (sbr - 1);
      const int jz = fz < 0 ? 1 + 8 * sbz : 2 + 8 * (sbz - 1);
      const int o = jr + kS * jz;
      T v = dmul<T>(T(0.5), cb[o]);
      v = dadd<T>(v, dmul<T>(T(0.25), cb[o + (2 * ir - 1)]));
      v = dadd<T>(v, dmul<T>(T(0.25), cb[o + kS * (2 * iz - 1)]));
      ub[x + kS * y] = v;
    }
  }
}


// ---- fused steps of the per-operation V-cycle (vcycle_fused) -------------------------
// The restriction half of a level's descent in one pass over its child edges: the fine
// block's residual is formed where it is restricted (residual_level! writes it and
// restrict_level! reads it back, two more launches), u and r restricted in the
// reference's order.  r's fine cells are not written.
template <typename T>
__device__ __forceinline__ void d_down(T *__restrict__ u, T *__restrict__ r, const T *__restrict__ b, const LevelView &lv,
                                       const int2 *__restrict__ coord_of, const OpParams<T> &p, const WTab<T> &wt) {
  const int64_t total = (int64_t)lv.nch * 64;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int e = (int)(t >> 6), c = (int)(t & 63);
    const int4 ch = lv.child[e];
    const int kx = c & 7, ky = c >> 3;
    const int2 fc = coord_of[ch.x];
    const T *ub = u + (int64_t)ch.x * kSS, *bb = b + (int64_t)ch.x * kSS;
    T f = T(0), g = T(0);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int x = 2 + 2 * kx + i, y = 2 + 2 * ky + j, o = x + kS * y;
        f = dadd<T>(f, ub[o]);
        const T Lu = lhs_apply<T>(ub, x, y, p, wt, fc.x, fc.y);
        g = dadd<T>(g, -(bb[o] + quot(Lu, p.s, p.rs)));
      }
    const int64_t co = (int64_t)ch.y * kSS + (2 + 8 * (ch.z - 1) + kx) + kS * (2 + 8 * (ch.w - 1) + ky);
    u[co] = dmul<T>(f, T(0.25));
    r[co] = dmul<T>(g, T(0.25));
  }
}

// Value of the field a - a1 that a ghost or valid cell (x, y) of block index bi holds after a
// fill_ghost! of it, refinement ghosts interpolated from the parent level of e (already
// filled): what copying or subtracting the whole blocks and filling them would leave, cell
// by cell.
template <typename T, class F, class E>
__device__ __forceinline__ T filled_diff(F a, F a1, E e, const LevelView &lv, const Signs &sg, int bi, int64_t blk,
                                         int x, int y) {
  auto diff = [&](int64_t X, int o) { return dadd<T>(tile_of(a, X)[o], -tile_of(a1, X)[o]); };
  const int fr = x < kG ? -1 : x >= kG + kM ? 1 : 0, fz = y < kG ? -1 : y >= kG + kM ? 1 : 0;
  const int o = x + kS * y;
  if (!fr && !fz) return diff(blk, o);
  const bool corner = fr && fz;
  if (corner && !lv.cfaces) return diff(blk, o);
  const int f = fr ? (fr < 0 ? 0 : 1) : (fz < 0 ? 2 : 3);
  const int4 fi = corner ? lv.cfaces[4 * bi + (fr + 1) / 2 + (fz + 1)] : lv.faces[4 * bi + f];
  if (fi.x == FACE_NEIGHBOR) return diff(fi.y, (x - kM * fr) + kS * (y - kM * fz));
  if (fi.x == FACE_BOUNDARY) {
    const int b0 = corner ? fi.z : fr, b1 = corner ? fi.w : fz;
    const int mx = b0 < 0 ? 2 * kG - 1 - x : b0 > 0 ? 2 * (kG + kM) - 1 - x : x;
    const int my = b1 < 0 ? 2 * kG - 1 - y : b1 > 0 ? 2 * (kG + kM) - 1 - y : y;
    T v;
    if (corner && (b0 == 0) != (b1 == 0)) {
      // the mirror lands in the ghosts of the face along the zero component, filled by the
      // copy and boundary passes (fill_corner_cell)
      const int g = b0 == 0 ? (fr < 0 ? 0 : 1) : (fz < 0 ? 2 : 3);
      const int4 ff = lv.faces[4 * bi + g];
      const int gr = g < 2 ? 2 * g - 1 : 0, gz = g < 2 ? 0 : 2 * g - 5;
      if (ff.x == FACE_NEIGHBOR) {
        v = diff(ff.y, (mx - kM * gr) + kS * (my - kM * gz));
      } else if (ff.x == FACE_BOUNDARY) {
        const int nx = gr < 0 ? 2 * kG - 1 - mx : gr > 0 ? 2 * (kG + kM) - 1 - mx : mx;
        const int ny = gz < 0 ? 2 * kG - 1 - my : gz > 0 ? 2 * (kG + kM) - 1 - my : my;
        v = dmul<T>(T(sg.v[face_sign_index(g)]), diff(blk, nx + kS * ny));
      } else {
        v = diff(blk, mx + kS * my);
      }
    } else {
      v = diff(blk, mx + kS * my);
    }
    return dmul<T>(T(sg.v[(1 + b0) + 3 * (1 + b1)]), v);
  }
  if (fi.x == FACE_REFBND) {
    const T *cb = tile_of(e, fi.y);
    const int jr = fr < 0 ? 1 + 8 * fi.z : fr > 0 ? 2 + 8 * (fi.z - 1) : 2 + 8 * (fi.z - 1) + ((x - kG) >> 1);
    const int jz = fz < 0 ? 1 + 8 * fi.w : fz > 0 ? 2 + 8 * (fi.w - 1) : 2 + 8 * (fi.w - 1) + ((y - kG) >> 1);
    const int ir = x & 1, iz = y & 1, q = jr + kS * jz;  // both ghost pairs start at an even index
    T v = dmul<T>(T(0.5), cb[q]);
    v = dadd<T>(v, dmul<T>(T(0.25), cb[q + (2 * ir - 1)]));
    return dadd<T>(v, dmul<T>(T(0.25), cb[q + kS * (2 * iz - 1)]));
  }
  return diff(blk, o);
}

// The coarse correction e = u - u1 of a level with its ghosts filled (e's parent level filled
// already), one launch instead of a difference and the fill passes.  e must be neither u nor u1.
template <typename T>
__device__ __forceinline__ void d_correction(T *__restrict__ e, const T *__restrict__ u, const T *__restrict__ u1,
                                             const LevelView &lv, const Signs &sg) {
  const int64_t total = (int64_t)lv.nblk * kSS;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int bi = (int)(t / kSS), c = (int)(t % kSS);
    const int64_t blk = lv.blocks[bi].x;
    e[blk * kSS + c] = filled_diff<T>(u, u1, e, lv, sg, bi, blk, c % kS, c / kS);
  }
}

// interp_add_level! that also leaves u's ghosts filled: each updated cell is written to the
// copy and mirror ghosts of it (PushView; nothing here reads a ghost of this level), and
// the level's refinement ghosts are interpolated from its parent level.  pv.cbi gives the
// index of a child edge's fine block in the level's block list.
template <typename T>
__device__ __forceinline__ void d_interp_push(T *__restrict__ u, const T *__restrict__ e, const LevelView &lv,
                                              const PushView &pv, unsigned sw, const Signs &sg, bool refined) {
  const int64_t total = (int64_t)lv.nch * 256;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int k = (int)(t >> 8), c = (int)(t & 255);
    const int4 ch = lv.child[k];
    const int dx = c & 15, dy = c >> 4;
    const int ir = dx & 1, iz = dy & 1;
    const int o = 2 + 8 * (ch.z - 1) + (dx >> 1) + kS * (2 + 8 * (ch.w - 1) + (dy >> 1));
    const T *cb = e + (int64_t)ch.y * kSS;
    T v = dmul<T>(T(0.5), cb[o]);
    v = dadd<T>(v, dmul<T>(T(0.25), cb[o + (2 * ir - 1)]));
    v = dadd<T>(v, dmul<T>(T(0.25), cb[o + kS * (2 * iz - 1)]));
    T *d = u + (int64_t)ch.x * kSS + (2 + dx) + kS * (2 + dy);
    v = dadd<T>(v, *d);
    *d = v;
    push_ghosts<T>(u, pv, sw, pv.cbi[k], 2 + dx, 2 + dy, v);
  }
  if (refined) d_fill_ghost<T>(u, lv, sg, 4);
}

// The saved copy of the coarse level (for the correction) and its FAS right-hand side under
// the children of lf: both read the coarse u after its ghost fill.
template <typename T>
__device__ __forceinline__ void d_save_rhs(T *__restrict__ u1, T *__restrict__ b, const T *__restrict__ u,
                                           const T *__restrict__ r, const LevelView &lc, const LevelView &lf,
                                           const int2 *__restrict__ coord_of, const OpParams<T> &pc, const WTab<T> &wt) {
  d_postrestrict<T>(b, u, r, lf, coord_of, pc, wt);
  d_copy_level<T>(u1, u, lc);
}

// The kernels of the per-operation path: each a grid-stride loop over its work, so the
// same bodies also run as the operations of one cooperative launch (srmg_seq.cu).
template <typename T>
__global__ void __launch_bounds__(256, 6) k_fill_ghost(T *__restrict__ u, LevelView lv, Signs sg, int mask) {
  pdl_enter(u);
  d_fill_ghost<T>(u, lv, sg, mask);
}

template <typename T>
__global__ void k_gs_colour(T *__restrict__ u, const T *__restrict__ b, LevelView lv,
                            OpParams<T> p, WTab<T> wt, int parity) {
  pdl_enter(u, b);
  d_gs_colour<T>(u, b, lv, p, wt, parity);
}

template <typename T>
__global__ void k_residual(T *__restrict__ r, const T *__restrict__ u, const T *__restrict__ b,
                           LevelView lv, OpParams<T> p, WTab<T> wt) {
  pdl_enter(r, u, b);
  d_residual<T>(r, u, b, lv, p, wt);
}

template <typename T>
__global__ void k_postrestrict(T *__restrict__ bf, const T *__restrict__ u, const T *__restrict__ r,
                               LevelView lv, const int2 *__restrict__ coord_of, OpParams<T> p,
                               WTab<T> wt) {
  pdl_enter(bf, u, r);
  d_postrestrict<T>(bf, u, r, lv, coord_of, p, wt);
}

template <typename T>
__global__ void k_restrict(T *__restrict__ u, LevelView lv) {
  pdl_enter(u);
  d_restrict<T>(u, lv);
}

template <typename T>
__global__ void k_interp_add(T *__restrict__ u, const T *__restrict__ u1, LevelView lv) {
  pdl_enter(u, u1);
  d_interp_add<T>(u, u1, lv);
}

template <typename T>
__global__ void k_copy_level(T *__restrict__ dst, const T *__restrict__ src, LevelView lv) {
  pdl_enter(dst, src);
  d_copy_level<T>(dst, src, lv);
}

template <typename T>
__global__ void k_diff_level(T *__restrict__ dst, const T *__restrict__ a1, const T *a2,
                             LevelView lv) {
  pdl_enter(dst, a1, a2);
  d_diff_level<T>(dst, a1, a2, lv);
}

template <typename T>
__global__ void k_gs4(T *__restrict__ u, const T *__restrict__ b, LevelView lv, OpParams<T> p, int p1, int p2) {
  pdl_enter(u, b);
  d_gs4<T>(u, b, lv, p, p1, p2);
}

template <typename T>
__global__ void __launch_bounds__(256, 1) k_down(T *__restrict__ u, T *__restrict__ r, const T *__restrict__ b, LevelView lv,
                       const int2 *__restrict__ coord_of, OpParams<T> p, WTab<T> wt) {
  pdl_enter(u, r, b);
  d_down<T>(u, r, b, lv, coord_of, p, wt);
}

template <typename T>
__global__ void __launch_bounds__(256, 1) k_save_rhs(T *__restrict__ u1, T *__restrict__ b, const T *__restrict__ u, const T *__restrict__ r,
                           LevelView lc, LevelView lf, const int2 *__restrict__ coord_of, OpParams<T> pc, WTab<T> wt) {
  pdl_enter(u1, b, u, r);
  d_save_rhs<T>(u1, b, u, r, lc, lf, coord_of, pc, wt);
}

template <typename T>
__global__ void __launch_bounds__(256, 1) k_correction(T *__restrict__ e, const T *__restrict__ u, const T *__restrict__ u1, LevelView lv,
                             Signs sg) {
  pdl_enter(e, u, u1);
  d_correction<T>(e, u, u1, lv, sg);
}

template <typename T>
__global__ void __launch_bounds__(256, 1) k_interp_push(T *__restrict__ u, const T *__restrict__ e, LevelView lv, PushView pv, unsigned sw,
                              Signs sg, bool refined) {
  pdl_enter(u, e);
  d_interp_push<T>(u, e, lv, pv, sw, sg, refined);
}

// The colour sweeps with their ghost pushes (PushView), the per-operation V-cycle's most
// frequent kernels and a chain of latencies: block record, coefficients, cells, a dozen
// dependent fp64 operations, then the push list and its entries.  All that comes from tables
// -- everything but u and b -- is loaded before the wait for the previous kernel: a thread's
// first cell (nearly always its only one) with its pushes.  u and b are not
// __restrict__, so that their loads stay below it.  Up to ~16k cells a sweep the time does
// not depend on the level's size: an order-4 sweep 1.7 us in a row of them (4.7 before, with
// coefficients from nine fp64 divisions a cell and nothing ahead of the wait).
template <typename T, bool FOUR, int GEOM>
__global__ void __launch_bounds__(128, 1) k_gs_push(T *u, const T *b, LevelView lv, OpParams<T> p, WTab<T> wt, int p1,
                                                 int p2, PushView pv, unsigned sg) {
  constexpr int N = FOUR ? 64 : 128;  // cells of a colour per block
  constexpr int kAhead = 3;           // a cell by a block's corner has that many pushes
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int total = lv.nblk * N, stride = gridDim.x * blockDim.x;  // a field holds fewer than 2^31 values here
  struct Cell {
    int at, e0, e1;
    int2 d[kAhead];
    Row4 r;   // FOUR
    W5<T> w;  // red-black
  };
  auto load = [&](int t) {
    Cell q;
    const int bi = t / N, c = t % N;
    const int y = FOUR ? 2 + 2 * (c >> 3) + p2 : 2 + (c >> 3);
    const int x = 2 + 2 * (c & 7) + (FOUR ? p1 : ((p1 ^ (y + 1)) & 1));
    const int *off = pv.off + bi * 256 + (x - kG) + kM * (y - kG);
    const int4 bk = lv.blocks[bi];
    q.e0 = off[0];
    q.e1 = off[1];
    q.at = bk.x * kSS + x + kS * y;
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      if (q.e0 + k < q.e1) q.d[k] = pv.ent[q.e0 + k];
    if (FOUR) {
      if (GEOM) q.r = row4(p, gidx(bk.y, x), gidx(bk.z, y));
    } else {
      q.w = weights<T>(wt, GEOM, bk.y, bk.z, x, y);
    }
    return q;
  };
  auto push = [&](int2 d, T v) {
    if (d.y != 255) {  // mirrors on the way
      const int k1 = d.y & 15, k2 = d.y >> 4;
      if (k1 < 9) v = dmul<T>(T((int)((sg >> (2 * k1)) & 3u) - 1), v);
      if (k2 < 9) v = dmul<T>(T((int)((sg >> (2 * k2)) & 3u) - 1), v);
    }
    u[d.x] = v;
  };
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  Cell q;
  if (t < total) q = load(t);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  while (t < total) {
    T *uc = u + q.at;
    const T bo = b[q.at];
    T nv;
    if (FOUR) {
      nv = gs4_value<T, GEOM>(uc, bo, p, q.r);
    } else {
      const T v = fma(p.s, bo, apply5<T>(uc, 0, 0, q.w, p.centre));
      nv = fma(p.nwc, v, uc[0]);
    }
    *uc = nv;
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      if (q.e0 + k < q.e1) push(q.d[k], nv);
    for (int e = q.e0 + kAhead; e < q.e1; ++e) push(pv.ent[e], nv);
    if (total - t <= stride) break;
    t += stride;
    q = load(t);
  }
}

// The coarse end of a V-cycle as one cluster runs it (srmg_coarse.cu): up to kCoarseCtas blocks
// per level and CTA slot, kCoarsePer slots a level.
constexpr int kCoarseLevels = 12, kCoarseCtas = 16, kCoarsePer = 16, kCoarseThreads = 256;
constexpr int kCoarseSmem = 227 * 1024;
struct CoarseCycle {
  OpParams<double> p[kCoarseLevels + 1];
  double *u, *b, *r;
  Signs sg;
  WTab<double> wt;
  int top, inner, known;      // inner: level top + 1 exists and has been restricted (residual in r);
                              // known: else, whether level top's ghosts are filled
  int ndown, ntop, nup, ncycles;
  // the tree's tables, set by coarse_launch
  const int4 *tab;
  int slots, levels, tabq, corners;
  unsigned refined, mref;     // per-level bits
  int base[kCoarseLevels + 2], nblk[kCoarseLevels + 1], per[kCoarseLevels + 1];  // slots of level l: base[l]..
  int pbase[kCoarseLevels + 2];                                                  // pushes of level l: pbase[l]..
};

// FMG's step up to level lf: level lf saved, and the correction of the level below it.
template <typename T>
__global__ void k_fmg_step(T *__restrict__ e, T *__restrict__ u1, const T *__restrict__ u, LevelView lf, LevelView lc,
                           Signs sg) {
  pdl_enter(e, u1, u);
  d_correction<T>(e, u, u1, lc, sg);
  d_copy_level<T>(u1, u, lf);
}

}  // namespace srmg
