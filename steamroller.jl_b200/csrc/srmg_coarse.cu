// srmg_coarse.cu -- the coarse end of a V-cycle (src/multigrid.jl:60-106 on levels 1..top) in
// one cluster of 16 CTAs, its fields in their shared memories.
//
// What it replaces is a chain of ~20 dependent steps a level, each on a few thousand cells: a
// launch or a grid barrier with its trips through L2 apart, 1.7 us a colour as launches, 4 us
// a sweep and 3 to 5 us a transfer as phases of the persistent kernel.  Here a block's tiles
// stay in one CTA, ghosts go to the neighbour's CTA by stores into its shared memory, and a
// step is a cluster barrier (0.3 us), a stencil from shared memory (0.2) and those stores (0.2)
// away from the next: latency all the way.  Two FP64 V-cycles (2, 4, 2) on the uniform tree of
// 1 to 256 blocks, whole in the cluster: 231 -> 130 us (one launch); order 4 on the 2725-block
// tree, levels of 1 to 64 blocks here: 164 -> 78 us of a cycle; full multigrid on the
// 400k-cell channel tree: 1507 -> 1130 us.  256 threads a CTA, one cell a thread at a time: more
// warps make the barriers dearer, more cells a thread the chain longer (order 4, 512 threads:
// 87 us of that cycle; two cells: 82).
#include <algorithm>

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

// Where a block is: CTA of the cluster and slot, its tile's index in that CTA's fields.
constexpr int kSlotBits = 6;
inline int pos_of(int cta, int slot) { return cta << kSlotBits | slot; }

// Tables of a CTA, one array over its slots after the other (in int4 a slot: 1 the block, 1 its
// parent, 4 faces, 4 corners), then 2 a level: where the level's pushes of each kind of cell
// begin, then the pushes.  Blocks go by position: blocks[].x, faces[].y; child[] = {block id,
// parent's position, sb_r, sb_z}.
constexpr int kSlotQ = 1 + 1 + 4 + 4;
// A push, the ghost x (9 bits cell, 6 slot, 4 CTA) that takes the value of cell y (9 bits cell, 6
// slot) times two boundary-table entries (4 bits each, above 8 none).  Cells are of four
// kinds, by the parities of x and y, in the order (0,1), (1,0), (0,0), (1,1): a colour of either
// smoother is a run of them.
constexpr int kKindAt[4] = {2, 0, 1, 3};  // [2 (x & 1) + (y & 1)]

// Coefficients kept per slot: 16 rows of Row4 or of a pair of weights.
constexpr int coef_n(bool four, int geom) { return geom == 0 ? 0 : four ? 16 * kCoef4 : 16 * 2; }

// Shared memory of a CTA with `all` slots, `below` of them on levels below the coarsest part's
// top: u and b for all, the correction below the top, the saved u there and, where finer
// levels follow, on the top too.
int64_t smem_bytes(int all, int below, bool inner, int top, int pushes, bool four, int geom) {
  const int64_t tiles = 2 * all + below + (inner ? all : below);
  return tiles * kSS * 8 + 16 * 8 + (int64_t)all * (16 * kSlotQ + 8 * coef_n(four, geom)) + 32 * top + 8 * pushes;
}

struct Tiles {  // a field by position
  double *own;
  int cta;
};
__device__ __forceinline__ double *tile_of(const Tiles &f, int64_t pos) {
  double *p = f.own + ((int)pos & ((1 << kSlotBits) - 1)) * kSS;
  const int cta = (int)pos >> kSlotBits;
  if (cta == f.cta) return p;
  double *q;
  asm("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(p), "r"(cta));
  return q;
}

__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void cp8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// Every step ends in cluster_arrive() and begins, after what it can prepare, with
// cluster_wait(); all threads of the cluster take all of them.
template <bool FOUR, int GEOM>
__global__ void __launch_bounds__(kCoarseThreads, 1) k_vcycle_coarse(const __grid_constant__ CoarseCycle L) {
  typedef double T;
  extern __shared__ __align__(16) unsigned char raw[];
  const int tid = threadIdx.x, cta = blockIdx.x, top = L.top;
  const int all = L.base[top + 1], below = L.base[top];
  constexpr int kCoef = coef_n(FOUR, GEOM);
  T *const su = reinterpret_cast<T *>(raw), *const sb = su + all * kSS, *const se = sb + all * kSS;
  T *const s1 = se + below * kSS, *const scoef = s1 + (L.inner ? all : below) * kSS;
  T *const sgn = scoef + all * kCoef;
  int4 *const blk = reinterpret_cast<int4 *>(sgn + 16), *const child = blk + all;
  int4 *const faces = child + all, *const cfaces = faces + 4 * all, *const headq = cfaces + 4 * all;
  const int *const head = reinterpret_cast<const int *>(headq);
  const int2 *const ent = reinterpret_cast<const int2 *>(headq + 2 * top);
  const Tiles fu{su, cta}, f1{s1, cta}, fe{se, cta};
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  {  // the part of levels 1..top of each array of this CTA's tables
    const int4 *src = L.tab + (int64_t)cta * L.tabq;
    int4 *dst = blk;
    const int have[6] = {all, all, 4 * all, 4 * all, 2 * top, L.pbase[top + 1] / 2};
    const int full[6] = {L.slots, L.slots, 4 * L.slots, 4 * L.slots, 2 * L.levels, 0};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      for (int i = tid; i < have[k]; i += kCoarseThreads) cp16(dst + i, src + i);
      dst += have[k];
      src += full[k];
    }
    if (tid < 16) sgn[tid] = tid < 9 ? L.sg.v[tid] : 1.0;
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  auto own = [&](int l) { return max(0, min(L.per[l], L.nblk[l] - cta * L.per[l])); };
  auto each = [&](auto f) {  // f(slot, level) for this CTA's blocks
    for (int l = 1; l <= top; ++l)
      for (int q = 0; q < own(l); ++q) f(L.base[l] + q, l);
  };
  each([&](int q, int) {
    const int64_t o = (int64_t)child[q].x * kSS;
    for (int i = tid; i < kSS; i += kCoarseThreads) {
      cp8(su + q * kSS + i, L.u + o + i);
      cp8(sb + q * kSS + i, L.b + o + i);
    }
    if (GEOM != 0)
      for (int i = tid; i < 16; i += kCoarseThreads) {
        const int gi = kG + i - 1 + kM * ((GEOM == 1 ? blk[q].y : blk[q].z) - 1);
        T *c = scoef + q * kCoef + i * (kCoef / 16);
        if (FOUR) {
          for (int k = 0; k < kCoef4; ++k) c[k] = L.p[1].c4[kCoef4 * gi + k];
        } else {
          c[0] = L.wt.wm[gi];
          c[1] = L.wt.wp[gi];
        }
      }
  });
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  __syncthreads();  // a sweep reads coefficients ahead of its wait
  cluster_arrive();

  auto kind = [](int c) { return (0x3102 >> (4 * c)) & 3; };  // kKindAt
  auto step = [&](auto body) {
    cluster_wait();
    body();
    cluster_arrive();
  };
  auto view = [&](int l) {
    const int q = L.base[l], n = own(l);
    return LevelView{blk + q, faces + 4 * q, child + q, n, n, l, L.corners ? cfaces + 4 * q : nullptr};
  };
  auto coef = [&](int q, int x, int y) { return scoef + q * kCoef + ((GEOM == 1 ? x : y) - kG) * (kCoef / 16); };
  auto weights_at = [&](int q, int x, int y) {
    W5<T> w{T(1), T(1), T(1), T(1)};
    if (GEOM != 0) {
      const double2 c = *reinterpret_cast<const double2 *>(coef(q, x, y));
      if (GEOM == 1) w.rm = c.x, w.rp = c.y;
      else w.zm = c.x, w.zp = c.y;
    }
    return w;
  };
  auto lhs = [&](const OpParams<T> &p, int q, int x, int y) {
    if (FOUR) return sum9<T, GEOM>(su + q * kSS + x + kS * y, GEOM ? Row4(coef(q, x, y)) : Row4());
    return apply5<T>(su + q * kSS, x, y, weights_at(q, x, y), p.centre);
  };
  // pushes i..end of the list, a thread every kCoarseThreads of them (its first one loaded)
  auto push = [&](int i, int end, int2 e) {
    while (i < end) {
      const T v = dmul<T>(dmul<T>(su[(e.y >> 9 & 63) * kSS + (e.y & 511)], sgn[e.y >> 15 & 15]), sgn[e.y >> 19]);
      T *to = su + (e.x >> 9 & 63) * kSS + (e.x & 511);
      const int dst = e.x >> 15;
      if (dst == cta) {
        *to = v;
      } else {
        uint32_t at;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(to)), "r"(dst));
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
      }
      i += kCoarseThreads;
      if (i < end) e = ent[i];
    }
  };
  // what a fill of level l (d_fill_ghost with this mask) would write
  auto fill = [&](int l, int mask) {
    if ((L.mref >> l) & 1) {
      d_fill_ghost<T>(fu, view(l), L.sg, mask, 0, 1);
      return;
    }
    const int i = head[8 * (l - 1)] + tid, end = head[8 * (l - 1) + 4];
    if (mask & 3) push(i, end, i < end ? ent[i] : int2());
    if (mask & 4) d_fill_ghost<T>(fu, view(l), L.sg, 4, 0, 1);
  };
  // gauss_seidel_iter! with ghost pushes, n sweeps.  known: the ghosts are what a fill would
  // make of the cells now (else, and where boundary corners mirror refinement ghosts, the
  // first colour is followed by a fill).  What comes from tables is loaded before
  // the wait; the pushes follow from a list of their own, a thread
  // each: at the cells, most lanes would wait for the few that have some, twice the time of
  // the rest.  A level of one block keeps to CTA 0's own barriers.
  auto gs = [&](int l, int n, bool known) {
    constexpr int N = FOUR ? 64 : 128;  // cells of a colour per block
    constexpr int kColours = FOUR ? 4 : 2;
    const OpParams<T> p = L.p[l];
    const int q0 = L.base[l], total = own(l) * N;
    const bool solo = L.nblk[l] == 1;
    if (solo && cta != 0) {
      cluster_wait();
      cluster_arrive();
      return;
    }
    struct Cell {
      int at;
      Row4 r;
      W5<T> w;
    };
    auto load = [&](int t, int c) {
      Cell k;
      const int q = q0 + t / N, j = t % N;
      const int y = FOUR ? 2 + 2 * (j >> 3) + (c & 1) : 2 + (j >> 3);
      const int x = 2 + 2 * (j & 7) + (FOUR ? c >> 1 : ((c ^ (y + 1)) & 1));
      k.at = q * kSS + x + kS * y;
      if (!FOUR) k.w = weights_at(q, x, y);
      else if (GEOM) k.r = Row4(coef(q, x, y));
      return k;
    };
    auto value = [&](const Cell &k) -> T {
      const T bo = sb[k.at];
      if (FOUR) return gs4_value<T, GEOM>(su + k.at, bo, p, k.r);
      return fma(p.nwc, fma(p.s, bo, apply5<T>(su + k.at, 0, 0, k.w, p.centre)), su[k.at]);
    };
    bool first = true;
    auto wait = [&] {
      if (first || !solo) cluster_wait();
      else __syncthreads();
      first = false;
    };
    for (int i = 0; i < n; ++i)
#pragma unroll 1
      for (int c = 0; c < kColours; ++c) {
        int t = tid;
        Cell k;
        if (t < total) k = load(t, c);
        const int *run = head + 8 * (l - 1) + (FOUR ? kind(c) : 2 * c);
        const int i0 = run[0] + tid, i1 = run[FOUR ? 1 : 2];
        const int2 e = i0 < i1 ? ent[i0] : int2();
        wait();
        while (t < total) {
          su[k.at] = value(k);
          t += kCoarseThreads;
          if (t < total) k = load(t, c);
        }
        __syncthreads();
        push(i0, i1, e);
        if (i == 0 && c == 0 && (!known || ((L.mref >> l) & 1))) {
          if (!solo) cluster_arrive();
          wait();
          fill(l, 3);
        }
        if (!solo || (i == n - 1 && c == kColours - 1)) cluster_arrive();
      }
  };
  // the coarse half of level l + 1's descent
  auto arrive_at = [&](int l) {
    step([&] { fill(l, (L.refined >> l) & 1 ? 7 : 3); });
    step([&] {
      const OpParams<T> p = L.p[l];
      for (int t = tid; t < own(l) * kSS; t += kCoarseThreads) {
        const int q = L.base[l] + t / kSS, o = t % kSS, x = o % kS, y = o / kS;
        s1[q * kSS + o] = su[q * kSS + o];
        if (x < kG || x >= kG + kM || y < kG || y >= kG + kM) continue;
        if (!((blk[q].w >> (((x - kG) >> 3) + 2 * ((y - kG) >> 3))) & 1)) continue;
        const T r = l == top ? L.r[(int64_t)child[q].x * kSS + o] : se[q * kSS + o];
        sb[q * kSS + o] = -(r + quot(lhs(p, q, x, y), p.s, p.rs));
      }
    });
  };
  if (L.inner) arrive_at(top);
#pragma unroll 1
  for (int cyc = 0; cyc < L.ncycles; ++cyc) {
    const bool known = L.known || L.inner || cyc > 0;  // level top's ghosts
#pragma unroll 1
    for (int l = top; l >= 2; --l) {
      gs(l, L.ndown, known || l < top);
      step([&] {
        const OpParams<T> p = L.p[l];
        for (int t = tid; t < own(l) * 64; t += kCoarseThreads) {
          const int q = L.base[l] + (t >> 6), kx = t & 7, ky = (t >> 3) & 7;
          const int4 ch = child[q];
          T f = T(0), g = T(0);
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int x = 2 + 2 * kx + i, y = 2 + 2 * ky + j, o = x + kS * y;
              f = dadd<T>(f, su[q * kSS + o]);
              g = dadd<T>(g, -(sb[q * kSS + o] + quot(lhs(p, q, x, y), p.s, p.rs)));
            }
          const int o = (2 + 8 * (ch.z - 1) + kx) + kS * (2 + 8 * (ch.w - 1) + ky);
          tile_of(fu, ch.y)[o] = dmul<T>(f, T(0.25));
          tile_of(fe, ch.y)[o] = dmul<T>(g, T(0.25));
        }
      });
      arrive_at(l - 1);
    }
    gs(1, L.ntop, known || top > 1);
#pragma unroll 1
    for (int l = 2; l <= top; ++l) {
      step([&] {
        const LevelView lc = view(l - 1);
        for (int t = tid; t < lc.nblk * kSS; t += kCoarseThreads) {
          const int bi = t / kSS, o = t % kSS;
          se[(L.base[l - 1] + bi) * kSS + o] = filled_diff<T>(fu, f1, fe, lc, L.sg, bi, lc.blocks[bi].x, o % kS, o / kS);
        }
      });
      step([&] {
        for (int t = tid; t < own(l) * 256; t += kCoarseThreads) {
          const int q = L.base[l] + (t >> 8), dx = t & 15, dy = (t >> 4) & 15;
          const int4 ch = child[q];
          const int ir = dx & 1, iz = dy & 1;
          const T *cb = tile_of(fe, ch.y) + 2 + 8 * (ch.z - 1) + (dx >> 1) + kS * (2 + 8 * (ch.w - 1) + (dy >> 1));
          T v = dmul<T>(T(0.5), cb[0]);
          v = dadd<T>(v, dmul<T>(T(0.25), cb[2 * ir - 1]));
          v = dadd<T>(v, dmul<T>(T(0.25), cb[kS * (2 * iz - 1)]));
          T *d = su + q * kSS + (2 + dx) + kS * (2 + dy);
          v = dadd<T>(v, *d);
          *d = v;
        }
        const int i = head[8 * (l - 1)] + tid, end = head[8 * (l - 1) + 4];
        const int2 first = i < end ? ent[i] : int2();
        __syncthreads();
        push(i, end, first);
        if ((L.refined >> l) & 1) d_fill_ghost<T>(fu, view(l), L.sg, 4, 0, 1);
      });
      gs(l, L.nup, true);
    }
  }
  cluster_wait();
  if (L.inner) {  // the correction of level top, for the prolongation of the next
    const LevelView lv = view(top);
    for (int t = tid; t < lv.nblk * kSS; t += kCoarseThreads) {
      const int bi = t / kSS, o = t % kSS;
      L.r[(int64_t)child[L.base[top] + bi].x * kSS + o] =
          filled_diff<T>(fu, f1, fe, lv, L.sg, bi, lv.blocks[bi].x, o % kS, o / kS);
    }
  }
  each([&](int q, int l) {
    const int64_t o = (int64_t)child[q].x * kSS;
    for (int i = tid; i < kSS; i += kCoarseThreads) {
      L.u[o + i] = su[q * kSS + i];
      if (l < top || L.inner) L.b[o + i] = sb[q * kSS + i];
    }
  });
  cluster_arrive();  // a CTA's shared memory stays until no one reads it
  cluster_wait();
}

typedef void (*CoarseKernel)(const CoarseCycle);
CoarseKernel coarse_kernel(bool four, int geom) {
  return four ? (geom == 0 ? k_vcycle_coarse<true, 0> : geom == 1 ? k_vcycle_coarse<true, 1> : k_vcycle_coarse<true, 2>)
              : (geom == 0   ? k_vcycle_coarse<false, 0>
                 : geom == 1 ? k_vcycle_coarse<false, 1>
                             : k_vcycle_coarse<false, 2>);
}

cudaError_t coarse_config(CoarseKernel k, int smem, cudaLaunchConfig_t *cfg, cudaLaunchAttribute *at) {
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  // the same limit on every launch: another thread's may be about to need more
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kCoarseSmem);
  cfg->gridDim = dim3(kCoarseCtas);
  cfg->blockDim = dim3(kCoarseThreads);
  cfg->dynamicSmemBytes = smem;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kCoarseCtas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg->attrs = at;
  cfg->numAttrs = 2;
  return e;
}

}  // namespace

// Positions, faces, parents and pushes of the levels from 1 up that the cluster can hold.
int srmg::ensure_coarse(srmg_ctx *ctx) {
  if (ctx->coarse.state != 0 || !ctx->has_tree || ctx->D != 2) return SRMG_OK;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  CK(cudaStreamIsCapturing(ctx->stream, &cap));
  if (cap != cudaStreamCaptureStatusNone) return SRMG_OK;
  CoarseTab &C = ctx->coarse;
  if (ctx->has_corners && ctx->push_state == 0) return SRMG_OK;
  C.state = -1;
  if (ctx->has_corners && ctx->push_state != 1) return SRMG_OK;
  const std::vector<CoarseTab::Level> &T = C.tree;
  int levels = 0;
  std::vector<int> pos((size_t)ctx->max_blk, -1);
  int slots = 0;
  for (int l = 1; l <= (int)T.size(); l++) {
    const DevLevel &L = ctx->lv[l - 1];
    const CoarseTab::Level &h = T[l - 1];
    const int per = (L.nblk + kCoarseCtas - 1) / kCoarseCtas;
    if (L.nblk < 1 || per > kCoarsePer || slots + per > (1 << kSlotBits) || (l > 1 && L.nch != L.nblk)) break;
    for (int bi = 0; bi < L.nblk; bi++) pos[h.blk[bi].x] = pos_of(bi / per, slots + bi % per);
    C.nblk[l] = L.nblk;
    C.per[l] = per;
    C.base[l] = slots;
    slots += per;
    C.base[l + 1] = slots;
    levels = l;
  }
  if (levels == 0) return SRMG_OK;
  // the pushes: of the star's faces by rule, of a BoxStencil tree from its push tables
  // Counted first, then placed: bin (level, CTA, kind).
  const int mask = (1 << kSlotBits) - 1;
  std::vector<int> bin((size_t)levels * kCoarseCtas * 4, 0);
  struct Push { int bin; int2 word; };
  std::vector<Push> list;
  list.reserve((size_t)slots * kCoarseCtas * 144);
  auto add = [&](int l, int src, int x, int y, int dst, int cell, int k1, int k2) {
    const int k = ((l - 1) * kCoarseCtas + (src >> kSlotBits)) * 4 + kKindAt[2 * (x & 1) + (y & 1)];
    bin[k]++;
    list.push_back({k, make_int2(cell | (dst & mask) << 9 | (dst >> kSlotBits) << 15,
                                 (x + kS * y) | (src & mask) << 9 | k1 << 15 | k2 << 19)});
  };
  for (int l = 1; l <= levels; l++) {
    const CoarseTab::Level &h = T[l - 1];
    const int nb = ctx->lv[l - 1].nblk;
    if (ctx->has_corners) {
      const PushView &pv = ctx->push_lv[l - 1];
      std::vector<int> off((size_t)nb * 256 + 1);
      CK(cudaMemcpy(off.data(), pv.off, off.size() * sizeof(int), cudaMemcpyDeviceToHost));
      std::vector<int2> ent(off.back());
      if (!ent.empty()) CK(cudaMemcpy(ent.data(), pv.ent, ent.size() * sizeof(int2), cudaMemcpyDeviceToHost));
      for (int k = 0; k < nb * 256; k++)
        for (int e = off[k]; e < off[k + 1]; e++) {
          const int dst = pos[ent[e].x / kSS];
          if (dst < 0) return SRMG_OK;
          add(l, pos[h.blk[k / 256].x], kG + k % 256 % kM, kG + k % 256 / kM, dst, ent[e].x % kSS, ent[e].y & 15,
              ent[e].y >> 4);
        }
      continue;
    }
    static const int kSign[4] = {3, 5, 1, 7};  // face_sign_index
    for (int k = 0; k < 4 * nb; k++) {
      const int me = pos[h.blk[k / 4].x], f = k % 4, type = h.face[k].x;
      if (type != FACE_NEIGHBOR && type != FACE_BOUNDARY) continue;
      if (type == FACE_NEIGHBOR && (h.face[k].y < 0 || h.face[k].y >= ctx->max_blk || pos[h.face[k].y] < 0))
        return SRMG_OK;
      for (int g = 0; g < kG; g++)
        for (int i = 0; i < kM; i++) {
          const int x = f == 0 ? g : f == 1 ? kG + kM + g : kG + i, y = f == 2 ? g : f == 3 ? kG + kM + g : kG + i;
          int sx = x, sy = y;
          if (type == FACE_NEIGHBOR) (f < 2 ? sx : sy) += f % 2 ? -kM : kM;
          else (f < 2 ? sx : sy) = (f % 2 ? 2 * (kG + kM) - 1 : 2 * kG - 1) - (f < 2 ? x : y);
          if (type == FACE_NEIGHBOR) add(l, pos[h.face[k].y], sx, sy, me, x + kS * y, 15, 15);
          else add(l, me, sx, sy, me, x + kS * y, kSign[f], 15);
        }
    }
  }
  C.pbase[1] = 0;
  for (int l = 1; l <= levels; l++) {
    int most = 0;
    for (int cta = 0; cta < kCoarseCtas; cta++) {
      const int *n = &bin[((l - 1) * kCoarseCtas + cta) * 4];
      most = std::max(most, n[0] + n[1] + n[2] + n[3]);
    }
    C.pbase[l + 1] = C.pbase[l] + (most + 1) / 2 * 2;
  }
  C.levels = levels;
  C.slots = slots;
  C.tabq = slots * kSlotQ + 2 * C.levels + C.pbase[C.levels + 1] / 2;
  std::vector<int4> img((size_t)kCoarseCtas * C.tabq, make_int4(0, 0, 0, 0));
  std::vector<int2 *> fillp(bin.size());
  for (int l = 1; l <= C.levels; l++)
    for (int cta = 0; cta < kCoarseCtas; cta++) {
      int4 *T4 = img.data() + (size_t)cta * C.tabq + slots * kSlotQ;
      int *head = reinterpret_cast<int *>(T4 + 2 * (l - 1));
      int2 *ent = reinterpret_cast<int2 *>(T4 + 2 * C.levels);
      int n = C.pbase[l];
      for (int k = 0; k < 4; k++) {
        const int b = ((l - 1) * kCoarseCtas + cta) * 4 + k;
        head[k] = n;
        fillp[b] = ent + n;
        n += bin[b];
      }
      head[4] = n;
    }
  for (const Push &e : list) *fillp[e.bin]++ = e.word;
  for (int l = 1; l <= levels; l++) {
    const CoarseTab::Level &h = T[l - 1];
    for (size_t bi = 0; bi < h.blk.size(); bi++) {
      const int p = pos[h.blk[bi].x], s = p & ((1 << kSlotBits) - 1);
      int4 *T4 = img.data() + (size_t)(p >> kSlotBits) * C.tabq;
      int4 *blk = T4 + s, *child = T4 + slots + s, *face = T4 + 2 * slots + 4 * s, *corner = T4 + 6 * slots + 4 * s;
      *blk = make_int4(p, h.blk[bi].y, h.blk[bi].z, h.blk[bi].w);  // w: the quadrants with finer blocks
      *child = make_int4(h.blk[bi].x, 0, 0, 0);
      auto placed = [&](int4 f) {
        if (f.x == FACE_NEIGHBOR || f.x == FACE_REFBND) f.y = f.y >= 0 && f.y < ctx->max_blk ? pos[f.y] : -1;
        return f;
      };
      for (int k = 0; k < 4; k++) {
        face[k] = placed(h.face[4 * bi + k]);
        if (!h.corner.empty()) corner[k] = placed(h.corner[4 * bi + k]);
        for (const int4 *f : {face + k, corner + k})
          if ((f->x == FACE_NEIGHBOR || f->x == FACE_REFBND) && f->y < 0) return SRMG_OK;
      }
    }
  }
  for (int l = 2; l <= levels; l++)  // parents
    for (const int4 &e : T[l - 1].child) {
      const int pc = pos[e.y], pf = pos[e.x];
      if (pc < 0 || pf < 0) return SRMG_OK;
      int4 &c = img[(size_t)(pf >> kSlotBits) * C.tabq + slots + (pf & mask)];
      c.y = pc, c.z = e.z, c.w = e.w;
    }
  // the GPU must have room for a cluster of this size
  int &able = ctx->coarse_able[ctx->has_corners];
  if (able == 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    const CoarseKernel k = coarse_kernel(ctx->has_corners, 1);
    int clusters = 0;
    cudaError_t e = coarse_config(k, kCoarseSmem, &cfg, attr);
    cfg.numAttrs = 1;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, k, &cfg);
    if (e != cudaSuccess) (void)cudaGetLastError();
    able = e == cudaSuccess && clusters >= 1 ? 1 : -1;
  }
  if (able < 0) return SRMG_OK;
  if (ensure(ctx, C.tab, img.size() * sizeof(int4))) {  // no memory for them: cycles run as without
    (void)cudaGetLastError();
    return SRMG_OK;
  }
  RC(upload(ctx, C.tab.p, img.data(), img.size() * sizeof(int4)));
  C.state = 1;
  return SRMG_OK;
}

// The levels from 1 up that a cycle with finest level lmax can run in the cluster, of up to
// `most` blocks each.
int srmg::coarse_top(const srmg_ctx *ctx, int lmax, bool four, int geom, int most) {
  const CoarseTab &C = ctx->coarse;
  if (C.state != 1) return 0;
  int levels = 0;
  while (levels < std::min(lmax, C.levels) && C.nblk[levels + 1] <= most) ++levels;
  for (int t = levels; t >= 1; t--)
    if (smem_bytes(C.base[t + 1], C.base[t], t < lmax, t, C.pbase[t + 1], four, geom) <= kCoarseSmem) return t;
  return 0;
}

int srmg::coarse_launch(srmg_ctx *ctx, CoarseCycle &A, bool four, int geom) {
  const CoarseTab &C = ctx->coarse;
  A.tab = (const int4 *)C.tab.p;
  A.slots = C.slots;
  A.levels = C.levels;
  A.tabq = C.tabq;
  A.corners = ctx->has_corners;
  for (int l = 1; l <= A.top; l++) {
    A.base[l] = C.base[l];
    A.nblk[l] = C.nblk[l];
    A.per[l] = C.per[l];
  }
  A.base[A.top + 1] = C.base[A.top + 1];
  for (int l = 1; l <= A.top + 1; l++) A.pbase[l] = C.pbase[l];
  A.refined = ctx->refbnd_levels;
  A.mref = ctx->has_corners ? ctx->mref_levels : 0;
  const CoarseKernel k = coarse_kernel(four, geom);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  const int64_t smem =
      smem_bytes(C.base[A.top + 1], C.base[A.top], A.inner, A.top, A.pbase[A.top + 1], four, geom);
  CK(coarse_config(k, (int)smem, &cfg, attr));
  cfg.stream = ctx->stream;
  CK(cudaLaunchKernelEx(&cfg, k, A));
  ctx->launches++;
  return SRMG_OK;
}
