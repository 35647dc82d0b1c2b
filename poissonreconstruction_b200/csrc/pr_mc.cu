// Extraction stage: iso value and marching cubes, bit-identical to the crate given the
// same FP64 coefficients.
//
//   iso  = mean of FEMTree::evaluate at the points      src/reconstructor.rs:56, src/fem_tree.rs:490-513
//   mesh = FEMTree::extract_surface                      src/fem_tree.rs:576-636
//
// The crate visits every leaf cell in Morton order, classifies the 8 corner values
// against iso, emits one vertex per cut edge (edge order 0..11), deduplicates vertices
// through a hash map keyed by ((x*1e9) as u64, (y*1e9) as u64, (z*1e9) as u64) and numbers
// them in order of first appearance, then emits TRI_TABLE triangles in row order.  The GPU
// version is a count / scan / emit pipeline:
//   1. per cell: case index; per block of cells: active-cell count      (k_mc_count)
//   2. exclusive scan; active cells written in Morton order             (k_mc_compact)
//   3. per active cell: vertex slots (cell order, then edge order) with position and key
//   4. a hash table of the keys holds the first slot of each, which is its vertex; vertex ids =
//      rank of first slots in slot order (= the crate's first-appearance numbering)
//   5. triangles from the packed table, vertices back-transformed to model space.
// Corner values at integer grid positions reduce to a shifted gather (the evaluation is
// offset by one cell, src/fem_tree.rs:645-649): node k-1 per axis, none at k = 0 and the
// last node counted twice at k = res.
#include <cub/cub.cuh>

#include "pr_internal.cuh"

#define PR_MC_TABLE_QUAL __constant__
#include "mc_tri_table.inc"

namespace pr {

namespace {

constexpr int kThreads = 256;

inline unsigned grid_for(uint64_t n, int threads = kThreads, uint64_t cap = 1u << 22) {
  uint64_t g = (n + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (unsigned)g;
}

__constant__ int c_co[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0}, {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
__constant__ int c_ev[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                                {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};

// edge e is cut iff its corners classify differently (== the crate's EDGE_TABLE)
__device__ __forceinline__ uint32_t edge_mask(uint32_t mc) {
  uint32_t m = 0;
#pragma unroll
  for (int e = 0; e < 12; ++e)
    if (((mc >> c_ev[e][0]) & 1u) != ((mc >> c_ev[e][1]) & 1u)) m |= 1u << e;
  return m;
}

// bspline1 (src/fem_tree.rs:640-642)
__device__ __forceinline__ double bspline1(double t) {
  if (t < 0.0 || t > 2.0) return 0.0;
  if (t <= 1.0) return t;
  return xsub(2.0, t);
}

// FEMTree::evaluate (src/fem_tree.rs:490-513), same operation order
__device__ double eval_fem(const double* __restrict__ x, uint32_t D, double px, double py, double pz) {
  const int64_t res = 1ll << D;
  const double h = 1.0 / (double)res;
  double s[3] = {xdiv(px, h), xdiv(py, h), xdiv(pz, h)};
  uint32_t o[3][2];
  double b[3][2];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int64_t f = sat_i64(floor(s[a]));
    int64_t lo = f - 1, hi = f;
    lo = lo < 0 ? 0 : (lo > res - 1 ? res - 1 : lo);
    hi = hi < 0 ? 0 : (hi > res - 1 ? res - 1 : hi);
    o[a][0] = (uint32_t)lo;
    o[a][1] = (uint32_t)hi;
    b[a][0] = bspline1(xsub(s[a], (double)o[a][0]));
    b[a][1] = bspline1(xsub(s[a], (double)o[a][1]));
  }
  double v = 0.0;
  for (int i = 0; i < 2; ++i) {
    if (b[0][i] == 0.0) continue;
    for (int j = 0; j < 2; ++j) {
      if (b[1][j] == 0.0) continue;
      for (int k = 0; k < 2; ++k) {
        if (b[2][k] == 0.0) continue;
        v = xadd(v, xmul(xmul(xmul(x[morton3(o[0][i], o[1][j], o[2][k])], b[0][i]), b[1][j]), b[2][k]));
      }
    }
  }
  return v;
}

// evaluate() at the integer grid position (kx,ky,kz) in [0,res]^3: the term of node k-1
// per axis, repeated twice at k = res, absent at k = 0; v accumulates the repeats.
__device__ __forceinline__ double corner_value(const double* __restrict__ x, int res, int kx, int ky, int kz) {
  int mx = kx == 0 ? 0 : (kx == res ? 2 : 1);
  int my = ky == 0 ? 0 : (ky == res ? 2 : 1);
  int mz = kz == 0 ? 0 : (kz == res ? 2 : 1);
  int m = mx * my * mz;
  if (m == 0) return 0.0;
  double s = x[morton3(kx == res ? res - 1 : kx - 1, ky == res ? res - 1 : ky - 1, kz == res ? res - 1 : kz - 1)];
  double v = 0.0;
  for (int i = 0; i < m; ++i) v = xadd(v, s);
  return v;
}

// Degree-2 coefficients come in Morton order (as every grid vector of the API) or, inside the
// reconstruction, in the natural order of the degree-2 solver (x + res (y + res z)). The extraction
// templates take DEG = 1 (the crate's basis), 2 (quadratic, Morton order) or 3 (quadratic, natural
// order); the arithmetic of 2 and 3 is the same.
template <bool NAT>
__device__ __forceinline__ uint64_t node_index(uint32_t x, uint32_t y, uint32_t z, uint32_t D) {
  return NAT ? (uint64_t)x + ((uint64_t)y << D) + ((uint64_t)z << (2 * D)) : (uint64_t)morton3(x, y, z);
}

// Degree-2 evaluation (the extension's quadratic node functions): per axis s = u / h, c = floor(s),
// t = s - c, weights (1-t)^2/2, (-2t^2 + 2t + 1)/2, t^2/2 of nodes c-1, c, c+1; nodes outside the
// grid are skipped; terms summed z-major, then y, then x, as ((x_j b_x) b_y) b_z.
template <bool NAT>
__device__ double eval_fem2(const double* __restrict__ x, uint32_t D, double px, double py, double pz) {
  const int64_t res = 1ll << D;
  const double h = 1.0 / (double)res;
  const double u[3] = {px, py, pz};
  int64_t c[3];
  double b[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double s = xdiv(u[a], h);
    c[a] = sat_i64(floor(s));
    const double t = xsub(s, (double)c[a]);
    const double omt = xsub(1.0, t);
    b[a][0] = xmul(xmul(0.5, omt), omt);
    b[a][1] = xmul(0.5, xadd(xadd(xmul(xmul(-2.0, t), t), xmul(2.0, t)), 1.0));
    b[a][2] = xmul(xmul(0.5, t), t);
  }
  double v = 0.0;
  for (int k = 0; k < 3; ++k) {
    const int64_t z = c[2] + k - 1;
    if (z < 0 || z >= res) continue;
    for (int j = 0; j < 3; ++j) {
      const int64_t y = c[1] + j - 1;
      if (y < 0 || y >= res) continue;
      for (int i = 0; i < 3; ++i) {
        const int64_t xx = c[0] + i - 1;
        if (xx < 0 || xx >= res) continue;
        v = xadd(v, xmul(xmul(xmul(x[node_index<NAT>((uint32_t)xx, (uint32_t)y, (uint32_t)z, D)], b[0][i]), b[1][j]),
                         b[2][k]));
      }
    }
  }
  return v;
}

// eval_fem2 at the integer grid position (kx,ky,kz): t = 0 on every axis, so the weights are
// 1/2, 1/2, 0 for nodes k-1, k, k+1; the zero-weight terms add +-0 and are left out (the sum
// never holds -0), which keeps the result identical.
template <bool NAT>
__device__ __forceinline__ double corner_value2(const double* __restrict__ x, uint32_t D, int kx, int ky, int kz) {
  const int res = 1 << D;
  double v = 0.0;
#pragma unroll
  for (int dz = -1; dz <= 0; ++dz) {
    const int z = kz + dz;
    if (z < 0 || z >= res) continue;
#pragma unroll
    for (int dy = -1; dy <= 0; ++dy) {
      const int y = ky + dy;
      if (y < 0 || y >= res) continue;
#pragma unroll
      for (int dx = -1; dx <= 0; ++dx) {
        const int xx = kx + dx;
        if (xx < 0 || xx >= res) continue;
        v = xadd(v, xmul(xmul(xmul(x[node_index<NAT>((uint32_t)xx, (uint32_t)y, (uint32_t)z, D)], 0.5), 0.5), 0.5));
      }
    }
  }
  return v;
}

template <int DEG>
__device__ __forceinline__ double eval_deg(const double* __restrict__ x, uint32_t D, double px, double py, double pz) {
  return DEG >= 2 ? eval_fem2<DEG == 3>(x, D, px, py, pz) : eval_fem(x, D, px, py, pz);
}

template <int DEG>
__device__ __forceinline__ uint32_t cell_case(const double* __restrict__ x, uint32_t D, uint32_t cell, double iso,
                                              double* cv) {
  const int res = 1 << D;
  uint32_t ox, oy, oz;
  unmorton3(cell, ox, oy, oz);
  uint32_t mc = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int kx = (int)ox + c_co[k][0], ky = (int)oy + c_co[k][1], kz = (int)oz + c_co[k][2];
    cv[k] = DEG >= 2 ? corner_value2<DEG == 3>(x, D, kx, ky, kz) : corner_value(x, res, kx, ky, kz);
    if (cv[k] < iso) mc |= 1u << k;
  }
  return mc;
}

// ------------------------------------------------------------------ iso value
// Per-point evaluate, then a deterministic compensated (Neumaier) sum.
template <int DEG>
__global__ void k_eval_points(const double* __restrict__ x, uint32_t D, const double* __restrict__ pts,
                              uint64_t stride_pt, uint64_t stride_axis, uint64_t n, double* __restrict__ out) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = eval_deg<DEG>(x, D, pts[i * stride_pt], pts[i * stride_pt + stride_axis],
                           pts[i * stride_pt + 2 * stride_axis]);
}

struct Neu {
  double s, c;
};
__device__ __forceinline__ Neu neu_add(Neu a, double v) {
  double t = a.s + v;
  if (fabs(a.s) >= fabs(v)) a.c += (a.s - t) + v;
  else a.c += (v - t) + a.s;
  a.s = t;
  return a;
}

template <int DEG>
__global__ void k_iso_partial(const double* __restrict__ x, uint32_t D, const double* __restrict__ upos, uint64_t P,
                              double* __restrict__ part) {
  Neu acc{0.0, 0.0};
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < P; i += (uint64_t)gridDim.x * blockDim.x)
    acc = neu_add(acc, eval_deg<DEG>(x, D, upos[i], upos[P + i], upos[2 * P + i]));
  __shared__ double ss[kThreads], sc[kThreads];
  ss[threadIdx.x] = acc.s;
  sc[threadIdx.x] = acc.c;
  __syncthreads();
  if (threadIdx.x == 0) {
    Neu t{0.0, 0.0};
    for (int i = 0; i < kThreads; ++i) {
      t = neu_add(t, ss[i]);
      t = neu_add(t, sc[i]);
    }
    part[2 * blockIdx.x] = t.s;
    part[2 * blockIdx.x + 1] = t.c;
  }
}

// the partials in order, one chain (thread 0); staged through shared memory, from which the chain reads
// ahead (from global memory it waits for every load): 40 us instead of 90 at 1M points, 15 instead of 30 at 100k
__global__ void __launch_bounds__(kThreads) k_iso_final(const double* __restrict__ part, int nb, double* __restrict__ out) {
  __shared__ double s[2 * kThreads];
  Neu t{0.0, 0.0};
  for (int b = 0; b < nb; b += kThreads) {
    const int m = min(kThreads, nb - b);
    for (int i = threadIdx.x; i < 2 * m; i += kThreads) s[i] = part[2 * b + i];
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll 8
      for (int i = 0; i < 2 * m; ++i) t = neu_add(t, s[i]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = t.s + t.c;
}

// ------------------------------------------------------------------ marching cubes
template <int DEG>
__global__ void k_mc_count(const double* __restrict__ x, uint32_t D, double iso, uint32_t* __restrict__ blockcnt) {
  const uint64_t n = 1ull << (3 * D);
  uint64_t cell = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  int active = 0;
  if (cell < n) {
    double cv[8];
    uint32_t mc = cell_case<DEG>(x, D, (uint32_t)cell, iso, cv);
    active = (mc != 0u && mc != 255u);
  }
  typedef cub::BlockReduce<int, kThreads> BR;
  __shared__ typename BR::TempStorage tmp;
  int tot = BR(tmp).Sum(active);
  if (threadIdx.x == 0) blockcnt[blockIdx.x] = (uint32_t)tot;
}

template <int DEG>
__global__ void k_mc_compact(const double* __restrict__ x, uint32_t D, double iso, const uint32_t* __restrict__ blockoff,
                             uint32_t* __restrict__ acell, uint8_t* __restrict__ acase, uint32_t* __restrict__ nedge,
                             uint32_t* __restrict__ ntri) {
  const uint64_t n = 1ull << (3 * D);
  uint64_t cell = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  uint32_t mc = 0;
  int active = 0;
  if (cell < n) {
    double cv[8];
    mc = cell_case<DEG>(x, D, (uint32_t)cell, iso, cv);
    active = (mc != 0u && mc != 255u);
  }
  typedef cub::BlockScan<int, kThreads> BS;
  __shared__ typename BS::TempStorage tmp;
  int off;
  BS(tmp).ExclusiveSum(active, off);
  if (active) {
    uint32_t a = blockoff[blockIdx.x] + (uint32_t)off;
    acell[a] = (uint32_t)cell;
    acase[a] = (uint8_t)mc;
    nedge[a] = __popc(edge_mask(mc));
    ntri[a] = PR_MC_NTRI[mc];
  }
}

// Vertex slots: position exactly as src/fem_tree.rs:613-624, key as :625
template <int DEG>
__global__ void k_mc_vertices(const double* __restrict__ x, uint32_t D, double iso, const uint32_t* __restrict__ acell,
                              uint64_t A, const uint32_t* __restrict__ eoff, double* __restrict__ pos,
                              uint64_t* __restrict__ k1, uint32_t* __restrict__ k2, uint64_t E,
                              int* __restrict__ err) {
  const int res = 1 << D;
  const double w = 1.0 / (double)res;  // (max_res >> d) as f64 / max_res as f64
  for (uint64_t a = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; a < A; a += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t cell = acell[a];
    double cv[8];
    uint32_t mc = cell_case<DEG>(x, D, cell, iso, cv);
    uint32_t em = edge_mask(mc);
    uint32_t ox, oy, oz;
    unmorton3(cell, ox, oy, oz);
    const int off[3] = {(int)ox, (int)oy, (int)oz};
    uint32_t sl = eoff[a];
    for (int e = 0; e < 12; ++e) {
      if (!((em >> e) & 1u)) continue;
      int ia = c_ev[e][0], ib = c_ev[e][1];
      double dv = xsub(cv[ib], cv[ia]);
      double t = fabs(dv) < 1e-15 ? 0.5 : xdiv(xsub(iso, cv[ia]), dv);
      uint64_t key[3];
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) {
        double base = xmul((double)(uint64_t)(off[ax] + c_co[ia][ax]), w);
        double d = (double)(c_co[ib][ax] - c_co[ia][ax]);
        double p = xadd(base, xmul(xmul(t, d), w));
        pos[(uint64_t)ax * E + sl] = p;
        key[ax] = sat_u64(xmul(p, 1e9));
      }
      if (key[0] >= (1ull << 30) || key[1] >= (1ull << 30) || key[2] >= (1ull << 30)) atomicOr(err, 1);
      k1[sl] = (key[0] << 30) | (key[1] & ((1ull << 30) - 1));
      k2[sl] = (uint32_t)(key[2] & ((1u << 30) - 1));
      ++sl;
    }
  }
}

// Vertices are slots with equal keys.  An open-addressing table (a power of two, 2 E entries or more)
// takes each key once; its entry ends as the smallest slot of that key, whatever the order of the
// insertions.  home[s] = the entry of slot s's key.  Scattered reads and atomics in L2 bound it: 46 us for
// the mesh of depth 9, k_mc_first 15, and k_mc_emit_tris 24 more than with ids in slot order.  By an LSD radix
// sort of the 90-bit keys, two gathers and two passes over the runs it is about 0.5 ms, and at depth 5 35
// launches more.
constexpr uint32_t kNoSlot = 0xffffffffu;
__global__ void k_mc_hash(const uint64_t* __restrict__ k1, const uint32_t* __restrict__ k2, uint64_t E, uint32_t mask,
                          uint32_t* __restrict__ table, uint32_t* __restrict__ home) {
  for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < E; s += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t a = k1[s];
    const uint32_t b = k2[s];
    uint64_t h = (a ^ ((uint64_t)b << 29)) * 0x9e3779b97f4a7c15ull;
    h ^= h >> 32;
    uint32_t e = (uint32_t)(h * 0xd6e8feb86659fd93ull >> 32) & mask;
    for (uint32_t probe = 0; probe < mask; ++probe, e = (e + 1) & mask) {  // ends early: entries stay free
      const uint32_t old = atomicCAS(table + e, kNoSlot, (uint32_t)s);
      if (old == kNoSlot) break;
      if (k1[old] == a && k2[old] == b) {
        if ((uint32_t)s < old) atomicMin(table + e, (uint32_t)s);
        break;
      }
    }
    home[s] = e;
  }
}
// first[s] = slot s is the first of its key
__global__ void k_mc_first(const uint32_t* __restrict__ table, const uint32_t* __restrict__ home, uint64_t E,
                           uint32_t* __restrict__ first) {
  for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < E; s += (uint64_t)gridDim.x * blockDim.x)
    first[s] = table[home[s]] == (uint32_t)s ? 1u : 0u;
}

struct Mat16 {
  double m[16];
};

__global__ void k_mc_emit_vertices(const double* __restrict__ pos, uint64_t E, const uint32_t* __restrict__ repflag,
                                   const uint32_t* __restrict__ vid_rep, int transform, Mat16 Mi,
                                   double* __restrict__ verts) {
  for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < E; s += (uint64_t)gridDim.x * blockDim.x) {
    if (!repflag[s]) continue;
    double p[3] = {pos[s], pos[E + s], pos[2 * E + s]};
    uint64_t v = vid_rep[s];
    if (transform) {
      // Mat4::transform_point (src/geometry.rs:256-262) with the inverse transform
#pragma unroll
      for (int r = 0; r < 3; ++r)
        verts[3 * v + r] =
            xadd(xadd(xadd(xmul(Mi.m[r], p[0]), xmul(Mi.m[4 + r], p[1])), xmul(Mi.m[8 + r], p[2])), Mi.m[12 + r]);
    } else {
#pragma unroll
      for (int r = 0; r < 3; ++r) verts[3 * v + r] = p[r];
    }
  }
}

__global__ void k_mc_emit_tris(const uint8_t* __restrict__ acase, uint64_t A, const uint32_t* __restrict__ eoff,
                               const uint32_t* __restrict__ toff, const uint32_t* __restrict__ table,
                               const uint32_t* __restrict__ home, const uint32_t* __restrict__ vid_rep,
                               uint64_t* __restrict__ tris) {
  for (uint64_t a = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; a < A; a += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t mc = acase[a];
    uint32_t em = edge_mask(mc);
    uint64_t packed = PR_MC_TRIS[mc];
    uint32_t nt = PR_MC_NTRI[mc];
    uint64_t t0 = toff[a];
    uint32_t e0 = eoff[a];
    for (uint32_t i = 0; i < 3 * nt; ++i) {
      uint32_t e = (uint32_t)((packed >> (4 * i)) & 15ull);
      uint32_t rank = __popc(em & ((1u << e) - 1u));
      tris[3 * t0 + i] = vid_rep[table[home[e0 + rank]]];
    }
  }
}

}  // namespace

// ------------------------------------------------------------------ block-tiled classification (depth >= 4)
// A CTA classifies the 16^3 cells of one Morton block.  Cell c has corners at grid positions c + co[k].
// The inside/outside bits of the block's 17^3 corner positions are one 17-bit word per (y, z) row: bit tx
// of row (ty, tz) is (corner value < iso) for grid position (o + t); a cell reads 4 words.
constexpr int MCW = 17;

__device__ __forceinline__ uint32_t sp4(uint32_t v) {
  return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4) | ((v & 8u) << 6);
}

// Degree 1: the corner value at a position is node (position - 1) per axis, so the bits are those of the
// block's own 16^3 nodes and of the low layer from the neighbour blocks (zeros outside the domain,
// matching the crate's empty evaluation at 0).  The value at a grid position equal to res on k axes is the
// node value added 2^k times in sequence, like the crate's evaluate() at the top boundary.  The values go
// from a coalesced 16-byte load (two nodes of a row) straight to bits: a lane's bits of one (y, z) row and
// its neighbour's (x bit 1 is lane bit 2) make the row.
__device__ void mc_masks1(uint32_t* mask, uint8_t* xbit, const double* __restrict__ x, uint32_t blk, int res,
                          double iso) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint32_t bx, by, bz;
  unmorton3(blk, bx, by, bz);
  const uint32_t last = (uint32_t)(res >> 4) - 1;
  const auto top = [](bool at_top, int l) { return at_top && l == 15 ? 2 : 1; };
  const bool tx = bx == last, ty = by == last, tz = bz == last;
  const auto bit = [iso](double s, int mult) {
    double v = s;
    for (int i = 1; i < mult; ++i) v = xadd(v, s);
    return (uint32_t)(v < iso);
  };
  const auto load2 = [x](uint64_t i) { return __ldg(reinterpret_cast<const double2*>(x + i)); };  // i even
  // node (lx, ly, lz) of the block dx, dy, dz below; ok: it lies in the domain
  const auto at = [&](int dx, int dy, int dz, int lx, int ly, int lz) {
    return ((uint64_t)morton3(bx - dx, by - dy, bz - dz) << 12) +
           (sp4((uint32_t)lx) | (sp4((uint32_t)ly) << 1) | (sp4((uint32_t)lz) << 2));
  };
  const bool okx = bx > 0, oky = by > 0, okz = bz > 0;
  double2 own[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {  // pair bits: y0 z0 x1 y1 z1 (lane), x2 (k) y2 z2 (warp, k), x3 (k) y3 z3 (warp)
    const uint32_t combo = 2 * warp + (k >> 2);
    const uint32_t q = lane | (k & 1) << 5 | (combo & 3u) << 6 | ((k >> 1) & 1) << 8 | (combo >> 2) << 9;
    own[k] = load2(((uint64_t)blk << 12) + 2 * q);
  }
  const int u = t & 127, xp = u & 7, yz = u >> 3;  // the low y layer (t < 128), the low z layer
  const bool on_y = t < 128;
  double2 low = make_double2(0.0, 0.0), edge = make_double2(0.0, 0.0);
  if (on_y ? oky : okz) low = load2(on_y ? at(0, 1, 0, 2 * xp, 15, yz) : at(0, 0, 1, 2 * xp, yz, 15));
  if (t < 32 && oky && okz) edge = load2(at(0, 1, 1, 2 * (t & 7), 15, 15));
  double side = 0.0, side2 = 0.0;  // the low x layer: row (t & 15, t >> 4), and its rows in the other low layers
  if (okx) side = __ldg(x + at(1, 0, 0, 15, t & 15, t >> 4));
  if (okx && t < 33) {
    if (t < 16) { if (oky) side2 = __ldg(x + at(1, 1, 0, 15, 15, t)); }
    else if (t < 32) { if (okz) side2 = __ldg(x + at(1, 0, 1, 15, t - 16, 15)); }
    else if (oky && okz) side2 = __ldg(x + at(1, 1, 1, 15, 15, 15));
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int combo = 2 * warp + c;
    const int y = (lane & 1) | ((lane >> 3) & 1) << 1 | (combo & 1) << 2 | ((combo >> 2) & 1) << 3;
    const int z = ((lane >> 1) & 1) | ((lane >> 4) & 1) << 1 | ((combo >> 1) & 1) << 2 | ((combo >> 3) & 1) << 3;
    const int m = top(ty, y) * top(tz, z), x1 = (lane >> 2) & 1;
    uint32_t bits = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int lx = 2 * x1 + 4 * (k & 1) + 8 * (k >> 1);
      bits |= bit(own[4 * c + k].x, m) << lx | bit(own[4 * c + k].y, m * top(tx, lx + 1)) << (lx + 1);
    }
    bits |= __shfl_xor_sync(0xffffffffu, bits, 4);
    if (!x1) mask[(z + 1) * MCW + y + 1] = bits << 1;
  }
  {
    const int m = on_y ? top(tz, yz) : top(ty, yz);
    uint32_t bits = bit(low.x, m) << (2 * xp) | bit(low.y, m * top(tx, 2 * xp + 1)) << (2 * xp + 1);
#pragma unroll
    for (int k = 1; k < 8; k *= 2) bits |= __shfl_xor_sync(0xffffffffu, bits, k);
    if (xp == 0) mask[on_y ? (yz + 1) * MCW : yz + 1] = bits << 1;
  }
  if (t < 32) {
    const int p = 2 * (t & 7);
    uint32_t bits = bit(edge.x, 1) << p | bit(edge.y, top(tx, p + 1)) << (p + 1);
#pragma unroll
    for (int k = 1; k < 8; k *= 2) bits |= __shfl_xor_sync(0xffffffffu, bits, k);
    if (t == 0) mask[0] = bits << 1;
  }
  xbit[((t >> 4) + 1) * MCW + (t & 15) + 1] = (uint8_t)bit(side, top(ty, t & 15) * top(tz, t >> 4));
  if (t < 16) xbit[(t + 1) * MCW] = (uint8_t)bit(side2, top(tz, t));
  else if (t < 32) xbit[t - 16 + 1] = (uint8_t)bit(side2, top(ty, t - 16));
  else if (t == 32) xbit[0] = (uint8_t)bit(side2, 1);
  __syncthreads();
  for (int r = t; r < MCW * MCW; r += blockDim.x) mask[r] |= xbit[r];
}
// Degree 2: the corner value at grid position p is the sum over the nodes p-1, p per axis of
// ((x 1/2) 1/2) 1/2, z-major, then y, then x (corner_value2).  The CTA stages the terms
// ((x 1/2) 1/2) 1/2 of nodes [-1, 16]^3 of its block (the same products, formed once per node;
// zeros outside the domain, which add +0 like the skipped terms).
constexpr int MCW2 = 18;  // node tile width, tile coordinate = node local + 1

__device__ __forceinline__ double mc_term2(double v) { return xmul(xmul(xmul(v, 0.5), 0.5), 0.5); }

// entry i of the 18^3 tile: its coordinates.  Natural order: row by row.  Morton order: the block's own
// nodes as they lie in memory, then the shell: the z faces (2 x 18 x 18), the y faces of the inner z range
// (2 x 16 x 18), the x faces of the inner y and z ranges (2 x 16 x 16)
template <bool NAT>
__device__ __forceinline__ void mc_tile2_entry(int i, int& tx, int& ty, int& tz) {
  if (NAT) {
    tx = i % MCW2;
    ty = (i / MCW2) % MCW2;
    tz = i / (MCW2 * MCW2);
  } else if (i < 4096) {
    uint32_t lx, ly, lz;
    unmorton3((uint32_t)i, lx, ly, lz);
    tx = (int)lx + 1;
    ty = (int)ly + 1;
    tz = (int)lz + 1;
  } else if (i < 4096 + 648) {
    const int r = (i - 4096) % 324;
    tz = i < 4096 + 324 ? 0 : 17;
    ty = r / 18;
    tx = r % 18;
  } else if (i < 4096 + 1224) {
    const int j = i - 4096 - 648, r = j % 288;
    ty = j < 288 ? 0 : 17;
    tz = 1 + r / 18;
    tx = r % 18;
  } else {
    const int j = i - 4096 - 1224, r = j % 256;
    tx = j < 256 ? 0 : 17;
    tz = 1 + r / 16;
    ty = 1 + r % 16;
  }
}
// Fills the tile, unless no cell can be cut: rounded addition is monotone, so where eight times the
// smallest term, added up like a corner value, is not below iso, no corner is, and likewise where eight
// times the largest is below it (both only without NaN).  Returns whether the tile is filled; all threads agree.
template <bool NAT>
__device__ bool mc_load_tile2(double* tile, const double* __restrict__ x, uint32_t blk, int res, double iso) {
  constexpr int kN = MCW2 * MCW2 * MCW2, kPer = (kN + 255) / 256;
  uint32_t bx, by, bz;
  unmorton3(blk, bx, by, bz);
  const uint32_t D = 31 - __clz(res);
  double v[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int i = threadIdx.x + 256 * k;
    int tx, ty, tz;
    mc_tile2_entry<NAT>(i, tx, ty, tz);
    const int gx = (int)bx * 16 + tx - 1, gy = (int)by * 16 + ty - 1, gz = (int)bz * 16 + tz - 1;
    v[k] = 0.0;
    if (i < kN && gx >= 0 && gy >= 0 && gz >= 0 && gx < res && gy < res && gz < res)
      v[k] = __ldg(x + node_index<NAT>((uint32_t)gx, (uint32_t)gy, (uint32_t)gz, D));
  }
  double lo = INFINITY, hi = -INFINITY;
  bool number = true;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    v[k] = mc_term2(v[k]);
    if (threadIdx.x + 256 * k < kN) {
      lo = fmin(lo, v[k]);
      hi = fmax(hi, v[k]);
      number = number && v[k] == v[k];
    }
  }
  double slo = 0.0, shi = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    slo = xadd(slo, lo);
    shi = xadd(shi, hi);
  }
  const bool above = __syncthreads_and(number && slo >= iso), below = __syncthreads_and(number && shi < iso);
  if (above || below) return false;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int i = threadIdx.x + 256 * k;
    int tx, ty, tz;
    mc_tile2_entry<NAT>(i, tx, ty, tz);
    if (i < kN) tile[NAT ? i : (tz * MCW2 + ty) * MCW2 + tx] = v[k];
  }
  return true;
}

__device__ __forceinline__ void mc_build_masks2(const double* tile, uint32_t* mask, double iso) {
  for (int r = threadIdx.x; r < MCW * MCW; r += blockDim.x) {
    const int ty = r % MCW, tz = r / MCW;
    uint32_t m = 0;
    for (int tx = 0; tx < MCW; ++tx) {
      double v = 0.0;
#pragma unroll
      for (int dz = 0; dz < 2; ++dz)
#pragma unroll
        for (int dy = 0; dy < 2; ++dy)
#pragma unroll
          for (int dx = 0; dx < 2; ++dx) v = xadd(v, tile[((tz + dz) * MCW2 + ty + dy) * MCW2 + tx + dx]);
      m |= (uint32_t)(v < iso) << tx;
    }
    mask[r] = m;
  }
}

template <int DEG>
struct McShared {
  double tile[DEG >= 2 ? MCW2 * MCW2 * MCW2 : 1];
  uint32_t mask[MCW * MCW];
  uint8_t xbit[DEG >= 2 ? 1 : MCW * MCW];
};
// fills s.mask, unless no cell of the block is cut (degree 2; false then)
template <int DEG>
__device__ __forceinline__ bool mc_block_masks(McShared<DEG>& s, const double* __restrict__ x, uint32_t blk, int res,
                                               double iso) {
  if (DEG >= 2) {
    if (!mc_load_tile2<DEG == 3>(s.tile, x, blk, res, iso)) return false;
    __syncthreads();
    mc_build_masks2(s.tile, s.mask, iso);
  } else {
    mc_masks1(s.mask, s.xbit, x, blk, res, iso);
  }
  __syncthreads();
  return true;
}

// case of local cell (lx, ly, lz) from the row masks (corner order of c_co)
__device__ __forceinline__ uint32_t mc_mask_case(const uint32_t* mask, int lx, int ly, int lz) {
  const uint32_t m00 = mask[lz * MCW + ly] >> lx, m10 = mask[lz * MCW + ly + 1] >> lx;
  const uint32_t m01 = mask[(lz + 1) * MCW + ly] >> lx, m11 = mask[(lz + 1) * MCW + ly + 1] >> lx;
  return (m00 & 1u) | ((m00 >> 1) & 1u) << 1 | ((m10 >> 1) & 1u) << 2 | (m10 & 1u) << 3 | (m01 & 1u) << 4 |
         ((m01 >> 1) & 1u) << 5 | ((m11 >> 1) & 1u) << 6 | (m11 & 1u) << 7;
}

// Reading the values bounds it: 8.6 GB at depth 10, 1.33 ms at the copy rate.  Degree 1: 1.62 ms (3.82
// through a tile in shared memory that a thread per row reads back); degree 2: 4.11 (6.66 where every
// block's corners are formed; rows of 128 bytes, and the index arithmetic of the 18^3 tile, hold it).
template <int DEG>
__global__ void __launch_bounds__(256) k_mc_block_count(const double* __restrict__ x, uint32_t D, double iso,
                                                        uint32_t* __restrict__ blockcnt) {
  __shared__ McShared<DEG> s;
  const int res = 1 << D;
  const uint32_t blk = blockIdx.x;
  int cnt = 0;
  if (mc_block_masks<DEG>(s, x, blk, res, iso)) {
    // thread = one x row of 16 cells; a cell is cut when its corners' bits differ
    const uint32_t* m = s.mask + (threadIdx.x >> 4) * MCW + (threadIdx.x & 15);
    const uint32_t any = m[0] | m[1] | m[MCW] | m[MCW + 1], all = m[0] & m[1] & m[MCW] & m[MCW + 1];
    cnt = __popc((any | any >> 1) & ~(all & all >> 1) & 0xffffu);
  }
  typedef cub::BlockReduce<int, 256> BR;
  __shared__ typename BR::TempStorage tmp;
  const int tot = BR(tmp).Sum(cnt);
  if (threadIdx.x == 0) blockcnt[blk] = (uint32_t)tot;
}

// active blocks only (list from a compaction of blockcnt > 0); cells written in Morton order, 16 to a
// thread (one scan of the block)
template <int DEG>
__global__ void __launch_bounds__(256) k_mc_block_emit(const double* __restrict__ x, uint32_t D, double iso,
                                                       const uint32_t* __restrict__ ablk,
                                                       const uint32_t* __restrict__ blockoff,
                                                       uint32_t* __restrict__ acell, uint8_t* __restrict__ acase,
                                                       uint32_t* __restrict__ nedge, uint32_t* __restrict__ ntri) {
  __shared__ McShared<DEG> s;
  const int res = 1 << D;
  const uint32_t blk = ablk[blockIdx.x];
  if (!mc_block_masks<DEG>(s, x, blk, res, iso)) return;
  typedef cub::BlockScan<int, 256> BS;
  __shared__ typename BS::TempStorage tmp;
  const uint32_t i0 = 16 * threadIdx.x;  // Morton-local cell index
  uint32_t lx, ly, lz, active = 0;
  unmorton3(i0, lx, ly, lz);
  const auto cell_of = [&](int k) {  // 4 x 2 x 2 cells
    return mc_mask_case(s.mask, (int)lx + ((k & 1) | (k >> 2 & 2)), (int)ly + (k >> 1 & 1), (int)lz + (k >> 2 & 1));
  };
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const uint32_t mc = cell_of(k);
    active |= (uint32_t)(mc != 0u && mc != 255u) << k;
  }
  int off;
  BS(tmp).ExclusiveSum(__popc(active), off);
  for (uint32_t a = blockoff[blk] + (uint32_t)off; active; active &= active - 1, ++a) {
    const int k = __ffs(active) - 1;
    const uint32_t mc = cell_of(k);
    acell[a] = (blk << 12) | (i0 + (uint32_t)k);
    acase[a] = (uint8_t)mc;
    nedge[a] = __popc(edge_mask(mc));
    ntri[a] = PR_MC_NTRI[mc];
  }
}

__global__ void k_flags_nonzero(const uint32_t* __restrict__ cnt, uint32_t n, uint32_t* __restrict__ flag) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) flag[i] = cnt[i] != 0;
}
__global__ void k_scatter_ids(const uint32_t* __restrict__ flag, const uint32_t* __restrict__ pos, uint32_t n,
                              uint32_t* __restrict__ ids) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (flag[i]) ids[pos[i]] = i;
}

// ====================================================================== host stages
void evaluate_points(pr_context* c, uint32_t D, const double* d_x64, const double* d_pts, uint64_t stride,
                     uint64_t n, double* d_out, int degree) {
  if (n == 0) return;
  if (degree == 3) k_eval_points<3><<<grid_for(n), kThreads, 0, c->stream>>>(d_x64, D, d_pts, stride, 1, n, d_out);
  else if (degree == 2) k_eval_points<2><<<grid_for(n), kThreads, 0, c->stream>>>(d_x64, D, d_pts, stride, 1, n, d_out);
  else k_eval_points<1><<<grid_for(n), kThreads, 0, c->stream>>>(d_x64, D, d_pts, stride, 1, n, d_out);
  PR_CHECK_LAUNCH();
}

double stage_iso(pr_context* c, const double* d_x64, bool natural) {
  const uint64_t P = c->P;
  int nb = (int)std::min<uint64_t>(kDotBlocks, (P + kThreads - 1) / kThreads);
  if (nb < 1) nb = 1;
  double* part = c->buf<double>("iso_part", 2 * (size_t)nb);
  double* out = c->buf<double>("iso_out", 1);
  const double* up = c->get<double>("upos");
  if (c->degree == 2 && natural) k_iso_partial<3><<<nb, kThreads, 0, c->stream>>>(d_x64, c->D, up, P, part);
  else if (c->degree == 2) k_iso_partial<2><<<nb, kThreads, 0, c->stream>>>(d_x64, c->D, up, P, part);
  else k_iso_partial<1><<<nb, kThreads, 0, c->stream>>>(d_x64, c->D, up, P, part);
  PR_CHECK_LAUNCH();
  k_iso_final<<<1, kThreads, 0, c->stream>>>(part, nb, out);
  PR_CHECK_LAUNCH();
  double sum = 0.0;
  PR_CUDA(cudaMemcpyAsync(&sum, out, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  c->sync();
  return sum / (double)P;
}

void stage_extract(pr_context* c, uint32_t D, const double* x, double iso, bool back_transform, int degree,
                   bool natural) {
  const uint64_t n = 1ull << (3 * D);
  cudaStream_t s = c->stream;
  c->nv = c->nt = 0;
  c->have_mesh = true;
  uint64_t A = 0;
  uint32_t *acell, *nedge, *ntri, *eoff, *toff;
  uint8_t* acase;
  size_t tb = 0;
  void* tmp = nullptr;
  if (D >= 4) {
    // 16^3 cell blocks: count per block, then emit the active blocks only
    const uint32_t nblk = 1u << (3 * (D - 4));
    uint32_t* blockcnt = c->buf<uint32_t>("mc_blockcnt", (size_t)nblk + 1);
    uint32_t* blockoff = c->buf<uint32_t>("mc_blockoff", (size_t)nblk + 1);
    uint32_t* flag = c->buf<uint32_t>("mc_flag", (size_t)nblk + 1);
    uint32_t* fpos = c->buf<uint32_t>("mc_fpos", (size_t)nblk + 1);
    uint32_t* ablk = c->buf<uint32_t>("mc_ablk", (size_t)nblk);
    if (degree == 2 && natural) k_mc_block_count<3><<<nblk, 256, 0, s>>>(x, D, iso, blockcnt);
    else if (degree == 2) k_mc_block_count<2><<<nblk, 256, 0, s>>>(x, D, iso, blockcnt);
    else k_mc_block_count<1><<<nblk, 256, 0, s>>>(x, D, iso, blockcnt);
    PR_CHECK_LAUNCH();
    PR_CUDA(cudaMemsetAsync(blockcnt + nblk, 0, sizeof(uint32_t), s));
    k_flags_nonzero<<<grid_for(nblk + 1), kThreads, 0, s>>>(blockcnt, nblk + 1, flag);
    PR_CHECK_LAUNCH();
    PR_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, blockcnt, blockoff, (int64_t)nblk + 1, s));
    tmp = c->buf<char>("cub_tmp", tb);
    PR_COUNT_PRIMITIVE();
    PR_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, blockcnt, blockoff, (int64_t)nblk + 1, s));
    PR_COUNT_PRIMITIVE();
    PR_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, flag, fpos, (int64_t)nblk + 1, s));
    k_scatter_ids<<<grid_for(nblk), kThreads, 0, s>>>(flag, fpos, nblk, ablk);
    PR_CHECK_LAUNCH();
    uint32_t hv[2] = {0, 0};
    PR_CUDA(cudaMemcpyAsync(&hv[0], blockoff + nblk, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    PR_CUDA(cudaMemcpyAsync(&hv[1], fpos + nblk, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    c->sync();
    A = hv[0];
    if (A == 0) return;
    acell = c->buf<uint32_t>("mc_acell", A);
    acase = c->buf<uint8_t>("mc_acase", A);
    nedge = c->buf<uint32_t>("mc_nedge", A + 1);
    ntri = c->buf<uint32_t>("mc_ntri", A + 1);
    if (degree == 2 && natural)
      k_mc_block_emit<3><<<hv[1], 256, 0, s>>>(x, D, iso, ablk, blockoff, acell, acase, nedge, ntri);
    else if (degree == 2)
      k_mc_block_emit<2><<<hv[1], 256, 0, s>>>(x, D, iso, ablk, blockoff, acell, acase, nedge, ntri);
    else k_mc_block_emit<1><<<hv[1], 256, 0, s>>>(x, D, iso, ablk, blockoff, acell, acase, nedge, ntri);
    PR_CHECK_LAUNCH();
  } else {
    const unsigned nblk = (unsigned)((n + kThreads - 1) / kThreads);
    uint32_t* blockcnt = c->buf<uint32_t>("mc_blockcnt", (size_t)nblk + 1);
    uint32_t* blockoff = c->buf<uint32_t>("mc_blockoff", (size_t)nblk + 1);
    if (degree == 2 && natural) k_mc_count<3><<<nblk, kThreads, 0, s>>>(x, D, iso, blockcnt);
    else if (degree == 2) k_mc_count<2><<<nblk, kThreads, 0, s>>>(x, D, iso, blockcnt);
    else k_mc_count<1><<<nblk, kThreads, 0, s>>>(x, D, iso, blockcnt);
    PR_CHECK_LAUNCH();
    PR_CUDA(cudaMemsetAsync(blockcnt + nblk, 0, sizeof(uint32_t), s));
    PR_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, blockcnt, blockoff, (int64_t)nblk + 1, s));
    tmp = c->buf<char>("cub_tmp", tb);
    PR_COUNT_PRIMITIVE();
    PR_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, blockcnt, blockoff, (int64_t)nblk + 1, s));
    uint32_t hA = 0;
    PR_CUDA(cudaMemcpyAsync(&hA, blockoff + nblk, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    c->sync();
    A = hA;
    if (A == 0) return;
    acell = c->buf<uint32_t>("mc_acell", A);
    acase = c->buf<uint8_t>("mc_acase", A);
    nedge = c->buf<uint32_t>("mc_nedge", A + 1);
    ntri = c->buf<uint32_t>("mc_ntri", A + 1);
    if (degree == 2 && natural) k_mc_compact<3><<<nblk, kThreads, 0, s>>>(x, D, iso, blockoff, acell, acase, nedge, ntri);
    else if (degree == 2) k_mc_compact<2><<<nblk, kThreads, 0, s>>>(x, D, iso, blockoff, acell, acase, nedge, ntri);
    else k_mc_compact<1><<<nblk, kThreads, 0, s>>>(x, D, iso, blockoff, acell, acase, nedge, ntri);
    PR_CHECK_LAUNCH();
  }
  eoff = c->buf<uint32_t>("mc_eoff", A + 1);
  toff = c->buf<uint32_t>("mc_toff", A + 1);
  PR_CUDA(cudaMemsetAsync(nedge + A, 0, sizeof(uint32_t), s));
  PR_CUDA(cudaMemsetAsync(ntri + A, 0, sizeof(uint32_t), s));
  tb = 0;
  PR_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, nedge, eoff, (int64_t)A + 1, s));
  tmp = c->buf<char>("cub_tmp", tb);
  PR_COUNT_PRIMITIVE();
  PR_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, nedge, eoff, (int64_t)A + 1, s));
  PR_COUNT_PRIMITIVE();
  PR_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, ntri, toff, (int64_t)A + 1, s));
  uint32_t hE = 0, hT = 0;
  PR_CUDA(cudaMemcpyAsync(&hE, eoff + A, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  PR_CUDA(cudaMemcpyAsync(&hT, toff + A, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  c->sync();
  const uint64_t E = hE, NT = hT;

  double* pos = c->buf<double>("mc_pos", 3 * E);
  uint64_t* k1 = c->buf<uint64_t>("mc_k1", E);
  uint32_t* k2 = c->buf<uint32_t>("mc_k2", E);
  int* err = c->buf<int>("mc_err", 1);
  PR_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
  if (degree == 2 && natural)
    k_mc_vertices<3><<<grid_for(A), kThreads, 0, s>>>(x, D, iso, acell, A, eoff, pos, k1, k2, E, err);
  else if (degree == 2)
    k_mc_vertices<2><<<grid_for(A), kThreads, 0, s>>>(x, D, iso, acell, A, eoff, pos, k1, k2, E, err);
  else k_mc_vertices<1><<<grid_for(A), kThreads, 0, s>>>(x, D, iso, acell, A, eoff, pos, k1, k2, E, err);
  PR_CHECK_LAUNCH();

  uint64_t cap = 1024;  // E < 2^32 - 1, so 2^32 entries always have room
  while (cap < 2 * E && cap < (1ull << 32)) cap *= 2;
  uint32_t* table = c->buf<uint32_t>("mc_table", cap);
  uint32_t* home = c->buf<uint32_t>("mc_home", E);
  uint32_t* first = c->buf<uint32_t>("mc_first", E + 1);
  uint32_t* vid_rep = c->buf<uint32_t>("mc_vidrep", E + 1);
  PR_CUDA(cudaMemsetAsync(table, 0xff, cap * sizeof(uint32_t), s));
  k_mc_hash<<<grid_for(E), kThreads, 0, s>>>(k1, k2, E, (uint32_t)(cap - 1), table, home);
  PR_CHECK_LAUNCH();
  k_mc_first<<<grid_for(E), kThreads, 0, s>>>(table, home, E, first);
  PR_CHECK_LAUNCH();
  PR_CUDA(cudaMemsetAsync(first + E, 0, sizeof(uint32_t), s));
  tb = 0;
  PR_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, first, vid_rep, (int64_t)E + 1, s));
  tmp = c->buf<char>("cub_tmp", tb);
  PR_COUNT_PRIMITIVE();
  PR_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, first, vid_rep, (int64_t)E + 1, s));
  uint32_t hNV = 0;
  int herr = 0;
  PR_CUDA(cudaMemcpyAsync(&hNV, vid_rep + E, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  PR_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s));
  c->sync();
  PR_REQUIRE(!herr, PR_ERR_INTERNAL, "marching cubes: vertex key outside [0, 2^30)");
  const uint64_t NV = hNV;
  double* verts = c->buf<double>("mesh_v", 3 * NV);
  uint64_t* tris = c->buf<uint64_t>("mesh_t", 3 * NT);
  Mat16 mi;
  for (int k = 0; k < 16; ++k) mi.m[k] = c->Minv[k];
  k_mc_emit_vertices<<<grid_for(E), kThreads, 0, s>>>(pos, E, first, vid_rep, back_transform ? 1 : 0, mi, verts);
  PR_CHECK_LAUNCH();
  k_mc_emit_tris<<<grid_for(A), kThreads, 0, s>>>(acase, A, eoff, toff, table, home, vid_rep, tris);
  PR_CHECK_LAUNCH();
  c->nv = NV;
  c->nt = NT;
}


}  // namespace pr
