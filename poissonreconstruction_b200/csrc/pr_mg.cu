// Block-tiled multigrid and CG kernels.
//
// Vectors live in Morton order, so a TB^3 block (TB = 8 or 16) is TB^3 consecutive
// entries: a CTA loads its block with coalesced loads, gathers the one-node halo of its
// 26 neighbour blocks, and works in shared memory.  No kernel writes a vector that it
// (or another CTA of the same launch) reads as halo: every halo-reading update writes a
// second buffer, so each launch is deterministic.
//
// Operator of level l (Galerkin, exact for the 1-D linear prolongation):
//   A_l = H (S_l (x) M_l (x) M_l + M_l (x) S_l (x) M_l + M_l (x) M_l (x) S_l) + shift I
// with H the finest spacing and 1-D matrices M_l, S_l that are tridiagonal Toeplitz except
// for the diagonal entry of node 0 (the coarse basis function at 0 is cut at the domain's
// low face: the fine grid has no node -1).  Interior nodes see the crate's constant
// stencil (src/fem_tree.rs:39-48) scaled to their level — centre, 12 edge and 8 corner
// neighbours; nodes on a low face use per-face coefficients from an 8 x 27 table.
//
// Smoother: multicolour Gauss-Seidel inside each block (8 parity colours, exact), blocks
// coupled through their halo values from before the sweep.  Forward sweeps relax colours
// 0..7 and backward sweeps 7..0, each the adjoint of the other, so the V-cycle (forward
// pre-, backward post-smoothing) is a symmetric preconditioner.  The smoother keeps its
// tile in a parity-split layout (8 sub-tiles, one per parity class), in which the nodes
// of one colour are contiguous and a warp's neighbour loads hit distinct banks.
#include <cub/cub.cuh>

#include <mutex>
#include <tuple>
#include <map>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <string>
#include <type_traits>
#include <vector>

#include "pr_mg.cuh"

namespace pr {

namespace {

template <int TB>
struct Geo {
  static constexpr int W = TB + 2;                  // tile width with a one-node halo
  static constexpr int H = W / 2;                   // parity sub-tile width
  static constexpr int H3 = H * H * H;
  static constexpr int N = TB * TB * TB;            // nodes of a block
  static constexpr int C = TB / 2;                  // colour lattice width
  static constexpr int C3 = C * C * C;
  static constexpr int LOGC = TB == 16 ? 3 : 2;
  static constexpr int THREADS = C3;                // one node per colour per thread
  static constexpr int HALO = W * W * W - N;
};

template <typename T>
struct DevCoef {
  T c0, ce, cc;       // interior: centre (+shift), edge, corner (faces are 0 in the interior)
  const T* table;     // [8 low-face masks][27 offsets], offset (dx+1) + 3(dy+1) + 9(dz+1)
  int has_faces;      // level has low-face modifications
};

// parity-split index of tile coordinate u in [0, W)^3
template <int TB>
__device__ __forceinline__ int ps_index(int ux, int uy, int uz) {
  constexpr int H = Geo<TB>::H, H3 = Geo<TB>::H3;
  const int sub = (ux & 1) | ((uy & 1) << 1) | ((uz & 1) << 2);
  return sub * H3 + ((uz >> 1) * H + (uy >> 1)) * H + (ux >> 1);
}

// h-th position of the one-node halo shell of a (TB+2)^3 tile: 6 faces, 12 edges, 8 corners
template <int TB>
__device__ __forceinline__ void halo_u(int h, int& ux, int& uy, int& uz) {
  constexpr int W = TB + 2, F = TB * TB, LT = TB == 16 ? 4 : 3;  // log2 TB
  if (h < 6 * F) {
    const int f = h >> (2 * LT), a = (h & (F - 1)) & (TB - 1), b = (h & (F - 1)) >> LT;
    const int axis = f >> 1, side = (f & 1) ? W - 1 : 0;
    if (axis == 0) { ux = side; uy = a + 1; uz = b + 1; }
    else if (axis == 1) { ux = a + 1; uy = side; uz = b + 1; }
    else { ux = a + 1; uy = b + 1; uz = side; }
    return;
  }
  h -= 6 * F;
  if (h < 12 * TB) {
    const int e = h >> LT, a = (h & (TB - 1)) + 1, axis = e >> 2;
    const int s0 = (e & 1) ? W - 1 : 0, s1 = (e & 2) ? W - 1 : 0;
    if (axis == 0) { ux = a; uy = s0; uz = s1; }
    else if (axis == 1) { ux = s0; uy = a; uz = s1; }
    else { ux = s0; uy = s1; uz = a; }
    return;
  }
  h -= 12 * TB;
  ux = (h & 1) ? W - 1 : 0;
  uy = (h & 2) ? W - 1 : 0;
  uz = (h & 4) ? W - 1 : 0;
}

template <typename T>
__device__ __forceinline__ T ldg_or0(const T* __restrict__ x, int gx, int gy, int gz, int res) {
  if (gx < 0 || gy < 0 || gz < 0 || gx >= res || gy >= res || gz >= res) return (T)0;
  return __ldg(x + morton3(gx, gy, gz));
}

// Gauss-Seidel value of one node of colour (cx, cy, cz) in a parity-split tile: `own` its sub-tile,
// pos its index there, mask its low-face mask (0: the interior row, else its row of the table).
template <typename T, int TB>
__device__ __forceinline__ T relax_colour(const T* tile, int own, int cx, int cy, int cz, int pos, int mask, T fi, T c0,
                                          T ce, T cc, const T* table) {
  constexpr int H = Geo<TB>::H, H3 = Geo<TB>::H3;
  T vals[27];
#pragma unroll
  for (int o = 0; o < 27; ++o) {
    const int dx = o % 3 - 1, dy = (o / 3) % 3 - 1, dz = o / 9 - 1;
    const int sub = own ^ ((dx != 0) | ((dy != 0) << 1) | ((dz != 0) << 2));
    const int hx = dx == 0 ? 0 : (dx < 0 ? -cx : 1 - cx);
    const int hy = dy == 0 ? 0 : (dy < 0 ? -cy : 1 - cy);
    const int hz = dz == 0 ? 0 : (dz < 0 ? -cz : 1 - cz);
    const int nzc = (dx != 0) + (dy != 0) + (dz != 0);
    // faces are only read on the (rare) low-face path
    vals[o] = (o == 13 || (nzc == 1 && mask == 0)) ? (T)0 : tile[sub * H3 + pos + (hz * H + hy) * H + hx];
  }
  T nv;
  if (mask == 0) {
    T se = 0, sc = 0;
#pragma unroll
    for (int o = 0; o < 27; ++o) {
      const int nzc = (o % 3 != 1) + ((o / 3) % 3 != 1) + (o / 9 != 1);
      if (nzc == 2) se += vals[o];
      else if (nzc == 3) sc += vals[o];
    }
    nv = (fi - ce * se - cc * sc) / c0;
  } else {
    const T* cm = table + 27 * mask;
    T off = 0;
#pragma unroll
    for (int o = 0; o < 27; ++o)
      if (o != 13) off += cm[o] * vals[o];
    nv = (fi - off) / cm[13];
  }
  return nv;
}

// P ec at fine node (gx, gy, gz) from a coarse tile of width CW whose entry 0 is coarse node (cox, coy, coz):
// even -> coarse g/2 (w 1), odd -> (g-1)/2, (g+1)/2 (w 1/2 each)
template <typename T, int CW>
__device__ __forceinline__ T prolong_node(const T* ctile, int gx, int gy, int gz, int cox, int coy, int coz) {
  const int ax = (gx >> 1) - cox, ay = (gy >> 1) - coy, az = (gz >> 1) - coz;
  const int nx = 1 + (gx & 1), ny = 1 + (gy & 1), nz = 1 + (gz & 1);
  T s = 0;
  for (int a = 0; a < nz; ++a)
    for (int b = 0; b < ny; ++b)
      for (int c = 0; c < nx; ++c) s += ctile[((az + a) * CW + (ay + b)) * CW + (ax + c)];
  const T w = (T)(((gx & 1) ? 0.5 : 1.0) * ((gy & 1) ? 0.5 : 1.0) * ((gz & 1) ? 0.5 : 1.0));
  return w * s;
}

// ------------------------------------------------------------------ smoother
// MODE 0: xo = sweep(xi); MODE 1: xo = sweep(0) (xi unused); MODE 2: xo = sweep(xi + P ec).
// DOT: part[block] = sum_i f_i xo_i over the block.
template <typename T, int TB, int MODE, bool DOT, bool FWD>
__global__ void __launch_bounds__(Geo<TB>::THREADS) k_smooth(uint32_t D, const T* __restrict__ xi, T* __restrict__ xo,
                                                           const T* __restrict__ f, const T* __restrict__ ec,
                                                           DevCoef<T> k, double* __restrict__ part) {
  using G = Geo<TB>;
  constexpr int W = G::W, H = G::H, H3 = G::H3, N = G::N, C = G::C, C3 = G::C3, LOGC = G::LOGC;
  constexpr int CW = TB / 2 + 2;  // coarse tile width (MODE 2): coarse [ox/2 - 1, ox/2 + TB/2]
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);  // W^3, parity-split
  T* fs = tile + W * W * W;                  // N, colour-major: fs[col * C3 + lattice index]
  T* ctile = fs + N;                         // CW^3 (MODE 2)
  const int res = 1 << D;
  {
    const uint64_t nl = 1ull << (3 * D);
    xi = cloud_slice(xi, nl);
    xo = cloud_slice(xo, nl);
    f = cloud_slice(f, nl);
    ec = cloud_slice(ec, nl / 8);
    part = cloud_slice(part, gridDim.x);
  }
  const uint32_t blk = blockIdx.x;
  const uint64_t base = (uint64_t)blk * N;
  uint32_t bx, by, bz;
  unmorton3(blk, bx, by, bz);
  const int ox = (int)bx * TB, oy = (int)by * TB, oz = (int)bz * TB;
  const int tid = threadIdx.x;
  const int cox = ox / 2 - 1, coy = oy / 2 - 1, coz = oz / 2 - 1;

  if (MODE == 2) {
    const int resc = res >> 1;
    for (int t = tid; t < CW * CW * CW; t += G::THREADS) {
      const int cx = cox + t % CW, cy = coy + (t / CW) % CW, cz = coz + t / (CW * CW);
      T v = 0;
      if (cx >= 0 && cx < resc && cy >= 0 && cy < resc && cz >= 0 && cz < resc) v = __ldg(ec + morton3(cx, cy, cz));
      ctile[t] = v;
    }
    __syncthreads();
  }
  auto prolong = [&](int gx, int gy, int gz) -> T { return prolong_node<T, CW>(ctile, gx, gy, gz, cox, coy, coz); };
  // interior + f
  for (int t = tid; t < N; t += G::THREADS) {
    uint32_t lx, ly, lz;
    unmorton3((uint32_t)t, lx, ly, lz);
    const int col = (lx & 1) | ((ly & 1) << 1) | ((lz & 1) << 2);
    const int lat = (lx >> 1) | ((ly >> 1) << LOGC) | ((lz >> 1) << (2 * LOGC));
    fs[col * C3 + lat] = __ldg(f + base + t);
    T v = 0;
    if (MODE != 1) v = __ldg(xi + base + t);
    if (MODE == 2) v += prolong(ox + (int)lx, oy + (int)ly, oz + (int)lz);
    tile[ps_index<TB>(lx + 1, ly + 1, lz + 1)] = v;
  }
  // halo
  for (int h = tid; h < G::HALO; h += G::THREADS) {
    int ux, uy, uz;
    halo_u<TB>(h, ux, uy, uz);
    T v = 0;
    if (MODE != 1) {
      const int gx = ox + ux - 1, gy = oy + uy - 1, gz = oz + uz - 1;
      if (gx >= 0 && gy >= 0 && gz >= 0 && gx < res && gy < res && gz < res) {
        v = __ldg(xi + morton3(gx, gy, gz));
        if (MODE == 2) v += prolong(gx, gy, gz);
      }
    }
    tile[ps_index<TB>(ux, uy, uz)] = v;
  }
  __syncthreads();

  // Gauss-Seidel over the 8 colours
  const int li = tid & (C - 1), lj = (tid >> LOGC) & (C - 1), lk = tid >> (2 * LOGC);
#pragma unroll
  for (int step = 0; step < 8; ++step) {
    const int col = FWD ? step : 7 - step;
    const int cx = col & 1, cy = (col >> 1) & 1, cz = col >> 2;
    const int own = (1 - cx) | ((1 - cy) << 1) | ((1 - cz) << 2);  // sub-tile of tile coordinate l + 1
    const int pos = ((lk + cz) * H + (lj + cy)) * H + (li + cx);
    const int self = own * H3 + pos;
    int mask = 0;
    if (k.has_faces)
      mask = ((ox == 0 && cx == 0 && li == 0) ? 1 : 0) | ((oy == 0 && cy == 0 && lj == 0) ? 2 : 0) |
             ((oz == 0 && cz == 0 && lk == 0) ? 4 : 0);
    const T nv = relax_colour<T, TB>(tile, own, cx, cy, cz, pos, mask, fs[col * C3 + tid], k.c0, k.ce, k.cc, k.table);
    tile[self] = nv;
    __syncthreads();
  }

  double acc = 0.0;
  for (int t = tid; t < N; t += G::THREADS) {
    uint32_t lx, ly, lz;
    unmorton3((uint32_t)t, lx, ly, lz);
    const T v = tile[ps_index<TB>(lx + 1, ly + 1, lz + 1)];
    xo[base + t] = v;
    if (DOT) {
      const int col = (lx & 1) | ((ly & 1) << 1) | ((lz & 1) << 2);
      const int lat = (lx >> 1) | ((ly >> 1) << LOGC) | ((lz >> 1) << (2 * LOGC));
      acc += (double)v * (double)fs[col * C3 + lat];
    }
  }
  if (DOT) {
    typedef cub::BlockReduce<double, Geo<TB>::THREADS> BR;
    __shared__ typename BR::TempStorage tmp;
    const double s = BR(tmp).Sum(acc);
    if (tid == 0) part[blk] = s;
  }
}

// ------------------------------------------------------------------ stencil rows on a natural tile
// tile index (ux,uy,uz) -> (uz*W + uy)*W + ux
template <typename T, int W>
__device__ __forceinline__ T row_general(const T* __restrict__ s, int idx, const T* __restrict__ cm) {
  T r = 0;
#pragma unroll
  for (int o = 0; o < 27; ++o) {
    const int dx = o % 3 - 1, dy = (o / 3) % 3 - 1, dz = o / 9 - 1;
    r += cm[o] * s[idx + dx + W * dy + W * W * dz];
  }
  return r;
}

template <typename T, int W>
__device__ __forceinline__ T row_interior(const T* __restrict__ s, int idx, T c0, T ce, T cc) {
  T se = 0, sc = 0;
#pragma unroll
  for (int o = 0; o < 27; ++o) {
    const int dx = o % 3 - 1, dy = (o / 3) % 3 - 1, dz = o / 9 - 1;
    const int nzc = (dx != 0) + (dy != 0) + (dz != 0);
    if (nzc == 2) se += s[idx + dx + W * dy + W * W * dz];
    else if (nzc == 3) sc += s[idx + dx + W * dy + W * W * dz];
  }
  return c0 * s[idx] + ce * se + cc * sc;
}

// Column sweep along z: for the column (ux,uy) of a natural tile, output A x at tile
// z coordinates uz0..uz0+ZL-1 through fn(k, centre value, row value).  Plane partial sums
// are shared by the three outputs that use them.
template <typename T, int W, int ZL, typename Fn>
__device__ __forceinline__ void column_apply(const T* __restrict__ s, int ux, int uy, int uz0, T c0, T ce, T cc,
                                             Fn fn) {
  auto plane = [&](int uz, T& pc, T& pf, T& pe) {
    const int b = (uz * W + uy) * W + ux;
    pc = s[b];
    pf = s[b - 1] + s[b + 1] + s[b - W] + s[b + W];
    pe = s[b - 1 - W] + s[b + 1 - W] + s[b - 1 + W] + s[b + 1 + W];
  };
  T pcm, pfm, pem, pc0, pf0, pe0;
  plane(uz0 - 1, pcm, pfm, pem);
  plane(uz0, pc0, pf0, pe0);
#pragma unroll
  for (int k = 0; k < ZL; ++k) {
    T pcp, pfp, pep;
    plane(uz0 + k + 1, pcp, pfp, pep);
    fn(k, pc0, c0 * pc0 + ce * (pe0 + pfm + pfp) + cc * (pem + pep));
    pcm = pc0;
    pfm = pf0;
    pem = pe0;
    pc0 = pcp;
    pf0 = pfp;
    pe0 = pep;
  }
  (void)pcm;
}

// ------------------------------------------------------------------ fine-level SpMV
// XPBY: dn = z + beta d (tile and halo), dn written; q = A dn (stencil part); part = dn.q
template <typename T, int TB, bool XPBY>
__global__ void __launch_bounds__(Geo<TB>::THREADS) k_spmv(uint32_t D, const T* __restrict__ z,
                                                         const T* __restrict__ d, T* __restrict__ dn, T beta,
                                                         T* __restrict__ q, DevCoef<T> k, double* __restrict__ part) {
  using G = Geo<TB>;
  constexpr int W = G::W, N = G::N;
  constexpr int SEG = G::THREADS / (TB * TB);  // z segments per column
  constexpr int ZL = TB / SEG;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);  // W^3 natural
  T* out = tile + W * W * W;                 // N, Morton-local
  const int res = 1 << D;
  {
    const uint64_t nl = 1ull << (3 * D);
    z = cloud_slice(z, nl);
    d = cloud_slice(d, nl);
    dn = cloud_slice(dn, nl);
    q = cloud_slice(q, nl);
    part = cloud_slice(part, gridDim.x);
  }
  const uint32_t blk = blockIdx.x;
  const uint64_t base = (uint64_t)blk * N;
  uint32_t bx, by, bz;
  unmorton3(blk, bx, by, bz);
  const int ox = (int)bx * TB, oy = (int)by * TB, oz = (int)bz * TB;
  const int tid = threadIdx.x;
  for (int t = tid; t < N; t += G::THREADS) {
    uint32_t lx, ly, lz;
    unmorton3((uint32_t)t, lx, ly, lz);
    T v = __ldg(d + base + t);
    if (XPBY) {
      v = __ldg(z + base + t) + beta * v;
      out[t] = v;  // staged dn for the coalesced store below
    }
    tile[((lz + 1) * W + (ly + 1)) * W + (lx + 1)] = v;
  }
  for (int h = tid; h < G::HALO; h += G::THREADS) {
    int ux, uy, uz;
    halo_u<TB>(h, ux, uy, uz);
    const int gx = ox + ux - 1, gy = oy + uy - 1, gz = oz + uz - 1;
    T v = 0;
    if (gx >= 0 && gy >= 0 && gz >= 0 && gx < res && gy < res && gz < res) {
      const uint32_t m = morton3(gx, gy, gz);
      v = __ldg(d + m);
      if (XPBY) v = __ldg(z + m) + beta * v;
    }
    tile[(uz * W + uy) * W + ux] = v;
  }
  __syncthreads();
  if (XPBY) {
    for (int t = tid; t < N; t += G::THREADS) dn[base + t] = out[t];
    __syncthreads();
  }
  const int col = tid % (TB * TB), seg = tid / (TB * TB);
  const int ux = col % TB + 1, uy = col / TB + 1;
  double acc = 0.0;
  column_apply<T, W, ZL>(tile, ux, uy, seg * ZL + 1, k.c0, k.ce, k.cc, [&](int kk, T dv, T y) {
    const int lz = seg * ZL + kk;
    out[morton3(ux - 1, uy - 1, lz)] = y;
    acc += (double)dv * (double)y;
  });
  __syncthreads();
  for (int t = tid; t < N; t += G::THREADS) q[base + t] = out[t];
  typedef cub::BlockReduce<double, Geo<TB>::THREADS> BR;
  __shared__ typename BR::TempStorage tmp;
  const double s = BR(tmp).Sum(acc);
  if (tid == 0) part[blk] = s;
}

// restriction to coarse node (cx, cy, cz) of the block from a WR^3 residual tile whose entry 0 is the
// fine node -1 per axis
template <typename T, int WR>
__device__ __forceinline__ T restrict_full(const T* rt, int cx, int cy, int cz) {
  const int fx = 2 * cx + 1, fy = 2 * cy + 1, fz = 2 * cz + 1;  // tile coordinate of the fine centre
  T s = 0;
#pragma unroll
  for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
      for (int dx = -1; dx <= 1; ++dx) {
        const T w = (T)((dx ? 0.5 : 1.0) * (dy ? 0.5 : 1.0) * (dz ? 0.5 : 1.0));
        s += w * rt[((fz + dz) * WR + (fy + dy)) * WR + (fx + dx)];
      }
  return s;
}

// ------------------------------------------------------------------ residual + restriction
// fc = P^T (f - A e) for the (TB/2)^3 coarse nodes whose fine centre lies in the block.
// r is needed on local [-1, TB-1]^3: the block interior (z columns) plus its low shell.
template <typename T, int TB>
__global__ void __launch_bounds__(Geo<TB>::THREADS) k_resid_restrict(uint32_t D, const T* __restrict__ e,
                                                                   const T* __restrict__ f, T* __restrict__ fc,
                                                                   DevCoef<T> k) {
  using G = Geo<TB>;
  constexpr int N = G::N;
  constexpr int WE = TB + 3;  // e over local [-2, TB]
  constexpr int WR = TB + 1;  // r over local [-1, TB-1]
  constexpr int TC = TB / 2;
  constexpr int SEG = G::THREADS / (TB * TB);
  constexpr int ZL = TB / SEG;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* et = reinterpret_cast<T*>(smem_raw);  // WE^3 natural, tile coordinate = local + 2
  T* rt = et + WE * WE * WE;               // WR^3 natural, coordinate = local + 1
  const int res = 1 << D;
  {
    const uint64_t nl = 1ull << (3 * D);
    e = cloud_slice(e, nl);
    f = cloud_slice(f, nl);
    fc = cloud_slice(fc, nl / 8);
  }
  const uint32_t blk = blockIdx.x;
  const uint64_t base = (uint64_t)blk * N;
  uint32_t bx, by, bz;
  unmorton3(blk, bx, by, bz);
  const int ox = (int)bx * TB, oy = (int)by * TB, oz = (int)bz * TB;
  const int tid = threadIdx.x;
  for (int t = tid; t < N; t += G::THREADS) {
    uint32_t lx, ly, lz;
    unmorton3((uint32_t)t, lx, ly, lz);
    et[((lz + 2) * WE + (ly + 2)) * WE + (lx + 2)] = __ldg(e + base + t);
    rt[((lz + 1) * WR + (ly + 1)) * WR + (lx + 1)] = __ldg(f + base + t);  // f first, r = f - A e below
  }
  for (int t = tid; t < WE * WE * WE; t += G::THREADS) {
    const int tx = t % WE, ty = (t / WE) % WE, tz = t / (WE * WE);
    if (tx >= 2 && tx < TB + 2 && ty >= 2 && ty < TB + 2 && tz >= 2 && tz < TB + 2) continue;
    et[t] = ldg_or0(e, ox + tx - 2, oy + ty - 2, oz + tz - 2, res);
  }
  __syncthreads();
  // interior: z columns with the interior rows
  {
    const int col = tid % (TB * TB), seg = tid / (TB * TB);
    const int lx = col % TB, ly = col / TB;
    column_apply<T, WE, ZL>(et, lx + 2, ly + 2, seg * ZL + 2, k.c0, k.ce, k.cc, [&](int kk, T, T y) {
      const int lz = seg * ZL + kk;
      rt[((lz + 1) * WR + (ly + 1)) * WR + (lx + 1)] -= y;
    });
  }
  // low shell of r: local coordinate -1 on at least one axis
  {
    constexpr int S1 = WR * WR, S2 = TB * WR, S3 = TB * TB;
    for (int t = tid; t < S1 + S2 + S3; t += G::THREADS) {
      int lx, ly, lz;
      if (t < S1) { lx = -1; ly = t % WR - 1; lz = t / WR - 1; }
      else if (t < S1 + S2) { const int u = t - S1; lx = u % TB; ly = -1; lz = u / TB - 1; }
      else { const int u = t - S1 - S2; lx = u % TB; ly = u / TB; lz = -1; }
      const int gx = ox + lx, gy = oy + ly, gz = oz + lz;
      T r = 0;
      if (gx >= 0 && gy >= 0 && gz >= 0) {
        const int ei = ((lz + 2) * WE + (ly + 2)) * WE + (lx + 2);
        const int mask = k.has_faces ? ((gx == 0) | ((gy == 0) << 1) | ((gz == 0) << 2)) : 0;
        const T y = mask ? row_general<T, WE>(et, ei, k.table + 27 * mask) : row_interior<T, WE>(et, ei, k.c0, k.ce, k.cc);
        r = __ldg(f + morton3(gx, gy, gz)) - y;
      }
      rt[((lz + 1) * WR + (ly + 1)) * WR + (lx + 1)] = r;
    }
  }
  __syncthreads();
  if (k.has_faces && (ox == 0 || oy == 0 || oz == 0)) {
    // interior nodes on a low domain face: replace the interior row by the face row
    for (int t = tid; t < N; t += G::THREADS) {
      uint32_t lx, ly, lz;
      unmorton3((uint32_t)t, lx, ly, lz);
      const int gx = ox + lx, gy = oy + ly, gz = oz + lz;
      const int mask = (gx == 0) | ((gy == 0) << 1) | ((gz == 0) << 2);
      if (!mask) continue;
      const int ei = ((lz + 2) * WE + (ly + 2)) * WE + (lx + 2);
      const T yi = row_interior<T, WE>(et, ei, k.c0, k.ce, k.cc);
      const T yf = row_general<T, WE>(et, ei, k.table + 27 * mask);
      rt[((lz + 1) * WR + (ly + 1)) * WR + (lx + 1)] += yi - yf;
    }
    __syncthreads();
  }
  const uint64_t cbase = (uint64_t)blk * (TC * TC * TC);
  for (int t = tid; t < TC * TC * TC; t += G::THREADS) {
    uint32_t cx, cy, cz;
    unmorton3((uint32_t)t, cx, cy, cz);
    fc[cbase + t] = restrict_full<T, WR>(rt, (int)cx, (int)cy, (int)cz);
  }
}

// fixed-order sum of two partial arrays by 1024 threads: sum(part) + scale2 * sum(part2), in thread 0
__device__ __forceinline__ double sum_parts_block(const double* __restrict__ part, int np, double scale2,
                                                  const double* __restrict__ part2, int np2) {
  part += (uint64_t)blockIdx.x * np;  // block k: cloud k's partials (packed launches)
  part2 += (uint64_t)blockIdx.x * np2;
  double s = 0.0, s2 = 0.0;
  for (int i = threadIdx.x; i < np; i += 1024) s += part[i];
  for (int i = threadIdx.x; i < np2; i += 1024) s2 += part2[i];
  typedef cub::BlockReduce<double, 1024> BR;
  __shared__ typename BR::TempStorage tmp;
  const double a = BR(tmp).Sum(s);
  __syncthreads();
  const double b = BR(tmp).Sum(s2);
  return a + scale2 * b;
}
__global__ void __launch_bounds__(1024) k_sum_parts(const double* __restrict__ part, int np, double scale2,
                                                    const double* __restrict__ part2, int np2,
                                                    double* __restrict__ out) {
  const double v = sum_parts_block(part, np, scale2, part2, np2);
  if (threadIdx.x == 0) out[blockIdx.x] = v;
}
__global__ void __launch_bounds__(1024) k_cg_step(int step, const double* __restrict__ part, int np, double scale2,
                                                  const double* __restrict__ part2, int np2, CgScalars cg) {
  const double v = sum_parts_block(part, np, scale2, part2, np2);
  if (threadIdx.x != 0) return;
  const int k = blockIdx.x;
  const bool act = cg.act[k] != 0;
  if (step == kCgRz0) {
    cg.rz[k] = v;
  } else if (step == kCgRz) {
    cg.beta[k] = act ? v / cg.rz[k] : 0.0;
    if (act) cg.rz[k] = v;
  } else if (step == kCgDq) {
    const bool ok = act && v > 0.0 && isfinite(v) && cg.rz[k] > 0.0;
    cg.alpha[k] = ok ? cg.rz[k] / v : 0.0;
    if (act && !ok) {
      cg.broke[k] = 1;
      cg.act[k] = 0;
    }
  } else if (act) {
    const int it = cg.iters[k] + 1;
    cg.iters[k] = it;
    cg.rr[k] = v;
    if (!isfinite(v)) {
      cg.broke[k] = 1;
      cg.act[k] = 0;
    } else if (__dsqrt_rn(v) <= cg.tol[k] || it >= cg.maxit[k]) {
      cg.act[k] = 0;
    }
  }
}

// ------------------------------------------------------------------ helpers of the 16^3 block kernels
namespace s16 {
// spread the 4 low bits of v to bit positions 0,3,6,9
__device__ __forceinline__ uint32_t sp4(uint32_t v) {
  return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4) | ((v & 8u) << 6);
}
// spread the 3 low bits of v to bit positions 0,2,4
__device__ __forceinline__ uint32_t sp2(uint32_t v) { return (v & 1u) | ((v & 2u) << 1) | ((v & 4u) << 2); }
template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
  typedef float4 type;
};
template <>
struct Vec4<double> {
  typedef double4 type;
};

__device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ double4 ld4(const double* p) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(p)), b = __ldg(reinterpret_cast<const double2*>(p) + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void st4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void st4(double* p, const double4& v) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v.x, v.y);
  reinterpret_cast<double2*>(p)[1] = make_double2(v.z, v.w);
}

__device__ __forceinline__ void neighbour_bases(uint32_t* nb, uint32_t bx, uint32_t by, uint32_t bz, int nblk_axis) {
  const int t = threadIdx.x;
  if (t < 27) {
    const int dx = t % 3 - 1, dy = (t / 3) % 3 - 1, dz = t / 9 - 1;
    const int x = (int)bx + dx, y = (int)by + dy, z = (int)bz + dz;
    nb[t] = (x < 0 || y < 0 || z < 0 || x >= nblk_axis || y >= nblk_axis || z >= nblk_axis)
                ? ~0u
                : (morton3((uint32_t)x, (uint32_t)y, (uint32_t)z) << 12);
  }
}

}  // namespace s16

// ------------------------------------------------------------------ 16^3 stencil rows
namespace n16 {
// in-plane sums of the quad's 4 nodes: tz = ce*faces + cc*diagonals (for the rows z-1, z+1),
// own = c0*centre + ce*diagonals (for row z)
template <typename T>
__device__ __forceinline__ void plane_terms(const T r[4][4], T c0, T ce, T cc, T tz[4], T own[4], T ctr[4]) {
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int e = 2 * j + i, R = j + 1, Cc = i + 1;
      const T pf = r[R][Cc - 1] + r[R][Cc + 1] + r[R - 1][Cc] + r[R + 1][Cc];
      const T pe = r[R - 1][Cc - 1] + r[R - 1][Cc + 1] + r[R + 1][Cc - 1] + r[R + 1][Cc + 1];
      tz[e] = ce * pf + cc * pe;
      own[e] = c0 * r[R][Cc] + ce * pe;
      ctr[e] = r[R][Cc];
    }
}

// in-plane sums of the quad's 4 nodes by themselves: the 4 face neighbours and the 4 diagonal ones
template <typename T>
__device__ __forceinline__ void plane_sums(const T r[4][4], T f[4], T d[4], T ctr[4]) {
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int e = 2 * j + i, R = j + 1, Cc = i + 1;
      f[e] = (r[R][Cc - 1] + r[R][Cc + 1]) + (r[R - 1][Cc] + r[R + 1][Cc]);
      d[e] = (r[R - 1][Cc - 1] + r[R - 1][Cc + 1]) + (r[R + 1][Cc - 1] + r[R + 1][Cc + 1]);
      ctr[e] = r[R][Cc];
    }
}

}  // namespace n16

// ------------------------------------------------------------------ the z-run tile of the 16^3 block kernels
// A 16^3 block with its one-node halo.  Column (x, y), x and y in -1..16, holds its 8 even planes, then
// its 8 odd ones, in consecutive words; the halo planes z = -1 and 16 are two small planes of their own.
// Thread = one 2x2 (x, y) quad column over ZT planes of one parity (ZT = 2 or 4), one 8- or 16-byte
// access of a column; the 16 / ZT segments of a quad column sit on neighbouring lanes, and the in-plane
// sums of the planes below and above come from those lanes by shuffle: only the block's first and last
// plane read the halo planes.  The parity is the lowest lane bit and the quads follow in Morton order, so
// that for each of its planes a warp loads (and stores) whole 128-byte lines, four 16-byte quads of two
// planes each.  (Segments of consecutive planes touched four times the lines, a quarter of each, and the
// L1's look-ups bounded the kernel; one 32-byte load per lane and two planes, one sector a cycle, too.)
// Bank conflicts: eight lanes of a 16-byte column access (ZT = 4: four segments of two quads 48 words
// apart) fill the 32 banks once; the halo planes' rows are 20 words and the planes 368 words apart, which
// puts the 16 lanes of a halo access on the 16 even banks.
// What bounds the kernels is the L1's data pipe (84% busy in the post-smoothing sweep: its own columns,
// 5 neighbouring ones per phase, shuffles, and the halo's sectors).  At depth 9 in FP32, in us, with the
// floor by HBM bytes and the time on a plane-by-plane tile with one quad per lane and plane:
//   post-smoothing 537 (floor 260; 753 plane by plane), CG update and pre-smoothing 556 (583; 750),
//   residual and restriction 482 (177; 560), first sweep 184 (167; 277), plain SpMV 311 (167; 338),
//   with d = z + beta d 462 (333; 454).
// Every value and every sum is the same for every ZT.
namespace z16 {
constexpr int kCS = 24, kRY = 18 * kCS + 4, kHR = 20, kHP = 368, TILE = 18 * kRY + 2 * kHP;
// word of column (x, y); of plane z in it
__device__ __forceinline__ int at(int x, int y) { return (y + 1) * kRY + (x + 1) * kCS; }
__device__ __forceinline__ int zw(int z) { return ((z & 1) << 3) | (z >> 1); }
// word of (x, y) on the halo plane z = -1 (hi 0) or 16 (hi 1)
__device__ __forceinline__ int halo_at(int hi, int x, int y) { return 18 * kRY + hi * kHP + (y + 1) * kHR + x + 1; }
// node (x, y) of plane z, -1..16, with its strides in x and y
template <typename T>
struct PlaneRef {
  const T* p;
  int sx, sy;
  __device__ __forceinline__ T operator()(int dx, int dy) const { return p[dx * sx + dy * sy]; }
};
template <typename T>
__device__ __forceinline__ PlaneRef<T> plane_ref(const T* tile, int x, int y, int z) {
  if (z < 0 || z > 15) return {tile + halo_at(z > 15, x, y), 1, kHR};
  return {tile + at(x, y) + zw(z), kCS, kRY};
}
// quad coordinates of quad qm (Morton order)
__device__ __forceinline__ void quad_of(int qm, int& qx, int& qy) {
  qx = (qm & 1) | ((qm >> 1) & 2) | ((qm >> 2) & 4);
  qy = ((qm >> 1) & 1) | ((qm >> 2) & 2) | ((qm >> 3) & 4);
}
template <typename T>
__device__ __forceinline__ void ld4q(const T* p, T (&o)[4]) {
  const typename s16::Vec4<T>::type v = s16::ld4(p);
  o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
template <typename T>
__device__ __forceinline__ void st4q(T* p, const T (&o)[4]) {
  typename s16::Vec4<T>::type v;
  v.x = o[0]; v.y = o[1]; v.z = o[2]; v.w = o[3];
  s16::st4(p, v);
}
template <int ZT>
struct Zt {
  static constexpr int SEG = 16 / ZT;       // z segments of a column
  static constexpr int NT = 64 * SEG;       // threads
  static constexpr int NSIDE = 36 * SEG;    // halo quad columns beside the block, a segment per thread
  static constexpr int NZF = NT - NSIDE;    // the other threads take the 2 x 100 quads of the z halo planes
  static constexpr int ZN = (200 + NZF - 1) / NZF;
  static constexpr int HV = ZT > ZN ? ZT : ZN;
};
// a segment: its parity, first plane, first word in a column, and place among the column's segments
template <int ZT>
struct Seg {
  int p, z0, w0, s;
  __device__ __forceinline__ explicit Seg(int lane) {
    s = lane % Zt<ZT>::SEG;
    p = s & 1;
    z0 = 2 * ZT * (s >> 1) + p;
    w0 = 8 * p + ZT * (s >> 1);
  }
  __device__ __forceinline__ int z(int k) const { return z0 + 2 * k; }
  __device__ __forceinline__ bool first() const { return s == 0; }                // holds plane 0 (k = 0)
  __device__ __forceinline__ bool last() const { return s == Zt<ZT>::SEG - 1; }  // holds plane 15 (k = ZT - 1)
};
// Values of the planes next to the segment's: y[k] those of plane z(k) + 1 (parity 0) or - 1 (parity 1),
// o[k] those of the other side; end: what lies beyond the block for its first and last plane.  Every lane
// of the warp takes part.
template <int ZT, typename T>
__device__ __forceinline__ void beside(const Seg<ZT>& g, const T (&x)[ZT], T end, T (&y)[ZT], T (&o)[ZT]) {
#pragma unroll
  for (int k = 0; k < ZT; ++k) y[k] = __shfl_xor_sync(0xffffffffu, x[k], 1);
  const int lane = threadIdx.x & 31;
  T w = __shfl_sync(0xffffffffu, g.p ? x[ZT - 1] : x[0], g.p ? lane + 1 : lane - 1);
  if (g.first() || g.last()) w = end;
#pragma unroll
  for (int k = 0; k < ZT; ++k) o[k] = g.p ? (k < ZT - 1 ? y[k < ZT - 1 ? k + 1 : k] : w) : (k > 0 ? y[k > 0 ? k - 1 : 0] : w);
}
template <int ZT>
__device__ __forceinline__ void ldz(const float* p, float (&o)[ZT]) {
  if constexpr (ZT == 2) {
    const float2 a = *reinterpret_cast<const float2*>(p);
    o[0] = a.x; o[1] = a.y;
  } else {
#pragma unroll
    for (int k = 0; k < ZT; k += 4) {
      const float4 a = *reinterpret_cast<const float4*>(p + k);
      o[k] = a.x; o[k + 1] = a.y; o[k + 2] = a.z; o[k + 3] = a.w;
    }
  }
}
template <int ZT>
__device__ __forceinline__ void ldz(const double* p, double (&o)[ZT]) {
#pragma unroll
  for (int k = 0; k < ZT; k += 2) {
    const double2 a = *reinterpret_cast<const double2*>(p + k);
    o[k] = a.x; o[k + 1] = a.y;
  }
}
template <int ZT>
__device__ __forceinline__ void stz(float* p, const float (&o)[ZT]) {
  if constexpr (ZT == 2) {
    *reinterpret_cast<float2*>(p) = make_float2(o[0], o[1]);
  } else {
#pragma unroll
    for (int k = 0; k < ZT; k += 4) *reinterpret_cast<float4*>(p + k) = make_float4(o[k], o[k + 1], o[k + 2], o[k + 3]);
  }
}
template <int ZT>
__device__ __forceinline__ void stz(double* p, const double (&o)[ZT]) {
#pragma unroll
  for (int k = 0; k < ZT; k += 2) *reinterpret_cast<double2*>(p + k) = make_double2(o[k], o[k + 1]);
}
// the quad's four columns of ZT planes
template <int ZT, typename T>
__device__ __forceinline__ void store_quad(T* tile, int x0, int y0, const Seg<ZT>& g, const T (&v)[ZT][4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    T c[ZT];
#pragma unroll
    for (int k = 0; k < ZT; ++k) c[k] = v[k][e];
    stz<ZT>(tile + at(x0 + (e & 1), y0 + (e >> 1)) + g.w0, c);
  }
}
// The coarse tile of the prolongation: coarse nodes -1..8 per axis, plane cz of column (cx, cy) at word
// cz + 4 of its kCC.  (Quads beside the block's last column read a column past it.)
constexpr int kCC = 20, kCX = 11, kCTile = kCX * kCX * kCC;
__device__ __forceinline__ int coarse_at(int cx, int cy) { return ((cy + 1) * kCX + cx + 1) * kCC + 4; }
// P ec on quad (qx, qy) (block-local, -1..8) from its four coarse columns on one coarse plane
template <typename T>
__device__ __forceinline__ void prolong_plane(T c00, T c10, T c01, T c11, T (&pl)[4]) {
  pl[0] = c00;
  pl[1] = (T)0.5 * (c00 + c10);
  pl[2] = (T)0.5 * (c00 + c01);
  pl[3] = (T)0.25 * ((c00 + c10) + (c01 + c11));
}
// v += P ec on the quad's segment (even planes lie on a coarse plane, odd ones halfway between two)
template <int ZT, typename T, int M>
__device__ __forceinline__ void prolong_quads(const T* ctile, int qx, int qy, const Seg<ZT>& g, T (&v)[M][4]) {
  const T* c = ctile + coarse_at(qx, qy) + (g.z0 >> 1);
  T q[4][ZT + 1];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    T a[ZT];
    const T* ci = c + (i & 1) * kCC + (i >> 1) * kCX * kCC;
    ldz<ZT>(ci, a);
#pragma unroll
    for (int k = 0; k < ZT; ++k) q[i][k] = a[k];
    q[i][ZT] = ci[ZT];
  }
  T lo[4], hi[4];
  prolong_plane<T>(q[0][0], q[1][0], q[2][0], q[3][0], lo);
#pragma unroll
  for (int k = 0; k < ZT; ++k) {
    prolong_plane<T>(q[0][k + 1], q[1][k + 1], q[2][k + 1], q[3][k + 1], hi);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[k][e] += g.p ? (T)0.5 * (lo[e] + hi[e]) : lo[e];
      lo[e] = hi[e];
    }
  }
}

// The halo in two steps, so that its loads are in flight with the block's own: halo quad columns beside
// the block (threads 0 .. NSIDE - 1) and the quads of the planes z = -1 and 16 (the others).
// quad(m, o): the four values of the quad at Morton index m of the vector.
__device__ __forceinline__ void side_quad(int h, int& qx, int& qy) {
  if (h < 20) {
    qy = h < 10 ? -1 : 8;
    qx = (h < 10 ? h : h - 10) - 1;
  } else {
    qy = (h - 20) >> 1;
    qx = (h & 1) ? 8 : -1;
  }
}
__device__ __forceinline__ void face_quad(int i, int& qx, int& qy) {  // the 64 of the block first
  if (i < 64) quad_of(i, qx, qy);
  else side_quad(i - 64, qx, qy);
}
__device__ __forceinline__ int side_of(int q) { return q < 0 ? -1 : (q > 7 ? 1 : 0); }
template <int ZT, typename T, typename Quad>
__device__ __forceinline__ void load_halo(const uint32_t* nb, Quad quad, T (&hv)[Zt<ZT>::HV][4]) {
  typedef Zt<ZT> Z;
  const int t = threadIdx.x;
  if (t < Z::NSIDE) {
    int qx, qy;
    side_quad(t / Z::SEG, qx, qy);
    const Seg<ZT> g(t);
    const uint32_t base = nb[13 + side_of(qx) + 3 * side_of(qy)];
    const uint32_t mq = s16::sp4(2 * (qx & 7)) | (s16::sp4(2 * (qy & 7)) << 1);
#pragma unroll
    for (int k = 0; k < ZT; ++k) {
      hv[k][0] = hv[k][1] = hv[k][2] = hv[k][3] = (T)0;
      if (base != ~0u) quad(base + (mq | (s16::sp4(g.z(k)) << 2)), hv[k]);
    }
  } else {
#pragma unroll
    for (int j = 0; j < Z::ZN; ++j) {
      const int i = t - Z::NSIDE + Z::NZF * j;
      if (i >= 200) break;
      const int hi = i >= 100;
      int qx, qy;
      face_quad(i - 100 * hi, qx, qy);
      const uint32_t base = nb[13 + side_of(qx) + 3 * side_of(qy) + (hi ? 9 : -9)];
      const uint32_t m = s16::sp4(2 * (qx & 7)) | (s16::sp4(2 * (qy & 7)) << 1) | (hi ? 0u : 0x249u << 2);
      hv[j][0] = hv[j][1] = hv[j][2] = hv[j][3] = (T)0;
      if (base != ~0u) quad(base + m, hv[j]);
    }
  }
}
// ctile (nullable): the coarse tile whose prolongation is added at nodes inside the domain
template <int ZT, bool PROLONG, typename T>
__device__ __forceinline__ void store_halo(T* tile, const uint32_t* nb, const T* ctile, T (&hv)[Zt<ZT>::HV][4]) {
  typedef Zt<ZT> Z;
  const int t = threadIdx.x;
  if (t < Z::NSIDE) {
    int qx, qy;
    side_quad(t / Z::SEG, qx, qy);
    const Seg<ZT> g(t);
    if (PROLONG && nb[13 + side_of(qx) + 3 * side_of(qy)] != ~0u) prolong_quads<ZT>(ctile, qx, qy, g, hv);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int x = 2 * qx + (e & 1), y = 2 * qy + (e >> 1);
      if (x < -1 || x > 16 || y < -1 || y > 16) continue;
      T c[ZT];
#pragma unroll
      for (int k = 0; k < ZT; ++k) c[k] = hv[k][e];
      stz<ZT>(tile + at(x, y) + g.w0, c);
    }
  } else {
#pragma unroll
    for (int j = 0; j < Z::ZN; ++j) {
      const int i = t - Z::NSIDE + Z::NZF * j;
      if (i >= 200) break;
      const int hi = i >= 100;
      int qx, qy;
      face_quad(i - 100 * hi, qx, qy);
      if (PROLONG && nb[13 + side_of(qx) + 3 * side_of(qy) + (hi ? 9 : -9)] != ~0u) {
        const T* c = ctile + coarse_at(qx, qy) + (hi ? 8 : -1);
        T lo[4], up[4];
        prolong_plane<T>(c[0], c[kCC], c[kCX * kCC], c[kCX * kCC + kCC], lo);
        if (!hi) prolong_plane<T>(c[1], c[kCC + 1], c[kCX * kCC + 1], c[kCX * kCC + kCC + 1], up);
#pragma unroll
        for (int e = 0; e < 4; ++e) hv[j][e] += hi ? lo[e] : (T)0.5 * (lo[e] + up[e]);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int x = 2 * qx + (e & 1), y = 2 * qy + (e >> 1);
        if (x >= -1 && x <= 16 && y >= -1 && y <= 16) tile[halo_at(hi, x, y)] = hv[j][e];
      }
    }
  }
}
// a zero halo (a sweep from zero reads no halo plane, only the columns beside the block)
template <int ZT, typename T>
__device__ __forceinline__ void zero_side_halo(T* tile) {
  const T zero[ZT] = {};
  for (int i = threadIdx.x; i < 68 * Zt<ZT>::SEG; i += Zt<ZT>::NT) {
    const int h = i / Zt<ZT>::SEG, z0 = ZT * (i % Zt<ZT>::SEG);  // (words)
    const int x = h < 36 ? (h < 18 ? h : h - 18) - 1 : ((h & 1) ? 16 : -1);
    const int y = h < 36 ? (h < 18 ? -1 : 16) : (h - 36) >> 1;
    stz<ZT>(tile + at(x, y) + z0, zero);
  }
}

// loads the coarse tile by quads: the block's 128 coarse ones in memory order, then the 232 around them
template <int NT, typename T>
__device__ __forceinline__ void load_coarse_tile(T* ctile, const T* __restrict__ ec, const uint32_t* nb) {
  for (int i = threadIdx.x; i < 360; i += NT) {
    int qx, qy, cz;
    if (i < 128) {
      qx = ((i >> 1) & 1) | ((i >> 3) & 2);
      qy = ((i >> 2) & 1) | ((i >> 4) & 2);
      cz = (i & 1) | ((i >> 2) & 2) | ((i >> 4) & 4);
    } else if (i < 200) {  // the planes below and above
      const int r = (i - 128) % 36;
      qx = r % 6 - 1;
      qy = r / 6 - 1;
      cz = i < 164 ? -1 : 8;
    } else {  // beside the block
      const int r = (i - 200) % 20;
      cz = (i - 200) / 20;
      if (r < 12) {
        qx = r % 6 - 1;
        qy = r < 6 ? -1 : 4;
      } else {
        qx = (r & 1) ? 4 : -1;
        qy = (r - 12) >> 1;
      }
    }
    const int dx = qx < 0 ? -1 : (qx > 3 ? 1 : 0), dy = qy < 0 ? -1 : (qy > 3 ? 1 : 0),
              dz = cz < 0 ? -1 : (cz > 7 ? 1 : 0);
    const uint32_t b = nb[13 + dx + 3 * dy + 9 * dz];
    T o[4] = {0, 0, 0, 0};
    if (b != ~0u) ld4q(ec + (b >> 3) + (s16::sp4(2 * (qx & 3)) | (s16::sp4(2 * (qy & 3)) << 1) | (s16::sp4(cz & 7) << 2)), o);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int cx = 2 * qx + (e & 1), cy = 2 * qy + (e >> 1);
      if (cx >= -1 && cx <= 8 && cy >= -1 && cy <= 8) ctile[coarse_at(cx, cy) + cz] = o[e];
    }
  }
}

// The sum over the block of one value per (quad column q, plane z), in an order fixed by the block: each
// column's planes in z order, then the 64 column sums by a fixed tree.  red: 64 x 18 doubles of shared
// memory, the value of (q, z) at red_at(q, z), written after a barrier that ends every other use of that
// memory.  Every thread calls this (it has barriers); thread 0 returns the sum.
__device__ __forceinline__ int red_at(int qx, int qy, int z) {  // columns in Morton order, as the writing lanes
  return 18 * (int)(s16::sp2(qx) | s16::sp2(qy) << 1) + z;
}
__device__ __forceinline__ double block_sum_fixed(double* red) {
  __syncthreads();
  const int t = threadIdx.x;
  double s = 0.0;
  if (t < 64) {
#pragma unroll
    for (int z = 0; z < 16; ++z) s += red[red_at(t & 7, t >> 3, z)];
  }
  __syncthreads();
  if (t < 64) red[t] = s;
  __syncthreads();
  if (t < 32) {
    s = red[t] + red[t + 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  }
  return s;
}

// the 4 x 4 patch around quad (x0, y0) on a halo plane
template <typename T>
__device__ __forceinline__ void halo_patch(const T* tile, int hi, int x0, int y0, T (&r)[4][4]) {
  const T* p = tile + halo_at(hi, x0, y0);
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) r[j][i] = p[(j - 1) * kHR + i - 1];
}
// the 4 x 4 columns around the quad over the thread's planes, the quad's own from v
template <int ZT, typename T>
__device__ __forceinline__ void load_columns(const T* tile, int x0, int y0, const Seg<ZT>& g, const T (&v)[ZT][4],
                                             T (&col)[4][4][ZT]) {
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if ((i == 1 || i == 2) && (j == 1 || j == 2)) {
#pragma unroll
        for (int k = 0; k < ZT; ++k) col[j][i][k] = v[k][2 * (j - 1) + i - 1];
      } else {
        ldz<ZT>(tile + at(x0 - 1 + i, y0 - 1 + j) + g.w0, col[j][i]);
      }
    }
}
// Stencil rows y = A v of the quad column's ZT planes (v: its own values, also in the tile): per plane the
// in-plane sums tz (for the planes above and below) and own; a row is (tz(z - 1) + own(z)) + tz(z + 1).
template <int ZT, typename T>
__device__ __forceinline__ void stencil_rows(const T* tile, int x0, int y0, const Seg<ZT>& g, const T (&v)[ZT][4],
                                             T c0, T ce, T cc, T (&y)[ZT][4]) {
  T tz[ZT][4];
  {
    T col[4][4][ZT];
    load_columns<ZT, T>(tile, x0, y0, g, v, col);
#pragma unroll
    for (int k = 0; k < ZT; ++k) {
      T r[4][4], ctr[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) r[j][i] = col[j][i][k];
      n16::plane_terms<T>(r, c0, ce, cc, tz[k], y[k], ctr);
    }
  }
  T te[4] = {0, 0, 0, 0};  // tz of the halo plane at the block's end
  if (g.first() || g.last()) {
    T r[4][4], own[4], ctr[4];
    halo_patch<T>(tile, g.last(), x0, y0, r);
    n16::plane_terms<T>(r, c0, ce, cc, te, own, ctr);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    T x[ZT], nx[ZT], ox[ZT];
#pragma unroll
    for (int k = 0; k < ZT; ++k) x[k] = tz[k][e];
    beside<ZT>(g, x, te[e], nx, ox);
#pragma unroll
    for (int k = 0; k < ZT; ++k) y[k][e] = ((g.p ? nx[k] : ox[k]) + y[k][e]) + (g.p ? ox[k] : nx[k]);
  }
}
// The same rows with a node's edge and corner neighbours summed before they meet their coefficients.
template <int ZT, typename T>
__device__ __forceinline__ void stencil_rows_summed(const T* tile, int x0, int y0, const Seg<ZT>& g,
                                                    const T (&v)[ZT][4], T c0, T ce, T cc, T (&y)[ZT][4]) {
  T fk[ZT][4], dk[ZT][4], ctr[4];
  {
    T col[4][4][ZT];
    load_columns<ZT, T>(tile, x0, y0, g, v, col);
#pragma unroll
    for (int k = 0; k < ZT; ++k) {
      T r[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) r[j][i] = col[j][i][k];
      n16::plane_sums<T>(r, fk[k], dk[k], ctr);
    }
  }
  T fe[4] = {0, 0, 0, 0}, de[4] = {0, 0, 0, 0};
  if (g.first() || g.last()) {
    T r[4][4];
    halo_patch<T>(tile, g.last(), x0, y0, r);
    n16::plane_sums<T>(r, fe, de, ctr);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    T f[ZT], d[ZT], fn[ZT], fo[ZT], dn[ZT], dO[ZT];
#pragma unroll
    for (int k = 0; k < ZT; ++k) {
      f[k] = fk[k][e];
      d[k] = dk[k][e];
    }
    beside<ZT>(g, f, fe[e], fn, fo);
    beside<ZT>(g, d, de[e], dn, dO);
#pragma unroll
    for (int k = 0; k < ZT; ++k) y[k][e] = c0 * v[k][e] + ce * (d[k] + (fn[k] + fo[k])) + cc * (dn[k] + dO[k]);
  }
}
}  // namespace z16

// ------------------------------------------------------------------ 16^3 stencil SpMV (finest level)
namespace n16 {
template <int ZT>
using Zt = z16::Zt<ZT>;
// CTAs per SM that the register budget is set for; FP64 at depth 9, 4 planes: two CTAs 749 us for the
// plain SpMV, one 926, three (spilling) 1246
template <typename T, int ZT>
constexpr int kCtas = sizeof(T) == 4 && ZT == 4 ? 4 : 2;

// KIND 0: q = A a, part = a.q;  1: an = bvec + beta a, q = A an, part = an.q;
// 3: q = A a for a caller's vector: a node's 12 edge and 8 corner neighbours are summed before they
// meet their coefficients, as in the per-node stencil, which rounds less than the solver's order;
// 2: an = a + beta bvec (FP64 solution + correction of type E; a null: zero), q = rhs - A an.
// beta_dev (packed launches): the cloud's beta, in place of the beta argument.
template <typename T, int KIND, typename E, int ZT>
__global__ void __launch_bounds__(Zt<ZT>::NT, kCtas<T, ZT>)
    k_spmv16(uint32_t D, const T* __restrict__ a, const E* __restrict__ bvec, T* __restrict__ an, T beta,
             T* __restrict__ q, T c0, T ce, T cc, const T* __restrict__ rhs, double* __restrict__ part,
             const double* __restrict__ beta_dev) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);
  __shared__ uint32_t nb[27];
  const int res = 1 << D;
  {
    const uint64_t nl = 1ull << (3 * D);
    a = cloud_slice(a, nl);
    bvec = cloud_slice(bvec, nl);
    an = cloud_slice(an, nl);
    q = cloud_slice(q, nl);
    rhs = cloud_slice(rhs, nl);
    part = cloud_slice(part, gridDim.x);
    if (beta_dev) beta = (T)beta_dev[blockIdx.y];
  }
  const uint32_t blk = blockIdx.x, base = blk << 12;
  uint32_t bx, by, bz;
  unmorton3(blk, bx, by, bz);
  const int t = threadIdx.x;
  const z16::Seg<ZT> g(t);
  int qx, qy;
  z16::quad_of(t / Zt<ZT>::SEG, qx, qy);
  const int x0 = 2 * qx, y0 = 2 * qy;
  const uint32_t mq = s16::sp4(x0) | (s16::sp4(y0) << 1);
  s16::neighbour_bases(nb, bx, by, bz, res >> 4);
  auto add = [&](T (&o)[4], const E (&bv)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (KIND == 1) o[i] = (T)bv[i] + beta * o[i];
      else if (beta != (T)0) o[i] += beta * (T)bv[i];  // beta 0: a cloud that has stopped keeps its solution
    }
  };
  auto quad = [&](uint32_t m, T (&o)[4]) {
    if (KIND != 2 || a) z16::ld4q(a + m, o);
    else o[0] = o[1] = o[2] = o[3] = (T)0;
    if (KIND == 1 || KIND == 2) {
      E bv[4];
      z16::ld4q(bvec + m, bv);
      add(o, bv);
    }
  };
  T v[ZT][4];
#pragma unroll
  for (int k = 0; k < ZT; ++k) quad(base + (mq | (s16::sp4(g.z(k)) << 2)), v[k]);
  __syncthreads();  // nb
  {
    T hv[Zt<ZT>::HV][4];
    z16::load_halo<ZT, T>(nb, quad, hv);
    z16::store_quad<ZT>(tile, x0, y0, g, v);
    if (KIND == 1 || KIND == 2) {
#pragma unroll
      for (int k = 0; k < ZT; ++k) z16::st4q(an + (base + (mq | (s16::sp4(g.z(k)) << 2))), v[k]);
    }
    z16::store_halo<ZT, false, T>(tile, nb, nullptr, hv);
  }
  __syncthreads();
  T y[ZT][4];
  if constexpr (KIND == 3) z16::stencil_rows_summed<ZT, T>(tile, x0, y0, g, v, c0, ce, cc, y);
  else z16::stencil_rows<ZT, T>(tile, x0, y0, g, v, c0, ce, cc, y);
  double pv[ZT];  // per plane: the quad's four products of the dot
#pragma unroll
  for (int k = 0; k < ZT; ++k) {
    const uint32_t m = base + (mq | (s16::sp4(g.z(k)) << 2));
    if (KIND == 2) {
      T rv[4];
      z16::ld4q(rhs + m, rv);
#pragma unroll
      for (int e = 0; e < 4; ++e) y[k][e] = rv[e] - y[k][e];
    } else {
      double a4 = 0.0;
#pragma unroll
      for (int e = 0; e < 4; ++e) a4 += (double)v[k][e] * (double)y[k][e];
      pv[k] = a4;
    }
    z16::st4q(q + m, y[k]);
  }
  if (KIND < 2) {
    __syncthreads();  // the tile's last reads: its memory takes the per-plane sums
    double* red = reinterpret_cast<double*>(smem_raw);
#pragma unroll
    for (int k = 0; k < ZT; ++k) red[z16::red_at(qx, qy, g.z(k))] = pv[k];
    const double sdot = z16::block_sum_fixed(red);
    if (t == 0) part[blk] = sdot;
  }
}
template <typename T>
constexpr size_t smem_bytes() {
  return sizeof(T) * z16::TILE;
}
}  // namespace n16

// ------------------------------------------------------------------ 16^3 residual + restriction
// Two launches, no redundant work.  k_resid16: r = f - A e on the block's 16^3 nodes (the
// SpMV's tile and quad columns; r then takes e's place in the tile), then (a) the part of the
// restriction to the block's 8^3 coarse nodes that comes from its own fine nodes, and (b) the
// restriction partials its high faces (local 15) owe the coarse nodes of its high neighbours: per
// face the sum over the face's other two axes (8 x 8), per edge over the remaining axis (8), and
// the corner (1), into a face buffer of 224 values per block.  k_restrict_faces adds to the coarse
// nodes on each block's low faces these partials of its low neighbours, scaled by 1/2 per crossed
// axis.  Restriction: coarse c gathers fine 2c-1, 2c, 2c+1 per axis with weights 1/2, 1, 1/2.
namespace r16 {
constexpr int FACE = 224;
// face buffer layout: [0,64) x face (cy + 8 cz), [64,128) y face (cx + 8 cz), [128,192) z face
// (cx + 8 cy), [192,200) xy edge (cz), [200,208) xz edge (cy), [208,216) yz edge (cx), 216 corner

// What the low-face row `cm` of a node changes in its residual: (interior row - face row) of A e, with
// at(dx, dy, dz) the node's neighbours.
template <typename T, typename At>
__device__ __forceinline__ T face_change(At at, const T* cm, T c0, T ce, T cc) {
  T yf = 0, se = 0, sc = 0;
#pragma unroll
  for (int o = 0; o < 27; ++o) {
    const int dx = o % 3 - 1, dy = (o / 3) % 3 - 1, dz = o / 9 - 1;
    const int nzc = (dx != 0) + (dy != 0) + (dz != 0);
    const T v = at(dx, dy, dz);
    yf += cm[o] * v;
    if (nzc == 2) se += v;
    else if (nzc == 3) sc += v;
  }
  const T yi = c0 * at(0, 0, 0) + ce * se + cc * sc;
  return yi - yf;
}

// r += what the low-face rows change at the quad column's nodes on a low domain face
template <int ZT, typename T>
__device__ __forceinline__ void face_residual(const T* tile, const T* table, int ox, int oy, int oz, int x0, int y0,
                                              const z16::Seg<ZT>& g, T c0, T ce, T cc, T (&r)[ZT][4]) {
#pragma unroll 1
  for (int i = 0; i < 4 * ZT; ++i) {
    const int x = x0 + (i & 1), y = y0 + ((i >> 1) & 1), z = g.z(i >> 2);
    const int mask = ((ox + x) == 0) | (((oy + y) == 0) << 1) | (((oz + z) == 0) << 2);
    if (!mask) continue;
    const z16::PlaneRef<T> pl[3] = {z16::plane_ref(tile, x, y, z - 1), z16::plane_ref(tile, x, y, z),
                                    z16::plane_ref(tile, x, y, z + 1)};
    const T dr = face_change<T>([&](int dx, int dy, int dz) { return pl[dz + 1](dx, dy); }, table + 27 * mask, c0, ce,
                                cc);
#pragma unroll
    for (int k = 0; k < ZT; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (4 * k + e == i) r[k][e] += dr;
  }
}

// restriction of the block's residual tile to its coarse node (cx, cy, cz) from its own fine nodes
template <typename T>
__device__ __forceinline__ T restrict_own(const T* tile, int cx, int cy, int cz) {
  T c[3][3][3];  // fine planes 2cz - 1, 2cz, 2cz + 1 of columns x, then y, 2c - 1 .. 2c + 1
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const T* p = tile + z16::at(2 * cx + i - 1, 2 * cy + j - 1) + cz;  // plane 2 cz; plane 2 cz + 1 at p[8]
      c[0][j][i] = cz > 0 ? p[7] : (T)0;
      c[1][j][i] = p[0];
      c[2][j][i] = p[8];
    }
  T s = 0;
#pragma unroll
  for (int dz = -1; dz <= 1; ++dz) {
    if (dz < 0 && cz == 0) continue;
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy) {
      if (dy < 0 && cy == 0) continue;
      const T wyz = (T)((dy == 0 ? 1.0 : 0.5) * (dz == 0 ? 1.0 : 0.5));
      const T* r = c[dz + 1][dy + 1];
      const T left = cx > 0 ? r[0] : (T)0;
      s += wyz * (r[1] + (T)0.5 * (r[2] + left));
    }
  }
  return s;
}

template <typename T, bool FACES, int ZT>
__global__ void __launch_bounds__(n16::Zt<ZT>::NT, n16::kCtas<T, ZT>)
    k_resid16(uint32_t D, const T* __restrict__ e, const T* __restrict__ f, T* __restrict__ fc,
              T* __restrict__ face, T c0, T ce, T cc, const T* __restrict__ table) {
  constexpr int NT = n16::Zt<ZT>::NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);
  __shared__ uint32_t nb[27];
  const int res = 1 << D;
  {
    const uint64_t nl = 1ull << (3 * D);
    e = cloud_slice(e, nl);
    f = cloud_slice(f, nl);
    fc = cloud_slice(fc, nl / 8);
    face = cloud_slice(face, (uint64_t)gridDim.x * FACE);
  }
  const uint32_t blk = blockIdx.x, base = blk << 12;
  uint32_t bx, by, bz;
  unmorton3(blk, bx, by, bz);
  const int ox = (int)bx * 16, oy = (int)by * 16, oz = (int)bz * 16;
  const int t = threadIdx.x;
  const z16::Seg<ZT> g(t);
  int qx, qy;
  z16::quad_of(t / n16::Zt<ZT>::SEG, qx, qy);
  const int x0 = 2 * qx, y0 = 2 * qy;
  const uint32_t mq = s16::sp4(x0) | (s16::sp4(y0) << 1);
  s16::neighbour_bases(nb, bx, by, bz, res >> 4);
  T r[ZT][4];
  {
    T v[ZT][4];
#pragma unroll
    for (int k = 0; k < ZT; ++k) z16::ld4q(e + (base + (mq | (s16::sp4(g.z(k)) << 2))), v[k]);
    __syncthreads();  // nb
    {
      T hv[n16::Zt<ZT>::HV][4];
      z16::load_halo<ZT, T>(nb, [&](uint32_t m, T (&o)[4]) { z16::ld4q(e + m, o); }, hv);
      z16::store_quad<ZT>(tile, x0, y0, g, v);
      z16::store_halo<ZT, false, T>(tile, nb, nullptr, hv);
    }
    __syncthreads();
    z16::stencil_rows<ZT, T>(tile, x0, y0, g, v, c0, ce, cc, r);
  }
#pragma unroll
  for (int k = 0; k < ZT; ++k) {
    T fq[4];
    z16::ld4q(f + (base + (mq | (s16::sp4(g.z(k)) << 2))), fq);
#pragma unroll
    for (int i = 0; i < 4; ++i) r[k][i] = fq[i] - r[k][i];
  }
  if (FACES && (ox == 0 || oy == 0 || oz == 0)) face_residual<ZT>(tile, table, ox, oy, oz, x0, y0, g, c0, ce, cc, r);
  __syncthreads();  // e is read
  z16::store_quad<ZT>(tile, x0, y0, g, r);
  __syncthreads();
  // own part of the restriction (lanes: eight coarse planes of a 2 x 2 of columns)
  const uint64_t cbase = (uint64_t)blk * 512;
#pragma unroll
  for (int i = t; i < 512; i += NT) {
    const int cz = i & 7, cx = ((i >> 3) & 1) | ((i >> 5) & 3) << 1, cy = ((i >> 4) & 1) | ((i >> 7) & 3) << 1;
    fc[cbase + (s16::sp4(cx) | (s16::sp4(cy) << 1) | (s16::sp4(cz) << 2))] = restrict_own<T>(tile, cx, cy, cz);
  }
  // restriction partials of the high faces, edges and corner
  {
    T* fb = face + (uint64_t)blk * FACE;
    auto w = [](int d) { return (T)(d == 0 ? 1.0 : 0.5); };
    for (int u = t; u < 217; u += NT) {
      if (u < 192) {  // faces: the two free axes restricted, the face axis at local 15
        const int axis = u >> 6, i = u & 7, j = (u >> 3) & 7;
        T acc = 0;
#pragma unroll
        for (int dj = -1; dj <= 1; ++dj) {
          const int fj = 2 * j + dj;
          if (fj < 0) continue;
#pragma unroll
          for (int di = -1; di <= 1; ++di) {
            const int fi = 2 * i + di;
            if (fi < 0) continue;
            const int x = axis == 0 ? 15 : fi, y = axis == 1 ? 15 : (axis == 0 ? fi : fj), z = axis == 2 ? 15 : fj;
            acc += w(di) * w(dj) * tile[z16::at(x, y) + z16::zw(z)];
          }
        }
        fb[u] = acc;
      } else if (u < 216) {  // edges: the free axis restricted
        const int e = (u - 192) >> 3, i = (u - 192) & 7;
        T acc = 0;
#pragma unroll
        for (int di = -1; di <= 1; ++di) {
          const int fi = 2 * i + di;
          if (fi < 0) continue;
          const int x = e == 2 ? fi : 15, y = e == 1 ? fi : 15, z = e == 0 ? fi : 15;
          acc += w(di) * tile[z16::at(x, y) + z16::zw(z)];
        }
        fb[u] = acc;
      } else {
        fb[216] = tile[z16::at(15, 15) + 15];
      }
    }
  }
}

// Adds to the coarse nodes on each block's low faces what the fine nodes at local -1 contribute:
// the partials of the low neighbours (k_resid16), 1/2 per axis crossed, fixed order.  Four
// blocks per CTA, 169 boundary coarse nodes per block.
template <typename T>
__global__ void __launch_bounds__(768) k_restrict_faces(uint32_t D, const T* __restrict__ face, T* __restrict__ fc,
                                                       uint32_t nblk) {
  const int nba = 1 << (D - 4);
  face = cloud_slice(face, (uint64_t)nblk * FACE);
  fc = cloud_slice(fc, (uint64_t)nblk * 512);
  const uint32_t blk = blockIdx.x * 4 + threadIdx.x / 192;
  const int j = threadIdx.x % 192;
  if (blk >= nblk || j >= 169) return;
  uint32_t bx, by, bz;
  unmorton3(blk, bx, by, bz);
  int cx, cy, cz;
  if (j < 64) { cx = 0; cy = j & 7; cz = j >> 3; }
  else if (j < 120) { cx = 1 + (j - 64) % 7; cy = 0; cz = (j - 64) / 7; }
  else { cx = 1 + (j - 120) % 7; cy = 1 + (j - 120) / 7; cz = 0; }
  T s = 0;
  bool any = false;
#pragma unroll
  for (int e = 1; e < 8; ++e) {
    const int ex = e & 1, ey = (e >> 1) & 1, ez = e >> 2;
    if ((ex && cx) || (ey && cy) || (ez && cz)) continue;  // only coarse index 0 reaches fine -1
    const int nx = (int)bx - ex, ny = (int)by - ey, nz = (int)bz - ez;
    if (nx < 0 || ny < 0 || nz < 0) continue;  // outside the domain
    (void)nba;
    const T* fb = face + (uint64_t)morton3((uint32_t)nx, (uint32_t)ny, (uint32_t)nz) * FACE;
    T v;
    switch (e) {
      case 1: v = (T)0.5 * fb[cy + 8 * cz]; break;
      case 2: v = (T)0.5 * fb[64 + cx + 8 * cz]; break;
      case 4: v = (T)0.5 * fb[128 + cx + 8 * cy]; break;
      case 3: v = (T)0.25 * fb[192 + cz]; break;
      case 5: v = (T)0.25 * fb[200 + cy]; break;
      case 6: v = (T)0.25 * fb[208 + cx]; break;
      default: v = (T)0.125 * fb[216]; break;
    }
    s += v;
    any = true;
  }
  if (any) fc[(uint64_t)blk * 512 + morton3((uint32_t)cx, (uint32_t)cy, (uint32_t)cz)] += s;
}
template <typename T>
constexpr size_t smem_bytes() {
  return sizeof(T) * z16::TILE;
}
}  // namespace r16

// ------------------------------------------------------------------ 16^3 smoother (levels >= 4)
// Multicolour Gauss-Seidel in the block, blocks coupled through the halo values from before
// the sweep.  Every level's interior stencil has no face couplings, so nodes that share the
// parity of x and y are uncoupled along z: the sweep has 4 phases, one per (x, y) parity class,
// each relaxing whole columns of that class at once (forward order (0,0) (1,0) (0,1) (1,1),
// backward the reverse, each the adjoint of the other).  Thread = one 2x2 quad column over ZT z
// planes of a parity-split tile (below); in phase k it relaxes the class-k column of its quad, sweeping
// the planes once: a plane's ring around the column gives its in-plane edge sum D (diagonals)
// and face-adjacent sum F, and the node at z uses D(z), F(z-1), F(z+1), D(z-1), D(z+1).
// FACES (coarse levels): nodes on the low domain faces use their 27-entry table row, which does
// couple z-neighbours of the same class; those take the values from before the phase (new
// values are written after a barrier), a Jacobi step along the column for those rows only.  On the
// coarse levels these rows are a phase's critical path (few blocks, most of them on a face), so a
// row is unrolled: its 26 tile and table loads (the table in shared memory) are in flight together
// before the chain of its multiply-adds: post-smoothing on 32^3 and 64^3 in FP32 8.1 us, the first sweep
// 6.1 (29 to 31 us in a rolled loop with the table in global memory).
namespace g16 {
// CTAs per SM that the register budget is set for: four, three where the face rows would spill
template <typename T, bool FACES, int ZT>
constexpr int kCtas = sizeof(T) == 8 ? 2 : (ZT == 2 ? 2 : (FACES ? 3 : 4));

// One phase: new values of the class-CLS column of the thread's quad (planes z0..z0+ZT-1).
// The ring members inside the thread's quad come from registers (v), the other five columns from the
// tile; the in-plane sums of the planes below and above from the neighbouring lanes, at the block's ends
// from the halo planes (zero there for a sweep from zero).
// ZERO: a forward sweep from zero, in which the classes after CLS are still zero everywhere
// (their loads are skipped; phase 0 needs none).
template <typename T, int CLS, bool FROM_ZERO, bool ZERO, int ZT>
__device__ __forceinline__ void relax_column(const T* tile, int x0, int y0, const z16::Seg<ZT>& g,
                                             const T (&fv)[ZT][4], const T (&v)[ZT][4], T ce, T cc, T c0inv,
                                             T (&nv)[ZT]) {
  constexpr int CX = CLS & 1, CY = CLS >> 1, CS = z16::kCS, RY = z16::kRY;
  constexpr int EDX = CX == 0 ? -1 : 1, EDY = CY == 0 ? -1 : 1;  // direction of the external ring side
  constexpr int EFX = (CX ^ 1) | (CY << 1), EFY = CX | ((CY ^ 1) << 1), ED = (CX ^ 1) | ((CY ^ 1) << 1);
  // classes updated before CLS in a forward sweep are 0..CLS-1
  constexpr bool NFX = !ZERO || EFX < CLS, NFY = !ZERO || EFY < CLS, ND = !ZERO || ED < CLS;
  if (ZERO && CLS == 0) {
#pragma unroll
    for (int k = 0; k < ZT; ++k) nv[k] = fv[k][CLS] * c0inv;
    return;
  }
  const T* c = tile + z16::at(x0 + CX, y0 + CY) + g.w0;
  T q0[ZT], q1[ZT], q2[ZT], ed[ZT], ex[ZT], Dk[ZT], Fk[ZT];
  if (ND) {
    z16::ldz<ZT>(c + EDY * RY - CS, q0);
    z16::ldz<ZT>(c + EDY * RY + CS, q2);
    z16::ldz<ZT>(c - EDY * RY + EDX * CS, ed);
  }
  if (NFY) z16::ldz<ZT>(c + EDY * RY, q1);
  if (NFX) z16::ldz<ZT>(c + EDX * CS, ex);
#pragma unroll
  for (int k = 0; k < ZT; ++k) {
    Dk[k] = Fk[k] = 0;
    if (ND) Dk[k] = (q0[k] + q2[k]) + (ed[k] + v[k][ED]);
    if (NFY) Fk[k] += q1[k] + v[k][EFY];
    if (NFX) Fk[k] += ex[k] + v[k][EFX];
  }
  T De = 0, Fe = 0;
  if (!FROM_ZERO && (g.first() || g.last())) {  // the halo plane: the whole ring from the tile
    const T* h = tile + z16::halo_at(g.last(), x0 + CX, y0 + CY);
    constexpr int HR = z16::kHR;
    De = (h[-HR - 1] + h[-HR + 1]) + (h[HR - 1] + h[HR + 1]);
    Fe = (h[-HR] + h[HR]) + (h[-1] + h[1]);
  }
  T Dn[ZT], Do[ZT], Fn[ZT], Fo[ZT];
  if (ND) {
    z16::beside<ZT>(g, Dk, De, Dn, Do);
  } else {
#pragma unroll
    for (int k = 0; k < ZT; ++k) Dn[k] = Do[k] = 0;
  }
  z16::beside<ZT>(g, Fk, Fe, Fn, Fo);
#pragma unroll
  for (int k = 0; k < ZT; ++k) {  // edges D(z) + F(z-1) + F(z+1), corners D(z-1) + D(z+1)
    const T fm = g.p ? Fn[k] : Fo[k], fp = g.p ? Fo[k] : Fn[k];
    nv[k] = (fv[k][CLS] - ce * (Dk[k] + fm + fp) - cc * (Dn[k] + Do[k])) * c0inv;
  }
}

// One sweep of the tile: the four phases, each ended by a barrier.  faces: the block holds nodes on a
// low domain face (uniform in the block), whose rows are in ftab.
template <typename T, bool FWD, bool FROM_ZERO, bool FACES, int ZT>
__device__ __forceinline__ void sweep(T* tile, const T* ftab, bool faces, int ox, int oy, int oz, int x0, int y0,
                                      const z16::Seg<ZT>& g, const T (&fv)[ZT][4], T (&v)[ZT][4], T ce, T cc,
                                      T c0inv) {
#pragma unroll
  for (int ph = 0; ph < 4; ++ph) {
    const int cls = FWD ? ph : 3 - ph;
    const int x = x0 + (cls & 1), y = y0 + (cls >> 1);
    T nv[ZT];
    constexpr bool ZERO = FROM_ZERO && FWD;
    switch (cls) {
      case 0: relax_column<T, 0, FROM_ZERO, ZERO, ZT>(tile, x0, y0, g, fv, v, ce, cc, c0inv, nv); break;
      case 1: relax_column<T, 1, FROM_ZERO, ZERO, ZT>(tile, x0, y0, g, fv, v, ce, cc, c0inv, nv); break;
      case 2: relax_column<T, 2, FROM_ZERO, ZERO, ZT>(tile, x0, y0, g, fv, v, ce, cc, c0inv, nv); break;
      default: relax_column<T, 3, FROM_ZERO, ZERO, ZT>(tile, x0, y0, g, fv, v, ce, cc, c0inv, nv); break;
    }
    T* self = tile + z16::at(x, y) + g.w0;
    if (faces) {  // low-domain-face nodes of this column: their table rows, neighbours from the tile
#pragma unroll 1
      for (int k = 0; k < ZT; ++k) {
        const int mask = ((ox + x) == 0) | (((oy + y) == 0) << 1) | (((oz + g.z(k)) == 0) << 2);
        if (!mask) continue;
        const T* cm = ftab + 27 * mask;
        const int z = g.z(k);
        const z16::PlaneRef<T> pl[3] = {z16::plane_ref<T>(tile, x, y, z - 1), z16::plane_ref<T>(tile, x, y, z),
                                        z16::plane_ref<T>(tile, x, y, z + 1)};
        T off = 0;
#pragma unroll
        for (int o = 0; o < 27; ++o) {
          if (o == 13) continue;
          off += cm[o] * pl[o / 9](o % 3 - 1, (o / 3) % 3 - 1);
        }
        T fk = fv[0][cls];
#pragma unroll
        for (int kk = 1; kk < ZT; ++kk)
          if (kk == k) fk = fv[kk][cls];
        const T nvk = (fk - off) / cm[13];
#pragma unroll
        for (int kk = 0; kk < ZT; ++kk)
          if (kk == k) nv[kk] = nvk;
      }
      __syncthreads();  // same-class column neighbours were read with their old values
    }
#pragma unroll
    for (int k = 0; k < ZT; ++k) v[k][cls] = nv[k];
    z16::stz<ZT>(self, nv);
    __syncthreads();
  }
}

// MODE 0: xo = sweep(xi); 1: xo = sweep(0); 2: xo = sweep(xi + P ec).  DOT: part = f.xo
// MODE 3 (finest level, forward): first the CG update x += alpha d, r -= alpha q in place
// (pointwise), then xo = sweep(0) with f = the new r; part = per-block sums of r^2.  A sweep
// from zero reads no halo, so updating r in place is race-free.
template <typename T, int MODE, bool DOT, bool FWD, bool FACES, int ZT>
__global__ void __launch_bounds__(n16::Zt<ZT>::NT, kCtas<T, FACES, ZT>)
    k_smooth16(uint32_t D, const T* __restrict__ xi, T* __restrict__ xo, const T* __restrict__ f,
               const T* __restrict__ ec, T c0inv, T ce, T cc, const T* __restrict__ table,
               double* __restrict__ part, CgFuse<T> cg) {
  static_assert(MODE != 3 || (FWD && !FACES), "the fused CG update is a forward sweep on the finest level");
  constexpr int NT = n16::Zt<ZT>::NT;
  constexpr bool FROM_ZERO = MODE == 1 || MODE == 3;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);  // z16::TILE
  T* ctile = tile + z16::TILE;               // z16::kCTile (MODE 2)
  __shared__ uint32_t nb[27];
  __shared__ T ftab[FACES ? 216 : 1];  // the face rows
  const int res = 1 << D;
  {
    const uint64_t nl = 1ull << (3 * D);
    xi = cloud_slice(xi, nl);
    xo = cloud_slice(xo, nl);
    f = cloud_slice(f, nl);
    ec = cloud_slice(ec, nl / 8);
    part = cloud_slice(part, gridDim.x);
    if (MODE == 3) {
      cg.x = cloud_slice(cg.x, nl);
      cg.d = cloud_slice(cg.d, nl);
      cg.q = cloud_slice(cg.q, nl);
      cg.r = cloud_slice(cg.r, nl);
      cg.rin = cloud_slice(cg.rin, nl);
      if (cg.alpha_dev) cg.alpha = (T)cg.alpha_dev[blockIdx.y];
    }
  }
  const uint32_t blk = blockIdx.x, base = blk << 12;
  uint32_t bx, by, bz;
  unmorton3(blk, bx, by, bz);
  const int ox = (int)bx * 16, oy = (int)by * 16, oz = (int)bz * 16;
  const int t = threadIdx.x;
  const z16::Seg<ZT> g(t);
  int qx, qy;
  z16::quad_of(t / n16::Zt<ZT>::SEG, qx, qy);
  const int x0 = 2 * qx, y0 = 2 * qy;
  const uint32_t mq = s16::sp4(x0) | (s16::sp4(y0) << 1);
  const bool faces = FACES && (ox == 0 || oy == 0 || oz == 0);  // uniform in the block
  if (faces)
    for (int i = t; i < 216; i += NT) ftab[i] = table[i];  // read after the barriers below
  if (!FROM_ZERO) s16::neighbour_bases(nb, bx, by, bz, res >> 4);
  T fv[ZT][4], v[ZT][4];
  double rr[ZT];  // MODE 3: per plane, the quad's r^2
#pragma unroll
  for (int k = 0; k < ZT; ++k) {
    const uint32_t m = base + (mq | (s16::sp4(g.z(k)) << 2));
    if (MODE == 3) {  // the CG update of this quad (plain loads: x and r are written here)
      typedef typename s16::Vec4<T>::type V4;
      const V4 rq = *reinterpret_cast<const V4*>((cg.rin ? cg.rin : cg.r) + m);
      fv[k][0] = rq.x; fv[k][1] = rq.y; fv[k][2] = rq.z; fv[k][3] = rq.w;
      if (cg.alpha != (T)0 || cg.rin) {  // alpha 0: a cloud that has stopped keeps x and r
        T xq[4] = {};
        if (!cg.rin) {
          const V4 xv = *reinterpret_cast<const V4*>(cg.x + m);
          xq[0] = xv.x; xq[1] = xv.y; xq[2] = xv.z; xq[3] = xv.w;
        }
        if (cg.alpha != (T)0) {
          T dq[4], qq[4];
          z16::ld4q(cg.d + m, dq);
          z16::ld4q(cg.q + m, qq);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            xq[e] += cg.alpha * dq[e];
            fv[k][e] -= cg.alpha * qq[e];
          }
        }
        z16::st4q(cg.x + m, xq);
        z16::st4q(cg.r + m, fv[k]);
      }
      rr[k] = (double)fv[k][0] * fv[k][0] + (double)fv[k][1] * fv[k][1] + (double)fv[k][2] * fv[k][2] +
              (double)fv[k][3] * fv[k][3];
    } else if (FROM_ZERO) {
      z16::ld4q(f + m, fv[k]);
    }
    if (FROM_ZERO) v[k][0] = v[k][1] = v[k][2] = v[k][3] = (T)0;
    else z16::ld4q(xi + m, v[k]);
  }
  if (FROM_ZERO) {
    z16::zero_side_halo<ZT, T>(tile);
    if (faces) {  // face rows read the planes above and below, and every class
      for (int i = t; i < z16::TILE; i += NT) tile[i] = 0;
    } else if (!FWD) {
      z16::store_quad<ZT>(tile, x0, y0, g, v);
    }
  } else {
    T hv[n16::Zt<ZT>::HV][4];
    __syncthreads();  // nb
    z16::load_halo<ZT, T>(nb, [&](uint32_t m, T (&o)[4]) { z16::ld4q(xi + m, o); }, hv);
    if (MODE == 2) {
      z16::load_coarse_tile<NT>(ctile, ec, nb);
      __syncthreads();  // ctile
      z16::prolong_quads<ZT>(ctile, qx, qy, g, v);
    }
#pragma unroll
    for (int k = 0; k < ZT; ++k) z16::ld4q(f + (base + (mq | (s16::sp4(g.z(k)) << 2))), fv[k]);
    z16::store_quad<ZT>(tile, x0, y0, g, v);
    z16::store_halo<ZT, MODE == 2, T>(tile, nb, ctile, hv);
  }
  __syncthreads();
  sweep<T, FWD, FROM_ZERO, FACES, ZT>(tile, ftab, faces, ox, oy, oz, x0, y0, g, fv, v, ce, cc, c0inv);
  double acc[ZT];  // DOT: per plane, the quad's f.x
#pragma unroll
  for (int k = 0; k < ZT; ++k) z16::st4q(xo + (base + (mq | (s16::sp4(g.z(k)) << 2))), v[k]);
#pragma unroll
  for (int k = 0; k < ZT; ++k) {
    acc[k] = 0.0;
    if (DOT)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[k] += (double)fv[k][e] * (double)v[k][e];
  }
  if (DOT || MODE == 3) {
    // the last phase ended with a barrier: the tile's memory takes the per-plane sums
    double* red = reinterpret_cast<double*>(smem_raw);
#pragma unroll
    for (int k = 0; k < ZT; ++k) red[z16::red_at(qx, qy, g.z(k))] = MODE == 3 ? rr[k] : acc[k];
    const double sum = z16::block_sum_fixed(red);
    if (t == 0) part[blk] = sum;
  }
}
template <typename T>
constexpr size_t smem_bytes(int mode) {
  return sizeof(T) * (z16::TILE + (mode == 2 ? z16::kCTile : 0));
}
}  // namespace g16

// ------------------------------------------------------------------ the coarsest levels in one block
// V-cycle of the levels 16^3, 8^3 and 4^3 (each a single block of its kernel) in one CTA per cloud:
// eight launches of one or a few warps' work each, whose time was launch and memory latency.  The
// level vectors, the face rows and the dense inverse stay in shared memory between the steps; every
// step is the arithmetic of its own kernel (k_smooth16, k_resid16, k_smooth, k_resid_restrict,
// k_dense_solve), so the result is the same, bit for bit.  512 threads: thread = one 2x2 quad column
// over 2 planes of the 16^3 level, or one node of the 8^3 level; the 64 nodes of an 8^3 colour and of
// the 4^3 level are two warps' work.
namespace t4 {
constexpr int NT = 512, ZT = 2;
constexpr int kInvStride = 65;  // the dense inverse's rows on disjoint banks
constexpr int WE = 11, WR = 9;  // the 8^3 level's natural tiles: e over local [-2, 8], r over [-1, 7]
constexpr int CW3 = 6;          // the 4^3 level with a zero border
template <typename T>
struct Coefs {  // of the 16^3 and the 8^3 level
  T c0inv4, c04, ce4, cc4, c03, ce3, cc3;
  const T *table4, *table3;  // face rows, 216 each
  const T* inv;              // 64 x 64
};
constexpr int kWords = z16::TILE + z16::kCTile + 1000 + 512 + WE * WE * WE + WR * WR * WR + 64 +
                       CW3 * CW3 * CW3 + 64 * kInvStride + 432;

// the 8 colours of an 8^3 sweep by threads 0..63 (two warps, their own barrier)
template <typename T, bool FWD>
__device__ __forceinline__ void sweep8(T* tile, const T* fs, const T* ftab, T c0, T ce, T cc, int t) {
  using G = Geo<8>;
  constexpr int H = G::H, H3 = G::H3, C = G::C, C3 = G::C3, LOGC = G::LOGC;
  const int li = t & (C - 1), lj = (t >> LOGC) & (C - 1), lk = t >> (2 * LOGC);
#pragma unroll
  for (int step = 0; step < 8; ++step) {
    const int col = FWD ? step : 7 - step;
    const int cx = col & 1, cy = (col >> 1) & 1, cz = col >> 2;
    const int own = (1 - cx) | ((1 - cy) << 1) | ((1 - cz) << 2);
    const int pos = ((lk + cz) * H + (lj + cy)) * H + (li + cx);
    const int mask = ((cx == 0 && li == 0) ? 1 : 0) | ((cy == 0 && lj == 0) ? 2 : 0) | ((cz == 0 && lk == 0) ? 4 : 0);
    const T nv = relax_colour<T, 8>(tile, own, cx, cy, cz, pos, mask, fs[col * C3 + t], c0, ce, cc, ftab);
    tile[own * H3 + pos] = nv;
    asm volatile("bar.sync 1, 64;" ::: "memory");
  }
}

template <typename T>
__global__ void __launch_bounds__(NT, 1) k_coarse_tail(const T* __restrict__ f, T* __restrict__ e, Coefs<T> k) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);  // 16^3 level: its tile, then its residual
  T* ctile = tile + z16::TILE;               // the 8^3 level with a one-node border, natural
  T* tile3 = ctile + z16::kCTile;            // 8^3 level: parity-split tile
  T* fs3 = tile3 + 1000;                     // its right-hand side, colour-major
  T* et3 = fs3 + 512;                        // natural tiles of its residual
  T* rt3 = et3 + WE * WE * WE;
  T* f2 = rt3 + WR * WR * WR;                // 4^3 level: right-hand side
  T* ctile3 = f2 + 64;                       // and solution with a zero border
  T* inv = ctile3 + CW3 * CW3 * CW3;
  T* tab4 = inv + 64 * kInvStride;
  T* tab3 = tab4 + 216;
  f = cloud_slice(f, 4096);
  e = cloud_slice(e, 4096);
  const int t = threadIdx.x;
  const z16::Seg<ZT> g(t);
  int qx, qy;
  z16::quad_of(t / z16::Zt<ZT>::SEG, qx, qy);
  const int x0 = 2 * qx, y0 = 2 * qy;
  const uint32_t mq = s16::sp4(x0) | (s16::sp4(y0) << 1);
  T fv[ZT][4], v[ZT][4];
#pragma unroll
  for (int p = 0; p < ZT; ++p) {
    const typename s16::Vec4<T>::type q = s16::ld4(f + (mq | (s16::sp4(g.z(p)) << 2)));
    fv[p][0] = q.x; fv[p][1] = q.y; fv[p][2] = q.z; fv[p][3] = q.w;
    v[p][0] = v[p][1] = v[p][2] = v[p][3] = (T)0;
  }
  for (int i = t; i < 64 * 64; i += NT) inv[(i >> 6) * kInvStride + (i & 63)] = k.inv[i];
  for (int i = t; i < 216; i += NT) {
    tab4[i] = k.table4[i];
    tab3[i] = k.table3[i];
  }
  // everything outside the domain is zero, and the sweeps start from zero
  for (int i = t; i < z16::TILE; i += NT) tile[i] = 0;
  for (int i = t; i < z16::kCTile; i += NT) ctile[i] = 0;
  for (int i = t; i < 1000; i += NT) tile3[i] = 0;
  for (int i = t; i < WE * WE * WE; i += NT) et3[i] = 0;
  for (int i = t; i < WR * WR * WR; i += NT) rt3[i] = 0;
  for (int i = t; i < CW3 * CW3 * CW3; i += NT) ctile3[i] = 0;
  __syncthreads();

  // 16^3: pre-smoothing from zero
  g16::sweep<T, true, true, true, ZT>(tile, tab4, true, 0, 0, 0, x0, y0, g, fv, v, k.ce4, k.cc4, k.c0inv4);
  {  // r = f - A a takes a's place in the tile (the threads keep a)
    T r[ZT][4];
    z16::stencil_rows<ZT, T>(tile, x0, y0, g, v, k.c04, k.ce4, k.cc4, r);
#pragma unroll
    for (int p = 0; p < ZT; ++p)
#pragma unroll
      for (int i = 0; i < 4; ++i) r[p][i] = fv[p][i] - r[p][i];
    r16::face_residual<ZT>(tile, tab4, 0, 0, 0, x0, y0, g, k.c04, k.ce4, k.cc4, r);
    __syncthreads();
    z16::store_quad<ZT>(tile, x0, y0, g, r);
  }
  __syncthreads();
  uint32_t nx, ny, nz;  // this thread's 8^3 node (Morton t)
  unmorton3((uint32_t)t, nx, ny, nz);
  const int ux = (int)nx + 1, uy = (int)ny + 1, uz = (int)nz + 1;
  {
    const T s = r16::restrict_own<T>(tile, (int)nx, (int)ny, (int)nz);
    const int col = (nx & 1) | ((ny & 1) << 1) | ((nz & 1) << 2);
    fs3[col * 64 + ((nx >> 1) | ((ny >> 1) << 2) | ((nz >> 1) << 4))] = s;
    rt3[(uz * WR + uy) * WR + ux] = s;  // f first, r = f - A a below
  }
  __syncthreads();

  // 8^3: pre-smoothing from zero, residual, restriction
  if (t < 64) sweep8<T, true>(tile3, fs3, tab3, k.c03, k.ce3, k.cc3, t);
  __syncthreads();
  const int self3 = ps_index<8>(ux, uy, uz);
  const T a3 = tile3[self3];
  et3[((uz + 1) * WE + (uy + 1)) * WE + (ux + 1)] = a3;
  __syncthreads();
  {
    const int ei = ((uz + 1) * WE + (uy + 1)) * WE + (ux + 1), ri = (uz * WR + uy) * WR + ux;
    column_apply<T, WE, 1>(et3, ux + 1, uy + 1, uz + 1, k.c03, k.ce3, k.cc3, [&](int, T, T y) { rt3[ri] -= y; });
    const int mask = (nx == 0) | ((ny == 0) << 1) | ((nz == 0) << 2);
    if (mask) {
      const T yi = row_interior<T, WE>(et3, ei, k.c03, k.ce3, k.cc3);
      const T yf = row_general<T, WE>(et3, ei, tab3 + 27 * mask);
      rt3[ri] += yi - yf;
    }
  }
  __syncthreads();
  if (t < 64) {
    uint32_t cx, cy, cz;
    unmorton3((uint32_t)t, cx, cy, cz);
    f2[t] = restrict_full<T, WR>(rt3, (int)cx, (int)cy, (int)cz);
    asm volatile("bar.sync 1, 64;" ::: "memory");
    // 4^3: the dense inverse
    double s = 0.0;
#pragma unroll 16
    for (int j = 0; j < 64; ++j) s += (double)inv[t * kInvStride + j] * (double)f2[j];
    ctile3[((cz + 1) * CW3 + (cy + 1)) * CW3 + (cx + 1)] = (T)s;
  }
  __syncthreads();

  // 8^3: post-smoothing on a + P e
  T v3 = a3;
  v3 += prolong_node<T, CW3>(ctile3, (int)nx, (int)ny, (int)nz, -1, -1, -1);
  tile3[self3] = v3;
  __syncthreads();
  if (t < 64) sweep8<T, false>(tile3, fs3, tab3, k.c03, k.ce3, k.cc3, t);
  __syncthreads();
  ctile[z16::coarse_at((int)nx, (int)ny) + (int)nz] = tile3[self3];
  __syncthreads();

  // 16^3: post-smoothing on a + P e
  z16::prolong_quads<ZT>(ctile, qx, qy, g, v);
  z16::store_quad<ZT>(tile, x0, y0, g, v);
  __syncthreads();
  g16::sweep<T, false, false, true, ZT>(tile, tab4, true, 0, 0, 0, x0, y0, g, fv, v, k.ce4, k.cc4, k.c0inv4);
#pragma unroll
  for (int p = 0; p < ZT; ++p) {
    typename s16::Vec4<T>::type o;
    o.x = v[p][0]; o.y = v[p][1]; o.z = v[p][2]; o.w = v[p][3];
    s16::st4(e + (mq | (s16::sp4(g.z(p)) << 2)), o);
  }
}
}  // namespace t4

template <typename T>
DevCoef<T> dev_coef(const LevelCoef& L, const T* table) {
  DevCoef<T> k;
  k.c0 = (T)L.c0;
  k.ce = (T)L.ce;
  k.cc = (T)L.cc;
  k.table = table;
  k.has_faces = L.has_faces ? 1 : 0;
  return k;
}

inline int tile_for(uint32_t D) { return D >= 4 ? 16 : 8; }

template <typename T, int TB, int MODE, bool DOT, bool FWD>
void launch_smooth(cudaStream_t s, uint32_t D, const T* xi, T* xo, const T* f, const T* ec, const DevCoef<T>& k,
                   double* part, uint32_t clouds) {
  using G = Geo<TB>;
  constexpr int CW = TB / 2 + 2;
  const size_t sm = sizeof(T) * (G::W * G::W * G::W + G::N + (MODE == 2 ? CW * CW * CW : 0));
  const unsigned nb = 1u << (3 * (D - (TB == 16 ? 4 : 3)));
  allow_smem(k_smooth<T, TB, MODE, DOT, FWD>, sm);
  k_smooth<T, TB, MODE, DOT, FWD><<<dim3(nb, clouds), G::THREADS, sm, s>>>(D, xi, xo, f, ec, k, part);
}

template <typename T, int TB>
void smooth_dispatch(cudaStream_t s, uint32_t D, const T* xi, T* xo, const T* f, const T* ec, const DevCoef<T>& k,
                     int mode, bool forward, double* part, uint32_t clouds) {
#define PR_SM(M, DT, FW) launch_smooth<T, TB, M, DT, FW>(s, D, xi, xo, f, ec, k, part, clouds)
  if (mode == 1) {
    if (forward) PR_SM(1, false, true);
    else PR_SM(1, false, false);
  } else if (mode == 2) {
    if (part) {
      if (forward) PR_SM(2, true, true);
      else PR_SM(2, true, false);
    } else {
      if (forward) PR_SM(2, false, true);
      else PR_SM(2, false, false);
    }
  } else {
    if (part) {
      if (forward) PR_SM(0, true, true);
      else PR_SM(0, true, false);
    } else {
      if (forward) PR_SM(0, false, true);
      else PR_SM(0, false, false);
    }
  }
#undef PR_SM
}

// ------------------------------------------------------------------ the z-segment autotuner
// The 16^3 block kernels (SpMV, residual + restriction, smoother) run with ZT = 2 or 4 planes per
// thread, i.e. 512 or 256 threads per 16^3 brick: 4 planes move a column in 16-byte accesses (faster
// on large levels by 20-30%), 2 put twice the warps on a level of few bricks.  Both compute the same
// values (per-block sums in a fixed order), so the choice is free and made by timing: the first FP32
// launch of a (kernel family, level, launch size, with or without face rows: the same level is one
// solve's finest and another's coarse) key times both (one warm-up and three timed launches on the
// launch's own buffers; every candidate writes what the real launch then overwrites) and keeps the
// faster for the process.  FP64 launches and launches inside a stream capture use ZT = 4.
// PR_AUTOTUNE=0 fixes ZT = 4; PR_ZT=2|4 forces one (8, an earlier shape, means 4).
enum TuneFamily { kTuneSpmv = 0, kTuneResid = 1, kTuneSmooth = 2, kTuneSmoothPost = 3 };
struct TuneTable {
  std::mutex mu;
  std::map<std::tuple<int, int, int, int, bool>, int> zt;  // (device, family, level, log2 blocks, faces) -> ZT
  std::string log;
};
TuneTable& tune_table() {
  static TuneTable* t = new TuneTable();  // never destroyed
  return *t;
}
const char* family_name(int f) {
  return f == kTuneSpmv ? "spmv16" : (f == kTuneResid ? "resid16" : (f == kTuneSmooth ? "smooth16" : "smooth16-post"));
}
// PR_ZT_<FAMILY> (e.g. PR_ZT_SPMV16), else PR_ZT, forces a choice; read at every launch, so that a
// process may switch
int forced_zt(int family) {
  auto choice = [](const char* v) {
    const int z = v ? std::atoi(v) : 0;
    return z == 8 ? 4 : (z == 2 || z == 4 ? z : 0);
  };
  char name[32];
  std::snprintf(name, sizeof(name), "PR_ZT_%s", family == kTuneSpmv ? "SPMV16" : (family == kTuneResid ? "RESID16" : "SMOOTH16"));
  // (both smoother families answer to PR_ZT_SMOOTH16)
  if (const int z = choice(std::getenv(name))) return z;
  if (const int z = choice(std::getenv("PR_ZT"))) return z;
  const char* a = std::getenv("PR_AUTOTUNE");
  return (a && std::atoi(a) == 0) ? 4 : 0;
}

// Runs launch(zt) with the ZT of the key, timing the candidates first for a new key.
template <typename L>
void tuned_launch(cudaStream_t s, int family, uint32_t level, uint64_t blocks, bool faces, bool tunable, L launch) {
  if (!tunable) {
    launch(4);
    return;
  }
  if (const int f = forced_zt(family)) {
    launch(f);
    return;
  }
  int dev = 0;
  PR_CUDA(cudaGetDevice(&dev));
  int bin = 0;
  while ((2ull << bin) <= blocks) ++bin;
  const auto key = std::make_tuple(dev, family, (int)level, bin, faces);
  TuneTable& tt = tune_table();
  {
    std::lock_guard<std::mutex> g(tt.mu);
    auto it = tt.zt.find(key);
    if (it != tt.zt.end()) {
      launch(it->second);
      return;
    }
  }
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  PR_CUDA(cudaStreamIsCapturing(s, &cs));
  if (cs != cudaStreamCaptureStatusNone) {
    launch(4);
    return;
  }
  cudaEvent_t e0, e1;
  PR_CUDA(cudaEventCreate(&e0));
  PR_CUDA(cudaEventCreate(&e1));
  const int cand[2] = {2, 4};
  float ms[2];
  for (int k = 0; k < 2; ++k) {
    launch(cand[k]);
    PR_CUDA(cudaEventRecord(e0, s));
    for (int r = 0; r < 3; ++r) launch(cand[k]);
    PR_CUDA(cudaEventRecord(e1, s));
    PR_CUDA(cudaEventSynchronize(e1));
    PR_CUDA(cudaEventElapsedTime(&ms[k], e0, e1));
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  const int best = ms[0] < ms[1] ? 0 : 1;
  {
    std::lock_guard<std::mutex> g(tt.mu);
    tt.zt[key] = cand[best];
    char line[200];
    std::snprintf(line, sizeof(line), "%s level %u%s blocks 2^%d: ZT 2/4 = %.4f/%.4f ms -> ZT %d\n",
                  family_name(family), level, faces ? " (faces)" : "", bin, ms[0] / 3, ms[1] / 3, cand[best]);
    tt.log += line;
  }
  launch(cand[best]);
}

template <typename T, int MODE, bool DOT, bool FWD, bool FACES>
void launch_s16(cudaStream_t s, uint32_t D, const T* xi, T* xo, const T* f, const T* ec, const LevelCoef& L,
                const T* table, double* part, uint32_t clouds) {
  const size_t sm = g16::smem_bytes<T>(MODE);
  const dim3 grid(1u << (3 * (D - 4)), clouds);
  auto go = [&](auto z) {
    constexpr int ZT = decltype(z)::value;
    allow_smem(g16::k_smooth16<T, MODE, DOT, FWD, FACES, ZT>, sm);
    g16::k_smooth16<T, MODE, DOT, FWD, FACES, ZT><<<grid, n16::Zt<ZT>::NT, sm, s>>>(
        D, xi, xo, f, ec, (T)(1.0 / L.c0), (T)L.ce, (T)L.cc, table, part, CgFuse<T>());
  };
  constexpr bool kTunable = std::is_same<T, float>::value && MODE != 0;
  tuned_launch(s, MODE == 2 ? kTuneSmoothPost : kTuneSmooth, D, (uint64_t)grid.x * grid.y, FACES, kTunable, [&](int zt) {
    if constexpr (kTunable) {
      if (zt == 2) return go(std::integral_constant<int, 2>());
    }
    go(std::integral_constant<int, 4>());
  });
}

template <typename T, int MODE, bool DOT, bool FWD>
void launch_s16f(cudaStream_t s, uint32_t D, const T* xi, T* xo, const T* f, const T* ec, const LevelCoef& L,
                 const T* table, double* part, uint32_t clouds) {
  if (L.has_faces) launch_s16<T, MODE, DOT, FWD, true>(s, D, xi, xo, f, ec, L, table, part, clouds);
  else launch_s16<T, MODE, DOT, FWD, false>(s, D, xi, xo, f, ec, L, table, part, clouds);
}

template <typename T>
void smooth16_dispatch(cudaStream_t s, const LevelCoef& L, uint32_t D, const T* xi, T* xo, const T* f, const T* ec,
                       const T* table, int mode, bool forward, double* part, uint32_t clouds) {
#define PR_S16(M, DT, FW) launch_s16f<T, M, DT, FW>(s, D, xi, xo, f, ec, L, table, part, clouds)
  if (mode == 1) {
    if (forward) PR_S16(1, false, true);
    else PR_S16(1, false, false);
  } else if (mode == 2) {
    if (part) {
      if (forward) PR_S16(2, true, true);
      else PR_S16(2, true, false);
    } else {
      if (forward) PR_S16(2, false, true);
      else PR_S16(2, false, false);
    }
  } else {
    if (part) {
      if (forward) PR_S16(0, true, true);
      else PR_S16(0, true, false);
    } else {
      if (forward) PR_S16(0, false, true);
      else PR_S16(0, false, false);
    }
  }
#undef PR_S16
}

}  // namespace

// ====================================================================== host side
LevelCoef level_coef(uint32_t D, uint32_t l, double shift_l) {
  // 1-D Galerkin recurrence (p^T m p for the linear prolongation p), from the fine level:
  //   interior diagonal m0 -> 1.5 m0 + 2 m1, off-diagonal m1 -> m1 + m0/4,
  //   node-0 diagonal  mb -> mb + m1 + m0/4  (the fine node -1 does not exist)
  double m0 = 2.0 / 3.0, m1 = 1.0 / 6.0, mb = 2.0 / 3.0;
  double s0 = 2.0, s1 = -1.0, sb = 2.0;
  for (uint32_t k = D; k > l; --k) {
    const double nm0 = 1.5 * m0 + 2.0 * m1, nm1 = m1 + 0.25 * m0, nmb = mb + m1 + 0.25 * m0;
    const double ns0 = 1.5 * s0 + 2.0 * s1, ns1 = s1 + 0.25 * s0, nsb = sb + s1 + 0.25 * s0;
    m0 = nm0;
    m1 = nm1;
    mb = nmb;
    s0 = ns0;
    s1 = ns1;
    sb = nsb;
  }
  const double H = 1.0 / (double)(1u << D);
  LevelCoef L;
  L.depth = l;
  L.shift = shift_l;
  auto M = [&](int d, bool b) { return d == 0 ? (b ? mb : m0) : m1; };
  auto S = [&](int d, bool b) { return d == 0 ? (b ? sb : s0) : s1; };
  for (int mask = 0; mask < 8; ++mask)
    for (int o = 0; o < 27; ++o) {
      const int dx = o % 3 - 1, dy = (o / 3) % 3 - 1, dz = o / 9 - 1;
      const bool bxm = mask & 1, bym = mask & 2, bzm = mask & 4;
      double v = H * (S(dx, bxm) * M(dy, bym) * M(dz, bzm) + M(dx, bxm) * S(dy, bym) * M(dz, bzm) +
                      M(dx, bxm) * M(dy, bym) * S(dz, bzm));
      if (o == 13) v += shift_l;
      L.table[mask][o] = v;
    }
  // interior values by offset class, o = (dx+1) + 3(dy+1) + 9(dz+1)
  L.c0 = L.table[0][13];
  L.ce = L.table[0][2 + 3 * 2 + 9 * 1];  // (1,1,0)
  L.cc = L.table[0][2 + 3 * 2 + 9 * 2];  // (1,1,1)
  L.cf = L.table[0][2 + 3 * 1 + 9 * 1];  // (1,0,0): 0 in exact arithmetic
  if (std::fabs(L.cf) > 1e-12 * std::fabs(L.c0))
    throw Error(PR_ERR_INTERNAL, "multigrid level has a non-zero interior face coupling");
  L.cf = 0.0;
  for (int mask = 0; mask < 8; ++mask)
    for (int o = 0; o < 27; ++o)
      if (std::fabs(L.table[mask][o]) <= 1e-12 * std::fabs(L.c0)) L.table[mask][o] = 0.0;
  L.has_faces = (l < D);
  return L;
}

template <typename T>
void mg_smooth(cudaStream_t s, const LevelCoef& L, const T* table, const T* xi, T* xo, const T* f, const T* ec,
               int mode, bool forward, double* part, uint32_t clouds) {
  const uint32_t D = L.depth;
  const DevCoef<T> k = dev_coef<T>(L, table);
  if (tile_for(D) == 16) smooth16_dispatch<T>(s, L, D, xi, xo, f, ec, table, mode, forward, part, clouds);
  else smooth_dispatch<T, 8>(s, D, xi, xo, f, ec, k, mode, forward, part, clouds);
  PR_CHECK_LAUNCH();
}

template <typename T>
void mg_cg_update_presmooth(cudaStream_t s, const LevelCoef& L, const T* table, const CgFuse<T>& cg, T* xo,
                            double* part, uint32_t clouds) {
  const uint32_t D = L.depth;
  if (D < 4 || L.has_faces) throw Error(PR_ERR_INTERNAL, "the fused CG update needs the finest level, depth >= 4");
  const size_t sm = g16::smem_bytes<T>(3);
  const dim3 grid(1u << (3 * (D - 4)), clouds);
  auto go = [&](auto z) {
    constexpr int ZT = decltype(z)::value;
    allow_smem(g16::k_smooth16<T, 3, false, true, false, ZT>, sm);
    g16::k_smooth16<T, 3, false, true, false, ZT><<<grid, n16::Zt<ZT>::NT, sm, s>>>(
        D, nullptr, xo, nullptr, nullptr, (T)(1.0 / L.c0), (T)L.ce, (T)L.cc, table, part, cg);
  };
  // in place (x and r), so not timed: ZT = 4 unless forced
  const int zt = std::is_same<T, float>::value && forced_zt(kTuneSmooth) ? forced_zt(kTuneSmooth) : 4;
  if constexpr (std::is_same<T, float>::value) {
    if (zt == 2) go(std::integral_constant<int, 2>());
    else go(std::integral_constant<int, 4>());
  } else {
    go(std::integral_constant<int, 4>());
  }
  PR_CHECK_LAUNCH();
}

template <typename T>
void mg_resid_restrict(cudaStream_t s, const LevelCoef& L, const T* table, const T* e, const T* f, T* fc, T* face,
                       uint32_t clouds) {
  const uint32_t D = L.depth;
  const DevCoef<T> k = dev_coef<T>(L, table);
  if (tile_for(D) == 16) {
    const size_t sm = r16::smem_bytes<T>();
    const unsigned nb = 1u << (3 * (D - 4));
    auto go = [&](auto z, auto fcs) {
      constexpr int ZT = decltype(z)::value;
      constexpr bool FC = decltype(fcs)::value;
      allow_smem(r16::k_resid16<T, FC, ZT>, sm);
      r16::k_resid16<T, FC, ZT><<<dim3(nb, clouds), n16::Zt<ZT>::NT, sm, s>>>(D, e, f, fc, face, (T)L.c0, (T)L.ce,
                                                                              (T)L.cc, table);
    };
    auto go_f = [&](auto z) {
      if (L.has_faces) go(z, std::true_type());
      else go(z, std::false_type());
    };
    constexpr bool kTunable = std::is_same<T, float>::value;
    tuned_launch(s, kTuneResid, D, (uint64_t)nb * clouds, L.has_faces, kTunable, [&](int zt) {
      if constexpr (kTunable) {
        if (zt == 2) return go_f(std::integral_constant<int, 2>());
      }
      go_f(std::integral_constant<int, 4>());
    });
    PR_CHECK_LAUNCH();
    r16::k_restrict_faces<T><<<dim3((nb + 3) / 4, clouds), 768, 0, s>>>(D, face, fc, nb);
  } else {
    const size_t sm = sizeof(T) * (11 * 11 * 11 + 9 * 9 * 9);
    allow_smem(k_resid_restrict<T, 8>, sm);
    k_resid_restrict<T, 8><<<dim3(1u << (3 * (D - 3)), clouds), Geo<8>::THREADS, sm, s>>>(D, e, f, fc, k);
  }
  PR_CHECK_LAUNCH();
}

template <typename T>
void mg_coarse_tail(cudaStream_t s, const LevelCoef& L4, const LevelCoef& L3, const T* table4, const T* table3,
                    const T* inv, const T* f, T* e, uint32_t clouds) {
  if (L4.depth != 4 || L3.depth != 3 || !L4.has_faces || !L3.has_faces)
    throw Error(PR_ERR_INTERNAL, "the coarse tail starts at a coarse 16^3 level");
  t4::Coefs<T> k;
  k.c0inv4 = (T)(1.0 / L4.c0);
  k.c04 = (T)L4.c0;
  k.ce4 = (T)L4.ce;
  k.cc4 = (T)L4.cc;
  k.c03 = (T)L3.c0;
  k.ce3 = (T)L3.ce;
  k.cc3 = (T)L3.cc;
  k.table4 = table4;
  k.table3 = table3;
  k.inv = inv;
  const size_t sm = t4::kWords * sizeof(T);
  allow_smem(t4::k_coarse_tail<T>, sm);
  t4::k_coarse_tail<T><<<dim3(1, clouds), t4::NT, sm, s>>>(f, e, k);
  PR_CHECK_LAUNCH();
}

size_t mg_face_entries(uint32_t D) { return D >= 4 ? (size_t)r16::FACE << (3 * (D - 4)) : 0; }

template <typename T>
void mg_spmv(cudaStream_t s, const LevelCoef& L, const T* table, const T* z, const T* d, T* dn, double beta,
             bool xpby, T* q, double* part, uint32_t clouds, const double* beta_dev) {
  const uint32_t D = L.depth;
  const DevCoef<T> k = dev_coef<T>(L, table);
  if (L.has_faces) throw Error(PR_ERR_INTERNAL, "mg_spmv is for the finest level");
  if (tile_for(D) == 16) {
    const dim3 g(1u << (3 * (D - 4)), clouds);
    const size_t sm = n16::smem_bytes<T>();
    auto go = [&](auto zc) {
      constexpr int ZT = decltype(zc)::value;
      if (xpby) {
        allow_smem(n16::k_spmv16<T, 1, T, ZT>, sm);
        n16::k_spmv16<T, 1, T, ZT><<<g, n16::Zt<ZT>::NT, sm, s>>>(D, d, z, dn, (T)beta, q, (T)L.c0, (T)L.ce,
                                                                  (T)L.cc, nullptr, part, beta_dev);
      } else {
        allow_smem(n16::k_spmv16<T, 0, T, ZT>, sm);
        n16::k_spmv16<T, 0, T, ZT><<<g, n16::Zt<ZT>::NT, sm, s>>>(D, d, nullptr, nullptr, (T)0, q, (T)L.c0,
                                                                  (T)L.ce, (T)L.cc, nullptr, part, nullptr);
      }
    };
    constexpr bool kTunable = std::is_same<T, float>::value;
    tuned_launch(s, kTuneSpmv, D, (uint64_t)g.x * g.y, false, kTunable, [&](int zt) {
      if constexpr (kTunable) {
        if (zt == 2) return go(std::integral_constant<int, 2>());
      }
      go(std::integral_constant<int, 4>());
    });
  } else {
    if (clouds != 1 || beta_dev) throw Error(PR_ERR_INTERNAL, "packed SpMV needs depth >= 4");
    const unsigned nb = 1u << (3 * (D - 3));
    const size_t sm = sizeof(T) * (10 * 10 * 10 + 512);
    if (xpby) k_spmv<T, 8, true><<<nb, Geo<8>::THREADS, sm, s>>>(D, z, d, dn, (T)beta, q, k, part);
    else k_spmv<T, 8, false><<<nb, Geo<8>::THREADS, sm, s>>>(D, z, d, dn, (T)beta, q, k, part);
  }
  PR_CHECK_LAUNCH();
}

template <typename T>
void mg_apply(cudaStream_t s, const LevelCoef& L, const T* x, T* y) {
  const uint32_t D = L.depth;
  if (D < 4 || L.has_faces) throw Error(PR_ERR_INTERNAL, "mg_apply needs the finest level, depth >= 4");
  const size_t sm = n16::smem_bytes<T>();
  constexpr int ZT = 4;
  allow_smem(n16::k_spmv16<T, 3, T, ZT>, sm);
  n16::k_spmv16<T, 3, T, ZT><<<1u << (3 * (D - 4)), n16::Zt<ZT>::NT, sm, s>>>(
      D, x, nullptr, nullptr, (T)0, y, (T)L.c0, (T)L.ce, (T)L.cc, nullptr, nullptr, nullptr);
  PR_CHECK_LAUNCH();
}

template <typename E>
void mg_resid_update(cudaStream_t s, const LevelCoef& L, const double* x, const E* e, double scale, double* xn,
                     const double* b, double* r, uint32_t clouds, const double* scale_dev) {
  const uint32_t D = L.depth;
  if (D < 4 || L.has_faces) throw Error(PR_ERR_INTERNAL, "mg_resid_update needs the finest level, depth >= 4");
  const size_t sm = n16::smem_bytes<double>();
  allow_smem(n16::k_spmv16<double, 2, E, 4>, sm);
  n16::k_spmv16<double, 2, E, 4><<<dim3(1u << (3 * (D - 4)), clouds), n16::Zt<4>::NT, sm, s>>>(
      D, x, e, xn, scale, r, L.c0, L.ce, L.cc, b, nullptr, scale_dev);
  PR_CHECK_LAUNCH();
}
template void mg_resid_update<float>(cudaStream_t, const LevelCoef&, const double*, const float*, double, double*,
                                     const double*, double*, uint32_t, const double*);
template void mg_resid_update<double>(cudaStream_t, const LevelCoef&, const double*, const double*, double, double*,
                                      const double*, double*, uint32_t, const double*);

uint32_t mg_blocks(uint32_t D) { return tile_for(D) == 16 ? (1u << (3 * (D - 4))) : (1u << (3 * (D - 3))); }

void sum_parts(cudaStream_t s, const double* part, int np, double scale2, const double* part2, int np2, double* out,
               uint32_t clouds) {
  k_sum_parts<<<clouds, 1024, 0, s>>>(part, np, scale2, part2, np2, out);
  PR_CHECK_LAUNCH();
}

void cg_step(cudaStream_t s, CgStep step, const double* part, int np, double scale2, const double* part2, int np2,
             const CgScalars& cg, uint32_t clouds) {
  k_cg_step<<<clouds, 1024, 0, s>>>(step, part, np, scale2, part2, np2, cg);
  PR_CHECK_LAUNCH();
}

// ------------------------------------------------------------------ kernel micro-benchmark
namespace {
template <typename T>
__global__ void k_fill(T* __restrict__ x, uint64_t n, uint32_t seed) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t h = (uint32_t)i * 2654435761u ^ seed;
    h ^= h >> 15;
    h *= 2246822519u;
    h ^= h >> 13;
    x[i] = (T)((double)(h & 0xffffff) / 16777216.0 - 0.5);
  }
}

template <typename T>
double bench_one(pr_context* c, int kid, uint32_t D, int reps, double* bytes) {
  cudaStream_t s = c->stream;
  const uint64_t n = 1ull << (3 * D), nc = n / 8;
  const std::string tn = std::is_same<T, double>::value ? "f64" : "f32";
  T* x = c->buf<T>("kb_x_" + tn, n);
  T* y = c->buf<T>("kb_y_" + tn, n);
  T* f = c->buf<T>("kb_f_" + tn, n);
  T* w = c->buf<T>("kb_w_" + tn, n);
  T* ec = c->buf<T>("kb_c_" + tn, nc);
  T* face = c->buf<T>("kb_face_" + tn, std::max<size_t>(mg_face_entries(D), 1));
  T* r2 = c->buf<T>("kb_r_" + tn, n);
  double* part = c->buf<double>("kb_part", std::max<uint32_t>(mg_blocks(D), kDotBlocks));
  const unsigned g = 148 * 16;
  k_fill<T><<<g, 256, 0, s>>>(x, n, 1u);
  k_fill<T><<<g, 256, 0, s>>>(f, n, 2u);
  k_fill<T><<<g, 256, 0, s>>>(w, n, 3u);
  k_fill<T><<<g, 256, 0, s>>>(ec, nc, 4u);
  k_fill<T><<<g, 256, 0, s>>>(r2, n, 5u);
  PR_CHECK_LAUNCH();
  // the finest level (no low-face rows: the variants that dominate a solve) and, for ids 7-8,
  // a coarse level (low-face table rows)
  const LevelCoef Lf = level_coef(D, D, 0.0), Lc = level_coef(D + 1, D, 0.0);
  std::vector<T> tab(216);
  for (int m = 0; m < 8; ++m)
    for (int o = 0; o < 27; ++o) tab[27 * m + o] = (T)Lc.table[m][o];
  T* table = c->buf<T>("kb_tab_" + tn, 216);
  PR_CUDA(cudaMemcpyAsync(table, tab.data(), 216 * sizeof(T), cudaMemcpyHostToDevice, s));
  const double es = sizeof(T);
  auto run = [&]() {
    switch (kid) {
      case 0: mg_spmv<T>(s, Lf, table, nullptr, x, nullptr, 0.0, false, y, part); break;
      case 1: mg_spmv<T>(s, Lf, table, f, x, w, 0.5, true, y, part); break;
      case 2: mg_smooth<T>(s, Lf, table, nullptr, y, f, nullptr, 1, true, nullptr); break;
      case 3: mg_smooth<T>(s, Lf, table, x, y, f, nullptr, 0, true, nullptr); break;
      case 4: mg_smooth<T>(s, Lf, table, x, y, f, ec, 2, false, part); break;
      case 5: mg_resid_restrict<T>(s, Lf, table, x, f, ec, face); break;
      case 7: mg_smooth<T>(s, Lc, table, x, y, f, ec, 2, false, part); break;
      case 8: mg_resid_restrict<T>(s, Lc, table, x, f, ec, face); break;
      case 9: {  // CG update fused with the first pre-smoothing sweep: x += a d, r -= a q, y = S(r)
        CgFuse<T> cg;
        cg.x = w;
        cg.d = x;
        cg.q = f;
        cg.r = r2;
        cg.alpha = (T)1e-3;  // small: the reps leave r and the update bounded
        mg_cg_update_presmooth<T>(s, Lf, table, cg, y, part);
        break;
      }
      case 6: stencil_apply<T>(s, D, x, nullptr, y, cast_coef<T>(stencil_coef(D, 0.0)), 0); break;
      default: throw Error(PR_ERR_INVALID_ARGUMENT, "unknown kernel id");
    }
  };
  const double nb = (double)n * es;
  const double algo[] = {2 * nb, 4 * nb, 2 * nb, 3 * nb, 3 * nb + nb / 8, 2 * nb + nb / 8, 2 * nb,
                         3 * nb + nb / 8, 2 * nb + nb / 8, 7 * nb};
  if (kid < 0 || kid > 9) throw Error(PR_ERR_INVALID_ARGUMENT, "unknown kernel id");
  *bytes = algo[kid];
  run();
  PR_CUDA(cudaStreamSynchronize(s));
  cudaEvent_t e0, e1;
  PR_CUDA(cudaEventCreate(&e0));
  PR_CUDA(cudaEventCreate(&e1));
  PR_CUDA(cudaEventRecord(e0, s));
  for (int r = 0; r < reps; ++r) run();
  PR_CUDA(cudaEventRecord(e1, s));
  PR_CUDA(cudaEventSynchronize(e1));
  float ms = 0.f;
  PR_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return (double)ms / reps;
}
}  // namespace

std::string autotune_log() {
  TuneTable& tt = tune_table();
  std::lock_guard<std::mutex> g(tt.mu);
  return tt.log;
}

double kernel_bench(pr_context* c, int kid, uint32_t D, int precision, int reps, double* bytes) {
  if (D < 4 || D > kMaxDepth) throw Error(PR_ERR_INVALID_ARGUMENT, "kernel bench depth must be in [4, 10]");
  if (kid >= 20) return deg2_kernel_bench(c, kid - 20, D, precision, reps, bytes);
  if (reps < 1) reps = 1;
  return precision == PR_PRECISION_FP64 ? bench_one<double>(c, kid, D, reps, bytes)
                                        : bench_one<float>(c, kid, D, reps, bytes);
}

#define PR_INST(T)                                                                                                 \
  template void mg_smooth<T>(cudaStream_t, const LevelCoef&, const T*, const T*, T*, const T*, const T*, int, bool, \
                             double*, uint32_t);                                                                  \
  template void mg_apply<T>(cudaStream_t, const LevelCoef&, const T*, T*);                                        \
  template void mg_coarse_tail<T>(cudaStream_t, const LevelCoef&, const LevelCoef&, const T*, const T*, const T*,   \
                                  const T*, T*, uint32_t);                                                        \
  template void mg_resid_restrict<T>(cudaStream_t, const LevelCoef&, const T*, const T*, const T*, T*, T*,        \
                                     uint32_t);                                                                   \
  template void mg_cg_update_presmooth<T>(cudaStream_t, const LevelCoef&, const T*, const CgFuse<T>&, T*, double*, \
                                          uint32_t);                                                              \
  template void mg_spmv<T>(cudaStream_t, const LevelCoef&, const T*, const T*, const T*, T*, double, bool, T*,    \
                           double*, uint32_t, const double*);
PR_INST(float)
PR_INST(double)
#undef PR_INST

}  // namespace pr
