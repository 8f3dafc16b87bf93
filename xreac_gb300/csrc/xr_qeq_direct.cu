// QEq by a dense FP32 factorization under FP64 refinement, one thread block or one cluster per system.
//
// A system of up to kQeqDirectMax atoms has its whole matrix in one block's shared memory. The CG
// it would take otherwise needs 30 to 140 iterations of 2 to 7 us (two team reductions each).
// Measured, CG then direct: 192 atoms 293 -> 112 us, 9 atoms 61 -> 38 us, a batch of 192 systems of
// up to 64 atoms 179 -> 56 us. The KKT system of
// src/xreac/energy.py:95-102 is solved by iterative refinement, as the FP32 CG's sweeps are: each
// step solves H y = -g, sum y = 0 for the FP64 gradient g = H x + chi - lambda projected onto the
// constraint, adds y to the FP64 charges, restores sum x = Q and forms the gradient again in FP64
// from the unscaled entries. The FP64 gradient's norm is held against the CG solver's target. The last
// correction has no gradient after it: it is made from one that meets the target already, or from one that a step as
// good as the one before it would bring to a hundredth of the target (of the squared norms). A step cuts the squared
// norm by some 1e12, so that is the third as a rule, from a norm 1 to 30 times the target's, which a cut by 1e3
// would do too. A step that does not cut the squared norm by 1e3 (a singular or badly indefinite matrix, or one whose
// smallest eigenvalue FP32 does not resolve; the elimination does not pivot) leaves the system to the CG
// solver, which starts over.
//
// The matrix is held as 32 x 32 tiles of its lower block triangle, column-major (rows of a column
// contiguous), and factorized as L D L' with D the 32 x 32 diagonal blocks, whose inverses replace
// them: W_ik = A_ik D_k^-1 replaces A_ik, and A_ij -= W_ik A_jk'. Four warps update and invert the
// next diagonal block (Gauss-Jordan, a row per lane and eight columns per warp, in registers) while
// the others update the rest. A tile product is bound by shared-memory loads: each lane forms 4 x 8
// entries, so that 12 load wavefronts feed 32 multiply-adds.
//
// What bounds it: the chain of diagonal blocks (16 dependent pairs of pivots each), and for the gradients the
// FP64 pipe (an entry is one of its multiply-adds, two a clock).
#include <algorithm>

#include "xr_common.cuh"
#include "xr_qeq_direct.h"

namespace {

constexpr double SELF_CONVERSION = 23.02;
constexpr int kTile = 32, kTileSize = kTile * kTile;
constexpr int kMaxTiles = kQeqDirectMax / kTile;

__device__ inline double atom_prm(const double* atab, int t, int col) { return __ldg(atab + t * XR_NATOM_COLS + col); }

// Shared state of one solve besides the dynamic part (tiles, then per-row vectors).
struct DirectShared {
  double red[8][16];  // warp partials of a block sum
  double tot[8];
  float redf[2][16], totf[2];
  float column[4][kTile];  // the two pivot columns of an inversion, two steps' in turn
  unsigned short map[kMaxTiles * (kMaxTiles + 1) / 2 + kMaxTiles];  // tile (i, j) -> slot; then the scratch slots
};

// Sum over 2 from lanes (from = 16: the warp).
template <class T>
__device__ inline T lane_sum(T v, int from) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    if (o <= from) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums over the block of NV values of every thread with a row; warps without rows skip the shuffles (an
// FP64 instruction costs the pipe the same for idle lanes). Thread 0 runs post(totals) before the
// others see them: divisions done once. A fixed order, so the same on every call. Two block barriers.
template <int NV, class Post>
__device__ inline void block_sums(DirectShared& sh, double (&v)[NV], int rows, Post post) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (rows + 31) >> 5;
  if (wid < nw) {
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = lane_sum(v[k], 16);
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < NV; ++k) sh.red[k][wid] = v[k];
  }
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      v[k] = lane < nw ? sh.red[k][lane] : 0.0;
      if (nw > 1) v[k] = lane_sum(v[k], 8);
    }
    if (lane == 0) {
      post(v);
#pragma unroll
      for (int k = 0; k < NV; ++k) sh.tot[k] = v[k];
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = sh.tot[k];
}

// The same for two FP32 values.
__device__ inline float2 block_sums2f(DirectShared& sh, float a, float b, int rows) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (rows + 31) >> 5;
  if (wid < nw) {
    a = lane_sum(a, 16);
    b = lane_sum(b, 16);
    if (lane == 0) {
      sh.redf[0][wid] = a;
      sh.redf[1][wid] = b;
    }
  }
  __syncthreads();
  if (wid < 2) {
    const float t = lane_sum(lane < nw ? sh.redf[wid][lane] : 0.0f, 16);
    if (lane == 0) sh.totf[wid] = t;
  }
  __syncthreads();
  return make_float2(sh.totf[0], sh.totf[1]);
}

// c[r][q] of the product sum_k a(row, k) b(col, k) of two column-major tiles: rows 4 rg .. 4 rg + 3 and
// columns c0 + NC cg .. c0 + NC cg + NC - 1 for lane = rg + 8 cg (a whole tile with NC = 8, half of its columns
// with NC = 4).
template <int NC>
__device__ inline void tile_product(const float* a, const float* b, int c0, float (&c)[4][NC]) {
  const int rg = threadIdx.x & 7, cg = (threadIdx.x >> 3) & 3;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < NC; ++q) c[r][q] = 0.0f;
#pragma unroll 8
  for (int k = 0; k < kTile; ++k) {
    const float4 x = *reinterpret_cast<const float4*>(a + kTile * k + 4 * rg);
    const float xr[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int h = 0; h < NC; h += 4) {
      const float4 y = *reinterpret_cast<const float4*>(b + kTile * k + c0 + NC * cg + h);
      const float yc[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) c[r][h + q] += xr[r] * yc[q];
    }
  }
}

// Warps 0 to 3: tile t less the product of w and a (null: of nothing), replaced by its inverse. Gauss-Jordan
// without pivoting, two pivots at a time, lane = row, warp q holds columns 8 q .. 8 q + 7; the pivot columns go through
// shared memory, one barrier of the four warps and one reciprocal (of the 2 x 2 block's determinant) a pair. With one
// pivot at a time QEq took 234 us for 375 atoms (224), 174 for a 288-atom slab (167) and 116 for 192 atoms (112).
// A vanishing determinant gives non-finite entries, which the refinement notices. (By one warp, all 32 columns
// unrolled, an inversion took 11 us: 4,000 instructions do not fit the instruction cache.)
__device__ __noinline__ void tile_inverse(float* t, const float* w, const float* a, DirectShared& sh) {
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
  float v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) v[c] = t[kTile * (8 * q + c) + lane];
  if (w != nullptr) {
#pragma unroll 8
    for (int k = 0; k < kTile; ++k) {
      const float x = w[kTile * k + lane];
      const float4 y0 = *reinterpret_cast<const float4*>(a + kTile * k + 8 * q);
      const float4 y1 = *reinterpret_cast<const float4*>(a + kTile * k + 8 * q + 4);
      v[0] -= x * y0.x;
      v[1] -= x * y0.y;
      v[2] -= x * y0.z;
      v[3] -= x * y0.w;
      v[4] -= x * y1.x;
      v[5] -= x * y1.y;
      v[6] -= x * y1.z;
      v[7] -= x * y1.w;
    }
  }
  for (int cb = 0; cb < 4; ++cb) {
#pragma unroll
    for (int ci = 0; ci < 8; ci += 2) {
      const int c = 8 * cb + ci;
      float* const ca = sh.column[ci & 2];
      float* const cd = sh.column[(ci & 2) + 1];
      if (q == cb) {
        ca[lane] = v[ci];
        cd[lane] = v[ci + 1];
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      // the pivot block's rows times its inverse (p11 -p01; -p10 p00) / det
      const float2 pa = *reinterpret_cast<const float2*>(ca + c), pb = *reinterpret_cast<const float2*>(cd + c);
      const float inv = __fdividef(1.0f, pa.x * pb.y - pb.x * pa.y);
      const float x = ca[lane], y = cd[lane];
      const bool first = lane == c, second = lane == c + 1, own = first || second;
      const float fa = (first ? -pb.y : second ? pa.y : x * pb.y - y * pa.y) * inv;
      const float fb = (first ? pb.x : second ? -pa.x : y * pa.x - x * pb.x) * inv;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float p0 = __shfl_sync(0xffffffffu, v[j], c), p1 = __shfl_sync(0xffffffffu, v[j], c + 1);
        v[j] = (own ? 0.0f : v[j]) - fa * p0 - fb * p1;
      }
      if (q == cb) {
        v[ci] = -fa;
        v[ci + 1] = -fb;
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) t[kTile * (8 * q + c) + lane] = v[c];
}

__device__ inline int tile_at(int i, int j) { return i * (i + 1) / 2 + j; }

// The dynamic shared memory of a system of n atoms in T = ceil(n / 32) tile rows: the lower triangle's
// tiles and T - 1 scratch tiles, then per row the FP64 charges and gradient and two FP32 vectors.
struct DirectLayout {
  int T;
  float* tiles;
  double *X, *G;
  float *b, *w1;
  __device__ DirectLayout(unsigned char* dyn, int n) {
    T = (n + kTile - 1) / kTile;
    tiles = reinterpret_cast<float*>(dyn);
    X = reinterpret_cast<double*>(dyn + (size_t)4 * kTileSize * (T * (T + 1) / 2 + T - 1));
    G = X + kTile * T;
    b = reinterpret_cast<float*>(G + kTile * T);
    w1 = b + kTile * T;
  }
  __device__ float* tile(const DirectShared& sh, int i, int j) const { return tiles + kTileSize * sh.map[tile_at(i, j)]; }
};

__host__ __device__ constexpr size_t direct_bytes(int n) {
  const size_t T = (n + kTile - 1) / kTile;
  return 4 * (size_t)kTileSize * (T * (T + 1) / 2 + T - 1) + T * kTile * (2 * sizeof(double) + 2 * sizeof(float));
}

// Factorizes the assembled tiles in place (see the head of the file). At least eight warps, or four for
// one tile row.
__device__ __noinline__ void factorize(const DirectLayout& L, DirectShared& sh) {
  const int T = L.T, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int rg = threadIdx.x & 7, cg = (threadIdx.x >> 3) & 3;
  unsigned short* scratch = sh.map + T * (T + 1) / 2;  // scratch[i - 1]: slot for W_ik
  if (wid < 4) tile_inverse(L.tile(sh, 0, 0), nullptr, nullptr, sh);
  __syncthreads();
  for (int k = 0; k + 1 < T; ++k) {
    const int m = T - 1 - k;
    // W_ik = A_ik D_k^-1 (symmetric) into the scratch tiles, half a tile a warp
    for (int u = wid; u < 2 * m; u += nw) {
      const int i = k + 1 + (u >> 1), c0 = 16 * (u & 1);
      float c[4][4];
      tile_product<4>(L.tile(sh, i, k), L.tile(sh, k, k), c0, c);
      float* o = L.tiles + kTileSize * scratch[i - 1] + kTile * c0;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<float4*>(o + kTile * (4 * cg + q) + 4 * rg) = make_float4(c[0][q], c[1][q], c[2][q], c[3][q]);
    }
    __syncthreads();
    // A_ij -= W_ik A_jk': the next diagonal tile and its inverse by warps 0 to 3, the rest by the others
    if (wid < 4) {
      tile_inverse(L.tile(sh, k + 1, k + 1), L.tiles + kTileSize * scratch[k], L.tile(sh, k + 1, k), sh);
    } else {
      for (int u = wid - 3; u < m * (m + 1) / 2; u += nw - 4) {
        int i = 0, r = u;
        while (r > i) r -= ++i;
        const int ti = k + 1 + i, tj = k + 1 + r;
        float c[4][8];
        tile_product<8>(L.tiles + kTileSize * scratch[ti - 1], L.tile(sh, tj, k), 0, c);
        float* o = L.tile(sh, ti, tj);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          float4* d = reinterpret_cast<float4*>(o + kTile * (8 * cg + q) + 4 * rg);
          float4 v = *d;
          v.x -= c[0][q];
          v.y -= c[1][q];
          v.z -= c[2][q];
          v.w -= c[3][q];
          *d = v;
        }
      }
    }
    __syncthreads();
    if ((int)threadIdx.x >= k + 1 && (int)threadIdx.x < T) {  // W_ik takes A_ik's place, whose slot is free
      const int i = threadIdx.x, at = tile_at(i, k);
      const unsigned short s = sh.map[at];
      sh.map[at] = scratch[i - 1];
      scratch[i - 1] = s;
    }
    __syncthreads();
  }
}

// H^-1 v for the NV vectors v[k] (kTile T floats each), in place. Every step of a substitution is a
// thread per row and a block barrier.
template <int NV>
__device__ inline void substitute(const DirectLayout& L, const DirectShared& sh, float* const (&v)[NV]) {
  const int T = L.T, rows = kTile * T;
  for (int k = 0; k + 1 < T; ++k) {
    for (int r = kTile * (k + 1) + threadIdx.x; r < rows; r += blockDim.x) {
      const float* w = L.tile(sh, r >> 5, k) + (r & 31);
      float s[NV][2];
#pragma unroll
      for (int q = 0; q < NV; ++q) s[q][0] = s[q][1] = 0.0f;
#pragma unroll 8
      for (int c = 0; c < kTile; c += 2) {
        const float w0 = w[kTile * c], w1 = w[kTile * c + kTile];
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          s[q][0] += w0 * v[q][kTile * k + c];
          s[q][1] += w1 * v[q][kTile * k + c + 1];
        }
      }
#pragma unroll
      for (int q = 0; q < NV; ++q) v[q][r] -= s[q][0] + s[q][1];
    }
    __syncthreads();
  }
  float z[NV];  // (a block has at least as many threads as rows)
  const int r = threadIdx.x;
  if (r < rows) {
    const float* d = L.tile(sh, r >> 5, r >> 5) + (r & 31);
#pragma unroll
    for (int q = 0; q < NV; ++q) z[q] = 0.0f;
#pragma unroll 8
    for (int c = 0; c < kTile; ++c) {
      const float x = d[kTile * c];
#pragma unroll
      for (int q = 0; q < NV; ++q) z[q] += x * v[q][(r & ~31) + c];
    }
  }
  __syncthreads();
  if (r < rows)
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q][r] = z[q];
  __syncthreads();
  for (int k = T - 1; k > 0; --k) {
    if (r < kTile * k) {
      const float* w = L.tile(sh, k, r >> 5) + kTile * (r & 31);
      float s[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) s[q] = 0.0f;
#pragma unroll 8
      for (int t = 0; t < kTile; ++t) {
        const int c = (t + r) & 31;  // a lane starts at its own column: no two share a bank
        const float x = w[c];
#pragma unroll
        for (int q = 0; q < NV; ++q) s[q] += x * v[q][kTile * k + c];
      }
#pragma unroll
      for (int q = 0; q < NV; ++q) v[q][r] -= s[q];
    }
    __syncthreads();
  }
}

// One warp: add(j, h) for the entries [beg, end) of a row, in the local column j (FP32 h). The images of one j
// are adjacent and added one after the other, so the sums are the same on every call.
template <class Add>
__device__ inline void add_row(const XrWork& w, int a0, int n, int beg, int end, Add add) {
  const int lane = threadIdx.x & 31;
  int before = -1;
  for (int e0 = beg; e0 < end; e0 += 128) {
    int j[4];
    float h[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + 32 * u + lane;
      j[u] = e < end ? w.edge[e].x - a0 : n;
      h[u] = e < end ? w.qch[e] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (e0 + 32 * u >= end) break;  // uniform per warp
      int prev = __shfl_up_sync(0xffffffffu, j[u], 1);
      if (lane == 0) prev = before;
      before = __shfl_sync(0xffffffffu, j[u], 31);
      const unsigned first = __ballot_sync(0xffffffffu, j[u] != prev) & ((2u << lane) - 1u);
      const int rank = j[u] < n ? (first ? lane - (31 - __clz(first)) : lane) : -1;  // images of j before this one
      const int last = __reduce_max_sync(0xffffffffu, rank);
      for (int q = 0; q <= last; ++q) {
        if (rank == q) add(j[u], h[u]);
        __syncwarp();
      }
    }
  }
}

// G[q] = (H X)_row(q) in FP64 for q < m (the caller adds the diagonal and chi): a group of lanes per
// row, X (of the whole system) in shared memory.
template <class Row>
__device__ inline void product64(const XrWork& w, const double* X, double* G, int a0, int m, Row row) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, wid = threadIdx.x >> 5;
  int gs = 32;
  while (gs > 4 && m * gs > 4 * (int)blockDim.x) gs >>= 1;
  const int sub = lane & (gs - 1), gpw = 32 / gs;
  for (int qb = wid * gpw; qb < m; qb += nw * gpw) {  // uniform per warp
    const int q = qb + lane / gs;
    double s = 0.0;
    if (q < m) {
      const int r = row(q), ee = w.cnt[a0 + r + 1];
      int e = w.cnt[a0 + r] + sub;
      for (; e + 3 * gs < ee; e += 4 * gs) {
        int j[4];
        double h[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          j[u] = w.edge[e + u * gs].x - a0;
          h[u] = w.hval[e + u * gs];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) s += h[u] * X[j[u]];
      }
      for (; e < ee; e += gs) s += w.hval[e] * X[w.edge[e].x - a0];
    }
    for (int o = gs / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (sub == 0 && q < m) G[q] = s;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(512, 1) k_qeq_direct(XrWork w, XrFF ff, const int* list, int adjoint) {
  __shared__ DirectShared sh;
  extern __shared__ __align__(16) unsigned char dyn[];
  const int sys = list[blockIdx.x];
  const XrSystem& S = w.sys[sys];
  const int a0 = S.atom_off, n = S.natoms, tid = threadIdx.x, wid = tid >> 5, nw = blockDim.x >> 5;
  const double* atab = xr_ff_at(ff, ff.nsets > 1 ? S.ff_set : 0).atom;
  const double Q = adjoint ? 0.0 : S.total_charge;
  const bool warm = !adjoint && S.has_guess != 0;
  const double x0 = Q == 0.0 ? 0.0 : Q / n;
  const DirectLayout L(dyn, n);
  const int T = L.T, rows = kTile * T, ntri = T * (T + 1) / 2;
  const int r = tid, a = a0 + min(r, n - 1), type = w.type[a];
  const bool row = r < n;
  const double eta = atom_prm(atab, type, A_ETA), chi = adjoint ? w.qrhs[a] : atom_prm(atab, type, A_CHI);
  // 1. The tiles: zeros, the hardness (padding: ones) on the diagonal, then the rows' entries.
  for (int k = tid; k < ntri * kTileSize / 4; k += blockDim.x) reinterpret_cast<float4*>(L.tiles)[k] = make_float4(0, 0, 0, 0);
  for (int k = tid; k < ntri + T - 1; k += blockDim.x) sh.map[k] = (unsigned short)k;
  if (r < rows) {
    L.X[r] = row ? (warm ? w.qguess[a] : x0) : 0.0;
    L.G[r] = 0.0;
  }
  __syncthreads();
  if (r < rows) L.tiles[kTileSize * tile_at(r >> 5, r >> 5) + (kTile + 1) * (r & 31)] = row ? (float)eta : 1.0f;
  __syncthreads();
  // Row i's last entries, as many as it has half edges, are those with j > i and one direction of its
  // self images; (j, i) lies in the lower triangle, whose rows j are contiguous.
  const int* const half = w.cnt + (w.A + 1) + a0;
  for (int i = wid; i < n; i += nw) {
    add_row(w, a0, n, w.cnt[a0 + i + 1] - (half[i + 1] - half[i]), w.cnt[a0 + i + 1], [&](int j, float h) {
      float* const t = L.tiles + kTileSize * tile_at(j >> 5, i >> 5);
      if (j == i) {
        t[(kTile + 1) * (i & 31)] += 2.0f * h;
      } else {
        t[kTile * (i & 31) + (j & 31)] += h;
        if ((j >> 5) == (i >> 5)) t[kTile * (j & 31) + (i & 31)] += h;
      }
    });
  }
  // 2. The start gradient, projected: g - lambda with lambda = <D^-1, g> / <D^-1, 1>; the target is the
  //    tolerance times the norm <D^-1, g^2> at the uniform start, as in the CG solver.
  const bool product = warm || x0 != 0.0;
  if (product) {
    __syncthreads();
    product64(w, L.X, L.G, a0, n, [](int q) { return q; });
  } else {
    __syncthreads();
  }
  const double di = row ? 1.0 / (double)L.tiles[kTileSize * tile_at(r >> 5, r >> 5) + (kTile + 1) * (r & 31)] : 0.0;
  double g = row ? L.G[min(r, rows - 1)] + eta * L.X[min(r, rows - 1)] + chi : 0.0, gu = g;
  if (warm) {  // the uniform start's gradient
    gu = row ? chi : 0.0;
    if (x0 != 0.0) {
      const double x = row ? L.X[r] : 0.0;
      __syncthreads();
      if (row) L.X[r] = x0;
      __syncthreads();
      product64(w, L.X, L.G, a0, n, [](int q) { return q; });
      if (row) {
        gu = L.G[r] + eta * x0 + chi;
        L.X[r] = x;
      }
      __syncthreads();
    }
  }
  double v5[5] = {di, di * g, di * g * g, di * gu, di * gu * gu};
  block_sums<5>(sh, v5, n, [](double* t) {
    t[1] /= t[0];
    t[3] /= t[0];
    t[2] = 1e-28 * fmax(t[2], t[4]);
  });
  const double s1 = v5[0], gfloor = v5[2];
  if (row) {
    g -= v5[1];
    gu -= v5[3];
  }
  double v2[2] = {di * g * g, di * gu * gu};
  block_sums<2>(sh, v2, n, [&](double* t) { t[1] *= w.cg_tol * w.cg_tol; });
  double gz = v2[0];
  const double target = v2[1];
  // 3. Refinement steps. The last one needs no gradient after it: it starts from one that meets the
  //    target, or from one that a step like the one before it, which cut the squared norm to the
  //    fraction c (the same linear map), brings to a hundredth of the target.
  int steps = 0;
  bool failed = false, last = false;
  double x = row ? L.X[r] : 0.0;
  auto correct = [&]() {  // x += y, the solution of H y = -g on sum y = 0, then sum x = Q exactly
    if (r < rows) L.b[r] = row ? (float)-g : 0.0f;
    if (steps == 0) {
      if (r < rows) L.w1[r] = row ? 1.0f : 0.0f;
      factorize(L, sh);
      float* const both[2] = {L.b, L.w1};
      substitute<2>(L, sh, both);
    } else {
      __syncthreads();
      float* const one[1] = {L.b};
      substitute<1>(L, sh, one);
    }
    ++steps;
    const float b = row ? L.b[r] : 0.0f, w1 = row ? L.w1[r] : 0.0f;
    const float2 t = block_sums2f(sh, b, w1, n);
    if (row) x += (double)(b - t.x / t.y * w1);
    double sx[1] = {x};
    block_sums<1>(sh, sx, n, [&](double* t) { t[0] = (Q - t[0]) / n; });
    if (row) x += sx[0];
  };
  bool more = gz > target && gz > gfloor && n >= 2;
  while (more) {
    if (steps == 8 && !last) {
      failed = true;
      break;
    }
    correct();
    if (last) break;
    if (row) L.X[r] = x;
    __syncthreads();
    product64(w, L.X, L.G, a0, n, [](int q) { return q; });
    g = row ? L.G[r] + eta * x + chi : 0.0;
    double vl[1] = {di * g};
    block_sums<1>(sh, vl, n, [&](double* t) { t[0] /= s1; });
    if (row) g -= vl[0];
    double vg[2] = {di * g * g, 0.0};
    const double before = gz;
    block_sums<2>(sh, vg, n, [&](double* t) { t[1] = t[0] / before; });
    gz = vg[0];
    if (!(vg[1] <= 1e-3) && !(gz <= target)) {  // (also when it is not finite)
      failed = true;
      break;
    }
    last = gz <= target || vg[1] * gz <= 1e-2 * target;
    more = last || gz > gfloor;
  }
  if (failed) {  // the CG solver's (xr_launch_qeq_retry)
    if (tid == 0) {
      int* const retry = w.qretry + (adjoint ? 2 : 0);
      w.qretry[4 + (adjoint ? w.S : 0) + atomicAdd(retry, 1)] = sys;
    }
    return;
  }
  if (tid == 0) {
    atomicMax(w.counts + 4, steps);
    w.qiters[sys] = max(w.qiters[sys], steps);
  }
  if (!row) return;
  const double q = x;
  if (adjoint) {
    w.qadj[a] = q;
    return;
  }
  w.q[a] = q;
  w.a_e[(size_t)6 * w.A + a] = SELF_CONVERSION * (chi * q + 0.5 * eta * q * q);
}

// ------------------------------------------------------------------------------------ clusters
// Larger systems: the same solve by the blocks of one thread-block cluster. Tile row i belongs to
// block i mod nb; a block holds its rows' tiles (W_ik in place once known), a copy of the current
// panel's tiles A_ik of every row, and the vectors whole. Step k of the factorization: the blocks send
// their A_ik, and the owner of row k its D_k^-1, to every block; then each forms its W_ik and updates
// its rows, the owner of row k + 1 inverting that row's diagonal tile meanwhile. A substitution sends
// one tile of the vector a step (forward), or adds its product to the other rows' tiles at their
// owners (backward). All control flow is the same in every block (it depends on cluster-wide sums
// only), so the blocks meet at the hardware cluster barrier. Measured, CG then direct: 375 atoms 541 -> 224 us, a
// 288-atom periodic slab 420 -> 167 us; a batch of 128 requests of up to 512 atoms, all classes side
// by side, 1165 -> 293 us. Larger systems' chain of diagonal blocks is longer than a grid-wide team's CG: 648
// atoms, warm-started, took 424 us on a cluster of 16 blocks and take 277 on a team.
__device__ inline unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ inline unsigned remote(const void* p, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
__device__ inline void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ inline void send(const float* at, int rank, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote(at, rank)), "f"(v) : "memory");
}
__device__ inline void send(const double* at, int rank, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote(at, rank)), "d"(v) : "memory");
}
__device__ inline void send4(const float* at, int rank, const float4& v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(remote(at, rank)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}
__device__ inline void send_add(const float* at, int rank, float v) {
  asm volatile("red.relaxed.cluster.shared::cluster.add.f32 [%0], %1;" ::"r"(remote(at, rank)), "f"(v) : "memory");
}

// Tiles of block p's rows before its l-th one (row p + nb l).
__host__ __device__ constexpr int row_offset(int p, int nb, int l) { return l * (p + 1) + nb * (l * (l - 1) / 2); }
__host__ __device__ constexpr int rows_of(int p, int nb, int T) { return p < T ? (T - 1 - p) / nb + 1 : 0; }
__host__ __device__ constexpr int most_tiles(int nb, int T) {
  int m = 0;
  for (int p = 0; p < nb; ++p) {
    const int t = row_offset(p, nb, rows_of(p, nb, T));
    m = t > m ? t : m;
  }
  return m;
}
__host__ __device__ constexpr size_t cluster_bytes(int n, int nb) {
  const int T = (n + kTile - 1) / kTile;
  return (size_t)4 * kTileSize * (most_tiles(nb, T) + T - 1 + 1) +
         (size_t)kTile * (T * (sizeof(double) + 2 * sizeof(float)) + rows_of(0, nb, T) * sizeof(double));
}

struct ClusterShared {
  DirectShared d;
  double slots[2][kQeqDirectBlocks][4];  // partial sums by block, two exchanges' in turn
};

struct ClusterLayout {
  static constexpr int nb = kQeqDirectBlocks;
  int T, rank, own;  // tile rows; this block and its number of rows (atoms, padding included)
  float *tiles, *panel, *dinv;
  double *X, *G;
  float *b, *w1;
  __device__ ClusterLayout(unsigned char* dyn, int n, int p) {
    T = (n + kTile - 1) / kTile;
    rank = p;
    own = kTile * rows_of(p, nb, T);
    tiles = reinterpret_cast<float*>(dyn);  // the same offsets in every block: remote addresses are local ones
    panel = tiles + kTileSize * most_tiles(nb, T);
    dinv = panel + kTileSize * (T - 1);
    X = reinterpret_cast<double*>(dinv + kTileSize);
    b = reinterpret_cast<float*>(X + kTile * T);
    w1 = b + kTile * T;
    G = reinterpret_cast<double*>(w1 + kTile * T);
  }
  __device__ float* tile(int i, int j) const { return tiles + kTileSize * (row_offset(rank, nb, i / nb) + j); }  // i own
  __device__ int owner(int i) const { return i % nb; }
  __device__ int row(int q) const { return kTile * (rank + nb * (q >> 5)) + (q & 31); }  // atom of own row q
};

// Sums over the cluster of NV values of every thread with a row, in block order; post as in block_sums.
template <int NV, class Post>
__device__ inline void cluster_sums(const ClusterLayout& L, ClusterShared& sh, unsigned& parity, double (&v)[NV], Post post) {
  static_assert(NV <= 4, "at most four values");
  const int rows = L.own > 0 ? L.own : 1;
  double (*slots)[4] = sh.slots[parity & 1];
  ++parity;
  block_sums<NV>(sh.d, v, rows, [](double*) {});
  if ((int)threadIdx.x < L.nb)
#pragma unroll
    for (int k = 0; k < NV; ++k) send(&slots[L.rank][k], threadIdx.x, v[k]);
  cluster_sync();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      v[k] = slots[0][k];
      for (int q = 1; q < L.nb; ++q) v[k] += slots[q][k];
    }
    post(v);
#pragma unroll
    for (int k = 0; k < NV; ++k) sh.d.tot[k] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = sh.d.tot[k];
}

__device__ __noinline__ void cluster_factorize(const ClusterLayout& L, ClusterShared& sh) {
  constexpr int nb = ClusterLayout::nb;
  const int T = L.T, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int rg = threadIdx.x & 7, cg = (threadIdx.x >> 3) & 3;
  if (L.rank == 0 && wid < 4) tile_inverse(L.tile(0, 0), nullptr, nullptr, sh.d);
  for (int k = 0; k + 1 < T; ++k) {
    cluster_sync();  // the last step's panel has been read everywhere
    const int first = L.rank + nb * ((k + nb - L.rank) / nb);  // this block's first row past k
    const int m = first < T ? (T - 1 - first) / nb + 1 : 0;    // and how many
    for (int u = threadIdx.x; u < m * (kTileSize / 4); u += blockDim.x) {
      const int i = first + nb * (u / (kTileSize / 4)), q = 4 * (u % (kTileSize / 4));
      const float4 v = *reinterpret_cast<const float4*>(L.tile(i, k) + q);
      for (int p = 0; p < nb; ++p) send4(L.panel + kTileSize * (i - 1) + q, p, v);
    }
    if (L.owner(k) == L.rank)
      for (int u = threadIdx.x; u < kTileSize / 4; u += blockDim.x) {
        const float4 v = *reinterpret_cast<const float4*>(L.tile(k, k) + 4 * u);
        for (int p = 0; p < nb; ++p) send4(L.dinv + 4 * u, p, v);
      }
    cluster_sync();
    for (int u = wid; u < 2 * m; u += nw) {  // W_ik = A_ik D_k^-1 in A_ik's place
      const int i = first + nb * (u >> 1), c0 = 16 * (u & 1);
      float c[4][4];
      tile_product<4>(L.panel + kTileSize * (i - 1), L.dinv, c0, c);
      float* o = L.tile(i, k) + kTile * c0;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<float4*>(o + kTile * (4 * cg + q) + 4 * rg) = make_float4(c[0][q], c[1][q], c[2][q], c[3][q]);
    }
    __syncthreads();
    const bool next = L.owner(k + 1) == L.rank;  // this block inverts the next diagonal tile
    if (next && wid < 4) {
      tile_inverse(L.tile(k + 1, k + 1), L.tile(k + 1, k), L.panel + kTileSize * k, sh.d);
    } else {
      // the tiles (i, j), k < j <= i, of own rows i, numbered row by row
      const int w0 = next ? wid - 4 : wid, ws = next ? nw - 4 : nw;
      int u = w0, i = first;
      for (;;) {
        while (i < T && u >= i - k) {
          u -= i - k;
          i += nb;
        }
        if (i >= T) break;
        const int j = k + 1 + u;
        if (!(next && i == k + 1)) {
          float c[4][8];
          tile_product<8>(L.tile(i, k), L.panel + kTileSize * (j - 1), 0, c);
          float* o = L.tile(i, j);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            float4* d = reinterpret_cast<float4*>(o + kTile * (8 * cg + q) + 4 * rg);
            float4 v = *d;
            v.x -= c[0][q];
            v.y -= c[1][q];
            v.z -= c[2][q];
            v.w -= c[3][q];
            *d = v;
          }
        }
        u += ws;
      }
    }
  }
  __syncthreads();
}

// H^-1 v for the NV vectors v[k], given and left in the owners' rows (a thread per own row).
template <int NV>
__device__ inline void cluster_substitute(const ClusterLayout& L, float* const (&v)[NV]) {
  constexpr int nb = ClusterLayout::nb;
  const int T = L.T, r = threadIdx.x;
  const bool mine = r < L.own;
  const int at = mine ? L.row(r) : 0, i = at >> 5;
  auto publish = [&](int q) {  // this thread's row of every vector, to every block
    for (int p = 0; p < nb; ++p) send(v[q] + at, p, v[q][at]);
  };
  if (mine && i == 0)
    for (int q = 0; q < NV; ++q) publish(q);
  cluster_sync();
  for (int k = 0; k + 1 < T; ++k) {
    if (mine && i > k) {
      const float* w = L.tile(i, k) + (at & 31);
      float s[NV][2];
#pragma unroll
      for (int q = 0; q < NV; ++q) s[q][0] = s[q][1] = 0.0f;
#pragma unroll 8
      for (int c = 0; c < kTile; c += 2) {
        const float w0 = w[kTile * c], w1 = w[kTile * c + kTile];
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          s[q][0] += w0 * v[q][kTile * k + c];
          s[q][1] += w1 * v[q][kTile * k + c + 1];
        }
      }
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        v[q][at] -= s[q][0] + s[q][1];
        if (i == k + 1) publish(q);
      }
    }
    cluster_sync();
  }
  float z[NV];
  if (mine) {
    const float* d = L.tile(i, i) + (at & 31);
#pragma unroll
    for (int q = 0; q < NV; ++q) z[q] = 0.0f;
#pragma unroll 8
    for (int c = 0; c < kTile; ++c) {
      const float x = d[kTile * c];
#pragma unroll
      for (int q = 0; q < NV; ++q) z[q] += x * v[q][kTile * i + c];
    }
  }
  __syncthreads();
  if (mine)
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q][at] = z[q];
  cluster_sync();
  for (int k = T - 1; k > 0; --k) {
    if (L.owner(k) == L.rank)
      for (int t = r; t < kTile * k; t += blockDim.x) {
        const float* w = L.tile(k, t >> 5) + kTile * (t & 31);
        float s[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) s[q] = 0.0f;
#pragma unroll 8
        for (int u = 0; u < kTile; ++u) {
          const int c = (u + t) & 31;  // a lane starts at its own column: no two share a bank
          const float x = w[c];
#pragma unroll
          for (int q = 0; q < NV; ++q) s[q] += x * v[q][kTile * k + c];
        }
#pragma unroll
        for (int q = 0; q < NV; ++q) send_add(v[q] + t, L.owner(t >> 5), -s[q]);
      }
    cluster_sync();
  }
}

__global__ void __launch_bounds__(512, 1) k_qeq_direct_cluster(XrWork w, XrFF ff, const int* list, int adjoint) {
  __shared__ ClusterShared sh;
  extern __shared__ __align__(16) unsigned char dyn[];
  constexpr int nb = kQeqDirectBlocks;
  const int sys = list[blockIdx.x / nb];
  const XrSystem& S = w.sys[sys];
  const int a0 = S.atom_off, n = S.natoms, tid = threadIdx.x, wid = tid >> 5, nw = blockDim.x >> 5;
  const double* atab = xr_ff_at(ff, ff.nsets > 1 ? S.ff_set : 0).atom;
  const double Q = adjoint ? 0.0 : S.total_charge;
  const bool warm = !adjoint && S.has_guess != 0;
  const double x0 = Q == 0.0 ? 0.0 : Q / n;
  const ClusterLayout L(dyn, n, blockIdx.x % nb);
  const int at = tid < L.own ? L.row(tid) : 0, m = min(L.own, max(0, L.own > 0 ? L.own - max(0, kTile * L.T - n) *
                                                                              (L.owner(L.T - 1) == L.rank ? 1 : 0) : 0));
  const bool row = tid < m;  // (only the last tile row has padding)
  const int a = a0 + min(at, n - 1), type = w.type[a];
  const double eta = atom_prm(atab, type, A_ETA), chi = adjoint ? w.qrhs[a] : atom_prm(atab, type, A_CHI);
  unsigned parity = 0;
  // 1. The own rows' tiles; the charges of every row.
  const int ntiles = row_offset(L.rank, nb, L.own / kTile);
  for (int k = tid; k < ntiles * kTileSize / 4; k += blockDim.x) reinterpret_cast<float4*>(L.tiles)[k] = make_float4(0, 0, 0, 0);
  for (int k = tid; k < kTile * L.T; k += blockDim.x) L.X[k] = k < n ? (warm ? w.qguess[a0 + k] : x0) : 0.0;
  __syncthreads();
  if (tid < L.own) L.tile(at >> 5, at >> 5)[(kTile + 1) * (at & 31)] = row ? (float)eta : 1.0f;
  __syncthreads();
  // Row i's first entries, all but as many as it has half edges, are those with j < i and one direction of its
  // self images.
  const int* const half = w.cnt + (w.A + 1) + a0;
  for (int q = wid; q < m; q += nw) {
    const int i = L.row(q);
    add_row(w, a0, n, w.cnt[a0 + i], w.cnt[a0 + i + 1] - (half[i + 1] - half[i]), [&](int j, float h) {
      float* const t = L.tile(i >> 5, j >> 5);
      if (j == i) {
        t[(kTile + 1) * (i & 31)] += 2.0f * h;
      } else {
        t[kTile * (j & 31) + (i & 31)] += h;
        if ((j >> 5) == (i >> 5)) t[kTile * (i & 31) + (j & 31)] += h;
      }
    });
  }
  __syncthreads();
  auto product = [&]() { product64(w, L.X, L.G, a0, m, [&](int q) { return L.row(q); }); };
  // 2. The start gradient and the target, as in k_qeq_direct.
  const double di = row ? 1.0 / (double)L.tile(at >> 5, at >> 5)[(kTile + 1) * (at & 31)] : 0.0;
  double x = row ? L.X[at] : 0.0, g = chi, gu = chi;
  if (warm || x0 != 0.0) {
    product();
    g = gu = row ? L.G[tid] + eta * x + chi : 0.0;
  }
  if (warm) {
    gu = chi;
    if (x0 != 0.0) {
      __syncthreads();
      for (int k = tid; k < n; k += blockDim.x) L.X[k] = x0;
      __syncthreads();
      product();
      gu = row ? L.G[tid] + eta * x0 + chi : 0.0;
    }
  }
  if (!row) g = gu = 0.0;
  double v3[3] = {di, di * g, di * gu}, vn[2] = {di * g * g, di * gu * gu};
  cluster_sync();  // every block runs before the first remote write
  cluster_sums<2>(L, sh, parity, vn, [](double*) {});
  cluster_sums<3>(L, sh, parity, v3, [](double* t) {
    t[1] /= t[0];
    t[2] /= t[0];
  });
  const double s1 = v3[0], gfloor = 1e-28 * fmax(vn[0], vn[1]);
  if (row) {
    g -= v3[1];
    gu -= v3[2];
  }
  double v2[2] = {di * g * g, di * gu * gu};
  cluster_sums<2>(L, sh, parity, v2, [&](double* t) { t[1] *= w.cg_tol * w.cg_tol; });
  double gz = v2[0];
  const double target = v2[1];
  // 3. Refinement steps, as in k_qeq_direct; y is made to sum to zero in FP64, so that one exchange gives its
  //    multiplier and the constraint's shift.
  int steps = 0;
  bool failed = false, last = false, more = gz > target && gz > gfloor && n >= 2;
  while (more) {
    if (steps == 8 && !last) {
      failed = true;
      break;
    }
    if (tid < L.own) L.b[at] = row ? (float)-g : 0.0f;
    if (steps == 0) {
      if (tid < L.own) L.w1[at] = row ? 1.0f : 0.0f;
      cluster_factorize(L, sh);
      float* const both[2] = {L.b, L.w1};
      cluster_substitute<2>(L, both);
    } else {
      float* const one[1] = {L.b};
      cluster_substitute<1>(L, one);
    }
    ++steps;
    const double b = row ? (double)L.b[at] : 0.0, w1 = row ? (double)L.w1[at] : 0.0;
    double vs[3] = {b, w1, x};
    cluster_sums<3>(L, sh, parity, vs, [&](double* t) {
      t[0] /= t[1];
      t[2] = (Q - t[2]) / n;
    });
    if (row) x += (b - vs[0] * w1) + vs[2];
    if (last) break;
    if (row)
      for (int p = 0; p < nb; ++p) send(L.X + at, p, x);
    cluster_sync();
    product();
    g = row ? L.G[tid] + eta * x + chi : 0.0;
    double vl[1] = {di * g};
    cluster_sums<1>(L, sh, parity, vl, [&](double* t) { t[0] /= s1; });
    if (row) g -= vl[0];
    double vg[2] = {di * g * g, 0.0};
    const double before = gz;
    cluster_sums<2>(L, sh, parity, vg, [&](double* t) { t[1] = t[0] / before; });
    gz = vg[0];
    if (!(vg[1] <= 1e-3) && !(gz <= target)) {
      failed = true;
      break;
    }
    last = gz <= target || vg[1] * gz <= 1e-2 * target;
    more = last || gz > gfloor;
  }
  // 4. Final charges: the constraint restored exactly.
  double sx[1] = {x};
  cluster_sums<1>(L, sh, parity, sx, [&](double* t) { t[0] = (Q - t[0]) / n; });
  cluster_sync();  // no block leaves while another may still write to it
  if (failed) {
    if (L.rank == 0 && tid == 0) {
      int* const retry = w.qretry + (adjoint ? 2 : 0);
      w.qretry[4 + (adjoint ? w.S : 0) + atomicAdd(retry, 1)] = sys;
    }
    return;
  }
  if (L.rank == 0 && tid == 0) {
    atomicMax(w.counts + 4, steps);
    w.qiters[sys] = max(w.qiters[sys], steps);
  }
  if (!row) return;
  const double q = x + sx[0];
  if (adjoint) {
    w.qadj[a] = q;
    return;
  }
  w.q[a] = q;
  w.a_e[(size_t)6 * w.A + a] = SELF_CONVERSION * (chi * q + 0.5 * eta * q * q);
}

cudaLaunchConfig_t cluster_config(int count, size_t bytes, cudaStream_t st, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kQeqDirectBlocks * count);
  cfg.blockDim = dim3(512);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kQeqDirectBlocks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

}  // namespace

int xr_qeq_direct_cluster_max() {
  constexpr int largest = kQeqDirectCluster;
  bool ok = cudaFuncSetAttribute(k_qeq_direct_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)cluster_bytes(largest, kQeqDirectBlocks)) ==
            cudaSuccess;
  int clusters = 0;
  if (ok) {
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = cluster_config(1, cluster_bytes(largest, kQeqDirectBlocks), nullptr, attr);
    ok = cudaOccupancyMaxActiveClusters(&clusters, (void*)k_qeq_direct_cluster, &cfg) == cudaSuccess;
  }
  if (!ok) cudaGetLastError();
  return ok && clusters > 0 ? largest : 0;
}

int xr_launch_qeq_direct_cluster(const XrWork& w, const XrFF& ff, cudaStream_t st, const int* list, int count, int largest,
                                 bool adjoint) {
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = cluster_config(count, cluster_bytes(largest, kQeqDirectBlocks), st, attr);
  return (int)cudaLaunchKernelEx(&cfg, k_qeq_direct_cluster, w, ff, list, adjoint ? 1 : 0);
}

bool xr_qeq_direct_ready() {
  const bool ok = cudaFuncSetAttribute(k_qeq_direct, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)direct_bytes(kQeqDirectMax)) == cudaSuccess;
  if (!ok) cudaGetLastError();
  return ok;
}

int xr_launch_qeq_direct(const XrWork& w, const XrFF& ff, cudaStream_t st, const int* list, int count, int largest, bool adjoint) {
  // a thread per row, four warps for the diagonal tiles and, past one tile, at least as many for the rest
  const int rows = (largest + kTile - 1) / kTile * kTile;
  const int threads = rows <= kTile ? 128 : rows <= kQeqDirectSmall ? 256 : 512;
  k_qeq_direct<<<count, threads, direct_bytes(largest), st>>>(w, ff, list, adjoint ? 1 : 0);
  return (int)cudaGetLastError();
}
