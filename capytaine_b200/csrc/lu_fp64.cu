// Batched blocked complex128 LU factorisation and triangular solves (sm_100a).
//
// Replaces the LAPACK zgetrf / zgetrs calls behind scipy.linalg.lu_factor /
// lu_solve in capytaine (tools/block_circulant_matrices.py:361-385, used by
// bem/engines.py:300-346).  Matrices are column-major complex128, one matrix per
// frequency, `batch` of them `stride` elements apart, each padded to a multiple
// of kNB = 64 with the identity on the padded diagonal.
//
// Factorisation (right-looking, one step per 64-column block):
//   1. diagonal block: LU in shared memory with partial pivoting among the rows
//      of the block (the permutation P is block diagonal, so P A = L U holds
//      exactly), and the inverses of its triangles;
//   2. panels: the block row is permuted (left part included, as LAPACK's
//      zlaswp does) and solved with L11; the block column below is solved with
//      U11 (both by substitution in blocks of 16);
//   3. trailing update A22 -= A21 A12; the CTA of the next diagonal block also
//      factors it.
// All products on double-precision tensor-core MMAs (mma.sync m16n8k8 f64),
// four real products per complex one.
// Solves: forward and backward block substitutions run as one persistent kernel each, block rows handed out in
// dependency order through an atomic ticket so that every wait targets a block
// row whose CTA is already running; waits are bounded and report a timeout.
#include <algorithm>
#include "dmma.cuh"
#include "reciprocals.cuh"

namespace bem {
namespace {

constexpr int kNB = 64;
constexpr int kLd = kNB + 1;  // shared-memory leading dimension of a 64x64 tile
constexpr int kLdD = kNB + 2;  // of the diagonal block being factored (MMA fragments)

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cfms(double2 acc, double2 a, double2 b) {  // acc - a*b
  return make_double2(acc.x - (a.x * b.x - a.y * b.y), acc.y - (a.x * b.y + a.y * b.x));
}
__device__ __forceinline__ double cabs1(double2 a) { return fabs(a.x) + fabs(a.y); }

// ---------------------------------------------------------------------------
// 1. Diagonal block: LU with partial pivoting among the block's 64 rows, and
// the inverses of both triangles, by one CTA of 256 threads, the block in
// shared memory (T[c * kLdD + r]).
// Panels of 8 columns are factored by one warp in registers, two rows per lane:
// the pivot by one warp reduction, no row moves (a row's place is settled at
// the panel's end), no barrier inside.  Meanwhile the other warps apply the
// previous panel to the columns beyond, as rank-8 products on the tensor
// cores; so are the levels of the inverses.  A barrier per step of 64 columns
// and an exchange through shared memory took 84 us per block (and the inverses
// a pass of 180 us over the matrix); this takes 40 us with the inverses, hidden behind the other tiles where they are many.
constexpr int kPW = 8;      // columns of a panel
constexpr int kTmpLd = 36;  // 4 mod 8: MMA B fragments

struct DiagShared {
  int perm[kNB];     // original row at each position
  int place[kNB];    // new position of each row after the panel
  int moved;         // 1: the panel exchanged rows
  double2 pivot_row[2][kPW];  // of the step (double-buffered)
};

__device__ __forceinline__ double2 shfl2(double2 v, int src) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
__device__ __forceinline__ int nth_bit(unsigned long long m, int n) {
  for (; n > 0; --n) m &= m - 1;
  return __ffsll((long long)m) - 1;
}

// Columns j0 .. j0 + 7 by one warp; kcol: the block's first column in the matrix.
__device__ __forceinline__ void factor_panel(double2* T, int j0, int lane, DiagShared& sh, int* info, int kcol) {
  double2 x[2][kPW];
  int pos[2] = {-1, -1};  // position of a row chosen as pivot
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int s = 0; s < kPW; ++s) x[h][s] = T[(j0 + s) * kLdD + lane + 32 * h];
  // The largest |re| + |im| of a column among the rows left: the high word of
  // the value with its last six bits replaced by the row, so that one reduction
  // finds both (values within 2^-14 of the largest count as equal and the first
  // row wins: multipliers up to 1 + 2^-14); a NaN is never chosen.
  auto pivot_key = [&](int s) {
    unsigned key = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = lane + 32 * h;
      const double c = cabs1(x[h][s]);
      if (r >= j0 && pos[h] < 0 && c == c)
        key = max(key, (((unsigned)__double2hiint(c) + 64u) & ~63u) | (unsigned)(63 - r));
    }
    return key;
  };
  unsigned key = __reduce_max_sync(0xffffffffu, pivot_key(0));
#pragma unroll
  for (int s = 0; s < kPW; ++s) {
    unsigned row = 63u - (key & 63u);
    if (key == 0) {  // only NaN left: the first row left
      const unsigned mine = (lane >= j0 && pos[0] < 0) ? lane : (lane + 32 >= j0 && pos[1] < 0) ? lane + 32 : 64u;
      row = __reduce_min_sync(0xffffffffu, mine);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (lane + 32 * h == (int)row) {
        pos[h] = j0 + s;
#pragma unroll
        for (int c = s; c < kPW; ++c) sh.pivot_row[s & 1][c] = x[h][c];
      }
    __syncwarp();
    double2 p[kPW];
#pragma unroll
    for (int c = s; c < kPW; ++c) p[c] = sh.pivot_row[s & 1][c];
    bool in_range;
    double2 inv = cinv_fast(p[s], in_range);
    if (!in_range) {
      const bool ok = cabs1(p[s]) > 0.0;
      if (!ok && lane == 0 && *info == 0) *info = kcol + j0 + s + 1;
      inv = ok ? cinv(p[s]) : make_double2(1.0, 0.0);
    }
    double2 l[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (lane + 32 * h >= j0 && pos[h] < 0) {
        x[h][s] = cmul(x[h][s], inv);
        l[h] = x[h][s];
      } else {
        l[h] = make_double2(0.0, 0.0);  // rows done keep their values
      }
    }
    // the next pivot's column first: its reduction runs beside the others' updates
    if (s + 1 < kPW) {
#pragma unroll
      for (int h = 0; h < 2; ++h) x[h][s + 1] = cfms(x[h][s + 1], l[h], p[s + 1]);
      key = __reduce_max_sync(0xffffffffu, pivot_key(s + 1));
#pragma unroll
      for (int c = s + 2; c < kPW; ++c)
#pragma unroll
        for (int h = 0; h < 2; ++h) x[h][c] = cfms(x[h][c], l[h], p[c]);
    }
  }
  // positions: pivots in order; a row that gave its place up takes the place
  // of a pivot that came from further down
  const unsigned long long sel = (unsigned long long)__ballot_sync(0xffffffffu, pos[0] >= 0) |
                                 (unsigned long long)__ballot_sync(0xffffffffu, pos[1] >= 0) << 32;
  const unsigned long long in_panel = ((1ull << kPW) - 1) << j0;
  const unsigned long long vacated = sel & ~in_panel, displaced = in_panel & ~sel;
  int old[2], to[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = lane + 32 * h;
    old[h] = sh.perm[r];
    to[h] = r;
    if (pos[h] >= 0) to[h] = pos[h];
    else if (displaced >> r & 1) to[h] = nth_bit(vacated, __popcll(displaced & ((1ull << r) - 1)));
    sh.place[r] = to[h];
  }
  __syncwarp();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    sh.perm[to[h]] = old[h];
#pragma unroll
    for (int s = 0; s < kPW; ++s) T[(j0 + s) * kLdD + to[h]] = x[h][s];
  }
  const bool moved = __any_sync(0xffffffffu, to[0] != lane || to[1] != lane + 32);
  if (lane == 0) sh.moved = moved;
}

// 16 x 16 inverse of one triangle of the block at (base, base), by one warp,
// in place.  Lane c < 16 holds column c.
__device__ __forceinline__ void invert_lower16(double2* T, int base, int lane) {
  const int c = lane & 15;
  double2 x[16];
#pragma unroll
  for (int r = 0; r < 16; ++r) x[r] = make_double2(r == c ? 1.0 : 0.0, 0.0);
#pragma unroll
  for (int i = 0; i < 15; ++i)
#pragma unroll
    for (int r = i + 1; r < 16; ++r) x[r] = cfms(x[r], T[(base + i) * kLdD + base + r], x[i]);
  __syncwarp();
  if (lane < 16) {
#pragma unroll
    for (int r = 0; r < 16; ++r)
      if (r > c) T[(base + c) * kLdD + base + r] = x[r];
  }
}
__device__ __forceinline__ void invert_upper16(double2* T, int base, int lane) {
  const int c = lane & 15;
  const double2 d = T[(base + c) * kLdD + base + c];
  bool in_range;
  double2 mine = cinv_fast(d, in_range);
  if (!in_range) mine = cabs1(d) > 0.0 ? cinv(d) : make_double2(0.0, 0.0);
  double2 x[16];
#pragma unroll
  for (int r = 0; r < 16; ++r) x[r] = make_double2(r == c ? 1.0 : 0.0, 0.0);
#pragma unroll
  for (int i = 15; i >= 0; --i) {
    x[i] = cmul(x[i], shfl2(mine, i));
#pragma unroll
    for (int r = 0; r < i; ++r) x[r] = cfms(x[r], T[(base + i) * kLdD + base + r], x[i]);
  }
  __syncwarp();
  if (lane < 16) {
#pragma unroll
    for (int r = 0; r < 16; ++r)
      if (r <= c) T[(base + c) * kLdD + base + r] = x[r];
  }
}

// T(16 rows from m0, 8 columns from n0) -= panel (8 columns from j0) times the
// rows j0 .. j0 + 7 of those columns, rows from first_row on only (a multiple of 8).
__device__ __forceinline__ void panel_update_tile(double2* T, int j0, int m0, int n0, int first_row, int lane) {
  const int g = lane >> 2, t = lane & 3;
  double2 c[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) c[e] = T[(n0 + 2 * t + (e & 1)) * kLdD + m0 + g + 8 * (e >> 1)];
  double ar[4], ai[4], ni[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const double2 v = T[(j0 + t + 4 * (e >> 1)) * kLdD + m0 + g + 8 * (e & 1)];
    ar[e] = v.x;
    ai[e] = v.y;
    ni[e] = -v.y;
  }
  const double2 b0 = T[(n0 + g) * kLdD + j0 + t], b1 = T[(n0 + g) * kLdD + j0 + t + 4];
  const double br[2] = {b0.x, b1.x}, bi[2] = {b0.y, b1.y};
  // the product on its own first: one rounding of the tile's size per entry
  double re[4] = {}, im[4] = {};
  dmma(re, ar, br);
  dmma(im, ar, bi);
  dmma(re, ni, bi);
  dmma(im, ai, br);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int r = m0 + g + 8 * (e >> 1);
    if (r >= first_row)
      T[(n0 + 2 * t + (e & 1)) * kLdD + r] = make_double2(c[e].x - re[e], c[e].y - im[e]);
  }
}

// The off-diagonal H x H blocks of the triangles' inverses from those of the
// diagonal ones (H = 16, then 32): with [A 0; C B] below the diagonal,
// -B^-1 (C A^-1); with [A C; 0 B] above it, -A^-1 (C B^-1).  In place in T, the
// inner product through tmp; 16 x 8 tiles of the products over the 8 warps,
// the zero blocks of the triangles skipped.
template <int H>
__device__ __forceinline__ void invert_level(double2* T, double2* tmp, int warp, int lane) {
  constexpr int kCombos = 64 / H;                     // (triangle, pair of blocks)
  constexpr int kTilesM = H / 16, kTilesN = H / 8;
  constexpr int kTiles = kCombos * kTilesM * kTilesN;
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int stage = 0; stage < 2; ++stage) {
#pragma unroll 1
    for (int tile = warp; tile < kTiles; tile += 8) {
      const int combo = tile / (kTilesM * kTilesN), in = tile % (kTilesM * kTilesN);
      const bool lower = combo & 1;
      const int base = (combo >> 1) * 2 * H, m0 = 16 * (in % kTilesM), n0 = 8 * (in / kTilesM);
      double2* W = tmp + combo * H * kTmpLd;
      const int rowC = lower ? base + H : base, colC = lower ? base : base + H;
      double re[4] = {}, im[4] = {};
#pragma unroll 1
      for (int k0 = 0; k0 < H; k0 += 8) {
        // stage 0: W = C (inverse at C's columns): its rows k against columns n0 ..
        // stage 1: (inverse at C's rows) W: its columns k against rows m0 ..
        if (stage == 0 ? (lower ? k0 < n0 : k0 > n0) : (lower ? k0 > m0 + 8 : k0 < m0)) continue;
        double ar[4], ai[4], na[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int k = k0 + t + 4 * (e >> 1), m = m0 + g + 8 * (e & 1);
          double2 v;
          if (stage == 0) {
            v = T[(colC + k) * kLdD + rowC + m];
          } else {
            v = T[(rowC + k) * kLdD + rowC + m];
            if (lower ? k > m : k < m) v = make_double2(0.0, 0.0);
            if (lower && k == m) v = make_double2(1.0, 0.0);
            v.x = -v.x;
            v.y = -v.y;
          }
          ar[e] = v.x;
          ai[e] = v.y;
          na[e] = -v.y;
        }
        double br[2], bi[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int k = k0 + t + 4 * e, n = n0 + g;
          double2 v;
          if (stage == 0) {
            v = T[(colC + n) * kLdD + colC + k];
            if (lower ? k < n : k > n) v = make_double2(0.0, 0.0);
            if (lower && k == n) v = make_double2(1.0, 0.0);
          } else {
            v = W[n * kTmpLd + k];
          }
          br[e] = v.x;
          bi[e] = v.y;
        }
        dmma(re, ar, br);
        dmma(im, ar, bi);
        dmma(re, na, bi);
        dmma(im, ai, br);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = m0 + g + 8 * (e >> 1), n = n0 + 2 * t + (e & 1);
        const double2 v = make_double2(re[e], im[e]);
        if (stage == 0) W[n * kTmpLd + m] = v;
        else T[(colC + n) * kLdD + rowC + m] = v;
      }
    }
    __syncthreads();
  }
}

// The whole diagonal block at row and column kk of a matrix, already in T:
// factors to the matrix, inverses to inv (L then U, 64 x 64 column-major).
__device__ void factor_diagonal(double2* T, double2* tmp, DiagShared& sh, double2* __restrict__ Ab, int64_t lda,
                                int kk, int* __restrict__ piv, int* __restrict__ info, double2* __restrict__ inv) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < kNB) sh.perm[tid] = tid;
  __syncthreads();
#pragma unroll 1
  for (int j0 = 0; j0 < kNB; j0 += kPW) {
    const int j1 = j0 + kPW;
    if (warp == 0) {
      factor_panel(T, j0, lane, sh, info, kk);
    } else if (j0 > 0) {
      // columns beyond this panel: the previous panel's update
      const int tiles_m = (kNB - (j0 & ~15)) / 16, tiles = tiles_m * ((kNB - j1) / 8);
      for (int i = warp - 1; i < tiles; i += 7)
        panel_update_tile(T, j0 - kPW, (j0 & ~15) + 16 * (i % tiles_m), j1 + 8 * (i / tiles_m), j0, lane);
    }
    __syncthreads();
    if (sh.moved) {
      for (int c = warp; c < kNB; c += 8) {
        if (c >= j0 && c < j1) continue;
        const double2 v0 = T[c * kLdD + lane], v1 = T[c * kLdD + lane + 32];
        __syncwarp();
        T[c * kLdD + sh.place[lane]] = v0;
        T[c * kLdD + sh.place[lane + 32]] = v1;
      }
      __syncthreads();
    }
    if (tid < kNB && tid >= j1) {  // rows of U: L11^-1 applied to column tid
      double2 x[kPW];
#pragma unroll
      for (int i = 0; i < kPW; ++i) x[i] = T[tid * kLdD + j0 + i];
#pragma unroll
      for (int i = 0; i < kPW - 1; ++i)
#pragma unroll
        for (int r = i + 1; r < kPW; ++r) x[r] = cfms(x[r], T[(j0 + i) * kLdD + j0 + r], x[i]);
#pragma unroll
      for (int i = 1; i < kPW; ++i) T[tid * kLdD + j0 + i] = x[i];
    }
    __syncthreads();
    // the next panel's columns
    if (j1 < kNB) {
      const int m0 = (j1 & ~15) + 16 * warp;
      if (m0 < kNB) panel_update_tile(T, j0, m0, j1, j1, lane);
    }
    __syncthreads();
  }
  for (int idx = tid; idx < kNB * kNB; idx += 256) {
    const int r = idx % kNB, c = idx / kNB;
    Ab[(size_t)(kk + r) + (size_t)(kk + c) * lda] = T[c * kLdD + r];
  }
  if (tid < kNB) piv[kk + tid] = sh.perm[tid];
  __syncthreads();
  if (warp < 4) invert_lower16(T, 16 * warp, lane);
  else invert_upper16(T, 16 * (warp - 4), lane);
  __syncthreads();
  invert_level<16>(T, tmp, warp, lane);
  invert_level<32>(T, tmp, warp, lane);
  for (int idx = tid; idx < kNB * kNB; idx += 256) {
    const int r = idx % kNB, c = idx / kNB;
    const double2 v = T[c * kLdD + r], zero = make_double2(0.0, 0.0);
    inv[idx] = r > c ? v : make_double2(r == c ? 1.0 : 0.0, 0.0);
    inv[kNB * kNB + idx] = r <= c ? v : zero;
  }
}

// ---------------------------------------------------------------------------
// 2. Panels by substitution in blocks of 16, each a product with the inverse of
// the triangle's 16 x 16 diagonal block.  blockIdx.x enumerates:
// [0, nleft) the block row's 64-column tiles left of the diagonal (permuted
// only, as LAPACK's zlaswp), then 32-column tiles right of it (permuted, times
// L11^-1 from the left), then 32-row tiles below it (times U11^-1 from the
// right).  In place: a CTA reads all that it overwrites first.
// One product with the whole inverse of the triangle is 3 us shorter per step
// (20 frequencies of 800 panels 4.80 ms in place of 4.92) but leaves up to ten
// times the error in the factors where the triangle is ill-conditioned.  A warp
// and its neighbour share a block of 16: with warps of one scheduler on it, 5.03 ms.
constexpr int kPanelTile = 32;
constexpr int kPanelLdB = kNB + 4;
constexpr int kPanelSmem = kNB * (kPanelTile + 2 + kPanelLdB) * (int)sizeof(double2);  // the tiles below need more
static_assert(kPanelSmem >= (kNB * (kNB + 2) + kPanelTile * kPanelLdB) * (int)sizeof(double2), "tiles to the right");
static_assert(kPanelSmem >= kNB * kLd * (int)sizeof(double2), "tiles to the left");

template <bool RIGHT>
__device__ __forceinline__ void panel_tile(double2* sm, double2* __restrict__ Ab, int64_t lda, int kk, int at,
                                           const double2* __restrict__ inv, const int* perm) {
  // RIGHT: (64 x 32) = L11^-1 (64 x 64) X (64 x 32); else (32 x 64) = X (32 x 64) U11^-1 (64 x 64)
  constexpr int kM = RIGHT ? kNB : kPanelTile, kN = RIGHT ? kPanelTile : kNB;
  constexpr int kLdA = kM + 2;
  double2* As = sm;
  double2* Bs = sm + kNB * kLdA;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double2* X = RIGHT ? Ab + kk + (size_t)at * lda : Ab + at + (size_t)kk * lda;
  const double2* D = Ab + kk + (size_t)kk * lda;
  // (r, c) of the triangle: its 16 x 16 diagonal blocks inverted, the blocks on its other side not read
  auto triangle = [&](int r, int c) {
    return (r >> 4) == (c >> 4) ? inv + (size_t)c * kNB + r : D + (size_t)r + (size_t)c * lda;
  };
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {  // a block of 16 of the inner dimension per copy group
    for (int idx = tid; idx < 16 * kM; idx += 256) {
      const int m = idx % kM, k = 16 * q + idx / kM;
      if (!RIGHT || m >= 16 * q)
        cp_async16(As + k * kLdA + m, RIGHT ? triangle(m, k) : X + (size_t)m + (size_t)k * lda, true);
    }
    for (int idx = tid; idx < 16 * kN; idx += 256) {
      const int k = 16 * q + (idx & 15), n = idx >> 4;
      if (RIGHT || n >= 16 * q)
        cp_async16(Bs + n * kPanelLdB + k, RIGHT ? X + (size_t)perm[k] + (size_t)n * lda : triangle(k, n), true);
    }
    cp_async_commit();
  }
  // eight warps of 16 x 16, each in one of the four blocks of the substitution
  const int own = warp >> 1, other = warp & 1;
  const int wm = 16 * (RIGHT ? own : other), wn = 16 * (RIGHT ? other : own);
  const int g = lane >> 2, t = lane & 3;
  double re[2][4] = {}, im[2][4] = {};    // products with the solved blocks
  double xr[2][4] = {}, xi[2][4] = {};    // this warp's part of the solution
  auto place = [&](int j, int e) -> double2& {  // of a fragment's element in the tile
    const int m = wm + g + 8 * (e >> 1), n = wn + 8 * j + 2 * t + (e & 1);
    return RIGHT ? Bs[n * kPanelLdB + m] : As[n * kLdA + m];
  };
  cp_async_wait<3>();
  __syncthreads();
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    const double2* a = As + 16 * q * kLdA + wm;
    const double2* bb = Bs + wn * kPanelLdB + 16 * q;
    if (own == q) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          double2& v = place(j, e);
          v = make_double2(v.x - re[j][e], v.y - im[j][e]);
        }
      __syncwarp();
      warp_zmma<2>(a, kLdA, bb, kPanelLdB, 16, xr, xi, lane);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) place(j, e) = make_double2(xr[j][e], xi[j][e]);
    }
    if (q == 0) cp_async_wait<2>();
    if (q == 1) cp_async_wait<1>();
    if (q >= 2) cp_async_wait<0>();
    __syncthreads();  // block q is solved, block q + 1 has landed
    if (own > q) warp_zmma<2>(a, kLdA, bb, kPanelLdB, 16, re, im, lane);
  }
  // every read of the tile (its rows permuted) lies before the last barrier
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      X[(size_t)(wm + g + 8 * (e >> 1)) + (size_t)(wn + 8 * j + 2 * t + (e & 1)) * lda] =
          make_double2(xr[j][e], xi[j][e]);
}

__global__ void __launch_bounds__(256, 2) zlu_panel_kernel(double2* __restrict__ A, int64_t lda, int64_t stride,
                                                           int n, int kk, const int* __restrict__ piv,
                                                           int64_t piv_stride, const double2* __restrict__ inv,
                                                           int nblk) {
  extern __shared__ double2 sm[];
  __shared__ int perm[kNB];
  const int b = blockIdx.y, tid = threadIdx.x;
  double2* Ab = A + (size_t)b * stride;
  const int nleft = kk / kNB, nrest = (n - kk - kNB) / kPanelTile;
  const int t = blockIdx.x;
  const double2* ib = inv + ((size_t)b * nblk + kk / kNB) * 2 * kNB * kNB;
  int own = 0;
  if (tid < kNB) {
    own = piv[(size_t)b * piv_stride + kk + tid];
    perm[tid] = own;
  }
  if (t < nleft) {
    if (!__syncthreads_or(tid < kNB && own != tid)) return;  // no row moves
    const int c0 = t * kNB;
    for (int idx = tid; idx < kNB * kNB; idx += 256) {
      const int r = idx % kNB, c = idx / kNB;
      sm[c * kLd + r] = Ab[(size_t)(kk + perm[r]) + (size_t)(c0 + c) * lda];
    }
    __syncthreads();
    for (int idx = tid; idx < kNB * kNB; idx += 256) {
      const int r = idx % kNB, c = idx / kNB;
      Ab[(size_t)(kk + r) + (size_t)(c0 + c) * lda] = sm[c * kLd + r];
    }
    return;
  }
  __syncthreads();
  const int u = t - nleft;
  if (u < nrest) panel_tile<true>(sm, Ab, lda, kk, kk + kNB + u * kPanelTile, ib, perm);
  else panel_tile<false>(sm, Ab, lda, kk, kk + kNB + (u - nrest) * kPanelTile, ib + kNB * kNB, perm);
}

// ---------------------------------------------------------------------------
// 3. C = beta C + alpha A B (alpha, beta real), column-major complex128, 64 x 64
// tiles by CTAs of 8 warps (16 x 32 each), depth 16 per stage of a three-stage
// cp.async ring, two CTAs per SM.  Edges of any size are filled with zeros and
// not stored.
// FACTOR (trailing update of the LU): the CTA of the tile that is the next
// diagonal block keeps its result in shared memory and factors it, beside the
// other CTAs' tiles: the chain of diagonal blocks is hidden behind the updates
// where these are long, and costs no launch.  Those CTAs come first in the
// grid.  4 x 2688: 8.97 ms, 27 TF/s in the largest update (9.25 ms with accumulators
// that start from C).
constexpr int kTile = 64, kDepth = 16, kStages = 3;
constexpr int kResident = 2 * 148;  // CTAs that the GPU holds at a time
constexpr int kLdTA = kTile + 2, kLdTB = kDepth + 4;
constexpr int kStageElems = kDepth * kLdTA + kTile * kLdTB;
constexpr int kGemmSmem = kStages * kStageElems * (int)sizeof(double2);
static_assert((kNB * kLdD + 2 * 32 * kTmpLd) * (int)sizeof(double2) <= kGemmSmem, "the diagonal block fits");

template <bool FACTOR>
__global__ void __launch_bounds__(256, 2)
    zgemm_dmma_kernel(int M, int N, int K, double alpha, const double2* A, int64_t lda, int64_t strideA,
                      const double2* B, int64_t ldb, int64_t strideB, double beta, double2* C, int64_t ldc,
                      int64_t strideC, int tiles_m, int tiles, int batch, int kk, int* __restrict__ piv,
                      int64_t piv_stride, int* __restrict__ info, double2* __restrict__ inv, int nblk) {
  extern __shared__ double2 sm[];
  __shared__ DiagShared sh;
  int t, b;
  if ((int)blockIdx.x < batch) {  // tile 0 of every matrix
    t = 0;
    b = blockIdx.x;
  } else {
    const int rest = blockIdx.x - batch;
    t = 1 + rest % (tiles - 1);
    b = rest / (tiles - 1);
  }
  A += (size_t)b * strideA;
  B += (size_t)b * strideB;
  C += (size_t)b * strideC;
  const int m0 = (t % tiles_m) * kTile, n0 = (t / tiles_m) * kTile;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nk = (K + kDepth - 1) / kDepth;
  auto issue = [&](int q) {
    if (q < nk) {
      double2* As = sm + (q % kStages) * kStageElems;
      double2* Bs = As + kDepth * kLdTA;
      const int k0 = q * kDepth;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int idx = tid + 256 * i;
        const int m = idx & 63, k = idx >> 6;
        const bool ok = m0 + m < M && k0 + k < K;
        cp_async16(As + k * kLdTA + m, ok ? A + (size_t)(m0 + m) + (size_t)(k0 + k) * lda : A, ok);
        const int kb = idx & 15, n = idx >> 4;
        const bool okb = n0 + n < N && k0 + kb < K;
        cp_async16(Bs + n * kLdTB + kb, okb ? B + (size_t)(k0 + kb) + (size_t)(n0 + n) * ldb : B, okb);
      }
    }
    cp_async_commit();
  };
  const int wm = 16 * (warp & 3), wn = 32 * (warp >> 2);
  const int g = lane >> 2, tt = lane & 3;
  double re[4][4] = {}, im[4][4] = {};
  issue(0);
  issue(1);
  if (FACTOR) {
    // this tile of C (the first CTAs') and the tile of the CTA that follows in this
    // place come into L2 meanwhile: their loads are the only ones that otherwise wait
    // for DRAM (2688 x 4: 9.66 -> 9.28 ms)
    auto prefetch = [&](const double2* tile) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int line = tid + 256 * i;  // 8 lines of 128 bytes per column
        asm volatile("prefetch.global.L2 [%0];" ::"l"(tile + 8 * (line & 7) + (int64_t)(line >> 3) * ldc));
      }
    };
    if ((int)blockIdx.x < kResident) prefetch(C + m0 + (int64_t)n0 * ldc);
    const int next = (int)blockIdx.x + kResident;
    if (next >= batch && next < tiles * batch) {  // the first `batch` CTAs take the first tiles
      const int tn = 1 + (next - batch) % (tiles - 1), bn = (next - batch) / (tiles - 1);
      prefetch(C + (int64_t)(bn - b) * strideC + (tn % tiles_m) * kTile + (int64_t)(tn / tiles_m) * kTile * ldc);
    }
  }
#pragma unroll 1
  for (int q = 0; q < nk; ++q) {
    cp_async_wait<1>();  // chunk q has landed (this thread's part)
    __syncthreads();     // everybody's part; and everybody is done with chunk q - 1
    issue(q + 2);
    const double2* As = sm + (q % kStages) * kStageElems;
    warp_zmma<4>(As + wm, kLdTA, As + kDepth * kLdTA + wn * kLdTB, kLdTB, kDepth, re, im, lane);
  }
  if constexpr (FACTOR) {
    const bool diagonal = t == 0;
    if (diagonal) {
      cp_async_wait<0>();
      __syncthreads();  // the ring becomes the block
    }
    // C - (the whole product): one rounding of C's size per entry (accumulators that
    // start from C round to its size with every product).  The loads run a
    // step ahead of the stores, which might alias them.
    auto at = [&](int j, int e) {
      return C + (size_t)(m0 + wm + g + 8 * (e >> 1)) + (size_t)(n0 + wn + 8 * j + 2 * tt + (e & 1)) * ldc;
    };
    double2 c[2][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) c[0][e] = *at(0, e);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j + 1 < 4) {
#pragma unroll
        for (int e = 0; e < 4; ++e) c[(j + 1) & 1][e] = *at(j + 1, e);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const double2 v = make_double2(c[j & 1][e].x - re[j][e], c[j & 1][e].y - im[j][e]);
        if (diagonal) sm[(wn + 8 * j + 2 * tt + (e & 1)) * kLdD + wm + g + 8 * (e >> 1)] = v;
        else *at(j, e) = v;
      }
    }
    if (!diagonal) return;
    __syncthreads();
    factor_diagonal(sm, sm + kNB * kLdD, sh, C - kk - (int64_t)kk * ldc, ldc, kk, piv + (size_t)b * piv_stride,
                    info + b, inv + ((size_t)b * nblk + kk / kNB) * 2 * kNB * kNB);
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int m = m0 + wm + g + 8 * (e >> 1), n = n0 + wn + 8 * j + 2 * tt + (e & 1);
      if (m < M && n < N) {
        double2* p = C + (size_t)m + (size_t)n * ldc;
        double2 c = beta == 0.0 ? make_double2(0.0, 0.0) : *p;
        c.x = beta * c.x + alpha * re[j][e];
        c.y = beta * c.y + alpha * im[j][e];
        *p = c;
      }
    }
}

// The first diagonal block of every matrix.
__global__ void __launch_bounds__(256, 2) zlu_first_kernel(double2* __restrict__ A, int64_t lda, int64_t stride,
                                                           int* __restrict__ piv, int64_t piv_stride,
                                                           int* __restrict__ info, double2* __restrict__ inv,
                                                           int nblk) {
  extern __shared__ double2 sm[];
  __shared__ DiagShared sh;
  const int b = blockIdx.x;
  double2* Ab = A + (size_t)b * stride;
  for (int idx = threadIdx.x; idx < kNB * kNB; idx += 256) {
    const int r = idx % kNB, c = idx / kNB;
    sm[c * kLdD + r] = Ab[(size_t)r + (size_t)c * lda];
  }
  __syncthreads();
  factor_diagonal(sm, sm + kNB * kLdD, sh, Ab, lda, 0, piv + (size_t)b * piv_stride, info + b,
                  inv + (size_t)b * nblk * 2 * kNB * kNB);
}

// ---------------------------------------------------------------------------
// Persistent block substitution.  forward: y = L^{-1} P b; backward: x = U^{-1} y.
// B: (n, nrhs) column-major per matrix, in place.  flags: batch*nblk ints counting
// the sweeps that have finished the block row (forward 1, backward 2), ticket: one
// int that runs on over both; both zero before the forward sweep.  err: set to 1
// when a wait times out.
//
// A CTA owns a 64-row block; the bound is the chain of block rows.  Its blocks
// stream through a cp.async ring of 32-column slots, two slots ahead, so that
// only the right-hand sides of a dependency wait for its flag; thread (r, g)
// accumulates row r over a quarter of each slot's columns in registers over all
// dependencies, and the quarters meet once, before the product with the diagonal
// inverse.  One block row (3008 unknowns): 3.7 us with one right-hand side and 6.2
// with 7, from 5.1 and 8.9 with each block loaded before its flag was read and
// one thread per row and right-hand side.
__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}

constexpr int kTrsmRhs = 16;             // right-hand sides per launch
constexpr int kTrsmCols = 32, kTrsmSlots = 4;
constexpr int kTrsmSlot = kTrsmCols * kNB;
constexpr int trsm_smem(int nc) {
  return (kTrsmSlots * kTrsmSlot + kNB * kNB + 2 * kNB * nc) * (int)sizeof(double2);
}

template <int NC>
__global__ void __launch_bounds__(256) ztrsm_persistent_kernel(const double2* __restrict__ A, int64_t lda,
                                                               int64_t stride, int nblk, int batch,
                                                               const int* __restrict__ piv, int64_t piv_stride,
                                                               const double2* __restrict__ inv, double2* B,
                                                               int64_t ldb, int64_t strideB, int nrhs, int forward,
                                                               int* flags, int* ticket, int* err, const int* skip,
                                                               long long spin_limit, const int* mskip) {
  if (skip && *skip) return;  // refinement already converged
  extern __shared__ double2 sm[];
  double2* ring = sm;                             // slots of 32 columns x 64 rows
  double2* Inv = ring + kTrsmSlots * kTrsmSlot;   // inverse of the diagonal block, Inv[m * 64 + r]
  double2* X = Inv + kNB * kNB;                   // own block, X[r * NC + c]
  double2* Y = X + kNB * NC;                      // dependency block, Y[m * NC + c]
  __shared__ int s_t;
  const int tid = threadIdx.x;
  const int r = tid & (kNB - 1), g = tid >> 6;
  if (tid == 0) s_t = atomicAdd(ticket, 1);
  __syncthreads();
  const int t = s_t - (forward ? 0 : nblk * batch);
  const int b = t % batch, step = t / batch;
  if (mskip && mskip[b]) return;  // converged matrix: every CTA of it returns, no wait targets it
  const int i = forward ? step : (nblk - 1 - step);
  const double2* Ab = A + (size_t)b * stride;
  double2* Bb = B + (size_t)b * strideB;
  const int r0 = i * kNB, target = forward ? 1 : 2;
  const int ndep = forward ? i : (nblk - 1 - i), nq = 2 * ndep;
  // dependencies in the order they complete: 0 .. i-1 forward, nblk-1 .. i+1 backward
  auto block_of = [&](int q) { return forward ? (q >> 1) : (nblk - 1 - (q >> 1)); };
  auto issue = [&](int q) {
    if (q < nq) {
      double2* slot = ring + (q % kTrsmSlots) * kTrsmSlot;
      const double2* src = Ab + (size_t)r0 + (size_t)(block_of(q) * kNB + (q & 1) * kTrsmCols) * lda;
#pragma unroll
      for (int u = 0; u < kTrsmSlot / 256; ++u) {
        const int idx = tid + 256 * u;
        cp_async16(slot + idx, src + (size_t)(idx & (kNB - 1)) + (size_t)(idx >> 6) * lda, true);
      }
    }
    cp_async_commit();
  };
  {  // the diagonal inverse with the first slot's group
    const double2* invg = inv + ((size_t)b * nblk + i) * 2 * kNB * kNB + (forward ? 0 : kNB * kNB);
#pragma unroll
    for (int u = 0; u < kNB * kNB / 256; ++u) cp_async16(Inv + tid + 256 * u, invg + tid + 256 * u, true);
  }
  issue(0);
  issue(1);
  // own right-hand sides (permuted rows for the forward sweep)
  for (int idx = tid; idx < kNB * NC; idx += 256) {
    const int rr = idx & (kNB - 1), c = idx >> 6;
    double2 v = make_double2(0.0, 0.0);
    if (c < nrhs) {
      const int src = forward ? piv[(size_t)b * piv_stride + r0 + rr] : rr;
      v = __ldcg(Bb + (size_t)(r0 + src) + (size_t)c * ldb);
    }
    X[rr * NC + c] = v;
  }
  double2 acc[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) acc[c] = make_double2(0.0, 0.0);
  auto add = [&](double2 a, const double2* y) {  // acc += a y
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const double2 v = y[c];
      acc[c].x = fma(a.x, v.x, fma(-a.y, v.y, acc[c].x));
      acc[c].y = fma(a.x, v.y, fma(a.y, v.x, acc[c].y));
    }
  };
#pragma unroll 1
  for (int q = 0; q < nq; ++q) {
    if ((q & 1) == 0) {
      const int j = block_of(q);
      if (tid == 0) {
        long long it = 0;
        while (ld_acquire(flags + (size_t)b * nblk + j) < target) {
          if (++it > spin_limit) {
            atomicExch(err, 1);
            break;
          }
          __nanosleep(20);
        }
      }
      __syncthreads();  // the dependency is there, and everyone is done with Y
      for (int idx = tid; idx < kNB * NC; idx += 256) {
        const int m = idx & (kNB - 1), c = idx >> 6;
        Y[m * NC + c] = c < nrhs ? __ldcg(Bb + (size_t)(j * kNB + m) + (size_t)c * ldb) : make_double2(0.0, 0.0);
      }
    }
    issue(q + 2);       // its slot was read two products ago: a barrier lies between
    cp_async_wait<2>();  // this thread's copies of slot q have landed
    __syncthreads();     // everyone's, and Y
    const double2* slot = ring + (q % kTrsmSlots) * kTrsmSlot + 8 * g * kNB + r;
    const double2* y = Y + ((q & 1) * kTrsmCols + 8 * g) * NC;
#pragma unroll 4
    for (int m = 0; m < 8; ++m) add(slot[m * kNB], y + m * NC);
  }
  cp_async_wait<0>();
  __syncthreads();
  // the quarters' sums through the ring: red[(g * NC + c) * 64 + r]
  double2* red = ring;
  static_assert(4 * NC * kNB <= kTrsmSlots * kTrsmSlot, "the sums fit the ring");
#pragma unroll
  for (int c = 0; c < NC; ++c) red[(g * NC + c) * kNB + r] = acc[c];
  __syncthreads();
  for (int idx = tid; idx < kNB * NC; idx += 256) {
    const int rr = idx & (kNB - 1), c = idx >> 6;
    double2 v = X[rr * NC + c];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const double2 o = red[(h * NC + c) * kNB + rr];
      v.x -= o.x;
      v.y -= o.y;
    }
    X[rr * NC + c] = v;
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) acc[c] = make_double2(0.0, 0.0);
  __syncthreads();
#pragma unroll 4
  for (int m = 16 * g; m < 16 * g + 16; ++m) add(Inv[m * kNB + r], X + m * NC);
#pragma unroll
  for (int c = 0; c < NC; ++c) red[(g * NC + c) * kNB + r] = acc[c];
  __syncthreads();
  for (int idx = tid; idx < kNB * NC; idx += 256) {
    const int rr = idx & (kNB - 1), c = idx >> 6;
    if (c >= nrhs) break;
    double2 v = red[c * kNB + rr];
#pragma unroll
    for (int h = 1; h < 4; ++h) {
      const double2 o = red[(h * NC + c) * kNB + rr];
      v.x += o.x;
      v.y += o.y;
    }
    Bb[(size_t)(r0 + rr) + (size_t)c * ldb] = v;
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    atomicAdd(flags + (size_t)b * nblk + i, 1);
  }
}

__global__ void pad_identity_kernel(double2* A, int64_t lda, int64_t stride, int n, int npad) {
  // zero the padded rows/columns and put ones on the padded diagonal
  const int b = blockIdx.y;
  double2* Ab = A + (size_t)b * stride;
  const long long total = (long long)npad * (npad - n) * 2;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long half = (long long)npad * (npad - n);
    long long e = idx < half ? idx : idx - half;
    int r, c;
    if (idx < half) {  // padded columns
      r = (int)(e % npad);
      c = n + (int)(e / npad);
    } else {  // padded rows of the first n columns... and all columns
      r = n + (int)(e % (npad - n));
      c = (int)(e / (npad - n));
    }
    Ab[(size_t)r + (size_t)c * lda] = make_double2(r == c ? 1.0 : 0.0, 0.0);
  }
}

}  // namespace
}  // namespace bem

using namespace bem;

namespace {
int check_lu_args(const void* A, int n, int64_t lda, int batch) {
  if (!A) return set_error(BEM_ERR_INVALID_ARGUMENT, "null matrix pointer");
  if (n <= 0 || n % kNB != 0) return set_error(BEM_ERR_INVALID_ARGUMENT, "n must be a positive multiple of 64");
  if (lda < n) return set_error(BEM_ERR_INVALID_ARGUMENT, "lda < n");
  if (batch <= 0) return set_error(BEM_ERR_INVALID_ARGUMENT, "batch <= 0");
  return BEM_OK;
}
int opt_in_smem() {
  BEM_CUDA_CHECK(cudaFuncSetAttribute(zlu_first_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem));
  BEM_CUDA_CHECK(
      cudaFuncSetAttribute(zgemm_dmma_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem));
  BEM_CUDA_CHECK(
      cudaFuncSetAttribute(zgemm_dmma_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem));
  BEM_CUDA_CHECK(cudaFuncSetAttribute(zlu_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPanelSmem));
  BEM_CUDA_CHECK(
      cudaFuncSetAttribute(ztrsm_persistent_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, trsm_smem(4)));
  BEM_CUDA_CHECK(
      cudaFuncSetAttribute(ztrsm_persistent_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, trsm_smem(8)));
  BEM_CUDA_CHECK(
      cudaFuncSetAttribute(ztrsm_persistent_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, trsm_smem(16)));
  return BEM_OK;
}
OncePerDevice g_smem;
int configure_smem() { return configure_device(g_smem, opt_in_smem); }
}  // namespace

extern "C" int bem_zpad_identity(void* A_dev, int64_t lda, int64_t stride, int batch, int n, int npad, void* stream) {
  if (!A_dev || n < 0 || npad < n || lda < npad || batch <= 0)
    return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_zpad_identity: bad arguments");
  if (npad == n) return BEM_OK;
  dim3 grid(256, batch);
  pad_identity_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((double2*)A_dev, lda, stride, n, npad);
  count_launches(1);
  BEM_CUDA_CHECK(cudaGetLastError());
  return BEM_OK;
}

extern "C" int bem_zgemm(int M, int N, int K, double alpha, const void* A_dev, int64_t lda, int64_t strideA,
                         const void* B_dev, int64_t ldb, int64_t strideB, double beta, void* C_dev, int64_t ldc,
                         int64_t strideC, int batch, void* stream) {
  if (M < 0 || N < 0 || K < 0 || batch <= 0) return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_zgemm: bad sizes");
  if (M == 0 || N == 0) return BEM_OK;
  if (!A_dev || !B_dev || !C_dev) return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_zgemm: null pointer");
  int st = configure_smem();
  if (st) return st;
  const int tiles_m = ceil_div(M, kTile), tiles = tiles_m * ceil_div(N, kTile);
  zgemm_dmma_kernel<false><<<tiles * batch, 256, kGemmSmem, (cudaStream_t)stream>>>(
      M, N, K, alpha, (const double2*)A_dev, lda, strideA, (const double2*)B_dev, ldb, strideB, beta,
      (double2*)C_dev, ldc, strideC, tiles_m, tiles, batch, 0, nullptr, 0, nullptr, nullptr, 0);
  count_launches(1);
  BEM_CUDA_CHECK(cudaGetLastError());
  return BEM_OK;
}

extern "C" int64_t bem_zlu_workspace_bytes(int n, int batch) {
  const int nblk = n / kNB;
  // inverses, block-row flags, then ticket, refinement flag and per-matrix convergence flags
  return (int64_t)batch * nblk * 2 * kNB * kNB * (int64_t)sizeof(double2) + (int64_t)batch * nblk * 4 +
         (int64_t)batch * 4 + 256;
}

extern "C" int bem_zlu_factor(void* A_dev, int n, int64_t lda, int64_t stride, int batch, int* piv_dev,
                              int* info_dev, void* work_dev, void* stream) {
  int st = check_lu_args(A_dev, n, lda, batch);
  if (st) return st;
  if (!piv_dev || !info_dev || !work_dev) return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_zlu_factor: null pointer");
  if ((st = configure_smem())) return st;
  cudaStream_t s = (cudaStream_t)stream;
  double2* A = (double2*)A_dev;
  double2* inv = (double2*)work_dev;
  const int nblk = n / kNB;
  BEM_CUDA_CHECK(cudaMemsetAsync(info_dev, 0, sizeof(int) * batch, s));
  {
    TimedLaunch tl(kKZluFirst, s);
    zlu_first_kernel<<<batch, 256, kGemmSmem, s>>>(A, lda, stride, piv_dev, n, info_dev, inv, nblk);
  }
  count_launches(1);
  for (int kk = 0; kk < n; kk += kNB) {
    const int m = n - kk - kNB;
    const int ntiles = kk / kNB + 2 * (m / kPanelTile);
    if (ntiles > 0) {
      TimedLaunch tl(kKZluPanel, s);
      zlu_panel_kernel<<<dim3(ntiles, batch), 256, kPanelSmem, s>>>(A, lda, stride, n, kk, piv_dev, n, inv, nblk);
      count_launches(1);
    }
    if (m > 0) {
      const int tiles_m = m / kTile, tiles = tiles_m * tiles_m, next = kk + kNB;
      TimedLaunch tl(kKZgemmDmma, s);
      zgemm_dmma_kernel<true><<<tiles * batch, 256, kGemmSmem, s>>>(
          m, m, kNB, -1.0, A + (size_t)next + (size_t)kk * lda, lda, stride, A + (size_t)kk + (size_t)next * lda, lda,
          stride, 1.0, A + (size_t)next + (size_t)next * lda, lda, stride, tiles_m, tiles, batch, next, piv_dev, n,
          info_dev, inv, nblk);
      count_launches(1);
    }
  }
  BEM_CUDA_CHECK(cudaGetLastError());
  return BEM_OK;
}

namespace bem {
// Address of the "converged" flag of a refinement with these factors: an int
// in the workspace tail after the block-row flags and the ticket.
int* zlu_done_flag(void* work_dev, int n, int batch) {
  const int nblk = n / kNB;
  int* flags = (int*)((char*)work_dev + (size_t)batch * nblk * 2 * kNB * kNB * sizeof(double2));
  return flags + (size_t)batch * nblk + 1;
}

// Forward and backward block substitutions with the float64 factors, in place
// on B; every launch returns at once while *skip != 0.
int zlu_solve_enqueue(const void* A_dev, int n, int64_t lda, int64_t stride, int batch, const int* piv_dev,
                      const void* work_dev, void* B_dev, int64_t ldb, int64_t strideB, int nrhs, int* err_dev,
                      cudaStream_t s, const int* skip, long long spin_limit, const int* mskip) {
  int st = configure_smem();
  if (st) return st;
  const int nblk = n / kNB;
  const double2* inv = (const double2*)work_dev;
  int* flags = (int*)((char*)work_dev + (size_t)batch * nblk * 2 * kNB * kNB * sizeof(double2));
  int* ticket = flags + (size_t)batch * nblk;
  for (int c0 = 0; c0 < nrhs; c0 += kTrsmRhs) {
    const int nc = std::min(kTrsmRhs, nrhs - c0);
    double2* Bc = (double2*)B_dev + (size_t)c0 * ldb;
    BEM_CUDA_CHECK(cudaMemsetAsync(flags, 0, sizeof(int) * ((size_t)batch * nblk + 1), s));
    auto* kernel = nc <= 4   ? ztrsm_persistent_kernel<4>
                   : nc <= 8 ? ztrsm_persistent_kernel<8>
                             : ztrsm_persistent_kernel<16>;
    const int smem = trsm_smem(nc <= 4 ? 4 : nc <= 8 ? 8 : 16);
    for (int forward = 1; forward >= 0; --forward) {
      TimedLaunch tl(kKZtrsm, s);
      kernel<<<nblk * batch, 256, smem, s>>>((const double2*)A_dev, lda, stride, nblk, batch, piv_dev, n, inv, Bc, ldb,
                                             strideB, nc, forward, flags, ticket, err_dev, skip, spin_limit, mskip);
      count_launches(1);
    }
  }
  BEM_CUDA_CHECK(cudaGetLastError());
  return BEM_OK;
}
}  // namespace bem

extern "C" int bem_zlu_solve(const void* A_dev, int n, int64_t lda, int64_t stride, int batch, const int* piv_dev,
                             const void* work_dev, void* B_dev, int64_t ldb, int64_t strideB, int nrhs,
                             int* err_dev, void* stream) {
  int st = check_lu_args(A_dev, n, lda, batch);
  if (st) return st;
  if (!piv_dev || !work_dev || !B_dev || !err_dev) return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_zlu_solve: null");
  if (nrhs <= 0 || nrhs > kNB) return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_zlu_solve: nrhs must be in [1, 64]");
  if (ldb < n) return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_zlu_solve: ldb < n");
  return zlu_solve_enqueue(A_dev, n, lda, stride, batch, piv_dev, work_dev, B_dev, ldb, strideB, nrhs, err_dev,
                           (cudaStream_t)stream, nullptr, kDefaultSpinLimit);
}

