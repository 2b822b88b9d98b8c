// Mixed-precision complex LU with float64-residual iterative refinement.
//
// Replaces the complex128 zgetrf/zgetrs solve of capytaine
// (tools/block_circulant_matrices.py:361-385, bem/engines.py:300-346) by:
//   * a float32 copy of K in two planes (real, imaginary), column-major, padded
//     to a multiple of 128 with the identity;
//   * a blocked right-looking block LU with 128-wide blocks, A = L U with L
//     unit block lower (L_ik = A_ik A_kk^{-1}) and U block upper (the updated
//     block rows): each diagonal block is inverted by Gauss-Jordan elimination
//     with partial pivoting among its rows, held in registers; the panel is the
//     product A21 A_kk^{-1}; the trailing update C -= L21 U12 runs on the
//     tcgen05 tensor cores (TF32 inputs, FP32 accumulation; tc_gemm.cu) from
//     packed operands (A12 and A21 by a pack kernel, L21 by the epilogue of
//     the panel product).  No row permutation leaves the diagonal blocks, so
//     the solves need none;
//   * block substitutions with these factors (persistent kernel); the block
//     rows of U are stored pre-multiplied by the diagonal inverses (U' =
//     A_kk^{-1} A12, computed beside the panel), so that the backward sweep
//     applies A_ii^{-1} to its own right-hand side before its dependencies;
//   * iterative refinement: x += LU^{-1} (b - K x) with the residual computed
//     in float64 against the float64 matrix until the relative residual of
//     every right-hand side is below the requested tolerance.
#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <vector>
#include "common.cuh"
#include "reciprocals.cuh"

namespace bem {

namespace {

constexpr int kB = 128;        // LU block
constexpr int kPT = 64;        // panel tile width
constexpr int kSplitK = 6 * kB;  // A row of the split-TF32 panel product: (hi, lo, hi) x (re, im) x 128
constexpr int kSplitB = 2 * kB;  // its B row: (hi, lo) x 128
// depths of the update (A row [Re | Im], B row of one part) and of the panel
// product (A_hi B_hi + A_lo B_hi + A_hi B_lo)
constexpr CgemmDepth kUpdateDepth{kB, 2 * kB, kB, 1, kB, 0, {0, 0, 0}, false};
constexpr CgemmDepth kSplitDepth{kB, kSplitK, kSplitB, 3, kB, 2 * kB, {0, 0, kB}, false};
constexpr int kRhs = 16;       // right-hand sides per solve launch
constexpr int kOpBuffers = 3;  // packed operands of the current, previous and next block steps

__device__ __forceinline__ float2 fmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// a b + c on a pair of floats in one instruction (fma.rn.f32x2: per element the
// correctly rounded fused multiply-add of fmaf)
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n.reg .b64 ra, rb, rc, rd;\n"
      "mov.b64 ra, {%2, %3};\nmov.b64 rb, {%4, %5};\nmov.b64 rc, {%6, %7};\n"
      "fma.rn.f32x2 rd, ra, rb, rc;\nmov.b64 {%0, %1}, rd;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

struct Planes {
  float* re;
  float* im;
  int64_t ld;      // = npad
  int64_t stride;  // floats between matrices (re and im planes of one matrix are plane apart)
};
// The part of x that TF32 keeps (the low 13 mantissa bits cleared); x - hi is
// exact in float32 and is the "lo" part of the split product.
__device__ __forceinline__ float tf32_hi(float x) { return __uint_as_float(__float_as_uint(x) & 0xffffe000u); }

__device__ __forceinline__ void stp(const Planes& W, int b, int r, int c, float2 v) {
  const size_t o = (size_t)b * W.stride + (size_t)r + (size_t)c * W.ld;
  W.re[o] = v.x;
  W.im[o] = v.y;
}

// K (complex128, n x n, leading dimension ldk) -> planes (npad x npad) with the
// identity on the padding.
__global__ void convert_pad_kernel(const double2* __restrict__ K, int64_t ldk, int64_t strideK, int n, int npad,
                                   Planes W) {
  const int b = blockIdx.z;
  const int c = blockIdx.y;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < npad; r += gridDim.x * blockDim.x) {
    float2 v;
    if (r < n && c < n) {
      const double2 z = K[(size_t)b * strideK + (size_t)r + (size_t)c * ldk];
      v = make_float2((float)z.x, (float)z.y);
    } else {
      v = make_float2(r == c ? 1.0f : 0.0f, 0.0f);
    }
    stp(W, b, r, c, v);
  }
}

// Gauss-Jordan inverse of a diagonal block in panels of 8 columns, one per warp:
// warp w has columns 8 w .. 8 w + 7 of the 128 x 128 block, which lies in shared
// memory as two planes; lane l has the rows 2 l, 2 l + 1, 64 + 2 l and 65 + 2 l.
// Pivoting is implicit: rows never move.  Step j picks the pivot of column j
// among the rows not yet used as pivot rows (row p_j) and eliminates column j
// from every other row with the unnormalised row p_j:
//   a_r -= (a_rj / a_pj) a_p   (r != p_j),
// the in-place inverse's column j ending as -a_rj / a_pj, with 1 in row p_j.
// The eight steps of a panel act on a column x outside it as
//   x <- x + sum_s (P_s - e_{p_s}) x_{p_s},
// P_s the panel's columns after its steps and x_{p_s} the column's entries in the
// pivot rows before them (each step is I - f e_p^T, and P_s is the product of the
// steps applied to e_{p_s}): a rank-8 update from the panel as it lies.
// Row p_j thus stays scaled by its pivot; at the end
//   A^{-1}(j', p_c) = a(p_j', c) / pivot_j'
// (row p_j' holds the j'-th pivot row, the place of column c the inverse's
// column p_c).
constexpr int kGjPanel = 8;               // columns per warp and panel
constexpr int kGjWarps = kB / kGjPanel;
constexpr int kGjDepth = 4;               // panels published ahead of the slowest warp
constexpr int kGjLd = kB + 2;             // column stride of a plane (row pairs aligned, two-way conflicts across)
constexpr int kGjSmem = (2 * kB * kGjLd + kGjDepth * kGjPanel * 2 * kB) * (int)sizeof(float);  // dynamic
constexpr long long kGjWaitLimit = 1ll << 22;  // polls of a bounded wait (about a second)

__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n.reg .b64 ra, rb, rd;\n"
      "mov.b64 ra, {%2, %3};\nmov.b64 rb, {%4, %5};\n"
      "mul.rn.f32x2 rd, ra, rb;\nmov.b64 {%0, %1}, rd;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

__device__ __forceinline__ uint32_t gj_smem(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void gj_bar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(gj_smem(bar)), "r"(count));
}
__device__ __forceinline__ void gj_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(gj_smem(bar)) : "memory");
}
__device__ __forceinline__ bool gj_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(gj_smem(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

struct GjShared {
  // full[s]: the panel of buffer s is published (32 arrivals, the owner's
  // lanes); empty[s]: every other warp has read it (15 arrivals, one per warp).
  uint64_t full[kGjDepth];
  uint64_t empty[kGjDepth];
  // per warp: entries (re, re, im, im) of pivot rows in its columns
  alignas(16) float4 rows[kGjWarps][kGjPanel][kGjPanel];
  float2 rowscale[kB];              // 1 / pivot of the step whose pivot row is this row
  alignas(16) int piv_row[kB];      // pivot row of each step
  alignas(16) int jinv[kB];         // step of each pivot row
  unsigned char used[kB];           // rows already used as pivot rows
  int abort;                        // a wait ran out: every warp leaves
};

// Bounded wait of a whole warp for phase `parity` of bar (every lane polls,
// so that every lane acquires the published data); false for the whole warp
// when a lane reached the limit or another warp gave up (the warp then leaves
// its loop, with no lane left behind in a warp-synchronous call).
__device__ __forceinline__ bool gj_wait(uint64_t* bar, uint32_t parity, GjShared& sh, int* __restrict__ err) {
  bool ok = false, gave_up = false;
  for (long long it = 0; it < kGjWaitLimit; ++it) {
    if (gj_try_wait(bar, parity)) {
      ok = true;
      break;
    }
    if (*(volatile int*)&sh.abort) {
      gave_up = true;
      break;
    }
  }
  if (!ok && !gave_up) {
    *(volatile int*)&sh.abort = 1;
    atomicExch(err, 1);
  }
  return __all_sync(0xffffffffu, ok);
}

// Ordered key of a pivot candidate: the bits of |re| + |im| with the last seven
// replaced by the row, so that one reduction finds the value and the row
// (values within 2^-16 of the largest count as equal and the first row wins).
// A NaN counts as zero; left: all ones, or 0 for a row already used (key 0).
__device__ __forceinline__ unsigned gj_key(float re, float im, int row, unsigned left) {
  const float m = fmaxf(fabsf(re) + fabsf(im), 0.0f);
  return (((__float_as_uint(m) + 128u) & ~127u) | (unsigned)(127 - row)) & left;
}

// A warp's columns in registers: [pair of rows][column], planes apart.
struct GjColumns {
  float2 re[2][kGjPanel], im[2][kGjPanel];
};

// acc += p y, y = (re, re, im, im) of one column's pivot-row entry, p two rows.
__device__ __forceinline__ void gj_fma(float2& re, float2& im, float2 pr, float2 pi, float2 npi, float4 y) {
  const float2 yr = make_float2(y.x, y.y), yi = make_float2(y.z, y.w);
  re = fma2(npi, yi, fma2(pr, yr, re));
  im = fma2(pi, yr, fma2(pr, yi, im));
}

// The eight steps of panel q on its own columns, by its warp: a becomes P.  The
// columns rotate through the register slots (the current one in slot 0, each
// update landing one slot below, the finished column in the last), so that the
// loop is 400 instructions; eight steps bring every column back to its slot.
__device__ __forceinline__ void gj_factor(GjColumns& a, int q, int kk, int b, int lane, GjShared& sh,
                                          int* __restrict__ info) {
  const int r0 = 2 * lane;
  unsigned left[4];  // rows r0, r0 + 1, r0 + 64, r0 + 65 not used yet
#pragma unroll
  for (int i = 0; i < 4; ++i) left[i] = sh.used[r0 + (i & 1) + 64 * (i >> 1)] ? 0u : ~0u;
  auto column_key = [&]() {
    const unsigned k0 = max(gj_key(a.re[0][0].x, a.im[0][0].x, r0, left[0]),
                            gj_key(a.re[0][0].y, a.im[0][0].y, r0 + 1, left[1]));
    const unsigned k1 = max(gj_key(a.re[1][0].x, a.im[1][0].x, r0 + 64, left[2]),
                            gj_key(a.re[1][0].y, a.im[1][0].y, r0 + 65, left[3]));
    return __reduce_max_sync(0xffffffffu, max(k0, k1));
  };
  unsigned key = column_key();
  int my_p = 0;  // of step s in lane s: stored once at the end
  float2 my_scale = make_float2(0.0f, 0.0f);
#pragma unroll 1
  for (int s = 0; s < kGjPanel; ++s) {
    const int p = 127 - (int)(key & 127u), src = (p & 63) >> 1;
    // the pivot row's entries from its lane (the branch is the warp's: p is)
    float ur[kGjPanel], ui[kGjPanel];
#define BEM_GJ_ROW(H, C)                                            \
  _Pragma("unroll") for (int m = 0; m < kGjPanel; ++m) {            \
    ur[m] = __shfl_sync(0xffffffffu, a.re[H][m].C, src);            \
    ui[m] = __shfl_sync(0xffffffffu, a.im[H][m].C, src);            \
  }
    if (p & 64) {
      if (p & 1) { BEM_GJ_ROW(1, y) } else { BEM_GJ_ROW(1, x) }
    } else {
      if (p & 1) { BEM_GJ_ROW(0, y) } else { BEM_GJ_ROW(0, x) }
    }
#undef BEM_GJ_ROW
    const float2 recip = gj_reciprocal(ur[0], ui[0]);
    const float dr = recip.x, di = recip.y;
    const bool own[4] = {p == r0, p == r0 + 1, p == r0 + 64, p == r0 + 65};
#pragma unroll
    for (int i = 0; i < 4; ++i) left[i] = own[i] ? 0u : left[i];
    // multipliers a_rj / pivot; 0 on the pivot row, which stays as it is
    float2 nr[2], fi[2], ni[2], done_re[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float2 ar = a.re[h][0], ai = a.im[h][0];
      float2 f = fma2(ai, make_float2(-di, -di), mul2(ar, make_float2(dr, dr)));
      fi[h] = fma2(ai, make_float2(dr, dr), mul2(ar, make_float2(di, di)));
      if (own[2 * h]) f.x = fi[h].x = 0.0f;
      if (own[2 * h + 1]) f.y = fi[h].y = 0.0f;
      nr[h] = neg2(f);
      ni[h] = neg2(fi[h]);
      done_re[h] = make_float2(own[2 * h] ? 1.0f : nr[h].x, own[2 * h + 1] ? 1.0f : nr[h].y);
    }
#pragma unroll
    for (int m = 1; m < kGjPanel; ++m) {
      const float4 y = make_float4(ur[m], ur[m], ui[m], ui[m]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float2 re = a.re[h][m], im = a.im[h][m];
        gj_fma(re, im, nr[h], ni[h], fi[h], y);
        a.re[h][m - 1] = re;
        a.im[h][m - 1] = im;
      }
      // the next pivot's column came first: its reduction runs beside the others' updates
      if (m == 1) key = column_key();
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      a.re[h][kGjPanel - 1] = done_re[h];
      a.im[h][kGjPanel - 1] = ni[h];
    }
    if (lane == s) {
      my_p = p;
      my_scale = make_float2(dr, di);
    }
  }
  if (lane < kGjPanel) {
    sh.piv_row[kGjPanel * q + lane] = my_p;
    sh.rowscale[my_p] = my_scale;
    sh.used[my_p] = 1;
  }
  const bool sound = isfinite(my_scale.x) && isfinite(my_scale.y) && (my_scale.x != 0.0f || my_scale.y != 0.0f);
  const unsigned bad = __ballot_sync(0xffffffffu, lane < kGjPanel && !sound);
  if (bad && lane == 0 && info[b] == 0) info[b] = kk + kGjPanel * q + __ffs(bad);
}

// Inverse of the diagonal block A_kk by Gauss-Jordan elimination with partial
// pivoting among its rows (implicit, in panels, see above).  The warps do not
// step together: panel q's warp factors it as soon as it has applied panel
// q - 1, and publishes it (shared-memory buffers guarded by mbarriers, kGjDepth
// panels deep) while the other warps still apply the earlier ones; those that
// share its scheduler (warps a multiple of four apart) stay a panel behind.
// Bound: the chain of panels on one SM, 8000 cycles each: the factorisation 4400
// (540 a column: shuffles of the pivot row, reciprocal, multipliers, the key and
// its reduction), the next warp's rank-8 update 2050, the exchange 1300; the
// other warps' updates (5000 a scheduler) run beside it.  79 us per block (77
// without the range check of the pivots' squares, 80 with a pass of its own for the
// scaling and a serial loop of the stores besides).  One
// step per exchange took 1800 cycles a column (121 us per block with the packed
// copies written by the same CTA): a pivot search, two trips through shared
// memory and a barrier each.  Row pairs and duplicated pivot entries feed the
// pair instructions without moves; interleaved complex entries in registers
// spent as much on moves and divergent row extraction as panels saved (170 us).
// Output: inv (128 x 128, column-major) = A_kk^{-1}; info flags a pivot without a
// finite reciprocal; err is set when a bounded wait runs out.
__global__ void __launch_bounds__(32 * kGjWarps, 1) clu_gj_kernel(Planes W, int kk, int* __restrict__ info,
                                                                 float2* __restrict__ inv, int nblk,
                                                                 int* __restrict__ err) {
  extern __shared__ __align__(16) float gj_smem_f[];
  float* Mre = gj_smem_f;              // the block: element (r, c) at c * kGjLd + r
  float* Mim = Mre + kB * kGjLd;
  float* panels = Mim + kB * kGjLd;    // [buffer][column][plane][row]
  __shared__ GjShared sh;
  const int b = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, w = tid >> 5;
  const int r0 = 2 * lane;
  {
    const float* gr = W.re + (size_t)b * W.stride + (size_t)kk + r0;
    const float* gi = W.im + (size_t)b * W.stride + (size_t)kk + r0;
#pragma unroll
    for (int m = 0; m < kGjPanel; ++m) {
      const int c = kGjPanel * w + m;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const size_t g = (size_t)(kk + c) * W.ld + 64 * h;
        *reinterpret_cast<float2*>(Mre + c * kGjLd + r0 + 64 * h) = *reinterpret_cast<const float2*>(gr + g);
        *reinterpret_cast<float2*>(Mim + c * kGjLd + r0 + 64 * h) = *reinterpret_cast<const float2*>(gi + g);
      }
    }
  }
  if (tid < kGjDepth) {
    gj_bar_init(&sh.full[tid], 32);
    gj_bar_init(&sh.empty[tid], kGjWarps - 1);
  }
  if (tid < kB) sh.used[tid] = 0;
  if (tid == 0) sh.abort = 0;
  __syncthreads();
  float* const mr = Mre + kGjPanel * w * kGjLd + r0;  // this lane's rows of the warp's columns
  float* const mi = Mim + kGjPanel * w * kGjLd + r0;
  GjColumns a;
#pragma unroll 1
  for (int q = 0; q < kGjWarps; ++q) {
    const int s = q % kGjDepth, parity = (q / kGjDepth) & 1;
    float* pan = panels + (size_t)s * kGjPanel * 2 * kB;
    const bool owner = q == w;
    if (!owner) {
      if (!gj_wait(&sh.full[s], parity, sh, err)) break;
      // the next panel's warp has its scheduler for itself until it has published
      const int next = q + 1;
      if (next < kGjWarps && w != next && ((w ^ next) & 3) == 0 &&
          !gj_wait(&sh.full[next % kGjDepth], (next / kGjDepth) & 1, sh, err))
        break;
      // this warp's entries of the pivot rows, which then start from zero
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int e = (lane >> 3) + 4 * u, m = lane & 7;
        const int o = (kGjPanel * w + m) * kGjLd + sh.piv_row[kGjPanel * q + e];
        const float re = Mre[o], im = Mim[o];
        sh.rows[w][e][m] = make_float4(re, re, im, im);
        Mre[o] = 0.0f;
        Mim[o] = 0.0f;
      }
      __syncwarp();
    }
#pragma unroll
    for (int m = 0; m < kGjPanel; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        a.re[h][m] = *reinterpret_cast<const float2*>(mr + m * kGjLd + 64 * h);
        a.im[h][m] = *reinterpret_cast<const float2*>(mi + m * kGjLd + 64 * h);
      }
    if (owner) {
      gj_factor(a, q, kk, b, lane, sh, info);
      // the buffer is free once every other warp has read panel q - kGjDepth
      if (q >= kGjDepth && !gj_wait(&sh.empty[s], parity ^ 1, sh, err)) break;
#pragma unroll
      for (int m = 0; m < kGjPanel; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          *reinterpret_cast<float2*>(pan + (2 * m) * kB + r0 + 64 * h) = a.re[h][m];
          *reinterpret_cast<float2*>(pan + (2 * m + 1) * kB + r0 + 64 * h) = a.im[h][m];
        }
      gj_arrive(&sh.full[s]);  // release: this lane's writes above
    } else {
#pragma unroll 2
      for (int e = 0; e < kGjPanel; ++e) {
        float2 pr[2], pi[2], npi[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          pr[h] = *reinterpret_cast<const float2*>(pan + (2 * e) * kB + r0 + 64 * h);
          pi[h] = *reinterpret_cast<const float2*>(pan + (2 * e + 1) * kB + r0 + 64 * h);
          npi[h] = neg2(pi[h]);
        }
#pragma unroll
        for (int m = 0; m < kGjPanel; ++m) {
          const float4 y = sh.rows[w][e][m];
#pragma unroll
          for (int h = 0; h < 2; ++h) gj_fma(a.re[h][m], a.im[h][m], pr[h], pi[h], npi[h], y);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < kGjPanel; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        *reinterpret_cast<float2*>(mr + m * kGjLd + 64 * h) = a.re[h][m];
        *reinterpret_cast<float2*>(mi + m * kGjLd + 64 * h) = a.im[h][m];
      }
    __syncwarp();  // the warp's reads of the panel are done, its columns are stored
    if (!owner && lane == 0) gj_arrive(&sh.empty[s]);
  }
  __syncthreads();
  if (sh.abort) return;
  if (tid < kB) sh.jinv[sh.piv_row[tid]] = tid;
  __syncthreads();
  // A_kk^{-1}(row, col) = a(piv_row[row], jinv[col]) / pivot of the row: column-major
  // 128 x 128, a lane's four rows 32 apart
  int p[4];
  float2 scale[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    p[u] = sh.piv_row[lane + 32 * u];
    scale[u] = sh.rowscale[p[u]];
  }
  float2* out = inv + ((size_t)b * nblk + kk / kB) * kB * kB + lane;
#pragma unroll 4
  for (int m = 0; m < kGjPanel; ++m) {
    const int col = w + kGjWarps * m, o = sh.jinv[col] * kGjLd;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      out[col * kB + 32 * u] = fmul(make_float2(Mre[o + p[u]], Mim[o + p[u]]), scale[u]);
  }
}

// The inverse of block kk as the operands of two products, 8 columns and 8 rows
// per CTA: the inverse's own CTA took 20 us to write them.
// binv: B operand of the split-TF32 product L21 = A21 A_kk^{-1} (see
// clu_pack_kernel for the A side): row t [hi Re X(:, t) | lo Re X(:, t)], row 128 + t
// the imaginary parts.
// ainv: A operand of U' = A_kk^{-1} A12, row r [Re A_kk^{-1}(r, :) | Im A_kk^{-1}(r, :)].
__global__ void __launch_bounds__(256) clu_inverse_pack_kernel(const float2* __restrict__ inv, int nblk, int kk,
                                                              float* __restrict__ binv, float* __restrict__ ainv) {
  const int b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, t = 8 * blockIdx.x + (tid >> 5);
  const float2* X = inv + ((size_t)b * nblk + kk / kB) * kB * kB;
  {
    const float4* col = reinterpret_cast<const float4*>(X + (size_t)t * kB) + 2 * lane;
    const float4 v0 = col[0], v1 = col[1];
    const float4 re = make_float4(v0.x, v0.z, v1.x, v1.z), im = make_float4(v0.y, v0.w, v1.y, v1.w);
    const float4 hr = make_float4(tf32_hi(re.x), tf32_hi(re.y), tf32_hi(re.z), tf32_hi(re.w));
    const float4 hi = make_float4(tf32_hi(im.x), tf32_hi(im.y), tf32_hi(im.z), tf32_hi(im.w));
    float* bo = binv + (size_t)b * (2 * kB) * kSplitB;
    float4* rr = reinterpret_cast<float4*>(bo + (size_t)t * kSplitB) + lane;
    float4* ri = reinterpret_cast<float4*>(bo + (size_t)(kB + t) * kSplitB) + lane;
    rr[0] = hr;
    rr[kB / 4] = make_float4(re.x - hr.x, re.y - hr.y, re.z - hr.z, re.w - hr.w);
    ri[0] = hi;
    ri[kB / 4] = make_float4(im.x - hi.x, im.y - hi.y, im.z - hi.z, im.w - hi.w);
  }
  float2 v[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) v[e] = X[(size_t)(4 * lane + e) * kB + t];
  float4* dst = reinterpret_cast<float4*>(ainv + (size_t)b * kB * 2 * kB + (size_t)t * 2 * kB) + lane;
  dst[0] = make_float4(tf32_rn(v[0].x), tf32_rn(v[1].x), tf32_rn(v[2].x), tf32_rn(v[3].x));
  dst[kB / 4] = make_float4(tf32_rn(v[0].y), tf32_rn(v[1].y), tf32_rn(v[2].y), tf32_rn(v[3].y));
}

// Operand packing of block step kk of the block LU (A_kk^{-1} is packed by
// clu_inverse_pack_kernel, L21 by the epilogue of the panel product).
// Blocks [0, nrest): the block row to the right of the diagonal, 64 columns
// each, packed as the B operand (U12 = A12).  Blocks [nrest, nrest +
// nrows/32): 32 rows of the block column [col0, col0 + 128) from row row0 on,
// packed K-major into A3 as the split-TF32 operand of the panel product (A21).
// Both through shared memory, so that reads and writes are coalesced.
// Bop: [batch][2*npad][kB]; A3: [batch][npad][kSplitK].
__global__ void __launch_bounds__(256) clu_pack_kernel(Planes W, int npad, int kk, int nrest, int row0, int col0,
                                                       float* __restrict__ Bop, float* __restrict__ A3, int t0) {
  __shared__ float tre[kB][33], tim[kB][33];  // [column][row] of a 32 x 128 tile
  const int b = blockIdx.y, tid = threadIdx.x;
  const int t = blockIdx.x + t0;  // a launch may cover a range of the blocks only
  if (t < nrest) {
    // 128 x 64 of A12: B operand rows of the complex columns c0 .. c0+63;
    // thread (q, cc): rows 4 q .. 4 q + 3 of column cc (16-byte loads and stores)
    const int c0 = kk + kB + t * kPT;
    const int j0 = c0 & ~(kB - 1);
    float* Bb = Bop + (size_t)b * 2 * npad * kB;
    const float* re = W.re + (size_t)b * W.stride;
    const float* im = W.im + (size_t)b * W.stride;
    const int q = tid & 31;
    for (int c = tid >> 5; c < kPT; c += 8) {
      const size_t g = (size_t)(c0 + c) * W.ld + kk + 4 * q;
      float4 ur = *reinterpret_cast<const float4*>(re + g);
      float4 ui = *reinterpret_cast<const float4*>(im + g);
      ur = make_float4(tf32_rn(ur.x), tf32_rn(ur.y), tf32_rn(ur.z), tf32_rn(ur.w));  // TF32 operands
      ui = make_float4(tf32_rn(ui.x), tf32_rn(ui.y), tf32_rn(ui.z), tf32_rn(ui.w));
      const int jj = c0 - j0 + c;
      reinterpret_cast<float4*>(Bb + (size_t)(2 * j0 + jj) * kB)[q] = ur;
      reinterpret_cast<float4*>(Bb + (size_t)(2 * j0 + kB + jj) * kB)[q] = ui;
    }
    return;
  }
  const int r0 = row0 + (t - nrest) * 32;
  const float* re = W.re + (size_t)b * W.stride;
  const float* im = W.im + (size_t)b * W.stride;
  {
    // thread (q, c): rows 4 q .. 4 q + 3 of column c, 16-byte loads
    const int q = tid & 7;
    for (int c = tid >> 3; c < kB; c += 32) {
      const size_t g = (size_t)(col0 + c) * W.ld + r0 + 4 * q;
      const float4 vr = *reinterpret_cast<const float4*>(re + g);
      const float4 vi = *reinterpret_cast<const float4*>(im + g);
      tre[c][4 * q] = vr.x;
      tre[c][4 * q + 1] = vr.y;
      tre[c][4 * q + 2] = vr.z;
      tre[c][4 * q + 3] = vr.w;
      tim[c][4 * q] = vi.x;
      tim[c][4 * q + 1] = vi.y;
      tim[c][4 * q + 2] = vi.z;
      tim[c][4 * q + 3] = vi.w;
    }
  }
  __syncthreads();
  // split rows [hi | lo | hi], each [Re(128) | Im(128)], for the panel
  // product; thread (q, i0): entries 4 q .. 4 q + 3 of rows i0, i0 + 4, ...
  float* dst = A3 + (size_t)b * npad * kSplitK + (size_t)r0 * kSplitK;
  const int q = tid & 63;
  const float(*src)[33] = q < 32 ? tre : tim;
  const int cb = 4 * (q & 31);
  for (int i = tid >> 6; i < 32; i += 4) {
    float h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float x = src[cb + e][i];
      h[e] = tf32_hi(x);
      l[e] = x - h[e];
    }
    float4* row = reinterpret_cast<float4*>(dst + (size_t)i * kSplitK);
    row[q] = make_float4(h[0], h[1], h[2], h[3]);
    row[2 * kB / 4 + q] = make_float4(l[0], l[1], l[2], l[3]);
    row[4 * kB / 4 + q] = make_float4(h[0], h[1], h[2], h[3]);
  }
}

// The next diagonal block's update by block step kk in one launch of its own,
// D -= A21 (A_kk^{-1} A12) in float32 from the unpacked blocks, as soon as the
// inverse is there: the chain of diagonal blocks need not wait for the packed
// inverse, the panel product over the whole block column (one 128 x 128 tile
// takes it 19 us whatever the column's height) and a tensor-core tile, which
// follow beside the next inverse.
// A CTA takes 4 columns: first A_kk^{-1} times theirs of A12, then A21 times
// that; a thread two rows of all four over a quarter of the depth (the quarters
// meet in shared memory).  Bound: the two 128 x 128 factors that every CTA
// reads from L2 (256 KB), 9.5 us in place of 34 between two inverses (packing
// 2.4, panel 19.4, tile 10-13 and their launches): one 3840 3.74 -> 2.97 ms.
constexpr int kNextCols = 4;
__global__ void __launch_bounds__(256) clu_next_diagonal_kernel(Planes W, int kk, const float2* __restrict__ inv,
                                                               int nblk) {
  __shared__ float4 rhs[kB][kNextCols];  // (re, re, im, im)
  __shared__ float2 part[4][2][kNextCols][kB / 2];
  const int b = blockIdx.y, tid = threadIdx.x, rp = tid & 63, quarter = tid >> 6;
  const int kn = kk + kB, c0 = kn + kNextCols * blockIdx.x;
  float* re = W.re + (size_t)b * W.stride;
  float* im = W.im + (size_t)b * W.stride;
  for (int idx = tid; idx < kB * kNextCols; idx += 256) {
    const int k = idx & (kB - 1), c = idx / kB;
    const size_t g = (size_t)(c0 + c) * W.ld + kk + k;
    const float x = re[g], y = im[g];
    rhs[k][c] = make_float4(x, x, y, y);
  }
  float2 ar[kNextCols], ai[kNextCols];
  auto clear = [&]() {
#pragma unroll
    for (int c = 0; c < kNextCols; ++c) ar[c] = ai[c] = make_float2(0.0f, 0.0f);
  };
  auto step = [&](int k, float2 xr, float2 xi) {
    const float2 ni = make_float2(-xi.x, -xi.y);
#pragma unroll
    for (int c = 0; c < kNextCols; ++c) {
      const float4 y = rhs[k][c];
      const float2 yr = make_float2(y.x, y.y), yi = make_float2(y.z, y.w);
      ar[c] = fma2(ni, yi, fma2(xr, yr, ar[c]));
      ai[c] = fma2(xi, yr, fma2(xr, yi, ai[c]));
    }
  };
  // the sum over the quarters: thread (rp, c) has the two rows of column c = quarter
  auto total = [&](float2& r, float2& i) {
#pragma unroll
    for (int c = 0; c < kNextCols; ++c) {
      part[quarter][0][c][rp] = ar[c];
      part[quarter][1][c][rp] = ai[c];
    }
    __syncthreads();
    r = i = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 u = part[q][0][quarter][rp], v = part[q][1][quarter][rp];
      r.x += u.x;
      r.y += u.y;
      i.x += v.x;
      i.y += v.y;
    }
  };
  __syncthreads();
  const int k0 = quarter * (kB / 4);
  clear();
  const float4* X = reinterpret_cast<const float4*>(inv + ((size_t)b * nblk + kk / kB) * kB * kB) + rp;
#pragma unroll 16
  for (int k = k0; k < k0 + kB / 4; ++k) {
    const float4 v = __ldcg(X + (size_t)k * (kB / 2));
    step(k, make_float2(v.x, v.z), make_float2(v.y, v.w));
  }
  float2 yr, yi;
  total(yr, yi);
  rhs[2 * rp][quarter] = make_float4(yr.x, yr.x, yi.x, yi.x);
  rhs[2 * rp + 1][quarter] = make_float4(yr.y, yr.y, yi.y, yi.y);
  __syncthreads();
  clear();
  const size_t a21 = (size_t)kk * W.ld + kn + 2 * rp;
#pragma unroll 16
  for (int k = k0; k < k0 + kB / 4; ++k)
    step(k, *reinterpret_cast<const float2*>(re + a21 + (size_t)k * W.ld),
         *reinterpret_cast<const float2*>(im + a21 + (size_t)k * W.ld));
  total(yr, yi);
  const size_t d = (size_t)(c0 + quarter) * W.ld + kn + 2 * rp;
  float2* dr = reinterpret_cast<float2*>(re + d);
  float2* di = reinterpret_cast<float2*>(im + d);
  const float2 oldr = *dr, oldi = *di;
  *dr = make_float2(oldr.x - yr.x, oldr.y - yr.y);
  *di = make_float2(oldi.x - yi.x, oldi.y - yi.y);
}

// 16-byte asynchronous global -> shared copy and its completion wait.
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))),
               "l"(gsrc)
               : "memory");
}

__device__ __forceinline__ int ld_acquire_i(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Persistent block substitution with the block LU factors.  Forward: y_i = b_i -
// sum_{j<i} L_ij y_j (unit block lower).  Backward: x_i = A_ii^{-1} y_i -
// sum_{j>i} U'_ij x_j with U'_ij = A_ii^{-1} U_ij stored in the factorisation, so
// each step of the dependency chain is one block product in both sweeps.
//
// A CTA owns 32 rows of a 128-row block, four CTAs per block.  What bounds the
// sweep is the chain of nblk steps, each the time from one block's publication
// to the next one's: a poll, the 128 x NC solution from L2, the product, the
// sum over the CTA's warps, the stores and the release.  With one CTA per
// block the product alone (128 x 128 x NC on one SM) was most of a step of
// 7 us with 4 right-hand sides and 23 with 16; a quarter of it on each of four SMs
// makes it 3.2 and 9.1 (forward and backward solve of one 3741: 0.43 -> 0.19 ms,
// of one 20493 with 16 right-hand sides 7.3 -> 2.9, of 15 x 6084 with 7 2.26 ->
// 1.42, half of the HBM rate).
//
// The rows' blocks stream through a ring of shared-memory slots, 64 columns
// (real and imaginary planes) each, copied two or three slots ahead of the products;
// only the right-hand sides of a dependency wait for its flag.  Warp w takes
// columns 8 w .. 8 w + 7 of a slot, a thread two rows and half of the columns of
// B; the partial sums stay in registers until the end (folded once per block, so
// that no float32 sum runs over more than 16 products before it is added to
// the rest), then the eight warps meet in shared memory.
// Solutions pass between CTAs as float32 in scratch (Yf: forward, Xb: backward,
// [matrix][row][NC]): half the bytes of complex128, and a CTA of a block may
// still read all of y_i while another already publishes x_i.  B gets the result
// of the backward sweep.  flags[b][i] counts the block's CTAs that have
// published (forward 1 .. 4, backward 5 .. 8), the ticket runs on as well: one
// memset per solve.
constexpr int kSubRows = 32, kSubs = kB / kSubRows;
constexpr int kSlotCols = 64;
constexpr int ring_slots(int nc) { return nc <= 8 ? 4 : 5; }  // the copies run this minus two slots ahead
constexpr int kSlotFloats = 2 * kSlotCols * kSubRows;  // [plane][column][row]

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

template <int NC, int CTAS>
__global__ void __launch_bounds__(256, CTAS)
    ctrsm_persistent_kernel(Planes W, int nblk, int batch, const float2* __restrict__ inv, double2* B, int64_t ldb,
                            int64_t strideB, int nrhs, int forward, float2* Yf, float2* Xb, int* flags, int* ticket,
                            int* err, const int* skip, long long spin_limit, int withheld, const int* mskip) {
  if (skip && *skip) return;  // refinement already converged
  constexpr int kC = NC / 2;  // columns of a thread
  constexpr int kSlots = ring_slots(NC), kAhead = kSlots - 2;
  extern __shared__ __align__(16) float fsmf[];
  float* ring = fsmf;
  float2* Y = reinterpret_cast<float2*>(ring + kSlots * kSlotFloats);  // Y[m * NC + c]
  __shared__ int s_t;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rp = lane & 15, ch = lane >> 4;  // rows 2 rp, 2 rp + 1; columns ch kC ..
  const int total = kSubs * nblk * batch;
  if (tid == 0) s_t = atomicAdd(ticket, 1);
  __syncthreads();
  const int t = s_t - (forward ? 0 : total);
  const int sub = t % kSubs, b = (t / kSubs) % batch, step = t / (kSubs * batch);
  if (mskip && mskip[b]) return;  // converged matrix: every CTA of it returns, no wait targets it
  const int i = forward ? step : (nblk - 1 - step);
  const int row0 = i * kB + sub * kSubRows;  // first row of this CTA
  const int ndep = forward ? i : (nblk - 1 - i);
  const int target = forward ? kSubs : 2 * kSubs;
  const float* Wre = W.re + (size_t)b * W.stride;
  const float* Wim = W.im + (size_t)b * W.stride;
  double2* Bb = B + (size_t)b * strideB;
  auto copy_solution = [&](const float2* src) {  // 128 x NC of another block into Y
    const float4* s4 = reinterpret_cast<const float4*>(src);
    float4* d4 = reinterpret_cast<float4*>(Y);
    float4 v[kB * NC / 512];
#pragma unroll
    for (int u = 0; u < kB * NC / 512; ++u) v[u] = __ldcg(s4 + tid + 256 * u);
#pragma unroll
    for (int u = 0; u < kB * NC / 512; ++u) d4[tid + 256 * u] = v[u];
  };
  // slot q: columns 64 (q % 2) .. of dependency q / 2
  const int nq = 2 * ndep;
  auto issue = [&](int q) {
    if (q < nq) {
      const int j = forward ? (q >> 1) : (nblk - 1 - (q >> 1));
      float* slot = ring + (q % kSlots) * kSlotFloats;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int idx = tid + 256 * u, col = idx >> 3, piece = idx & 7;
        const size_t g = (size_t)(row0 + piece * 4) + (size_t)(j * kB + (q & 1) * kSlotCols + col) * W.ld;
        cp_async16(slot + col * kSubRows + piece * 4, Wre + g);
        cp_async16(slot + kSlotCols * kSubRows + col * kSubRows + piece * 4, Wim + g);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int q = 0; q < kAhead; ++q) issue(q);
  // the outputs of this thread: idx = tid + 256 u, row idx / NC, column idx % NC
  constexpr int kOut = kSubRows * NC / 256;
  float2 own[kOut];
#pragma unroll
  for (int u = 0; u < kOut; ++u) {
    const int idx = tid + 256 * u, row = idx / NC, c = idx % NC;
    own[u] = make_float2(0.0f, 0.0f);
    if (forward && c < nrhs) {
      const double2 d = __ldcg(Bb + (size_t)(row0 + row) + (size_t)c * ldb);
      own[u] = make_float2((float)d.x, (float)d.y);
    }
  }
  float2 tot[2][kC], acc[2][kC], acci[2][kC];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int c = 0; c < kC; ++c) tot[h][c] = acc[h][c] = acci[h][c] = make_float2(0.0f, 0.0f);
  // acc += Re(A) y, acci += Im(A) y for one column of A; fold: tot += their complex product
  auto column = [&](float2 ar, float2 ai, const float2* y) {
    const float2 r0 = make_float2(ar.x, ar.x), r1 = make_float2(ar.y, ar.y);
    const float2 i0 = make_float2(ai.x, ai.x), i1 = make_float2(ai.y, ai.y);
    const float4* y4 = reinterpret_cast<const float4*>(y + ch * kC);
#pragma unroll
    for (int c2 = 0; c2 < kC / 2; ++c2) {
      const float4 v = y4[c2];
      const float2 v0 = make_float2(v.x, v.y), v1 = make_float2(v.z, v.w);
      acc[0][2 * c2] = fma2(r0, v0, acc[0][2 * c2]);
      acci[0][2 * c2] = fma2(i0, v0, acci[0][2 * c2]);
      acc[1][2 * c2] = fma2(r1, v0, acc[1][2 * c2]);
      acci[1][2 * c2] = fma2(i1, v0, acci[1][2 * c2]);
      acc[0][2 * c2 + 1] = fma2(r0, v1, acc[0][2 * c2 + 1]);
      acci[0][2 * c2 + 1] = fma2(i0, v1, acci[0][2 * c2 + 1]);
      acc[1][2 * c2 + 1] = fma2(r1, v1, acc[1][2 * c2 + 1]);
      acci[1][2 * c2 + 1] = fma2(i1, v1, acci[1][2 * c2 + 1]);
    }
  };
  auto fold = [&](float sign) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int c = 0; c < kC; ++c) {
        tot[h][c].x += sign * (acc[h][c].x - acci[h][c].y);
        tot[h][c].y += sign * (acc[h][c].y + acci[h][c].x);
        acc[h][c] = acci[h][c] = make_float2(0.0f, 0.0f);
      }
  };
  if (!forward) {
    // - A_ii^{-1} y_i, off the chain of dependencies: the inverse straight from
    // global memory, two rows of a column per thread
    copy_solution(Yf + ((size_t)b * nblk + i) * kB * NC);
    __syncthreads();
    const float2* Inv = inv + ((size_t)b * nblk + i) * kB * kB + sub * kSubRows + 2 * rp;
    float4 v[8];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
#pragma unroll
      for (int mm = 0; mm < 8; ++mm)
        v[mm] = __ldg(reinterpret_cast<const float4*>(Inv + (size_t)(16 * warp + 8 * half + mm) * kB));
#pragma unroll
      for (int mm = 0; mm < 8; ++mm)
        column(make_float2(v[mm].x, v[mm].z), make_float2(v[mm].y, v[mm].w), Y + (16 * warp + 8 * half + mm) * NC);
    }
    fold(-1.0f);
  }
#pragma unroll 1
  for (int q = 0; q < nq; ++q) {
    if ((q & 1) == 0) {
      const int j = forward ? (q >> 1) : (nblk - 1 - (q >> 1));
      if (tid == 0) {
        long long it = 0;
        while (ld_acquire_i(flags + (size_t)b * nblk + j) < target) {
          if (++it > spin_limit) {
            atomicExch(err, 1);
            break;
          }
          __nanosleep(20);
        }
      }
      __syncthreads();  // the dependency is there, and everyone is done with Y
      copy_solution((forward ? Yf : Xb) + ((size_t)b * nblk + j) * kB * NC);
    }
    // that slot was read two products ago: a barrier lies between
    issue(q + kAhead);
    cp_async_wait_group<kAhead>();  // this thread's copies of slot q have landed
    __syncthreads();                // everyone's, and Y
    const float* re = ring + (q % kSlots) * kSlotFloats + 8 * warp * kSubRows + 2 * rp;
    const float* im = re + kSlotCols * kSubRows;
    const float2* y = Y + ((q & 1) * kSlotCols + 8 * warp) * NC;
#pragma unroll 4
    for (int mm = 0; mm < 8; ++mm)
      column(*reinterpret_cast<const float2*>(re + mm * kSubRows), *reinterpret_cast<const float2*>(im + mm * kSubRows),
             y + mm * NC);
    if (q & 1) fold(1.0f);
  }
  cp_async_wait_group<0>();
  __syncthreads();
  // the warps' sums: red[warp][row][column] in the ring
  float2* red = reinterpret_cast<float2*>(ring);
  static_assert(8 * kSubRows * NC * sizeof(float2) <= kSlots * kSlotFloats * sizeof(float), "the sums fit the ring");
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int c = 0; c < kC; c += 2)
      *reinterpret_cast<float4*>(red + (warp * kSubRows + 2 * rp + h) * NC + ch * kC + c) =
          make_float4(tot[h][c].x, tot[h][c].y, tot[h][c + 1].x, tot[h][c + 1].y);
  __syncthreads();
  float2* dst = (forward ? Yf : Xb) + ((size_t)b * nblk + i) * kB * NC + sub * kSubRows * NC;
#pragma unroll
  for (int u = 0; u < kOut; ++u) {
    const int idx = tid + 256 * u;
    float2 v = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const float2 o = red[w * kSubRows * NC + idx];
      v.x += o.x;
      v.y += o.y;
    }
    own[u] = make_float2(own[u].x - v.x, own[u].y - v.y);
    dst[idx] = own[u];
  }
  __syncthreads();
  // withheld >= 0 only from the bounded-wait test entry point: that block row
  // never publishes, so the waits on it run out
  if (tid == 0 && i != withheld) {
    __threadfence();
    atomicAdd(flags + (size_t)b * nblk + i, 1);
  }
  if (!forward) {
#pragma unroll
    for (int u = 0; u < kOut; ++u) {
      const int idx = tid + 256 * u, row = idx / NC, c = idx % NC;
      if (c < nrhs) Bb[(size_t)(row0 + row) + (size_t)c * ldb] = make_double2((double)own[u].x, (double)own[u].y);
    }
  }
}

constexpr int trsm_smem_bytes(int nc) {
  return ring_slots(nc) * kSlotFloats * (int)sizeof(float) + kB * nc * (int)sizeof(float2);
}

// x += r (the correction solved in place in r), then r = b for the residual.
__global__ void ir_update_kernel(double2* __restrict__ X, double2* __restrict__ R, const double2* __restrict__ Bv,
                                 int n, int nrhs, int64_t ld, int64_t stride, const int* skip, const int* mskip) {
  if (skip && *skip) return;
  const int b = blockIdx.z, c = blockIdx.y;
  if (mskip && mskip[b]) return;  // this matrix has converged
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const size_t o = (size_t)b * stride + (size_t)c * ld + r;
    const double2 x = X[o], d = R[o];
    X[o] = make_double2(x.x + d.x, x.y + d.y);
    R[o] = Bv[o];
  }
}

// Squared norms of columns: out[(b*nrhs + c)] = sum |V(:, c)|^2 over n rows.
__global__ void colnorm2_kernel(const double2* __restrict__ V, int n, int64_t ld, int64_t stride,
                                double* __restrict__ out, const int* skip, const int* mskip) {
  if (skip && *skip) return;
  const int c = blockIdx.x, b = blockIdx.y, nrhs = gridDim.x;
  if (mskip && mskip[b]) return;
  const double2* v = V + (size_t)b * stride + (size_t)c * ld;
  double s = 0.0;
  for (int r = threadIdx.x; r < n; r += blockDim.x) s += v[r].x * v[r].x + v[r].y * v[r].y;
  __shared__ double red[256];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int off = blockDim.x / 2; off > 0; off >>= 1) {
    if ((int)threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[(size_t)b * nrhs + c] = red[0];
}

// Convergence test of one refinement iteration on the device: relative
// residual sqrt(|r_v|^2 / |b_v|^2) (absolute where b_v = 0) of every column,
// per matrix the worst of its nrhs columns: a matrix whose worst is <= tol is
// marked converged in mdone (the next iterations skip its work); *done when
// every matrix has converged (the iterations enqueued after return at once).
// state: [worst over all matrices, iterations].
__global__ void refine_check_kernel(const double* __restrict__ bn, const double* __restrict__ rn, int nrhs,
                                    int batch, double tol, int* done, double* state, int* mdone) {
  if (*done) return;
  __shared__ double red[32];
  __shared__ int all_done;
  if (threadIdx.x == 0) all_done = 1;
  __syncthreads();
  double worst = 0.0;
  for (int b = threadIdx.x; b < batch; b += blockDim.x) {
    double wb = 0.0;
    for (int c = 0; c < nrhs; ++c) {
      const int v = b * nrhs + c;
      wb = fmax(wb, bn[v] > 0.0 ? sqrt(rn[v] / bn[v]) : sqrt(rn[v]));
    }
    if (wb <= tol) mdone[b] = 1;
    else all_done = 0;  // benign race: every writer writes 0
    worst = fmax(worst, wb);
  }
  for (int off = 16; off > 0; off >>= 1) worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, off));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = worst;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) worst = fmax(worst, red[w]);
    state[0] = worst;
    state[1] += 1.0;
    if (all_done) *done = 1;
  }
}

int opt_in_mixed() {
  BEM_CUDA_CHECK(cudaFuncSetAttribute(clu_gj_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGjSmem));
  BEM_CUDA_CHECK(cudaFuncSetAttribute(ctrsm_persistent_kernel<8, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      trsm_smem_bytes(8)));
  BEM_CUDA_CHECK(cudaFuncSetAttribute(ctrsm_persistent_kernel<8, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      trsm_smem_bytes(8)));
  BEM_CUDA_CHECK(cudaFuncSetAttribute(ctrsm_persistent_kernel<16, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      trsm_smem_bytes(16)));
  return BEM_OK;
}
OncePerDevice g_mixed;
int configure_mixed() { return configure_device(g_mixed, opt_in_mixed); }

// Streaming multiprocessors of the current device (cached per device).
int sm_count(int* out) {
  static int counts[64] = {0};
  int dev = 0;
  BEM_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return set_error(BEM_ERR_UNSUPPORTED, "device index out of range");
  if (!counts[dev]) BEM_CUDA_CHECK(cudaDeviceGetAttribute(&counts[dev], cudaDevAttrMultiProcessorCount, dev));
  *out = counts[dev];
  return BEM_OK;
}

// Workspace layout, each part for the whole batch: planes 2 npad^2 floats per matrix,
// three A operands of npad x 2 kB floats, three B operands of 2 npad x kB floats,
// diagonal inverses nblk x kB x kB float2, the packed operands of the current block
// (see the members), then batch nblk + 2 + batch ints (flags, ticket, refinement).
struct MixedWork {
  float* W;
  float* Aop;
  float* Bop;
  float2* inv;
  float* binv;  // batch x 256 x kSplitB: packed A_kk^{-1} of the current block
  float* a3;    // batch x npad x kSplitK: split A21 of the current block
  float* ainv;  // 2 x batch x 128 x 256: A_kk^{-1} of the last two blocks as the A operand [Re | Im]
  int* flags;
};
MixedWork carve(void* work, int npad, int batch) {
  char* p = (char*)work;
  const int nblk = npad / kB;
  MixedWork w;
  w.W = (float*)p;
  p += (size_t)batch * 2 * npad * npad * sizeof(float);
  w.Aop = (float*)p;  // three buffers of batch x npad x 256
  p += kOpBuffers * (size_t)batch * npad * 2 * kB * sizeof(float);
  w.Bop = (float*)p;  // three buffers of batch x 2 npad x 128
  p += kOpBuffers * (size_t)batch * 2 * npad * kB * sizeof(float);
  w.inv = (float2*)p;
  p += (size_t)batch * nblk * kB * kB * sizeof(float2);
  w.binv = (float*)p;
  p += (size_t)batch * (2 * kB) * kSplitB * sizeof(float);
  w.a3 = (float*)p;
  p += (size_t)batch * npad * kSplitK * sizeof(float);
  w.ainv = (float*)p;
  p += 2 * (size_t)batch * kB * 2 * kB * sizeof(float);
  w.flags = (int*)p;
  return w;
}
Planes planes_of(const MixedWork& w, int npad) {
  return Planes{w.W, w.W + (size_t)npad * npad, npad, 2 * (int64_t)npad * npad};
}

// Streams and events of the lookahead in the block LU, one set per (device,
// caller stream): factorisations enqueued on different streams (concurrent
// requests of a server) overlap on the device without sharing a side stream.
// `chain` and `side` (highest priority) run the diagonal blocks (update,
// inverse) and the panels, `upper` (lowest priority) the block rows of U' that
// only the solves need.  The mutex is held while a factorisation is enqueued, so the events are never re-recorded by
// another caller in between.
struct Lookahead {
  std::mutex mu;
  cudaStream_t chain = nullptr;
  cudaStream_t side = nullptr;
  cudaStream_t upper = nullptr;
  cudaEvent_t inverse = nullptr;
  cudaEvent_t diag = nullptr;
  cudaEvent_t pre = nullptr;
  cudaEvent_t rows = nullptr;
  cudaEvent_t big = nullptr;
  cudaEvent_t strips = nullptr;
  cudaEvent_t colpack = nullptr;
  cudaEvent_t panel = nullptr;
  cudaEvent_t upper_done[2] = {nullptr, nullptr};
};
std::mutex g_lookahead_mu;
std::map<std::pair<int, cudaStream_t>, std::unique_ptr<Lookahead>> g_lookahead;
int lookahead_for(cudaStream_t caller, Lookahead** out) {
  int dev = 0;
  BEM_CUDA_CHECK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(g_lookahead_mu);
  std::unique_ptr<Lookahead>& la = g_lookahead[std::make_pair(dev, caller)];
  if (!la) {
    auto fresh = std::make_unique<Lookahead>();
    int least = 0, greatest = 0;
    BEM_CUDA_CHECK(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    BEM_CUDA_CHECK(cudaStreamCreateWithPriority(&fresh->chain, cudaStreamNonBlocking, greatest));
    BEM_CUDA_CHECK(cudaStreamCreateWithPriority(&fresh->side, cudaStreamNonBlocking, greatest));
    BEM_CUDA_CHECK(cudaStreamCreateWithPriority(&fresh->upper, cudaStreamNonBlocking, least));
    for (cudaEvent_t* e : {&fresh->inverse, &fresh->diag, &fresh->pre, &fresh->rows, &fresh->big, &fresh->strips,
                           &fresh->colpack, &fresh->panel, &fresh->upper_done[0], &fresh->upper_done[1]})
      BEM_CUDA_CHECK(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
    la = std::move(fresh);
  }
  *out = la.get();
  return BEM_OK;
}

}  // namespace
}  // namespace bem

using namespace bem;

extern "C" int64_t bem_clu_workspace_bytes(int npad, int batch) {
  if (npad <= 0 || npad % kB || batch <= 0) return -1;
  const int64_t nblk = npad / kB;
  return (int64_t)batch * 2 * npad * (int64_t)npad * 4 + kOpBuffers * (int64_t)batch * npad * 2 * kB * 4 +
         kOpBuffers * (int64_t)batch * 2 * npad * kB * 4 + (int64_t)batch * nblk * kB * kB * 8 +
         (int64_t)batch * (2 * kB) * kSplitB * 4 + (int64_t)batch * npad * kSplitK * 4 +
         2 * (int64_t)batch * kB * 2 * kB * 4 +
         ((int64_t)batch * nblk + 2 + batch) * 4 + 1024;
}

namespace bem {
namespace {
int clu_factor_impl(const void* K_dev, int64_t ldk, int64_t strideK, int n, int npad, int batch, const int* act,
                    int* piv_dev, int* info_dev, void* work_dev, int* err_dev, void* stream,
                    bool planes_ready = false);

// Identity on the padding of planes that already hold K (rows or columns n ..
// npad - 1), the counterpart of convert_pad_kernel when the assembly wrote
// the float32 planes itself.
// One warp per column (blockDim 32 x 8): columns below n only have their
// rows n .. npad - 1 written, the columns from n on all of theirs.
__global__ void pad_planes_kernel(int n, int npad, Planes W) {
  const int b = blockIdx.y, c = blockIdx.x * blockDim.y + threadIdx.y;
  if (c >= npad) return;
  for (int r = (c < n ? n : 0) + threadIdx.x; r < npad; r += blockDim.x)
    stp(W, b, r, c, make_float2(r == c ? 1.0f : 0.0f, 0.0f));
}
}  // namespace

int clu_planes(void* work_dev, int npad, float** re, int64_t* ld, int64_t* stride, int64_t* im) {
  if (!work_dev || npad <= 0 || npad % kB || (reinterpret_cast<uintptr_t>(work_dev) & 1023))
    return set_error(BEM_ERR_INVALID_ARGUMENT, "mixed LU workspace: npad a multiple of 128, 1024-byte alignment");
  // the planes come first in the workspace (carve)
  *re = reinterpret_cast<float*>(work_dev);
  *ld = npad;
  *stride = 2 * (int64_t)npad * npad;
  *im = (int64_t)npad * npad;
  return BEM_OK;
}
}  // namespace bem

extern "C" int bem_clu_factor_planes(int n, int npad, int batch, int* piv_dev, int* info_dev, void* work_dev,
                                     int* err_dev, void* stream) {
  return clu_factor_impl(nullptr, n, (int64_t)n * n, n, npad, batch, nullptr, piv_dev, info_dev, work_dev, err_dev,
                         stream, true);
}

extern "C" int bem_clu_factor(const void* K_dev, int64_t ldk, int64_t strideK, int n, int npad, int batch,
                              int* piv_dev, int* info_dev, void* work_dev, int* err_dev, void* stream) {
  return clu_factor_impl(K_dev, ldk, strideK, n, npad, batch, nullptr, piv_dev, info_dev, work_dev, err_dev, stream);
}

extern "C" int bem_clu_factor_grouped(const void* K_dev, int64_t ldk, int64_t strideK, int n, int npad, int batch,
                                      const int* active_host, int* piv_dev, int* info_dev, void* work_dev,
                                      int* err_dev, void* stream) {
  if (!active_host) return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_clu_factor_grouped: null active sizes");
  for (int b = 0; b < batch; ++b)
    if (active_host[b] <= 0 || active_host[b] % kB || active_host[b] > npad)
      return set_error(BEM_ERR_INVALID_ARGUMENT,
                       "bem_clu_factor_grouped: active sizes must be multiples of 128 in (0, npad]");
  return clu_factor_impl(K_dev, ldk, strideK, n, npad, batch, active_host, piv_dev, info_dev, work_dev, err_dev,
                         stream);
}

namespace bem {
namespace {
int clu_factor_impl(const void* K_dev, int64_t ldk, int64_t strideK, int n, int npad, int batch, const int* act,
                    int* piv_dev, int* info_dev, void* work_dev, int* err_dev, void* stream, bool planes_ready) {
  if ((!K_dev && !planes_ready) || !piv_dev || !info_dev || !work_dev || !err_dev || n <= 0 || npad < n ||
      npad % kB || batch <= 0 || ldk < n)
    return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_clu_factor: bad arguments (npad multiple of 128, >= n)");
  if (reinterpret_cast<uintptr_t>(work_dev) & 1023)
    return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_clu_factor: workspace must be 1024-byte aligned");
  int st = configure_mixed();
  if (st) return st;
  cudaStream_t s = (cudaStream_t)stream;
  MixedWork w = carve(work_dev, npad, batch);
  Planes W = planes_of(w, npad);
  const int nblk = npad / kB;
  int launches = 0;
  BEM_CUDA_CHECK(cudaMemsetAsync(info_dev, 0, sizeof(int) * batch, s));
  if (planes_ready) {  // K is in the planes already: the identity padding only
    if (npad > n)
      pad_planes_kernel<<<dim3(ceil_div(npad, 8), batch), dim3(32, 8), 0, s>>>(n, npad, W);
  } else {
    convert_pad_kernel<<<dim3(ceil_div(npad, 256), npad, batch), 256, 0, s>>>((const double2*)K_dev, ldk, strideK,
                                                                             n, npad, W);
  }
  ++launches;
  const size_t abuf = (size_t)batch * npad * 2 * kB, bbuf = (size_t)batch * 2 * npad * kB;
  // The updates and the panel product give each CTA an even share of up to
  // 32 tiles (the accumulator double buffer pays over a run; the runs end at
  // staggered times, so an SM frees up every few microseconds); U' (low
  // priority, off the chain) one tile per CTA, so that it never holds SMs
  // the chain needs for long.
  constexpr int kBigRun = 0, kSideRun = 1;
  float* Aop[kOpBuffers] = {w.Aop, w.Aop + abuf, w.Aop + 2 * abuf};
  float* Bop[kOpBuffers] = {w.Bop, w.Bop + bbuf, w.Bop + 2 * bbuf};
  const size_t ainv_buf = (size_t)batch * kB * 2 * kB;
  const int64_t a_stride = (int64_t)npad * 2 * kB;
  auto inverse = [&](int kk, cudaStream_t on) {
    TimedLaunch tl(kKCluGj, on);
    clu_gj_kernel<<<batch, 32 * kGjWarps, kGjSmem, on>>>(W, kk, info_dev, w.inv, nblk, err_dev);
    ++launches;
  };
  // its copies as the operands of the panel product and of U' (ainv buffer of
  // the block's parity)
  auto inverse_pack = [&](int kk, cudaStream_t on) {
    TimedLaunch tl(kKCluPanel, on);
    clu_inverse_pack_kernel<<<dim3(kB / 8, batch), 256, 0, on>>>(w.inv, nblk, kk, w.binv,
                                                                 w.ainv + ((kk / kB) & 1) * ainv_buf);
    ++launches;
  };
  // L21 = A21 A_kk^{-1} (split TF32: A_hi B_hi + A_lo B_hi + A_hi B_lo,
  // float32-level multipliers) into the working matrix and, packed, into the
  // A operand buffer of the block.
  auto panel = [&](int kk, int buf, cudaStream_t on) -> int {
    const int m = npad - kk - kB;
    if (m <= 0) return BEM_OK;
    TimedLaunch tl(kKCluPanel, on);
    return cgemm_tf32_update(w.a3, npad, kk + kB, w.binv, 2 * kB, 0, kSplitDepth, W.re, W.im, npad, W.stride, kk + kB,
                             kk, m, kB, batch, err_dev, on, 1, nullptr, nullptr, kBigRun, 0, act, Aop[buf],
                             kPackRows, a_stride);
  };
  // Block row of U scaled by the diagonal inverse, U' = A_kk^{-1} A12 (TF32),
  // for the backward substitution only (A12 itself is packed in Bop).
  auto upper = [&](int kk, int buf, cudaStream_t on) -> int {
    const int m = npad - kk - kB;
    if (m <= 0) return BEM_OK;
    TimedLaunch tl(kKCluPanel, on);
    return cgemm_tf32_update(w.ainv + ((kk / kB) & 1) * ainv_buf, kB, 0, Bop[buf], 2 * (int64_t)npad,
                             2 * (kk + kB), kUpdateDepth, W.re, W.im, npad, W.stride, kk, kk + kB, kB, m, batch, err_dev,
                             on, 1, nullptr, nullptr, kSideRun, 0, act);
  };
  // C rows r0.. (m), complex columns c0.. (nc) -= L21 U12 of the block step whose
  // packed operands are in buffer buf, and of a second step (buffer buf2 >= 0)
  // in the same pass over C (depth 256); optionally a packed copy of the result.
  auto update = [&](int buf, int r0, int c0, int m, int nc, int buf2, int run, cudaStream_t on,
                    TileRegion region = kTilesAll, int reserve = 0) -> int {
    if (m <= 0 || nc <= 0) return BEM_OK;
    return cgemm_tf32_update(Aop[buf], npad, r0, Bop[buf], 2 * (int64_t)npad, 2 * c0, kUpdateDepth, W.re, W.im, npad,
                             W.stride, r0, c0, m, nc, batch, err_dev, on, 0, buf2 >= 0 ? Aop[buf2] : nullptr,
                             buf2 >= 0 ? Bop[buf2] : nullptr, run, 0, act, nullptr, kPackNone, 0, region, reserve);
  };
  Lookahead* la = nullptr;
  if ((st = lookahead_for(s, &la))) return st;
  std::lock_guard<std::mutex> lock(la->mu);
  auto record = [](cudaEvent_t e, cudaStream_t on) -> int {
    BEM_CUDA_CHECK(cudaEventRecord(e, on));
    return BEM_OK;
  };
  auto wait = [](cudaStream_t on, cudaEvent_t e) -> int {
    BEM_CUDA_CHECK(cudaStreamWaitEvent(on, e, 0));
    return BEM_OK;
  };
#define BEM_TRY(call) \
  if ((st = (call))) return st
  // Right-looking block LU with a lookahead, the trailing updates of two
  // consecutive block steps applied in one pass over C (depth 256: the update
  // is bound by reading and writing C).  Step k, its inverse and operands
  // (A12 as the B operand, A21 split for the panel product) given:
  //   chain (highest priority): the diagonal block k+1 gets the update of step
  //     k and is inverted;
  //   side (highest priority): the panel product L21 (its epilogue packs the A
  //     operand), then the updates pending on the diagonal block k+2;
  //   upper (lowest priority): U', which only the solves need;
  //   the caller's stream: block row and block column k+1 get their updates
  //     (one L-shaped launch) and are packed as the operands of step k+1; at
  //     every second step the rest of the trailing matrix gets the updates of
  //     steps k-1 and k together.
  // direct: the diagonal block k+1 gets step k's update straight from A12, A21
  // and the inverse (clu_next_diagonal_kernel), what is pending on it having
  // been applied before; otherwise all of it as a tile behind the panel product.
  // Operands of steps k-1, k, k+1 live in three buffers; A_kk^{-1} for U' in
  // two.
  // direct while the chain is the bound: fewer than 200 blocks below block k+1
  // in all matrices together (8 x 3072: 4.13 -> 3.70 ms with 200, 3.88 with 100;
  // 15 x 6144 the same with 100, 200 and 400), and up to 24 matrices, whose
  // next blocks still fit the GPU at once (24 x 1024 1.18 -> 1.13 ms, but
  // 32 x 1536 2.41 -> 2.46, 60 x 1536 3.81 -> 3.95).  The two ways round
  // differently, so that the factors of a matrix follow its batch; one way for
  // every batch costs 29% without (3840: 2.96 -> 3.82 ms) or 20% with it (60 x 1536:
  // 3.82 -> 4.58 ms)
  auto direct = [&](int kk) {
    return batch <= 24 && (long long)batch * (npad - kk - 2 * kB) < 200ll * kB;
  };
  BEM_TRY(record(la->rows, s));
  BEM_TRY(wait(la->chain, la->rows));
  inverse(0, la->chain);
  BEM_TRY(record(la->inverse, la->chain));
  if (npad > kB) {  // the operands of block 0 come straight from the converted matrix
    const int m = npad - kB;
    TimedLaunch tl(kKCluPanel, s);
    clu_pack_kernel<<<dim3(m / kPT + m / 32, batch), 256, 0, s>>>(W, npad, 0, m / kPT, kB, 0, Bop[0], w.a3, 0);
    ++launches;
    BEM_TRY(record(la->colpack, s));
    BEM_TRY(record(la->strips, s));
  }
  for (int kk = 0, step = 0; kk + kB < npad; kk += kB, ++step) {
    const int cur = step % kOpBuffers, prev = (step + kOpBuffers - 1) % kOpBuffers;
    const int nxt = (step + 1) % kOpBuffers;
    const int kn = kk + kB, rest = npad - kn - kB;
    const int pend = (step & 1) ? prev : -1;  // step k-1 still pending beyond block k
    if (step >= 2) {
      // U' of block k-2 has read the A^{-1} copy that this block's overwrites
      // and the operand buffer that the strips below overwrite
      BEM_TRY(wait(la->side, la->upper_done[step & 1]));
      BEM_TRY(wait(s, la->upper_done[step & 1]));
    }
    BEM_TRY(wait(la->side, la->inverse));
    inverse_pack(kk, la->side);
    if (direct(kk)) {
      BEM_TRY(wait(la->chain, la->rows));
      if (step > 0) BEM_TRY(wait(la->chain, la->pre));
      {
        TimedLaunch tl(kKCluPanel, la->chain);
        clu_next_diagonal_kernel<<<dim3(kB / kNextCols, batch), 256, 0, la->chain>>>(W, kk, w.inv, nblk);
        ++launches;
      }
      BEM_TRY(record(la->diag, la->chain));
      inverse(kn, la->chain);
      BEM_TRY(record(la->inverse, la->chain));
      BEM_TRY(wait(la->side, la->diag));  // the panel product overwrites A21
    }
    BEM_TRY(wait(la->side, la->colpack));
    BEM_TRY(panel(kk, cur, la->side));
    BEM_TRY(record(la->panel, la->side));
    // U' reads the block row's B operand and the inverse, and overwrites A12
    BEM_TRY(wait(la->upper, la->strips));
    BEM_TRY(wait(la->upper, la->panel));
    BEM_TRY(upper(kk, cur, la->upper));
    BEM_TRY(record(la->upper_done[step & 1], la->upper));
    BEM_TRY(wait(s, la->panel));
    if (!direct(kk)) {
      BEM_TRY(update(cur, kn, kn, kB, kB, pend, kSideRun, s));
      BEM_TRY(record(la->diag, s));
      BEM_TRY(wait(la->chain, la->diag));
      inverse(kn, la->chain);
      BEM_TRY(record(la->inverse, la->chain));
    }
    if (rest == 0) break;
    const bool ahead = direct(kn);
    if (ahead) {  // what is pending on the next step's diagonal block
      BEM_TRY(wait(la->side, la->strips));
      if (step >= 2) BEM_TRY(wait(la->side, la->big));
      BEM_TRY(update(cur, kn + kB, kn + kB, kB, kB, pend, kSideRun, la->side));
      BEM_TRY(record(la->pre, la->side));
    }
    // block row kn and block column kn below the diagonal; the inverse of
    // block kn holds one SM per matrix meanwhile
    BEM_TRY(update(cur, kn, kn, rest + kB, rest + kB, pend, 0, s, kTilesL, batch));
    BEM_TRY(record(la->rows, s));
    // the block column's split copy first: the panel product starts on it
    // while the block row is packed as the next step's B operand.  (Strips and
    // packs on a stream of their own beside the big update: 15 x 6144 29.4 ->
    // 30.4 ms; they share its SMs and HBM.)
    {
      TimedLaunch tl(kKCluPanel, s);
      clu_pack_kernel<<<dim3(rest / 32, batch), 256, 0, s>>>(W, npad, kn, rest / kPT, kn + kB, kn, Bop[nxt], w.a3,
                                                            rest / kPT);
      BEM_TRY(record(la->colpack, s));
      clu_pack_kernel<<<dim3(rest / kPT, batch), 256, 0, s>>>(W, npad, kn, rest / kPT, kn + kB, kn, Bop[nxt], w.a3,
                                                             0);
      launches += 2;
    }
    BEM_TRY(record(la->strips, s));
    if (step & 1) {
      BEM_TRY(update(cur, kn + kB, kn + kB, rest, rest, prev, kBigRun, s, ahead ? kTilesNoCorner : kTilesAll));
      BEM_TRY(record(la->big, s));
    }
  }
  BEM_TRY(wait(s, la->inverse));
  if (npad > kB) {  // the last block rows of U' are part of the factors
    BEM_TRY(record(la->upper_done[0], la->upper));
    BEM_TRY(wait(s, la->upper_done[0]));
  }
#undef BEM_TRY
  count_launches(launches);
  BEM_CUDA_CHECK(cudaGetLastError());
  return BEM_OK;
}
}  // namespace
}  // namespace bem

namespace bem {
// Forward and backward block substitution with the float32 factors, in place on
// B (npad x nrhs complex128 per matrix); returns at once while *skip != 0.  Also
// the preconditioner of the GMRES solver.
int clu_solve_enqueue(void* work_dev, int npad, int batch, void* B_dev, int64_t ldb, int64_t strideB, int nrhs,
                      int* err_dev, cudaStream_t s, const int* skip, long long spin_limit, int withheld,
                      const int* mskip) {
  int st = configure_mixed();
  if (st) return st;
  MixedWork w = carve(work_dev, npad, batch);
  Planes W = planes_of(w, npad);
  const int nblk = npad / kB;
  int* ticket = w.flags + (size_t)batch * nblk;
  int launches = 0;
  int sms = 0;
  if ((st = sm_count(&sms))) return st;
  // more CTAs than two per SM hold: three per SM (85 registers, a few spilled)
  // stream the factors faster (15 x 6144: 1.42 ms a solve against 1.49; 60 x
  // 1536: 0.36 against 0.39), where all are resident the chain alone counts
  // (one 3741: 0.21 against 0.19)
  const bool crowded = (long long)kSubs * nblk * batch > 2 * sms;
  // scratch for the solutions passed between CTAs: the factorisation's packed
  // operands are free by now (2 x npad x 16 of their 3 x npad x 256 values)
  float2* Yf = reinterpret_cast<float2*>(w.Aop);
  float2* Xb = Yf + (size_t)batch * npad * kRhs;
  for (int c0 = 0; c0 < nrhs; c0 += kRhs) {
    const int nc = std::min(kRhs, nrhs - c0);
    double2* Bc = (double2*)B_dev + (size_t)c0 * ldb;
    BEM_CUDA_CHECK(cudaMemsetAsync(w.flags, 0, sizeof(int) * ((size_t)batch * nblk + 1), s));
    for (int forward = 1; forward >= 0; --forward) {
      TimedLaunch tl(kKCtrsm, s);
      auto* kernel = nc > 8   ? ctrsm_persistent_kernel<16, 2>
                     : crowded ? ctrsm_persistent_kernel<8, 3>
                               : ctrsm_persistent_kernel<8, 2>;
      kernel<<<kSubs * nblk * batch, 256, trsm_smem_bytes(nc <= 8 ? 8 : 16), s>>>(
          W, nblk, batch, w.inv, Bc, ldb, strideB, nc, forward, Yf, Xb, w.flags, ticket, err_dev, skip, spin_limit,
          withheld, mskip);
      ++launches;
    }
  }
  count_launches(launches);
  BEM_CUDA_CHECK(cudaGetLastError());
  return BEM_OK;
}
}  // namespace bem

extern "C" int bem_clu_solve(void* work_dev, int npad, int batch, const int* piv_dev, void* B_dev, int64_t ldb,
                             int64_t strideB, int nrhs, int* err_dev, void* stream) {
  if (!work_dev || !piv_dev || !B_dev || !err_dev || npad <= 0 || npad % kB || batch <= 0 || nrhs <= 0 ||
      ldb < npad)
    return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_clu_solve: bad arguments");
  return clu_solve_enqueue(work_dev, npad, batch, B_dev, ldb, strideB, nrhs, err_dev, (cudaStream_t)stream,
                           nullptr);
}

extern "C" int bem_clu_solve_bounded(void* work_dev, int npad, int batch, const int* piv_dev, void* B_dev,
                                     int64_t ldb, int64_t strideB, int nrhs, long long spin_limit, int withheld_block,
                                     int* err_dev, void* stream) {
  if (!work_dev || !piv_dev || !B_dev || !err_dev || npad <= 0 || npad % kB || batch <= 0 || nrhs <= 0 ||
      ldb < npad || spin_limit <= 0 || withheld_block < -1 || withheld_block >= npad / kB)
    return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_clu_solve_bounded: bad arguments");
  return clu_solve_enqueue(work_dev, npad, batch, B_dev, ldb, strideB, nrhs, err_dev, (cudaStream_t)stream,
                           nullptr, spin_limit, withheld_block);
}

extern "C" int bem_zgemm_ts(int M, int K, int nrhs, double alpha_re, double alpha_im, const void* A_dev, int64_t lda,
                            int64_t strideA, const void* X_dev, int64_t ldx, int64_t strideX, double beta_re,
                            double beta_im, void* Y_dev, int64_t ldy, int64_t strideY, int batch, void* work_dev,
                            void* stream);

namespace bem {
// Iterative refinement x += F^{-1} (b - K x) with the residual in float64
// against the float64 K, where F^{-1} is `solve_in_place` (the float32 block
// LU of the mixed engine, or the float64 block LU itself, whose pivoting stays
// inside the diagonal blocks: the residual test then checks, and the
// iteration repairs, what that pivoting loses).  x = 0, r = b to start; per
// iteration: r <- F^{-1} r, x += r, r = b - K x, worst relative residual per
// column, convergence flag on the device.  `done` is an int of the solver's
// workspace; norms_dev holds 2 batch nrhs + 2 doubles.
template <class Solve>
int refine_loop(Solve solve_in_place, int* done, int* mdone, const void* K_dev, int64_t ldk, int64_t strideK, int n,
                int npad,
                int batch, const void* B_dev, void* X_dev, void* R_dev, int64_t ldb, int64_t strideB, int nrhs,
                double tol, int max_iter, void* ts_work_dev, double* norms_dev, int* iters_out, double* resid_out,
                cudaStream_t s, int first_group = 4) {
  const int nvec = batch * nrhs;
  double* bn = norms_dev;
  double* rn = norms_dev + nvec;
  double* state = norms_dev + 2 * nvec;  // [worst, iterations]
  int launches = 1;
  // |b|^2 per column; x = 0, r = b, not converged
  colnorm2_kernel<<<dim3(nrhs, batch), 256, 0, s>>>((const double2*)B_dev, n, ldb, strideB, bn, nullptr,
                                                    nullptr);
  // Only the nrhs columns of each matrix: the caller may interleave other
  // columns (a wider right-hand-side block solved in chunks) between them.
  for (int b = 0; b < batch; ++b) {
    const size_t o = (size_t)b * strideB;
    BEM_CUDA_CHECK(cudaMemset2DAsync((double2*)X_dev + o, ldb * sizeof(double2), 0, npad * sizeof(double2), nrhs, s));
    BEM_CUDA_CHECK(cudaMemcpy2DAsync((double2*)R_dev + o, ldb * sizeof(double2), (const double2*)B_dev + o,
                                     ldb * sizeof(double2), npad * sizeof(double2), nrhs, cudaMemcpyDeviceToDevice,
                                     s));
  }
  BEM_CUDA_CHECK(cudaMemsetAsync(done, 0, sizeof(int), s));
  BEM_CUDA_CHECK(cudaMemsetAsync(mdone, 0, sizeof(int) * batch, s));
  BEM_CUDA_CHECK(cudaMemsetAsync(state, 0, 2 * sizeof(double), s));
  // Iterations are enqueued in groups without host synchronisation; once the
  // device-side test has converged the rest of the group returns at once.
  // first_group: the first group's size (float64 factors converge in one
  // iteration, and the kernels of three more cost 30 launches for nothing).
  constexpr int kGroup = 4;
  double host_state[2] = {0.0, 0.0};
  int enqueued = 0;
  while (enqueued < max_iter) {
    const int group = std::min(enqueued == 0 ? first_group : kGroup, max_iter - enqueued);
    for (int g = 0; g < group; ++g) {
      // r <- F^{-1} r in place (the padded rows of r stay zero)
      int st = solve_in_place(R_dev, (const int*)done, (const int*)mdone);
      if (st) return st;
      // x += r ; r = b ; r -= K x (float64); matrices already converged skip all of it
      ir_update_kernel<<<dim3(ceil_div(n, 256), nrhs, batch), 256, 0, s>>>(
          (double2*)X_dev, (double2*)R_dev, (const double2*)B_dev, n, nrhs, ldb, strideB, done, mdone);
      st = zgemm_ts_enqueue(n, n, nrhs, -1.0, 0.0, K_dev, ldk, strideK, X_dev, ldb, strideB, 1.0, 0.0, R_dev, ldb,
                            strideB, batch, ts_work_dev, s, done, mdone);
      if (st) return st;
      colnorm2_kernel<<<dim3(nrhs, batch), 256, 0, s>>>((const double2*)R_dev, n, ldb, strideB, rn, done, mdone);
      refine_check_kernel<<<1, 256, 0, s>>>(bn, rn, nrhs, batch, tol, done, state, mdone);
      launches += 3;
    }
    enqueued += group;
    const double before = host_state[0];
    BEM_CUDA_CHECK(cudaMemcpyAsync(host_state, state, sizeof(host_state), cudaMemcpyDeviceToHost, s));
    BEM_CUDA_CHECK(cudaStreamSynchronize(s));
    if (host_state[0] <= tol && host_state[1] > 0.0) break;
    // A contracting iteration gains far more than a factor 2 per group; one
    // that does not (the factors too far from K, e.g. near an irregular
    // frequency) stops here and reports non-convergence.
    if (enqueued > group && !(host_state[0] < 0.5 * before)) break;
  }
  count_launches(launches);
  *iters_out = (int)host_state[1];
  *resid_out = host_state[0];
  BEM_CUDA_CHECK(cudaGetLastError());
  if (!(host_state[0] <= tol)) {
    char msg[160];
    std::snprintf(msg, sizeof(msg), "iterative refinement stopped at relative residual %.3e after %d iterations",
                  host_state[0], (int)host_state[1]);
    return set_error(BEM_ERR_NOT_CONVERGED, msg);
  }
  return BEM_OK;
}
}  // namespace bem

extern "C" int bem_refine_solve(const void* K_dev, int64_t ldk, int64_t strideK, int n, int npad, int batch,
                                void* work_dev, const int* piv_dev, const void* B_dev, void* X_dev, void* R_dev,
                                int64_t ldb, int64_t strideB, int nrhs, double tol, int max_iter, void* ts_work_dev,
                                double* norms_dev, int* err_dev, int* iters_out, double* resid_out, void* stream) {
  if (!K_dev || !work_dev || !piv_dev || !B_dev || !X_dev || !R_dev || !ts_work_dev || !norms_dev || !err_dev ||
      !iters_out || !resid_out || nrhs <= 0 || nrhs > 16 || max_iter <= 0 || ldb < npad || npad % kB || n > npad ||
      batch <= 0)
    return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_refine_solve: bad arguments (nrhs <= 16)");
  cudaStream_t s = (cudaStream_t)stream;
  MixedWork w = carve(work_dev, npad, batch);
  int* done = w.flags + (size_t)batch * (npad / kB) + 1;
  int* mdone = done + 1;  // batch ints (bem_clu_workspace_bytes counts them)
  auto solve = [&](void* R, const int* skip, const int* mskip) {
    return clu_solve_enqueue(work_dev, npad, batch, R, ldb, strideB, nrhs, err_dev, s, skip, kDefaultSpinLimit, -1,
                             mskip);
  };
  return refine_loop(solve, done, mdone, K_dev, ldk, strideK, n, npad, batch, B_dev, X_dev, R_dev, ldb, strideB, nrhs, tol,
                     max_iter, ts_work_dev, norms_dev, iters_out, resid_out, s);
}

extern "C" int bem_zlu_refine_solve(const void* K_dev, int64_t ldk, int64_t strideK, int n, const void* LU_dev,
                                    int npad, int64_t ldlu, int64_t strideLU, int batch, const int* piv_dev,
                                    void* lu_work_dev, const void* B_dev, void* X_dev, void* R_dev, int64_t ldb,
                                    int64_t strideB, int nrhs, double tol, int max_iter, void* ts_work_dev,
                                    double* norms_dev, int* err_dev, int* iters_out, double* resid_out,
                                    void* stream) {
  if (!K_dev || !LU_dev || !lu_work_dev || !piv_dev || !B_dev || !X_dev || !R_dev || !ts_work_dev || !norms_dev ||
      !err_dev || !iters_out || !resid_out || nrhs <= 0 || nrhs > 16 || max_iter <= 0 || npad <= 0 || npad % 64 ||
      n > npad || n <= 0 || ldk < n || ldlu < npad || ldb < npad || batch <= 0)
    return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_zlu_refine_solve: bad arguments (nrhs <= 16, npad % 64 == 0)");
  cudaStream_t s = (cudaStream_t)stream;
  int* done = zlu_done_flag(lu_work_dev, npad, batch);
  int* mdone = done + 1;  // batch ints (bem_zlu_workspace_bytes counts them)
  auto solve = [&](void* R, const int* skip, const int* mskip) {
    return zlu_solve_enqueue(LU_dev, npad, ldlu, strideLU, batch, piv_dev, lu_work_dev, R, ldb, strideB, nrhs,
                             err_dev, s, skip, kDefaultSpinLimit, mskip);
  };
  return refine_loop(solve, done, mdone, K_dev, ldk, strideK, n, npad, batch, B_dev, X_dev, R_dev, ldb, strideB, nrhs, tol,
                     max_iter, ts_work_dev, norms_dev, iters_out, resid_out, s, 1);
}
