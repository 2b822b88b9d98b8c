// Right-hand sides, potentials and forces of the indirect BEM solve.
//
// * bem_build_rhs: radiation boundary conditions -i*omega*(dof . n) and
//   diffraction boundary conditions -(u_Airy . n) on the hull, zero on lid
//   panels (capytaine bem/problems_and_results.py:373-381, 440-449;
//   bem/airy_waves.py:56-95, infinite or finite depth).
// * bem_zgemm_ts: Y = alpha A X + beta Y for a tall matrix A (n x K, complex128,
//   column-major) and a few columns X (K x nrhs): the potential S @ sigma
//   (bem/solver.py:197-198) and the residuals b - K x.  Memory-bound on A: split
//   over K into partial sums reduced in a fixed order (deterministic).
// * bem_integrate_pressure / bem_froude_krylov: force integrals
//   F_d = sum_i p_i (-dof_d . n_i) area_i (bodies/bodies.py:238-250) of the
//   radiated/diffracted pressure i*omega*rho*phi and of the incident-wave
//   pressure (airy_waves.py:19-53, 98-102).
#include <algorithm>
#include <cmath>

#include "dmma.cuh"

namespace bem {
namespace {


// Depth profiles of the Airy wave at height z (airy_waves.py:41-47, 80-85):
// cosh(k (z + h)) / cosh(k h) and sinh(k (z + h)) / cosh(k h) when 0 <= k h < 20,
// else both e^{k z} (the infinite-depth profile).
template <bool FINITE_DEPTH>
__device__ __forceinline__ void airy_profiles(double k, double z, double depth, double& cih, double& sih) {
  if constexpr (FINITE_DEPTH) {
    const double kh = k * depth;
    if (kh >= 0.0 && kh < 20.0) {
      const double ch = cosh(kh);
      cih = cosh(k * (z + depth)) / ch;
      sih = sinh(k * (z + depth)) / ch;
      return;
    }
  }
  cih = exp(k * z);
  sih = cih;
}

template <bool FINITE_DEPTH>
__global__ void build_rhs_kernel(int n, int64_t ldb, int64_t strideB, int batch, const double* __restrict__ omega,
                                 const double* __restrict__ wavenumber, double g, double depth, int ndof,
                                 const double* __restrict__ dofn, int nhead, const double* __restrict__ headings,
                                 const double* __restrict__ centers, const double* __restrict__ normals,
                                 const int* __restrict__ hull, double2* __restrict__ B) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (i >= n) return;
  double2* Bb = B + (size_t)b * strideB;
  const double w = omega[b], k = wavenumber[b];
  const bool on_hull = hull == nullptr || hull[i] != 0;
  for (int d = 0; d < ndof; ++d) {
    const double v = on_hull ? dofn[(size_t)d * n + i] : 0.0;
    Bb[(size_t)i + (size_t)d * ldb] = make_double2(0.0, -w * v);  // -1j * omega * (dof . n)
  }
  const double x = centers[3 * i], y = centers[3 * i + 1], z = centers[3 * i + 2];
  const double nx = normals[3 * i], ny = normals[3 * i + 1], nz = normals[3 * i + 2];
  for (int h = 0; h < nhead; ++h) {
    double2 bc = make_double2(0.0, 0.0);
    if (on_hull) {
      const double beta = headings[h];
      double sb, cb;
      sincos(beta, &sb, &cb);
      const double wbar = x * cb + y * sb;
      double s, c;
      sincos(k * wbar, &s, &c);
      double cih, sih;
      airy_profiles<FINITE_DEPTH>(k, z, depth, cih, sih);
      const double amp_c = g * k / w * cih, amp_s = g * k / w * sih;
      // v = (g k / w) e^{i k wbar} (cos b cih, sin b cih, -i sih); v . n
      const double2 ec = make_double2(amp_c * c, amp_c * s);
      const double2 es = make_double2(amp_s * c, amp_s * s);
      const double horiz = cb * nx + sb * ny;
      // ec * horiz + es * (-i) * nz
      const double2 vn = make_double2(ec.x * horiz + es.y * nz, ec.y * horiz - es.x * nz);
      bc = make_double2(-vn.x, -vn.y);
    }
    Bb[(size_t)i + (size_t)(ndof + h) * ldb] = bc;
  }
}

constexpr int kTsMaxRhs = 16;

// Partial products of the split-K tall GEMM on the double-precision tensor cores,
// 8 or 16 columns of X.  The reads of A are the bound (16 bytes per entry); with
// plain multiply-adds (27 TF/s, one row per thread, X from shared memory) 8
// columns already cost as much as the reads and 16 twice as much.  A CTA owns 128
// rows, 16 per warp; A and X stream through a five-stage cp.async ring of depth 8.
// 15 x 6084^2, 7 columns: 1.91 -> 1.31 ms (6.8 TB/s, a little above the measured copy
// rate: reads only); 20493^2, 16 columns: 3.31 -> 1.83 ms (1.5 of MMAs).
constexpr int kTsRows = 128, kTsDepth = 8, kTsStages = 5;
constexpr int kTsLdA = kTsRows + 2, kTsLdX = kTsDepth + 4;
constexpr int kTsStage = kTsDepth * kTsLdA + kTsMaxRhs * kTsLdX;
constexpr int kTsSmem = kTsStages * kTsStage * (int)sizeof(double2);

template <int NT>
__global__ void __launch_bounds__(256, 2) zgemm_ts_partial_kernel(int M, int K, int nrhs, int kchunk,
                                                             const double2* __restrict__ A, int64_t lda,
                                                             int64_t strideA, const double2* __restrict__ X,
                                                             int64_t ldx, int64_t strideX,
                                                             double2* __restrict__ part, const int* skip,
                                                             const int* mskip) {
  if (skip && *skip) return;
  extern __shared__ double2 ring[];
  const int b = blockIdx.z;
  if (mskip && mskip[b]) return;  // matrix b is not needed (converged)
  const int split = blockIdx.y;
  const int k0 = split * kchunk, kc = min(K, k0 + kchunk) - k0;
  const int m0 = blockIdx.x * kTsRows;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  A += (size_t)b * strideA + (size_t)k0 * lda;
  X += (size_t)b * strideX + k0;
  const int nk = (kc + kTsDepth - 1) / kTsDepth;
  auto issue = [&](int q) {
    if (q < nk) {
      double2* As = ring + (q % kTsStages) * kTsStage;
      double2* Xs = As + kTsDepth * kTsLdA;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int idx = tid + 256 * i, m = idx & (kTsRows - 1), k = idx >> 7, kq = q * kTsDepth + k;
        const bool ok = m0 + m < M && kq < kc;
        cp_async16(As + k * kTsLdA + m, ok ? A + (size_t)(m0 + m) + (size_t)kq * lda : A, ok);
      }
      if (tid < 8 * NT * kTsDepth) {
        const int k = tid & (kTsDepth - 1), c = tid / kTsDepth, kq = q * kTsDepth + k;
        const bool ok = c < nrhs && kq < kc;
        cp_async16(Xs + c * kTsLdX + k, ok ? X + (size_t)kq + (size_t)c * ldx : X, ok);
      }
    }
    cp_async_commit();
  };
  double re[NT][4] = {}, im[NT][4] = {};
#pragma unroll
  for (int q = 0; q < kTsStages - 1; ++q) issue(q);
#pragma unroll 1
  for (int q = 0; q < nk; ++q) {
    cp_async_wait<kTsStages - 2>();  // stage q has landed (this thread's part)
    __syncthreads();                 // everybody's; and everybody is done with stage q - 1
    issue(q + kTsStages - 1);
    const double2* As = ring + (q % kTsStages) * kTsStage;
    warp_zmma<NT>(As + 16 * warp, kTsLdA, As + kTsDepth * kTsLdA, kTsLdX, kTsDepth, re, im, lane);
  }
  const int g = lane >> 2, t = lane & 3;
  double2* p = part + ((size_t)b * gridDim.y + split) * (size_t)M * nrhs;
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = m0 + 16 * warp + g + 8 * (e >> 1), c = 8 * j + 2 * t + (e & 1);
      if (row < M && c < nrhs) p[(size_t)c * M + row] = make_double2(re[j][e], im[j][e]);
    }
}

__global__ void zgemm_ts_reduce_kernel(int M, int nrhs, int nsplit, double2 alpha, double2 beta,
                                       const double2* __restrict__ part, double2* __restrict__ Y, int64_t ldy,
                                       int64_t strideY, const int* skip, const int* mskip) {
  if (skip && *skip) return;
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.y, b = blockIdx.z;
  if (mskip && mskip[b]) return;
  if (row >= M) return;
  double2 s = make_double2(0.0, 0.0);
  for (int sp = 0; sp < nsplit; ++sp) {
    const double2 v = part[(((size_t)b * nsplit + sp) * nrhs + c) * (size_t)M + row];
    s.x += v.x;
    s.y += v.y;
  }
  double2* y = Y + (size_t)b * strideY + (size_t)c * ldy + row;
  double2 out = make_double2(alpha.x * s.x - alpha.y * s.y, alpha.x * s.y + alpha.y * s.x);
  if (beta.x != 0.0 || beta.y != 0.0) {
    const double2 o = *y;
    out.x += beta.x * o.x - beta.y * o.y;
    out.y += beta.x * o.y + beta.y * o.x;
  }
  *y = out;
}

// F[b][c][d] = coef_b * sum_i phi[b][i][c] * w[d][i], coef_b = i omega_b rho
__global__ void integrate_pressure_kernel(int n, int nrhs, int ndof, const double2* __restrict__ phi, int64_t ldp,
                                          int64_t strideP, const double* __restrict__ omega, double rho,
                                          const double* __restrict__ wdof, double2* __restrict__ F) {
  const int d = blockIdx.x, c = blockIdx.y, b = blockIdx.z;
  const double2* p = phi + (size_t)b * strideP + (size_t)c * ldp;
  const double* w = wdof + (size_t)d * n;
  double sx = 0.0, sy = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double2 v = p[i];
    sx += v.x * w[i];
    sy += v.y * w[i];
  }
  __shared__ double rx[256], ry[256];
  rx[threadIdx.x] = sx;
  ry[threadIdx.x] = sy;
  __syncthreads();
  for (int off = blockDim.x / 2; off > 0; off >>= 1) {
    if ((int)threadIdx.x < off) {
      rx[threadIdx.x] += rx[threadIdx.x + off];
      ry[threadIdx.x] += ry[threadIdx.x + off];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double cw = omega[b] * rho;  // coef = (0, cw)
    F[((size_t)b * nrhs + c) * ndof + d] = make_double2(-cw * ry[0], cw * rx[0]);
  }
}

// Froude-Krylov: p0 = rho g cih(z) e^{i k (x cos b + y sin b)}, F[b][h][d] = sum_i p0_i w[d][i]
template <bool FINITE_DEPTH>
__global__ void froude_krylov_kernel(int n, int ndof, int nhead, const double* __restrict__ wavenumber, double rho,
                                     double g, double depth, const double* __restrict__ headings,
                                     const double* __restrict__ centers, const double* __restrict__ wdof,
                                     double2* __restrict__ F) {
  const int d = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const double k = wavenumber[b];
  double sb, cb;
  sincos(headings[h], &sb, &cb);
  const double* w = wdof + (size_t)d * n;
  double sx = 0.0, sy = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double x = centers[3 * i], y = centers[3 * i + 1], z = centers[3 * i + 2];
    double s, c;
    sincos(k * (x * cb + y * sb), &s, &c);
    double cih, sih;
    airy_profiles<FINITE_DEPTH>(k, z, depth, cih, sih);
    const double amp = rho * g * cih * w[i];
    sx += amp * c;
    sy += amp * s;
  }
  __shared__ double rx[256], ry[256];
  rx[threadIdx.x] = sx;
  ry[threadIdx.x] = sy;
  __syncthreads();
  for (int off = blockDim.x / 2; off > 0; off >>= 1) {
    if ((int)threadIdx.x < off) {
      rx[threadIdx.x] += rx[threadIdx.x + off];
      ry[threadIdx.x] += ry[threadIdx.x + off];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) F[((size_t)b * nhead + h) * ndof + d] = make_double2(rx[0], ry[0]);
}

}  // namespace
}  // namespace bem

using namespace bem;

extern "C" int bem_build_rhs(int n, int batch, const double* omega_dev, const double* wavenumber_dev, double g,
                             double water_depth, int ndof, const double* dofn_dev, int nhead,
                             const double* headings_dev, const double* centers_dev, const double* normals_dev,
                             const int32_t* hull_dev, void* B_dev, int64_t ldb, int64_t strideB, void* stream) {
  if (n <= 0 || batch <= 0 || ndof < 0 || nhead < 0 || ldb < n || !B_dev || !omega_dev || !wavenumber_dev ||
      (ndof > 0 && !dofn_dev) || (nhead > 0 && (!headings_dev || !centers_dev || !normals_dev)) ||
      !(water_depth > 0.0))
    return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_build_rhs: bad arguments");
  dim3 grid(ceil_div(n, 128), batch);
  if (std::isinf(water_depth))
    build_rhs_kernel<false><<<grid, 128, 0, (cudaStream_t)stream>>>(n, ldb, strideB, batch, omega_dev, wavenumber_dev,
                                                                    g, water_depth, ndof, dofn_dev, nhead,
                                                                    headings_dev, centers_dev, normals_dev, hull_dev,
                                                                    (double2*)B_dev);
  else
    build_rhs_kernel<true><<<grid, 128, 0, (cudaStream_t)stream>>>(n, ldb, strideB, batch, omega_dev, wavenumber_dev,
                                                                   g, water_depth, ndof, dofn_dev, nhead,
                                                                   headings_dev, centers_dev, normals_dev, hull_dev,
                                                                   (double2*)B_dev);
  count_launches(1);
  BEM_CUDA_CHECK(cudaGetLastError());
  return BEM_OK;
}

// Splits of the K dimension: two waves of the two CTAs that an SM holds, in shares
// of at least 32 columns (a 735 x 735 product in 9 CTAs took 58 us, in 132 it
// takes 15), and up to 32 CTAs per SM (an even last wave) while the shares keep
// 256 columns: shorter ones spend their time filling the ring (3741 in shares of
// 47 columns 66 us, of 187 58 us), and every split writes and reads M x nrhs
// partial sums.  The splits, and with them the rounding of the sums, follow the
// batch: splits from M and K alone would be 13 in place of 6 for 15 x 6084^2 (7
// columns 1.31 -> 1.54 ms) and 12 for 60 x 1521^2 in place of 5 (0.38 -> 0.45).
constexpr int kTsFill = 4 * 148, kTsFillCols = 32;
constexpr int kTsEven = 32 * 148, kTsEvenCols = 256;
static int ts_nsplit(int M, int K, int batch) {
  const long long rows = (long long)ceil_div(M, kTsRows) * batch;
  return std::max(1, std::max(std::min(ceil_div(kTsFill, rows), K / kTsFillCols),
                              std::min(ceil_div(kTsEven, rows), K / kTsEvenCols)));
}

// For these sizes and all smaller ones (which may take more splits): rows blocks
// of 128 rows have at most `kTsFill / rows + 1` splits by the first rule,
// `kTsEven / rows + 1` by the second.
extern "C" int64_t bem_zgemm_ts_workspace_bytes(int M, int K, int nrhs, int batch) {
  const int64_t rows = (int64_t)ceil_div(std::max(M, 1), kTsRows) * std::max(batch, 1);
  const int64_t blocks = std::max({rows, std::min(rows + kTsFill, rows * (K / kTsFillCols)),
                                   std::min(rows + kTsEven, rows * (K / kTsEvenCols))});
  return blocks * kTsRows * nrhs * (int64_t)sizeof(double2);
}

namespace bem {
int zgemm_ts_enqueue(int M, int K, int nrhs, double alpha_re, double alpha_im, const void* A_dev, int64_t lda,
                     int64_t strideA, const void* X_dev, int64_t ldx, int64_t strideX, double beta_re,
                     double beta_im, void* Y_dev, int64_t ldy, int64_t strideY, int batch, void* work_dev,
                     void* stream, const int* skip, const int* mskip) {
  if (M <= 0 || K <= 0 || nrhs <= 0 || nrhs > kTsMaxRhs || batch <= 0 || !A_dev || !X_dev || !Y_dev || !work_dev ||
      lda < M || ldx < K || ldy < M)
    return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_zgemm_ts: bad arguments (nrhs must be <= 16)");
  const int nsplit = ts_nsplit(M, K, batch), kchunk = ceil_div(K, nsplit);
  cudaStream_t s = (cudaStream_t)stream;
  static OncePerDevice once;
  const int st = configure_device(once, [] {
    BEM_CUDA_CHECK(
        cudaFuncSetAttribute(zgemm_ts_partial_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTsSmem));
    BEM_CUDA_CHECK(
        cudaFuncSetAttribute(zgemm_ts_partial_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTsSmem));
    return BEM_OK;
  });
  if (st) return st;
  TimedLaunch tl(kKZgemmTs, s);
  auto* kernel = nrhs <= 8 ? zgemm_ts_partial_kernel<1> : zgemm_ts_partial_kernel<2>;
  kernel<<<dim3(ceil_div(M, kTsRows), nsplit, batch), 256, kTsSmem, s>>>(
      M, K, nrhs, kchunk, (const double2*)A_dev, lda, strideA, (const double2*)X_dev, ldx, strideX,
      (double2*)work_dev, skip, mskip);
  zgemm_ts_reduce_kernel<<<dim3(ceil_div(M, 256), nrhs, batch), 256, 0, s>>>(
      M, nrhs, nsplit, make_double2(alpha_re, alpha_im), make_double2(beta_re, beta_im), (const double2*)work_dev,
      (double2*)Y_dev, ldy, strideY, skip, mskip);
  count_launches(2);
  BEM_CUDA_CHECK(cudaGetLastError());
  return BEM_OK;
}
}  // namespace bem

extern "C" int bem_zgemm_ts(int M, int K, int nrhs, double alpha_re, double alpha_im, const void* A_dev, int64_t lda,
                            int64_t strideA, const void* X_dev, int64_t ldx, int64_t strideX, double beta_re,
                            double beta_im, void* Y_dev, int64_t ldy, int64_t strideY, int batch, void* work_dev,
                            void* stream) {
  return bem::zgemm_ts_enqueue(M, K, nrhs, alpha_re, alpha_im, A_dev, lda, strideA, X_dev, ldx, strideX, beta_re,
                               beta_im, Y_dev, ldy, strideY, batch, work_dev, stream, nullptr, nullptr);
}

extern "C" int bem_integrate_pressure(int n, int batch, int nrhs, int ndof, const void* phi_dev, int64_t ldp,
                                      int64_t strideP, const double* omega_dev, double rho, const double* wdof_dev,
                                      void* F_dev, void* stream) {
  if (n <= 0 || batch <= 0 || nrhs <= 0 || ndof <= 0 || !phi_dev || !omega_dev || !wdof_dev || !F_dev || ldp < n)
    return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_integrate_pressure: bad arguments");
  integrate_pressure_kernel<<<dim3(ndof, nrhs, batch), 256, 0, (cudaStream_t)stream>>>(
      n, nrhs, ndof, (const double2*)phi_dev, ldp, strideP, omega_dev, rho, wdof_dev, (double2*)F_dev);
  count_launches(1);
  BEM_CUDA_CHECK(cudaGetLastError());
  return BEM_OK;
}

extern "C" int bem_froude_krylov(int n, int batch, int ndof, int nhead, const double* wavenumber_dev, double rho,
                                 double g, double water_depth, const double* headings_dev, const double* centers_dev,
                                 const double* wdof_dev, void* F_dev, void* stream) {
  if (n <= 0 || batch <= 0 || ndof <= 0 || nhead <= 0 || !wavenumber_dev || !headings_dev || !centers_dev ||
      !wdof_dev || !F_dev || !(water_depth > 0.0))
    return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_froude_krylov: bad arguments");
  const dim3 grid(ndof, nhead, batch);
  if (std::isinf(water_depth))
    froude_krylov_kernel<false><<<grid, 256, 0, (cudaStream_t)stream>>>(
        n, ndof, nhead, wavenumber_dev, rho, g, water_depth, headings_dev, centers_dev, wdof_dev, (double2*)F_dev);
  else
    froude_krylov_kernel<true><<<grid, 256, 0, (cudaStream_t)stream>>>(
        n, ndof, nhead, wavenumber_dev, rho, g, water_depth, headings_dev, centers_dev, wdof_dev, (double2*)F_dev);
  count_launches(1);
  BEM_CUDA_CHECK(cudaGetLastError());
  return BEM_OK;
}
