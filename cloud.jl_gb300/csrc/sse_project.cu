// sse_project.cu -- L2 projection of initial data onto the modal basis, FP64.
//
// project_function (src/Solvers/Solvers.jl:396-418): per element the mass
// matrix M = VDM' diag(W J) VDM is formed, factorised by Cholesky and solved
// against VDM' (W J u_q), all in one CTA: the weights, nodal data, mass
// matrix, factor and right-hand sides live in shared memory; VDM is read
// through L1/L2 by every CTA.
#include <cmath>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/sse_gb300.h"
#include "sse_kernels.cuh"
#include "sse_fixed_ops.cuh"

namespace sse {
namespace {

struct ProjArgs {
  int np, nq, nc;
  const double *V, *W, *J, *uq;
  Fx *Vf;  // V row i times 2^k_i times 2^-eV (at most 1/2), node-major; k_i <= 0
  int *k;  // about the square root of the node's weight
  int *eV;
  double *u0;
  int *flag;  // set when a mass matrix is not positive definite
};

// Vf, k and eV from V, by one block
__global__ void __launch_bounds__(256) fix_vandermonde_kernel(ProjArgs a) {
  __shared__ unsigned least, top;
  const int np = a.np, nq = a.nq;
  if (threadIdx.x == 0) {
    least = 0x7ff00000u;
    top = 0u;
  }
  __syncthreads();
  // node i: its largest entry, brought down to the smallest such
  auto largest = [&](int i) {
    unsigned m = 0u;
    for (int r = 0; r < np; ++r) m = max(m, (unsigned)__double2hiint(a.V[i + (size_t)nq * r]) & 0x7fffffffu);
    return m;
  };
  for (int i = threadIdx.x; i < nq; i += blockDim.x) atomicMin(&least, largest(i));
  __syncthreads();
  for (int i = threadIdx.x; i < nq; i += blockDim.x) {
    const unsigned m = largest(i);
    const int k = max(-200, fx_exponent(least) - fx_exponent(m));
    a.k[i] = k;
    atomicMax(&top, m + ((unsigned)k << 20));
  }
  __syncthreads();
  const int e = top >= 0x7ff00000u ? kFxBad : min(300, max(-300, fx_exponent(top) + 1));
  if (threadIdx.x == 0) *a.eV = e;
  for (int t = threadIdx.x; t < nq * np; t += blockDim.x) {
    const int i = t / np, r = t - i * np;
    a.Vf[t] = fo_from_double(a.V[i + (size_t)nq * r], e - a.k[i]);
  }
}

// 1/sqrt(x) for positive normal x: the hardware approximation (relative error
// about 2^-22) and one third-order step y <- y (1 + e/2 + 3 e^2/8), e = 1 - x y^2
__device__ __forceinline__ double rsqrt_step(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

constexpr int kTile = 3;  // rows and columns of M a thread forms

// Shared memory: WJ[nq], U[nc][nq], M[np][np] (lower triangle, overwritten by the
// Cholesky factor), Y[nc][np], the factor's inverse diagonal [np].
//
// M = VDM' diag(W J) VDM is most of the work (630 sums of 125 terms at p = 4,
// against 7 K FMAs of the factorisation).  In FP64 with an entry a thread it was
// bound by the FP64 pipe, and the factorisation by one lane's chains of FMAs.  M
// and the right-hand sides are formed in block fixed point (sse_fixed_ops.cuh)
// with the rows of VDM scaled by 2^k_i, M in 3 x 3 entries a thread, the cross
// products carried every four terms; the factorisation and the solves update
// all remaining entries after each column.  10,368 p = 4 tets, the whole call: 5.79 -> 2.51 ms.
__global__ void __launch_bounds__(128) project_function_kernel(ProjArgs a) {
  extern __shared__ double sm[];
  __shared__ unsigned key[2];
  __shared__ int bad;
  const int64_t k = blockIdx.x;
  const int np = a.np, nq = a.nq, nc = a.nc, eV = *a.eV;
  double *WJ = sm, *U = WJ + nq, *M = U + (size_t)nc * nq, *Y = M + (size_t)np * np, *inv = Y + (size_t)nc * np;
  Fx *wf = reinterpret_cast<Fx *>(WJ), *Uf = reinterpret_cast<Fx *>(U);
  if (threadIdx.x == 0) {
    bad = 0;
    key[0] = key[1] = 0u;
  }
  __syncthreads();
  // W J 2^-2k and W J u_q 2^-k, in units small enough for sums of nq terms
  unsigned m0 = 0u, m1 = 0u;
  for (int i = threadIdx.x; i < nq; i += blockDim.x) {
    const double w = a.W[i] * a.J[(size_t)nq * k + i], up = fx_pow2(-a.k[i]);
    WJ[i] = w * up * up;
    m0 = max(m0, (unsigned)__double2hiint(WJ[i]) & 0x7fffffffu);
    for (int e = 0; e < nc; ++e) {
      const double u = a.uq[((size_t)nc * k + e) * nq + i] * w * up;
      U[e * nq + i] = u;
      m1 = max(m1, (unsigned)__double2hiint(u) & 0x7fffffffu);
    }
  }
  fx_team_max(key, m0, threadIdx.x, blockDim.x);
  fx_team_max(key + 1, m1, threadIdx.x, blockDim.x);
  __syncthreads();
  const int spare = 32 - __clz(nq);
  auto unit_of = [&](unsigned m) { return m >= (1023u + 900u) << 20 ? kFxBad : max(-700, fx_exponent(m)) + spare; };
  const int uW = unit_of(key[0]), uU = unit_of(key[1]);
  for (int i = threadIdx.x; i < nq; i += blockDim.x) {
    wf[i] = fo_from_double(WJ[i], uW);
    for (int e = 0; e < nc; ++e) Uf[e * nq + i] = fo_from_double(U[e * nq + i], uU);
  }
  __syncthreads();
  // M[r][c] (r >= c) = sum_i (VDM[i, r] W J) VDM[i, c]
  const int nt = (np + kTile - 1) / kTile, ntri = nt * (nt + 1) / 2;
  for (int t = threadIdx.x; t < ntri; t += blockDim.x) {
    // t -> (tr, tc) with tc <= tr, rows in order
    int tr = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
    while (tr * (tr + 1) / 2 > t) --tr;
    while ((tr + 1) * (tr + 2) / 2 <= t) ++tr;
    const int r0 = tr * kTile, c0 = (t - tr * (tr + 1) / 2) * kTile;
    int rr[kTile], cc[kTile];
#pragma unroll
    for (int q = 0; q < kTile; ++q) {
      rr[q] = min(r0 + q, np - 1);
      cc[q] = min(c0 + q, np - 1);
    }
    FxSums<kTile> s[kTile];
#pragma unroll 2
    for (int i = 0; i < nq; ++i) {
      const Fx w = wf[i];
      Fx v[kTile];
#pragma unroll
      for (int q = 0; q < kTile; ++q) v[q] = a.Vf[i * np + cc[q]];
#pragma unroll
      for (int p = 0; p < kTile; ++p) {
        FxSums<1> wv;
        wv.add(a.Vf[i * np + rr[p]], &w, 0);
        s[p].add(fo_split(wv.template value<0>(0)), v, 1);
      }
      if ((i & 3) == 3)
#pragma unroll
        for (int p = 0; p < kTile; ++p) s[p].fold();
    }
#pragma unroll
    for (int p = 0; p < kTile; ++p)
#pragma unroll
      for (int q = 0; q < kTile; ++q)
        if (r0 + p < np && c0 + q <= r0 + p)
          M[(r0 + p) * np + c0 + q] = fx_value(s[p].template value<0>(q), max(uW, eV) == kFxBad ? kFxBad : uW + 2 * eV);
  }
  // right-hand sides Y[e][r] = sum_i VDM[i, r] (WJ u_q)[e][i]
  for (int t = threadIdx.x; t < nc * np; t += blockDim.x) {
    const int e = t / np, r = t - e * np;
    FxSums<1> s;
#pragma unroll 4
    for (int i = 0; i < nq; ++i) {
      s.add(a.Vf[i * np + r], Uf + e * nq + i, 0);
      if ((i & 3) == 3) s.fold();
    }
    Y[t] = fx_value(s.template value<0>(0), max(uU, eV) == kFxBad ? kFxBad : uU + eV);
  }
  __syncthreads();
  // Cholesky M = L L' by columns (L overwrites the lower triangle), and L z = y
  // along with it
  for (int j = 0; j < np; ++j) {
    if (threadIdx.x == 0) {
      double d = M[j * np + j];
      if (!(d > 0.0)) {
        bad = 1;
        d = 1.0;
      }
      inv[j] = rsqrt_step(d);
    }
    __syncthreads();
    const int below = np - 1 - j;
    const double f = inv[j];
    for (int t = threadIdx.x; t < below + nc; t += blockDim.x) {
      double *x = t < below ? M + (j + 1 + t) * np + j : Y + (t - below) * np + j;
      *x *= f;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < below * (below + nc); t += blockDim.x) {
      const int row = t / below, col = t - row * below + j + 1;
      if (row < nc) {
        Y[row * np + col] = fma(-M[col * np + j], Y[row * np + j], Y[row * np + col]);
      } else {
        const int r = row - nc + j + 1;
        if (col <= r) M[r * np + col] = fma(-M[r * np + j], M[col * np + j], M[r * np + col]);
      }
    }
    __syncthreads();
  }
  // L' x = z
  for (int r = np - 1; r >= 0; --r) {
    for (int e = threadIdx.x; e < nc; e += blockDim.x) Y[e * np + r] *= inv[r];
    __syncthreads();
    for (int t = threadIdx.x; t < nc * r; t += blockDim.x) {
      const int e = t / r, q = t - e * r;
      Y[e * np + q] = fma(-M[r * np + q], Y[e * np + r], Y[e * np + q]);
    }
    __syncthreads();
  }
  for (int t = threadIdx.x; t < nc * np; t += blockDim.x) a.u0[(size_t)nc * np * k + t] = Y[t];
  if (threadIdx.x == 0 && bad) atomicExch(a.flag, 1);
}

struct Buffers {
  std::vector<void *> ptrs;
  ~Buffers() {
    for (void *p : ptrs) cudaFree(p);
  }
  cudaError_t alloc(size_t bytes, void **out) {
    *out = nullptr;
    cudaError_t e = cudaMalloc(out, bytes > 0 ? bytes : 8);
    if (e == cudaSuccess) ptrs.push_back(*out);
    return e;
  }
};

}  // namespace

int project_function_run(int np, int nq, int nc, int64_t ne, const double *V, const double *W,
                         const double *J, const double *uq, double *u0, int memory, std::string *err) {
  auto bad = [&](const char *msg) {
    *err = msg;
    return (int)SSE_ERR_INVALID_ARGUMENT;
  };
  if (np <= 0 || nq <= 0 || nc <= 0 || nc > 8 || ne <= 0 || ne > 0x7fffffff) return bad("bad sizes");
  if (np > nq) return bad("n_p must not exceed n_q");
  if (!V || !W || !J || !uq || !u0) return bad("null array");
  if (memory != SSE_HOST && memory != SSE_DEVICE) return bad("memory must be SSE_HOST or SSE_DEVICE");
  const size_t smem = ((size_t)nq + (size_t)nc * nq + (size_t)np * np + (size_t)nc * np + np) * sizeof(double);
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (smem > (size_t)optin) {
    *err = "element too large for one CTA's shared memory";
    return SSE_ERR_UNSUPPORTED;
  }
  Buffers buf;
  auto cuda = [&](cudaError_t e, const char *where) {
    *err = std::string(where) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? (int)SSE_ERR_OUT_OF_MEMORY : (int)SSE_ERR_CUDA;
  };
  cudaError_t e;
  void *p;
  ProjArgs a{};
  a.np = np;
  a.nq = nq;
  a.nc = nc;
  if ((e = buf.alloc(((size_t)nq * np + nq) * sizeof(double), &p)) != cudaSuccess) return cuda(e, "allocate");
  a.V = (const double *)p;
  a.W = a.V + (size_t)nq * np;
  if ((e = cudaMemcpy(p, V, (size_t)nq * np * sizeof(double), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy((double *)p + (size_t)nq * np, W, nq * sizeof(double), cudaMemcpyHostToDevice)) != cudaSuccess)
    return cuda(e, "upload VDM, W");
  if ((e = buf.alloc((size_t)nq * np * sizeof(Fx) + (nq + 2) * sizeof(int), &p)) != cudaSuccess)
    return cuda(e, "allocate");
  a.Vf = (Fx *)p;
  a.k = (int *)(a.Vf + (size_t)nq * np);
  a.eV = a.k + nq;
  a.flag = a.eV + 1;
  if ((e = cudaMemset(a.flag, 0, sizeof(int))) != cudaSuccess) return cuda(e, "memset");
  const size_t n_j = (size_t)nq * ne, n_u = (size_t)nq * nc * ne, n_o = (size_t)np * nc * ne;
  if (memory == SSE_DEVICE) {
    a.J = J;
    a.uq = uq;
    a.u0 = u0;
  } else {
    if ((e = buf.alloc((n_j + n_u + n_o) * sizeof(double), &p)) != cudaSuccess) return cuda(e, "allocate");
    double *d = (double *)p;
    if ((e = cudaMemcpy(d, J, n_j * sizeof(double), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(d + n_j, uq, n_u * sizeof(double), cudaMemcpyHostToDevice)) != cudaSuccess)
      return cuda(e, "upload J_q, u_q");
    a.J = d;
    a.uq = d + n_j;
    a.u0 = d + n_j + n_u;
  }
  cudaFuncSetAttribute(project_function_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  fix_vandermonde_kernel<<<1, 256>>>(a);
  project_function_kernel<<<(unsigned)ne, 128, smem>>>(a);
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda(e, "projection kernel launch");
  if ((e = cudaDeviceSynchronize()) != cudaSuccess) return cuda(e, "projection kernel");
  int flag = 0;
  if ((e = cudaMemcpy(&flag, a.flag, sizeof(int), cudaMemcpyDeviceToHost)) != cudaSuccess) return cuda(e, "flag");
  if (memory == SSE_HOST &&
      (e = cudaMemcpy(u0, a.u0, n_o * sizeof(double), cudaMemcpyDeviceToHost)) != cudaSuccess)
    return cuda(e, "copy u0 to the host");
  if (flag) {
    *err = "a mass matrix is not positive definite";
    return SSE_ERR_NONPHYSICAL;
  }
  return SSE_OK;
}

}  // namespace sse
