// sse_project.cu -- L2 projection of initial data onto the modal basis, FP64.
//
// project_function (src/Solvers/Solvers.jl:396-418): per element the mass
// matrix M = VDM' diag(W J) VDM is formed, factorised by Cholesky and solved
// against VDM' (W J u_q), one to four elements in a CTA: the weights, nodal
// data, mass matrix, factor and right-hand sides live in shared memory; VDM is
// staged there a chunk of nodes at a time.
#include <cmath>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/sse_gb300.h"
#include "sse_kernels.cuh"

namespace sse {
namespace {

struct ProjArgs {
  int np, nq, nc;
  int64_t ne;
  int epb;           // elements per block
  int chunk;         // nodes staged at a time
  const int *tri;    // r << 16 | c of the lower triangle's entries, rows in order
  const double *V, *W, *J, *uq;
  double *u0;
  int *flag;  // set when a mass matrix is not positive definite
};

constexpr int kThreads = 256;

// Shared memory: of each element WJ[nq], U[nc][nq] (then W J u), M[np][np] (lower
// triangle, overwritten by the Cholesky factor) and Y[nc][np]; then, STAGED,
// chunk nodes of VDM and, of each element, of W J VDM, node-major.
//
// Bound by the FP64 pipe (a warp instruction takes it for 16 cycles however few
// lanes are live): the mass matrix is 630 sums of 125 terms at p = 4.  So the
// products W J VDM are formed once a chunk rather than once a term, and the
// factorisation updates all remaining entries after each column, with the
// elements of a block sharing the warps of the square roots, divisions and
// solves.  Each entry's sum keeps its order, so the results do not change.
// 10,368 p = 4 tets, the whole call: 5.79 ms with a product a term, one element
// a block and the factorisation by dot products; 3.20 ms.
template <bool STAGED>
__global__ void __launch_bounds__(kThreads) project_function_kernel(ProjArgs a) {
  extern __shared__ double sm[];
  __shared__ int bad;
  const int np = a.np, nq = a.nq, nc = a.nc;
  const int64_t k0 = (int64_t)blockIdx.x * a.epb;
  const int live = (int)(a.ne - k0 < a.epb ? a.ne - k0 : a.epb);
  const int per = nq + nc * nq + np * np + nc * np;  // doubles an element
  const int oU = nq, oM = oU + nc * nq, oY = oM + np * np;
  double *Vc = sm + (size_t)a.epb * per, *VWc = Vc + a.chunk * np;
  if (threadIdx.x == 0) bad = 0;
  for (int t = threadIdx.x; t < live * nq; t += kThreads) {
    const int el = t / nq, i = t - el * nq;
    double *E = sm + (size_t)el * per;
    const double w = a.W[i] * a.J[(size_t)nq * k0 + t];
    E[i] = w;
    // lmul!(WJ, u_q): U <- WJ .* U
    for (int e = 0; e < nc; ++e) E[oU + e * nq + i] = a.uq[((size_t)nc * (k0 + el) + e) * nq + i] * w;
  }
  const int ntri = np * (np + 1) / 2, tasks = ntri + nc * np;
  for (int i0 = 0; i0 < nq; i0 += a.chunk) {
    const int n = min(a.chunk, nq - i0);
    __syncthreads();
    if constexpr (STAGED) {
      for (int t = threadIdx.x; t < n * np; t += kThreads) {
        const int r = t / n, i = t - r * n;
        const double v = a.V[i0 + i + (size_t)nq * r];
        Vc[i * np + r] = v;
        for (int el = 0; el < live; ++el) VWc[(el * a.chunk + i) * np + r] = v * sm[(size_t)el * per + i0 + i];
      }
      __syncthreads();
    }
    // M[r][c] (r >= c) = sum_i VDM[i, r] WJ[i] VDM[i, c] and
    // Y[e][r] = sum_i VDM[i, r] (WJ u_q)[e][i]
    for (int t = threadIdx.x; t < live * tasks; t += kThreads) {
      const int el = t / tasks, q = t - el * tasks;
      double *E = sm + (size_t)el * per;
      if (q < ntri) {
        const int rc = __ldg(a.tri + q), r = rc >> 16, c = rc & 0xffff;
        double acc = i0 ? E[oM + r * np + c] : 0.0;
        if constexpr (STAGED) {
          const double *x = VWc + el * a.chunk * np + r, *y = Vc + c;
#pragma unroll 4
          for (int i = 0; i < n; ++i) acc = fma(x[i * np], y[i * np], acc);
        } else {
          const double *vr = a.V + i0 + (size_t)nq * r, *vc = a.V + i0 + (size_t)nq * c;
          for (int i = 0; i < n; ++i) acc = fma(__ldg(vr + i) * E[i0 + i], __ldg(vc + i), acc);
        }
        E[oM + r * np + c] = acc;
      } else {
        const int e = (q - ntri) / np, r = q - ntri - e * np;
        const double *u = E + oU + e * nq + i0;
        double acc = i0 ? E[oY + e * np + r] : 0.0;
        for (int i = 0; i < n; ++i)
          acc = fma(STAGED ? Vc[i * np + r] : __ldg(a.V + i0 + i + (size_t)nq * r), u[i], acc);
        E[oY + e * np + r] = acc;
      }
    }
  }
  __syncthreads();
  // Cholesky M = L L' by columns (L overwrites the lower triangle), and L z = y
  // along with it
  for (int j = 0; j < np; ++j) {
    if (threadIdx.x < live) {
      double *d = sm + (size_t)threadIdx.x * per + oM + j * np + j;
      double v = *d;
      if (!(v > 0.0)) {
        bad = 1;
        v = 1.0;
      }
      *d = sqrt(v);
    }
    __syncthreads();
    const int below = np - 1 - j;
    for (int t = threadIdx.x; t < live * (below + nc); t += kThreads) {
      const int el = t / (below + nc), q = t - el * (below + nc);
      double *E = sm + (size_t)el * per;
      double *x = q < below ? E + oM + (j + 1 + q) * np + j : E + oY + (q - below) * np + j;
      *x /= E[oM + j * np + j];
    }
    __syncthreads();
    const int rest = below * (below + 1) / 2, all = rest + nc * below;
    for (int t = threadIdx.x; t < live * all; t += kThreads) {
      const int el = t / all, q = t - el * all;
      double *M = sm + (size_t)el * per + oM, *Y = M + np * np;
      if (q < rest) {
        const int rc = __ldg(a.tri + q), r = (rc >> 16) + j + 1, c = (rc & 0xffff) + j + 1;
        M[r * np + c] = fma(-M[r * np + j], M[c * np + j], M[r * np + c]);
      } else {
        const int e = (q - rest) / below, r = q - rest - e * below + j + 1;
        Y[e * np + r] = fma(-M[r * np + j], Y[e * np + j], Y[e * np + r]);
      }
    }
    __syncthreads();
  }
  // L' x = z, one right-hand side per thread
  for (int t = threadIdx.x; t < live * nc; t += kThreads) {
    const double *M = sm + (size_t)(t / nc) * per + oM;
    double *y = sm + (size_t)(t / nc) * per + oY + (t % nc) * np;
    for (int r = np - 1; r >= 0; --r) {
      double s = y[r];
      for (int q = r + 1; q < np; ++q) s = fma(-M[q * np + r], y[q], s);
      y[r] = s / M[r * np + r];
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < live * nc * np; t += kThreads) {
    const int el = t / (nc * np);
    a.u0[(size_t)nc * np * k0 + t] = sm[(size_t)el * per + oY + t - el * nc * np];
  }
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
  const size_t element = ((size_t)nq + (size_t)nc * nq + (size_t)np * np + (size_t)nc * np) * sizeof(double);
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const size_t static_bytes = 16;
  if (element + static_bytes > (size_t)optin) {
    *err = "element too large for one CTA's shared memory";
    return SSE_ERR_UNSUPPORTED;
  }
  // as many elements a block as leave room for three blocks on an SM; the chunk
  // shrinks, and at last goes, where one element alone fills shared memory
  int epb = 4, chunk = 16;
  auto bytes = [&](int n, int ch) { return n * element + (size_t)(n + 1) * ch * np * sizeof(double); };
  while (epb > 1 && bytes(epb, chunk) > (size_t)74 * 1024) epb /= 2;
  while (chunk > 0 && bytes(epb, chunk) + static_bytes > (size_t)optin) --chunk;
  const bool staged = chunk > 0;
  const size_t smem = bytes(epb, chunk);
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
  std::vector<int> tri;
  for (int r = 0; r < np; ++r)
    for (int c = 0; c <= r; ++c) tri.push_back(r << 16 | c);
  if ((e = buf.alloc(tri.size() * sizeof(int), &p)) != cudaSuccess) return cuda(e, "allocate");
  a.tri = (const int *)p;
  if ((e = cudaMemcpy(p, tri.data(), tri.size() * sizeof(int), cudaMemcpyHostToDevice)) != cudaSuccess)
    return cuda(e, "upload triangle");
  a.ne = ne;
  a.epb = epb;
  a.chunk = staged ? chunk : nq;
  if ((e = buf.alloc(sizeof(int), &p)) != cudaSuccess) return cuda(e, "allocate");
  a.flag = (int *)p;
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
  auto *kernel = staged ? project_function_kernel<true> : project_function_kernel<false>;
  raise_smem_limit((const void *)kernel, smem);
  kernel<<<(unsigned)((ne + epb - 1) / epb), kThreads, smem>>>(a);
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
