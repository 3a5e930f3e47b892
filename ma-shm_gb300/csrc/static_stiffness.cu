// static_stiffness.cu -- allocation-free internal-force entry point.
//
// shm_stiffness_static() computes the assembled flat-shell internal force
// F = K*U for a mesh whose arrays already live in device memory, without
// allocating anything: no cudaMalloc, no cudaFree, no library call that
// allocates.  It exists for callers that cannot allocate device memory on
// their own terms:
//   * a MATLAB MEX gateway working on gpuArray data owned by MATLAB's GPU
//     memory manager, which keeps a pool of the device memory and whose
//     accounting a hidden cudaMalloc would bypass (and can fail when MATLAB
//     has reserved most of the memory);
//   * monitoring loops that run for days on a fixed memory budget and forbid
//     any allocation after start-up, so that a run never dies on an
//     out-of-memory error half way.
// The element-local forces (the reference's F2, main_flat_shell.m:716-721)
// are kept in a file-scope device array of SHM_STATIC_MAX_ELEMS elements
// (5 x 36 doubles each, 5.9 MB), which every GPU that loads the library holds
// until the process exits.  The assembly is the reference's 12-basket scatter
// F(I_G(:,b)) += F2(I_L(:,b)), b = 1..12 (main_flat_shell.m:724-726), driven by
// the caller's I_G / I_L maps (nodesMaps_Fiborek.m), so the summation order is
// the reference's.
//
// A call is two launches.  The first computes the element forces and, in
// further CTAs, turns the maps round: slot b of node g in a second file-scope
// array (12 ints per node, 7.1 MB) receives the row of basket b that names g
// and an element node.
// The second sums each node's element forces in basket order and writes F; it
// takes a slot only if the caller's map does name g in that row, so whatever
// earlier calls left in the array does no harm and nothing is cleared.  (The
// former memset, element kernel and twelve basket kernels cost 138 us for 99
// elements, 57 us of it one SM's FP64 pipe working through 32 elements.)  The
// basket kernels remain for nnode beyond the slot array, which a mesh of at
// most SHM_STATIC_MAX_ELEMS elements only has with nodes that no element uses.
//
// Set-up: the first call on a device (with that device current) looks up the
// device address of the array with cudaGetSymbolAddress, copies the GLL
// derivative matrix to this file's constant memory and raises the kernel's
// shared-memory limit.  Make that first call before any stream capture.
// Every call uses the same array and leaves its contents behind; calls that
// overlap on the GPU (two streams at once) race on it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>

#include "internal.h"
#include "shmsem.h"
#include "shell_element.cuh"

using namespace shm;

namespace {

__device__ __align__(256) double g_static_f2[(size_t)5 * NPE * SHM_STATIC_MAX_ELEMS];

constexpr int kMaxNodes = NPE * SHM_STATIC_MAX_ELEMS, kBaskets = 12;
__device__ __align__(256) int g_static_slot[(size_t)kBaskets * kMaxNodes];  // [node][basket] row of the maps

constexpr int kMaxDevices = 64;
double* s_f2_addr[kMaxDevices] = {nullptr};
int* s_slot_addr[kMaxDevices] = {nullptr};
int s_sms[kMaxDevices] = {0};
std::mutex s_setup_mutex;
thread_local std::string t_err;  // text of this thread's last failed call

// records which step failed; the error of a CUDA call made here is cleared so
// that it does not surface in the caller's next error check
shm_status fail(const char* stage, cudaError_t e, bool clear) {
  if (clear) cudaGetLastError();
  t_err = std::string("shm_stiffness_static: ") + stage + ": " + cudaGetErrorString(e);
  return e == cudaErrorMemoryAllocation ? SHM_ERR_OOM : SHM_ERR_CUDA;
}

// The element part in FP64, which runs at two operations per clock and SM: the
// elements are spread over all SMs (1 to 7 per CTA), and each phase is split
// over the CTA's threads as finely as its results allow -- derivatives and
// transposed operators by (field, node), geometry and resultants by node.
constexpr int kElemMax = 7;                      // elements per CTA: 252 nodes on 256 threads
constexpr int kElemThreads = 256;
constexpr int kElemVals = 21 * NPE;              // per element: u (5), x, y; their xi- and eta-derivatives
constexpr int kSlotThreads = 64;                 // nodes per CTA of the assembly

size_t static_smem_bytes(int ne) { return sizeof(double) * (size_t)ne * kElemVals; }

__global__ void __launch_bounds__(kElemThreads) k_static_elem(int fen, int nnode, int ne, int ecta,
                                                              const int* __restrict__ nodes,
                                                              const double* __restrict__ coords,
                                                              const double* __restrict__ lam,
                                                              const double* __restrict__ U, double* f2, int rows,
                                                              const int* __restrict__ IG,
                                                              const int* __restrict__ IL, int* slot) {
  if ((int)blockIdx.x >= ecta) {  // turn the basket maps round
    const int64_t n = (int64_t)kBaskets * rows, step = (int64_t)(gridDim.x - ecta) * kElemThreads;
    for (int64_t q = ((int64_t)blockIdx.x - ecta) * kElemThreads + threadIdx.x; q < n; q += step) {
      const int g = IG[q], l = IL[q];
      // empty (0) or out of range; a row that names a node without an element node must
      // not take the place of one with (maps padded with a node's number)
      if (g < 1 || g > nnode || l < 1 || l > fen * NPE) continue;
      const int b = (int)(q / rows);
      slot[(int64_t)(g - 1) * kBaskets + b] = (int)(q - (int64_t)b * rows);
    }
    return;
  }
  extern __shared__ __align__(16) unsigned char smraw[];
  double* sm = reinterpret_cast<double*>(smraw);
  __shared__ double sD[NPE];
  const int e0 = blockIdx.x * ne, nel = min(ne, fen - e0);
  for (int w = threadIdx.x; w < NPE; w += kElemThreads) sD[w] = Dm<double>(w / NP, w % NP);
  for (int w = threadIdx.x; w < NPE * nel; w += kElemThreads) {
    const int le = w / NPE, n = w % NPE;
    int node = nodes[(int64_t)n * fen + e0 + le] - 1;
    if (node >= nnode) node = -1;  // out-of-range entries read as zero
    double* v = sm + le * kElemVals + n;
#pragma unroll
    for (int f = 0; f < 5; ++f) v[f * NPE] = node >= 0 ? U[5 * (int64_t)node + f] : 0.0;
    v[5 * NPE] = node >= 0 ? coords[node] : 0.0;
    v[6 * NPE] = node >= 0 ? coords[(int64_t)nnode + node] : 0.0;
  }
  __syncthreads();
  for (int w = threadIdx.x; w < 7 * NPE * nel; w += kElemThreads) {
    const int le = w / (7 * NPE), r = w % (7 * NPE), f = r / NPE, n = r % NPE, i = n % NP, k = n / NP;
    double* v = sm + le * kElemVals + f * NPE;
    double x = 0.0, y = 0.0;
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      x = fma(sD[i * NP + q], v[k * NP + q], x);
      y = fma(sD[k * NP + q], v[q * NP + i], y);
    }
    v[7 * NPE + n] = x;
    v[14 * NPE + n] = y;
  }
  __syncthreads();
  for (int w = threadIdx.x; w < NPE * nel; w += kElemThreads) {
    const int le = w / NPE, n = w % NPE, i = n % NP, k = n / NP, e = e0 + le;
    double* v = sm + le * kElemVals + n;
    double* dx = v + 7 * NPE;
    double* de = v + 14 * NPE;
    const double J11 = dx[5 * NPE], J21 = dx[6 * NPE], J12 = de[5 * NPE], J22 = de[6 * NPE];
    const double det = J11 * J22 - J12 * J21, a = 1.0 / det;
    const double i11 = a * J22, i12 = -a * J12, i21 = -a * J21, i22 = a * J11;
    const double W = Wg<double>(i) * Wg<double>(k) * det;
    double gx[5], gy[5];
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      gx[f] = dx[f * NPE] * i11 + de[f * NPE] * i21;
      gy[f] = dx[f * NPE] * i12 + de[f * NPE] * i22;
    }
    auto L = [&](int q) { return lam[(int64_t)q * fen + e]; };
    const double ex = gx[0], ey = gy[2], gxy = gy[0] + gx[2], kx = gx[1], ky = gy[3], kxy = gy[1] + gx[3];
    const double gyz = v[3 * NPE] + gy[4], gxz = v[NPE] + gx[4];
    const double Nxx = L(0) * ex + L(1) * ey + L(2) * gxy + L(9) * kx + L(10) * ky + L(11) * kxy;
    const double Nyy = L(1) * ex + L(3) * ey + L(4) * gxy + L(10) * kx + L(12) * ky + L(13) * kxy;
    const double Nxy = L(2) * ex + L(4) * ey + L(5) * gxy + L(11) * kx + L(13) * ky + L(14) * kxy;
    const double Mxx = L(9) * ex + L(10) * ey + L(11) * gxy + L(15) * kx + L(16) * ky + L(17) * kxy;
    const double Myy = L(10) * ex + L(12) * ey + L(13) * gxy + L(16) * kx + L(18) * ky + L(19) * kxy;
    const double Mxy = L(11) * ex + L(13) * ey + L(14) * gxy + L(17) * kx + L(19) * ky + L(20) * kxy;
    const double Qy = L(6) * gyz + L(7) * gxz, Qx = L(7) * gyz + L(8) * gxz;
    const double w11 = W * i11, w12 = W * i12, w21 = W * i21, w22 = W * i22;
    const double Sx[5] = {Nxx, Mxx, Nxy, Mxy, Qx}, Sy[5] = {Nxy, Mxy, Nyy, Myy, Qy};
#pragma unroll
    for (int f = 0; f < 5; ++f) {  // fluxes over the node's own derivatives
      dx[f * NPE] = w11 * Sx[f] + w12 * Sy[f];
      de[f * NPE] = w21 * Sx[f] + w22 * Sy[f];
    }
    v[NPE] = W * Qx;      // + Sxz.*WWDetJ into mx
    v[3 * NPE] = W * Qy;  // + Syz.*WWDetJ into my
  }
  __syncthreads();
  // element-local forces in the reference's F2 layout (5 per local node)
  for (int w = threadIdx.x; w < 5 * NPE * nel; w += kElemThreads) {
    const int le = w / (5 * NPE), r = w % (5 * NPE), f = r / NPE, n = r % NPE, i = n % NP, k = n / NP;
    const double* v = sm + le * kElemVals + f * NPE;
    double F = (f == 1 || f == 3) ? v[n] : 0.0;
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      F = fma(sD[q * NP + i], v[7 * NPE + k * NP + q], F);
      F = fma(sD[q * NP + k], v[14 * NPE + q * NP + i], F);
    }
    f2[((int64_t)(e0 + le) * NPE + n) * 5 + f] = F;
  }
}

// F of each node: its element forces in basket order
__global__ void __launch_bounds__(kSlotThreads) k_static_nodes(int nnode, int nlocal, int rows,
                                                               const int* __restrict__ IG, const int* __restrict__ IL,
                                                               const int* __restrict__ slot,
                                                               const double* __restrict__ f2, double* F) {
  const int g = blockIdx.x * kSlotThreads + threadIdx.x;
  if (g >= nnode) return;
  const int4* s4 = reinterpret_cast<const int4*>(slot + (int64_t)g * kBaskets);
  int r[kBaskets], l[kBaskets];
#pragma unroll
  for (int q = 0; q < kBaskets / 4; ++q) {
    const int4 v = s4[q];
    r[4 * q] = v.x;
    r[4 * q + 1] = v.y;
    r[4 * q + 2] = v.z;
    r[4 * q + 3] = v.w;
  }
#pragma unroll
  for (int b = 0; b < kBaskets; ++b) {  // (the maps confirm the slot)
    l[b] = 0;
    if (r[b] >= 0 && r[b] < rows && IG[(int64_t)b * rows + r[b]] == g + 1) l[b] = IL[(int64_t)b * rows + r[b]];
  }
  double a[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int b = 0; b < kBaskets; ++b)
    if (l[b] >= 1 && l[b] <= nlocal) {
#pragma unroll
      for (int f = 0; f < 5; ++f) a[f] += f2[5 * (int64_t)(l[b] - 1) + f];
    }
#pragma unroll
  for (int f = 0; f < 5; ++f) F[5 * (int64_t)g + f] = a[f];
}

__global__ void k_static_basket(int rows, int b, int nnode, int nlocal, const int* __restrict__ IG,
                                const int* __restrict__ IL, const double* __restrict__ f2, double* F) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  const int g = IG[(int64_t)b * rows + r];
  const int l = IL[(int64_t)b * rows + r];
  if (g < 1 || g > nnode || l < 1 || l > nlocal) return;  // empty slot (0) or out of range
#pragma unroll
  for (int f = 0; f < 5; ++f) F[5 * (int64_t)(g - 1) + f] += f2[5 * (int64_t)(l - 1) + f];
}

void gll6(double* D, double* w) {
  // GLL nodes of order 5 (Newton on P5'), weights 2/(30 P5(x)^2), and the
  // Lagrange derivative matrix by barycentric weights; |D| < 1e-12 -> 0
  const int n = NP, N = n - 1;
  double x[NP];
  x[0] = -1.0;
  x[N] = 1.0;
  auto leg = [N](double t, double& p, double& dp) {
    double p0 = 1.0, p1 = t;
    for (int k = 2; k <= N; ++k) {
      const double p2 = ((2.0 * k - 1.0) * t * p1 - (k - 1.0) * p0) / k;
      p0 = p1;
      p1 = p2;
    }
    p = p1;
    dp = N * (t * p1 - p0) / (t * t - 1.0);
  };
  for (int k = 1; k < N; ++k) {
    double t = -std::cos(M_PI * k / N);
    for (int it = 0; it < 100; ++it) {
      double p, dp;
      leg(t, p, dp);
      const double d2p = (2.0 * t * dp - N * (N + 1.0) * p) / (1.0 - t * t);
      const double step = dp / d2p;
      t -= step;
      if (std::fabs(step) < 1e-16) break;
    }
    x[k] = t;
  }
  for (int k = 0; k <= N / 2; ++k) {
    const double s = 0.5 * (x[N - k] - x[k]);
    x[k] = -s;
    x[N - k] = s;
  }
  for (int k = 0; k < n; ++k) {
    double p, dp;
    if (k == 0 || k == N) {
      p = (k == 0) ? -1.0 : 1.0;  // P5(+-1) = +-1
    } else {
      leg(x[k], p, dp);
    }
    w[k] = 2.0 / (N * (N + 1.0) * p * p);
  }
  double lam[NP];
  for (int j = 0; j < n; ++j) {
    lam[j] = 1.0;
    for (int k = 0; k < n; ++k)
      if (k != j) lam[j] /= (x[j] - x[k]);
  }
  for (int r = 0; r < n; ++r) {
    double diag = 0.0;
    for (int c = 0; c < n; ++c)
      if (c != r) {
        D[r * n + c] = (lam[c] / lam[r]) / (x[r] - x[c]);
        diag -= D[r * n + c];
      }
    D[r * n + r] = diag;
  }
  for (int q = 0; q < n * n; ++q)
    if (std::fabs(D[q]) < 1e-12) D[q] = 0.0;
}

// once per device, with the device current
shm_status setup_device(double** f2, int** slot, int* sms) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail("cudaGetDevice", e, true);
  if (dev < 0 || dev >= kMaxDevices) {
    t_err = "shm_stiffness_static: device ordinal beyond the library's table";
    return SHM_ERR_CUDA;
  }
  std::lock_guard<std::mutex> lock(s_setup_mutex);
  if (s_f2_addr[dev] == nullptr) {
    void* ptr = nullptr;
    if ((e = cudaGetSymbolAddress(&ptr, g_static_f2)) != cudaSuccess) return fail("cudaGetSymbolAddress", e, true);
    if (ptr == nullptr) return fail("cudaGetSymbolAddress", cudaErrorInvalidSymbol, false);
    void* sp = nullptr;
    if ((e = cudaGetSymbolAddress(&sp, g_static_slot)) != cudaSuccess) return fail("cudaGetSymbolAddress", e, true);
    if (sp == nullptr) return fail("cudaGetSymbolAddress", cudaErrorInvalidSymbol, false);
    if ((e = cudaDeviceGetAttribute(&s_sms[dev], cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
      return fail("cudaDeviceGetAttribute", e, true);
    double D[NP * NP], w[NP];
    gll6(D, w);
    if ((e = cudaMemcpyToSymbol(c_D64, D, sizeof(D))) != cudaSuccess) return fail("cudaMemcpyToSymbol", e, true);
    if ((e = cudaMemcpyToSymbol(c_w64, w, sizeof(w))) != cudaSuccess) return fail("cudaMemcpyToSymbol", e, true);
    if ((e = cudaFuncSetAttribute(k_static_elem, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)static_smem_bytes(kElemMax))) != cudaSuccess)
      return fail("cudaFuncSetAttribute", e, true);
    // (the caller's stream need not wait for the legacy one)
    if ((e = cudaStreamSynchronize(cudaStreamLegacy)) != cudaSuccess) return fail("cudaStreamSynchronize", e, true);
    s_slot_addr[dev] = static_cast<int*>(sp);
    s_f2_addr[dev] = static_cast<double*>(ptr);
  }
  *f2 = s_f2_addr[dev];
  *slot = s_slot_addr[dev];
  *sms = s_sms[dev];
  return SHM_OK;
}

}  // namespace

extern "C" shm_status shm_stiffness_static(int32_t fen, int32_t nnode, const int32_t* nodes, const double* coords,
                                           const double* lam, int32_t basket_rows, const int32_t* I_G,
                                           const int32_t* I_L, const double* U, double* F, void* stream) {
  if (fen < 1 || fen > SHM_STATIC_MAX_ELEMS || nnode < 1 || basket_rows < 1) {
    t_err = "shm_stiffness_static: fen must be 1..SHM_STATIC_MAX_ELEMS, nnode and basket_rows >= 1";
    return SHM_ERR_BAD_ARG;
  }
  if (!nodes || !coords || !lam || !I_G || !I_L || !U || !F) {
    t_err = "shm_stiffness_static: NULL array";
    return SHM_ERR_BAD_ARG;
  }
  // an error left pending by earlier work of the caller would be read back
  // as a failed launch below: report it before anything is queued (and leave
  // it pending for the caller's own check)
  cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) return fail("a CUDA error was already pending, nothing queued", e, false);
  double* f2 = nullptr;
  int *slot = nullptr, sms = 1;
  shm_status st = setup_device(&f2, &slot, &sms);
  if (st != SHM_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int ne = std::max(1, std::min(kElemMax, (fen + sms - 1) / sms)), ecta = (fen + ne - 1) / ne;
  const bool turn = nnode <= kMaxNodes;
  const int64_t entries = (int64_t)kBaskets * basket_rows;
  const int mcta = turn ? (int)std::min<int64_t>((entries + kElemThreads - 1) / kElemThreads, 2 * sms) : 0;
  if (!turn && (e = cudaMemsetAsync(F, 0, sizeof(double) * 5 * (size_t)nnode, s)) != cudaSuccess)
    return fail("cudaMemsetAsync of F", e, true);
  k_static_elem<<<ecta + mcta, kElemThreads, static_smem_bytes(ne), s>>>(fen, nnode, ne, ecta, nodes, coords, lam, U, f2,
                                                                         basket_rows, I_G, I_L, slot);
  if ((e = cudaGetLastError()) != cudaSuccess) return fail("k_static_elem launch", e, false);
  if (turn) {
    k_static_nodes<<<(nnode + kSlotThreads - 1) / kSlotThreads, kSlotThreads, 0, s>>>(nnode, fen * NPE, basket_rows, I_G,
                                                                                      I_L, slot, f2, F);
    if ((e = cudaGetLastError()) != cudaSuccess) return fail("k_static_nodes launch", e, false);
  } else {
    const int tb = 256, nb = (basket_rows + tb - 1) / tb;
    for (int b = 0; b < kBaskets; ++b) {
      k_static_basket<<<nb, tb, 0, s>>>(basket_rows, b, nnode, fen * NPE, I_G, I_L, f2, F);
      if ((e = cudaGetLastError()) != cudaSuccess) return fail("k_static_basket launch", e, false);
    }
  }
  t_err.clear();
  return SHM_OK;
}

const char* shm::static_last_error() { return t_err.empty() ? nullptr : t_err.c_str(); }
