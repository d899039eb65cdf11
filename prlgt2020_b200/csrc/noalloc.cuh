// Allocation-free static plaquette of a caller-owned device field.
//
// Same quantity as nspt_plaquette_measure (plaquette_measure, OpenMP
// branch, nspt.cc:1362-1404: sum over links of Tr(U_mu(x) * staples) / 72V
// per order) computed without a context.  The field is read where the caller
// keeps it -- the reference's AoS layout (ptGluon_fld, QCDenvNODEpt_test.h:
// 331-338) in device memory -- and the only scratch is a fixed, file-scope
// device array: one row of per-order partial sums per CTA plus one result
// row.  Nothing is allocated, on the device or the host.
//
// Scratch contents: every call writes each partial row it later reads and
// the result row before reading them, so nothing in the array has to start
// at zero and stale contents from an earlier call are never used.  Two calls
// that overlap on one device (different host threads or streams) share the
// array and race; callers serialise them.
#pragma once

#include <mutex>

namespace nspt {

constexpr int NOALLOC_BLOCKS = 1024;               // partial rows (max CTAs per call)
constexpr int NOALLOC_ROW = NSPT_MAX_ORDER + 1;    // orders 0..NSPT_MAX_ORDER
constexpr int NOALLOC_MAX_DEVICES = 64;
// (NOALLOC_BLOCKS + 1) rows of NOALLOC_ROW complex doubles: 803,600 bytes
static __device__ __align__(256) double2 g_noalloc_scratch[(NOALLOC_BLOCKS + 1) * NOALLOC_ROW];

// Sum the CTAs' partial rows in block order into the result row.
__global__ void k_plaq_noalloc_sum(const double2 *partial, int nblocks, int N, double2 *out) {
  for (int k = threadIdx.x; k <= N; k += blockDim.x) {
    double2 s = cz();
    for (int b = 0; b < nblocks; b++) s = cadd(s, partial[(size_t)b * NOALLOC_ROW + k]);
    out[k] = s;
  }
}

}  // namespace nspt

namespace {

// Per-device set-up, done once with that device current: the scratch
// array's address, the launch limits and the twist matrices.  It is kept
// until the process exits; a cudaDeviceReset after the first call reloads
// the module and leaves these values stale, which the header documents as
// unsupported.
struct NoallocDevice {
  bool ready;
  double2 *scratch;
  int nsm;
  int smem_optin;
};
NoallocDevice g_noalloc_dev[nspt::NOALLOC_MAX_DEVICES];
std::mutex g_noalloc_mu;

int noalloc_setup(int dev, NoallocDevice **out) {
  using namespace nspt;
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  NoallocDevice &d = g_noalloc_dev[dev];
  if (!d.ready) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess) return NSPT_ERR_CUDA;
    if (!p || (reinterpret_cast<uintptr_t>(p) & 255u)) return NSPT_ERR_CUDA;
    if (cudaDeviceGetAttribute(&d.nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      return NSPT_ERR_CUDA;
    if (cudaDeviceGetAttribute(&d.smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
        cudaSuccess)
      return NSPT_ERR_CUDA;
    if (cudaFuncSetAttribute(k_plaq_trace<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             d.smem_optin) != cudaSuccess)
      return NSPT_ERR_CUDA;
    // twist matrices (twistmatrices.h:158-240), the values nspt_create uploads
    double2 om[4][9], omd[4][9];
    for (int a = 0; a < 4; a++)
      for (int e = 0; e < 9; e++) om[a][e] = make_double2(0.0, 0.0);
    for (int a = 0; a < 2; a++)
      for (int e = 0; e < 9; e += 4) om[a][e] = make_double2(1.0, 0.0);
    om[1][0] = make_double2(cos(-2. * M_PI / 3.), sin(-2. * M_PI / 3.));
    om[1][8] = make_double2(cos(2. * M_PI / 3.), sin(2. * M_PI / 3.));
    om[2][1] = om[2][5] = om[2][6] = make_double2(1.0, 0.0);
    om[3][1] = make_double2(cos(-2. * M_PI / 3.), sin(-2. * M_PI / 3.));
    om[3][5] = make_double2(1.0, 0.0);
    om[3][6] = make_double2(cos(2. * M_PI / 3.), sin(2. * M_PI / 3.));
    for (int a = 0; a < 4; a++)
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++)
          omd[a][3 * i + j] = make_double2(om[a][3 * j + i].x, -om[a][3 * j + i].y);
    if (cudaMemcpyToSymbol(c_om, om, sizeof(om)) != cudaSuccess) return NSPT_ERR_CUDA;
    if (cudaMemcpyToSymbol(c_omd, omd, sizeof(omd)) != cudaSuccess) return NSPT_ERR_CUDA;
    d.scratch = static_cast<double2 *>(p);
    d.ready = true;
  }
  *out = &d;
  return NSPT_OK;
}

}  // namespace

extern "C" int nspt_plaquette_measure_noalloc(const void *links_dev, int allocORD, const int L[4],
                                              int N, unsigned flags, double *plaq, void *stream) {
  using namespace nspt;
  if (!links_dev || !L || !plaq) return NSPT_ERR_ARG;
  if (N < 1 || N > NSPT_MAX_ORDER) return NSPT_ERR_ORDER;  // beyond the scratch rows
  if (allocORD < N) return NSPT_ERR_ARG;
  if (flags & ~(NSPT_TWIST_Y | NSPT_TWIST_Z | NSPT_TWIST_T)) return NSPT_ERR_ARG;
  if (reinterpret_cast<uintptr_t>(links_dev) & 15u) return NSPT_ERR_ARG;
  long V = 1;
  for (int d = 0; d < 4; d++) {
    if (L[d] < 1) return NSPT_ERR_ARG;
    V *= L[d];
  }
  if (V > (1L << 29)) return NSPT_ERR_ARG;  // 4V links index an int site range
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return NSPT_ERR_NODEVICE;
  if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return NSPT_ERR_ARG;
  NoallocDevice *d = nullptr;
  int rc = noalloc_setup(dev, &d);
  if (rc) return rc;

  const size_t ser = 1 + 9 * (size_t)allocORD;
  const int SS = (int)link_rec(N);
  Geo g;
  for (int k = 0; k < 4; k++) g.L[k] = L[k];
  g.s2 = L[3];
  g.s1 = L[2] * g.s2;
  g.s0 = L[1] * g.s1;
  g.V = (int)V;
  g.twist = 0;
  if (flags & NSPT_TWIST_Y) g.twist |= 2u;
  if (flags & NSPT_TWIST_Z) g.twist |= 4u;
  if (flags & NSPT_TWIST_T) g.twist |= 8u;

  const Shape sh = group_shape(32, 4, MEASURE_SLOTS, SS, (size_t)d->smem_optin);
  if (sh.gpc < 1) return NSPT_ERR_ORDER;
  const long want = (6 * V + sh.gpc - 1) / sh.gpc;
  const int blocks = (int)std::min<long>(want, NOALLOC_BLOCKS);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  double2 *partial = d->scratch;
  double2 *result = d->scratch + (size_t)NOALLOC_BLOCKS * NOALLOC_ROW;
  const double2 *U = static_cast<const double2 *>(links_dev);
  k_plaq_trace<32><<<blocks, 32 * sh.warps, sh.smem, st>>>(U, ser, N, SS, g, partial, NOALLOC_ROW,
                                                       sh.gpc);
  if (cudaGetLastError() != cudaSuccess) return NSPT_ERR_CUDA;
  k_plaq_noalloc_sum<<<1, 64, 0, st>>>(partial, blocks, N, result);
  if (cudaGetLastError() != cudaSuccess) return NSPT_ERR_CUDA;
  if (cudaMemcpyAsync(plaq, result, (size_t)(N + 1) * sizeof(double2), cudaMemcpyDeviceToHost,
                      st) != cudaSuccess)
    return NSPT_ERR_CUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess) return NSPT_ERR_CUDA;
  for (int k = 0; k <= N; k++) {  // nspt.cc:1398-1404
    plaq[2 * k] /= (double)(V * 72);
    plaq[2 * k + 1] /= (double)(V * 72);
  }
  return NSPT_OK;
}
