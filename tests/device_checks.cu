// device_checks.cu -- small calls into the engine's device code that no entry
// point of the library makes by itself, for tests/test_device_functions.py:
// the branch-free divisions of hg_phys.cuh on given operands, and the FP32
// flux kernels of hg_mixed.cu (hg::launch_flux_f32 of libharmgpu.so) on given
// states and geometry.  Every function returns 0 or the CUDA error.
#include <cstring>
#include <vector>

#include "harmgpu.h"
#include "hg_phys.cuh"

namespace hg {
void launch_flux_f32(const GridDev &G, const LaunchCfg &L, cudaStream_t s, int d, const int *lo, const int *n,
                     unsigned int mult, int slot, int all);
}
using namespace hg;

// Device memory freed with the object; err holds the first error.
struct Pool {
  std::vector<void *> ptrs;
  cudaError_t err = cudaSuccess;
  void note(cudaError_t e) { if (err == cudaSuccess) err = e; }
  template <class T>
  T *make(size_t n, const T *src)
  {
    void *p = nullptr;
    note(cudaMalloc(&p, n * sizeof(T)));
    if (err != cudaSuccess) return nullptr;
    ptrs.push_back(p);
    note(src ? cudaMemcpy(p, src, n * sizeof(T), cudaMemcpyHostToDevice) : cudaMemset(p, 0, n * sizeof(T)));
    return (T *)p;
  }
  template <class T>
  void get(T *dst, const T *src, size_t n) { note(cudaMemcpy(dst, src, n * sizeof(T), cudaMemcpyDeviceToHost)); }
  ~Pool() { for (void *p : ptrs) cudaFree(p); }
};

// out: a/b, 1/b, 1/b by rcp_any, a/b by div_any, within(a, b, tol); ok of each
__global__ void k_divisions(int n, const double *a, const double *b, double tol, double *out, unsigned char *ok)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  FastDiv dv[5];
  out[t] = dv[0].div(a[t], b[t]);
  out[n + t] = dv[1].rcp(b[t]);
  out[2 * n + t] = dv[2].rcp_any(b[t]);
  out[3 * n + t] = dv[3].div_any(a[t], b[t]);
  out[4 * n + t] = dv[4].within(a[t], b[t], tol);
  for (int q = 0; q < 5; q++) ok[q * n + t] = dv[q].ok;
}

extern "C" int check_divisions(int n, const double *a, const double *b, double tol, double *out, unsigned char *ok)
{
  Pool m;
  double *da = m.make(n, a), *db = m.make(n, b), *dout = m.make<double>(5 * (size_t)n, nullptr);
  unsigned char *dok = m.make<unsigned char>(5 * (size_t)n, nullptr);
  if (m.err != cudaSuccess) return m.err;
  k_divisions<<<(n + 127) / 128, 128>>>(n, da, db, tol, dout, dok);
  m.note(cudaGetLastError());
  m.get(out, dout, 5 * (size_t)n);
  m.get(ok, dok, 5 * (size_t)n);
  return m.err;
}

// Fluxes of the three directions on a grid of n physical zones (every
// direction resolved) from FP32 primitives (8 planes, x1 fastest).  geom: one
// row of 42 (metric_dim 0) or HG_NPOS x T1 x T0 rows (metric_dim 2), gk the
// HG_GK_* the kernels are chosen by.  F: 3 x 8 planes, maxs: the largest
// speeds, booked: the failures of gamma_calc per zone.
extern "C" int check_flux_f32(const int *n, int recon, int flux, int mdim, int gk, int strip_nf, int strip_x1,
                              double gam, const float *prims, const double *geom, double *F, double *maxs,
                              unsigned *booked)
{
  Pool m;
  GridDev G;
  memset(&G, 0, sizeof(G));
  int st = 1;
  for (int a = 0; a < 3; a++) {
    G.N[a] = n[a];
    G.T[a] = n[a] + 2 * HG_NGH;
    G.NE[a] = n[a] + HG_NGH - 1;
    G.st[a] = st;
    st *= G.T[a];
  }
  G.S = st;
  G.recon = recon;
  G.flux = flux;
  G.ct_para = 1;
  G.bc = 10;
  G.mdim = mdim;
  G.gk = gk;
  G.prec = HG_PREC_MIXED;
  G.gam = gam;
  memcpy(G.g0.gcon, geom, 16 * 8);
  memcpy(G.g0.gcov, geom + 16, 16 * 8);
  G.g0.g = geom[32];
  G.g0.g_inv = geom[33];
  G.g0.alpha = geom[34];
  for (int a = 0; a < 3; a++) G.g0.beta[a] = geom[35 + a];
  for (int a = 0; a < 4; a++) G.g0.ncon[a] = geom[38 + a];
  if (mdim == 2) {
    G.gS = (long)HG_NPOS * G.T[0] * G.T[1];
    std::vector<float> t((size_t)HG_GF * G.gS);
    for (long o = 0; o < G.gS; o++) {
      const double *s = geom + 42 * o;
      for (int a = 0; a < 16; a++) t[a * G.gS + o] = (float)s[16 + a];
      t[16 * G.gS + o] = (float)s[0];
      for (int j = 1; j <= 3; j++) {
        t[(16 + j) * G.gS + o] = (float)s[j];
        t[(19 + j) * G.gS + o] = (float)s[j * 4 + j];
      }
      t[23 * G.gS + o] = (float)s[38];
      for (int a = 0; a < 3; a++) t[(24 + a) * G.gS + o] = (float)s[35 + a];
      t[27 * G.gS + o] = (float)s[32];
    }
    G.geomF = m.make(t.size(), t.data());
  }
  G.p32 = m.make(HG_NPR * (size_t)G.S, prims);
  for (int d = 0; d < 3; d++) G.F[d] = m.make<double>(HG_NPR * (size_t)G.S, nullptr);
  G.nfail = m.make<unsigned>(HG_NF * (size_t)G.S, nullptr);
  G.sc = m.make<DevScalars>(1, nullptr);
  if (m.err != cudaSuccess) return m.err;
  LaunchCfg L;
  memset(&L, 0, sizeof(L));
  L.grid_flux32 = 5;  // a few strips for each thread
  L.strip_nf = strip_nf;
  L.strip_x1 = strip_x1;
  for (int d = 0; d < 3; d++) {
    int lo[3], c[3];
    for (int a = 0; a < 3; a++) {
      lo[a] = a == d ? HG_NGH : 0;
      c[a] = a == d ? n[a] + 1 : G.T[a];
    }
    launch_flux_f32(G, L, 0, d, lo, c, 1u, 0, 0);
    m.note(cudaGetLastError());
  }
  m.note(cudaDeviceSynchronize());
  if (m.err != cudaSuccess) return m.err;
  for (int d = 0; d < 3; d++) m.get(F + d * HG_NPR * (size_t)G.S, G.F[d], HG_NPR * (size_t)G.S);
  m.get(booked, G.nfail + NF_GAMMA_CALC * G.S, (size_t)G.S);
  DevScalars sc;
  m.get(&sc, G.sc, 1);
  for (int d = 0; d < 3; d++) memcpy(maxs + d, &sc.maxs[d + 1], 8);
  return m.err;
}
