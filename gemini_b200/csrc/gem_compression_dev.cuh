// Device form of the compression sub-step (app/main.f90:320-338): one thread per index of
// the per-index bodies in gem_compression.cuh, behind the C ABI (include/gem_fluid.h).
// Included by gem_fluid.cu (one translation unit with the plain path).

#include "gem_compression.cuh"

namespace gemk {

__global__ void kc_artvisc(gemc::View v, long long n, const double* __restrict__ ns,
                           const double* __restrict__ vs1, double* __restrict__ Q) {
  step_entry();
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    gemc::artvisc(v, t, ns, vs1, Q);
}
__global__ void kc_rk2_x1(gemc::View v, long long n, double* vs1) {
  step_entry();
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    gemc::rk2_x1(v, t, vs1);
}
__global__ void kc_rk2_x2(gemc::View v, long long n, double* vs1, double* vs2, double* vs3) {
  step_entry();
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    gemc::rk2_x2(v, t, vs1, vs2, vs3);
}
__global__ void kc_rk2_x3(gemc::View v, long long n, double* vs1, double* vs2, double* vs3) {
  step_entry();
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    gemc::rk2_x3(v, t, vs1, vs2, vs3);
}
__global__ void kc_compression(gemc::View v, long long n, const double* __restrict__ vs1,
                               const double* __restrict__ vs2, const double* __restrict__ vs3,
                               const double* __restrict__ Q, double* rhoes, const double* __restrict__ dtp) {
  step_entry();
  const double dt = *dtp;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    gemc::cmp(v, t, vs1, vs2, vs3, Q, rhoes, dt);
}

// VNRicht_artvisc, compression, rhoe2T and clean_param(3) of the interior cells in one pass:
// Q and the new temperature of one cell and species (blockIdx.y).  The ghost velocities that
// halo_fluidvars and RK2_global_boundary would leave are read as the interior cells they copy
// (the edge cell, or the wrapped one along a periodic x3); Q reads the x1 ghosts as the
// advection left them.  rhoes is not stored: after this only its conversion to T is used, and
// the diffusion's store rewrites it.  Quotients through the grid's reciprocal tables (exact).
// One pass instead of four; 384x96x96: 0.93 -> 0.47 ms at eight blocks per SM (32 registers, 32-48
// bytes spilled; 0.50 ms at 48 registers), half the copy peak by the eight doubles a cell and species needs.
template <bool UNIT>
__global__ void __launch_bounds__(256, 8) kc_compress_T(GridDev G, Blocks B, double* __restrict__ Q, const double* __restrict__ dtp) {
  step_entry();
  const Dims d = G.d;
  const double dt = *dtp;
  const int s = blockIdx.y;
  const long long nc = nci(d);
  const double *v1 = B.vs1(s), *v2 = B.vs2(s), *v3 = B.vs3(s);
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < nc; c += (long long)gridDim.x * blockDim.x) {
    int i1, i2, i3;
    if (c <= 0xffffffffll) {
      const unsigned u = (unsigned)c, r = u / (unsigned)d.lx1, q = r / (unsigned)d.lx2;
      i1 = (int)(u - r * (unsigned)d.lx1) + 1;
      i2 = (int)(r - q * (unsigned)d.lx2) + 1;
      i3 = (int)q + 1;
    } else {
      i1 = (int)(c % d.lx1) + 1;
      i2 = (int)(c / d.lx1 % d.lx2) + 1;
      i3 = (int)(c / d.lx1 / d.lx2) + 1;
    }
    const long long k = gi(d, i1, i2, i3);
    const double um = v1[k - 1], u0 = v1[k], up = v1[k + 1], n = B.ns(s)[k];
    double q = 0.0;
    if (s < LSP - 1) {  // multifluid.f90:237-268
      const double vl = 0.5 * (um + u0), vr = 0.5 * (u0 + up);
      const double dv = vr - vl;
      const double mn = (dv < 0.0) ? dv : 0.0;
      q = n * c_ms[s] * 0.25 * 9.0 * (mn * mn);
    }
    Q[(long long)s * nc + c] = q;
    // div3D_curv_23 (calculus/div.f90:110-200)
    auto area = [&](const double* a, const double* b, int j1, int j2, int j3) {
      if (UNIT) return 1.0;
      const long long m = cmi(G, j1, j2, j3);
      return __ldg(a + m) * __ldg(b + m);
    };
    double div;
    {
      const double tp = area(G.h2, G.h3, i1 + 1, i2, i3) * (i1 < d.lx1 ? up : u0);
      const double tm = area(G.h2, G.h3, i1 - 1, i2, i3) * (i1 > 1 ? um : u0);
      div = mdiv(tp - tm, __ldg(G.L[0].dxs + i1), __ldg(G.L[0].ydxs + i1));
    }
    if (d.lx2 > 1) {
      const double fp = v2[i2 < d.lx2 ? k + d.s2 : k], fm = v2[i2 > 1 ? k - d.s2 : k];
      const double tp = area(G.h1, G.h3, i1, i2 + 1, i3) * fp, tm = area(G.h1, G.h3, i1, i2 - 1, i3) * fm;
      div = div + mdiv(tp - tm, __ldg(G.L[1].dxs + i2), __ldg(G.L[1].ydxs + i2));
    }
    if (d.lx3 > 1) {
      const long long wrap = G.flagper ? (d.lx3 - 1) * d.s3 : 0;
      const double fp = v3[i3 < d.lx3 ? k + d.s3 : k - wrap], fm = v3[i3 > 1 ? k - d.s3 : k + wrap];
      const double tp = area(G.h1, G.h2, i1, i2, i3 + 1) * fp, tm = area(G.h1, G.h2, i1, i2, i3 - 1) * fm;
      div = div + mdiv(tp - tm, __ldg(G.L[2].dxs + i3), __ldg(G.L[2].ydxs + i3));
    }
    if (!UNIT) {
      const long long m = cmi(G, i1, i2, i3);
      div = mdiv(div, __ldg(G.ha1_0 + m), __ldg(G.yha1_0 + m));
    }
    // compression (multifluid.f90:274-302), then rhoe2T and clean_param(3)
    const double p = B.re(s)[k], gm1 = c_gammas[s] - 1;
    const double half = p - dt / 2 * (p * gm1 + q) * div;
    const double e = p - dt * (half * gm1 + q) * div;
    double T = fmax_f(c_gm1kb[s] * e / fmax_f(n, MINDENSDIV), 100.0);
    if (is_null(G, i1, i2, i3)) T = 100;
    B.Ts(s)[k] = T;
  }
}

// the View of a grid: device metric tables (null on unit-metric grids) and the species
// constants from the same literal expressions as the device constants
gemc::View cmp_view(const gem_grid* g) {
  const GridDev& G = g->dev;
  const Dims& d = G.d;
  gemc::View v;
  v.lx1 = d.lx1;
  v.lx2 = d.lx2;
  v.lx3 = d.lx3;
  v.flagper = G.flagper;
  v.s2 = d.s2;
  v.s3 = d.s3;
  v.ng = d.ng;
  v.c3 = G.c3;
  v.h1 = G.unit ? nullptr : G.h1;
  v.h2 = G.unit ? nullptr : G.h2;
  v.h3 = G.unit ? nullptr : G.h3;
  v.dx1 = G.L[0].dx;
  v.dx2 = G.L[1].dx;
  v.dx3 = G.L[2].dx;
  const double ms[LSP] = {16.0 * AMU, 30.0 * AMU, 28.0 * AMU, 32.0 * AMU, 14.0 * AMU, 1.0 * AMU, 5.485799090e-4 * AMU};
  const double gam[LSP] = {5.0 / 3, 7.0 / 5, 7.0 / 5, 7.0 / 5, 5.0 / 3, 5.0 / 3, 5.0 / 3};
  for (int s = 0; s < LSP; ++s) {
    v.ms[s] = ms[s];
    v.gm1[s] = gam[s] - 1;
  }
  return v;
}

}  // namespace gemk

extern "C" {

int gem_vnricht_artvisc_dev(const gem_grid* g, const double* fluidvars, double* Q, void* stream) {
  if (check_grid(g) || !fluidvars || !Q) return set_err(GEM_EINVAL, "null argument");
  const gemc::View v = gemk::cmp_view(g);
  const long long n = gemc::ncell(v) * LSP;
  step_launch(gemk::kc_artvisc, grid_for(n, 256), 256, 0, S(stream), v, n, fluidvars, fluidvars + LSP * v.ng, Q);
  GEM_LAUNCHED("kc_artvisc");
  return GEM_OK;
}

int gem_rk2_global_boundary_allspec_dev(const gem_grid* g, double* fluidvars, void* stream) {
  if (check_grid(g) || !fluidvars) return set_err(GEM_EINVAL, "null argument");
  const gemc::View v = gemk::cmp_view(g);
  double* vs1 = fluidvars + LSP * v.ng;
  double* vs2 = fluidvars + 2 * LSP * v.ng;
  double* vs3 = fluidvars + 3 * LSP * v.ng;
  cudaStream_t st = S(stream);
  const long long n1 = (long long)(v.lx2 + 4) * (v.lx3 + 4) * LSP;
  step_launch(gemk::kc_rk2_x1, grid_for(n1, 256), 256, 0, st, v, n1, vs1);
  GEM_LAUNCHED("kc_rk2_x1");
  const long long n2 = (long long)(v.lx1 + 4) * (v.lx3 + 4) * LSP * 3;
  step_launch(gemk::kc_rk2_x2, grid_for(n2, 256), 256, 0, st, v, n2, vs1, vs2, vs3);
  GEM_LAUNCHED("kc_rk2_x2");
  if (!v.flagper) {
    const long long n3 = (long long)(v.lx1 + 4) * (v.lx2 + 4) * LSP * 3;
    step_launch(gemk::kc_rk2_x3, grid_for(n3, 256), 256, 0, st, v, n3, vs1, vs2, vs3);
    GEM_LAUNCHED("kc_rk2_x3");
  }
  return GEM_OK;
}

int gem_compression_dev(const gem_grid* g, const double* fluidvars, double* fluidauxvars, const double* Q,
                        const double* dt, void* stream) {
  if (check_grid(g) || !fluidvars || !fluidauxvars || !Q || !dt) return set_err(GEM_EINVAL, "null argument");
  const gemc::View v = gemk::cmp_view(g);
  const long long n = gemc::ncell(v) * LSP;
  step_launch(gemk::kc_compression, grid_for(n, 256), 256, 0, S(stream), v, n, fluidvars + LSP * v.ng,
                                                                  fluidvars + 2 * LSP * v.ng,
                                                                  fluidvars + 3 * LSP * v.ng, Q,
                                                                  fluidauxvars + LSP * v.ng, dt);
  GEM_LAUNCHED("kc_compression");
  return GEM_OK;
}

}  // extern "C"
