// K2: Zalesak-limited horizontal FCT deferred-correction source.
//
// Replaces compute_horizontal_fct_source (orbit/core/fct.py:459-492) with its
// helpers _vanleer_phi (fct.py:235-247), _horizontal_antidiffusive
// (fct.py:256-357, with or without the lateral-inflow ghost field),
// _zalesak_2d (fct.py:381-447) and
// _net_antidiffusive_into_cells (fct.py:360-378).  Pass 1 computes, per cell,
// the Zalesak ratios R+/R- from the four face fluxes touching it and the
// 5-point bounds; pass 2 limits every face with the ratios of its two cells
// and forms d = -div(C A) times rho.  k_fct_source does both on tiles in shared
// memory; the frozen-gain operator keeps a kernel per pass, which recompute the
// face fluxes where they need them (each needs at most four cells along its
// axis).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"

namespace orbit {

namespace {

constexpr double kEarthRadius = 6378137.0;
constexpr double kGravity = 9.80665;
constexpr double kDegToRad = 3.14159265358979323846 / 180.0;

struct FctGeom {
  orbit_met_t g;
  int nz, ny, nx;
  double dt;
  // optional lateral-inflow concentration per vector (c-space, same layout as
  // c): its edge-cell values stand for the cells beyond each lateral edge
  const double* ghost = nullptr;
};


// State weight of a cell: rho = dP / (g Dz) in the concentration form, 1 in the
// pressure form (_state_weights, fct.py:451-456).
__device__ __forceinline__ double rho_at(const orbit_met_t& g, int64_t c) {
  if (g.pressure_form) return 1.0;
  const double dP = g.dP[c], Dz = g.Dz[c];
  return (dP > 0.0 && Dz > 0.0) ? dP / (kGravity * Dz) : 1.0;
}

// Value beyond the edge at edge cell e, in x = c / rho.
__device__ __forceinline__ double ghost_x(const orbit_met_t& g, const double* gh, int64_t e) {
  return gh[e] / rho_at(g, e);
}

__device__ __forceinline__ double vl_phi(double up, double far, double down) {
  const double num = up - far;
  const double den = down - up;
  const bool tiny = fabs(den) < 1e-30;
  double r = num / (tiny ? 1e-30 : den);
  if (tiny) r = fabs(num) < 1e-30 ? 1.0 : 1e6;
  return (r + fabs(r)) / (1.0 + fabs(r));
}

__device__ __forceinline__ double dx_at(const orbit_met_t& g, int j) {
  return kEarthRadius * cos(g.lat[j] * kDegToRad) * g.dlon * kDegToRad;
}

// Face between lo = (k, j, i-1) [x] or (k, j-1, i) [y] and hi = cell index `hi`.
// Returns flux = A * inv and the terrain weights; valid flag.
struct Face {
  double flux, trL, trR, beta, inv;
  bool ok;
};

// gh: the ghost field of this vector or null (fct.py:283-292: with a ghost
// field the far-upwind value beyond an edge is the ghost value of the edge
// cell; without one the face drops to first order there).
__device__ Face x_face(const FctGeom& G, const double* x, int k, int j, int ihi, const double* gh) {
  const orbit_met_t& g = G.g;
  const int nx = G.nx;
  const int64_t base = ((int64_t)k * G.ny + j) * nx;
  const int64_t hi = base + ihi, lo = hi - 1;
  const double cL = x[lo], cR = x[hi];
  const double cLL = ihi - 1 > 0 ? x[lo - 1] : gh ? ghost_x(g, gh, lo) : cL;
  const double cRR = ihi < nx - 1 ? x[hi + 1] : gh ? ghost_x(g, gh, hi) : cR;
  double pL = vl_phi(cL, cLL, cR);
  double pR = vl_phi(cR, cRR, cL);
  if (!gh && ihi - 1 == 0) pL = 0.0;
  if (!gh && ihi == nx - 1) pR = 0.0;
  const double up = G.g.split ? g.u_plus[hi] : fmax(g.u[hi], 0.0);
  const double um = G.g.split ? g.u_minus[hi] : fmax(-g.u[hi], 0.0);
  const double beta = 0.5 * (up * pL + um * pR);
  const double A = beta * (cR - cL);
  const double d = dx_at(g, j);
  const double inv = 1.0 / (d > 0.0 ? d : 1.0);
  const double dl = g.dP[lo], dr = g.dP[hi];
  Face f;
  f.ok = dl > 0.0 && dr > 0.0;
  const double face = 0.5 * (dl + dr);
  f.trL = f.ok ? face / (dl > 0.0 ? dl : 1.0) : 1.0;
  f.trR = f.ok ? face / (dr > 0.0 ? dr : 1.0) : 1.0;
  f.flux = A * inv;
  f.beta = beta;
  f.inv = inv;
  return f;
}

__device__ Face y_face(const FctGeom& G, const double* x, int k, int jhi, int i, const double* gh) {
  const orbit_met_t& g = G.g;
  const int nx = G.nx, ny = G.ny;
  const int64_t hi = ((int64_t)k * ny + jhi) * nx + i, lo = hi - nx;
  const double cS = x[lo], cN = x[hi];
  const double cSS = jhi - 1 > 0 ? x[lo - nx] : gh ? ghost_x(g, gh, lo) : cS;
  const double cNN = jhi < ny - 1 ? x[hi + nx] : gh ? ghost_x(g, gh, hi) : cN;
  double pS = vl_phi(cS, cSS, cN);
  double pN = vl_phi(cN, cNN, cS);
  if (!gh && jhi - 1 == 0) pS = 0.0;
  if (!gh && jhi == ny - 1) pN = 0.0;
  const double vp = G.g.split ? g.v_plus[hi] : fmax(g.v[hi], 0.0);
  const double vm = G.g.split ? g.v_minus[hi] : fmax(-g.v[hi], 0.0);
  const double beta = 0.5 * (vp * pS + vm * pN);
  const double A = beta * (cN - cS);
  const double dy = kEarthRadius * g.dlat * kDegToRad;
  const double inv = 1.0 / (dy > 0.0 ? dy : 1.0);
  const double dxs = dx_at(g, jhi - 1), dxn = dx_at(g, jhi);
  const double dxf = 0.5 * (dxs + dxn);
  const double ds = g.dP[lo], dn = g.dP[hi];
  Face f;
  f.ok = ds > 0.0 && dn > 0.0;
  const double face = 0.5 * (ds + dn);
  f.trL = f.ok ? (dxf / (dxs > 0.0 ? dxs : 1.0)) * (face / (ds > 0.0 ? ds : 1.0)) : 1.0;
  f.trR = f.ok ? (dxf / (dxn > 0.0 ? dxn : 1.0)) * (face / (dn > 0.0 ? dn : 1.0)) : 1.0;
  f.flux = A * inv;
  f.beta = beta;
  f.inv = inv;
  return f;
}

// x = c / rho for all vectors
__global__ void k_fct_x(FctGeom G, const double* c, double* x, int64_t N) {
  const double* cv = c + (int64_t)blockIdx.y * N;
  double* xv = x + (int64_t)blockIdx.y * N;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < N; e += (int64_t)gridDim.x * blockDim.x)
    xv[e] = cv[e] / rho_at(G.g, e);
}

__global__ void k_fct_ratio(FctGeom G, const double* x_all, double* Rp_all, double* Rm_all, int64_t N) {
  const int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= N) return;
  const double* x = x_all + (int64_t)blockIdx.y * N;
  const double* gh = G.ghost ? G.ghost + (int64_t)blockIdx.y * N : nullptr;
  const int nx = G.nx, ny = G.ny;
  const int i = (int)(cell % nx), j = (int)((cell / nx) % ny), k = (int)(cell / ((int64_t)nx * ny));
  const double c = x[cell];
  double cmax = c, cmin = c;
  // beyond an edge: the edge cell's ghost value, or the cell itself (clamped)
  const double out = gh ? ghost_x(G.g, gh, cell) : c;
  const double w = i > 0 ? x[cell - 1] : out, e = i < nx - 1 ? x[cell + 1] : out;
  const double s = j > 0 ? x[cell - nx] : out, n = j < ny - 1 ? x[cell + nx] : out;
  cmax = fmax(fmax(fmax(cmax, w), fmax(e, s)), n);
  cmin = fmin(fmin(fmin(cmin, w), fmin(e, s)), n);
  double Pp = 0.0, Pm = 0.0;
  auto acc = [&](double into) {
    Pp += fmax(into, 0.0);
    Pm += fmax(-into, 0.0);
  };
  if (nx > 1) {
    if (i > 0) {
      Face f = x_face(G, x, k, j, i, gh);
      acc(f.ok ? f.trR * f.flux : 0.0);
    }
    if (i < nx - 1) {
      Face f = x_face(G, x, k, j, i + 1, gh);
      acc(f.ok ? -f.trL * f.flux : 0.0);
    }
  }
  if (ny > 1) {
    if (j > 0) {
      Face f = y_face(G, x, k, j, i, gh);
      acc(f.ok ? f.trR * f.flux : 0.0);
    }
    if (j < ny - 1) {
      Face f = y_face(G, x, k, j + 1, i, gh);
      acc(f.ok ? -f.trL * f.flux : 0.0);
    }
  }
  const double Qp = (cmax - c) / G.dt, Qm = (c - cmin) / G.dt;
  Rp_all[(int64_t)blockIdx.y * N + cell] = Pp > 0.0 ? fmin(1.0, Qp / Pp) : 0.0;
  Rm_all[(int64_t)blockIdx.y * N + cell] = Pm > 0.0 ? fmin(1.0, Qm / Pm) : 0.0;
}

// The whole source in one pass over the field.  Bound by instruction issue (66 % of
// the cycles, DRAM 2 %): double-precision divisions, two for each face's van Leer
// factors, one or two for each cell's ratios, one for x = c / rho, and the index
// arithmetic of each halo cell, face and ratio.  With a kernel per pass every face was computed by
// each of its cells in both passes (eight times four divisions and its geometry,
// a cosine among it, per cell); here a block computes a tile's faces and ratios
// once, in shared memory, and the geometry of its faces once for all the vectors
// that it takes.  12 vectors on the 80x72x15 grid: 228 -> 82 us a bin (3 vectors per block; 6 or 12: 91-96 us; the faces kept in registers instead: 102).
//
// Tiles of 16 x 16 cells of one layer; the ratios reach one cell beyond the
// tile, its faces one more and the field three.  Beyond a lateral edge the field
// holds the edge cell's ghost value, or the edge cell itself.
constexpr int kFT = 16, kFH = kFT + 6, kFR = kFT + 2, kFF = kFT + 3;

// van Leer's factor of the ratio r = num / den, (r + |r|) / (1 + |r|), with one
// division: 2 num / (den + num) where r > 0, else 0 (NaN stays NaN).
__device__ __forceinline__ double vl_factor(double num, double den) {
  if (fabs(den) < 1e-30) return fabs(num) < 1e-30 ? 1.0 : 2e6 / (1.0 + 1e6);
  const bool not_positive = num == 0.0 || (num > 0.0 && den < 0.0) || (num < 0.0 && den > 0.0);
  return not_positive ? 0.0 : (2.0 * num) / (den + num);
}

// weight times that factor; a wind of one sign leaves one weight of a face 0,
// whose division is saved (0 times the numerator keeps its NaN or infinity).
__device__ __forceinline__ double vl_term(double weight, double num, double den) {
  return weight == 0.0 ? weight * num : weight * vl_factor(num, den);
}

__global__ void __launch_bounds__(kFT * kFT) k_fct_source(FctGeom G, const double* c_all, int n_vec, int per_block,
                                                          int limited, double* d_all, int64_t N) {
  __shared__ double xs[kFH * kFH], rho[kFH * kFH];
  // faces [axis]: weights of the two factors (wind / (2 width)), terrain weights
  // of the low and the high cell (0: no face), flux
  __shared__ double up[2][kFR * kFF], um[2][kFR * kFF], tl[2][kFR * kFF], th[2][kFR * kFF], fl[2][kFR * kFF];
  __shared__ double rp[kFR * kFR], rm[kFR * kFR];
  __shared__ double dxr[kFT + 4];
  const orbit_met_t& g = G.g;
  const int nx = G.nx, ny = G.ny, tid = threadIdx.x;
  const int tiles_x = (nx + kFT - 1) / kFT, tiles = tiles_x * ((ny + kFT - 1) / kFT);
  const int tile = blockIdx.x % tiles, k = blockIdx.x / tiles;
  const int i0 = (tile % tiles_x) * kFT, j0 = (tile / tiles_x) * kFT;
  const int64_t layer = (int64_t)k * ny * nx;
  for (int q = tid; q < kFT + 4; q += kFT * kFT) {
    const int j = min(max(j0 - 2 + q, 0), ny - 1);
    dxr[q] = dx_at(g, j);
  }
  for (int q = tid; q < kFH * kFH; q += kFT * kFT) {
    const int i = min(max(i0 - 3 + q % kFH, 0), nx - 1), j = min(max(j0 - 3 + q / kFH, 0), ny - 1);
    rho[q] = rho_at(g, layer + (int64_t)j * nx + i);
  }
  __syncthreads();
  // x-faces: face i between cells i - 1 and i, rows j0 - 1 ..; y-faces: face j
  // between rows j - 1 and j, columns i0 - 1 ..
  for (int q = tid; q < 2 * kFR * kFF; q += kFT * kFT) {
    const int axis = q >= kFR * kFF, e = q - axis * kFR * kFF;
    const int fast = e % (axis ? kFR : kFF), slow = e / (axis ? kFR : kFF);
    const int i = i0 - 1 + fast, j = j0 - 1 + slow;
    double wp = 0.0, wm = 0.0, wl = 0.0, wh = 0.0;
    if (i >= 0 && i < nx && j >= 0 && j < ny && (axis ? j : i) > 0) {
      const int64_t hi = layer + (int64_t)j * nx + i, lo = hi - (axis ? nx : 1);
      const double pl = g.dP[lo], ph = g.dP[hi];
      if (pl > 0.0 && ph > 0.0) {
        const double face = 0.5 * (pl + ph);
        wl = face / pl;
        wh = face / ph;
        double width;
        if (axis) {
          width = kEarthRadius * g.dlat * kDegToRad;
          const double ds = dxr[j - 1 - j0 + 2], dn = dxr[j - j0 + 2], mid = 0.5 * (ds + dn);
          wl *= mid / (ds > 0.0 ? ds : 1.0);
          wh *= mid / (dn > 0.0 ? dn : 1.0);
        } else {
          width = dxr[j - j0 + 2];
        }
        const double inv = 0.5 / (width > 0.0 ? width : 1.0);
        const double* net = axis ? g.v : g.u;
        const int at = axis ? j : i, last = axis ? ny - 1 : nx - 1;
        wp = (g.split ? (axis ? g.v_plus : g.u_plus)[hi] : fmax(net[hi], 0.0)) * inv;
        wm = (g.split ? (axis ? g.v_minus : g.u_minus)[hi] : fmax(-net[hi], 0.0)) * inv;
        // without a ghost field the faces next to an edge are first order there
        if (!G.ghost && at == 1) wp = 0.0;
        if (!G.ghost && at == last) wm = 0.0;
      }
    }
    up[axis][e] = wp;
    um[axis][e] = wm;
    tl[axis][e] = wl;
    th[axis][e] = wh;
  }
  const int v1 = min(n_vec, ((int)blockIdx.y + 1) * per_block);
  for (int v = blockIdx.y * per_block; v < v1; ++v) {
    const double* c = c_all + (int64_t)v * N + layer;
    const double* gh = G.ghost ? G.ghost + (int64_t)v * N + layer : nullptr;
    __syncthreads();
    for (int q = tid; q < kFH * kFH; q += kFT * kFT) {
      const int i = i0 - 3 + q % kFH, j = j0 - 3 + q / kFH;
      const int ic = min(max(i, 0), nx - 1), jc = min(max(j, 0), ny - 1);
      const double* src = gh && (i != ic || j != jc) ? gh : c;
      xs[q] = src[(int64_t)jc * nx + ic] / rho[q];
    }
    __syncthreads();
    for (int q = tid; q < 2 * kFR * kFF; q += kFT * kFT) {
      const int axis = q >= kFR * kFF, e = q - axis * kFR * kFF;
      double f = 0.0;
      if (th[axis][e] != 0.0) {
        const int at = (2 + e / (axis ? kFR : kFF)) * kFH + 2 + e % (axis ? kFR : kFF), step = axis ? kFH : 1;
        const double ll = xs[at - 2 * step], l = xs[at - step], h = xs[at], hh = xs[at + step];
        const double jump = h - l;
        f = (vl_term(up[axis][e], l - ll, jump) + vl_term(um[axis][e], h - hh, -jump)) * jump;
      }
      fl[axis][e] = f;
    }
    __syncthreads();
    if (limited) {
      for (int q = tid; q < kFR * kFR; q += kFT * kFT) {
        const int ii = q % kFR, jj = q / kFR, i = i0 - 1 + ii, j = j0 - 1 + jj;
        double p = 0.0, m = 0.0;
        if (i >= 0 && i < nx && j >= 0 && j < ny) {
          const int xf = jj * kFF + ii, yf = jj * kFR + ii, at = (jj + 2) * kFH + ii + 2;
          const double into[4] = {th[0][xf] * fl[0][xf], -tl[0][xf + 1] * fl[0][xf + 1], th[1][yf] * fl[1][yf],
                                  -tl[1][yf + kFR] * fl[1][yf + kFR]};
          double gain = 0.0, loss = 0.0;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            gain += fmax(into[e], 0.0);
            loss += fmax(-into[e], 0.0);
          }
          const double x = xs[at], w = xs[at - 1], e = xs[at + 1], s = xs[at - kFH], n = xs[at + kFH];
          const double top = fmax(fmax(fmax(x, w), fmax(e, s)), n), low = fmin(fmin(fmin(x, w), fmin(e, s)), n);
          if (gain > 0.0) p = fmin(1.0, (top - x) / (G.dt * gain));
          if (loss > 0.0) m = fmin(1.0, (x - low) / (G.dt * loss));
        }
        rp[q] = p;
        rm[q] = m;
      }
      __syncthreads();
    }
    const int ii = tid % kFT, jj = tid / kFT, i = i0 + ii, j = j0 + jj;
    if (i < nx && j < ny) {
      const int cell = (jj + 1) * kFR + ii + 1, xf = (jj + 1) * kFF + ii + 1, yf = (jj + 1) * kFR + ii + 1;
      // limited flux of a face between the cells lo and hi of the ratios
      auto flux = [&](int axis, int f, int lo, int hi) {
        const double a = fl[axis][f];
        if (!limited) return a;
        const double q = th[axis][f] * a >= 0.0 ? fmin(rp[hi], rm[lo]) : fmin(rm[hi], rp[lo]);
        return fmin(fmax(q, 0.0), 1.0) * a;
      };
      double d = th[0][xf] * flux(0, xf, cell - 1, cell);
      d -= tl[0][xf + 1] * flux(0, xf + 1, cell, cell + 1);
      d += th[1][yf] * flux(1, yf, cell - kFR, cell);
      d -= tl[1][yf + kFR] * flux(1, yf + kFR, cell, cell + kFR);
      d_all[(int64_t)v * N + layer + (int64_t)j * nx + i] = d * rho[(jj + 3) * kFH + ii + 3];
    }
  }
}

// Frozen-gain linearisation of the limited flux (assemble_fct_linear_operator,
// orbit/core/fct.py:495-572): each face's gain w = C beta / dx (C the Zalesak
// coefficient and beta the van Leer reconstruction factor of the baseline),
// distributed with the terrain weights so that L_AD x = -div(w (x_R - x_L)),
// then the similarity diag(rho) L diag(1/rho).  Output: the 7-point stencil
// layout of the transport blocks (centre, W, E, S, N, below, above; the
// vertical entries are zero), so L_low + L_AD is a plain stencil sum.
__global__ void k_fct_linop(FctGeom G, const double* x_all, const double* Rp_all, const double* Rm_all,
                            double* st_all, int64_t N) {
  const int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= N) return;
  const double* x = x_all + (int64_t)blockIdx.y * N;
  const double* Rp = Rp_all + (int64_t)blockIdx.y * N;
  const double* Rm = Rm_all + (int64_t)blockIdx.y * N;
  double* st = st_all + (int64_t)blockIdx.y * 7 * N;
  const double* gh = nullptr;  // the frozen operator has no ghost field (fct.py:495-572)
  const int nx = G.nx, ny = G.ny;
  const int i = (int)(cell % nx), j = (int)((cell / nx) % ny), k = (int)(cell / ((int64_t)nx * ny));
  auto gain = [&](const Face& f, int64_t lo, int64_t hi) {
    if (!f.ok) return 0.0;
    const double into_hi = f.trR * f.flux;
    const double C = into_hi >= 0.0 ? fmin(Rp[hi], Rm[lo]) : fmin(Rm[hi], Rp[lo]);
    return fmin(fmax(C, 0.0), 1.0) * f.beta * f.inv;
  };
  const double rp = rho_at(G.g, cell);
  double cen = 0.0, w = 0.0, e = 0.0, s = 0.0, n = 0.0;
  if (nx > 1) {
    if (i > 0) {  // west face: this cell is its high side
      const Face f = x_face(G, x, k, j, i, gh);
      const double wr = f.trR * gain(f, cell - 1, cell);
      cen -= wr;
      w = wr * rp / rho_at(G.g, cell - 1);
    }
    if (i < nx - 1) {  // east face: low side
      const Face f = x_face(G, x, k, j, i + 1, gh);
      const double wl = f.trL * gain(f, cell, cell + 1);
      cen -= wl;
      e = wl * rp / rho_at(G.g, cell + 1);
    }
  }
  if (ny > 1) {
    if (j > 0) {
      const Face f = y_face(G, x, k, j, i, gh);
      const double wr = f.trR * gain(f, cell - nx, cell);
      cen -= wr;
      s = wr * rp / rho_at(G.g, cell - nx);
    }
    if (j < ny - 1) {
      const Face f = y_face(G, x, k, j + 1, i, gh);
      const double wl = f.trL * gain(f, cell, cell + nx);
      cen -= wl;
      n = wl * rp / rho_at(G.g, cell + nx);
    }
  }
  st[cell] = cen;
  st[N + cell] = w;
  st[2 * N + cell] = e;
  st[3 * N + cell] = s;
  st[4 * N + cell] = n;
  st[5 * N + cell] = 0.0;
  st[6 * N + cell] = 0.0;
}

}  // namespace

// SMs of the current device, asked for once per ordinal (0.4 us of the 16 that a
// call takes on the smallest domains).
static cudaError_t sm_count(int* sms) {
  static std::atomic<int> known[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::atomic<int>* k = dev < 64 ? &known[dev] : nullptr;
  *sms = k ? k->load(std::memory_order_relaxed) : 0;
  if (*sms > 0) return cudaSuccess;
  e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess && k) k->store(*sms, std::memory_order_relaxed);
  return e;
}

// Whether the source may not be written while c is read (the caller then
// passes a copy of c).
bool fct_overlaps(const double* c, const double* d, int64_t n) { return c < d + n && d < c + n; }

int fct_source(int nz, int ny, int nx, const orbit_met_t* met, int n_vec, const double* c, double dt,
               int limited, double* d, cudaStream_t st, const double* ghost = nullptr) {
  const int64_t N = (int64_t)nz * ny * nx;
  FctGeom G{*met, nz, ny, nx, dt, ghost};
  const int tiles = ((nx + kFT - 1) / kFT) * ((ny + kFT - 1) / kFT);
  int sms = 0;
  ORBIT_CUDA_TRY(sm_count(&sms));
  // as many vectors per block (sharing its geometry) as leave about eight blocks
  // per SM
  const int64_t blocks = (int64_t)tiles * nz;
  const int groups = (int)std::max<int64_t>(1, std::min<int64_t>(n_vec, (8 * sms + blocks - 1) / blocks));
  const int per = (n_vec + groups - 1) / groups;
  k_fct_source<<<dim3((unsigned)blocks, (n_vec + per - 1) / per), kFT * kFT, 0, st>>>(G, c, n_vec, per, limited, d, N);
  note_launch();
  ORBIT_CUDA_TRY(cudaGetLastError());
  return ORBIT_OK;
}

int fct_linear_operator(int nz, int ny, int nx, const orbit_met_t* met, int n_vec, const double* c, double dt,
                        double* stencil, double* scratch, cudaStream_t st) {
  const int64_t N = (int64_t)nz * ny * nx;
  FctGeom G{*met, nz, ny, nx, dt};
  double* x = scratch;
  double* Rp = scratch + (int64_t)n_vec * N;
  double* Rm = Rp + (int64_t)n_vec * N;
  dim3 g((unsigned)((N + 127) / 128), n_vec);
  k_fct_x<<<g, 128, 0, st>>>(G, c, x, N);
  note_launch();
  k_fct_ratio<<<g, 128, 0, st>>>(G, x, Rp, Rm, N);
  note_launch();
  k_fct_linop<<<g, 128, 0, st>>>(G, x, Rp, Rm, stencil, N);
  note_launch();
  ORBIT_CUDA_TRY(cudaGetLastError());
  return ORBIT_OK;
}

}  // namespace orbit

// ---------------------------------------------------------------------------
// FCT source without any device allocation.
//
// Some callers cannot allocate device memory when they apply the correction:
// a host model that hands this library a fixed device-memory budget and owns
// every other byte through its own pool, or a time-stepping loop that must not
// stall on the implicit synchronization cudaFree may cause.  The source needs
// no scratch; only where d overlaps c is c copied first, here to one file-scope
// device array in place of a stream-ordered allocation.  Every GPU that loads
// the library holds the array (kFctNoAllocMaxCells doubles, 8 MiB) until the
// process exits.
// ---------------------------------------------------------------------------
#include <mutex>

namespace orbit {

// n_vec * nz * ny * nx may not exceed this (e.g. 12 vectors of 86,400 cells).
constexpr int64_t kFctNoAllocMaxCells = int64_t(1) << 20;

static __device__ __align__(256) double g_fct_scratch[kFctNoAllocMaxCells];

namespace {
std::mutex g_fct_scratch_mu;
constexpr int kMaxDevices = 64;
double* g_fct_scratch_ptr[kMaxDevices] = {nullptr};
}  // namespace

int fct_source_noalloc(int nz, int ny, int nx, const orbit_met_t* met, int n_vec, const double* c,
                       double dt, int limited, double* d, cudaStream_t st) {
  const int64_t cells = (int64_t)nz * ny * nx * n_vec;
  if (cells > kFctNoAllocMaxCells) {
    set_last_error("orbit_fct_source_noalloc: n_vec*nz*ny*nx = " + std::to_string(cells) +
                   " exceeds the static scratch limit of " + std::to_string(kFctNoAllocMaxCells) +
                   " cells; split the vectors over several calls or use orbit_fct_source");
    return ORBIT_ERR_ARG;
  }
  int dev = 0;
  ORBIT_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) {
    set_last_error("orbit_fct_source_noalloc: device ordinal out of range");
    return ORBIT_ERR_ARG;
  }
  double* scratch = nullptr;
  {
    // The array's name is only a host-side stand-in for the symbol; its device
    // address is looked up once per device, with that device current.  The
    // cached address belongs to the device's current primary context: after a
    // cudaDeviceReset the module may load elsewhere, so the entry point must
    // not be called after one.
    std::lock_guard<std::mutex> lk(g_fct_scratch_mu);
    if (!g_fct_scratch_ptr[dev]) {
      void* p = nullptr;
      ORBIT_CUDA_TRY(cudaGetSymbolAddress(&p, g_fct_scratch));
      g_fct_scratch_ptr[dev] = static_cast<double*>(p);
    }
    scratch = g_fct_scratch_ptr[dev];
  }
  if (fct_overlaps(c, d, cells)) {
    ORBIT_CUDA_TRY(cudaMemcpyAsync(scratch, c, sizeof(double) * cells, cudaMemcpyDeviceToDevice, st));
    c = scratch;
  }
  return fct_source(nz, ny, nx, met, n_vec, c, dt, limited, d, st);
}

}  // namespace orbit
