// Hydrodynamic step of FLUXOS-OVERLAND for sm_100a, FP64 and FP32.
//
// One launch of k_hydro_* performs, tile by tile (31 x BY-1 cells):
//   * the snowmelt forcing of common.cpp:210-262 (add_meteo), including the
//     solute dilution, applied on the fly to every cell the tile reads;
//   * Loop 1 of hydrodynamics_calc.cpp:53-73 (depth, wet flag, wet time);
//   * Loop 2 (:76-90): the east and north face fluxes of solver_wet
//     (solver_wetdomain.cpp:27-342) and solver_dry (solver_drydomain.cpp:27-194)
//     for the tile and its west/south halo, each face once, by one thread,
//     and used by both cells that share it;
//   * Loop 3 (:93-120) and Loop 4 (:123-154): divergence and update;
//   * the optional Manning friction extension;
//   * the per-cell part of the NEXT step's Courant scan (main.cpp:300-323),
//     kept per thread and reduced once per block with one atomic.
// k_finalize then turns the reduction into the next dt and advances the
// clock on the device, so a run of steps needs no host round trip.
//
// Every expression keeps the reference's operand types and evaluation order
// (the library is built with --fmad=false), so results match the CPU
// reference bit for bit except where noted at fx_pow15.
#include <cuda_runtime.h>

#include <type_traits>
#include <vector>

#include "fx_common.cuh"
#include "fx_div.cuh"

namespace fx {

// A block of 32 x BY threads owns a tile of 31 rows (irow) x BY-1 columns
// (icol): with its west row and south column of halo faces the tile has
// exactly 32 x BY face-flux cells, one per thread, so the flux phase runs in
// a single wave and no warp waits at the barrier for a second round. BY (the
// tile rows along icol: 4, 8 or 16) is chosen per domain or batch, by the
// autotuner (fx_autotune) or fx_set_option("tile_rows").
constexpr int BX = 32;          // threads along irow: one warp
constexpr int TX = 31;          // owned rows
constexpr int SX = TX + 3;      // stencil rows irow0-2..irow0+TX
constexpr int FXN = TX + 1;     // flux rows irow0-1..irow0+TX-1
template <int BY>
struct Tile {
  static constexpr int TY = BY - 1;            // owned columns
  static constexpr int SY = TY + 3;            // stencil columns icol0-2..icol0+TY
  static constexpr int FYN = TY + 1;           // flux columns icol0-1..icol0+TY-1
  static constexpr int NSTEN = SX * SY, NFLUX = FXN * FYN, NTHREADS = BX * BY;
  static_assert(NFLUX == NTHREADS, "one face-flux cell per thread");
};

// stencil cell classes
constexpr unsigned char C_DRY = 1;   // Loop-1 ldry == 1 (interior cells only)
constexpr unsigned char C_WALL = 2;  // innerNeumannBCWeir == 1
constexpr unsigned char C_INT = 4;   // interior cell (1..NROWS, 1..NCOLS)

template <int BY, bool STAGED>
struct HydroSmem64 {
  static constexpr int NSTEN = Tile<BY>::NSTEN, NFLUX = Tile<BY>::NFLUX, NW = Tile<BY>::NTHREADS / 32;
  double budget[2 * NW];
  double z[NSTEN], qx[NSTEN], qy[NSTEN];
  double mi[STAGED ? NSTEN : 1];  // the step's melt depth, of the cells that take it
  double zb[STAGED ? 1 : NSTEN];  // a staged tile reads the bed where TMA left it
  // cell velocities q / max(h, hdry, ks) of the stencil, formed once per
  // cell for the wet solver's shear terms (the same expression and operands
  // the solver divides for each face, so the same values); kept for tiles
  // up to 8 rows, the largest tile's state stays within 48 KB
  static constexpr bool VEL = BY <= 8;
  double u[VEL ? NSTEN : 1], v[VEL ? NSTEN : 1];
  double f[3][NFLUX];  // north face fluxes
  unsigned char cls[NSTEN];
  double red_dt[NW], red_h[NW];
};

// sqrt(h)^3 = pow(h, 1.5) for h >= 0, correctly rounded: s = sqrt(h) is
// refined to a double-double with its exact residual (fma(-s, s, h)), and the
// product h * (s + s_lo) is formed with an exact fma error term (Dekker/Knuth
// error-free transformations; Muller et al., Handbook of Floating-Point
// Arithmetic, ch. 4-5). glibc's pow differs from the correctly rounded value
// in about 1e-3 of arguments, so the edge weir flux may differ from the CPU
// reference by one unit in the last place there.
__device__ __forceinline__ double fx_pow15(double h) {
  if (h == 0.0) return 0.0;
  double s = sqrt(h);
  double e = fma(-s, s, h);
  double slo = e / (2.0 * s);
  double p = h * s;
  double pe = fma(h, s, -p);
  return p + (pe + h * slo);
}

// x / dxy of the FP64 state. Out of line for the same reason; at a spacing of
// 3, 1000 x 700 cells took 131 us a step with plain divisions, 112 us so.
__device__ __noinline__ double over_dxy(double x, double dxy, double inv) { return over(x, dxy, inv); }
__device__ __forceinline__ double div_dxy(const fx_dev& d, double x) {
  return d.dxy_pow2 ? x * d.inv_dxy : over_dxy(x, d.dxy, d.inv_dxy);
}
constexpr double DAY_MM = 1000. * 3600. * 24.;  // mm/day to m/s

// max(x, c) for a c that is a number, by a compare and a select: the bits of
// fmax (an x that is no number gives c, and max(-0, 0) is 0), which takes a
// few instructions more.
__device__ __forceinline__ double at_least(double x, double c) { return x > c ? x : c; }
__device__ __forceinline__ double max0(double x) { return at_least(x, 0.0); }

// The edge weir's flux (solver_wetdomain.cpp:302-307): out of line, only edge
// cells of the domain have one.
__device__ __noinline__ double edge_weir(double volrat, double sqrt_g, double hp) {
  return fmin(volrat, sqrt_g * fx_pow15(fmax(hp, 0.0)));
}

// Cube root of x >= 0 by Newton iteration on the mantissa, using only
// frexp/ldexp and IEEE +,-,*,/, so the oracle's C (ox_cbrt) computes the
// same bits. Used by the Manning extension only.
__device__ __forceinline__ double fx_cbrt(double x) {
  if (!(x > 0.0) || isinf(x)) return x;
  int e;
  double m = frexp(x, &e);
  int r = e % 3;
  if (r < 0) r += 3;
  m = ldexp(m, r);
  e -= r;
  double y = 0.5 + 0.35 * m;
#pragma unroll 1
  for (int i = 0; i < 7; ++i) {
    y = y - (y * y * y - m) / (3.0 * y * y);
  }
  return ldexp(y, e / 3);
}

// The stencil cells a thread reads, in two passes without an integer division: warp
// ly reads column ly, then warps 0 and 1 the last two columns and the others
// the two rows beyond the warp's 32. False: none in this pass.
template <int BY>
__device__ __forceinline__ bool stencil_cell(int pass, int lx, int ly, int& sr, int& sc) {
  sr = lx;
  sc = ly;
  if (pass == 0) return true;
  if (ly < 2) {
    sc = BY + ly;
    return true;
  }
  const int e = (ly - 2) * BX + lx;
  sr = BX + (e & 1);
  sc = e >> 1;
  return e < 2 * Tile<BY>::SY;
}

__device__ __forceinline__ int sidx(int sr, int sc) { return sc * SX + sr; }
// The bed of the tile's stencil: columns LD doubles apart.
template <int LD>
struct Bed {
  const double* p;
  __device__ __forceinline__ double operator()(int sr, int sc) const { return p[sc * LD + sr]; }
};

// solver_wetdomain.cpp:27-342 for the flux cell at stencil (sr, sc).
template <class SM, class BED>
__device__ void solver_wet(const fx_dev& d, const SM& S, const BED& bed, int sr, int sc, int irow, int icol,
                           Over dt, double out[6]) {
  const double hdryl = d.hdry, gaccl = d.gaccl;
  const int P = sidx(sr, sc), W = sidx(sr - 1, sc), E = sidx(sr + 1, sc);
  const int Sx = sidx(sr, sc - 1), N = sidx(sr, sc + 1);
  const int ES = sidx(sr + 1, sc - 1), EN = sidx(sr + 1, sc + 1), WN = sidx(sr - 1, sc + 1);
  auto ksat = [&](int k) { return (S.cls[k] & C_INT) ? d.ks : 0.0; };
  auto hat = [&](int r, int q) { return max0(S.z[sidx(r, q)] - bed(r, q)); };
  const double nueml = d.nueml, cvdefl = d.cvdefl;
  const unsigned dx = d.dxy_u, dy = d.dxy_u;
  bool lroe = true;
  double volrat = d.volrat_mode == 0 ? __longlong_as_double(0x7ff0000000000000LL) : 0.0;

  const bool lde_dry = S.cls[E] & C_DRY;
  const bool ldn_dry = S.cls[N] & C_DRY;

  const double zbw = bed(sr - 1, sc), zbp = bed(sr, sc), zbe = bed(sr + 1, sc);
  const double zbs = bed(sr, sc - 1), zbn = bed(sr, sc + 1);
  const double zw = S.z[W], zp = S.z[P], ze = S.z[E], zs = S.z[Sx], zn = S.z[N];
  double qp = S.qx[P], qe = S.qx[E], qn = S.qx[N];
  double rw = S.qy[W], rp = S.qy[P], re = S.qy[E], rn = S.qy[N];

  const double zbpe = .5 * (zbe + zbp);
  const double zbpn = .5 * (zbn + zbp);
  const double hp = max0(zp - zbp);
  const double hw = max0(zw - zbw);
  double he = max0(ze - zbe);
  const double hs = max0(zs - zbs);
  double hn = max0(zn - zbn);

  double hme = .5 * (hp + he);
  double qme = .5 * (qp + qe);
  double rme = .5 * (rp + re);
  double hmn = .5 * (hp + hn);
  double qmn = .5 * (qp + qn);
  double rmn = .5 * (rp + rn);

  double dze = ze - zp;
  const double dqe = qe - qp;
  const double dre = re - rp;
  double dzn = zn - zp;
  const double drn = rn - rp;
  const double dqn = qn - qp;

  if (lde_dry) {  // :121-147
    hme = max0(zp - zbpe);
    he = 0.0;
    qe = 0.0;
    re = 0.0;
    if (hme > hdryl) {
      if (ze >= zp) {
        qme = 0.0;
        rme = 0.0;
      } else {
        dze = fmin(fabs(dze), hme);
        qme = 0.296 * dze * sqrt(gaccl * dze);
        volrat = dt.of(0.5 * dx * hp);
        qme = fmin(qme, volrat);
        rme = 0.0;
      }
    } else {
      qme = 0.0;
      rme = 0.0;
      hme = 0.0;
    }
    lroe = false;
  }
  if (ldn_dry) {  // :148-175
    hmn = max0(zp - zbpn);
    hn = 0.0;
    qn = 0.0;
    rn = 0.0;
    if (hmn > hdryl) {
      if (zn >= zp) {
        qmn = 0.0;
        rmn = 0.0;
      } else {
        dzn = fmin(fabs(dzn), hmn);
        rmn = 0.296 * dzn * sqrt(gaccl * dzn);
        qmn = 0.0;
        volrat = dt.of(0.5 * dy * hp);
        rmn = fmin(rmn, volrat);
      }
    } else {
      qmn = 0.0;
      rmn = 0.0;
      hmn = 0.0;
    }
    lroe = false;
  }

  // :177-203 turbulent stress; the shear velocity us is identically 0 in
  // the reference (set to 0 by initiate.cpp:176 and both update loops).
  const double cme = sqrt(gaccl * hme);
  const double cmn = sqrt(gaccl * hmn);
  const Over he_(at_least(hme, hdryl)), hn_(at_least(hmn, hdryl));
  const double ume = he_.of(qme);
  const double vme = he_.of(rme);
  const double umn = hn_.of(qmn);
  const double vmn = hn_.of(rmn);
  const double cnp = cvdefl * 0.0 * hp + nueml;
  const double cne = cvdefl * 0.0 * he + nueml;
  const double cnn = cvdefl * 0.0 * hn + nueml;
  const double hne = .5 * (cnp + cne) * sqrt(hp * he);
  const double hnn = .5 * (cnp + cnn) * sqrt(hp * hn);

  // neighbour velocities from the stencil (solver_wetdomain.cpp: each is
  // q / max(max(h, hdry), ks) of its cell; a dry neighbour's discharge is 0,
  // so its velocity is 0 whatever depth the division uses)
  double up, vp, un, us0, use0, une, ve, vw, vwn, ven;
  if constexpr (SM::VEL) {
    up = S.u[P];
    vp = S.v[P];
    un = S.u[N];
    us0 = S.u[Sx];
    use0 = S.u[ES];
    une = S.u[EN];
    ve = S.v[E];
    vw = S.v[W];
    vwn = S.v[WN];
    ven = S.v[EN];
  } else {
    const Over hp_(fmax(fmax(hdryl, hp), ksat(P)));
    up = hp_.of(qp);
    vp = hp_.of(rp);
    un = qn / fmax(fmax(hn, hdryl), ksat(N));
    us0 = S.qx[Sx] / fmax(fmax(hs, hdryl), ksat(Sx));
    use0 = S.qx[ES] / fmax(fmax(hat(sr + 1, sc - 1), hdryl), ksat(ES));
    une = S.qx[EN] / fmax(fmax(hat(sr + 1, sc + 1), hdryl), ksat(EN));
    ve = re / fmax(fmax(he, hdryl), ksat(E));
    vw = rw / fmax(fmax(hw, hdryl), ksat(W));
    vwn = S.qy[WN] / fmax(fmax(hat(sr - 1, sc + 1), hdryl), ksat(WN));
    ven = S.qy[EN] / fmax(fmax(hat(sr + 1, sc + 1), hdryl), ksat(EN));
  }

  const double txye = hne * (div_dxy(d, ve - vp) + div_dxy(d, .25 * (un + une - us0 - use0)));
  const double txyn = hnn * (div_dxy(d, un - up) + div_dxy(d, .25 * (ve + ven - vw - vwn)));

  const double fe1c = qme;
  const double fe2c = qme * ume;
  const double fe3c = qme * vme - txye;
  const double fn1c = rmn;
  const double fn2c = rmn * umn - txyn;
  const double fn3c = rmn * vmn;

  double fe1r, fe2r, fe3r, fn1r, fn2r, fn3r;
  if (lroe) {  // :213-285
    double cc;
    if (hme > d.hdry) {
      double dzea = fabs(dze);
      if (dzea > 0.5 * hme) {
        double dhea = fabs(he - hp);
        dzea = fmin(dzea, dhea);
        dze = copysign(dzea, dze);
      }
      cc = .25 / cme;
    } else {
      cc = 0.0;
    }
    double c1 = ume, c2 = ume + cme, c3 = ume - cme;
    double c1a = fabs(c1), c2a = fabs(c2), c3a = fabs(c3);
    double a11 = c2 * c3a - c2a * c3;
    double a12 = c2a - c3a;
    double a21 = c2 * c3 * (c3a - c2a);
    double a22 = c2a * c2 - c3a * c3;
    double a31 = vme * (c2 * c3a - 2. * cme * c1a - c2a * c3);
    double a32 = vme * (c2a - c3a);
    double a33 = 2. * cme * c1a;
    fe1r = -(a11 * dze + a12 * dqe) * cc;
    fe2r = -(a21 * dze + a22 * dqe) * cc;
    fe3r = -(a31 * dze + a32 * dqe + a33 * dre) * cc;

    if (hmn > d.hdry) {  // this cell is wet (ldp == 0)
      double dzna = fabs(dzn);
      double dhna = fabs(hn - hp);
      dzna = fmin(dzna, dhna);
      dzn = copysign(dzna, dzn);
      cc = .25 / cmn;
    } else {
      cc = 0.0;
    }
    c1 = vmn;
    c2 = vmn + cmn;
    c3 = vmn - cmn;
    c1a = fabs(c1);
    c2a = fabs(c2);
    c3a = fabs(c3);
    a11 = c2 * c3a - c2a * c3;
    double a13 = c2a - c3a;
    a21 = umn * (c2 * c3a - 2. * cmn * c1a - c2a * c3);
    a22 = 2. * cmn * c1a;
    double a23 = umn * (c2a - c3a);
    a31 = c2 * c3 * (c3a - c2a);
    a33 = c2a * c2 - c3a * c3;
    fn1r = -(a11 * dzn + a13 * drn) * cc;
    fn2r = -(a21 * dzn + a22 * dqn + a23 * drn) * cc;
    fn3r = -(a31 * dzn + a33 * drn) * cc;
  } else {
    fe1r = fe2r = fe3r = fn1r = fn2r = fn3r = 0.0;
  }

  const double fe2p = .5 * gaccl * (hme * hme);
  const double fn3p = .5 * gaccl * (hmn * hmn);
  double fe1 = fe1c + fe1r;
  const double fe2 = fe2c + fe2r + fe2p;
  const double fe3 = fe3c + fe3r;
  double fn1 = fn1c + fn1r;
  const double fn2 = fn2c + fn2r;
  const double fn3 = fn3c + fn3r + fn3p;

  if (icol == 1 || icol == d.nc) fn1 = edge_weir(volrat, d.sqrt_gaccl, hp);
  if (irow == 1 || irow == d.nr) fe1 = edge_weir(volrat, d.sqrt_gaccl, hp);

  const double volpot = d.arbase * hp;
  volrat = dt.of(volpot);
  if (volrat > 0.0) {  // :309-332
    if ((fe1 > 0.0) & (fn1 > 0.0)) {
      if (fe1 * dy + fn1 * dx > volrat) {
        double cf = fn1 * dx / (fe1 * dy + fn1 * dx);
        fe1 = div_dxy(d, (1. - cf) * volrat);
        fn1 = div_dxy(d, cf * volrat);
      }
    } else if (fe1 > 0.0) {
      fe1 = div_dxy(d, fmin(fe1 * dy, volrat));
    } else if (fn1 > 0.0) {
      fn1 = div_dxy(d, fmin(fn1 * dx, volrat));
    }
  } else {
    fe1 = 0.0;
    fn1 = 0.0;
  }
  out[0] = fe1;
  out[1] = fe2;
  out[2] = fe3;
  out[3] = fn1;
  out[4] = fn2;
  out[5] = fn3;
}

// solver_drydomain.cpp:78-194 (the cell is dry and has a wet neighbour).
template <class SM, class BED>
__device__ void solver_dry(const fx_dev& d, const SM& S, const BED& bed, int sr, int sc, int irow, int icol,
                           double dtl, double out[6]) {
  const int P = sidx(sr, sc), E = sidx(sr + 1, sc), N = sidx(sr, sc + 1);
  const double gaccl = d.gaccl;
  double volrat = d.volrat_mode == 0 ? __longlong_as_double(0x7ff0000000000000LL) : 0.0;
  const bool lde_dry = S.cls[E] & C_DRY, ldn_dry = S.cls[N] & C_DRY;
  const double zbp = bed(sr, sc), zbe = bed(sr + 1, sc), zbn = bed(sr, sc + 1);
  const double zp = S.z[P], ze = S.z[E], zn = S.z[N];
  const double hp = fmax(0.0, zp - zp);  // :85 reads z - z
  const double he = fmax(0.0, ze - zbe);
  const double hn = fmax(0.0, zn - zbn);
  const double zbpe = .5 * (zbe + zbp);
  const double zbpn = .5 * (zbn + zbp);
  double dze = ze - zp, dzn = zn - zp;
  double fe1 = 0.0, fe2 = 0.0, fe3 = 0.0, fn1 = 0.0, fn2 = 0.0, fn3 = 0.0;
  if (!lde_dry) {  // :115-145
    double hme = fmax(0.0, ze - zbpe);
    if (hme > d.hdry) {
      if (ze <= zp) {
        double fe2p = .5 * gaccl * hme * hme;
        fe1 = 0.0;
        fe2 = fe2p;
        fe3 = 0.0;
      } else {
        dze = fmin(fabs(dze), hme);
        double qme = 0.296 * dze * sqrt(gaccl * dze);
        hme = 0.444 * dze;
        volrat = d.dxy * he / dtl;
        qme = -fmin(qme, volrat);
        double ume = qme / hme;
        fe1 = qme;
        fe2 = qme * ume + .5 * gaccl * hme * hme;
        fe3 = 0.0;
      }
    }
  }
  if (!ldn_dry) {  // :146-175
    double hmn = fmax(0.0, zn - zbpn);
    if (hmn > d.hdry) {
      if (zn <= zp) {
        double fn3p = .5 * gaccl * hmn * hmn;
        fn1 = 0.0;
        fn2 = 0.0;
        fn3 = fn3p;
      } else {
        dzn = fmin(fabs(dzn), hmn);
        double rmn = 0.296 * dzn * sqrt(gaccl * dzn);
        hmn = 0.444 * dzn;
        volrat = d.dxy * hn / dtl;
        rmn = -fmin(rmn, volrat);
        double vmn = rmn / hmn;
        fn1 = rmn;
        fn2 = 0.0;
        fn3 = rmn * vmn + .5 * gaccl * hmn * hmn;
      }
    }
  }
  if (icol == 1 || icol == d.nc) fn1 = edge_weir(volrat, d.sqrt_gaccl, hp);
  if (irow == 1 || irow == d.nr) fe1 = edge_weir(volrat, d.sqrt_gaccl, hp);
  out[0] = fe1;
  out[1] = fe2;
  out[2] = fe3;
  out[3] = fn1;
  out[4] = fn2;
  out[5] = fn3;
}

// The Courant candidate of one cell (main.cpp:308-316), or +inf if dry.
__device__ __forceinline__ void courant_cell(const fx_dev& d, double h, double qx, double qy, double& dtc,
                                             double& hm) {
  dtc = __longlong_as_double(0x7ff0000000000000LL);
  hm = 0.0;
  if (h > d.hdry) {
    double c0 = sqrt(d.gaccl * h);
    const Over hp(h);  // max(h, hdry) is h here
    double u0 = fmax(.000001, fabs(hp.of(qx)));
    double v0 = fmax(.000001, fabs(hp.of(qy)));
    // min(a / (u0 + c0), a / (v0 + c0)) with a > 0 is a / (max(u0, v0) + c0)
    // bit for bit: rounded addition and division are monotone
    double c = d.cfl_dxy / (fmax(u0, v0) + c0);
    if (c == c) dtc = c;
    hm = h;
  }
}

// Block-wide min/max followed by one atomic each on the control block.
template <class SM>
__device__ void reduce_courant(const fx_dev& d, SM& S, double dtc, double hm) {
  for (int o = 16; o > 0; o >>= 1) {
    dtc = fmin(dtc, __shfl_xor_sync(0xffffffffu, dtc, o));
    hm = fmax(hm, __shfl_xor_sync(0xffffffffu, hm, o));
  }
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  const int nw = (blockDim.x * blockDim.y) / 32;
  if ((tid & 31) == 0) {
    S.red_dt[tid >> 5] = dtc;
    S.red_h[tid >> 5] = hm;
  }
  __syncthreads();
  if (tid == 0) {
    double a = S.red_dt[0], b = S.red_h[0];
    for (int w = 1; w < nw; ++w) {
      a = fmin(a, S.red_dt[w]);
      b = fmax(b, S.red_h[w]);
    }
    if (a < __longlong_as_double(0x7ff0000000000000LL))
      atomicMin(&d.ctl->acc_dtmin, (unsigned long long)__double_as_longlong(a));
    if (b > 0.0) atomicMax(&d.ctl->acc_hmax, (unsigned long long)__double_as_longlong(b));
  }
}

// Shared-memory staging of a tile's stencil by TMA (k_hydro_tma). Each field
// of the stencil (rows irow0-2..irow0+TX, columns icol0-2..icol0+TY) arrives
// as one box of W elements x (BY+2) columns. A TMA box must start on a
// 16-byte boundary along irow, so the box starts at the stencil's first row
// rounded down to 4 (4-byte elements), 2 (8-byte) or 16 (1-byte) elements,
// and the stencil sits `xo` elements into it. Rows and columns outside the
// field read 0 (TMA out-of-bounds fill; the field padding is 0 as well), as
// the per-thread loads of the unstaged path do.
constexpr int STG_W4 = 40, STG_W8 = 36, STG_W1 = 64;  // box widths: 34 + largest offset, 16-byte multiples
__host__ __device__ constexpr int stg_round(int b) { return (b + 127) / 128 * 128; }
template <bool P32, int BY>
struct StageLayout {
  static constexpr int SY = BY + 2;
  static constexpr int B4 = stg_round(STG_W4 * SY * 4), B8 = stg_round(STG_W8 * SY * 8), B1 = stg_round(STG_W1 * SY);
  // FP64 stage: z, zb, qx, qy, melt multiplier (8-byte boxes), flags (1-byte)
  // FP32 stage: eta, eta_lo, qx, qy, melt multiplier (4-byte boxes), zb (8-byte), flags
  static constexpr int O_Z = 0;                                   // z | eta
  static constexpr int O_LO = P32 ? B4 : 0;                       // - | eta_lo
  static constexpr int O_ZB = P32 ? 2 * B4 : B8;                  // zb
  static constexpr int O_QX = P32 ? 2 * B4 + B8 : 2 * B8;         // qx
  static constexpr int O_QY = P32 ? 3 * B4 + B8 : 3 * B8;         // qy
  static constexpr int O_MM = P32 ? 4 * B4 + B8 : 4 * B8;         // melt multiplier
  static constexpr int O_FL = P32 ? 5 * B4 + B8 : 5 * B8;         // flags
  static constexpr int BYTES = O_FL + B1;
};

// x offsets of the stencil in the staged boxes of tile column bx.
struct StageOff {
  int o4, o8, o1;
};
__device__ __forceinline__ StageOff stage_off(int bx) {
  const int x = TX * bx;  // element index of stencil row 0: irow0 - 2 + FX_ROFF
  return StageOff{x & 3, x & 1, x & 15};
}

// A thread's share of a launch's reductions, kept across the tiles it works
// on and reduced once per block (reduce_part): the smallest Courant dt and
// the largest wet depth (exact in any order) and the FP64 water budget.
struct TilePart {
  double dtc, hm, melt, out;
  float hmf;       // FP32 state: high part of hm
  unsigned speed;  // largest approximate wave speed (float bits) whose Courant candidate is in dtc, the warp's
  __device__ __forceinline__ void add(double dt, double h, double m, double o) {
    dtc = fmin(dtc, dt);
    hm = fmax(hm, h);
    melt += m;
    out += o;
  }
};
__device__ __forceinline__ TilePart tile_part() {
  TilePart p;
  p.dtc = __longlong_as_double(0x7ff0000000000000LL);
  p.hm = p.melt = p.out = 0.0;
  p.hmf = 0.0f;
  p.speed = 0u;
  return p;
}

// The fields of the control block a step kernel reads.
struct StepCtl {
  double dtfl, meteoi, meteo_rate, mconc, inflowi;
  double twet_inc;  // dtfl / 3600, the wet-time increment (hydrodynamics_calc.cpp:69-70), once per tile
  Over dt;          // quotients over dtfl, FP64 state
  float dtf, twet_f;  // dtfl and twet_inc in FP32
  // Slot planes (fx_slot) of the state after the previous step and of the one
  // this step writes, and the same of the two-plane fields (fx_pp): here, once
  // per block, because the slot is a 64-bit remainder (the FP32 kernel at
  // 4096 x 4096 cells 1.11 ms a step with it in every tile and with stencil
  // indices by division, 1.02 ms without)
  long long sprev, scur, pprev, pcur;
  long long steps;
  int live, active;
};
__device__ __forceinline__ void read_ctl(const fx_dev& d, StepCtl& c) {
  const fx_ctl& g = *d.ctl;
  c.dtfl = g.dtfl;
  c.meteoi = g.meteoi;
  c.meteo_rate = g.meteo_rate;
  c.mconc = g.mconc;
  c.inflowi = g.inflowi;
  c.twet_inc = g.dtfl / 3600;
  c.dt = Over(g.dtfl);
  c.dtf = (float)g.dtfl;
  c.twet_f = (float)c.twet_inc;
  c.sprev = fx_slot(d, g.steps - 1);
  c.scur = fx_slot(d, g.steps);
  c.pprev = fx_pp(d, g.steps - 1);
  c.pcur = fx_pp(d, g.steps);
  c.steps = g.steps;
  c.live = g.live;
  c.active = g.active;
}

// Block sum of the step's water budget terms, one double atomic each.
__device__ void reduce_budget(const fx_dev& d, double* red, double melt, double out) {
  for (int o = 16; o > 0; o >>= 1) {
    melt += __shfl_xor_sync(0xffffffffu, melt, o);
    out += __shfl_xor_sync(0xffffffffu, out, o);
  }
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  const int nw = (blockDim.x * blockDim.y) / 32;
  __syncthreads();
  if ((tid & 31) == 0) {
    red[2 * (tid >> 5)] = melt;
    red[2 * (tid >> 5) + 1] = out;
  }
  __syncthreads();
  if (tid == 0) {
    double a = 0.0, b = 0.0;
    for (int w = 0; w < nw; ++w) {
      a += red[2 * w];
      b += red[2 * w + 1];
    }
    if (a != 0.0) atomicAdd(&d.ctl->budget_melt, a);
    if (b != 0.0) atomicAdd(&d.ctl->budget_out, b);
  }
}

// The block's reductions of a launch: Courant dt and wet depth, then the
// budget (every thread of the block calls it).
template <class SM>
__device__ __forceinline__ void reduce_part(const fx_dev& d, SM& S, const TilePart& acc) {
  reduce_courant(d, S, acc.dtc, acc.hm);
  reduce_budget(d, S.budget, acc.melt, acc.out);
}

__device__ __forceinline__ double melt_depth(const fx_dev& d, const StepCtl& c, long long gi) {
  if (d.melt_mult) return over((double)c.meteo_rate * d.melt_mult[gi], DAY_MM, 1.0 / DAY_MM) * c.dtfl;
  if (d.melt_mult_f) return (double)c.meteo_rate * (double)d.melt_mult_f[gi] / (1000. * 3600. * 24.) * c.dtfl;
  return c.meteoi;
}

// The point inflow of common.cpp:300-309 on its cell's water level (after
// the melt): a level below the bed is first raised to the bed, then the
// step's inflow depth is added.
__device__ __forceinline__ double inflow_z(double z, double zb, double inflowi) {
  if (z <= zb) z = zb;
  return z + inflowi;
}
// The same on the FP32 state's compensated depth.
__device__ __forceinline__ void inflow_eta(float& eta, float& lo, double inflowi) {
  if (fx_dd_val(eta, lo) <= 0.0) {
    eta = 0.0f;
    lo = 0.0f;
  }
  fx_dd_add(eta, lo, (float)inflowi);
}
__device__ __forceinline__ bool is_inflow(const fx_dev& d, int r, int q) {
  return d.has_inflow && r == d.inflow_irow && q == d.inflow_icol;
}
// The depth the inflow cell had after the melt, for the ADE's dilution.
__device__ __forceinline__ void record_inflow_hm(const fx_dev& d, const StepCtl& c, double hm) {
  d.ctl->rec[c.steps % d.nslot].inflow_hm = hm;
}


// ===================== single-precision step (prec32) =======================
// The same step as the FP64 body, on the depth eta = z - zb and the bed
// differences sx = zb(E) - zb(P), sy = zb(N) - zb(P), formed exactly in FP64
// from the stencil's bed values: every water-surface difference of the
// reference is rewritten without the bed elevation itself,
//   ze - zp = sx(P) + (eta_E - eta_P),  zp - zbpe = eta_P - sx(P)/2,
//   ze - zbpe = eta_E + sx(P)/2,        h = max(0, eta),
// and likewise to the north with sy. Flux, update and friction arithmetic is
// FP32 on the high part of the compensated depth; the branch tests on
// near-zero depths (wet/dry, the face-depth thresholds of both solvers) and
// the signs of near-zero surface differences are decided in FP64 on the
// compensated depth; the Courant candidates and the water budget are FP64.

template <int BY, bool STAGED>
struct HydroSmem32 {
  static constexpr int NSTEN = Tile<BY>::NSTEN, NFLUX = Tile<BY>::NFLUX, NW = Tile<BY>::NTHREADS / 32;
  double budget[2 * NW];
  double red_dt[NW], red_h[NW];
  double zb[STAGED ? 1 : NSTEN];
  float eta[NSTEN], eta_lo[NSTEN], qx[NSTEN], qy[NSTEN];
  // cell velocities q / max(h, hdry, ks) of the stencil, formed once per
  // cell for the wet solver's shear terms (each face reads eight of them)
  static constexpr bool VEL = true;
  float u[NSTEN], v[NSTEN];
  float mi[NSTEN];  // the step's melt depth, of the cells that take it
  float f[3][NFLUX];  // north face fluxes
  unsigned char cls[NSTEN];
};

template <bool P32, int BY, bool STAGED>
using HydroSmem = std::conditional_t<P32, HydroSmem32<BY, STAGED>, HydroSmem64<BY, STAGED>>;

// FP32 arithmetic divides and takes square roots by the approximate hardware
// reciprocal and square root (PTX rcp.approx / sqrt.approx) refined by one
// Newton step with fused multiply-adds: close to correctly rounded for the
// finite, normal operands of this scheme, without the IEEE code paths; the
// FP64 path keeps IEEE-rounded operations for bit parity with the reference.
__device__ __forceinline__ float frcp(float a) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return fmaf(fmaf(-a, r, 1.0f), r, r);
}
__device__ __forceinline__ float fdiv(float a, float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  const float q = a * r;
  return fmaf(fmaf(-b, q, a), r, q);
}
__device__ __forceinline__ float fsqrt(float a) {
  float s, r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(s) : "f"(a));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
  const float t = fmaf(fmaf(-s, s, a), 0.5f * r, s);
  return a > 0.0f ? t : s;
}
// Cube root of h > 0 as 2^(log2(h) / 3) (the friction term only).
__device__ __forceinline__ float fcbrt(float h) {
  float l, r;
  asm("lg2.approx.f32 %0, %1;" : "=f"(l) : "f"(h));
  l = l * (1.0f / 3.0f);
  asm("ex2.approx.f32 %0, %1;" : "=f"(r) : "f"(l));
  return r;
}

// The melt depth the FP32 state adds to a cell this step: the step's
// uniform depth c.meteoi (rate / (1000*3600*24) * dt, computed once in
// k_finalize) times the cell's melt multiplier, rounded once to float. The
// budget counts this float value, the water actually added.
__device__ __forceinline__ float melt32(const fx_dev& d, const StepCtl& c, float mm) {
  return d.melt_mult_f ? (float)(c.meteoi * (double)mm) : (float)c.meteoi;
}

// The Courant candidate of main.cpp:300-323 for the FP32 state. It stays
// FP64, so the FP32 state's dt sequence follows the reference's formula to
// the last bits, but with two divisions instead of four: depth > hdry, so
// the reference's max(h, hdry) is h; u0 and v0 share one reciprocal; and
// min(cfl dxy / (u0 + c0), cfl dxy / (v0 + c0)) = cfl dxy / (max(u0, v0) + c0).
__device__ __forceinline__ void courant_cell32(const fx_dev& d, double depth, float qx, float qy, double& dtc,
                                               double& hm) {
  dtc = __longlong_as_double(0x7ff0000000000000LL);
  hm = 0.0;
  if (depth > d.hdry) {
    const double rh = 1.0 / depth;
    const double c0 = sqrt(d.gaccl * depth);
    const double u0 = fmax(.000001, fabs((double)qx * rh)), v0 = fmax(.000001, fabs((double)qy * rh));
    const double cc = d.cfl_dxy / (fmax(u0, v0) + c0);
    if (cc == cc) dtc = cc;
    hm = depth;
  }
}

// The Courant candidates and depths of a warp's cells into its partials. The
// step's dt needs only the smallest candidate, cfl dxy / speed, so a cell
// whose approximate speed (relative error below 2^-18: two approximate
// operations and a handful of roundings on FP32 operands) is more than 2^-15
// below one whose candidate is in the partials already cannot be the
// smallest, and its two FP64 divisions and root are skipped: a warp evaluates
// its first cells and then the few that set a record. The same for the FP64
// depth, by its high part. The results are those of evaluating every cell.
__device__ __forceinline__ void courant_tile32(const fx_dev& d, bool wet, float eta, float lo, float qx, float qy,
                                               TilePart& acc) {
  float speed = 0.0f;
  if (wet) {
    float r, s;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(eta));
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(d.f.gaccl * eta));
    speed = fmaxf(.000001f, fmaxf(fabsf(qx), fabsf(qy)) * r) + s;
    if (eta >= acc.hmf) {
      acc.hm = fmax(acc.hm, fx_dd_val(eta, lo));
      acc.hmf = eta;
    }
  }
  const bool odd = !(speed < 1e30f);  // an overflow or a NaN bounds nothing
  const unsigned bits = odd ? 0u : __float_as_uint(speed);
  acc.speed = max(acc.speed, __reduce_max_sync(0xffffffffu, bits));
  if (wet && (odd || speed >= __uint_as_float(acc.speed) * (1.0f - 0x1p-15f))) {
    double dtc, hm;
    courant_cell32(d, fmax(0.0, fx_dd_val(eta, lo)), qx, qy, dtc, hm);
    acc.dtc = fmin(acc.dtc, dtc);
  }
}

__device__ __forceinline__ float div_dxy_f(const fx_dev& d, float x) {
  return d.dxy_pow2 ? x * d.f.inv_dxy : fdiv(x, d.f.dxy);
}

// The Roe face-depth test of the FP32 state, `.5 * (max(0, dP) + max(0, dQ))
// > hdry` on the two cells' compensated FP64 depths, decided from its FP32
// value x = .5f * (max(0, eta_P) + max(0, eta_Q)) where that is safe: each
// eta differs from its compensated depth by at most half an ulp and the sum
// rounds once, so |x - exact| <= x * 2^-23, and outside the band
// [hdry (1 - 2^-19), hdry (1 + 2^-19)] (bounds rounded to float) x and the
// exact value lie on the same side of hdry. Inside the band the FP64 test
// (`exact`) decides. The outcome is the FP64 test's in every case.
template <class F>
__device__ __forceinline__ bool above_hdry(float x, float lo, float hi, F exact) {
  if (x > hi) return true;
  if (x < lo) return false;
  return exact();
}

// The compensated depth eta + lo against hdry, decided from eta where that is
// safe (|lo| is at most half an ulp of eta, so the same band serves).
__device__ __forceinline__ bool dd_le_hdry(const fx_dev& d, float eta, float lo) {
  if (eta > d.f.hdry_hi) return false;
  if (eta < d.f.hdry_lo) return true;
  return fx_dd_val(eta, lo) <= d.hdry;
}
// Above it: not the opposite of the one before, as neither holds for a NaN.
__device__ __forceinline__ bool dd_gt_hdry(const fx_dev& d, float eta, float lo) {
  if (eta > d.f.hdry_hi) return true;
  if (eta < d.f.hdry_lo) return false;
  return fx_dd_val(eta, lo) > d.hdry;
}
__device__ __forceinline__ bool dd_lt_hdry(const fx_dev& d, float eta, float lo) {
  if (eta > d.f.hdry_hi) return false;
  if (eta < d.f.hdry_lo) return true;
  return fx_dd_val(eta, lo) < d.hdry;
}

template <class SM, class BED>
__device__ void solver_wet32(const fx_dev& d, const SM& S, const BED& bed, int sr, int sc, int irow, int icol,
                             float dtl, float out[6]) {
  const double hdry = d.hdry;
  const float hdryl = d.f.hdry, gaccl = d.f.gaccl, hdry_lo = d.f.hdry_lo, hdry_hi = d.f.hdry_hi;
  const int P = sidx(sr, sc), W = sidx(sr - 1, sc), E = sidx(sr + 1, sc);
  const int Sx = sidx(sr, sc - 1), N = sidx(sr, sc + 1);
  const int ES = sidx(sr + 1, sc - 1), EN = sidx(sr + 1, sc + 1), WN = sidx(sr - 1, sc + 1);
  auto ksat = [&](int k) { return (S.cls[k] & C_INT) ? d.f.ks : 0.0f; };
  const float kspl = ksat(P);
  const float nueml = d.f.nueml;
  const float dx = d.f.dxy, dy = dx;
  bool lroe = true;
  float volrat = d.volrat_mode == 0 ? __int_as_float(0x7f800000) : 0.0f;
  const bool ldp_dry = S.cls[P] & C_DRY, lde_dry = S.cls[E] & C_DRY, ldn_dry = S.cls[N] & C_DRY;
  // bed differences: exact in FP64 for the branch tests, rounded for the flux arithmetic
  const double sx_d = bed(sr + 1, sc) - bed(sr, sc), sy_d = bed(sr, sc + 1) - bed(sr, sc);
  const float etap = S.eta[P], sxp = (float)sx_d, syp = (float)sy_d;
  // compensated depths for the branch tests (FP64, as the FP64 path decides
  // them), formed where a test needs them
  auto dd = [&](int k) { return fx_dd_val(S.eta[k], S.eta_lo[k]); };
  float qp = S.qx[P], qe = S.qx[E], qn = S.qx[N];
  float rw = S.qy[W], rp = S.qy[P], re = S.qy[E], rn = S.qy[N];
  const float hp = fmaxf(0.0f, etap);
  const float hp0 = fmaxf(fmaxf(hdryl, hp), kspl);
  const float hw = fmaxf(0.0f, S.eta[W]);
  float he = fmaxf(0.0f, S.eta[E]);
  const float hs = fmaxf(0.0f, S.eta[Sx]);
  float hn = fmaxf(0.0f, S.eta[N]);
  float hme = .5f * (hp + he), qme = .5f * (qp + qe), rme = .5f * (rp + re);
  float hmn = .5f * (hp + hn), qmn = .5f * (qp + qn), rmn = .5f * (rp + rn);
  float dze = sxp + (S.eta[E] - etap);
  const float dqe = qe - qp, dre = re - rp;
  float dzn = syp + (S.eta[N] - etap);
  const float drn = rn - rp, dqn = qn - qp;
  if (lde_dry) {
    hme = fmaxf(0.0f, etap - .5f * sxp);
    he = qe = re = 0.0f;
    const double dP = dd(P), dE = dd(E);
    const double dze_d = sx_d + (dE - dP);
    if (fmax(0.0, dP - .5 * sx_d) > hdry) {
      if (dze_d >= 0.0) {
        qme = rme = 0.0f;
      } else {
        dze = fminf((float)fabs(dze_d), hme);
        qme = 0.296f * dze * fsqrt(gaccl * dze);
        volrat = fdiv(0.5f * dx * hp, dtl);
        qme = fminf(qme, volrat);
        rme = 0.0f;
      }
    } else {
      qme = rme = hme = 0.0f;
    }
    lroe = false;
  }
  if (ldn_dry) {
    hmn = fmaxf(0.0f, etap - .5f * syp);
    hn = qn = rn = 0.0f;
    const double dP = dd(P), dN = dd(N);
    const double dzn_d = sy_d + (dN - dP);
    if (fmax(0.0, dP - .5 * sy_d) > hdry) {
      if (dzn_d >= 0.0) {
        qmn = rmn = 0.0f;
      } else {
        dzn = fminf((float)fabs(dzn_d), hmn);
        rmn = 0.296f * dzn * fsqrt(gaccl * dzn);
        qmn = 0.0f;
        volrat = fdiv(0.5f * dy * hp, dtl);
        rmn = fminf(rmn, volrat);
      }
    } else {
      qmn = rmn = hmn = 0.0f;
    }
    lroe = false;
  }
  const float cme = fsqrt(gaccl * hme), cmn = fsqrt(gaccl * hmn);
  const float rhme = frcp(fmaxf(hme, hdryl)), rhmn = frcp(fmaxf(hmn, hdryl));
  const float ume = qme * rhme, vme = rme * rhme;
  const float umn = qmn * rhmn, vmn = rmn * rhmn;
  const float hne = nueml * fsqrt(hp * he);  // (cvdef*us*h + nuem), us = 0
  const float hnn = nueml * fsqrt(hp * hn);
  const float rhp0 = frcp(hp0);
  const float up = qp * rhp0;
  // neighbour velocities from the stencil (a dry neighbour's discharge is 0,
  // so its velocity is 0 whatever depth the division uses)
  const float un = S.u[N];
  const float us0 = S.u[Sx];
  const float use0 = S.u[ES];
  const float une = S.u[EN];
  const float vp = rp * rhp0;
  const float ve = S.v[E];
  const float vw = S.v[W];
  const float vwn = S.v[WN];
  const float ven = S.v[EN];
  const float txye = hne * (div_dxy_f(d, ve - vp) + div_dxy_f(d, .25f * (un + une - us0 - use0)));
  const float txyn = hnn * (div_dxy_f(d, un - up) + div_dxy_f(d, .25f * (ve + ven - vw - vwn)));
  const float fe1c = qme, fe2c = qme * ume, fe3c = qme * vme - txye;
  const float fn1c = rmn, fn2c = rmn * umn - txyn, fn3c = rmn * vmn;
  float fe1r = 0.f, fe2r = 0.f, fe3r = 0.f, fn1r = 0.f, fn2r = 0.f, fn3r = 0.f;
  if (lroe) {
    float cc;
    if (above_hdry(hme, hdry_lo, hdry_hi, [&] { return .5 * (fmax(0.0, dd(P)) + fmax(0.0, dd(E))) > hdry; })) {
      float dzea = fabsf(dze);
      if (dzea > 0.5f * hme) {
        dzea = fminf(dzea, fabsf(he - hp));
        dze = copysignf(dzea, dze);
      }
      cc = fdiv(.25f, cme);
    } else {
      cc = 0.0f;
    }
    float c1 = ume, c2 = ume + cme, c3 = ume - cme;
    float c1a = fabsf(c1), c2a = fabsf(c2), c3a = fabsf(c3);
    fe1r = -((c2 * c3a - c2a * c3) * dze + (c2a - c3a) * dqe) * cc;
    fe2r = -(c2 * c3 * (c3a - c2a) * dze + (c2a * c2 - c3a * c3) * dqe) * cc;
    fe3r = -(vme * (c2 * c3a - 2.f * cme * c1a - c2a * c3) * dze + vme * (c2a - c3a) * dqe + 2.f * cme * c1a * dre) * cc;
    if (!ldp_dry &&
        above_hdry(hmn, hdry_lo, hdry_hi, [&] { return .5 * (fmax(0.0, dd(P)) + fmax(0.0, dd(N))) > hdry; })) {
      float dzna = fminf(fabsf(dzn), fabsf(hn - hp));
      dzn = copysignf(dzna, dzn);
      cc = fdiv(.25f, cmn);
    } else {
      cc = 0.0f;
    }
    c1 = vmn;
    c2 = vmn + cmn;
    c3 = vmn - cmn;
    c1a = fabsf(c1);
    c2a = fabsf(c2);
    c3a = fabsf(c3);
    fn1r = -((c2 * c3a - c2a * c3) * dzn + (c2a - c3a) * drn) * cc;
    fn2r = -(umn * (c2 * c3a - 2.f * cmn * c1a - c2a * c3) * dzn + 2.f * cmn * c1a * dqn + umn * (c2a - c3a) * drn) * cc;
    fn3r = -(c2 * c3 * (c3a - c2a) * dzn + (c2a * c2 - c3a * c3) * drn) * cc;
  }
  float fe1 = fe1c + fe1r;
  const float fe2 = fe2c + fe2r + .5f * gaccl * (hme * hme);
  const float fe3 = fe3c + fe3r;
  float fn1 = fn1c + fn1r;
  const float fn2 = fn2c + fn2r;
  const float fn3 = fn3c + fn3r + .5f * gaccl * (hmn * hmn);
  if (icol == 1 || icol == d.nc || irow == 1 || irow == d.nr) {  // the edge weir, on edge cells only
    const float weir = fsqrt(gaccl) * hp * fsqrt(hp);
    if (icol == 1 || icol == d.nc) fn1 = fminf(volrat, weir);
    if (irow == 1 || irow == d.nr) fe1 = fminf(volrat, weir);
  }
  volrat = fdiv(d.f.area * hp, dtl);
  {  // solver_wetdomain.cpp:309-332 as selects: one straight-line block, the
     // quotient of the split kept only when the split applies
    const float sdy = fe1 * dy, sdx = fn1 * dx, sum = sdy + sdx;
    const bool pos = volrat > 0.0f, pe = fe1 > 0.0f, pn = fn1 > 0.0f;
    const bool split = pos & pe & pn & (sum > volrat);
    const float cf = fdiv(sdx, split ? sum : 1.0f);
    const float e = div_dxy_f(d, split ? (1.f - cf) * volrat : fminf(sdy, volrat));
    const float n = div_dxy_f(d, split ? cf * volrat : fminf(sdx, volrat));
    fe1 = !pos ? 0.0f : ((split | (pe & !pn)) ? e : fe1);
    fn1 = !pos ? 0.0f : ((split | (pn & !pe)) ? n : fn1);
  }
  out[0] = fe1;
  out[1] = fe2;
  out[2] = fe3;
  out[3] = fn1;
  out[4] = fn2;
  out[5] = fn3;
}

template <class SM, class BED>
__device__ void solver_dry32(const fx_dev& d, const SM& S, const BED& bed, int sr, int sc, int irow, int icol,
                             float dtl, float out[6]) {
  const int P = sidx(sr, sc), E = sidx(sr + 1, sc), N = sidx(sr, sc + 1);
  const float gaccl = d.f.gaccl;
  float volrat = d.volrat_mode == 0 ? __int_as_float(0x7f800000) : 0.0f;
  const bool lde_dry = S.cls[E] & C_DRY, ldn_dry = S.cls[N] & C_DRY;
  const double sx_d = bed(sr + 1, sc) - bed(sr, sc), sy_d = bed(sr, sc + 1) - bed(sr, sc);
  const float etap = S.eta[P], etae = S.eta[E], etan = S.eta[N], sxp = (float)sx_d, syp = (float)sy_d;
  const double dP = fx_dd_val(etap, S.eta_lo[P]), dE = fx_dd_val(etae, S.eta_lo[E]);
  const double dN = fx_dd_val(etan, S.eta_lo[N]);
  const float he = fmaxf(0.0f, etae), hn = fmaxf(0.0f, etan);
  float dze = sxp + (etae - etap), dzn = syp + (etan - etap);
  float fe1 = 0.f, fe2 = 0.f, fe3 = 0.f, fn1 = 0.f, fn2 = 0.f, fn3 = 0.f;
  if (!lde_dry) {
    float hme = fmaxf(0.0f, etae + .5f * sxp);
    const double dze_d = sx_d + (dE - dP);
    if (fmax(0.0, dE + .5 * sx_d) > d.hdry) {
      if (dze_d <= 0.0) {
        fe2 = .5f * gaccl * hme * hme;
      } else {
        // the surface difference is positive (decided in FP64); its FP32
        // value can round to 0, where the inflow and its momentum are 0
        dze = fminf((float)dze_d, hme);
        volrat = fdiv(d.f.dxy * he, dtl);
        if (dze > 0.0f) {
          float qme = 0.296f * dze * fsqrt(gaccl * dze);
          hme = 0.444f * dze;
          qme = -fminf(qme, volrat);
          fe1 = qme;
          fe2 = qme * fdiv(qme, hme) + .5f * gaccl * hme * hme;
        }
      }
    }
  }
  if (!ldn_dry) {
    float hmn = fmaxf(0.0f, etan + .5f * syp);
    const double dzn_d = sy_d + (dN - dP);
    if (fmax(0.0, dN + .5 * sy_d) > d.hdry) {
      if (dzn_d <= 0.0) {
        fn3 = .5f * gaccl * hmn * hmn;
      } else {
        dzn = fminf((float)dzn_d, hmn);
        volrat = fdiv(d.f.dxy * hn, dtl);
        if (dzn > 0.0f) {
          float rmn = 0.296f * dzn * fsqrt(gaccl * dzn);
          hmn = 0.444f * dzn;
          rmn = -fminf(rmn, volrat);
          fn1 = rmn;
          fn3 = rmn * fdiv(rmn, hmn) + .5f * gaccl * hmn * hmn;
        }
      }
    }
  }
  // the dry cell's own depth is taken as 0 (solver_drydomain.cpp:85): the weir is 0
  if (icol == 1 || icol == d.nc) fn1 = fminf(volrat, 0.0f);
  if (irow == 1 || irow == d.nr) fe1 = fminf(volrat, 0.0f);
  out[0] = fe1;
  out[1] = fe2;
  out[2] = fe3;
  out[3] = fn1;
  out[4] = fn2;
  out[5] = fn3;
}

// The FP64 per-step record of an owned cell in the step's slot
// (fx_dev::rec64), as three 16-byte stores.
__device__ __forceinline__ void put_rec64(const fx_dev& d, long long o, double h0, double h, double hp, double fe1,
                                          double fn1, uint8_t fl) {
  double2* r = reinterpret_cast<double2*>(fx_rec64(d, o));
  r[0] = make_double2(h0, h);
  r[1] = make_double2(hp, fe1);
  r[2] = make_double2(fn1, __longlong_as_double((long long)fl));
}

// The per-step record of an owned cell in the step's slot (fx_dev::rec32).
__device__ __forceinline__ void put_rec32(const fx_dev& d, long long o, float h0, float h, float hp, float mi,
                                          float fe1, float fn1, uint8_t fl) {
  float4* r = d.rec32 + 2 * o;
  r[0] = make_float4(h0, h, hp, mi);
  r[1] = make_float4(fe1, fn1, __uint_as_float((unsigned)fl), 0.0f);
}

// A step without solver (no wet cell): the Courant scan and add_meteo only
// (main.cpp:300-370, the solver block at :385 is skipped).
template <int BY>
__device__ __forceinline__ void idle_tile32(const fx_dev& d, const StepCtl& c, const fx_tile& tile, TilePart& acc) {
  const int irow = 1 + tile.bx * TX + threadIdx.x, icol = 1 + tile.by * Tile<BY>::TY + threadIdx.y;
  const bool own = threadIdx.x < TX && threadIdx.y < Tile<BY>::TY && irow <= d.nr && icol <= d.nc;
  const bool melt_on = d.has_meteo != 0;
  const long long sprev = c.sprev, scur = c.scur, pprev = c.pprev, pcur = c.pcur;
  double dtc = __longlong_as_double(0x7ff0000000000000LL), hm = 0.0, bmelt = 0.0;
  if (own) {
    const long long gi = fx_ix(d, irow, icol);
    const float etapre = d.eta[pprev + gi];
    float eta1 = etapre, lo1 = d.eta_lo[pprev + gi];
    const uint8_t fl = d.flags[sprev + gi];
    const float hpre = fmaxf(0.0f, etapre);
    uint8_t ld = fx_dd_val(etapre, lo1) > d.hdry ? 0 : 1;
    float h1 = hpre;
    double depth = fx_dd_val(etapre, lo1);
    float mir = 0.0f;  // the record's melt depth
    if (melt_on && !(fl & FX_F_NODATA)) {
      const float mi = melt32(d, c, d.melt_mult_f ? d.melt_mult_f[gi] : 1.0f);
      mir = mi;
      bmelt = (double)mi * d.arbase;
      fx_dd_add(eta1, lo1, mi);
      h1 = fmaxf(eta1, 0.0f);
      depth = fx_dd_val(eta1, lo1);
      if (depth <= d.hdry) ld = 0;
    }
    if (is_inflow(d, irow, icol)) {  // common.cpp:300-315
      const double dm = fx_dd_val(eta1, lo1);
      record_inflow_hm(d, c, fmax(dm, 0.0));
      inflow_eta(eta1, lo1, c.inflowi);
      depth = fx_dd_val(eta1, lo1);
      bmelt += (depth - dm) * d.arbase;
      h1 = fmaxf(eta1, 0.0f);
      ld = depth <= d.hdry ? 1 : 0;
    }
    const float qx = d.qx_f[pprev + gi], qy = d.qy_f[pprev + gi];
    d.eta[pcur + gi] = eta1;
    d.eta_lo[pcur + gi] = lo1;
    d.qx_f[pcur + gi] = qx;
    d.qy_f[pcur + gi] = qy;
    const uint8_t fl1 = (fl & (FX_F_WALL | FX_F_NODATA)) | ((fl & FX_F_LDRY) ? FX_F_LDRY_PREV : 0) | ld;
    d.flags[scur + gi] = fl1;
    // fluxes are unchanged by a step without solver
    const float* rp = fx_rec(d, sprev + gi);
    const bool melted = melt_on && !(fl & FX_F_NODATA);
    put_rec32(d, scur + gi, h1, h1, melted ? hpre : 0.0f, mir,
              rp[FX_R_FE1], rp[FX_R_FN1], fl1);
    courant_cell32(d, fmax(0.0, depth), qx, qy, dtc, hm);
  }
  acc.add(dtc, hm, bmelt, 0.0);
}

template <int BY, bool STAGED, class F>
__device__ __forceinline__ bool hydro_tile32(const fx_dev& d, const StepCtl& c, const fx_tile& tile,
                                             HydroSmem32<BY, STAGED>& S, TilePart& acc, const unsigned char* stg, int bad, F stage_free) {
  using L = StageLayout<true, BY>;
  const StageOff so = stage_off(tile.bx);
  constexpr int TY = Tile<BY>::TY;
  const int lx = threadIdx.x, ly = threadIdx.y;
  const int tid = ly * BX + lx;
  const int irow0 = 1 + tile.bx * TX, icol0 = 1 + tile.by * TY;
  // The thread's face-flux cell and, but for the west row and south column of
  // the tile, the cell it owns.
  const int irow = irow0 - 1 + lx, icol = icol0 - 1 + ly;
  const bool own = lx > 0 && ly > 0 && irow <= d.nr && icol <= d.nc;
  const float dtl = c.dtf;
  const bool melt_on = d.has_meteo != 0;
  const long long sprev = c.sprev, scur = c.scur, pprev = c.pprev, pcur = c.pcur;
  double bmelt = 0.0, bout = 0.0;


  const auto bed = [&] {
    if constexpr (STAGED) return Bed<STG_W8>{reinterpret_cast<const double*>(stg + L::O_ZB) + so.o8};
    else return Bed<SX>{S.zb};
  }();
  if constexpr (STAGED) {
    // staged by TMA: the same values, read from shared memory
    const float* g_eta = reinterpret_cast<const float*>(stg + L::O_Z);
    const float* g_lo = reinterpret_cast<const float*>(stg + L::O_LO);
    const float* g_qx = reinterpret_cast<const float*>(stg + L::O_QX);
    const float* g_qy = reinterpret_cast<const float*>(stg + L::O_QY);
    const float* g_mm = reinterpret_cast<const float*>(stg + L::O_MM);
    const uint8_t* g_fl = stg + L::O_FL;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      int sr, scc;
      if (!stencil_cell<BY>(pass, lx, ly, sr, scc)) break;
      const int k = sidx(sr, scc);
      const int r = irow0 - 2 + sr, q = icol0 - 2 + scc;
      const int i4 = scc * STG_W4 + sr + so.o4;
      float eta = g_eta[i4], lo = g_lo[i4], qx = g_qx[i4], qy = g_qy[i4];
      unsigned char cl = 0;
      if (r >= 1 && r <= d.nr && q >= 1 && q <= d.nc) {
        cl = C_INT;
        const uint8_t fl = g_fl[scc * STG_W1 + sr + so.o1];
        if (fl & FX_F_WALL) cl |= C_WALL;
        if (melt_on && !(fl & FX_F_NODATA)) {
          const float mi = melt32(d, c, g_mm[i4]);
          S.mi[k] = mi;
          fx_dd_add(eta, lo, mi);
        }
        if (is_inflow(d, r, q)) inflow_eta(eta, lo, c.inflowi);
        if (dd_le_hdry(d, eta, lo)) {
          qx = 0.f;
          qy = 0.f;
          cl |= C_DRY;
        }
      }
      S.eta[k] = eta;
      S.eta_lo[k] = lo;
      S.qx[k] = qx;
      S.qy[k] = qy;
      S.cls[k] = cl;
      {
        const float den = fmaxf(fmaxf(fmaxf(0.0f, eta), d.f.hdry), (cl & C_INT) ? d.f.ks : 0.0f);
        S.u[k] = fdiv(qx, den);
        S.v[k] = fdiv(qy, den);
      }
    }
  } else {
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      int sr, scc;
      if (!stencil_cell<BY>(pass, lx, ly, sr, scc)) break;
      const int k = sidx(sr, scc);
      const int r = irow0 - 2 + sr, q = icol0 - 2 + scc;
      float eta = 0.f, lo = 0.f, qx = 0.f, qy = 0.f;
      double zb = 0.0;
      unsigned char cl = 0;
      if (r >= 0 && r <= d.nr + 1 && q >= 0 && q <= d.nc + 1) {
        const long long gi = fx_ix(d, r, q);
        eta = d.eta[pprev + gi];
        lo = d.eta_lo[pprev + gi];
        zb = d.zb[gi];
        qx = d.qx_f[pprev + gi];
        qy = d.qy_f[pprev + gi];
        if (r >= 1 && r <= d.nr && q >= 1 && q <= d.nc) {
          cl = C_INT;
          const uint8_t fl = d.flags[sprev + gi];
          if (fl & FX_F_WALL) cl |= C_WALL;
          if (melt_on && !(fl & FX_F_NODATA)) {
            const float mi = melt32(d, c, d.melt_mult_f ? d.melt_mult_f[gi] : 1.0f);
            S.mi[k] = mi;
            fx_dd_add(eta, lo, mi);
          }
          if (is_inflow(d, r, q)) inflow_eta(eta, lo, c.inflowi);
          if (dd_le_hdry(d, eta, lo)) {
            qx = 0.f;
            qy = 0.f;
            cl |= C_DRY;
          }
        }
      }
      S.eta[k] = eta;
      S.eta_lo[k] = lo;
      S.zb[k] = zb;
      S.qx[k] = qx;
      S.qy[k] = qy;
      S.cls[k] = cl;
        {
          const float den = fmaxf(fmaxf(fmaxf(0.0f, eta), d.f.hdry), (cl & C_INT) ? d.f.ks : 0.0f);
          S.u[k] = fdiv(qx, den);
          S.v[k] = fdiv(qy, den);
        }
    }
  }
  // the stencil is complete; a thread whose stage wait gave up (bad) stops
  // the whole block here, before anything is written to global memory
  if (__syncthreads_or(bad)) return false;
  // Each thread computes its own face-flux cell (NFLUX == NTHREADS), wet, dry
  // or kept: gathering each kind's cells in lists cost more than the
  // divergence it avoids (4096^2 wet start 1.4 % and the 64-scenario batch 6 %
  // faster without).
  // Its six fluxes stay in registers for the update of the cell itself; the
  // east faces' go to the neighbour's lane by shuffle, the north faces' to the
  // next column's warp through shared memory.
  const int sr = lx + 1, sc = ly + 1, sP = sidx(sr, sc);
  const unsigned char cl = S.cls[sP];
  const bool wall = cl & C_WALL;
  bool computed = false;
  float o[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};  // of wall cells and outside: never written in the reference
  if ((cl & C_INT) && !wall) {
    const bool alldry = S.cls[sidx(sr - 1, sc)] & S.cls[sidx(sr + 1, sc)] & S.cls[sidx(sr, sc - 1)] &
                        S.cls[sidx(sr, sc + 1)] & cl & C_DRY;
    if (alldry) {
      // all five cells dry: the reference returns before storing
      // (solver_drydomain.cpp:60-76), so the fluxes of the last step that
      // computed them stay in effect
      const long long gi = fx_ix(d, irow, icol);
      const float* rp = fx_rec(d, sprev + gi);
      o[0] = rp[FX_R_FE1];
      o[1] = d.fe2_f[gi];
      o[2] = d.fe3_f[gi];
      o[3] = rp[FX_R_FN1];
      o[4] = d.fn2_f[gi];
      o[5] = d.fn3_f[gi];
    } else {
      computed = true;
      if (cl & C_DRY) solver_dry32(d, S, bed, sr, sc, irow, icol, dtl, o);
      else solver_wet32(d, S, bed, sr, sc, irow, icol, dtl, o);
    }
  }
  for (int j = 0; j < 3; ++j) S.f[j][tid] = o[3 + j];
  float w[3];  // the west neighbour's east faces
  for (int j = 0; j < 3; ++j) w[j] = __shfl_up_sync(0xffffffffu, o[j], 1);
  // What the update takes from the stage and the stencil is read here, before
  // the barrier: after it the stage is free for the tile after next, and a
  // warp that is done with its update may read the next tile's stencil while
  // others are still at it, so a tile has two barriers. The wet time and the
  // roughness are loaded here for the update behind the barrier: 4096 x 4096
  // cells 0.92 ms a step before, 0.91 with two barriers, 0.86 with the loads.
  bool wet = false, outE = false, outN = false;
  uint8_t fl = 0;
  float eta = 0.f, lo = 0.f, qx = 0.f, qy = 0.f;  // this thread's cell, before and after the update
  float tw = 0.f, n = 0.f;
  float h0v = 0.f, hpv = 0.f, miv = 0.f;          // the record's depths: at the start of the step, pre-melt, of the melt
  if (own) {
    const int i4 = sc * STG_W4 + sr + so.o4;
    const long long gi = fx_ix(d, irow, icol);
    fl = STAGED ? stg[L::O_FL + sc * STG_W1 + sr + so.o1] : d.flags[sprev + gi];
    if (!(cl & C_DRY)) tw = d.twet_f[gi];
    if (d.manning_f) n = d.manning_f[gi];
    eta = S.eta[sP];
    lo = S.eta_lo[sP];
    qx = S.qx[sP];
    qy = S.qy[sP];
    outE = irow == d.nr || (S.cls[sidx(sr + 1, sc)] & C_WALL);
    outN = icol == d.nc || (S.cls[sidx(sr, sc + 1)] & C_WALL);
    const float etapre = STAGED ? reinterpret_cast<const float*>(stg + L::O_Z)[i4] : d.eta[pprev + gi];
    h0v = fmaxf(0.0f, etapre);
    if (melt_on && !(fl & FX_F_NODATA)) {
      h0v = fmaxf(eta, 0.0f);
      hpv = fmaxf(etapre, 0.0f);
      miv = S.mi[sP];
      bmelt = (double)miv * d.arbase;
    }
    if (is_inflow(d, irow, icol)) {  // common.cpp:300-315 (h0 = the depth after the inflow)
      float em = etapre, lm = STAGED ? reinterpret_cast<const float*>(stg + L::O_LO)[i4] : d.eta_lo[pprev + gi];
      if (melt_on && !(fl & FX_F_NODATA)) fx_dd_add(em, lm, miv);
      const double dm = fx_dd_val(em, lm);
      record_inflow_hm(d, c, fmax(dm, 0.0));
      bmelt += (fx_dd_val(eta, lo) - dm) * d.arbase;
      h0v = fmaxf(eta, 0.0f);
    }
  }
  __syncthreads();
  stage_free();
  if (own) {
    const long long gi = fx_ix(d, irow, icol);
    const int S0 = tid - BX;  // the south neighbour's north faces
    if (!(cl & C_DRY)) d.twet_f[gi] = tw + c.twet_f;
    float dh = 0.f, dqx = 0.f, dqy = 0.f, qxfP = 0.f, qyfP = 0.f;
    if (!wall) {
      dh = (div_dxy_f(d, w[0] - o[0]) + div_dxy_f(d, S.f[0][S0] - o[3])) * dtl;
      dqx = (div_dxy_f(d, w[1] - o[1]) + div_dxy_f(d, S.f[1][S0] - o[4])) * dtl;
      dqy = (div_dxy_f(d, w[2] - o[2]) + div_dxy_f(d, S.f[2][S0] - o[5])) * dtl;
      qxfP = o[0] * dtl;
      qyfP = o[3] * dtl;
      if (outE) bout += (double)o[0] * d.dxy * c.dtfl;
      if (outN) bout += (double)o[3] * d.dxy * c.dtfl;
    }
    const float qxfW = w[0] * dtl, qyfS = S.f[0][S0] * dtl;
    fx_dd_add(eta, lo, dh);
    const float h = fmaxf(0.0f, eta);
    uint8_t ld;
    if (dd_lt_hdry(d, eta, lo) || wall) {
      qx = qy = 0.0f;
      ld = 1;
    } else {
      qx += dqx;
      qy += dqy;
      qx = .1f * qxfW + .8f * qx + .1f * qxfP;
      qy = .1f * qyfS + .8f * qy + .1f * qyfP;
      ld = 0;
    }
    if (d.manning_f && ld == 0 && !wall) {
      if (n != 0.0f) {
        const float qm = fsqrt(qx * qx + qy * qy);
        const float den = 1.0f + fdiv(dtl * d.f.gaccl * n * n * qm, h * h * fcbrt(h));
        const float rden = frcp(den);
        qx = qx * rden;
        qy = qy * rden;
      }
    }
    d.eta[pcur + gi] = eta;
    d.eta_lo[pcur + gi] = lo;
    d.qx_f[pcur + gi] = qx;
    d.qy_f[pcur + gi] = qy;
    const uint8_t fl1 = (fl & (FX_F_WALL | FX_F_NODATA)) | ((fl & FX_F_LDRY) ? FX_F_LDRY_PREV : 0) | ld;
    d.flags[scur + gi] = fl1;
    if (computed && (d.store_all_fluxes || !dd_gt_hdry(d, eta, lo))) {
      d.fe2_f[gi] = o[1];
      d.fe3_f[gi] = o[2];
      d.fn2_f[gi] = o[4];
      d.fn3_f[gi] = o[5];
    }
    // fe_1 and fn_1 of every cell go to this step's slot, kept ones too
    put_rec32(d, scur + gi, h0v, h, hpv, miv, o[0], o[3], fl1);
    wet = d.f.below_zero || (eta > 0.0f && dd_gt_hdry(d, eta, lo));
  }
  courant_tile32(d, wet, eta, lo, qx, qy, acc);
  acc.melt += bmelt;
  acc.out += bout;
  return true;
}

// A step without solver (no wet cell): the Courant scan and add_meteo only
// (main.cpp:300-370, the solver block at :385 is skipped). The solute
// dilution of add_meteo is applied by the ADE sweep (fx_ade.cu).
template <int BY>
__device__ __forceinline__ void idle_tile64(const fx_dev& d, const StepCtl& c, const fx_tile& tile, TilePart& acc) {
  const int irow = 1 + tile.bx * TX + threadIdx.x, icol = 1 + tile.by * Tile<BY>::TY + threadIdx.y;
  const bool own = threadIdx.x < TX && threadIdx.y < Tile<BY>::TY && irow <= d.nr && icol <= d.nc;
  const bool melt_on = d.has_meteo != 0;
  const long long sprev = c.sprev, scur = c.scur, pprev = c.pprev, pcur = c.pcur;
  double dtc = __longlong_as_double(0x7ff0000000000000LL), hm = 0.0, bmelt = 0.0;
  if (own) {
    const long long gi = fx_ix(d, irow, icol);
    const double zb = d.zb[gi], zpre = d.z[pprev + gi];
    const uint8_t fl = d.flags[sprev + gi];
    const double hpre = max0(zpre - zb);
    uint8_t ld = hpre > d.hdry ? 0 : 1;  // Courant scan (:308-320)
    double z1 = zpre, h1 = hpre, hpv = 0.0;
    if (melt_on && zb != d.nodata) {
      const double mi = melt_depth(d, c, gi);
      bmelt = mi * d.arbase;
      hpv = max0(zpre - zb);  // the dilution's hp (common.cpp:216)
      z1 = zpre + mi;
      h1 = max0(z1 - zb);
      if (h1 <= d.hdry) ld = 0;  // common.cpp:219-222
    }
    if (is_inflow(d, irow, icol)) {  // common.cpp:300-315
      const double zm = z1;
      record_inflow_hm(d, c, max0(zm - zb));
      z1 = inflow_z(z1, zb, c.inflowi);
      h1 = max0(z1 - zb);
      ld = h1 <= d.hdry ? 1 : 0;
      bmelt += (z1 - zm) * d.arbase;
    }
    const double qx = d.qx[pprev + gi], qy = d.qy[pprev + gi];
    d.z[pcur + gi] = z1;
    d.qx[pcur + gi] = qx;
    d.qy[pcur + gi] = qy;
    const uint8_t fl1 = (fl & (FX_F_WALL | FX_F_NODATA)) | ((fl & FX_F_LDRY) ? FX_F_LDRY_PREV : 0) | ld;
    d.flags[scur + gi] = fl1;
    const double* rp = fx_rec64(d, sprev + gi);  // fluxes are unchanged by a step without solver
    put_rec64(d, scur + gi, h1, h1, hpv, rp[FX_R64_FE1], rp[FX_R64_FN1], fl1);
    courant_cell(d, h1, qx, qy, dtc, hm);
  }
  acc.add(dtc, hm, bmelt, 0.0);
}

// The FP64 step of one tile (the reference's arithmetic, bit for bit).
template <int BY, bool STAGED, class F>
__device__ __forceinline__ bool hydro_tile64(const fx_dev& d, const StepCtl& c, const fx_tile& tile,
                                             HydroSmem64<BY, STAGED>& S, TilePart& acc, const unsigned char* stg, int bad, F stage_free) {
  using SM = HydroSmem64<BY, STAGED>;
  using L = StageLayout<false, BY>;
  const StageOff so = stage_off(tile.bx);
  constexpr int TY = Tile<BY>::TY;
  const int lx = threadIdx.x, ly = threadIdx.y;
  const int tid = ly * BX + lx;
  const int irow0 = 1 + tile.bx * TX, icol0 = 1 + tile.by * TY;
  // The thread's face-flux cell and, but for the west row and south column of
  // the tile, the cell it owns.
  const int irow = irow0 - 1 + lx, icol = icol0 - 1 + ly;
  const bool own = lx > 0 && ly > 0 && irow <= d.nr && icol <= d.nc;
  const double dtl = c.dtfl;
  const bool melt_on = d.has_meteo != 0;

  // Slot planes: the state after the previous step, and the one this step
  // writes (h, h0, fe_1, fn_1, flags), and the two planes of z, qx, qy (see
  // fx_common.cuh): every block reads the previous step's plane, halo
  // included, and writes the other.
  const long long sprev = c.sprev, scur = c.scur, pprev = c.pprev, pcur = c.pcur;


  const auto bed = [&] {
    if constexpr (STAGED) return Bed<STG_W8>{reinterpret_cast<const double*>(stg + L::O_ZB) + so.o8};
    else return Bed<SX>{S.zb};
  }();
  // ---- phase A: stencil load, melt, Loop 1 ---------------------------------
  if constexpr (STAGED) {
    // staged by TMA: the same values, read from shared memory
    const double* g_z = reinterpret_cast<const double*>(stg + L::O_Z);
    const double* g_zb = reinterpret_cast<const double*>(stg + L::O_ZB);
    const double* g_qx = reinterpret_cast<const double*>(stg + L::O_QX);
    const double* g_qy = reinterpret_cast<const double*>(stg + L::O_QY);
    const double* g_mm = reinterpret_cast<const double*>(stg + L::O_MM);
    const uint8_t* g_fl = stg + L::O_FL;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      int sr, sc;
      if (!stencil_cell<BY>(pass, lx, ly, sr, sc)) break;
      const int k = sidx(sr, sc);
      const int r = irow0 - 2 + sr, q = icol0 - 2 + sc;
      const int i8 = sc * STG_W8 + sr + so.o8;
      double z = g_z[i8], qx = g_qx[i8], qy = g_qy[i8];
      const double zb = g_zb[i8];
      unsigned char cl = 0;
      if (r >= 1 && r <= d.nr && q >= 1 && q <= d.nc) {
        cl = C_INT;
        if (g_fl[sc * STG_W1 + sr + so.o1] & FX_F_WALL) cl |= C_WALL;
        if (melt_on && zb != d.nodata) {
          const double mi = d.melt_mult ? over((double)c.meteo_rate * g_mm[i8], DAY_MM, 1.0 / DAY_MM) * c.dtfl : c.meteoi;
          S.mi[k] = mi;
          z = z + mi;
        }
        if (is_inflow(d, r, q)) z = inflow_z(z, zb, c.inflowi);
        const double h1 = max0(z - zb);
        if (h1 <= d.hdry) {
          qx = 0.0;
          qy = 0.0;
          cl |= C_DRY;
        }
      }
      S.z[k] = z;
      S.qx[k] = qx;
      S.qy[k] = qy;
      S.cls[k] = cl;
      if constexpr (SM::VEL) {
        const Over den(at_least(at_least(max0(z - zb), d.hdry), (cl & C_INT) ? d.ks : 0.0));
        S.u[k] = den.of(qx);
        S.v[k] = den.of(qy);
      }
    }
  } else {
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      int sr, sc;
      if (!stencil_cell<BY>(pass, lx, ly, sr, sc)) break;
      const int k = sidx(sr, sc);
      const int r = irow0 - 2 + sr, q = icol0 - 2 + sc;
      double z = 0.0, zb = 0.0, qx = 0.0, qy = 0.0;
      unsigned char cl = 0;
      if (r >= 0 && r <= d.nr + 1 && q >= 0 && q <= d.nc + 1) {
        const long long gi = fx_ix(d, r, q);
        z = d.z[pprev + gi];
        zb = d.zb[gi];
        qx = d.qx[pprev + gi];
        qy = d.qy[pprev + gi];
        if (r >= 1 && r <= d.nr && q >= 1 && q <= d.nc) {
          cl = C_INT;
          if (d.flags[sprev + gi] & FX_F_WALL) cl |= C_WALL;
          if (melt_on && zb != d.nodata) z = z + melt_depth(d, c, gi);
          if (is_inflow(d, r, q)) z = inflow_z(z, zb, c.inflowi);
          const double h1 = max0(z - zb);
          if (h1 <= d.hdry) {
            qx = 0.0;
            qy = 0.0;
            cl |= C_DRY;
          }
        }
      }
      S.z[k] = z;
      S.zb[k] = zb;
      S.qx[k] = qx;
      S.qy[k] = qy;
      S.cls[k] = cl;
      if constexpr (SM::VEL) {
        const Over den(at_least(at_least(max0(z - zb), d.hdry), (cl & C_INT) ? d.ks : 0.0));
        S.u[k] = den.of(qx);
        S.v[k] = den.of(qy);
      }
    }
  }
  // the stencil is complete; a thread whose stage wait gave up (bad) stops
  // the whole block here, before anything is written to global memory
  if (__syncthreads_or(bad)) return false;

  // ---- face fluxes ----------------------------------------------------------
  // Each thread computes its own face-flux cell (NFLUX == NTHREADS). Lists of
  // wet, dry and kept cells, which would fill the warps with one kind each,
  // cost a pass and a barrier more than the divergence they avoid: 2048 x 2048
  // cells and a 384 x 384 basin take the same time without, 1000 x 700 cells 1 % less.
  // Its six fluxes stay in registers for the update of the cell itself; the
  // east faces' go to the neighbour's lane by shuffle, the north faces' to the
  // next column's warp through shared memory.
  const int sr = lx + 1, sc = ly + 1, sP = sidx(sr, sc);
  const unsigned char cl = S.cls[sP];
  const bool wall = cl & C_WALL;
  bool computed = false;
  double o[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};  // of wall cells and outside: never written in the reference
  if ((cl & C_INT) && !wall) {
    const bool alldry = S.cls[sidx(sr - 1, sc)] & S.cls[sidx(sr + 1, sc)] & S.cls[sidx(sr, sc - 1)] &
                        S.cls[sidx(sr, sc + 1)] & cl & C_DRY;
    if (alldry) {
      // all five cells dry: the reference returns before storing
      // (solver_drydomain.cpp:60-76), so the fluxes of the last step that
      // computed them stay in effect
      const long long gi = fx_ix(d, irow, icol);
      const double* rp = fx_rec64(d, sprev + gi);
      o[0] = rp[FX_R64_FE1];
      o[1] = d.fe2[gi];
      o[2] = d.fe3[gi];
      o[3] = rp[FX_R64_FN1];
      o[4] = d.fn2[gi];
      o[5] = d.fn3[gi];
    } else {
      computed = true;
      if (cl & C_DRY) solver_dry(d, S, bed, sr, sc, irow, icol, dtl, o);
      else solver_wet(d, S, bed, sr, sc, irow, icol, c.dt, o);
    }
  }
  for (int j = 0; j < 3; ++j) S.f[j][tid] = o[3 + j];
  double w[3];  // the west neighbour's east faces
  for (int j = 0; j < 3; ++j) w[j] = __shfl_up_sync(0xffffffffu, o[j], 1);
  // ---- what the update takes from the stage and the stencil, read before the
  // barrier: after it the stage is free for the tile after next, and a warp
  // that is done with its update may read the next tile's stencil while others
  // are still at it, so a tile has two barriers. The wet time and the roughness
  // are loaded here for the update behind it: 2048 x 2048 cells 0.607 ms a step
  // with three barriers and without the early loads, 0.584 so.
  double bmelt = 0.0, bout = 0.0;
  double c_h = 0.0;  // this thread's depth after the update
  bool outE = false, outN = false;
  uint8_t fl = 0;
  double zb = 0.0, z1 = 0.0, qx = 0.0, qy = 0.0;  // this thread's cell
  double tw = 0.0, n = 0.0;
  double h0v = 0.0, hpv = 0.0;                    // the record's depths
  if (own) {
    const long long gi = fx_ix(d, irow, icol);
    const int i8 = sc * STG_W8 + sr + so.o8;
    fl = STAGED ? stg[L::O_FL + sc * STG_W1 + sr + so.o1] : d.flags[sprev + gi];
    if (!(cl & C_DRY)) tw = d.twet[gi];
    if (d.manning) n = d.manning[gi];
    zb = bed(sr, sc);
    z1 = S.z[sP];
    qx = S.qx[sP];
    qy = S.qy[sP];
    // water leaves the domain through the outflow faces, and into wall cells
    // (which never take it up, hydrodynamics_calc.cpp:111-117)
    outE = irow == d.nr || (S.cls[sidx(sr + 1, sc)] & C_WALL);
    outN = icol == d.nc || (S.cls[sidx(sr, sc + 1)] & C_WALL);
    const double zpre = STAGED ? reinterpret_cast<const double*>(stg + L::O_Z)[i8] : d.z[pprev + gi];

    // add_meteo's h0 (common.cpp:223): the depth after the melt, or the
    // Courant scan's copy of h (main.cpp:305) for cells it skips. Its solute
    // dilution (:226-234) is applied by the ADE sweep (fx_ade.cu).
    h0v = max0(zpre - zb);
    double mi = 0.0;
    if (melt_on && zb != d.nodata) {
      h0v = max0(z1 - zb);
      hpv = max0(zpre - zb);  // the dilution's hp (common.cpp:216)
      mi = STAGED ? S.mi[sP] : melt_depth(d, c, gi);
      bmelt = mi * d.arbase;
    }
    if (is_inflow(d, irow, icol)) {  // common.cpp:300-315 (h0 = the depth after the inflow)
      const double zm = (melt_on && zb != d.nodata) ? zpre + mi : zpre;
      record_inflow_hm(d, c, max0(zm - zb));
      bmelt += (z1 - zm) * d.arbase;
      h0v = max0(z1 - zb);
    }
  }
  __syncthreads();
  stage_free();

  // ---- Loop 3, Loop 4, friction, store, next Courant ------------------------
  if (own) {
    const long long gi = fx_ix(d, irow, icol);
    const int S0 = tid - BX;  // the south neighbour's north faces
    // Loop 1 wet time (:69-70)
    if (!(cl & C_DRY)) d.twet[gi] = tw + c.twet_inc;  // dtl / 3600

    // Loop 3 (:93-120)
    double dh = 0.0, dqx = 0.0, dqy = 0.0, qxfP = 0.0, qyfP = 0.0;
    if (!wall) {
      dh = (div_dxy(d, w[0] - o[0]) + div_dxy(d, S.f[0][S0] - o[3])) * dtl;
      dqx = (div_dxy(d, w[1] - o[1]) + div_dxy(d, S.f[1][S0] - o[4])) * dtl;
      dqy = (div_dxy(d, w[2] - o[2]) + div_dxy(d, S.f[2][S0] - o[5])) * dtl;
      qxfP = o[0] * dtl;
      qyfP = o[3] * dtl;
    }
    if (!wall && outE) bout += o[0] * d.dxy * dtl;
    if (!wall && outN) bout += o[3] * d.dxy * dtl;
    const double qxfW = w[0] * dtl, qyfS = S.f[0][S0] * dtl;

    // Loop 4 (:123-154)
    const double z = z1 + dh;
    const double h = max0(z - zb);
    uint8_t ld;
    if (h < d.hdry || wall) {
      qx = 0.0;
      qy = 0.0;
      ld = 1;
    } else {
      qx += dqx;
      qy += dqy;
      qx = .1 * qxfW + .8 * qx + .1 * qxfP;
      qy = .1 * qyfS + .8 * qy + .1 * qyfP;
      ld = 0;
    }
    // Extension: semi-implicit Manning friction (n = 0 leaves q unchanged).
    if (d.manning && ld == 0 && !wall) {
      if (n != 0.0) {
        const double qm = sqrt(qx * qx + qy * qy);
        const double h73 = h * h * fx_cbrt(h);
        const Over den(1.0 + dtl * d.gaccl * n * n * qm / h73);
        qx = den.of(qx);
        qy = den.of(qy);
      }
    }
    d.z[pcur + gi] = z;
    d.qx[pcur + gi] = qx;
    d.qy[pcur + gi] = qy;
    const uint8_t fl1 = (fl & (FX_F_WALL | FX_F_NODATA)) | ((fl & FX_F_LDRY) ? FX_F_LDRY_PREV : 0) | ld;
    d.flags[scur + gi] = fl1;
    // Fluxes computed this step become the grid values (stale ones are
    // already there). fe_2/fe_3/fn_2/fn_3 are read back only when this cell
    // is dry with four dry neighbours at a later solver step; a cell that
    // ends the step wet (h > hdry) is wet again at the next solver step as
    // long as forcing adds water, so those three-quarters of the flux
    // traffic are skipped for it.
    if (computed && (d.store_all_fluxes || !(h > d.hdry))) {
      d.fe2[gi] = o[1];
      d.fe3[gi] = o[2];
      d.fn2[gi] = o[4];
      d.fn3[gi] = o[5];
    }
    // fe_1 and fn_1 of every cell go to this step's slot, kept ones too
    put_rec64(d, scur + gi, h0v, h, hpv, o[0], o[3], fl1);
    c_h = h;
  }
  double dtc, hm;
  courant_cell(d, c_h, qx, qy, dtc, hm);
  acc.add(dtc, hm, bmelt, bout);
  return true;
}

// The kernels of a step follow one another by programmatic dependent launch: a
// kernel is launched when every block of the one before it has called
// let_next(), and waits in follow(), ahead of its first access to global
// memory, until that one is done and its writes are visible. k_finalize calls
// let_next() at its start, the hydrodynamic kernels when their tiles are done
// (called at their start, the next blocks wait on the SMs that still work).
// Water alone, a step of 64 x 64 cells in FP64 takes 12.9 us (14.0 with full
// launches, 12.7 with the call at the start), of 200 x 200 15.2 (16.7, 15.8),
// of 1024 x 1024 in FP32 67.6 (69.2, 70.3).
__device__ __forceinline__ void let_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void follow() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// One tile of a step without solver, in the domain's precision.
template <bool P32, int BY>
__device__ __forceinline__ void idle_tile(const fx_dev& d, const StepCtl& c, const fx_tile& tile, TilePart& acc) {
  if constexpr (P32) idle_tile32<BY>(d, c, tile, acc);
  else idle_tile64<BY>(d, c, tile, acc);
}
// One tile's step. STAGED: its stencil is in the stage at `stg`, else it is
// read from global memory. `bad`: this thread's wait for the stage gave up.
// stage_free() is called when no thread reads the stage any more.
template <bool P32, int BY, bool STAGED, class F>
__device__ __forceinline__ bool hydro_tile(const fx_dev& d, const StepCtl& c, const fx_tile& tile,
                                           HydroSmem<P32, BY, STAGED>& S, TilePart& acc, const unsigned char* stg,
                                           int bad, F stage_free) {
  if constexpr (P32) return hydro_tile32<BY, STAGED>(d, c, tile, S, acc, stg, bad, stage_free);
  else return hydro_tile64<BY, STAGED>(d, c, tile, S, acc, stg, bad, stage_free);
}

// Reads the step's fields of the control block (written by k_finalize) into
// shared memory, then runs the tile.
template <bool P32, int BY>
__device__ __forceinline__ void hydro_block(const fx_dev& d, const fx_tile& tile, HydroSmem<P32, BY, false>& S,
                                            StepCtl& sc) {
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    read_ctl(d, sc);
  }
  __syncthreads();
  const StepCtl c = sc;
  if (!c.live) return;
  TilePart acc = tile_part();
  if (!c.active) idle_tile<P32, BY>(d, c, tile, acc);
  else hydro_tile<P32, BY, false>(d, c, tile, S, acc, nullptr, 0, [] {});
  let_next();
  reduce_part(d, S, acc);
}

// Blocks per SM the launch bounds ask for: 768 threads for FP64 (at most 80
// registers each), 1024 for FP32 (at most 64). The kernel is bound by the
// instructions it issues (FP32: 71 % of the issue slots) and by their latency
// and the tile barriers (FP64: 52 %), so resident warps pay for the spills
// this costs: at 4096 x 4096 cells the FP32 kernel took 1.50 ms per step at
// 64 registers against 1.73 ms at 80 (3 blocks); at 2048 x 2048 the FP64 one
// took 0.68 ms at 80 against 0.71 ms at 128 (2 blocks), in tiles of 8 rows.
// FP64 tiles of 4 rows serve the small grids, whose blocks have a tile or two
// and little company on their SM: with 96 registers (5 blocks) they take
// 16.4 us at 200 x 200 and 126 us at 1000 x 700, with 80 18.2 and 140 us.
template <bool P32, int BY>
constexpr int min_blocks() { return (P32 ? 32 : BY == 4 ? 20 : 24) / BY; }

// One domain: the descriptor is a kernel parameter (constant bank), so its
// fields are instruction operands. Block (x, y) is tile (x, y).
template <bool P32, int BY>
__global__ void __launch_bounds__(BX * BY, min_blocks<P32, BY>()) k_hydro_one(const __grid_constant__ fx_dev d) {
  __shared__ HydroSmem<P32, BY, false> S;
  __shared__ StepCtl sc;
  const fx_tile tile{0, (int)blockIdx.x, (int)blockIdx.y, 0};
  follow();
  hydro_block<P32, BY>(d, tile, S, sc);
}

// A batch of domains: one block per entry of the tile table; the block copies
// its domain's descriptor to shared memory.
template <bool P32, int BY>
__global__ void __launch_bounds__(BX * BY, min_blocks<P32, BY>()) k_hydro_batch(const fx_dev* __restrict__ devs,
                                                                        const fx_tile* __restrict__ tiles) {
  __shared__ HydroSmem<P32, BY, false> S;
  __shared__ fx_dev sd;
  __shared__ StepCtl sc;
  follow();
  const fx_tile tile = tiles[blockIdx.x];
  {
    const int tid = threadIdx.y * BX + threadIdx.x;
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(devs + tile.dom);
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(&sd);
    for (int i = tid; i < (int)(sizeof(fx_dev) / 8); i += BX * BY) dst[i] = src[i];
  }
  __syncthreads();
  hydro_block<P32, BY>(sd, tile, S, sc);
}
static_assert(sizeof(fx_dev) % 8 == 0, "descriptor copied as 8-byte words");

// ---- TMA-staged persistent form -------------------------------------------
// One block per SM slot loops over the domain's tiles. Thread 0 loads the
// tiles' stencils into two shared-memory stages with TMA (cp.async.bulk.tensor,
// completion counted on an mbarrier), each as soon as its stage is free, two
// tiles ahead, so the halo reads of a tile overlap the arithmetic of the ones
// before it.

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const void* map, int x, int y, int z,
                                            unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// Issue the loads of tile t's stencil into stage `stg` (thread 0).
template <bool P32, int BY>
__device__ __forceinline__ void stage_issue(const fx_dev& d, const fx_tmaps& tm, int t, int ntx, long long step_prev,
                                            unsigned char* stg, unsigned long long* bar) {
  using L = StageLayout<P32, BY>;
  const int bx = t % ntx, by = t / ntx;
  const int x = TX * bx, y = (BY - 1) * by - 1;  // stencil origin (irow0 - 2 + FX_ROFF, icol0 - 2)
  const int x4 = x & ~3, x8 = x & ~1, x1 = x & ~15;
  const int pp = (int)(step_prev & 1), sl = (int)(step_prev % d.nslot);
  const bool mm = P32 ? d.melt_mult_f != nullptr : d.melt_mult != nullptr;
  const unsigned bytes = (unsigned)((P32 ? 4 * STG_W4 * L::SY * 4 + STG_W8 * L::SY * 8
                                         : 4 * STG_W8 * L::SY * 8) +
                                    (mm ? (P32 ? STG_W4 * L::SY * 4 : STG_W8 * L::SY * 8) : 0) + STG_W1 * L::SY);
  mbar_expect_tx(bar, bytes);
  if (P32) {
    tma_load_3d(stg + L::O_Z, &tm.m[FX_TM_Z], x4, y, pp, bar);
    tma_load_3d(stg + L::O_LO, &tm.m[FX_TM_LO], x4, y, pp, bar);
    tma_load_3d(stg + L::O_ZB, &tm.m[FX_TM_ZB], x8, y, 0, bar);
    tma_load_3d(stg + L::O_QX, &tm.m[FX_TM_QX], x4, y, pp, bar);
    tma_load_3d(stg + L::O_QY, &tm.m[FX_TM_QY], x4, y, pp, bar);
    if (mm) tma_load_3d(stg + L::O_MM, &tm.m[FX_TM_MM], x4, y, 0, bar);
  } else {
    tma_load_3d(stg + L::O_Z, &tm.m[FX_TM_Z], x8, y, pp, bar);
    tma_load_3d(stg + L::O_ZB, &tm.m[FX_TM_ZB], x8, y, 0, bar);
    tma_load_3d(stg + L::O_QX, &tm.m[FX_TM_QX], x8, y, pp, bar);
    tma_load_3d(stg + L::O_QY, &tm.m[FX_TM_QY], x8, y, pp, bar);
    if (mm) tma_load_3d(stg + L::O_MM, &tm.m[FX_TM_MM], x8, y, 0, bar);
  }
  tma_load_3d(stg + L::O_FL, &tm.m[FX_TM_FL], x1, y, sl, bar);
}

constexpr long long STAGE_SPIN_LIMIT = 1LL << 22;  // polls of a stage's mbarrier before giving up

template <bool P32, int BY>
__global__ void __launch_bounds__(BX * BY, min_blocks<P32, BY>())
    k_hydro_tma(const __grid_constant__ fx_dev d, const __grid_constant__ fx_tmaps tm, int ntx, int nty) {
  using L = StageLayout<P32, BY>;
  __shared__ HydroSmem<P32, BY, true> S;
  __shared__ StepCtl sc;
  __shared__ __align__(8) unsigned long long bar[2];
  extern __shared__ __align__(128) unsigned char dyn[];
  unsigned char* stage0 = dyn + ((128 - (smem_u32(dyn) & 127)) & 127);
  const int tid = threadIdx.y * BX + threadIdx.x;
  const int ntiles = ntx * nty;
  follow();
  if (tid == 0) read_ctl(d, sc);
  __syncthreads();
  const StepCtl c = sc;
  if (!c.live) return;
  TilePart acc = tile_part();
  if (!c.active) {  // no solver this step: cell-local work only, nothing to stage
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
      const fx_tile tile{0, t % ntx, t / ntx, 0};
      idle_tile<P32, BY>(d, c, tile, acc);
    }
    let_next();
    reduce_part(d, S, acc);
    return;
  }
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int q = 0, t = blockIdx.x; q < 2 && t < ntiles; ++q, t += gridDim.x)
      stage_issue<P32, BY>(d, tm, t, ntx, c.steps - 1, stage0 + q * L::BYTES, &bar[q]);
  }
  __syncthreads();
  unsigned parity = 0u;  // bit q: phase of stage q's barrier
  int st = 0;
  // the block's tiles are gridDim.x apart in the row-major order: in FP32 bx,
  // by step along without a division (1 % of the kernel); in FP64 the
  // registers this takes cost as much
  int bx = blockIdx.x % ntx, by = blockIdx.x / ntx;
  const int dbx = gridDim.x % ntx, dby = gridDim.x / ntx;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    // wait for this tile's stencil, bounded; each thread waits for itself,
    // and the tile's first barrier (after the stencil is read) tells the
    // whole block whether any wait gave up
    long long it = 0;
    int bad = 0;
    while (!mbar_try_wait(&bar[st], (parity >> st) & 1u)) {
      if (++it > STAGE_SPIN_LIMIT) {
        bad = 1;
        break;
      }
    }
    parity ^= 1u << st;
    const fx_tile tile = P32 ? fx_tile{0, bx, by, 0} : fx_tile{0, t % ntx, t / ntx, 0};
    bx += dbx;
    by += dby;
    if (bx >= ntx) {
      bx -= ntx;
      ++by;
    }
    unsigned char* stg = stage0 + st * L::BYTES;
    const auto next = [&] {  // the stage is free: the tile after next
      const int tn = t + 2 * gridDim.x;
      if (tid == 0 && tn < ntiles) stage_issue<P32, BY>(d, tm, tn, ntx, c.steps - 1, stg, &bar[st]);
    };
    if (!hydro_tile<P32, BY, true>(d, c, tile, S, acc, stg, bad, next)) {
      // every thread of the block takes this branch
      if (tid == 0) {
        atomicCAS(&d.ctl->error, 0, FX_DEVERR_WAIT_TIMEOUT);
        // let the copy of the next tile, if one was issued, land before the block exits
        long long w = 0;
        if (t + gridDim.x < ntiles)
          while (!mbar_try_wait(&bar[st ^ 1], (parity >> (st ^ 1)) & 1u) && ++w < STAGE_SPIN_LIMIT) {
          }
      }
      return;
    }
    st ^= 1;
  }
  let_next();
  reduce_part(d, S, acc);
}

// ---- TMA-staged persistent form for a batch --------------------------------
// Each block walks a contiguous range of the packed tile table of all the
// batch's domains (so it crosses few domain boundaries). Thread 0 stages the
// stencil of the block's tile after next with that domain's own tensor maps (a
// device array, one set per domain) while the block computes the current
// tile; a domain without a solver step this launch (stopped, or no wet cell)
// gets no stage. The domain's descriptor and step fields sit in shared
// memory while the block works on its tiles, and the block's Courant and
// budget partials go to a domain when the block leaves it.

// Thread 0: stage tile `tl` into `stg` if its domain runs the solver this step;
// returns whether a copy was issued.
template <bool P32, int BY>
__device__ __forceinline__ bool batch_stage(const fx_dev& d, bool runs, long long step_prev, const fx_tmaps& tm,
                                            const fx_tile& tl, unsigned char* stg, unsigned long long* bar, int& fenced) {
  if (!runs) return false;
  if (fenced != tl.dom) {
    // the maps were written by a host copy before the launch; order the
    // tensor-map proxy's reads of a domain's maps after it, once per domain
    for (int f = 0; f < FX_TM_COUNT; ++f)
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(&tm.m[f]) : "memory");
    fenced = tl.dom;
  }
  const int ntx = (d.nr + TX - 1) / TX;
  stage_issue<P32, BY>(d, tm, tl.by * ntx + tl.bx, ntx, step_prev, stg, bar);
  return true;
}

template <bool P32, int BY>
__global__ void __launch_bounds__(BX * BY, min_blocks<P32, BY>())
    k_hydro_batch_tma(const fx_dev* __restrict__ devs, const fx_tmaps* __restrict__ tms,
                      const fx_tile* __restrict__ tiles, int ntiles) {
  using L = StageLayout<P32, BY>;
  __shared__ HydroSmem<P32, BY, true> S;
  __shared__ fx_dev sd;
  __shared__ StepCtl sc;
  __shared__ __align__(8) unsigned long long bar[2];
  __shared__ int staged[2];      // the tile each stage holds (-1: none)
  __shared__ fx_tile entry[4];   // the table's entries of the tiles under way
  extern __shared__ __align__(128) unsigned char dyn[];
  unsigned char* stage0 = dyn + ((128 - (smem_u32(dyn) & 127)) & 127);
  const int tid = threadIdx.y * BX + threadIdx.x;
  follow();
  const int t0 = (int)((long long)ntiles * blockIdx.x / gridDim.x);
  const int t1 = (int)((long long)ntiles * (blockIdx.x + 1) / gridDim.x);
  if (t0 >= t1) return;
  int fenced = -1;  // thread 0: the domain whose maps it last fenced
  // Thread 0: stage tile t, whose entry is `tl`, into stage q. The descriptor
  // and control block of the domain at hand are in shared memory; another
  // domain's are read from global memory, once per domain and block.
  const auto stage = [&](int t, const fx_tile& tl, int q, int at_hand) {
    entry[t & 3] = tl;
    bool on;
    if (tl.dom == at_hand) {
      on = batch_stage<P32, BY>(sd, sc.live && sc.active, sc.steps - 1, tms[tl.dom], tl, stage0 + q * L::BYTES, &bar[q],
                                fenced);
    } else {
      const fx_dev& d = devs[tl.dom];
      const fx_ctl& g = *d.ctl;
      on = batch_stage<P32, BY>(d, g.live && g.active, g.steps - 1, tms[tl.dom], tl, stage0 + q * L::BYTES, &bar[q],
                                fenced);
    }
    staged[q] = on ? t : -1;
  };
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    staged[1] = -1;
    stage(t0, tiles[t0], 0, -1);
    if (t0 + 1 < t1) stage(t0 + 1, tiles[t0 + 1], 1, -1);
  }
  __syncthreads();
  unsigned parity = 0u;  // bit q: phase of stage q's barrier
  int st = 0, dom = -1;
  TilePart acc = tile_part();
  for (int t = t0; t < t1; ++t) {
    const fx_tile tl = entry[t & 3];
    fx_tile after{};  // thread 0: the entry of the tile after next, loaded ahead of its use
    if (tid == 0 && t + 2 < t1) after = tiles[t + 2];
    if (tl.dom != dom) {
      if (dom >= 0) reduce_part(sd, S, acc);  // the partials of the domain the block leaves
      acc = tile_part();
      __syncthreads();
      const unsigned long long* src = reinterpret_cast<const unsigned long long*>(devs + tl.dom);
      unsigned long long* dst = reinterpret_cast<unsigned long long*>(&sd);
      for (int i = tid; i < (int)(sizeof(fx_dev) / 8); i += BX * BY) dst[i] = src[i];
      __syncthreads();
      if (tid == 0) read_ctl(sd, sc);
      __syncthreads();
      dom = tl.dom;
    }
    const bool mine = staged[st] == t;  // this tile's stencil is (being) staged
    int bad = 0;
    if (mine) {
      long long it = 0;
      while (!mbar_try_wait(&bar[st], (parity >> st) & 1u)) {
        if (++it > STAGE_SPIN_LIMIT) {
          bad = 1;
          break;
        }
      }
      parity ^= 1u << st;
    }
    const auto next = [&] {  // the stage is free: the tile after next
      if (tid == 0) {
        if (t + 2 < t1) stage(t + 2, after, st, dom);
        else staged[st] = -1;
      }
    };
    const StepCtl c = sc;
    const fx_tile tile{0, tl.bx, tl.by, 0};
    if (c.live && c.active) {  // such a domain's tiles are staged
      if (!hydro_tile<P32, BY, true>(sd, c, tile, S, acc, stage0 + st * L::BYTES, bad, next)) {
        // every thread of the block takes this branch
        if (tid == 0) {
          atomicCAS(&sd.ctl->error, 0, FX_DEVERR_WAIT_TIMEOUT);
          long long w = 0;  // let a copy already issued for the next tile land before the block exits
          if (staged[st ^ 1] >= 0)
            while (!mbar_try_wait(&bar[st ^ 1], (parity >> (st ^ 1)) & 1u) && ++w < STAGE_SPIN_LIMIT) {
            }
        }
        return;
      }
    } else {
      if (c.live) idle_tile<P32, BY>(sd, c, tile, acc);
      next();
      __syncthreads();  // what next() wrote is read two tiles on, with no barrier between when the next is idle too
    }
    st ^= 1;
  }
  let_next();
  if (dom >= 0) reduce_part(sd, S, acc);
}

// Courant scan of the state as uploaded (the scan at the top of the first
// step). Also used after a host edit of the state.
template <int BY>
__global__ void __launch_bounds__(BX * BY) k_courant_scan(const fx_dev* __restrict__ devs,
                                                         const fx_tile* __restrict__ tiles) {
  constexpr int TY = Tile<BY>::TY;
  __shared__ HydroSmem64<BY, true> S;
  __shared__ fx_dev sd;
  const fx_tile tile = tiles[blockIdx.x];
  if (threadIdx.x == 0 && threadIdx.y == 0) sd = devs[tile.dom];
  __syncthreads();
  const fx_dev& d = sd;
  const int irow = 1 + tile.bx * TX + threadIdx.x, icol = 1 + tile.by * TY + threadIdx.y;
  double dtc = __longlong_as_double(0x7ff0000000000000LL), hm = 0.0;
  if (threadIdx.x < TX && threadIdx.y < TY && irow <= d.nr && icol <= d.nc) {
    const long long gi = fx_ix(d, irow, icol);
    const long long sl = fx_slot(d, d.ctl->steps), pl = fx_pp(d, d.ctl->steps);
    if (d.prec32)
      courant_cell32(d, fmax(0.0, fx_dd_val(d.eta[pl + gi], d.eta_lo[pl + gi])), d.qx_f[pl + gi],
                     d.qy_f[pl + gi], dtc, hm);
    else
      courant_cell(d, fx_rec64(d, sl + gi)[FX_R64_H], d.qx[pl + gi], d.qy[pl + gi], dtc, hm);
  }
  reduce_courant(d, S, dtc, hm);
}

// First row a (0-based) of the forcing table with t[a] > tim
// (common.cpp:195-200), the warp's lanes on 32 rows at a time. Returns -1
// when no row qualifies.
__device__ __forceinline__ int forcing_row(const float* t, double tim) {
  for (int a = 0; a < FX_METEO_ROWS; a += 32) {
    const int q = a + (int)(threadIdx.x & 31);
    const unsigned m = __ballot_sync(0xffffffffu, q < FX_METEO_ROWS && t[q] > tim);
    if (m) return a + __ffs(m) - 1;
  }
  return -1;
}

// The clock update of one step (main.cpp:271-325 and common.cpp:195-208), by
// the 32 lanes of a warp.
__device__ __forceinline__ void finalize_step(const fx_dev& d) {
  fx_ctl& c = *d.ctl;
  const bool lane0 = (threadIdx.x & 31) == 0;
  const double tim0 = c.tim, print_next = c.print_next;
  const long long steps = c.steps + 1;
  if (c.error || c.print_pending || c.finished || steps > c.stop_after) {
    if (lane0) c.live = 0;
    return;
  }
  if (!(tim0 <= c.ntim)) {
    if (lane0) {
      c.live = 0;
      c.finished = 1;
    }
    return;
  }
  const double dtmin = __longlong_as_double((long long)c.acc_dtmin);
  const double hpall = __longlong_as_double((long long)c.acc_hmax);
  double dt = fmin(9.e10, dtmin);
  dt = fmin(print_next - tim0, dt);
  const double tim = tim0 + dt;
  int row = 0, irow = 0;
  bool overrun = false;
  if (d.has_meteo) {
    row = forcing_row(d.meteo_t, tim);
    overrun |= row < 0;
    if (row < 0) row = FX_METEO_ROWS - 1;
  }
  if (d.has_inflow) {
    irow = forcing_row(d.inflow_t, tim);
    overrun |= irow < 0;
    if (irow < 0) irow = FX_METEO_ROWS - 1;
  }
  if (!lane0) return;
  if (overrun) c.forcing_overrun = 1;
  fx_steprec& r = c.rec[steps % d.nslot];
  c.dtfl = r.dtfl = dt;
  c.hpall = hpall;
  c.tim = tim;
  if (d.has_meteo) {
    c.meteo_rate = r.meteo_rate = (double)d.meteo_r[row];
    c.meteoi = r.meteoi = (double)d.meteo_r[row] / (1000. * 3600. * 24.) * dt;
    c.mconc = r.mconc = (double)d.meteo_c[row];
  } else {
    c.meteo_rate = r.meteo_rate = 0.0;
    c.meteoi = r.meteoi = 0.0;
    c.mconc = r.mconc = 0.0;
  }
  if (d.has_inflow) {  // common.cpp:300-311; table rows from 0 (read_functions.cpp:311)
    c.inflowi = r.inflowi = (double)d.inflow_r[irow] * dt / d.arbase;  // / pow(dxy, 2), exact
    c.iconc = r.iconc = (double)d.inflow_c[irow];
  } else {
    c.inflowi = r.inflowi = 0.0;
    c.iconc = r.iconc = 0.0;
  }
  const int active = hpall != 0.0, it = c.it + (active ? 1 : 0);
  c.active = r.active = active;
  c.it = r.it = it;
  c.print_pending = tim >= print_next;
  c.steps = r.step = steps;
  r.inflow_hm = 0.0;
  r.batch = c.batch;
  r.live = 1;
  c.acc_dtmin = (unsigned long long)__double_as_longlong(__longlong_as_double(0x7ff0000000000000LL));
  c.acc_hmax = 0ull;
  c.live = 1;
}

__global__ void __launch_bounds__(32) k_finalize(const fx_dev* __restrict__ devs) {
  let_next();
  follow();
  finalize_step(devs[blockIdx.x]);
}

// Opens a batch of steps whose ADE sweeps run together (fx_ade.cu).
__global__ void k_batch_begin(const fx_dev* __restrict__ devs, int ndom) {
  const int dom = blockIdx.x * blockDim.x + threadIdx.x;
  if (dom >= ndom) return;
  devs[dom].ctl->batch = devs[dom].ctl->batch + 1;
  devs[dom].ctl->ade_next = 0;
}

// Sets the bed flags that never change (NODATA bed) in every slot plane.
// One thread per 4 cells of a column (ld is a multiple of 32, so the 4 share
// the column): the four flags bytes of a slot move as one 32-bit word.
__global__ void k_mark_static(const fx_dev* __restrict__ devs, int dom) {
  const fx_dev& d = devs[dom];
  const long long i = 4 * (blockIdx.x * (long long)blockDim.x + threadIdx.x);
  if (i >= d.plane) return;
  const int icol = (int)(i / d.ld), irow0 = (int)(i - (long long)icol * d.ld) - FX_ROFF;
  if (icol < 1 || icol > d.nc) return;
  const double2 z01 = *reinterpret_cast<const double2*>(d.zb + i);
  const double2 z23 = *reinterpret_cast<const double2*>(d.zb + i + 2);
  const double zb[4] = {z01.x, z01.y, z23.x, z23.y};
  unsigned keep = 0xffffffffu, set = 0u;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int irow = irow0 + j;
    if (irow < 1 || irow > d.nr) continue;
    keep &= ~((unsigned)FX_F_NODATA << (8 * j));
    if (zb[j] == d.nodata) set |= (unsigned)FX_F_NODATA << (8 * j);
  }
  if (keep == 0xffffffffu) return;
  unsigned* f = reinterpret_cast<unsigned*>(d.flags + i);
  const long long step = d.plane / 4;
  for (int k = 0; k < d.nslot; ++k) f[k * step] = (f[k * step] & keep) | set;
}

// FP32 state: the compensated depth (eta, eta_lo) = z - zb over the whole
// grid (ghost ring included), from a staged FP64 z in the field layout, into
// both planes.
__global__ void k_eta_from_z(const __grid_constant__ fx_dev d, const double* __restrict__ z) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < d.plane;
       i += (long long)gridDim.x * blockDim.x) {
    const double depth = z[i] - d.zb[i];
    const float hi = (float)depth;
    d.eta[i] = d.eta[d.plane + i] = hi;
    d.eta_lo[i] = d.eta_lo[d.plane + i] = (float)(depth - (double)hi);
  }
}

// Stored water sum(z - zb) * dxy^2 over the interior cells that are not
// walls (the quantity the update conserves: a cell overdrawn by its
// neighbours' outflow holds a small negative depth until it refills, where h
// reads 0) and solute mass sum(c * h) * dxy^2, FP64 block sums added into
// out[0] and out[1 + k].
__global__ void __launch_bounds__(256) k_mass(const __grid_constant__ fx_dev d, double* __restrict__ out) {
  __shared__ double red[8][1 + FX_MAX_CHEM];
  const long long sl = fx_slot(d, d.ctl->steps), pl = fx_pp(d, d.ctl->steps);
  double acc[1 + FX_MAX_CHEM];
  for (int k = 0; k <= FX_MAX_CHEM; ++k) acc[k] = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < d.plane;
       i += (long long)gridDim.x * blockDim.x) {
    const int icol = (int)(i / d.ld), irow = (int)(i % d.ld) - FX_ROFF;
    if (irow < 1 || irow > d.nr || icol < 1 || icol > d.nc) continue;
    if (d.flags[sl + i] & FX_F_WALL) continue;
    const double h = d.prec32 ? (double)fx_rec(d, sl + i)[FX_R_H] : fx_rec64(d, sl + i)[FX_R64_H];
    acc[0] += d.prec32 ? fx_dd_val(d.eta[pl + i], d.eta_lo[pl + i]) : d.z[pl + i] - d.zb[i];
    for (int k = 0; k < d.nchem; ++k)
      acc[1 + k] += h * (d.prec32 ? (double)d.conc_f[k * d.plane + i] : d.conc[k * d.plane + i]);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int k = 0; k <= d.nchem; ++k) {
    double v = acc[k];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[w][k] = v;
  }
  __syncthreads();
  if (threadIdx.x <= d.nchem) {
    double v = 0.0;
    for (int j = 0; j < 8; ++j) v += red[j][threadIdx.x];
    atomicAdd(&out[threadIdx.x], v * d.arbase);
  }
}

}  // namespace fx

// Launch helpers used by fx_capi.cu and fx_batch.cu. `devs` is a device
// array of ndom domain descriptors; tile tables are built by fx_tiles_of.
// A launch that may start before the one ahead of it in the stream is done
// (see follow(), which every kernel launched so calls first).
template <class... P, class... A>
static void launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
void fx_launch_finalize(const fx_dev* devs, int ndom, cudaStream_t s) {
  launch_after(fx::k_finalize, ndom, 32, 0, s, devs);
}
void fx_launch_batch_begin(const fx_dev* devs, int ndom, cudaStream_t s) {
  fx::k_batch_begin<<<(ndom + 127) / 128, 128, 0, s>>>(devs, ndom);
}
void fx_launch_mark_static(const fx_dev* devs, int dom, long long plane, cudaStream_t s) {
  fx::k_mark_static<<<(unsigned)((plane / 4 + 255) / 256), 256, 0, s>>>(devs, dom);
}
namespace {
template <int BY>
void launch_hydro_batch(const fx_dev* devs, const fx_tile* tiles, int ntiles, bool prec32, cudaStream_t s) {
  if (prec32) launch_after(fx::k_hydro_batch<true, BY>, ntiles, dim3(fx::BX, BY), 0, s, devs, tiles);
  else launch_after(fx::k_hydro_batch<false, BY>, ntiles, dim3(fx::BX, BY), 0, s, devs, tiles);
}
template <int BY>
void launch_hydro_one(const fx_dev& d, cudaStream_t s) {
  const dim3 grid((d.nr + fx::TX - 1) / fx::TX, (d.nc + fx::Tile<BY>::TY - 1) / fx::Tile<BY>::TY);
  if (d.prec32) launch_after(fx::k_hydro_one<true, BY>, grid, dim3(fx::BX, BY), 0, s, d);
  else launch_after(fx::k_hydro_one<false, BY>, grid, dim3(fx::BX, BY), 0, s, d);
}
}  // namespace

bool fx_tile_rows_ok(int r) { return r == 4 || r == 8 || r == 16; }

static long long tiles_of(int nr, int nc, int rows) {
  return (long long)((nr + fx::TX - 1) / fx::TX) * ((nc + rows - 2) / (rows - 1));
}
// The tile shape where none is set, for domains of nr[i] x nc[i] cells.
// * 4 rows while all such tiles are resident at once (5 blocks an SM): a step
//   is then one tile's latency, and the smallest tile's is the shortest
//   (200 x 200 cells FP64 16.3 us against 18.0 with 8 rows, FP32 13.3 against
//   13.8; 257 x 257 FP64, one tile in 20 too many, 22.1 against 20.3).
// * 16 rows in FP32 when every block has ten such tiles or more: fewer halo
//   cells are read and updated (2048 x 2048 cells 0.223 ms against 0.236,
//   1280 x 1280 96 us against 101, 64 domains of 200 x 200 199 us against 204);
//   with eight a block (1024 x 1024) it is 2 % less with water everywhere and
//   5 % more after a dam break. In FP64 they spill (2048 x 2048 0.73 against 0.58 ms).
// * 8 rows otherwise.
int fx_default_tile_rows(bool prec32, const std::vector<int>& nr, const std::vector<int>& nc) {
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 8;
  long long small = 0, large = 0;
  bool staged = true;  // boxes of 16 rows fit every domain
  for (size_t i = 0; i < nr.size(); ++i) {
    small += tiles_of(nr[i], nc[i], 4);
    large += tiles_of(nr[i], nc[i], 16);
    staged &= nc[i] >= 16;
  }
  if (small <= 5LL * nsm) return 4;
  return prec32 && staged && large >= 10LL * fx::min_blocks<true, 16>() * nsm ? 16 : 8;
}

void fx_launch_hydro(const fx_dev* devs, const fx_tile* tiles, int ntiles, bool prec32, int tile_rows,
                     cudaStream_t s) {
  if (tile_rows == 4) launch_hydro_batch<4>(devs, tiles, ntiles, prec32, s);
  else if (tile_rows == 16) launch_hydro_batch<16>(devs, tiles, ntiles, prec32, s);
  else launch_hydro_batch<8>(devs, tiles, ntiles, prec32, s);
}
void fx_launch_hydro_one(const fx_dev& d, cudaStream_t s) {
  if (d.tile_rows == 4) launch_hydro_one<4>(d, s);
  else if (d.tile_rows == 16) launch_hydro_one<16>(d, s);
  else launch_hydro_one<8>(d, s);
}
namespace {
template <int BY>
void launch_hydro_tma(const fx_dev& d, const fx_tmaps& tm, int nblocks, cudaStream_t s) {
  const int ntx = (d.nr + fx::TX - 1) / fx::TX, nty = (d.nc + fx::Tile<BY>::TY - 1) / fx::Tile<BY>::TY;
  const size_t dyn = (size_t)2 * (d.prec32 ? fx::StageLayout<true, BY>::BYTES : fx::StageLayout<false, BY>::BYTES) + 128;
  if (d.prec32) launch_after(fx::k_hydro_tma<true, BY>, nblocks, dim3(fx::BX, BY), dyn, s, d, tm, ntx, nty);
  else launch_after(fx::k_hydro_tma<false, BY>, nblocks, dim3(fx::BX, BY), dyn, s, d, tm, ntx, nty);
}
template <bool P32, int BY>
int tma_blocks(int* out) {
  const size_t dyn = (size_t)2 * fx::StageLayout<P32, BY>::BYTES + 128;
  if (cudaFuncSetAttribute(fx::k_hydro_tma<P32, BY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn) !=
      cudaSuccess)
    return -1;
  int dev = 0, nsm = 0, per = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fx::k_hydro_tma<P32, BY>, fx::BX * BY, dyn) !=
      cudaSuccess)
    return -1;
  *out = per * nsm;
  return 0;
}
}  // namespace

namespace {
template <bool P32, int BY>
size_t batch_tma_dyn() { return (size_t)2 * fx::StageLayout<P32, BY>::BYTES + 128; }
template <int BY>
void launch_hydro_batch_tma(const fx_dev* devs, const fx_tmaps* tms, const fx_tile* tiles, int ntiles, int nblocks,
                            bool prec32, cudaStream_t s) {
  if (prec32)
    launch_after(fx::k_hydro_batch_tma<true, BY>, nblocks, dim3(fx::BX, BY), batch_tma_dyn<true, BY>(), s, devs, tms, tiles, ntiles);
  else
    launch_after(fx::k_hydro_batch_tma<false, BY>, nblocks, dim3(fx::BX, BY), batch_tma_dyn<false, BY>(), s, devs, tms, tiles, ntiles);
}
template <bool P32, int BY>
int batch_tma_blocks(int* out) {
  const size_t dyn = batch_tma_dyn<P32, BY>();
  if (cudaFuncSetAttribute(fx::k_hydro_batch_tma<P32, BY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn) !=
      cudaSuccess)
    return -1;
  int dev = 0, nsm = 0, per = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fx::k_hydro_batch_tma<P32, BY>, fx::BX * BY, dyn) !=
      cudaSuccess)
    return -1;
  *out = per * nsm;
  return 0;
}
}  // namespace

// The TMA-staged persistent hydrodynamic launch of a batch: `tms` holds one
// set of tensor maps per domain, built for `tile_rows`.
void fx_launch_hydro_batch_tma(const fx_dev* devs, const fx_tmaps* tms, const fx_tile* tiles, int ntiles,
                               int nblocks, bool prec32, int tile_rows, cudaStream_t s) {
  if (tile_rows == 4) launch_hydro_batch_tma<4>(devs, tms, tiles, ntiles, nblocks, prec32, s);
  else if (tile_rows == 16) launch_hydro_batch_tma<16>(devs, tms, tiles, ntiles, nblocks, prec32, s);
  else launch_hydro_batch_tma<8>(devs, tms, tiles, ntiles, nblocks, prec32, s);
}
int fx_hydro_batch_tma_blocks(bool prec32, int tile_rows, int* out) {
  if (tile_rows == 4) return prec32 ? batch_tma_blocks<true, 4>(out) : batch_tma_blocks<false, 4>(out);
  if (tile_rows == 16) return prec32 ? batch_tma_blocks<true, 16>(out) : batch_tma_blocks<false, 16>(out);
  return prec32 ? batch_tma_blocks<true, 8>(out) : batch_tma_blocks<false, 8>(out);
}

void fx_launch_hydro_tma(const fx_dev& d, const fx_tmaps& tm, int nblocks, cudaStream_t s) {
  if (d.tile_rows == 4) launch_hydro_tma<4>(d, tm, nblocks, s);
  else if (d.tile_rows == 16) launch_hydro_tma<16>(d, tm, nblocks, s);
  else launch_hydro_tma<8>(d, tm, nblocks, s);
}

// Resident blocks of the TMA-staged hydrodynamic kernel (after raising its
// dynamic shared memory limit); the persistent grid is at most this.
int fx_hydro_tma_blocks(bool prec32, int tile_rows, int* out) {
  if (tile_rows == 4) return prec32 ? tma_blocks<true, 4>(out) : tma_blocks<false, 4>(out);
  if (tile_rows == 16) return prec32 ? tma_blocks<true, 16>(out) : tma_blocks<false, 16>(out);
  return prec32 ? tma_blocks<true, 8>(out) : tma_blocks<false, 8>(out);
}

void fx_launch_courant_scan(const fx_dev* devs, const fx_tile* tiles, int ntiles, int tile_rows, cudaStream_t s) {
  if (tile_rows == 4) fx::k_courant_scan<4><<<ntiles, dim3(fx::BX, 4), 0, s>>>(devs, tiles);
  else if (tile_rows == 16) fx::k_courant_scan<16><<<ntiles, dim3(fx::BX, 16), 0, s>>>(devs, tiles);
  else fx::k_courant_scan<8><<<ntiles, dim3(fx::BX, 8), 0, s>>>(devs, tiles);
}
void fx_launch_eta_from_z(const fx_dev& d, const double* z, cudaStream_t s) {
  fx::k_eta_from_z<<<592, 256, 0, s>>>(d, z);
}
void fx_launch_mass(const fx_dev& d, double* out, cudaStream_t s) { fx::k_mass<<<296, 256, 0, s>>>(d, out); }
// Appends the tiles of domain `dom` (nr x nc interior cells) to a table.
void fx_tiles_of(int dom, int nr, int nc, int tile_rows, std::vector<fx_tile>& out) {
  const int ty = tile_rows - 1;
  const int gx = (nr + fx::TX - 1) / fx::TX, gy = (nc + ty - 1) / ty;
  for (int by = 0; by < gy; ++by)
    for (int bx = 0; bx < gx; ++bx) out.push_back(fx_tile{dom, bx, by, 0});
}
