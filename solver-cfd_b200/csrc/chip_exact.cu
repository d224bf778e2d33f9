// chip_exact.cu -- the on-chip engine with the reference's exact arithmetic: every product, sum and
// quotient is rounded as in the reference's expressions (the file is built with -fmad=false), so the
// results are bit-identical to points_exact.cuh and to the CPU oracle.
//
// What differs from points_exact.cuh is how quotients are found, not their values:
//   * a quotient by a metric difference, a porosity or another constant of the case is computed from
//     the constant's correctly rounded reciprocal (exact_div), five dependent FP64 instructions instead
//     of a division routine of about 114 cycles;
//   * a quotient by a porosity of 1 and, unless it has overflowed, the drag of a node without porous
//     structure (a product with 0) are left out.
// Reference (OpenMp_Multicore/): RESU equations.f90:2-116 (+ upwind_Ui/Uj :120-240), RESV :305-420
// (+ upwind_Vi/Vj :423-542), solve_P :607-665, RESZ :723-765, RESC :823-867.
#include "chip_engine.cuh"

namespace acs {

// RN(a / b) from z = RN(1 / b).  a*z is within two units in the last place of a/b; one residual step
// makes it faithful, and by Markstein's theorem (P. Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990) a residual step on a faithful
// quotient with a correctly rounded reciprocal gives the correctly rounded one, while nothing
// underflows or overflows.  b is in [2^-60, 2^60] (chip_divisors), a in [2^-900, 2^900) in magnitude.
__device__ __forceinline__ double const_div(double a, double b, double z) {  // a a constant in range
  double q = a * z;
  q = __fma_rn(__fma_rn(-b, q, a), z, q);
  return __fma_rn(__fma_rn(-b, q, a), z, q);
}
// The same for any a; `bad` is set when the result may be wrong (the node is then computed again with
// plain divisions).  The sign is restored for a = -0.
__device__ __forceinline__ double exact_div(double a, double b, double z, bool& bad) {
  const double q = const_div(a, b, z);
  const int ha = __double2hiint(a);
  bad |= (unsigned)(ha & 0x7ff00000) - (123u << 20) >= (1800u << 20) && ((ha << 1) | __double2loint(a)) != 0;
  return __hiloint2double(__double2hiint(q) | (ha & 0x80000000), __double2loint(q));
}

__device__ __forceinline__ double pos_part(double a) { return a > 0.0 ? a : 0.0; }

__device__ __noinline__ double plain_quotient(double a, double b) { return a / b; }

struct ChipExact {
  enum { K_IPHI, K_E1RE, K_EPRE, K_REDA, K_IREDA, K_CFS, K_KT, K_KC, K_CAP, K_ICAP };
  // constants of the case, each the value that the reference's expression has
  static __device__ void constants(const CaseDev& d, double* k) {
    k[K_IPHI] = 1.0 / d.phi;
    k[K_E1RE] = 1.0 / d.Re;
    k[K_EPRE] = d.phi / d.Re;
    k[K_REDA] = d.Re * d.Da;
    k[K_IREDA] = 1.0 / k[K_REDA];
    k[K_CFS] = d.Cf / sqrt(d.phi * d.Da);
    k[K_KT] = 1.0 / d.Pe;
    k[K_KC] = 1.0 / d.Re / d.Sc;
    k[K_CAP] = 1.0 * (d.phi - 1.0) + 1.0;
    k[K_ICAP] = 1.0 / k[K_CAP];
  }
  static __device__ __forceinline__ double buoy(const ChipCtx& x, double T0, double T1) {
    return x.d.InvFr2 * (1.0 - 1.0 / ((T0 + T1) * 0.5));
  }
  // Arithmetic of one node with fast quotients (SAFE = false; sets bad) or plain ones.
  template <bool SAFE>
  static __device__ __forceinline__ double quo(double a, double b, double z, bool& bad) {
    return SAFE ? a / b : exact_div(a, b, z, bad);
  }
  // -(ap*c) + sum of the neighbours (QUICK and upwind coefficients of equations.f90:44-70, :146-160).
  // The alpha flags are 0 or 1: coefficient * flag is selected, and its product with the flux kept.
  template <bool QUICK>
  static __device__ __forceinline__ double balance(bool quick, double fw, double fe, double fs, double fn, double Dw,
                                                   double De, double Ds, double Dn, const double* f, int P) {
    const double df = fe - fw + fn - fs;
    const double c = f[0], W = f[-1], E = f[1], S = f[-P], N = f[P];
    if (QUICK && quick) {
      const bool pw = fw > 0.0, pe = fe > 0.0, ps = fs > 0.0, pn = fn > 0.0;
      const double w75 = (pw ? 0.75 : 0.0) * fw, w37 = (pw ? 0.0 : 0.375) * fw, w12 = (pw ? 0.0 : 0.125) * fw;
      const double e12 = (pe ? 0.125 : 0.0) * fe, e37 = (pe ? 0.375 : 0.0) * fe, e75 = (pe ? 0.0 : 0.75) * fe;
      const double s75 = (ps ? 0.75 : 0.0) * fs, s37 = (ps ? 0.0 : 0.375) * fs, s12 = (ps ? 0.0 : 0.125) * fs;
      const double n12 = (pn ? 0.125 : 0.0) * fn, n37 = (pn ? 0.375 : 0.0) * fn, n75 = (pn ? 0.0 : 0.75) * fn;
      const double aw = Dw + w75 + e12 + w37, ae = De - e37 - e75 - w12;
      const double as = Ds + s75 + n12 + s37, an = Dn - n37 - n75 - s12;
      const double aww = (pw ? -0.125 : -0.0) * fw, aee = (pe ? 0.0 : 0.125) * fe;
      const double ass = (ps ? -0.125 : -0.0) * fs, ann = (pn ? 0.0 : 0.125) * fn;
      const double ap = aw + ae + as + an + aww + aee + ass + ann + df;
      return -(ap * c) + aww * f[-2] + aw * W + aee * f[2] + ae * E + ass * f[-2 * P] + as * S +
             ann * f[2 * P] + an * N;
    }
    const double aw = Dw + pos_part(fw), as = Ds + pos_part(fs), ae = De + pos_part(-fe), an = Dn + pos_part(-fn);
    const double ap = aw + ae + as + an + df;
    return -(ap * c) + aw * W + ae * E + as * S + an * N;
  }
  template <bool SAFE>
  static __device__ __forceinline__ void by_porosity(const ChipCtx& x, double& a, double& b, double& c, double& e, bool& bad) {
    a = quo<SAFE>(a, x.d.phi, x.k[K_IPHI], bad);
    b = quo<SAFE>(b, x.d.phi, x.k[K_IPHI], bad);
    c = quo<SAFE>(c, x.d.phi, x.k[K_IPHI], bad);
    e = quo<SAFE>(e, x.d.phi, x.k[K_IPHI], bad);
  }
  // r minus the Darcy-Forchheimer drag of velocity a at a node with velocity (u, v).  Without porous structure
  // the reference multiplies the drag with liga = 0: nothing, or NaN where it has overflowed, which takes
  // u*u + v*v above 2^600 (chip_divisors and Cf); such a node is computed in full.
  template <bool SAFE>
  static __device__ __forceinline__ double drag(const ChipCtx& x, double r, double a, double u, double v, bool por, bool& bad) {
    const double s = u * u + v * v;
    if (por)
      return r - x.d.phi * (quo<SAFE>(a, x.k[K_REDA], x.k[K_IREDA], bad) + x.k[K_CFS] * a * sqrt(s)) * 1.0;
    if (SAFE) return r - 1.0 * (a / x.k[K_REDA] + x.d.Cf / sqrt(1.0 * x.d.Da) * a * sqrt(s)) * 0.0;
    bad |= (unsigned)__double2hiint(s) >= (1023u + 600u) << 20;
    return r;
  }
  // RESU and RESV at a node: U, V the stage inputs, ut, vt the tau arrays, p the pressure, each at the
  // node (neighbours at +-1 and +-P)
  template <bool QUICK, bool SAFE>
  static __device__ __forceinline__ double ru_t(const ChipCtx& x, const ChipNode& n, const double* U, const double* vt,
                                                const double* p, bool& bad) {
    const CaseDev& d = x.d;
    const int P = x.P;
    const double e = n.por ? d.phi : 1.0, eRe = n.por ? x.k[K_EPRE] : x.k[K_E1RE];
    const double uP = U[0], vP = vt[0];
    double fn = 0.5 * (vt[P] + vt[P - 1]) * n.xd.d, fs = 0.5 * (vP + vt[-1]) * n.xd.d;
    double fe = 0.5 * (U[1] + uP) * n.ym.d, fw = 0.5 * (uP + U[-1]) * n.ym.d;
    if (n.por) by_porosity<SAFE>(x, fn, fs, fe, fw, bad);
    const double Dn = const_div(eRe * n.xd.d, n.yn.d, n.yn.rd), Ds = const_div(eRe * n.xd.d, n.yd.d, n.yd.rd);
    const double De = const_div(eRe * n.ym.d, n.xm.d, n.xm.rd), Dw = const_div(eRe * n.ym.d, n.xw.d, n.xw.rd);
    const double q_art = quo<SAFE>(e * (p[0] - p[-1]), n.xd.d, n.xd.rd, bad);
    double r = const_div(n.xd.rd, n.yd.d, n.yd.rd) *
                   balance<QUICK>(n.j >= 3 && n.j <= d.ny - 2, fw, fe, fs, fn, Dw, De, Ds, Dn, U, P) - q_art;
    if (d.flags & F_POROUS) r = drag<SAFE>(x, r, uP, uP, vP, n.por, bad);
    return r - d.g * e;
  }
  template <bool QUICK, bool SAFE>
  static __device__ __forceinline__ double rv_t(const ChipCtx& x, const ChipNode& n, const double* ut, const double* V,
                                                const double* p, double w, bool& bad) {
    const CaseDev& d = x.d;
    const int P = x.P;
    const double e = n.por ? d.phi : 1.0, eRe = n.por ? x.k[K_EPRE] : x.k[K_E1RE];
    const double vP = V[0], uP = ut[0];
    double fn = 0.5 * (vP + V[P]) * n.xm.d, fs = 0.5 * (vP + V[-P]) * n.xm.d;
    double fe = 0.5 * (ut[1] + ut[1 - P]) * n.yd.d, fw = 0.5 * (uP + ut[-P]) * n.yd.d;
    if (n.por) by_porosity<SAFE>(x, fn, fs, fe, fw, bad);
    const double Dn = const_div(eRe * n.xm.d, n.ym.d, n.ym.rd), Ds = const_div(eRe * n.xm.d, n.ys.d, n.ys.rd);
    const double De = const_div(eRe * n.yd.d, n.xe.d, n.xe.rd), Dw = const_div(eRe * n.yd.d, n.xd.d, n.xd.rd);
    const double q_art = quo<SAFE>(e * (p[0] - p[-P]), n.yd.d, n.yd.rd, bad);
    double r = const_div(n.xd.rd, n.yd.d, n.yd.rd) *
                   balance<QUICK>(n.i >= 3 && n.i <= d.nx - 2, fw, fe, fs, fn, Dw, De, Ds, Dn, V, P) - q_art;
    if (d.flags & F_BUOY) r = r + w;
    if (d.flags & F_POROUS) r = drag<SAFE>(x, r, vP, uP, vP, n.por, bad);
    return r;
  }
  // The rare nodes whose operands leave the fast quotients' range.
  template <bool QUICK>
  static __device__ __noinline__ double2 uv_safe(ChipCtx x, ChipNode n, const double* U, const double* V, const double* ut,
                                                 const double* vt, const double* p, double w) {
    bool bad = false;
    return make_double2(ru_t<QUICK, true>(x, n, U, vt, p, bad), rv_t<QUICK, true>(x, n, ut, V, p, w, bad));
  }
  template <bool QUICK>
  static __device__ __forceinline__ void uv(const ChipCtx& x, const ChipNode& n, const double* U, const double* V,
                                            const double* ut, const double* vt, const double* p, double w, double& Ru,
                                            double& Rv) {
    bool bad = false;
    Ru = ru_t<QUICK, false>(x, n, U, vt, p, bad);
    Rv = rv_t<QUICK, false>(x, n, ut, V, p, w, bad);
    if (bad) {
      const double2 R = uv_safe<QUICK>(x, n, U, V, ut, vt, p, w);
      Ru = R.x;
      Rv = R.y;
    }
  }
  // RESZ (k = 1/Pe) or RESC (k = 1/Re/Sc) at a node; ee, en: the neighbour at i+1, j+1 is the
  // extrapolated boundary
  template <bool IS_C>
  static __device__ __forceinline__ double rs(const ChipCtx& x, const ChipNode& n, bool ee, bool en, const double* un, const double* vn,
                                              const double* z) {
    const int P = x.P;
    const double k = x.k[IS_C ? K_KC : K_KT];
    const double zp = z[0], zw = z[-1], zs = z[-P];
    const double ze = ee ? zp + 1.0 * (zp - zw) : z[1], zn = en ? zp + 1.0 * (zp - zs) : z[P];
    const double dzu = 0.5 * (ze + zp) * un[1] * n.ym.d - 0.5 * (zw + zp) * un[0] * n.ym.d;
    const double dzv = 0.5 * (zn + zp) * vn[P] * n.xm.d - 0.5 * (zs + zp) * vn[0] * n.xm.d;
    const double De = const_div(n.ym.d * k, n.xe.d, n.xe.rd), Dw = const_div(n.ym.d * k, n.xd.d, n.xd.rd);
    const double Dn = const_div(n.xm.d * k, n.yn.d, n.yn.rd), Ds = const_div(n.xm.d * k, n.yd.d, n.yd.rd);
    const double Dp = De + Dw + Dn + Ds;
    const double pre = const_div(n.xm.rd, n.ym.d, n.ym.rd), sum = -(Dp * zp) + De * ze + Dw * zw + Dn * zn + Ds * zs;
    const double cv = dzu + dzv;
    if (!n.por) return pre * (sum - cv);  // a porosity of 1: (1 - liga) = 1, capacity 1
    bool bad = false;
    const double a = IS_C ? cv : pre * (sum - 0.0 * cv);
    double c = exact_div(a, x.k[K_CAP], x.k[K_ICAP], bad);
    if (bad) c = plain_quotient(a, x.k[K_CAP]);
    return IS_C ? pre * (sum - c) : c;
  }
  static __device__ __forceinline__ void tc(const ChipCtx& x, const ChipNode& n, bool ee, bool en, const double* un, const double* vn,
                                            const double* t, const double* c, double& Rt, double& Rc) {
    Rt = rs<false>(x, n, ee, en, un, vn, t);
    Rc = rs<true>(x, n, ee, en, un, vn, c);
  }
  // solve_P's three stages at one node (equations.f90:620-662); *r = dtau*RP*beta
  static __device__ __forceinline__ double p_update(const ChipCtx& x, const ChipNode& n, double p0, const double* un,
                                                    const double* vn, double* r) {
    const CaseDev& d = x.d;
    const double dudx = un[1] * n.ym.d - un[0] * n.ym.d;
    const double dvdy = vn[x.P] * n.xm.d - vn[0] * n.xm.d;
    double RP = -(dudx + dvdy);
    if (d.continuity == 1) RP = RP / (n.ym.d * n.xm.d);
    const double pi1 = p0 + d.dtau * RP * d.beta;
    const double pi2 = 0.75 * p0 + 0.25 * (pi1 + d.dtau * RP * d.beta);
    *r = d.dtau * RP * d.beta;
    return 1.0 / 3.0 * p0 + 2.0 / 3.0 * (pi2 + *r);
  }
};

namespace {
using PT = ChipExact;
}  // namespace
#define CHIP_LAUNCH launch_chip_exact
#define CHIP_RESIDENT chip_resident_exact
#include "chip_launch.inl"

}  // namespace acs
