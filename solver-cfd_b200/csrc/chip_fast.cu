// chip_fast.cu -- the on-chip engine with FAST arithmetic (the forms of points_fast.cuh).
#include "chip_engine.cuh"

namespace acs {

// Value carried over a face by the flux f (points_fast.cuh: quick_face, upw_face) as k.a * upwind +
// k.b * downwind + k.c * far upwind node; the operands are selected before the products.
struct FaceK { double a, b, c; };
__device__ __forceinline__ FaceK face_k(bool quick) { return {quick ? 0.75 : 1.0, quick ? 0.375 : 0.0, quick ? -0.125 : 0.0}; }
__device__ __forceinline__ double face(const FaceK& k, double f, double up2, double up, double dn, double dn2) {
  const bool pos = f > 0.0;
  return fma(k.a, pos ? up : dn, fma(k.b, pos ? dn : up, k.c * (pos ? up2 : dn2)));
}

struct ChipFast {
  static __device__ void constants(const CaseDev&, double*) {}
  static __device__ __forceinline__ double buoy(const ChipCtx&, double T0, double T1) { return 1.0 - 2.0 / (T0 + T1); }
  // RESU and RESV at a node: U, V the stage inputs, ut, vt the tau arrays, p the pressure, each at the
  // node (neighbours at +-1 and +-P)
  template <bool QUICK>
  static __device__ __forceinline__ void uv(const ChipCtx& x, const ChipNode& n, const double* U, const double* V,
                                            const double* ut, const double* vt, const double* p, double w, double& Ru,
                                            double& Rv) {
    const CaseDev& d = x.d;
    const int P = x.P;
    const double e = n.por ? d.phi : 1.0, ie = n.por ? d.fc[FC_IPHI] : 1.0;
    const double er = e * d.fc[FC_IRE], pP = p[0], rr = n.xd.rd * n.yd.rd;
    {
      const double uP = U[0], uW = U[-1], uE = U[1], uS = U[-P], uN = U[P];
      const double hx = 0.5 * n.xd.d * ie, hy = 0.5 * n.ym.d * ie;
      const double fn = (vt[P] + vt[P - 1]) * hx, fs = (vt[0] + vt[-1]) * hx, fe = (uE + uP) * hy, fw = (uP + uW) * hy;
      double cw, ce, cs, cn;
      if (QUICK) {
        const FaceK q = face_k(n.j >= 3 && n.j <= d.ny - 2);
        cw = face(q, fw, U[-2], uW, uP, uE);
        ce = face(q, fe, uW, uP, uE, U[2]);
        cs = face(q, fs, U[-2 * P], uS, uP, uN);
        cn = face(q, fn, uS, uP, uN, U[2 * P]);
      } else {
        cw = fw > 0.0 ? uW : uP;
        ce = fe > 0.0 ? uP : uE;
        cs = fs > 0.0 ? uS : uP;
        cn = fn > 0.0 ? uP : uN;
      }
      const double conv = fw * cw - fe * ce + fs * cs - fn * cn;
      const double diff = er * (n.xd.d * (n.yn.rd * (uN - uP) - n.yd.rd * (uP - uS)) +
                                n.ym.d * (n.xm.rd * (uE - uP) - n.xw.rd * (uP - uW)));
      Ru = rr * (conv + diff) - e * (pP - p[-1]) * n.xd.rd - d.g * e;
    }
    {
      const double vP = V[0], vW = V[-1], vE = V[1], vS = V[-P], vN = V[P];
      const double hx = 0.5 * n.xm.d * ie, hy = 0.5 * n.yd.d * ie;
      const double fn = (vP + vN) * hx, fs = (vP + vS) * hx, fe = (ut[1] + ut[1 - P]) * hy, fw = (ut[0] + ut[-P]) * hy;
      double cw, ce, cs, cn;
      if (QUICK) {
        const FaceK q = face_k(n.i >= 3 && n.i <= d.nx - 2);
        cw = face(q, fw, V[-2], vW, vP, vE);
        ce = face(q, fe, vW, vP, vE, V[2]);
        cs = face(q, fs, V[-2 * P], vS, vP, vN);
        cn = face(q, fn, vS, vP, vN, V[2 * P]);
      } else {
        cw = fw > 0.0 ? vW : vP;
        ce = fe > 0.0 ? vP : vE;
        cs = fs > 0.0 ? vS : vP;
        cn = fn > 0.0 ? vP : vN;
      }
      const double conv = fw * cw - fe * ce + fs * cs - fn * cn;
      const double diff = er * (n.xm.d * (n.ym.rd * (vN - vP) - n.ys.rd * (vP - vS)) +
                                n.yd.d * (n.xe.rd * (vE - vP) - n.xd.rd * (vP - vW)));
      Rv = rr * (conv + diff) - e * (pP - p[-P]) * n.yd.rd + d.InvFr2 * w;
    }
    if (n.por) {
      const double uP = U[0], vu = vt[0], uv = ut[0], vP = V[0];
      Ru -= e * uP * (d.fc[FC_IREDA] + d.fc[FC_CFS] * sqrt(fma(uP, uP, vu * vu)));
      Rv -= e * vP * (d.fc[FC_IREDA] + d.fc[FC_CFS] * sqrt(fma(uv, uv, vP * vP)));
    }
  }
  // RESZ and RESC at a node; ee, en: the neighbour at i+1, j+1 is the extrapolated boundary
  static __device__ __forceinline__ void tc(const ChipCtx& x, const ChipNode& n, bool ee, bool en, const double* un, const double* vn,
                                            const double* t, const double* c, double& Rt, double& Rc) {
    const CaseDev& d = x.d;
    const int P = x.P;
    const double ue = 0.5 * n.ym.d * un[1], uw = 0.5 * n.ym.d * un[0], vN = 0.5 * n.xm.d * vn[P], vS = 0.5 * n.xm.d * vn[0];
    const double ax = n.ym.d * n.xe.rd, bx = n.ym.d * n.xd.rd, ay = n.xm.d * n.yn.rd, by = n.xm.d * n.yd.rd;
    const double rr = n.xm.rd * n.ym.rd, icap = n.por ? d.fc[FC_IPHI] : 1.0;
    auto res = [&](const double* z, double k, double& conv, double& diff) {
      const double zp = z[0], zw = z[-1], zs = z[-P];
      const double ze = ee ? zp + (zp - zw) : z[1], zn = en ? zp + (zp - zs) : z[P];
      conv = (ze + zp) * ue - (zw + zp) * uw + (zn + zp) * vN - (zs + zp) * vS;
      diff = k * (ax * (ze - zp) - bx * (zp - zw) + ay * (zn - zp) - by * (zp - zs));
    };
    double conv, diff;
    res(t, d.fc[FC_IPE], conv, diff);
    Rt = rr * ((diff - (n.por ? 0.0 : conv)) * icap);
    res(c, d.fc[FC_IRESC], conv, diff);
    Rc = rr * (diff - conv * icap);
  }
  // solve_P at one node: with RP frozen the three stages give pn = p + dtau*beta*RP
  static __device__ __forceinline__ double p_update(const ChipCtx& x, const ChipNode& n, double p0, const double* un,
                                                    const double* vn, double* r) {
    double RP = -((un[1] - un[0]) * n.ym.d + (vn[x.P] - vn[0]) * n.xm.d);
    if (x.d.continuity == 1) RP *= n.xm.rd * n.ym.rd;
    *r = x.d.fc[FC_DTB] * RP;
    return p0 + *r;
  }
};

namespace {
using PT = ChipFast;
}  // namespace
#define CHIP_LAUNCH launch_chip_fast
#define CHIP_RESIDENT chip_resident_fast
#include "chip_launch.inl"

}  // namespace acs
