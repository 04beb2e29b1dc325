// nodemath.cuh -- the fused path's per-node arithmetic (collision + Recolor,
// Source1.f90:599-732) over a value type V: double, or F2, two nodes' FP32
// values in one register pair (one instruction does both: FP32 arithmetic is
// bound by instruction issue, not by the FP32 units).
//
// The 19x19 moment transform of the reference is factored through the sums
// and differences of opposite populations: an even row of M sees only
// f_i + f_opc(i), an odd row only f_i - f_opc(i), and within each kind the
// rows are combinations of the same three axis sums and three face sums.  That
// takes about a third of the operations of the rows written out pair by pair
// (256x256x256 FP64 collide 2260 -> 2060 us together with the curvature's six
// sums, the split normals and one reciprocal square root per normal; what bounds
// it now is the latency of its loads at 16 warps per SM, the FP64 pipe is 25 %
// busy).
#pragma once
#include "lattice.cuh"

namespace symb200 {
namespace fused {

__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }

struct F2 {
  float2 v;
  __device__ __forceinline__ F2() {}
  __device__ __forceinline__ explicit F2(float a) : v(make_float2(a, a)) {}
  __device__ __forceinline__ F2(float a, float b) : v(make_float2(a, b)) {}
  __device__ __forceinline__ explicit F2(float2 a) : v(a) {}
  __device__ __forceinline__ float operator[](int k) const { return k ? v.y : v.x; }
};
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) { return F2(__ffma2_rn(a.v, b.v, c.v)); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return F2(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return F2(__fmul2_rn(a.v, b.v)); }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return vfma(b, F2(-1.0f), a); }

// Moments of one node in the order of the reference's M (density and momentum
// first): what a node holds between its loads and its pushes.
template <typename V>
struct Moments {
  V rho, jx, jy, jz;
  V e, eps, pxx, pixx, pww, piww, pxy, pyz, pxz;
  V qx, qy, qz, mx, my, mz;
};

template <typename V, typename R>
__device__ __forceinline__ void to_moments(const V (&f)[19], Moments<V>& m) {
  auto k = [](double v) { return V(R(v)); };
  // axis pairs
  const V X = f[1] + f[2], Y = f[3] + f[4], Z = f[5] + f[6];
  const V dx = f[1] - f[2], dy = f[3] - f[4], dz = f[5] - f[6];
  // face diagonals: (+,+) and (+,-) pairs of each face
  const V a = f[7] + f[10], b = f[8] + f[9], c = f[11] + f[14], d = f[12] + f[13], g = f[15] + f[18],
          h = f[16] + f[17];
  const V ao = f[7] - f[10], bo = f[8] - f[9], co = f[11] - f[14], od = f[12] - f[13], go = f[15] - f[18],
          ho = f[16] - f[17];
  const V sxy = a + b, sxz = c + d, syz = g + h;
  m.pxy = a - b; m.pxz = c - d; m.pyz = g - h;
  const V A = X + Y + Z, D = sxy + sxz + syz;
  m.rho = f[0] + A + D;
  m.e = vfma(k(-30), f[0], vfma(k(-11), A, k(8) * D));
  m.eps = vfma(k(12), f[0], vfma(k(-4), A, D));
  // the stresses from differences of nearly equal sums, which are exact near
  // equilibrium (3 X - (X + Y + Z) would carry the rounding of the sum)
  const V p1 = (X - Y) + (X - Z), p2 = (sxy - syz) + (sxz - syz);
  m.pxx = p1 + p2;
  m.pixx = vfma(k(-2), p1, p2);
  const V w1 = Y - Z, w2 = sxy - sxz;
  m.pww = w1 + w2;
  m.piww = vfma(k(-2), w1, w2);
  // odd: the x, y and z components of the face diagonals
  const V x1 = ao - bo, y1 = ao + bo, x2 = co - od, z1 = co + od, y2 = go - ho, z2 = go + ho;
  const V x12 = x1 + x2, y12 = y1 + y2, z12 = z1 + z2;
  m.jx = dx + x12; m.jy = dy + y12; m.jz = dz + z12;
  m.qx = vfma(k(-4), dx, x12); m.qy = vfma(k(-4), dy, y12); m.qz = vfma(k(-4), dz, z12);
  m.mx = x1 - x2; m.my = y2 - y1; m.mz = z1 - z2;
}

// Reciprocal density and relaxation rates of a node (:674-684).  FP64 takes
// one division for all three quotients.
template <typename R>
__device__ __forceinline__ void node_rates_fused(const TileParams<R>& P, R phi, R rho, R& irho, R& su, R& sq) {
  const NodeParams<R>& q = P.np;
  if (P.same_nu) {
    irho = qdiv<R>(R(1), rho);
    su = q.su;
    sq = q.sq;
    return;
  }
  const R ph = fmin(fmax(phi, R(-1)), R(1));
  const R D = (R(1) + ph) * q.inu_r + (R(1) - ph) * q.inu_b;
  const R a = R(12) + D, b = R(16) + D;
  if constexpr (sizeof(R) == 8) {
    const R ab = a * b, t = R(1) / (rho * ab), rt = rho * t;
    irho = ab * t;
    su = R(2) * D * b * rt;
    sq = R(32) * a * rt;
  } else {
    irho = qdiv<R>(R(1), rho);
    su = qdiv<R>(R(2) * D, a);
    sq = qdiv<R>(R(32), b);
  }
}

// Relaxation with Guo forcing (:686): m - s (m - meq) + (1 - s/2) fk per row, the
// equilibrium and forcing moments of equilf (:397-450).  Density and momentum
// relax with rate 1: meq + fk/2.  u already carries half the force.
// m may hold the moments of f - w rho_ref for any rho_ref (w rho_ref is the rest
// equilibrium, its own fixed point); rho is the node's whole density.
template <typename V, typename R>
__device__ __forceinline__ void relax(Moments<V>& m, V rho, V ux, V uy, V uz, V fx, V fy, V fz, V su, V se, V seps,
                                      V sq, V spi, V sm) {
  auto k = [](double v) { return V(R(v)); };
  const V rx = rho * ux, ry = rho * uy, rz = rho * uz;
  const V xx = rx * ux, yy = ry * uy, zz = rz * uz;
  const V yz = yy + zz, us = xx + yz;                         // rho u^2
  const V gx = ux * fx, gy = uy * fy, gz = uz * fz;
  const V gyz = gy + gz, uf = gx + gyz;
  const V one = k(1), half = k(-0.5);
  const V hu = vfma(half, su, one), he = vfma(half, se, one), hp = vfma(half, seps, one), hq = vfma(half, sq, one),
          hi = vfma(half, spi, one);
  // row = row + s (eq - row) + h fk
  auto row = [](V& v, V s, V eq, V h, V fk) { v = vfma(s, eq - v, vfma(h, fk, v)); };
  row(m.e, se, vfma(k(19), us, k(-11) * m.rho), he, k(38) * uf);
  row(m.eps, seps, vfma(k(-5.5), us, k(3) * m.rho), hp, k(-11) * uf);
  const V exx = vfma(k(2), xx, k(-1) * yz), fxx = vfma(k(4), gx, k(-2) * gyz);
  row(m.pxx, su, exx, hu, fxx);
  row(m.pixx, spi, half * exx, half * hi, fxx);
  const V eww = yy - zz, fww = k(2) * (gy - gz);
  row(m.pww, su, eww, hu, fww);
  row(m.piww, spi, half * eww, half * hi, fww);
  row(m.pxy, su, rx * uy, hu, vfma(ux, fy, uy * fx));
  row(m.pyz, su, ry * uz, hu, vfma(uy, fz, uz * fy));
  row(m.pxz, su, rx * uz, hu, vfma(ux, fz, uz * fx));
  // q: eq = -2/3 rho u, fk = -2/3 f
  const V hqt = hq * k(-2.0 / 3.0), nq = k(-1) * sq, c = k(2.0 / 3.0);
  m.qx = vfma(nq, vfma(c, rx, m.qx), vfma(hqt, fx, m.qx));
  m.qy = vfma(nq, vfma(c, ry, m.qy), vfma(hqt, fy, m.qy));
  m.qz = vfma(nq, vfma(c, rz, m.qz), vfma(hqt, fz, m.qz));
  const V om = one - sm;
  m.mx = om * m.mx; m.my = om * m.my; m.mz = om * m.mz;
  m.jx = vfma(k(0.5), fx, rx); m.jy = vfma(k(0.5), fy, ry); m.jz = vfma(k(0.5), fz, rz);
}

// f = M^-1 m, M_inv(i,r) = M(r,i) / |M(r,:)|^2
template <typename V, typename R>
__device__ __forceinline__ void from_moments(const Moments<V>& m, V (&f)[19]) {
  auto k = [](double v) { return V(R(v)); };
  const V r19 = k(1.0 / 19.0) * m.rho;
  const V ka = vfma(k(-11.0 / 2394.0), m.e, vfma(k(-4.0 / 252.0), m.eps, r19));
  const V kd = vfma(k(8.0 / 2394.0), m.e, vfma(k(1.0 / 252.0), m.eps, r19));
  f[0] = vfma(k(-30.0 / 2394.0), m.e, vfma(k(12.0 / 252.0), m.eps, r19));
  // even parts: axes, then the (+,+) and (+,-) diagonals of each face
  const V t = m.pxx - m.pixx, w = m.pww - m.piww;
  const V Ex = vfma(k(1.0 / 18.0), t, ka);
  const V kt = vfma(k(-1.0 / 36.0), t, ka);
  const V Ey = vfma(k(1.0 / 12.0), w, kt), Ez = vfma(k(-1.0 / 12.0), w, kt);
  const V s = vfma(k(0.5), m.pixx, m.pxx), q = vfma(k(0.5), m.piww, m.pww);
  const V ks = vfma(k(1.0 / 36.0), s, kd), kyz = vfma(k(-1.0 / 18.0), s, kd);
  const V kxy = vfma(k(1.0 / 12.0), q, ks), kxz = vfma(k(-1.0 / 12.0), q, ks);
  const V quarter = k(0.25), mquarter = k(-0.25);
  // odd parts
  const V tenth = k(0.1);
  const V jx = tenth * m.jx, jy = tenth * m.jy, jz = tenth * m.jz;
  const V Ox = vfma(k(-0.1), m.qx, jx), Oy = vfma(k(-0.1), m.qy, jy), Oz = vfma(k(-0.1), m.qz, jz);
  const V gx = vfma(k(0.025), m.qx, jx), gy = vfma(k(0.025), m.qy, jy), gz = vfma(k(0.025), m.qz, jz);
  const V e8 = k(0.125), n8 = k(-0.125);
  const V xy = vfma(e8, m.mx, gx), xz = vfma(n8, m.mx, gx);   // x component on the xy and xz faces
  const V yx = vfma(n8, m.my, gy), yz = vfma(e8, m.my, gy);
  const V zx = vfma(e8, m.mz, gz), zy = vfma(n8, m.mz, gz);
  auto pair = [](V& a, V& b, V ev, V od) { a = ev + od; b = ev - od; };
  pair(f[1], f[2], Ex, Ox);
  pair(f[3], f[4], Ey, Oy);
  pair(f[5], f[6], Ez, Oz);
  pair(f[7], f[10], vfma(quarter, m.pxy, kxy), xy + yx);
  pair(f[8], f[9], vfma(mquarter, m.pxy, kxy), yx - xy);
  pair(f[11], f[14], vfma(quarter, m.pxz, kxz), xz + zx);
  pair(f[12], f[13], vfma(mquarter, m.pxz, kxz), zx - xz);
  pair(f[15], f[18], vfma(quarter, m.pyz, kyz), yz + zy);
  pair(f[16], f[17], vfma(mquarter, m.pyz, kyz), zy - yz);
}

// Curvature of the normal field from its central differences (:635-663): D(i, a)
// is w_i-unweighted n_a(x + c_i) - n_a(x - c_i) for the pair representative i.
// Only the symmetric sums of the gradient enter:
//   kurv = nx ny (dxy + dyx) + nx nz (dxz + dzx) + ny nz (dyz + dzy)
//          - (ny^2 + nz^2) dxx - (nx^2 + nz^2) dyy - (nx^2 + ny^2) dzz.
// An axis pair weighs twice a diagonal one; the common factor 3/36 comes last.
template <typename V, typename R, typename F>
__device__ __forceinline__ V curvature(F&& diff, V nx, V ny, V nz) {
  auto k = [](double v) { return V(R(v)); };
  V dxx, dyy, dzz, sxy, sxz, syz;
  {
    V x[3], y[3], z[3];
    diff(std::integral_constant<int, 1>{}, x);
    diff(std::integral_constant<int, 3>{}, y);
    diff(std::integral_constant<int, 5>{}, z);
    dxx = x[0] + x[0]; dyy = y[1] + y[1]; dzz = z[2] + z[2];
    sxy = x[1] + y[0]; sxz = x[2] + z[0]; syz = y[2] + z[1];
    sxy = sxy + sxy; sxz = sxz + sxz; syz = syz + syz;
  }
  // a face's diagonals (+,+) and (+,-): their sum is twice the first axis'
  // derivative, their difference the second's
  V p[3], m[3];
  diff(std::integral_constant<int, 7>{}, p);
  diff(std::integral_constant<int, 8>{}, m);   // (-,+)
  dxx = dxx + (p[0] - m[0]); dyy = dyy + (p[1] + m[1]);
  sxy = sxy + (p[1] - m[1]) + (p[0] + m[0]); sxz = sxz + (p[2] - m[2]); syz = syz + (p[2] + m[2]);
  diff(std::integral_constant<int, 11>{}, p);
  diff(std::integral_constant<int, 12>{}, m);
  dxx = dxx + (p[0] - m[0]); dzz = dzz + (p[2] + m[2]);
  sxz = sxz + (p[2] - m[2]) + (p[0] + m[0]); sxy = sxy + (p[1] - m[1]); syz = syz + (p[1] + m[1]);
  diff(std::integral_constant<int, 15>{}, p);
  diff(std::integral_constant<int, 16>{}, m);
  dyy = dyy + (p[1] - m[1]); dzz = dzz + (p[2] + m[2]);
  syz = syz + (p[2] - m[2]) + (p[1] + m[1]); sxy = sxy + (p[0] - m[0]); sxz = sxz + (p[0] + m[0]);
  const V x2 = nx * nx, y2 = ny * ny, z2 = nz * nz;
  const V cross = vfma(nx * ny, sxy, vfma(nx * nz, sxz, (ny * nz) * syz));
  const V diag = vfma(y2 + z2, dxx, vfma(x2 + z2, dyy, (x2 + y2) * dzz));
  return k(3.0 / 36.0) * (cross - diag);
}

}  // namespace fused
}  // namespace symb200
