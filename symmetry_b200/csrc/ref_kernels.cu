// ref_kernels.cu -- the reference's per-timestep subroutines as device kernels
// on the canonical state (FP64 SoA arrays mirroring the reference's arrays).
//
// These kernels keep the reference's subroutine boundaries one to one so that
// each Fortran call site maps to one library call (the drop-in path).  Each
// kernel cites the loop it replaces.  Indices are 0-based: a reference node
// (x,y,z) (1-based) is (x-1,y-1,z-1) here.
#include <cstdio>
#include <utility>
#include <vector>
#include "nodemath.cuh"
#include "state.cuh"

namespace symb200 {

namespace {

constexpr int TPB = 256;

inline unsigned blocks_for(long long n, int tpb = TPB) { return (unsigned)((n + tpb - 1) / tpb); }

// thread t -> node of the update range (z fastest)
__device__ __forceinline__ bool range_node(const DevParams& P, long long t, int& x, int& y, int& z) {
  // (32-bit arithmetic: a domain has at most 4e9 nodes)
  const unsigned ry = P.hi[1] - P.lo[1] + 1, rz = P.hi[2] - P.lo[2] + 1;
  const unsigned u = (unsigned)t, q = u / rz, r = q / ry;
  z = P.lo[2] + (int)(u - q * rz);
  y = P.lo[1] + (int)(q - r * ry);
  x = P.lo[0] + (int)r;
  return t <= 0xffffffffLL && x <= P.hi[0];
}
inline long long range_count(const DevParams& P) {
  return (long long)(P.hi[0] - P.lo[0] + 1) * (P.hi[1] - P.lo[1] + 1) * (P.hi[2] - P.lo[2] + 1);
}

// node L's coordinates; whether it is in the update range
__device__ __forceinline__ bool update_node(const DevParams& P, long long L, int& x, int& y, int& z) {
  const unsigned Lu = (unsigned)L, q = Lu / (unsigned)P.nz;
  z = (int)(Lu - q * (unsigned)P.nz); x = (int)(q / (unsigned)P.ny); y = (int)(q - (unsigned)x * P.ny);
  return x >= P.lo[0] && x <= P.hi[0] && y >= P.lo[1] && y <= P.hi[1] && z >= P.lo[2] && z <= P.hi[2];
}
// For kernels that work on the few nodes with mask[L] >= 1: a block reads the
// masks of 4 TPB nodes, 16 bytes a thread, and hands the marked ones (node and
// mask, any order) out one per thread.  (One thread per node is bound by the
// launch of its blocks, several nodes per thread by the marked ones that sit
// side by side: curve at 152^3 147 and 71 us, at 48x88x48 37 and 62.)
struct Marked {
  unsigned n;
  unsigned node[4 * TPB];
  int32_t mask[4 * TPB];
};
__device__ __forceinline__ void load_mask4(const DevParams& P, const int32_t* __restrict__ mask, long long L0,
                                           int (&p)[4]);
template <typename F>
__device__ __forceinline__ void for_marked(const DevParams& P, const int32_t* __restrict__ mask, F&& f) {
  __shared__ Marked m;
  if (threadIdx.x == 0) m.n = 0;
  __syncthreads();
  const long long L0 = 4 * (blockIdx.x * (long long)TPB + threadIdx.x);
  int p[4];
  load_mask4(P, mask, L0, p);
  for (int k = 0; k < 4; k++)
    if (p[k] >= 1) {
      const unsigned q = atomicAdd(&m.n, 1u);
      m.node[q] = (unsigned)(L0 + k);
      m.mask[q] = p[k];
    }
  __syncthreads();
  for (unsigned q = threadIdx.x; q < m.n; q += TPB) {
    int x, y, z;
    if (update_node(P, m.node[q], x, y, z)) f((long long)m.node[q], (int)m.mask[q], x, y, z);
  }
}
// four consecutive nodes' masks from L0, a multiple of 4 (0 past the end); the
// arrays start on 256-byte boundaries
__device__ __forceinline__ void load_mask4(const DevParams& P, const int32_t* __restrict__ mask, long long L0,
                                           int (&p)[4]) {
  p[0] = p[1] = p[2] = p[3] = 0;
  if (L0 + 4 <= P.N) {
    const int4 v = *reinterpret_cast<const int4*>(mask + L0);
    p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w;
  } else {
    for (int k = 0; k < 4; k++)
      if (L0 + k < P.N) p[k] = mask[L0 + k];
  }
}

__device__ __forceinline__ long long nbr(const DevParams& P, int x, int y, int z, int i) {
  return lin(P, wrapi(x + CX(i), P.nx), wrapi(y + CY(i), P.ny), wrapi(z + CZ(i), P.nz));
}

// ---- mirror planes (symmetry_X/Y/Z_phi/_u/_fi, Source1.f90:1443-1542) ---------
// The reference copies plane n-1 onto plane n of x, then planes 2 and n-1 onto
// 1 and n of y, then plane n-1 onto n of z.  A node on several mirror planes
// ends with the value of the node mirrored in each of those axes, and no source
// lies on a mirror plane, so one launch over the planes' nodes does all three
// passes for every array (24 launches of calmacros before; 152^3: 380 us of a
// 3.4 ms step were plane copies).
struct MirrorSet {
  double* scalar[4] = {};   // copied
  double* vec[2][3] = {};   // the component along a mirrored axis changes sign
  double* pop[2] = {};      // velocities mirrored
  int32_t* mask[4] = {};
  double* low = nullptr;    // also copied onto the wall planes x = 0 and z = 0 from their neighbours
  int ns = 0, nv = 0, np = 0, nm = 0;
};

// velocity index of (cx, cy, cz)
__constant__ unsigned char kDir[27] = {0, 10, 0, 14, 2, 12, 0, 8, 0, 18, 4, 16, 6, 0, 5, 17, 3, 15, 0, 9, 0, 13, 1, 11, 0, 7, 0};
__device__ __forceinline__ int dir_index(int cx, int cy, int cz) { return kDir[(cx + 1) * 9 + (cy + 1) * 3 + cz + 1]; }

// node (x, y, z) mirrored off the mirror planes; which axes were mirrored
struct Image {
  int x, y, z;
  bool fx, fy, fz;
  __device__ __forceinline__ int dir(int cx, int cy, int cz) const {
    return dir_index(fx ? -cx : cx, fy ? -cy : cy, fz ? -cz : cz);
  }
};
__device__ __forceinline__ Image image_of(const DevParams& P, int x, int y, int z) {
  Image m;
  m.fx = x == P.nx - 1;
  m.fy = y == 0 || y == P.ny - 1;
  m.fz = z == P.nz - 1;
  m.x = m.fx ? P.nx - 2 : x;
  m.y = y == 0 ? 1 : (m.fy ? P.ny - 2 : y);
  m.z = m.fz ? P.nz - 2 : z;
  return m;
}

// t-th node of the boundary planes: x = nx-1, y = 0, y = ny-1, z = nz-1 and, with
// `walls`, x = 0 and z = 0 (nodes on several planes come up once per plane, with
// the same result)
__device__ __forceinline__ bool plane_node(const DevParams& P, int t, bool walls, int& x, int& y, int& z) {
  const int yz = P.ny * P.nz, xz = P.nx * P.nz, xy = P.nx * P.ny;
  if (t < yz) { x = P.nx - 1; y = t / P.nz; z = t % P.nz; return true; }
  t -= yz;
  if (t < 2 * xz) {
    y = t < xz ? 0 : P.ny - 1;
    if (t >= xz) t -= xz;
    x = t / P.nz; z = t % P.nz;
    return true;
  }
  t -= 2 * xz;
  if (t < xy) { x = t / P.ny; y = t % P.ny; z = P.nz - 1; return true; }
  t -= xy;
  if (!walls) return false;
  if (t < yz) { x = 0; y = t / P.nz; z = t % P.nz; return true; }
  t -= yz;
  if (t < xy) { x = t / P.ny; y = t % P.ny; z = 0; return true; }
  return false;
}
inline long long plane_count(const DevParams& P, bool walls) {
  const long long yz = (long long)P.ny * P.nz, xz = (long long)P.nx * P.nz, xy = (long long)P.nx * P.ny;
  return yz + 2 * xz + xy + (walls ? yz + xy : 0);
}

__global__ void __launch_bounds__(TPB) k_mirror(DevParams P, MirrorSet S) {
  int x, y, z;
  if (!plane_node(P, blockIdx.x * TPB + threadIdx.x, S.low != nullptr, x, y, z)) return;
  const Image m = image_of(P, x, y, z);
  const long long Ld = lin(P, x, y, z), N = P.N;
  if (S.low) S.low[Ld] = S.low[lin(P, m.x == 0 ? 1 : m.x, m.y, m.z == 0 ? 1 : m.z)];
  if (!(m.fx || m.fy || m.fz)) return;
  const long long Ls = lin(P, m.x, m.y, m.z);
  // every array's value is read before the first is written (the planes of z are
  // one sector per value: latency, not bandwidth)
  double v[4 + 6];
  int32_t k4[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (k < S.ns) v[k] = S.scalar[k][Ls];
    if (k < S.nm) k4[k] = S.mask[k][Ls];
  }
#pragma unroll
  for (int k = 0; k < 6; k++)
    if (k / 3 < S.nv) v[4 + k] = S.vec[k / 3][k % 3][Ls];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (k < S.ns) S.scalar[k][Ld] = v[k];
    if (k < S.nm) S.mask[k][Ld] = k4[k];
  }
#pragma unroll
  for (int k = 0; k < 6; k++)
    if (k / 3 < S.nv) {
      const bool flip = k % 3 == 0 ? m.fx : (k % 3 == 1 ? m.fy : m.fz);
      S.vec[k / 3][k % 3][Ld] = flip ? -v[4 + k] : v[4 + k];
    }
#pragma unroll 1
  for (int k = 0; k < S.np; k++) {
    double* const f = S.pop[k];
    double tmp[19];
#pragma unroll
    for (int i = 0; i < 19; i++) tmp[i] = f[m.dir(CX(i), CY(i), CZ(i)) * N + Ls];
#pragma unroll
    for (int i = 0; i < 19; i++) f[i * N + Ld] = tmp[i];
  }
}
void mirror(sym_handle* h, const MirrorSet& S) {
  k_mirror<<<blocks_for(plane_count(h->dp, S.low != nullptr)), TPB, 0, h->st>>>(h->dp, S);
}

// ---- calmacros (Source1.f90:770-831) --------------------------------------
__global__ void k_calmacros(DevParams P, const double* __restrict__ ri, const double* __restrict__ bi,
                            double* __restrict__ fi, double* rho, double* ux, double* uy, double* uz, double* rhoN,
                            double* rhoR, double* rhoB, const int32_t* __restrict__ walls_all) {
  int x, y, z;
  if (!range_node(P, blockIdx.x * (long long)blockDim.x + threadIdx.x, x, y, z)) return;
  const long long L = lin(P, x, y, z), N = P.N;
  if (walls_all[L] >= 1) {
    rhoN[L] = 0.0; ux[L] = 0.0; uy[L] = 0.0; uz[L] = 0.0; rho[L] = P.rho0;
    return;
  }
  double f[19], sr = 0.0, sb = 0.0;
#pragma unroll
  for (int i = 0; i < 19; i++) {
    const double r = ri[i * N + L], b = bi[i * N + L];
    f[i] = r + b;
    fi[i * N + L] = f[i];
    sr = sr + r;
  }
#pragma unroll
  for (int i = 0; i < 19; i++) sb = sb + bi[i * N + L];
  rhoR[L] = sr; rhoB[L] = sb;
  const double rh = sr + sb;
  rho[L] = rh;
  double mx = 0.0, my = 0.0, mz = 0.0;
#pragma unroll
  for (int i = 0; i < 19; i++) {
    if (CX(i)) mx = mx + f[i] * (double)CX(i);
    if (CY(i)) my = my + f[i] * (double)CY(i);
    if (CZ(i)) mz = mz + f[i] * (double)CZ(i);
  }
  ux[L] = mx / rh; uy[L] = my / rh; uz[L] = mz / rh;
  rhoN[L] = (sr - sb) / rh;
}

// rho_N, rho_R, rho_B, rho, u and fi; wall_phi: rho_N also onto the wall planes
void mirror_macros(sym_handle* h, bool wall_phi) {
  MirrorSet S;
  S.scalar[S.ns++] = h->rhoR;
  S.scalar[S.ns++] = h->rhoB;
  S.scalar[S.ns++] = h->rho;
  if (wall_phi) S.low = h->rhoN;
  else S.scalar[S.ns++] = h->rhoN;
  S.vec[0][0] = h->ux; S.vec[0][1] = h->uy; S.vec[0][2] = h->uz;
  S.nv = 1;
  S.pop[S.np++] = h->fi;
  mirror(h, S);
}
void mirror_colours(sym_handle* h) {
  MirrorSet S;
  S.pop[S.np++] = h->ri;
  S.pop[S.np++] = h->bi;
  mirror(h, S);
}

// ---- derivatives (Source1.f90:452-597) ------------------------------------
// images: the filled node's images on the mirror planes too
__global__ void __launch_bounds__(TPB) k_pin_fill(DevParams P, const int32_t* __restrict__ pin,
                                                  const int32_t* __restrict__ walls_all, double* rhoN, bool images) {
  for_marked(P, pin, [&](long long L, int, int x, int y, int z) {
    int wall[19];
    double ph[19];
#pragma unroll
    for (int i = 1; i < 19; i++) {
      const long long nb = nbr(P, x, y, z, i);
      wall[i] = walls_all[nb];
      ph[i] = rhoN[nb];
    }
    double ws = 0.0, v = 0.0;
#pragma unroll
    for (int i = 1; i < 19; i++)
      if (wall[i] <= 0) { ws = ws + W(i); v = v + W(i) * ph[i]; }
    rhoN[L] = v / ws;
    if (images) for_images(P, x, y, z, false, [&](long long Li, bool, bool, bool) { rhoN[Li] = v / ws; });
  });
}

// REF: no neighbour of an updated node is across a periodic face
template <bool REF>
__global__ void k_gradient(DevParams P, const sym_particles* __restrict__ S, const int32_t* __restrict__ pout,
                           const int32_t* __restrict__ walls_all, const double* __restrict__ rhoN, double* gx, double* gy, double* gz, double* nx, double* ny, double* nz, int32_t* flag) {
  int x, y, z;
  if (!range_node(P, blockIdx.x * (long long)blockDim.x + threadIdx.x, x, y, z)) return;
  const long long L = lin(P, x, y, z);
  double g0 = 0.0, g1 = 0.0, g2 = 0.0, n0 = 0.0, n1 = 0.0, n2 = 0.0;
  int fl = 0;
  if (walls_all[L] <= 0) {
#pragma unroll
    for (int i = 1; i < 19; i++) {
      const double val = W(i) * (REF ? (rhoN + L)[CZ(i) + P.nz * (CY(i) + P.ny * CX(i))] : rhoN[nbr(P, x, y, z, i)]);
      if (CX(i)) g0 = g0 + val * (double)CX(i);
      if (CY(i)) g1 = g1 + val * (double)CY(i);
      if (CZ(i)) g2 = g2 + val * (double)CZ(i);
    }
    g0 = 3.0 * g0; g1 = 3.0 * g1; g2 = 3.0 * g2;
    const double fnorm = sqrt(g0 * g0 + g1 * g1 + g2 * g2);
    if (fnorm > P.evap) { n0 = g0 / fnorm; n1 = g1 / fnorm; n2 = g2 / fnorm; fl = 1; }
  }
  // rotated to the contact angle next to a solid (:535-587)
  const int pp = fl ? pout[L] : 0;
  if (pp >= 1) {
    double nw[3], n[3] = {n0, n1, n2}, v[3];
    wall_normal_dev(P, S, pp, x, y, z, nw);
    akai_rotate<double>(P.cita, nw, n, true, v);
    n0 = v[0]; n1 = v[1]; n2 = v[2];
    const double fnorm = sqrt(g0 * g0 + g1 * g1 + g2 * g2);
    g0 = fnorm * v[0]; g1 = fnorm * v[1]; g2 = fnorm * v[2];
  }
  gx[L] = g0; gy[L] = g1; gz[L] = g2; nx[L] = n0; ny[L] = n1; nz[L] = n2; flag[L] = fl;
  if (REF)
    for_images(P, x, y, z, false, [&](long long Li, bool fx, bool fy, bool fz) {
      gx[Li] = fx ? -g0 : g0; gy[Li] = fy ? -g1 : g1; gz[Li] = fz ? -g2 : g2;
      nx[Li] = fx ? -n0 : n0; ny[Li] = fy ? -n1 : n1; nz[Li] = fz ? -n2 : n2;
    });
}

// ---- collision (Source1.f90:599-695) --------------------------------------
__global__ void __launch_bounds__(128) k_collision(
    DevParams P, const int32_t* __restrict__ walls_all, const int32_t* __restrict__ pout,
    const int32_t* __restrict__ flag, const double* __restrict__ nxv, const double* __restrict__ nyv,
    const double* __restrict__ nzv, const double* __restrict__ gx, const double* __restrict__ gy,
    const double* __restrict__ gz, const double* __restrict__ rho, const double* __restrict__ rhoN, double* ux,
    double* uy, double* uz, double* fi, double* ffi) {
  int x, y, z;
  if (!range_node(P, blockIdx.x * (long long)blockDim.x + threadIdx.x, x, y, z)) return;
  const long long L = lin(P, x, y, z), N = P.N;
  if (walls_all[L] > 0) return;
  double fx = 0.0, fy = 0.0, fz = 0.0;
  const bool edge_ok = P.ref ? (z >= 2 && x >= 2) : true;  // z>=3 .and. x>=3 (1-based), :624
  if (flag[L] && pout[L] <= 0 && edge_ok) {
    double d00 = 0, d01 = 0, d02 = 0, d10 = 0, d11 = 0, d12 = 0, d20 = 0, d21 = 0, d22 = 0;
#pragma unroll
    for (int i = 1; i < 19; i++) {
      const long long nb = nbr(P, x, y, z, i);
      double tmp = W(i) * nxv[nb];
      if (CX(i)) d00 = d00 + tmp * (double)CX(i);
      if (CY(i)) d01 = d01 + tmp * (double)CY(i);
      if (CZ(i)) d02 = d02 + tmp * (double)CZ(i);
      tmp = W(i) * nyv[nb];
      if (CX(i)) d10 = d10 + tmp * (double)CX(i);
      if (CY(i)) d11 = d11 + tmp * (double)CY(i);
      if (CZ(i)) d12 = d12 + tmp * (double)CZ(i);
      tmp = W(i) * nzv[nb];
      if (CX(i)) d20 = d20 + tmp * (double)CX(i);
      if (CY(i)) d21 = d21 + tmp * (double)CY(i);
      if (CZ(i)) d22 = d22 + tmp * (double)CZ(i);
    }
    d00 *= 3.0; d01 *= 3.0; d02 *= 3.0; d10 *= 3.0; d11 *= 3.0; d12 *= 3.0; d20 *= 3.0; d21 *= 3.0; d22 *= 3.0;
    const double nx = nxv[L], ny = nyv[L], nz = nzv[L];
    const double kurv = nx * ny * (d10 + d01) + nx * nz * (d20 + d02) + ny * nz * (d12 + d21) -
                        (ny * ny + nz * nz) * d00 - (nx * nx + nz * nz) * d11 - (nx * nx + ny * ny) * d22;
    const double val = 0.5 * P.sigma * kurv;
    fx = val * gx[L]; fy = val * gy[L]; fz = val * gz[L];
  }
  const double rh = rho[L];
  if (!P.ref) { fx = fx + rh * P.body[0]; fy = fy + rh * P.body[1]; fz = fz + rh * P.body[2]; }
  const double u0 = ux[L] + 0.5 * fx / rh, u1 = uy[L] + 0.5 * fy / rh, u2 = uz[L] + 0.5 * fz / rh;
  ux[L] = u0; uy[L] = u1; uz[L] = u2;
  double f[19];
#pragma unroll
  for (int i = 0; i < 19; i++) f[i] = fi[i * N + L];
  mrt_collide<double>(P, f, rh, u0, u1, u2, fx, fy, fz, rhoN[L]);
#pragma unroll
  for (int i = 0; i < 19; i++) { fi[i * N + L] = f[i]; ffi[i * N + L] = f[i]; }
}

// ---- Recolor (Source1.f90:697-732) ----------------------------------------
__global__ void k_recolor(DevParams P, const int32_t* __restrict__ walls_all, const int32_t* __restrict__ flag,
                          const double* __restrict__ fi, double* ri, double* bi, const double* __restrict__ rhoR,
                          const double* __restrict__ rhoB, const double* __restrict__ rho,
                          const double* __restrict__ nxv, const double* __restrict__ nyv,
                          const double* __restrict__ nzv) {
  int x, y, z;
  if (!range_node(P, blockIdx.x * (long long)blockDim.x + threadIdx.x, x, y, z)) return;
  const long long L = lin(P, x, y, z), N = P.N;
  if (walls_all[L] >= 1) return;
  const double R = rhoR[L], B = rhoB[L], rh = rho[L];
  const double ratio = R / rh;
  const bool fl = flag[L] != 0;
  const double coef = R * B / rh * P.beta;
  const double n0 = nxv[L], n1 = nyv[L], n2 = nzv[L];
#pragma unroll
  for (int i = 0; i < 19; i++) {
    const double f = fi[i * N + L];
    double r = ratio * f;
    if (i > 0 && fl) r = r + coef * W(i) * (n0 * (double)CX(i) + n1 * (double)CY(i) + n2 * (double)CZ(i));
    if (R <= P.evap) r = 0.0;
    if (B <= P.evap) r = f;
    ri[i * N + L] = r;
    bi[i * N + L] = f - r;
  }
}

// ---- boundary (Source1.f90:1544-1592), REFERENCE geometry -------------------
// Mirror planes, then the halfway bounce-back of the bottom wall z = 0 and of
// the back wall x = 0 (0-based): link i of a node next to a wall comes back as
// opc(i) of the wall node it enters.  One thread per boundary node gathers its
// new populations; the reads go to nodes off the mirror planes, and on the wall
// planes only to velocities that no thread writes.
// FULL: every velocity of every boundary node.  Otherwise (inside a run of
// steps) a node on mirror planes only gets the velocities that enter the domain;
// those that leave it or run along the planes reach no interior node, and the
// run's last step writes them all.  Nodes of the wall planes, whose populations
// along the walls a run carries from step to step, get all of theirs, and
// (1,0,-1) of the plane x = nx-1 wraps to the row beside both walls, where no
// bounce-back replaces it.
template <bool FULL>
__global__ void __launch_bounds__(TPB) k_boundary(DevParams P, double* ri, double* bi) {
  int x, y, z;
  if (!plane_node(P, blockIdx.x * TPB + threadIdx.x, true, x, y, z)) return;
  const long long N = P.N, Ld = lin(P, x, y, z);
  const Image own = image_of(P, x, y, z);
  const bool mirrored = own.fx || own.fy || own.fz;
  const long long Lo = lin(P, own.x, own.y, own.z);
  const bool all = FULL || x == 0 || z == 0;
  auto enters = [&](int cx, int cy, int cz) {
    return (x == P.nx - 1 && (cx < 0 || (cx > 0 && cy == 0 && cz < 0))) || (y == 0 && cy > 0) ||
           (y == P.ny - 1 && cy < 0) || (z == P.nz - 1 && cz < 0);
  };
  double tr[19], tb[19];
#pragma unroll
  for (int i = 0; i < 19; i++) {
    // (1,0,-1) of the row beside both walls: the back wall would return what
    // the bottom wall just put there, its own value
    const bool back = x == 0 && CX(i) > 0 && !(i == 13 && z == 1);
    if ((z == 0 && CZ(i) > 0) || back) {
      const Image m = image_of(P, wrapi(x + CX(i), P.nx), wrapi(y + CY(i), P.ny), wrapi(z + CZ(i), P.nz));
      const long long q = m.dir(-CX(i), -CY(i), -CZ(i)) * N + lin(P, m.x, m.y, m.z);
      tr[i] = ri[q];
      tb[i] = bi[q];
    } else if (mirrored && (all || enters(CX(i), CY(i), CZ(i)))) {
      const long long q = own.dir(CX(i), CY(i), CZ(i)) * N + Lo;
      tr[i] = ri[q];
      tb[i] = bi[q];
    }
  }
#pragma unroll
  for (int i = 0; i < 19; i++) {
    const bool back = x == 0 && CX(i) > 0 && !(i == 13 && z == 1);
    if ((z == 0 && CZ(i) > 0) || back || (mirrored && (all || enters(CX(i), CY(i), CZ(i))))) {
      ri[i * N + Ld] = tr[i];
      bi[i * N + Ld] = tb[i];
    }
  }
}

// ---- streaming (Source1.f90:735-768): periodic pull, i = 1..18 ---------------
// REST: the velocity at rest is carried over too
template <bool REST>
__global__ void k_stream_pull(DevParams P, const double* __restrict__ f, double* __restrict__ ft) {
  const long long L = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (L >= P.N) return;
  const int z = (int)(L % P.nz), y = (int)((L / P.nz) % P.ny), x = (int)(L / ((long long)P.nz * P.ny));
  const long long N = P.N;
  if (REST) ft[L] = f[L];
#pragma unroll
  for (int i = 1; i < 19; i++) {
    const long long src = lin(P, wrapi(x - CX(i), P.nx), wrapi(y - CY(i), P.ny), wrapi(z - CZ(i), P.nz));
    ft[i * N + L] = f[i * N + src];
  }
}

// ---- curve (Source1.f90:990-1034) -----------------------------------------
__device__ __forceinline__ void curve_node(const DevParams& P, const sym_particles* __restrict__ S,
                                           const int32_t* __restrict__ walls, int pp, double* ri, double* bi,
                                           const double* __restrict__ rhoR, const double* __restrict__ rhoB, int x,
                                           int y, int z) {
  const long long L = lin(P, x, y, z), N = P.N;
  const int par = P.par;
  // the neighbours' masks are read together, then the populations of every link
  // from a solid, which no thread writes (one link after another, each waited for
  // the store before it: 23 us at 48x88x48)
  int wbs[19];
  long long Bs[19];
#pragma unroll
  for (int i = 1; i < 19; i++) {
    const int xb = P.ref ? x - CX(i) : wrapi(x - CX(i), P.nx);
    const int yb = P.ref ? y - CY(i) : wrapi(y - CY(i), P.ny);
    const int zb = P.ref ? z - CZ(i) : wrapi(z - CZ(i), P.nz);
    Bs[i] = lin(P, xb, yb, zb);
    wbs[i] = walls[Bs[i]];
  }
  const double cr = rhoR[L], cb = rhoB[L];
  double r[19], b[19];
  bool link[19];
#pragma unroll
  for (int i = 1; i < 19; i++) {
    link[i] = wbs[i] == pp || (!P.ref && wbs[i] > par);
    r[i] = b[i] = 0.0;
    if (link[i]) {
      r[i] = ri[OPC(i) * N + Bs[i]];
      b[i] = bi[OPC(i) * N + Bs[i]];
    }
  }
  // a link from a particle comes from pp's (of a flat wall: no velocity)
  double uw0 = 0.0, uw1 = 0.0, uw2 = 0.0;
  if (pp <= par) {
    const double xr = disp(P, (double)(x + P.origin), S->center[0 * par + pp - 1], 0);
    const double yr = disp(P, (double)(y + P.origin), S->center[1 * par + pp - 1], 1);
    const double zr = disp(P, (double)(z + P.origin), S->center[2 * par + pp - 1], 2);
    const double* up = S->up;
    const double* rp = S->rp;
    uw0 = up[0 * par + pp - 1] + zr * rp[1 * par + pp - 1] - yr * rp[2 * par + pp - 1];
    uw1 = up[1 * par + pp - 1] + xr * rp[2 * par + pp - 1] - zr * rp[0 * par + pp - 1];
    uw2 = up[2 * par + pp - 1] + yr * rp[0 * par + pp - 1] - xr * rp[1 * par + pp - 1];
  }
#pragma unroll
  for (int i = 1; i < 19; i++) {
    if (!link[i]) continue;
    double star = 0.0;
    if (wbs[i] <= par) star = uw0 * (double)CX(i) + uw1 * (double)CY(i) + uw2 * (double)CZ(i);
    ri[i * N + L] = r[i] + 6.0 * W(i) * cr * star;
    bi[i * N + L] = b[i] + 6.0 * W(i) * cb * star;
  }
}

__global__ void __launch_bounds__(TPB) k_curve(DevParams P, const sym_particles* __restrict__ S,
                                               const int32_t* __restrict__ walls, const int32_t* __restrict__ pout,
                                               double* ri, double* bi, const double* __restrict__ rhoR,
                                               const double* __restrict__ rhoB) {
  for_marked(P, pout, [&](long long, int pp, int x, int y, int z) {
    curve_node(P, S, walls, pp, ri, bi, rhoR, rhoB, x, y, z);
  });
}

// curve2 (Source1.f90:1036-1101): bounce-back interpolated with the link
// fraction, the wall velocity at the wall point; one thread per node updates
// its links in index order like the reference's loop.  CONFIG wall planes keep
// the halfway bounce-back.
__global__ void k_curve2(DevParams P, const sym_particles* __restrict__ S, const int32_t* __restrict__ walls,
                         const int32_t* __restrict__ pout, double* ri, double* bi, const double* __restrict__ rhoR,
                         const double* __restrict__ rhoB) {
  int x, y, z;
  if (!range_node(P, blockIdx.x * (long long)blockDim.x + threadIdx.x, x, y, z)) return;
  const long long L = lin(P, x, y, z), N = P.N;
  const int pp = pout[L];
  if (pp < 1) return;
  const int par = P.par;
#pragma unroll 1
  for (int i = 1; i < 19; i++) {
    const int xb = P.ref ? x - CX(i) : wrapi(x - CX(i), P.nx);
    const int yb = P.ref ? y - CY(i) : wrapi(y - CY(i), P.ny);
    const int zb = P.ref ? z - CZ(i) : wrapi(z - CZ(i), P.nz);
    const long long B = lin(P, xb, yb, zb);
    const int wb = walls[B];
    const int j = OPC(i);
    if (wb == pp && pp <= par) {
      const int xf = P.ref ? x + CX(i) : wrapi(x + CX(i), P.nx);
      const int yf = P.ref ? y + CY(i) : wrapi(y + CY(i), P.ny);
      const int zf = P.ref ? z + CZ(i) : wrapi(z + CZ(i), P.nz);
      const long long F = lin(P, xf, yf, zf);
      const double cx = CX(i), cy = CY(i), cz = CZ(i);
      const double* c = S->center;
      const double x0 = disp(P, (double)(x + P.origin), c[0 * par + pp - 1], 0);
      const double y0 = disp(P, (double)(y + P.origin), c[1 * par + pp - 1], 1);
      const double z0 = disp(P, (double)(z + P.origin), c[2 * par + pp - 1], 2);
      const double qq = link_fraction(x0, y0, z0, cx, cy, cz, P.rad);
      const double xr = disp(P, (double)(x + P.origin) - cx * qq, c[0 * par + pp - 1], 0);
      const double yr = disp(P, (double)(y + P.origin) - cy * qq, c[1 * par + pp - 1], 1);
      const double zr = disp(P, (double)(z + P.origin) - cz * qq, c[2 * par + pp - 1], 2);
      const double* up = S->up;
      const double* rp = S->rp;
      const double uw0 = up[0 * par + pp - 1] + zr * rp[1 * par + pp - 1] - yr * rp[2 * par + pp - 1];
      const double uw1 = up[1 * par + pp - 1] + xr * rp[2 * par + pp - 1] - zr * rp[0 * par + pp - 1];
      const double uw2 = up[2 * par + pp - 1] + yr * rp[0 * par + pp - 1] - xr * rp[1 * par + pp - 1];
      const double star = uw0 * cx + uw1 * cy + uw2 * cz;
      ri[i * N + L] = 1.0 / (1.0 + qq) *
                      (qq * (ri[i * N + F] + ri[j * N + B]) + (1.0 - qq) * ri[j * N + L] + 6.0 * W(i) * rhoR[L] * star);
      bi[i * N + L] = 1.0 / (1.0 + qq) *
                      (qq * (bi[i * N + F] + bi[j * N + B]) + (1.0 - qq) * bi[j * N + L] + 6.0 * W(i) * rhoB[L] * star);
    } else if (wb == pp || (!P.ref && wb > par)) {
      ri[i * N + L] = ri[j * N + B];
      bi[i * N + L] = bi[j * N + B];
    }
  }
}

// ---- whole steps (sym_step, REFERENCE geometry, halfway bounce-back) -------------
// A run of n steps is the reference's loop body n times, cut between the calls
// so that passes over the populations fall together (152^3 per step, bytes per
// node: separate subroutines about 2,700, these about 1,150):
//   streaming of both colours, curve and the next step's calmacros in one pass
//   (k_step_macros<true>), and collision with Recolor in one (k_collide_recolor).
//   Both passes pull the streamed populations from the ones boundary left; only
//   those that curve, refilling or the walls' carry-over make or need are
//   written in between (`kept`: boundary planes, solids, nodes next to a
//   particle), so a step reads the populations twice and writes them once.
// What no later call of the same run reads is written by the run's last step
// only (FULL): fi and ffi away from the particles, rho and u, and the mirror
// planes' copies of them.

// calmacros (:770-831) of the populations (ri, bi); PULL: of the populations
// that streaming (:735-768) and curve (:990-1034) make of them, which go to
// (ro, bo) on every node (FULL) or on those it marks in kept.  !FULL: fi only
// next to particles (the momentum exchange reads it there), no rho and u.
template <bool PULL, bool FULL>
__global__ void __launch_bounds__(TPB) k_step_macros(DevParams P, const sym_particles* __restrict__ S,
                                                     const double* __restrict__ ri, const double* __restrict__ bi,
                                                     double* __restrict__ ro, double* __restrict__ bo,
                                                     unsigned char* __restrict__ kept, double* fi, double* rho,
                                                     double* ux, double* uy, double* uz, double* rhoN, double* rhoR,
                                                     double* rhoB, const int32_t* __restrict__ walls,
                                                     const int32_t* __restrict__ walls_all,
                                                     const int32_t* __restrict__ pout) {
  const long long N = P.N, L = blockIdx.x * (long long)TPB + threadIdx.x;
  if (L >= N) return;
  const unsigned Lu = (unsigned)L, q = Lu / (unsigned)P.nz;
  const int z = (int)(Lu - q * (unsigned)P.nz), x = (int)(q / (unsigned)P.ny), y = (int)(q - (unsigned)x * P.ny);
  const bool in = x >= P.lo[0] && x <= P.hi[0] && y >= P.lo[1] && y <= P.hi[1] && z >= P.lo[2] && z <= P.hi[2];
  if (!PULL && !in) return;
  const int pp = in ? pout[L] : 0;
  const bool solid = in && walls_all[L] >= 1;
  double r[19], b[19];
  if (PULL) {
    // 32-bit offsets along each axis, from one pointer per velocity
    const int sx = P.ny * P.nz, sy = P.nz;
    const int ox[3] = {x + 1 < P.nx ? sx : -(P.nx - 1) * sx, 0, x > 0 ? -sx : (P.nx - 1) * sx};
    const int oy[3] = {y + 1 < P.ny ? sy : -(P.ny - 1) * sy, 0, y > 0 ? -sy : (P.ny - 1) * sy};
    const int oz[3] = {z + 1 < P.nz ? 1 : -(P.nz - 1), 0, z > 0 ? -1 : P.nz - 1};
    const double* const rL = ri + L;
    const double* const bL = bi + L;
#pragma unroll
    for (int i = 0; i < 19; i++) {
      const int o = ox[CX(i) + 1] + oy[CY(i) + 1] + oz[CZ(i) + 1];
      r[i] = (rL + i * N)[o];
      b[i] = (bL + i * N)[o];
    }
    if (pp >= 1) {
      // link i comes from a node of particle pp: this node's own opposite
      // population, with the wall's velocity
      const int par = P.par;
      const double xr = disp(P, (double)(x + P.origin), S->center[0 * par + pp - 1], 0);
      const double yr = disp(P, (double)(y + P.origin), S->center[1 * par + pp - 1], 1);
      const double zr = disp(P, (double)(z + P.origin), S->center[2 * par + pp - 1], 2);
      const double* up = S->up;
      const double* rp = S->rp;
      const double uw0 = up[0 * par + pp - 1] + zr * rp[1 * par + pp - 1] - yr * rp[2 * par + pp - 1];
      const double uw1 = up[1 * par + pp - 1] + xr * rp[2 * par + pp - 1] - zr * rp[0 * par + pp - 1];
      const double uw2 = up[2 * par + pp - 1] + yr * rp[0 * par + pp - 1] - xr * rp[1 * par + pp - 1];
      const double cr = rhoR[L], cb = rhoB[L];
#pragma unroll
      for (int i = 1; i < 19; i++) {
        if (walls[lin(P, x - CX(i), y - CY(i), z - CZ(i))] != pp) continue;
        const double star = uw0 * (double)CX(i) + uw1 * (double)CY(i) + uw2 * (double)CZ(i);
        r[i] = ri[OPC(i) * N + L] + 6.0 * W(i) * cr * star;
        b[i] = bi[OPC(i) * N + L] + 6.0 * W(i) * cb * star;
      }
    }
    const bool keep = !in || solid || pp >= 1;
    if (FULL || keep) {
#pragma unroll
      for (int i = 0; i < 19; i++) {
        ro[i * N + L] = r[i];
        bo[i * N + L] = b[i];
      }
    }
    if (!FULL) kept[L] = keep;
    if (!in) return;
  }
  if (solid) {
    rhoN[L] = 0.0;
    if (FULL) { ux[L] = 0.0; uy[L] = 0.0; uz[L] = 0.0; rho[L] = P.rho0; }
    return;
  }
  if (!PULL) {
#pragma unroll
    for (int i = 0; i < 19; i++) {
      r[i] = ri[i * N + L];
      b[i] = bi[i * N + L];
    }
  }
  double sr = 0.0, sb = 0.0, mx = 0.0, my = 0.0, mz = 0.0;
#pragma unroll
  for (int i = 0; i < 19; i++) {
    sr = sr + r[i];
    sb = sb + b[i];
    if (FULL || pp > 0) fi[i * N + L] = r[i] + b[i];
    if (FULL) {
      const double f = r[i] + b[i];
      if (CX(i)) mx = mx + f * (double)CX(i);
      if (CY(i)) my = my + f * (double)CY(i);
      if (CZ(i)) mz = mz + f * (double)CZ(i);
    }
  }
  rhoR[L] = sr; rhoB[L] = sb;
  const double rh = sr + sb;
  rhoN[L] = (sr - sb) / rh;
  if (FULL) {
    rho[L] = rh;
    ux[L] = mx / rh; uy[L] = my / rh; uz[L] = mz / rh;
  }
}

// collision (:599-695) and Recolor (:697-732) of one node from its populations
// (ri, bi), in place; the collision in the fused path's arithmetic
// (nodemath.cuh), bound by memory instead of FP64 issue (the two kernels: 816 +
// 366 us at 152^3).  PULL: the populations of nodes that k_step_macros did not
// keep are streamed here from (rs, bs), without curve, which they were not part
// of; a node that has become solid since gets them unchanged.
// A node uncovered without being refilled (it is next to no particle any more: one
// that moved by more than a node) collides what calmacros left of a solid node:
// the totals fi of the step that covered it, rho0, no velocity, its old colour
// densities.
template <bool FULL, bool PULL>
__global__ void __launch_bounds__(128, 4) k_collide_recolor(
    DevParams P, const __grid_constant__ TileParams<double> T, const int32_t* __restrict__ walls_all,
    const int32_t* __restrict__ pout, const int32_t* __restrict__ flag, const double* __restrict__ nxv,
    const double* __restrict__ nyv, const double* __restrict__ nzv, const double* __restrict__ gx,
    const double* __restrict__ gy, const double* __restrict__ gz, const double* __restrict__ rhoN, double* ux,
    double* uy, double* uz, double* fi, double* ffi, double* ri, double* bi, const double* __restrict__ rs,
    const double* __restrict__ bs, const unsigned char* __restrict__ kept, const int32_t* __restrict__ walls_old,
    const double* __restrict__ rhoR, const double* __restrict__ rhoB) {
  using namespace fused;
  const unsigned t = blockIdx.x * 128u + threadIdx.x;
  const unsigned rz = P.hi[2] - P.lo[2] + 1, ry = P.hi[1] - P.lo[1] + 1;
  const unsigned q = t / rz;
  const int z = P.lo[2] + (int)(t - q * rz), x = P.lo[0] + (int)(q / ry), y = P.lo[1] + (int)(q % ry);
  if (x > P.hi[0]) return;
  const long long L = lin(P, x, y, z), N = P.N;
  const bool solid = walls_all[L] > 0;
  const bool pull = PULL && !kept[L];
  const bool covered = !FULL && solid && walls_old[L] <= 0;
  if (solid && !pull && !covered) return;
  const int pp = pout[L];
  const bool fl = flag[L] != 0;
  double f[19], cr[19];
  const double* const fr = pull ? rs : ri;
  const double* const fb = pull ? bs : bi;
#pragma unroll
  for (int i = 0; i < 19; i++) {
    // an updated node's neighbours are inside the arrays
    const long long o = i * N + L - (pull ? CZ(i) + P.nz * (CY(i) + P.ny * CX(i)) : 0);
    cr[i] = fr[o];
    f[i] = fb[o];
  }
  if (solid) {
#pragma unroll
    for (int i = 0; i < 19; i++) {
      if (pull) {
        ri[i * N + L] = cr[i];
        bi[i * N + L] = f[i];
      }
      if (covered) fi[i * N + L] = cr[i] + f[i];
    }
    return;
  }
  auto sum = [](const double (&c)[19]) {
    return c[0] + ((c[1] + c[2]) + (c[3] + c[4]) + (c[5] + c[6])) +
           (((c[7] + c[10]) + (c[8] + c[9])) + ((c[11] + c[14]) + (c[12] + c[13])) + ((c[15] + c[18]) + (c[16] + c[17])));
  };
  // each colour's own sum: as a difference of densities the smaller one would
  // carry the rounding of the larger (at EVAP_LIM 1e-9 of itself)
  double sr = sum(cr), sb = sum(f);
#pragma unroll
  for (int i = 0; i < 19; i++) f[i] = cr[i] + f[i];
  const double phi = rhoN[L];
  const bool stale = phi == 0.0 && pp <= 0 && walls_old[L] >= 1;   // (phi of a solid node is 0)
  if (stale) {
    sr = rhoR[L];
    sb = rhoB[L];
#pragma unroll
    for (int i = 0; i < 19; i++) f[i] = fi[i * N + L];
  }
  Moments<double> m;
  to_moments<double, double>(f, m);
  if (stale) {
    m.rho = P.rho0;
    m.jx = m.jy = m.jz = 0.0;
  }
  const double rh = m.rho;
  double irho, su, sq;
  node_rates_fused<double>(T, phi, rh, irho, su, sq);
  const double n0 = nxv[L], n1 = nyv[L], n2 = nzv[L];
  double fx = 0.0, fy = 0.0, fz = 0.0;
  if (fl && pp <= 0 && z >= 2 && x >= 2) {   // z>=3 .and. x>=3 (1-based), :624
    const double kurv = curvature<double, double>(
        [&](auto ic, double (&d)[3]) {
          constexpr int i = decltype(ic)::value;
          const int o = CZ(i) + P.nz * (CY(i) + P.ny * CX(i));
          d[0] = nxv[L + o] - nxv[L - o];
          d[1] = nyv[L + o] - nyv[L - o];
          d[2] = nzv[L + o] - nzv[L - o];
        },
        n0, n1, n2);
    const double val = T.np.half_sigma * kurv;
    fx = val * gx[L]; fy = val * gy[L]; fz = val * gz[L];
  }
  const double u0 = (m.jx + 0.5 * fx) * irho, u1 = (m.jy + 0.5 * fy) * irho, u2 = (m.jz + 0.5 * fz) * irho;
  if (FULL) { ux[L] = u0; uy[L] = u1; uz[L] = u2; }
  const NodeParams<double>& np = T.np;
  relax<double, double>(m, rh, u0, u1, u2, fx, fy, fz, su, np.s_e > 0 ? np.s_e : su, np.s_eps > 0 ? np.s_eps : su,
                        np.s_q > 0 ? np.s_q : sq, np.s_pi > 0 ? np.s_pi : su, np.s_m > 0 ? np.s_m : sq);
  from_moments<double, double>(m, f);
  if (FULL || pp > 0) {
#pragma unroll
    for (int i = 0; i < 19; i++) { fi[i * N + L] = f[i]; ffi[i * N + L] = f[i]; }
  }
  const bool rzero = sr <= P.evap, bzero = sb <= P.evap;
  const double ratio = bzero ? 1.0 : (rzero ? 0.0 : sr * irho);
  const double coef = (rzero || bzero || !fl) ? 0.0 : sr * sb * irho * np.beta;
#pragma unroll
  for (int i = 0; i < 19; i++) {
    double r = ratio * f[i];
    if (i > 0) r = fma(coef * W(i), n0 * (double)CX(i) + n1 * (double)CY(i) + n2 * (double)CZ(i), r);
    ri[i * N + L] = r;
    bi[i * N + L] = f[i] - r;
  }
}

// streaming of both colours (every node, the velocity at rest carried over)
__global__ void __launch_bounds__(TPB) k_stream_both(DevParams P, const double* __restrict__ ri,
                                                     const double* __restrict__ bi, double* __restrict__ ro,
                                                     double* __restrict__ bo) {
  const long long N = P.N, L = blockIdx.x * (long long)TPB + threadIdx.x;
  if (L >= N) return;
  const unsigned Lu = (unsigned)L, q = Lu / (unsigned)P.nz;
  const int z = (int)(Lu - q * (unsigned)P.nz), x = (int)(q / (unsigned)P.ny), y = (int)(q - (unsigned)x * P.ny);
#pragma unroll
  for (int i = 0; i < 19; i++) {
    const long long src = i * N + lin(P, wrapi(x - CX(i), P.nx), wrapi(y - CY(i), P.ny), wrapi(z - CZ(i), P.nz));
    ro[i * N + L] = ri[src];
    bo[i * N + L] = bi[src];
  }
}

// ---- initial state -----------------------------------------------------------
// initialization (Source1.f90:850-896), REFERENCE geometry
__global__ void k_initialization(DevParams P, double* rhoN, double* rho, double* rhoR, double* rhoB, double* ux,
                                 double* uy, double* uz, double* ri, double* bi, double* fi, double* ffi) {
  const long long L = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (L >= P.N) return;
  const int z = (int)(L % P.nz) + 1, y = (int)((L / P.nz) % P.ny) + 1,
            x = (int)(L / ((long long)P.nz * P.ny)) + 1;  // 1-based like the reference
  const double Rad_c = 30.0, lamda_d = ((double)P.ny - 2.0) * 2.0;
  const double x0 = (double)P.nx - 0.5, z0 = (double)P.nz - 0.5;
  const double dis = ((double)x - x0) * ((double)x - x0) + ((double)z - z0) * ((double)z - z0);
  const double dis_x = 0.1 * Rad_c * cos(2.0 * M_PI * ((double)y - 1.5) / lamda_d);
  const double star = Rad_c + dis_x - sqrt(dis);
  const double phi = tanh(star * 6.0 * P.beta * 0.134);
  const double plus = P.sigma / (Rad_c + dis_x) * 3.0;
  const double rh = phi > 0.0 ? P.rho0 + plus : P.rho0;
  const double R = rh * (phi + 1.0) / 2.0;
  const double B = rh - R;
  rhoN[L] = phi; rho[L] = rh; rhoR[L] = R; rhoB[L] = B; ux[L] = 0.0; uy[L] = 0.0; uz[L] = 0.0;
  const long long N = P.N;
#pragma unroll
  for (int i = 0; i < 19; i++) {
    const double r = feq_srt<double>(i, R, 0.0, 0.0, 0.0, 0.0), b = feq_srt<double>(i, B, 0.0, 0.0, 0.0, 0.0);
    ri[i * N + L] = r; bi[i * N + L] = b;
    if (fi) { fi[i * N + L] = r + b; ffi[i * N + L] = r + b; }
  }
}

// equilibrium fill from rhoN and rho (the fill of :883-894)
__global__ void k_init_fill(DevParams P, const double* rhoN, const double* rho, double* rhoR, double* rhoB,
                            double* ux, double* uy, double* uz, double* ri, double* bi, double* fi, double* ffi) {
  const long long L = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (L >= P.N) return;
  const double phi = rhoN[L], rh = rho[L];
  const double R = rh * (phi + 1.0) / 2.0;
  const double B = rh - R;
  rhoR[L] = R; rhoB[L] = B; ux[L] = 0.0; uy[L] = 0.0; uz[L] = 0.0;
  const long long N = P.N;
#pragma unroll
  for (int i = 0; i < 19; i++) {
    const double r = feq_srt<double>(i, R, 0.0, 0.0, 0.0, 0.0), b = feq_srt<double>(i, B, 0.0, 0.0, 0.0, 0.0);
    ri[i * N + L] = r; bi[i * N + L] = b;
    if (fi) { fi[i * N + L] = r + b; ffi[i * N + L] = r + b; }
  }
}

// splitmix64 finaliser (Steele, Lea, Flood 2014)
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
  unsigned long long z = x + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ double node_noise(long long L, double amp, unsigned long long seed) {
  const unsigned long long hsh = splitmix64(seed ^ (unsigned long long)L);
  const double u = (double)(hsh >> 11) * 0x1.0p-53;
  return u * (2.0 * amp) - amp;
}
// CONFIG Rayleigh-Plateau thread along z (same formula as configs.thread_phase)
__global__ void k_init_thread(DevParams P, double* rhoN, double* rho, double radius, double amp, double wavelength,
                              double width, double noise, unsigned long long seed) {
  const long long L = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (L >= P.N) return;
  const int z = (int)(L % P.nz), y = (int)((L / P.nz) % P.ny), x = (int)(L / ((long long)P.nz * P.ny));
  const double xc = (P.nx - 1) / 2.0, yc = (P.ny - 1) / 2.0;
  const double rz = radius * (1.0 + amp * cos(2.0 * M_PI * (double)z / wavelength));
  const double d = sqrt((x - xc) * (x - xc) + (y - yc) * (y - yc));
  double phi = tanh(2.0 * (rz - d) / width);
  if (noise > 0) phi = phi + node_noise(L, noise, seed);
  phi = fmin(fmax(phi, -1.0), 1.0);
  rhoN[L] = phi;
  rho[L] = phi > 0.0 ? P.rho0 + 3.0 * P.sigma / rz : P.rho0;
}
__global__ void k_init_slab(DevParams P, double* rhoN, double* rho, double z0, double z1, double width, double noise,
                            unsigned long long seed) {
  const long long L = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (L >= P.N) return;
  const int z = (int)(L % P.nz);
  const double dz = fmin((double)z - z0, z1 - (double)z);
  double phi = tanh(2.0 * dz / width);
  if (noise > 0) phi = phi + node_noise(L, noise, seed);
  phi = fmin(fmax(phi, -1.0), 1.0);
  rhoN[L] = phi;
  rho[L] = P.rho0;
}

// ---- diagnostics -----------------------------------------------------------
// deterministic block reduction of doubles (fixed tree for a fixed blockDim)
template <int NT>
__device__ __forceinline__ double block_sum(double v, double* sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
#pragma unroll
  for (int s = NT / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) sh[threadIdx.x] = sh[threadIdx.x] + sh[threadIdx.x + s];
    __syncthreads();
  }
  const double r = sh[0];
  __syncthreads();
  return r;
}

// per-z-plane sum of (1+phi)/2 over fluid nodes: one block per z
__global__ void k_plane_red(DevParams P, const double* __restrict__ rhoN, const int32_t* __restrict__ walls_all,
                            double* out) {
  __shared__ double sh[256];
  const int z = blockIdx.x;
  double s = 0.0;
  for (int t = threadIdx.x; t < P.nx * P.ny; t += 256) {
    const int x = t / P.ny, y = t % P.ny;
    const long long L = lin(P, x, y, z);
    if (walls_all[L] <= 0) s += (1.0 + rhoN[L]) * 0.5;
  }
  s = block_sum<256>(s, sh);
  if (threadIdx.x == 0) out[z] = s;
}

// output3 (Source1.f90:1686-1699): per y, the last phi sign change along z on plane x = xl-1
__global__ void k_output3(DevParams P, const double* __restrict__ rhoN, const int32_t* __restrict__ walls_all,
                          const int32_t* __restrict__ pout, double* bottom) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x + 1;  // 0-based y = 1..ny-2
  if (y > P.ny - 2) return;
  const int x = P.nx - 2;
  double b = 1.0;
  for (int z = 1; z <= P.nz - 2; z++) {
    const long long L = lin(P, x, y, z);
    if (pout[L] == 0 && walls_all[L] == 0) {
      const long long Ln = lin(P, x, y, z + 1);
      if (pout[Ln] == 0 && walls_all[Ln] == 0)
        if (rhoN[L] * rhoN[Ln] < 0.0) b = (double)(z + 2) - rhoN[Ln] / (rhoN[Ln] - rhoN[L]);
    }
  }
  bottom[y] = b;
}

// FP64 mass and momentum over fluid nodes: per-block partials
__global__ void k_mass_mom(DevParams P, const double* __restrict__ ri, const double* __restrict__ bi,
                           const int32_t* __restrict__ walls_all, double* part) {
  __shared__ double sh[256];
  const long long L = blockIdx.x * 256LL + threadIdx.x;
  double v[5] = {0, 0, 0, 0, 0};
  if (L < P.N && walls_all[L] <= 0) {
    const long long N = P.N;
#pragma unroll
    for (int i = 0; i < 19; i++) {
      const double r = ri[i * N + L], b = bi[i * N + L], f = r + b;
      v[0] += r; v[1] += b;
      v[2] += f * CX(i); v[3] += f * CY(i); v[4] += f * CZ(i);
    }
  }
  for (int k = 0; k < 5; k++) {
    const double s = block_sum<256>(v[k], sh);
    if (threadIdx.x == 0) part[blockIdx.x * 5LL + k] = s;
  }
}
__global__ void k_sum_partials(const double* part, long long nblk, int width, double* out) {
  __shared__ double sh[256];
  for (int k = 0; k < width; k++) {
    double s = 0.0;
    for (long long b = threadIdx.x; b < nblk; b += 256) s += part[b * width + k];
    s = block_sum<256>(s, sh);
    if (threadIdx.x == 0) out[k] = s;
  }
}

__global__ void k_aos_to_soa(const double* __restrict__ aos, double* __restrict__ soa, long long N) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= 19 * N) return;
  const long long L = t / 19;
  const int i = (int)(t % 19);
  soa[i * N + L] = aos[t];
}
__global__ void k_soa_to_aos(const double* __restrict__ soa, double* __restrict__ aos, long long N) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= 19 * N) return;
  const long long L = t / 19;
  const int i = (int)(t % 19);
  aos[t] = soa[i * N + L];
}

}  // namespace

// ===========================================================================
// host launchers
int ref_calmacros(sym_handle* h) {
  const DevParams& P = h->dp;
  k_calmacros<<<blocks_for(range_count(P)), TPB, 0, h->st>>>(P, h->ri, h->bi, h->fi, h->rho, h->ux, h->uy, h->uz,
                                                              h->rhoN, h->rhoR, h->rhoB, h->walls_all);
  if (P.ref) mirror_macros(h, true);
  return check_cuda(h, cudaGetLastError(), "calmacros");
}

// mirrored: rho_N is already on the mirror planes (inside a run of steps)
int ref_derivatives(sym_handle* h, bool mirrored) {
  const DevParams& P = h->dp;
  const unsigned g = blocks_for(range_count(P));
  k_pin_fill<<<blocks_for((P.N + 3) / 4), TPB, 0, h->st>>>(P, h->pin, h->walls_all, h->rhoN, mirrored);
  if (P.ref && !mirrored) {
    MirrorSet S;
    S.scalar[S.ns++] = h->rhoN;
    mirror(h, S);
  }
  auto go = [&](auto kern) {
    kern<<<g, TPB, 0, h->st>>>(P, h->dpart, h->pout, h->walls_all, h->rhoN, h->gx, h->gy, h->gz, h->nx, h->ny, h->nz,
                               h->flag);
  };
  if (P.ref) go(k_gradient<true>);
  else go(k_gradient<false>);
  return check_cuda(h, cudaGetLastError(), "derivatives");
}

int ref_collision(sym_handle* h) {
  const DevParams& P = h->dp;
  k_collision<<<blocks_for(range_count(P), 128), 128, 0, h->st>>>(P, h->walls_all, h->pout, h->flag, h->nx, h->ny,
                                                                   h->nz, h->gx, h->gy, h->gz, h->rho, h->rhoN,
                                                                   h->ux, h->uy, h->uz, h->fi, h->ffi);
  return check_cuda(h, cudaGetLastError(), "collision");
}

int ref_recolor(sym_handle* h) {
  const DevParams& P = h->dp;
  k_recolor<<<blocks_for(range_count(P)), TPB, 0, h->st>>>(P, h->walls_all, h->flag, h->fi, h->ri, h->bi, h->rhoR,
                                                            h->rhoB, h->rho, h->nx, h->ny, h->nz);
  return check_cuda(h, cudaGetLastError(), "recolor");
}

int ref_boundary(sym_handle* h, bool full) {
  const DevParams& P = h->dp;
  if (!P.ref) return SYM_OK;
  if (full) k_boundary<true><<<blocks_for(plane_count(P, true)), TPB, 0, h->st>>>(P, h->ri, h->bi);
  else k_boundary<false><<<blocks_for(plane_count(P, true)), TPB, 0, h->st>>>(P, h->ri, h->bi);
  return check_cuda(h, cudaGetLastError(), "boundary");
}

int ref_streaming(sym_handle* h, int which) {
  const DevParams& P = h->dp;
  double*& f = which == 0 ? h->ri : h->bi;
  if (P.ref) {
    // the streamed populations are the handle's from here on (the old array
    // becomes the temporary): no copy back of 18 of 19 velocities (152^3: 158 us
    // per colour)
    k_stream_pull<true><<<blocks_for(P.N), TPB, 0, h->st>>>(P, f, h->ft);
    std::swap(f, h->ft);
  } else {
    // a CONFIG handle's arrays stay where the fused path's tables point
    k_stream_pull<false><<<blocks_for(P.N), TPB, 0, h->st>>>(P, f, h->ft);
    cudaMemcpyAsync(f + P.N, h->ft + P.N, sizeof(double) * 18 * P.N, cudaMemcpyDeviceToDevice, h->st);
  }
  return check_cuda(h, cudaGetLastError(), "streaming");
}

int ref_curve(sym_handle* h) {
  const DevParams& P = h->dp;
  if (P.bounce)
    k_curve2<<<blocks_for(range_count(P)), TPB, 0, h->st>>>(P, h->dpart, h->walls, h->pout, h->ri, h->bi, h->rhoR,
                                                             h->rhoB);
  else
    k_curve<<<blocks_for((P.N + 3) / 4), TPB, 0, h->st>>>(P, h->dpart, h->walls, h->pout, h->ri, h->bi, h->rhoR,
                                                          h->rhoB);
  if (P.ref) mirror_colours(h);
  return check_cuda(h, cudaGetLastError(), "curve");
}

int ref_initialization(sym_handle* h) {
  const DevParams& P = h->dp;
  k_initialization<<<blocks_for(P.N), TPB, 0, h->st>>>(P, h->rhoN, h->rho, h->rhoR, h->rhoB, h->ux, h->uy, h->uz,
                                                        h->ri, h->bi, h->fi, h->ffi);
  return check_cuda(h, cudaGetLastError(), "initialization");
}

int ref_init_fill(sym_handle* h) {
  const DevParams& P = h->dp;
  k_init_fill<<<blocks_for(P.N), TPB, 0, h->st>>>(P, h->rhoN, h->rho, h->rhoR, h->rhoB, h->ux, h->uy, h->uz, h->ri,
                                                   h->bi, h->fi, h->ffi);
  return check_cuda(h, cudaGetLastError(), "init_fill");
}

int ref_init_thread(sym_handle* h, double radius, double amp, double wavelength, double width, double noise,
                    unsigned long long seed) {
  const DevParams& P = h->dp;
  k_init_thread<<<blocks_for(P.N), TPB, 0, h->st>>>(P, h->rhoN, h->rho, radius, amp, wavelength, width, noise, seed);
  return ref_init_fill(h);
}

int ref_init_slab(sym_handle* h, double z0, double z1, double width, double noise, unsigned long long seed) {
  const DevParams& P = h->dp;
  k_init_slab<<<blocks_for(P.N), TPB, 0, h->st>>>(P, h->rhoN, h->rho, z0, z1, width, noise, seed);
  return ref_init_fill(h);
}

int ref_neck_radius(sym_handle* h, double* rmin) {
  const DevParams& P = h->dp;
  k_plane_red<<<P.nz, 256, 0, h->st>>>(P, h->rhoN, h->walls_all, h->red);
  std::vector<double> s(P.nz);
  cudaMemcpyAsync(s.data(), h->red, sizeof(double) * P.nz, cudaMemcpyDeviceToHost, h->st);
  if (int e = check_cuda(h, cudaStreamSynchronize(h->st), "neck_radius")) return e;
  double mn = 1e300;
  for (int z = 0; z < P.nz; z++) mn = fmin(mn, sqrt(s[z] / M_PI));
  *rmin = mn;
  return SYM_OK;
}

int ref_output3(sym_handle* h, double* hmin, int32_t* y0) {
  const DevParams& P = h->dp;
  k_output3<<<blocks_for(P.ny), TPB, 0, h->st>>>(P, h->rhoN, h->walls_all, h->pout, h->red);
  std::vector<double> b(P.ny);
  cudaMemcpyAsync(b.data(), h->red, sizeof(double) * P.ny, cudaMemcpyDeviceToHost, h->st);
  if (int e = check_cuda(h, cudaStreamSynchronize(h->st), "output3")) return e;
  double hm = (double)P.nz;
  int yy = 0;
  const double top = (double)P.nz - 0.5;
  for (int y = 1; y <= P.ny - 2; y++) {
    const double hh = top - b[y];
    if (hh < hm) { hm = hh; yy = y + 1; }
  }
  *hmin = hm;
  *y0 = yy;
  return SYM_OK;
}

int ref_mass_momentum(sym_handle* h, double out[5]) {
  const DevParams& P = h->dp;
  const long long nblk = (P.N + 255) / 256;
  if ((size_t)(nblk * 5 + 8) > h->red_len) return set_error(h, SYM_ERR_STATE, "reduction scratch too small");
  k_mass_mom<<<(unsigned)nblk, 256, 0, h->st>>>(P, h->ri, h->bi, h->walls_all, h->red);
  k_sum_partials<<<1, 256, 0, h->st>>>(h->red, nblk, 5, h->red + nblk * 5);
  cudaMemcpyAsync(out, h->red + nblk * 5, sizeof(double) * 5, cudaMemcpyDeviceToHost, h->st);
  return check_cuda(h, cudaStreamSynchronize(h->st), "mass_momentum");
}

int aos_to_soa(sym_handle* h, const double* aos, double* soa) {
  k_aos_to_soa<<<blocks_for(19 * (long long)h->N), TPB, 0, h->st>>>(aos, soa, (long long)h->N);
  return check_cuda(h, cudaGetLastError(), "aos_to_soa");
}
int soa_to_aos(sym_handle* h, const double* soa, double* aos) {
  k_soa_to_aos<<<blocks_for(19 * (long long)h->N), TPB, 0, h->st>>>(soa, aos, (long long)h->N);
  return check_cuda(h, cudaGetLastError(), "soa_to_aos");
}

// ---- the pieces of a run of steps (see k_step_macros) ----
int ref_step_macros(sym_handle* h, bool pull, bool full) {
  const DevParams& P = h->dp;
  auto go = [&](auto kern) {
    kern<<<blocks_for(P.N), TPB, 0, h->st>>>(P, h->dpart, h->ri, h->bi, h->ft, h->ft2, h->kept, h->fi, h->rho, h->ux,
                                             h->uy, h->uz, h->rhoN, h->rhoR, h->rhoB, h->walls, h->walls_all, h->pout);
  };
  if (pull && full) go(k_step_macros<true, true>);
  else if (pull) go(k_step_macros<true, false>);
  else if (full) go(k_step_macros<false, true>);
  else go(k_step_macros<false, false>);
  if (pull) {
    std::swap(h->ri, h->ft);
    std::swap(h->bi, h->ft2);
  }
  if (full) {
    mirror_macros(h, true);
  } else {   // (images written by the kernel itself cost it 60 us in divergence, the pass 10)
    MirrorSet S;
    S.scalar[S.ns++] = h->rhoR;
    S.scalar[S.ns++] = h->rhoB;
    S.low = h->rhoN;
    mirror(h, S);
  }
  return check_cuda(h, cudaGetLastError(), "step macros");
}

// pulled: ref_step_macros(pull, !full) ran before it
int ref_collide_recolor(sym_handle* h, bool full, bool pulled) {
  const DevParams& P = h->dp;
  const unsigned g = blocks_for(range_count(P), 128);
  auto go = [&](auto kern) {
    kern<<<g, 128, 0, h->st>>>(P, tile_params<double>(P), h->walls_all, h->pout, h->flag, h->nx, h->ny, h->nz, h->gx,
                               h->gy, h->gz, h->rhoN, h->ux, h->uy, h->uz, h->fi, h->ffi, h->ri, h->bi, h->ft, h->ft2,
                               h->kept, h->walls_old, h->rhoR, h->rhoB);
  };
  if (full) go(k_collide_recolor<true, false>);
  else if (pulled) go(k_collide_recolor<false, true>);
  else go(k_collide_recolor<false, false>);
  return check_cuda(h, cudaGetLastError(), "collision and recolour");
}

int ref_stream_both(sym_handle* h) {
  k_stream_both<<<blocks_for(h->dp.N), TPB, 0, h->st>>>(h->dp, h->ri, h->bi, h->ft, h->ft2);
  std::swap(h->ri, h->ft);
  std::swap(h->bi, h->ft2);
  return check_cuda(h, cudaGetLastError(), "streaming");
}

// exported for particles.cu (the mirrors of set_walls and refilling)
void mirror_masks(sym_handle* h) {
  MirrorSet S;
  S.mask[0] = h->walls; S.mask[1] = h->walls_all; S.mask[2] = h->pin; S.mask[3] = h->pout;
  S.nm = 4;
  mirror(h, S);
}
void mirror_macros_all(sym_handle* h) { mirror_macros(h, false); }

}  // namespace symb200
