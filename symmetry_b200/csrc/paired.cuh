// paired.cuh -- the fused collide step for FP32 arithmetic (FP32 and 16-bit
// storage): a tile of 32(z) x 16(y) nodes marched along x by 256 threads, each
// of which holds two nodes, rows y and y + 8, in packed FP32 register pairs
// (nodemath.cuh, F2).
//
// Bound by instruction issue before (one node per thread: 1,943 instructions a
// node in 16-bit storage, 62 % of issue slots): packing halves the arithmetic.
// Rows 8 apart because every access then stays a contiguous warp access, and
// the shared-memory ring of normals can hold the two rows' values side by side
// -- pair row j is rows j and j + 8, so a stencil neighbour of a pair is again
// a pair (rows 7 and 8 are held twice).
//
// Populations are handled as their deviation g = f - w rho_ref from a rest
// equilibrium (16-bit storage: the node's own reference, which is how they are
// stored; FP32: rho0): the moments then carry no rounding of sums near 1,
// which in FP32 would drift the mass and drive a spurious flow.
#pragma once
#include "fused.cuh"

namespace symb200 {
namespace fused {

// 256-thread tile, pair rows -1 .. 8 and their z halo
constexpr int kPairRows = 8;
struct PairNormals {
  float4 xy[4][kPairRows + 2][BZ + 2];   // n_x of both rows, n_y of both rows
  float2 z_[4][kPairRows + 2][BZ + 2];
  float2 g[4][kPairRows + 2][BZ + 2];    // |grad phi|
};
template <typename S>
struct PairSmem {
  static constexpr int BY = 2 * kPairRows;
  static constexpr int kTile = (BY + 4) * (BZ + 4);
  static constexpr int kPhiSlot = (kTile * 4 + 127) / 128 * 128 / 4;
  static constexpr int kRefSlot = (kTile * 8 + 127) / 128 * 128 / 8;
  alignas(128) float phi[5][kPhiSlot];
  alignas(128) Ref ref[Codec<S>::kRef ? kIrrRing : 1][kRefSlot];
  alignas(16) PairNormals n;
  uint64_t bar[kIrrRing];
  unsigned char near_solid[kMaxExtent + 2];   // planes xa-1 .. xb
};

__host__ __device__ __forceinline__ constexpr float WF(int i) { return float(W(i)); }
constexpr float kFloatMax = 3.40282347e+38f;

template <typename S, bool SOLID>
__device__ __forceinline__ void collide_pair_tile(const TileParams<float>& P, const Pad& pd, const S* __restrict__ pin_,
                                                  S* __restrict__ pout_, const int32_t* __restrict__ walls,
                                                  const int32_t* __restrict__ walls_all,
                                                  const int32_t* __restrict__ pout,
                                                  const sym_particles* __restrict__ Sp, double* __restrict__ ffi,
                                                  const Ref* __restrict__ rr_old, int* status,
                                                  const CUtensorMap* tm_phi, const CUtensorMap* tm_ref, int z0, int y0,
                                                  int xa, int xb, PairSmem<S>& sm, unsigned& nload,
                                                  bool solid_rt = true) {
  constexpr int H = kPairRows;
  constexpr bool REF = Codec<S>::kRef;
  constexpr int kRow = BZ + 4;
  const bool SOLIDX = SOLID && solid_rt;
  const int tz = threadIdx.x % BZ, ty = threadIdx.x / BZ;
  const int sy = P.nz, sx = P.nz * P.ny;
  const int Ni = sx * P.nx;   // 19 N < 2^31 on the fused path
  const NodeParams<float>& np = P.np;
  const float evap = np.evap;

  // phi (and reference pairs) of plane xp by TMA, as in collide_tile
  const unsigned nl0 = nload;
  auto load_no = [&](int xp) { return nl0 + (unsigned)(xp - (xa - 2)); };
  constexpr uint32_t kTx = PairSmem<S>::kTile * (4 + (REF ? 8 : 0));
  auto load_phi = [&](int xp) {   // thread 0 only
    uint64_t* bar = &sm.bar[load_no(xp) % kIrrRing];
    tma::mbar_expect_tx(bar, kTx);
    tma::load_3d(sm.phi[(unsigned)(xp + 5) % 5u], tm_phi, z0, y0, xp + 2, bar);
    if (REF) tma::load_3d(sm.ref[(unsigned)(xp + kIrrRing) % kIrrRing], tm_ref, z0, y0, xp + 2, bar);
  };
  auto wait_phi = [&](int xp) {   // every thread
    const unsigned q = load_no(xp);
    if (!tma::mbar_wait(&sm.bar[q % kIrrRing], (q / kIrrRing) & 1u)) atomicOr(status, 2);
  };
  int ring_y, ring_z;
  ring_node(threadIdx.x, H, ring_y, ring_z);
  constexpr int kRing = 2 * (BZ + 2) + 2 * H;
  // unit normals (rotated at wetting nodes) and |grad phi| of plane xp: pair
  // row py - 1 is rows y0 + py - 1 and y0 + py + 7
  auto compute_n_as = [&](auto solidc, int xp) __attribute__((always_inline)) {
    constexpr bool solid = decltype(solidc)::value;
    const int s = xp & 3;
    const float* const pm = sm.phi[(unsigned)(xp + 4) % 5u];
    const float* const p0 = sm.phi[(unsigned)(xp + 5) % 5u];
    const float* const pp1 = sm.phi[(unsigned)(xp + 6) % 5u];
    auto one = [&](int py, int pz) __attribute__((always_inline)) {
      const int b = (py + 1) * kRow + pz + 1;
      auto at = [&](const float* p, int o) { return F2(p[b + o], p[b + o + H * kRow]); };
      // grad phi = 3 sum_i w_i c_i phi(x + c_i) (:510-521) from the differences
      // over opposite neighbours: an axis pair weighs twice a diagonal one
      const F2 ax = at(pp1, 0) - at(pm, 0), ay = at(p0, kRow) - at(p0, -kRow), az = at(p0, 1) - at(p0, -1);
      const F2 xyp = at(pp1, kRow) - at(pm, -kRow), xym = at(pp1, -kRow) - at(pm, kRow);
      const F2 xzp = at(pp1, 1) - at(pm, -1), xzm = at(pp1, -1) - at(pm, 1);
      const F2 yzp = at(p0, kRow + 1) - at(p0, -kRow - 1), yzm = at(p0, kRow - 1) - at(p0, -kRow + 1);
      const F2 k6 = F2(1.0f / 6.0f), k12 = F2(1.0f / 12.0f);
      const F2 g0 = vfma(k6, ax, k12 * ((xyp + xym) + (xzp + xzm)));
      const F2 g1 = vfma(k6, ay, k12 * ((xyp - xym) + (yzp + yzm)));
      const F2 g2 = vfma(k6, az, k12 * ((xzp - xzm) + (yzp - yzm)));
      const F2 g2s = vfma(g0, g0, vfma(g1, g1, g2 * g2));
      // |grad phi| and its reciprocal from one rsqrt
      F2 rf(g2s[0] > evap * evap ? rsqrtf(g2s[0]) : 0.f, g2s[1] > evap * evap ? rsqrtf(g2s[1]) : 0.f);
      F2 fn = g2s * rf;
      F2 n0 = g0 * rf, n1 = g1 * rf, n2 = g2 * rf;
      // a gradient that is not finite is none, as in the reference, whose test
      // against EVAP_LIM a NaN fails (0 times it would hand it to the neighbours)
      if (!(g2s[0] <= kFloatMax && g2s[1] <= kFloatMax)) {
        if (!(g2s[0] <= kFloatMax)) n0.v.x = n1.v.x = n2.v.x = fn.v.x = 0.f;
        if (!(g2s[1] <= kFloatMax)) n0.v.y = n1.v.y = n2.v.y = fn.v.y = 0.f;
      }
      if (solid) {
        // both rows' masks are read at once (nodes beyond the halo, read by
        // nobody, take the last one's)
        int wall[2], near[2];
        const int z = wrapi(min(z0 - 1 + pz, P.nz), P.nz);
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const unsigned Lw =
              (unsigned)(z + sy * wrapi(min(y0 - 1 + py + q * H, P.ny), P.ny) + sx * wrapi(xp, P.nx));
          wall[q] = walls_all[Lw];
          near[q] = pout[Lw];
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
          float a0 = n0[q], a1 = n1[q], a2 = n2[q];
          bool hit = false;
          if (wall[q] > 0) {
            a0 = a1 = a2 = 0.f;
            (q ? fn.v.y : fn.v.x) = 0.f;
            hit = true;
          } else {
            if (near[q] >= 1 && fn[q] > 0.f) {
              wet_rotate<float>(P, Sp, near[q], wrapi(xp, P.nx), wrapi(min(y0 - 1 + py + q * H, P.ny), P.ny), z, a0, a1,
                                a2);
              hit = true;
            }
          }
          if (hit) {
            (q ? n0.v.y : n0.v.x) = a0;
            (q ? n1.v.y : n1.v.x) = a1;
            (q ? n2.v.y : n2.v.x) = a2;
          }
        }
      }
      sm.n.xy[s][py][pz] = make_float4(n0[0], n0[1], n1[0], n1[1]);
      sm.n.z_[s][py][pz] = n2.v;
      sm.n.g[s][py][pz] = fn.v;
    };
    one(ty + 1, tz + 1);   // the thread's own pair, then the ring around the tile
    if (threadIdx.x < kRing) one(ring_y, ring_z);
  };
  // every plane is compiled twice, with and without solids; a plane's flag is
  // the whole CTA's, and the code of the planes without stays that of a domain
  // without (switching solids node by node inside one code took 1.6 times as long)
  auto near_solid = [&](int xp) { return SOLIDX && sm.near_solid[xp - xa + 1]; };
  auto compute_n = [&](int xp) {
    if constexpr (SOLID) {
      if (near_solid(xp)) {
        compute_n_as(std::true_type{}, xp);
        return;
      }
    }
    compute_n_as(std::false_type{}, xp);
  };

  if (threadIdx.x == 0)
    for (int xp = xa - 2; xp <= xa + 2; xp++) load_phi(xp);
  if (SOLIDX) {
    for (int t = threadIdx.x; t < xb - xa + 2; t += kTPB)
      sm.near_solid[t] = solid_near(P, Sp, PairSmem<S>::BY, xa - 1 + t, y0, z0);
    __syncthreads();
  }
  wait_phi(xa - 2);
  wait_phi(xa - 1);
  nload = nl0 + (unsigned)(xb - xa + 4);   // loads of this tile: planes xa-2 .. xb+1

  const int z = z0 + tz;
  int yc[2], y[2];
  bool inr[2];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    y[q] = y0 + ty + q * H;
    inr[q] = y[q] < P.ny && z < P.nz;
    yc[q] = min(y[q], P.ny - 1);
  }
  const int zc = min(z, P.nz - 1);
  const int ozp = (zc == P.nz - 1) ? -(P.nz - 1) : 1, ozm = (zc == 0) ? (P.nz - 1) : -1;
  int oyp[2], oym[2];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    oyp[q] = (yc[q] == P.ny - 1) ? -(P.ny - 1) * sy : sy;
    oym[q] = (yc[q] == 0) ? (P.ny - 1) * sy : -sy;
  }
  using Raw = typename std::conditional<REF, __half2, float2>::type;
  // 16-bit storage: a plane's populations are loaded before its normals are
  // computed (38 registers; 128x128x256: 197 -> 165 us); FP32's 76 do not fit
  // beside them.
  constexpr bool kEarly = REF;
  // the node arithmetic and pushes of plane x
  auto plane = [&](auto solidc, int x) __attribute__((always_inline)) {
    constexpr bool solid = decltype(solidc)::value;
    Raw raw[2][19];   // this plane's populations
    Ref ref[2] = {Ref{}, Ref{}};
    unsigned L[2];
    auto load = [&](int x) __attribute__((always_inline)) {
#pragma unroll
      for (int q = 0; q < 2; q++) {
        L[q] = (unsigned)(zc + sy * yc[q] + sx * x);
        const Raw* const in = reinterpret_cast<const Raw*>(pin_) + L[q];
#pragma unroll
        for (int i = 0; i < 19; i++) raw[q][i] = in[i * Ni];
        if (REF) ref[q] = rr_old[pd.idx(x, yc[q], zc)];
      }
    };
    load(x);
    if constexpr (kEarly) {
      wait_phi(x + 2);
      compute_n(x + 1);
      __syncthreads();
    }
    bool act[2] = {inr[0], inr[1]};
    int pp[2] = {0, 0};
    if (solid) {
      const int w0 = walls_all[L[0]], w1 = walls_all[L[1]], p0 = pout[L[0]], p1 = pout[L[1]];
      if (w0 > 0) act[0] = false; else pp[0] = p0;
      if (w1 > 0) act[1] = false; else pp[1] = p1;
    }
    if (!(act[0] || act[1])) return;
    // deviations from the rest equilibrium, and the colour densities
    F2 g[19], rho_ref, rho, sr, sb;
    Moments<F2> m;
    if constexpr (REF) {
      rho_ref = F2(ref[0].x, ref[1].x);
      const F2 chi(ref[0].y, ref[1].y);
      F2 d[19];
#pragma unroll
      for (int i = 0; i < 19; i++) {
        const float2 a = __half22float2(raw[0][i]), b = __half22float2(raw[1][i]);
        g[i] = F2(a.x, b.x) * F2(float(W(i) / 4096.0));
        d[i] = F2(a.y, b.y);
      }
      to_moments<F2, float>(g, m);
      rho = rho_ref + m.rho;
      F2 da = d[1], dd = d[7];
#pragma unroll
      for (int i = 2; i < 7; i++) da = da + d[i];
#pragma unroll
      for (int i = 8; i < 19; i++) dd = dd + d[i];
      // sr = chi rho + sum of the red deviations: exactly rho or 0 in a pure phase
      const F2 dev = vfma(F2(float(W(0) / 4096.0)), d[0],
                          vfma(F2(float(W(1) / 4096.0)), da, F2(float(W(7) / 4096.0)) * dd));
      sr = vfma(chi, rho, dev);
      sb = rho - sr;
    } else {
      rho_ref = F2(P.rho0);
      F2 c0(raw[0][0]), c1(raw[1][0]);   // (red, blue) sums of each node
#pragma unroll
      for (int i = 0; i < 19; i++) {
        const float w = WF(i) * P.rho0;
        g[i] = F2((raw[0][i].x - w) + raw[0][i].y, (raw[1][i].x - w) + raw[1][i].y);
        if (i) {
          c0 = c0 + F2(raw[0][i]);
          c1 = c1 + F2(raw[1][i]);
        }
      }
      to_moments<F2, float>(g, m);
      rho = rho_ref + m.rho;
      sr = F2(c0[0], c1[0]);
      sb = F2(c0[1], c1[1]);
    }
    const float4 nxy = sm.n.xy[x & 3][ty + 1][tz + 1];
    const F2 nx(nxy.x, nxy.y), ny(nxy.z, nxy.w), nz(sm.n.z_[x & 3][ty + 1][tz + 1]);
    const F2 fn(sm.n.g[x & 3][ty + 1][tz + 1]);
    F2 irho, su, sq;
    {
      const float* const ph = sm.phi[(unsigned)(x + 5) % 5u] + (ty + 2) * kRow + tz + 2;
      float a[2], b[2], c[2];
#pragma unroll
      for (int q = 0; q < 2; q++) node_rates_fused<float>(P, ph[q * H * kRow], rho[q], a[q], b[q], c[q]);
      irho = F2(a[0], a[1]);
      su = F2(b[0], b[1]);
      sq = F2(c[0], c[1]);
    }
    // CSF surface tension from the curvature of the normal field (:624-667);
    // nodes without a normal have n = 0 and |grad phi| = 0
    F2 val;
    {
      const F2 kurv = curvature<F2, float>(
          [&](auto ic, F2 (&d)[3]) {
            constexpr int i = decltype(ic)::value;
            const int sp = (x + CX(i)) & 3, s2 = (x - CX(i)) & 3;
            const float4 p = sm.n.xy[sp][ty + 1 + CY(i)][tz + 1 + CZ(i)];
            const float4 q = sm.n.xy[s2][ty + 1 - CY(i)][tz + 1 - CZ(i)];
            d[0] = F2(p.x, p.y) - F2(q.x, q.y);
            d[1] = F2(p.z, p.w) - F2(q.z, q.w);
            d[2] = F2(sm.n.z_[sp][ty + 1 + CY(i)][tz + 1 + CZ(i)]) - F2(sm.n.z_[s2][ty + 1 - CY(i)][tz + 1 - CZ(i)]);
          },
          nx, ny, nz);
      val = F2(np.half_sigma) * kurv * fn;
      if (solid) val = F2(pp[0] > 0 ? 0.f : val[0], pp[1] > 0 ? 0.f : val[1]);
    }
    const F2 fx = vfma(val, nx, rho * F2(np.body[0])), fy = vfma(val, ny, rho * F2(np.body[1])),
             fz = vfma(val, nz, rho * F2(np.body[2]));
    const F2 h(0.5f);
    relax<F2, float>(m, rho, vfma(h, fx, m.jx) * irho, vfma(h, fy, m.jy) * irho, vfma(h, fz, m.jz) * irho, fx, fy, fz,
                     su, np.s_e > 0.f ? F2(np.s_e) : su, np.s_eps > 0.f ? F2(np.s_eps) : su,
                     np.s_q > 0.f ? F2(np.s_q) : sq, np.s_pi > 0.f ? F2(np.s_pi) : su,
                     np.s_m > 0.f ? F2(np.s_m) : sq);
    from_moments<F2, float>(m, g);
    // Latva-Kokko recolouring (:712-726) as in collide_tile
    F2 ratio, cd;
    {
      const F2 t = sr * irho;
      const F2 c = sb * t * F2(np.beta * (REF ? 4096.0f : 1.0f / 36.0f));
      float a[2], b[2];
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const bool rz = sr[q] <= evap, bz = sb[q] <= evap;
        a[q] = bz ? 1.f : (rz ? 0.f : t[q]);
        b[q] = bz || rz ? 0.f : c[q];
      }
      ratio = F2(a[0], a[1]);
      cd = F2(b[0], b[1]);
    }
    const F2 cnx = cd * nx, cny = cd * ny, cnz = cd * nz;
    const int oxp = (x == P.nx - 1) ? -(P.nx - 1) * sx : sx, oxm = (x == 0) ? (P.nx - 1) * sx : -sx;
    // links that come back (bit i: the push along c_i enters a solid, curve
    // :1001-1019), from a wall without velocity (flat) or from particle pp; the
    // neighbours' masks are read together, not one per push
    unsigned back[2] = {0, 0}, flat[2] = {0, 0};
    float uw[2][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
    if (solid) {
#pragma unroll
      for (int q = 0; q < 2; q++) {
        if (!(act[q] && pp[q] >= 1)) continue;
        const int par = P.par;
        static_for<18>([&](auto kc) {
          constexpr int i = decltype(kc)::value + 1;
          const int wb = walls[(int)L[q] + (CX(i) > 0 ? oxp : (CX(i) < 0 ? oxm : 0)) +
                               (CY(i) > 0 ? oyp[q] : (CY(i) < 0 ? oym[q] : 0)) +
                               (CZ(i) > 0 ? ozp : (CZ(i) < 0 ? ozm : 0))];
          if (wb > par) flat[q] |= 1u << i;
          else if (wb == pp[q]) back[q] |= 1u << i;
        });
        back[q] |= flat[q];
        if (pp[q] <= par) {
          // rigid-body velocity of the particle at this node (curve :1009-1014)
          const int k = pp[q] - 1;
          const float xr = float(disp(P, (double)(x + P.origin), Sp->center[0 * par + k], 0));
          const float yr = float(disp(P, (double)(y[q] + P.origin), Sp->center[1 * par + k], 1));
          const float zr = float(disp(P, (double)(z + P.origin), Sp->center[2 * par + k], 2));
          const float w0 = float(Sp->rp[0 * par + k]), w1 = float(Sp->rp[1 * par + k]), w2 = float(Sp->rp[2 * par + k]);
          uw[q][0] = float(Sp->up[0 * par + k]) + zr * w1 - yr * w2;
          uw[q][1] = float(Sp->up[1 * par + k]) + xr * w2 - zr * w0;
          uw[q][2] = float(Sp->up[2 * par + k]) + yr * w0 - xr * w1;
          // post-collision populations for the momentum exchange (:1241-1243),
          // read only next to particles
#pragma unroll
          for (int i = 0; i < 19; i++) ffi[(size_t)i * Ni + L[q]] = (double)fmaf(WF(i), rho_ref[q], g[i][q]);
        }
      }
    }
    // pushes.  16-bit storage: with F = 4096 f / w the stored pair is
    //   q = F - 4096 rho_dst = g 4096/w + 4096 (rho_ref - rho_dst)
    //   d = 4096 (r - chi_dst f) / w = (ratio - chi_dst) F + 4096 a / w
    // where (4096 (rho_ref - rho_dst), ratio - chi_dst) is one packed
    // multiply-add on the destination's reference pair and a, the recolouring
    // of the link, is cn summed over its axes on axis and diagonal links alike
    // after the division by w.  d is exactly 0 in a pure phase.
    const F2 r4 = rho_ref * F2(4096.0f);
    const F2 src[2] = {F2(r4[0], ratio[0]), F2(r4[1], ratio[1])};
    Raw* const out[2] = {reinterpret_cast<Raw*>(pout_) + L[0], reinterpret_cast<Raw*>(pout_) + L[1]};
    [[maybe_unused]] const Ref* refp[3];   // this node's place in the reference pairs of planes x-1, x, x+1
    if constexpr (REF) {
#pragma unroll
      for (int k = 0; k < 3; k++)
        refp[k] = sm.ref[(unsigned)(x + k - 1 + kIrrRing) % kIrrRing] + (ty + 2) * kRow + tz + 2;
    }
    const F2 c2x = cnx + cnx, c2y = cny + cny, c2z = cnz + cnz;
    static_for<19>([&](auto kc) __attribute__((always_inline)) {
      constexpr int i = decltype(kc)::value;
      F2 a(0.f);   // recolouring of the link
      if constexpr (i >= 1 && i < 7) {
        const F2 c = REF ? (CX(i) ? cnx : (CY(i) ? cny : cnz)) : (CX(i) ? c2x : (CY(i) ? c2y : c2z));
        a = CX(i) + CY(i) + CZ(i) > 0 ? c : F2(0.f) - c;
      } else if constexpr (i >= 7) {
        constexpr int s1 = CX(i) ? CX(i) : CY(i), s2 = CZ(i) ? CZ(i) : CY(i);
        const F2 c1 = CX(i) ? cnx : cny, c2 = CZ(i) ? cnz : cny;
        a = s1 > 0 ? (s2 > 0 ? c1 + c2 : c1 - c2) : (s2 > 0 ? c2 - c1 : F2(0.f) - (c1 + c2));
      }
      constexpr float c = float(4096.0 / W(i));
      const F2 f = REF ? vfma(g[i], F2(c), r4) : vfma(F2(WF(i)), rho_ref, g[i]);
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int o = i * Ni + (CX(i) > 0 ? oxp : (CX(i) < 0 ? oxm : 0)) +
                      (CY(i) > 0 ? oyp[q] : (CY(i) < 0 ? oym[q] : 0)) + (CZ(i) > 0 ? ozp : (CZ(i) < 0 ? ozm : 0));
        if (solid && act[q] && pp[q] >= 1) {
          const float fi = fmaf(WF(i), rho_ref[q], g[i][q]);
          const float r = fmaf(ratio[q], fi, REF ? a[q] * float(W(i) / 4096.0) : a[q]);
          // interpolated bounce-back: the red post-collision populations of the
          // nodes next to particles, for the link update after this kernel
          if (P.bounce && pp[q] <= P.par) ffi[(size_t)(19 + i) * Ni + L[q]] = (double)r;
          if (i > 0 && (back[q] >> i & 1u)) {
            // comes back as the opposite link of this node
            constexpr int j = OPC(i);
            const float star = (flat[q] >> i & 1u) ? 0.f
                                                   : float(6.0 * W(j)) * (uw[q][0] * float(CX(j)) +
                                                                          uw[q][1] * float(CY(j)) +
                                                                          uw[q][2] * float(CZ(j)));
            const float rr = fmaf(sr[q], star, r), ff = rr + fmaf(sb[q], star, fi - r);
            Raw v;
            if constexpr (REF) {
              const Ref rd = refp[1][q * H * kRow];
              v = __floats2half2_rn((ff - __fmul_rn(WF(j), rd.x)) * c, fmaf(-rd.y, ff, rr) * c);
            } else {
              v = make_float2(rr, ff - rr);
            }
            out[q][j * Ni] = v;
            continue;
          }
        }
        Raw v;
        if constexpr (REF) {
          const Ref rd = refp[CX(i) + 1][q * H * kRow + CY(i) * kRow + CZ(i)];
          const F2 t = vfma(F2(rd), F2(-4096.0f, -1.0f), src[q]);
          v = __floats2half2_rn(fmaf(g[i][q], c, t[0]), fmaf(t[1], f[q], a[q]));
        } else {
          const float r = fmaf(ratio[q], f[q], a[q]);
          v = make_float2(r, f[q] - r);
        }
        if (act[q]) out[q][o] = v;
      }
    });
  };
  if constexpr (kEarly) {
#pragma unroll 1
    for (int x = xa - 2; x < xa; x++) {
      wait_phi(x + 2);
      compute_n(x + 1);
    }
    // the first phi load below reuses the slot of plane xa-2, read by the first turn
    __syncthreads();
  }
  // (otherwise the first two turns only compute normals)
#pragma unroll 1
  for (int x = kEarly ? xa : xa - 2; x < xb; x++) {
    // phi of plane x+3 on its way; normals of plane x+1 from phi planes x..x+2.
    // The slots the load overwrites (phi of plane x-2, reference pairs of plane
    // x-3) were last read before the previous plane's barrier.
    if (threadIdx.x == 0 && x >= xa && x + 3 <= xb + 1) load_phi(x + 3);
    if constexpr (!kEarly) {
      wait_phi(x + 2);
      compute_n(x + 1);
      if (x != xa - 2) __syncthreads();
      if (x < xa) continue;
    }
    if constexpr (SOLID) {
      if (near_solid(x)) {
        plane(std::true_type{}, x);
        continue;
      }
    }
    plane(std::false_type{}, x);
  }
}

// ---- one tile of any storage -------------------------------------------------------
template <typename S>
using TileSmem = typename std::conditional<std::is_same<S, double>::value, Smem, PairSmem<S>>::type;
// dynamic shared memory of the collide kernels: the TileSmem block on a 128-byte
// boundary inside the allocation
template <typename S>
constexpr size_t smem_bytes() { return sizeof(TileSmem<S>) + 128; }
template <typename S>
__device__ __forceinline__ TileSmem<S>& smem_view(unsigned char* raw) {
  // an offset from the shared array, so that the accesses stay shared-memory
  // instructions (an aligned integer address would make them generic ones)
  const uint32_t pad = (128u - (tma::smem_addr(raw) & 127u)) & 127u;
  return *reinterpret_cast<TileSmem<S>*>(raw + pad);
}
// the CTA's mbarriers: initialised once per kernel by thread 0
template <typename S>
__device__ __forceinline__ void collide_init_barriers(TileSmem<S>& sm) {
  if (threadIdx.x == 0) {
    for (int k = 0; k < kIrrRing; k++) tma::mbar_init(&sm.bar[k], 1);
    tma::mbar_fence_init();
  }
  __syncthreads();
}
// Resident CTAs per SM the collide kernels are compiled for: 2 of 256 threads at
// 128 registers.
template <typename S>
constexpr int collide_ctas() { return 2; }

template <typename S, bool SOLID>
__device__ __forceinline__ void collide_any(const TileParams<typename Codec<S>::R>& P, const Pad& pd, const S* pin_, S* pout_,
                                            const int32_t* walls, const int32_t* walls_all, const int32_t* pout,
                                            const sym_particles* Sp, double* ffi, const Ref* rr_old,
                                            Acc::T* acc, int* status,
                                            const CUtensorMap* tm_phi, const CUtensorMap* tm_ref, int z0, int y0, int xa,
                                            int xb, TileSmem<S>& sm, unsigned& nload, bool solid_rt = true) {
  if constexpr (std::is_same<S, double>::value)
    collide_tile<SOLID>(P, pin_, pout_, walls, walls_all, pout, Sp, ffi, acc, status, tm_phi, z0, y0, xa, xb, sm, nload,
                        solid_rt);
  else
    collide_pair_tile<S, SOLID>(P, pd, pin_, pout_, walls, walls_all, pout, Sp, ffi, rr_old, status, tm_phi, tm_ref, z0,
                                y0, xa, xb, sm, nload, solid_rt);
}

template <typename S, bool SOLID>
__global__ void __launch_bounds__(kTPB, collide_ctas<S>())
    k_collide(const __grid_constant__ TileParams<typename Codec<S>::R> P, Pad pd, const S* __restrict__ pin_, S* __restrict__ pout_,
              const int32_t* __restrict__ walls, const int32_t* __restrict__ walls_all,
              const int32_t* __restrict__ pout, const sym_particles* __restrict__ Sp, double* __restrict__ ffi,
              const Ref* __restrict__ rr_old, Acc::T* acc, int* status,
              const __grid_constant__ CUtensorMap tm_phi, const __grid_constant__ CUtensorMap tm_ref, int xchunk) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  TileSmem<S>& sm = smem_view<S>(smem_raw);
  collide_init_barriers<S>(sm);
  unsigned nload = 0;
  const int xa = blockIdx.z * xchunk;
  collide_any<S, SOLID>(P, pd, pin_, pout_, walls, walls_all, pout, Sp, ffi, rr_old, acc, status, &tm_phi, &tm_ref,
                        blockIdx.x * BZ, blockIdx.y * kBY<S>, xa, min(xa + xchunk, P.nx), sm, nload);
}

}  // namespace fused
}  // namespace symb200
