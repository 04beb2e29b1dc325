// fused.cuh -- device code of the fused fast path, shared by the
// single-domain driver (fast.cu) and the batch engine (batch.cu).
// See fast.cu for the per-step kernel sequence.
#pragma once
#include <cuda_fp16.h>
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <utility>
#include <vector>
#include "nodemath.cuh"
#include "state.cuh"
#include "tma.cuh"

namespace symb200 {
namespace fused {

constexpr int BZ = 32;   // tile width along z: one warp per row
constexpr int XCHUNK = 32;   // most x planes marched by one CTA

// A pointer read from a descriptor, marked as one to global memory: its accesses
// are then global loads and stores (through a pointer of unknown space they are
// generic ones, which also wait for the shared-memory writes around them:
// 16-bit collide of a one-domain batch 328 us against 163 alone).
template <typename T>
__device__ __forceinline__ T* as_global(T* p) {
  return static_cast<T*>(__cvta_global_to_generic(__cvta_generic_to_global(p)));
}

// ---- halo-padded phase field -----------------------------------------------------
struct Pad {
  int nxp, nyp, nzp;
  __host__ __device__ long long idx(int x, int y, int z) const {
    return (long long)(z + 2) + (long long)nzp * ((long long)(y + 2) + (long long)nyp * (long long)(x + 2));
  }
  __host__ __device__ long long size() const { return (long long)nxp * nyp * nzp; }
};
inline Pad make_pad(const DevParams& P) {
  Pad d;
  d.nxp = P.nx + 4;
  d.nyp = P.ny + 4;
  d.nzp = ((P.nz + 4) + 3) / 4 * 4;   // row stride a multiple of 16 bytes
  return d;
}

// store v at (x,y,z) and at each periodic image inside the 2-deep ghost layers
// (per axis: +n when within 2 of the low face, -n within 2 of the high face;
// both for n = 3).  Nodes 2 or more from every face store once.
template <typename R>
__device__ __forceinline__ void phi_store(const DevParams& P, const Pad& pd, R* phi, int x, int y, int z, R v) {
  if (x >= 2 && x < P.nx - 2 && y >= 2 && y < P.ny - 2 && z >= 2 && z < P.nz - 2) {
    phi[pd.idx(x, y, z)] = v;
    return;
  }
  int xs[3], ys[3], zs[3], nx = 1, ny = 1, nz = 1;
  xs[0] = x; ys[0] = y; zs[0] = z;
  if (x < 2) xs[nx++] = x + P.nx;
  if (x >= P.nx - 2) xs[nx++] = x - P.nx;
  if (y < 2) ys[ny++] = y + P.ny;
  if (y >= P.ny - 2) ys[ny++] = y - P.ny;
  if (z < 2) zs[nz++] = z + P.nz;
  if (z >= P.nz - 2) zs[nz++] = z - P.nz;
  for (int a = 0; a < nx; a++)
    for (int b = 0; b < ny; b++)
      for (int c = 0; c < nz; c++) phi[pd.idx(xs[a], ys[b], zs[c])] = v;
}

// ---- population storage codecs --------------------------------------------------
// Each velocity i holds an array of N slot pairs, pair index i*N + L: one
// aligned 2-slot load or store per velocity (8/16-byte pairs, 4-byte for the
// 16-bit storage), so a warp moves whole 128-byte lines per instruction.
// FP64 / FP32: the pair is (r, b).
// 16-bit storage (shifted storage, FP32 arithmetic): the pair is two FP16
// numbers relative to a reference pair (rho_ref, chi_ref) -- the density and
// red fraction of the node the population is stored at, from the step that
// wrote it (FP32):
//   q = 4096 (f - w rho_ref) / w    the total's deviation from its rest
//                                   equilibrium (the Laplace pressure jump
//                                   does not eat the significand; the 2^12
//                                   scale keeps deviations down to 1e-8 out
//                                   of the FP16 subnormal range)
//   d = 4096 (r - chi_ref f) / w    the red population's deviation from the
//                                   node's colour split of f: exactly 0 in a
//                                   pure phase, and the small colour
//                                   perturbations that seed an instability
//                                   keep FP16's 2^-11 relative precision
//                                   instead of a fixed step (no quotient)
// Encoder and decoder share the rounded rest equilibrium e = w rho_ref (one
// product, never contracted), so the rounding of the scale factors multiplies
// only the deviation and adds no bias to the mass.
// Indices are 32-bit pair offsets (the fused path requires 38*N < 2^32).
// load and store take the reference pair of the node the population is
// stored at (only the 16-bit codec uses it; kRef says whether it does).
using Ref = float2;
template <typename S>
struct Codec;
template <>
struct Codec<double> {
  using R = double;
  static constexpr bool kRef = false;
  template <int I>
  __device__ __forceinline__ static void load(const double* __restrict__ p, unsigned N, unsigned L, Ref, R& r, R& b) {
    const double2 v = reinterpret_cast<const double2*>(p)[I * N + L];
    r = v.x;
    b = v.y;
  }
  // total f = r + b and red r
  template <int I>
  __device__ __forceinline__ static void load_fr(const double* __restrict__ p, unsigned N, unsigned L, Ref, R& f,
                                                 R& r) {
    const double2 v = reinterpret_cast<const double2*>(p)[I * N + L];
    r = v.x;
    f = v.x + v.y;
  }
  template <int I>
  __device__ __forceinline__ static void store(double* p, unsigned N, unsigned L, Ref, R r, R f) {
    reinterpret_cast<double2*>(p)[I * N + L] = make_double2(r, f - r);
  }
};
template <>
struct Codec<float> {
  using R = float;
  static constexpr bool kRef = false;
  template <int I>
  __device__ __forceinline__ static void load(const float* __restrict__ p, unsigned N, unsigned L, Ref, R& r, R& b) {
    const float2 v = reinterpret_cast<const float2*>(p)[I * N + L];
    r = v.x;
    b = v.y;
  }
  template <int I>
  __device__ __forceinline__ static void load_fr(const float* __restrict__ p, unsigned N, unsigned L, Ref, R& f,
                                                 R& r) {
    const float2 v = reinterpret_cast<const float2*>(p)[I * N + L];
    r = v.x;
    f = v.x + v.y;
  }
  template <int I>
  __device__ __forceinline__ static void store(float* p, unsigned N, unsigned L, Ref, R r, R f) {
    reinterpret_cast<float2*>(p)[I * N + L] = make_float2(r, f - r);
  }
};
template <>
struct Codec<__half> {
  using R = float;
  static constexpr bool kRef = true;
  // total f and red r
  template <int I>
  __device__ __forceinline__ static void load_fr(const __half* __restrict__ p, unsigned N, unsigned L, Ref ref, R& f,
                                                 R& r) {
    const float2 q = __half22float2(reinterpret_cast<const __half2*>(p)[I * N + L]);
    f = fmaf(q.x, float(W(I) / 4096.0), __fmul_rn(float(W(I)), ref.x));
    r = fmaf(q.y, float(W(I) / 4096.0), ref.y * f);
  }
  template <int I>
  __device__ __forceinline__ static void load(const __half* __restrict__ p, unsigned N, unsigned L, Ref ref, R& r,
                                              R& b) {
    R f;
    load_fr<I>(p, N, L, ref, f, r);
    b = f - r;
  }
  template <int I>
  __device__ __forceinline__ static void store(__half* p, unsigned N, unsigned L, Ref ref, R r, R f) {
    constexpr float c = float(4096.0 / W(I));   // 12288, 73728 or 147456: exact
    const R q = (f - __fmul_rn(float(W(I)), ref.x)) * c;
    // exactly 0 in a pure phase: r = f with chi_ref = 1, r = 0 with chi_ref = 0
    const R d = fmaf(-ref.y, f, r) * c;
    reinterpret_cast<__half2*>(p)[I * N + L] = __floats2half2_rn(q, d);
  }
};
// the reference pair of node colour densities (sr, sb): density and red
// fraction (a pure phase exactly 1 or 0)
__device__ __forceinline__ Ref ref_pair(float sr, float sb) {
  const float rho = sr + sb;
  return make_float2(rho, sr / rho);
}
// the reference pair of a node with no populations of its own (solid): the
// rest density, half red
__device__ __forceinline__ Ref ref_rest(const DevParams& P) { return make_float2(float(P.rho0), 0.5f); }

// ---- next-step colour densities accumulated by the collide kernel ----------------
// The collide kernel of a step pushes every post-collision population to the
// node that holds it after streaming; it also adds the pushed values per
// destination node into two fixed-point accumulators (red, blue), so the next
// step's phase field (calmacros) reads 2 numbers per node instead of all 38
// populations.  Integer addition is associative, so the totals do not depend
// on the order in which the tiles' atomic adds land: the accumulated densities
// are deterministic.  64-bit integers in units of 2^-52 (|rho| < 1024).  The
// share that each of three planes sends to a node is rounded by itself, three
// roundings of 1.1e-16 where one of the whole sum would do: the price of totals
// that do not depend on the tiles' x extents.  A value outside the range or not
// finite sets the domain's status word, and the next phase field is written as
// NaN (the NaN test of the stop rule then retires the run).
struct Acc {
  using T = unsigned long long;
  __device__ __forceinline__ static T fix(double v) { return (T)__double2ll_rn(v * 0x1p52); }
  __device__ __forceinline__ static double val(T a) { return (double)(long long)a * 0x1p-52; }
  __device__ __forceinline__ static bool ok(double v) { return fabs(v) < 1024.0; }
};
// Whether the collide kernel of storage S accumulates the next step's colour
// densities (the phase field then reads 2 values per node) or the phase field
// re-reads the populations (38 per node).  The accumulation costs arithmetic
// (warp shuffles, a shared-memory exchange, atomics), the re-read costs
// bytes: FP64 storage, bound by memory, accumulates; the 16-bit storage, bound
// by arithmetic, re-reads, and FP32 does (accumulating was measured slower for
// both with one node per thread: +2.7 ms of collide for -0.4 ms of phase on 45 M
// nodes in 16 bits).
template <typename S>
constexpr bool kAccumulate = sizeof(S) == 8;

// add v to accumulator p (a reduction: nothing is returned); an out-of-range
// value sets *status and counts as nothing
__device__ __forceinline__ void acc_add(Acc::T* p, double v, int* status) {
  if (Acc::ok(v)) atomicAdd(p, Acc::fix(v));
  else atomicOr(status, 1);
}

template <typename F, int... Is>
__device__ __forceinline__ void unroll19_impl(F&& f, std::integer_sequence<int, Is...>) {
  (f(std::integral_constant<int, Is>{}), ...);
}
template <typename F>
__device__ __forceinline__ void unroll19(F&& f) {
  unroll19_impl(f, std::make_integer_sequence<int, 19>{});
}

// ---- calmacros (Source1.f90:770-831) on the fused state ---------------------------
// Storages that do not accumulate: phi = (rhoR - rhoB) / rho from the node's
// own post-stream populations; 0 on solid nodes.  16-bit storage decodes with
// the reference pairs rr_old and records the node's (rho, red fraction) in rr_new:
// the references this step's encoders use and the next step decodes with.
template <typename S, bool SOLID>
__device__ __forceinline__ void phase_node(const DevParams& P, const Pad& pd, const S* __restrict__ pops,
                                           typename Codec<S>::R* __restrict__ phi,
                                           const int32_t* __restrict__ walls_all, const Ref* __restrict__ rr_old,
                                           Ref* __restrict__ rr_new, long long L) {
  using R = typename Codec<S>::R;
  if (L >= P.N) return;
  const unsigned Lu = (unsigned)L, q = Lu / (unsigned)P.nz;
  const int z = (int)(Lu - q * (unsigned)P.nz), x = (int)(q / (unsigned)P.ny), y = (int)(q - (unsigned)x * P.ny);
  R v = R(0);
  Ref nref = ref_rest(P);
  if (!(SOLID && walls_all[L] >= 1)) {
    const unsigned N = (unsigned)P.N;
    if constexpr (Codec<S>::kRef) {
      const Ref ref = rr_old[pd.idx(x, y, z)];
      // the deviations summed by weight, both of a velocity in one packed addition,
      // and decoded once, as the collide kernel does (decoding every velocity was
      // bound by instruction issue: 527 instructions a node)
      const __half2* const in = reinterpret_cast<const __half2*>(pops) + Lu;
      const F2 rest(__half22float2(in[0]));
      F2 axis(__half22float2(in[N])), diag(__half22float2(in[7 * N]));
#pragma unroll
      for (unsigned i = 2; i < 7; i++) axis = axis + F2(__half22float2(in[i * N]));
#pragma unroll
      for (unsigned i = 8; i < 19; i++) diag = diag + F2(__half22float2(in[i * N]));
      const F2 dev = vfma(F2(float(W(0) / 4096.0)), rest,
                          vfma(F2(float(W(1) / 4096.0)), axis, F2(float(W(7) / 4096.0)) * diag));
      // sr is exactly rho or 0 in a pure phase
      const float rho = ref.x + dev[0], sr = fmaf(ref.y, rho, dev[1]), sb = rho - sr;
      v = qdiv<R>(sr - sb, rho);
      nref = make_float2(rho, sr / rho);
    } else {
      R sr = R(0), sf = R(0);
      unroll19([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        R f, r;
        Codec<S>::template load_fr<i>(pops, N, Lu, Ref{}, f, r);
        sr = sr + r;
        sf = sf + f;
      });
      v = qdiv<R>(sr - (sf - sr), sf);
    }
  }
  phi_store<R>(P, pd, phi, x, y, z, v);
  if constexpr (Codec<S>::kRef) phi_store<Ref>(P, pd, rr_new, x, y, z, nref);
}

template <typename S, bool SOLID>
__global__ void __launch_bounds__(256) k_phase(DevParams P, Pad pd, const S* __restrict__ pops,
                                               typename Codec<S>::R* __restrict__ phi,
                                               const int32_t* __restrict__ walls_all, const Ref* __restrict__ rr_old,
                                               Ref* __restrict__ rr_new) {
  phase_node<S, SOLID>(P, pd, pops, phi, walls_all, rr_old, rr_new, blockIdx.x * 256LL + threadIdx.x);
}

// From the accumulated colour densities (FP64, the steady-state phase field):
// phi = (rhoR - rhoB) / rho on fluid nodes, 0 on solid nodes, written with its
// periodic ghost images; the accumulators are cleared for the collide kernel
// of this step.
// Nodes L0, L0 + 256, ..., L0 + 256 (NPT-1) per thread: every load of all of
// them is issued before the first store, so a thread keeps 2 NPT accumulator
// reads in flight (nothing waits on a store).
template <bool SOLID, int NPT>
__device__ __forceinline__ void finalize_nodes(const DevParams& P, const Pad& pd, Acc::T* __restrict__ acc,
                                               double* __restrict__ phi, const int32_t* __restrict__ walls_all,
                                               const int* __restrict__ status, long long L0) {
  const int bad = *status;
  Acc::T ar[NPT], ab[NPT];
  bool solid[NPT];
#pragma unroll
  for (int k = 0; k < NPT; k++) {
    const long long L = L0 + 256LL * k;
    ar[k] = ab[k] = 0;
    solid[k] = false;
    if (L < P.N) {
      ar[k] = acc[L];
      ab[k] = acc[L + P.N];
      solid[k] = SOLID && walls_all[L] >= 1;
    }
  }
#pragma unroll
  for (int k = 0; k < NPT; k++) {
    const long long L = L0 + 256LL * k;
    if (L >= P.N) break;
    acc[L] = 0;
    acc[L + P.N] = 0;
    // 32-bit index arithmetic (the fused path keeps 38*N < 2^32)
    const unsigned Lu = (unsigned)L, q = Lu / (unsigned)P.nz;
    const int z = (int)(Lu - q * (unsigned)P.nz), x = (int)(q / (unsigned)P.ny), y = (int)(q - (unsigned)x * P.ny);
    const double sr = Acc::val(ar[k]), sb = Acc::val(ab[k]);
    double v = solid[k] ? 0.0 : (sr - sb) / (sr + sb);
    if (bad) v = NAN;
    phi_store<double>(P, pd, phi, x, y, z, v);
  }
}

// nodes finalised per thread by the single-domain kernel
constexpr int kFinalizeNPT = 4;

template <bool SOLID>
__global__ void __launch_bounds__(256) k_finalize(DevParams P, Pad pd, Acc::T* acc, double* __restrict__ phi,
                                                  const int32_t* __restrict__ walls_all,
                                                  const int* __restrict__ status) {
  finalize_nodes<SOLID, kFinalizeNPT>(P, pd, acc, phi, walls_all, status,
                                      blockIdx.x * (256LL * kFinalizeNPT) + threadIdx.x);
}

// ---- wetting rotation of a node normal (derivatives :535-587) ---------------------
template <typename R, typename PT>
__device__ __forceinline__ void wet_rotate(const PT& P, const sym_particles* S, int pp, int x, int y, int z,
                                           R& n0, R& n1, R& n2) {
  double nwd[3];
  wall_normal_dev(P, S, pp, x, y, z, nwd);
  const R nw[3] = {R(nwd[0]), R(nwd[1]), R(nwd[2])};
  const R n[3] = {n0, n1, n2};
  R v[3];
  akai_rotate_sc<R>(R(P.sin_cita), R(P.cos_cita), nw, n, true, v);
  n0 = v[0]; n1 = v[1]; n2 = v[2];
}

// ---- k_collide ------------------------------------------------------------------
// phi ring of 5 planes, normal ring of 4 planes, reference-pair ring of 6 planes:
// normals are computed one plane ahead and phi / reference-pair loaded three planes
// ahead, before the plane's single barrier.  A warp that has finished plane x
// runs those writes for plane x+1 while slower warps still read plane x's
// slots: phi at x, normals at x-1..x+1 and reference-pair at x-1..x+1 (the push
// targets).  The rings are sized so that the slots written for plane x+1
// (phi x+4 -> slot (x-1)%5, normals x+2 -> (x-2)%4, reference-pair x+4 -> (x-2)%6)
// are never among them.
constexpr int kIrrRing = 6;
// The unit normals and |grad phi| of four planes of a tile, [plane][y][z], split
// so that a warp's accesses are contiguous (16-byte x, y pairs and 8-byte z: 6
// shared-memory wavefronts for a warp's normals, against 16 of a 32-byte
// record); only a node's own |grad phi| is read.
template <int ROWS>
struct NormalTile {
  double2 xy[4][ROWS][BZ + 2];
  double z_[4][ROWS][BZ + 2];
  double g[4][ROWS][BZ + 2];
  __device__ __forceinline__ void set(int s, int y, int z, double nx, double ny, double nz, double gr) {
    xy[s][y][z] = make_double2(nx, ny);
    z_[s][y][z] = nz;
    g[s][y][z] = gr;
  }
  __device__ __forceinline__ void get(int s, int y, int z, double (&n)[3]) const {
    const double2 t = xy[s][y][z];
    n[0] = t.x; n[1] = t.y; n[2] = z_[s][y][z];
  }
  __device__ __forceinline__ double grad(int s, int y, int z) const { return g[s][y][z]; }
};
// Tile height (rows of BZ nodes) of the collide kernels per storage, on 256
// threads: 8 rows for FP64 (16 would fit one CTA per SM and was slower,
// 256x256x512: 4.70 against 4.52 ms), 16 for FP32 arithmetic (two nodes a thread,
// paired.cuh).
template <typename S>
constexpr int kBY = sizeof(S) == 8 ? 8 : 16;
constexpr int kTPB = 256;
// the same for a storage mode chosen at run time (SYM_STORE_*)
inline int tile_rows(int storage) {
  return storage == SYM_STORE_FP16 ? kBY<__half> : (storage == SYM_STORE_FP32 ? kBY<float> : kBY<double>);
}
// most x planes of a tile
constexpr int kMaxExtent = 64;
// phi plane tiles ((BY+4) x (BZ+4), z fastest) arrive by TMA: each slot starts on
// a 128-byte boundary
struct Smem {
  static constexpr int BY = kBY<double>;
  static constexpr int kTile = (BY + 4) * (BZ + 4);
  static constexpr int kPhiSlot = (kTile * 8 + 127) / 128 * 128 / 8;
  alignas(128) double phi[5][kPhiSlot];
  alignas(16) NormalTile<BY + 2> n;
  double xch[3][2][2][BY][BZ];   // [cx+1][to row y+1, y-1][colour]: density sums crossing rows
  // [beside lane 0, beside the last lane][cx+1][cy = 0, +1, -1][colour][row]:
  // pushes crossing the tile's z edges (cy = +-1 for cx = 0 only)
  double zx[2][3][3][2][BY];
  uint64_t bar[kIrrRing];   // one mbarrier per plane load, used round robin
  unsigned char near_solid[kMaxExtent + 2];   // planes xa-1 .. xb
};
// Whether plane xp of the tile at (z0, y0) may hold a solid or a node next to
// one: where the masks had any when the fused state was built, and around the
// particles where they are now (a solid reaches rad from its centre, the nodes
// next to it one more).  Planes without take no masks: two dependent reads a
// node and plane made the solid variant 1.2 to 2 times slower than the plain one.
template <typename R>
__device__ __forceinline__ bool solid_near(const TileParams<R>& P, const sym_particles* __restrict__ S, int rows, int xp,
                                           int y0, int z0) {
  if (P.solid_tiles[((size_t)wrapi(xp, P.nx) * P.tiles_y + y0 / rows) * P.tiles_z + z0 / BZ]) return true;
  const double reach = P.rad + 2.0;
  const double yc = y0 + 0.5 * (rows - 1), yh = 0.5 * (rows - 1) + 1.0;
  const double zc = z0 + 0.5 * (BZ - 1), zh = 0.5 * (BZ - 1) + 1.0;
  for (int k = 0; k < P.par; k++)
    if (fabs(disp(P, (double)xp, S->center[k], 0)) <= reach &&
        fabs(disp(P, yc, S->center[P.par + k], 1)) <= reach + yh &&
        fabs(disp(P, zc, S->center[2 * P.par + k], 2)) <= reach + zh)
      return true;
  return false;
}
// node t of the one-node ring around a tile of `rows` rows, in normal-ring
// coordinates (the tile's own nodes are y 1 .. rows, z 1 .. BZ): rows 0 and
// rows + 1, then the two z columns
__device__ __forceinline__ void ring_node(int t, int rows, int& y, int& z) {
  if (t < 2 * (BZ + 2)) {
    y = t < BZ + 2 ? 0 : rows + 1;
    z = t < BZ + 2 ? t : t - (BZ + 2);
  } else {
    t -= 2 * (BZ + 2);
    y = 1 + t % rows;
    z = t < rows ? 0 : BZ + 1;
  }
}
// One FP64 tile: the 32(z) x 8(y) footprint at (z0, y0), planes xa..xb-1.  Called
// by the single-domain kernel (tile from blockIdx) and by the batched
// persistent kernel (tile from the work-tile table).  solid_rt: solid handling
// wanted by this domain (the batched kernel compiles one variant and decides
// per tile).
//
// Besides the pushed populations the tile adds up the next step's colour
// densities.  Per plane the pushes are summed over z by warp shuffles and over
// y through shared memory; what leaves the tile along z is handed over as ten
// numbers per row in shared memory, and what leaves along y is a row of the
// exchange.  The sum a plane sends to each destination node is turned into
// fixed point and added to the sums of the planes before and after it in
// registers -- the tile's own nodes by their threads, the one-node ring around
// it by 168 threads beside that work -- so each node gets one addition per
// tile and plane.  The totals are integer sums of terms that do not depend on
// where the march starts or ends: a domain's result is the same bit for bit
// whatever x extent its tiles have.
template <bool SOLID>
__device__ __forceinline__ void collide_tile(const TileParams<double>& P, const double* __restrict__ pin_,
                                             double* __restrict__ pout_, const int32_t* __restrict__ walls,
                                             const int32_t* __restrict__ walls_all,
                                             const int32_t* __restrict__ pout,
                                             const sym_particles* __restrict__ Sp, double* __restrict__ ffi,
                                             Acc::T* acc, int* status, const CUtensorMap* tm_phi,
                                             int z0, int y0, int xa, int xb, Smem& sm, unsigned& nload,
                                             bool solid_rt = true) {
  using R = double;
  using A = Acc;
  using AT = A::T;
  constexpr int BY = kBY<double>, kRow = BZ + 4;
  const bool SOLIDX = SOLID && solid_rt;
  const int tz = threadIdx.x % BZ, ty = threadIdx.x / BZ;
  const int sy = P.nz, sx = P.nz * P.ny;   // element strides of y and x
  const int Ni = sx * P.nx;                // 19 N < 2^31 on the fused path
  const NodeParams<R>& np = P.np;
  const R evap = np.evap;

  // phi of plane xp by TMA: one box of (BY+4) x (BZ+4) at the padded origin
  // (z0, y0, xp+2) -- z0 is a multiple of 32 elements, so the innermost
  // coordinate is 128-byte aligned; rows past the padded extent read as zeros.
  // Plane xp is load number nl0 + xp - (xa - 2) of this CTA, on mbarrier
  // (number mod 6) with phase parity (number / 6) mod 2.
  const unsigned nl0 = nload;
  auto load_no = [&](int xp) { return nl0 + (unsigned)(xp - (xa - 2)); };
  auto load_phi = [&](int xp) {   // thread 0 only
    uint64_t* bar = &sm.bar[load_no(xp) % kIrrRing];
    tma::mbar_expect_tx(bar, Smem::kTile * sizeof(R));
    tma::load_3d(sm.phi[(unsigned)(xp + 5) % 5u], tm_phi, z0, y0, xp + 2, bar);
  };
  auto wait_phi = [&](int xp) {   // every thread
    const unsigned q = load_no(xp);
    if (!tma::mbar_wait(&sm.bar[q % kIrrRing], (q / kIrrRing) & 1u)) atomicOr(status, 2);
  };
  int ring_y, ring_z;
  ring_node(threadIdx.x, BY, ring_y, ring_z);
  constexpr int kRing = 2 * (BZ + 2) + 2 * BY;
  // unit normals (rotated at wetting nodes) and |grad phi| of plane xp, halo 1
  auto compute_n_as = [&](auto solidc, int xp) __attribute__((always_inline)) {
    constexpr bool solid = decltype(solidc)::value;
    const int s = xp & 3;   // xp >= -1: the slot in the 4-plane normal ring
    // phi planes xp-1, xp, xp+1 in the 5-plane ring (xp >= -1)
    const R* const pm = sm.phi[(unsigned)(xp + 4) % 5u];
    const R* const p0 = sm.phi[(unsigned)(xp + 5) % 5u];
    const R* const pp1 = sm.phi[(unsigned)(xp + 6) % 5u];
    auto one = [&](int py, int pz) __attribute__((always_inline)) {
      R n0 = 0, n1 = 0, n2 = 0, fn = 0;
      bool ok = true;
      int id = 0, y = 0, z = 0;
      if (solid) {   // nodes beyond the halo, read by nobody, take the last one's masks
        y = wrapi(min(y0 - 1 + py, P.ny), P.ny);
        z = wrapi(min(z0 - 1 + pz, P.nz), P.nz);
        const unsigned Lw = (unsigned)(z + sy * y + sx * wrapi(xp, P.nx));
        const int wall = walls_all[Lw];
        id = pout[Lw];
        ok = wall <= 0;
      }
      if (ok) {
        // grad phi = 3 sum_i w_i c_i phi(x + c_i) (:510-521) from the
        // differences over opposite neighbours: an axis pair weighs twice a
        // diagonal one
        const int b = (py + 1) * kRow + pz + 1;
        const R xyp = pp1[b + kRow] - pm[b - kRow], xym = pp1[b - kRow] - pm[b + kRow];
        const R xzp = pp1[b + 1] - pm[b - 1], xzm = pp1[b - 1] - pm[b + 1];
        const R yzp = p0[b + kRow + 1] - p0[b - kRow - 1], yzm = p0[b + kRow - 1] - p0[b - kRow + 1];
        const R g0 = (1.0 / 12.0) * fma(2.0, pp1[b] - pm[b], (xyp + xym) + (xzp + xzm));
        const R g1 = (1.0 / 12.0) * fma(2.0, p0[b + kRow] - p0[b - kRow], (xyp - xym) + (yzp + yzm));
        const R g2 = (1.0 / 12.0) * fma(2.0, p0[b + 1] - p0[b - 1], (xzp - xzm) + (yzp - yzm));
        const R g2s = g0 * g0 + g1 * g1 + g2 * g2;
        // |grad phi| and its reciprocal from one rsqrt
        if (g2s > evap * evap) {
          const R rf = rsqrt(g2s);
          fn = g2s * rf;
          n0 = g0 * rf; n1 = g1 * rf; n2 = g2 * rf;
          if (solid && id >= 1) {
            // the rotation has to know a gradient along the wall's normal, whose
            // unit vector is exactly 1 there (the reference's quotient) and with
            // rsqrt may be an ulp to either side
            const R m = fmax(fabs(g0), fmax(fabs(g1), fabs(g2)));
            if (m * m == g2s) {
              fn = m;
              if (fabs(g0) == m) n0 = copysign(R(1), g0);
              if (fabs(g1) == m) n1 = copysign(R(1), g1);
              if (fabs(g2) == m) n2 = copysign(R(1), g2);
            }
            wet_rotate<R>(P, Sp, id, wrapi(xp, P.nx), y, z, n0, n1, n2);
          }
        }
      }
      sm.n.set(s, py, pz, n0, n1, n2, fn);
    };
    one(ty + 1, tz + 1);   // the thread's own node, then the ring around the tile
    if (threadIdx.x < kRing) one(ring_y, ring_z);
  };
  // every plane is compiled twice, with and without solids; a plane's flag is
  // the whole CTA's, and the code of the planes without stays that of a domain
  // without
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
  if (SOLIDX) {
    for (int t = threadIdx.x; t < xb - xa + 2; t += kTPB)
      sm.near_solid[t] = solid_near(P, Sp, BY, xa - 1 + t, y0, z0);
    __syncthreads();
  }

  if (threadIdx.x == 0)
    for (int xp = xa - 2; xp <= xa + 2; xp++) load_phi(xp);
  wait_phi(xa - 2);
  wait_phi(xa - 1);
  nload = nl0 + (unsigned)(xb - xa + 4);   // loads of this tile: planes xa-2 .. xb+1

  // last row and lane of the tile inside the domain; rows past the last one
  // have no work, lanes past the last one run the node arithmetic on a clamped
  // node for the shuffles' sake (nothing of theirs is stored or added)
  const int ylast = min(BY - 1, P.ny - 1 - y0), zlast = min(BZ - 1, P.nz - 1 - z0);
  const int y = y0 + ty, z = z0 + min(tz, zlast);
  const bool inr = ty <= ylast && tz <= zlast;
  const bool ezp = tz == zlast, ezm = tz == 0;
  const int oyp = (y == P.ny - 1) ? -(P.ny - 1) * sy : sy, oym = (y == 0) ? (P.ny - 1) * sy : -sy;
  const int ozp = (z == P.nz - 1) ? -(P.nz - 1) : 1, ozm = (z == 0) ? (P.nz - 1) : -1;
  // ring nodes: threads 0..127 the rows before and after the tile (two
  // colours, 32 lanes), threads 128..167 the columns beside it, their rows -1
  // to ylast + 1 (the corners included)
  constexpr int kRowItems = 4 * BZ, kColItems = 4 * (BY + 2);
  const bool row_item = threadIdx.x < kRowItems;
  const int u = (int)threadIdx.x - kRowItems;
  const int o_side = row_item ? (int)threadIdx.x / (2 * BZ) : u / (2 * (BY + 2));
  const int o_col = row_item ? ((int)threadIdx.x / BZ) & 1 : (u / (BY + 2)) & 1;
  const int o_row = row_item ? (o_side ? ylast + 1 : -1) : u % (BY + 2) - 1;
  const bool o_valid =
      row_item ? tz <= zlast : ((int)threadIdx.x < kRowItems + kColItems && o_row <= ylast + 1);
  const int o_z = row_item ? z0 + min(tz, zlast) : wrapi(o_side ? z0 + zlast + 1 : z0 - 1, P.nz);
  AT* const o_acc = acc + (o_col ? Ni : 0) + (o_z + sy * wrapi(y0 + o_row, P.ny));
  AT* const n_acc = acc + (z + sy * min(y, P.ny - 1));
  AT aPr = 0, aPb = 0, aCr = 0, aCb = 0, oP = 0, oC = 0;   // planes x-1 and x
  bool fine = true;   // every density finite and in the fixed-point range
  // the node arithmetic, pushes and density sums of plane x
  auto plane = [&](auto solidc, int x) __attribute__((always_inline)) {
    constexpr bool solid = decltype(solidc)::value;
    wait_phi(x + 2);
    compute_n(x + 1);
    __syncthreads();
    const int oxp = (x == P.nx - 1) ? -(P.nx - 1) * sx : sx, oxm = (x == 0) ? (P.nx - 1) * sx : -sx;
    R cen[3][2];   // sums this row sends to its own row in planes x-1, x, x+1
    if (ty <= ylast) {
      const int L = z + sy * y + sx * x;
      int pp = 0;
      bool act = inr;
      if (solid) {
        const int wall = walls_all[L], id = pout[L];
        if (wall > 0) act = false;
        else pp = id;
      }
      // calmacros on the own populations
      R f[19];
      const double2* const in = reinterpret_cast<const double2*>(pin_) + L;
      auto ld = [&](auto ic) __attribute__((always_inline)) -> R {   // f[i]; returns the red population
        constexpr int i = decltype(ic)::value;
        const double2 v = in[i * Ni];
        f[i] = v.x + v.y;
        return v.x;
      };
#define SYM_LD(i) ld(std::integral_constant<int, i>{})
      // red density, added in the order to_moments adds the totals: a pure red
      // node (r = f) gets sr = rho exactly
      const R rest = SYM_LD(0);
      const R rx = SYM_LD(1) + SYM_LD(2), ry = SYM_LD(3) + SYM_LD(4), rz = SYM_LD(5) + SYM_LD(6);
      const R rxp = SYM_LD(7) + SYM_LD(10), rxm = SYM_LD(8) + SYM_LD(9);
      const R rzp = SYM_LD(11) + SYM_LD(14), rzm = SYM_LD(12) + SYM_LD(13);
      const R ryp = SYM_LD(15) + SYM_LD(18), rym = SYM_LD(16) + SYM_LD(17);
#undef SYM_LD
      const R sr = rest + (rx + ry + rz) + ((rxp + rxm) + (rzp + rzm) + (ryp + rym));
      Moments<R> m;
      to_moments<R, R>(f, m);
      const R rho = m.rho, sb = rho - sr;
      R nown[3];
      sm.n.get(x & 3, ty + 1, tz + 1, nown);
      const R nx = nown[0], ny = nown[1], nz = nown[2], fn = sm.n.grad(x & 3, ty + 1, tz + 1);
      R irho, su, sq;
      node_rates_fused<R>(P, sm.phi[(unsigned)(x + 5) % 5u][(ty + 2) * kRow + tz + 2], rho, irho, su, sq);
      // CSF surface tension from the curvature of the normal field (:624-667);
      // a node without a normal has n = 0 and |grad phi| = 0
      R val = 0;
      if (!solid || pp <= 0) {
        const R kurv = curvature<R, R>(
            [&](auto ic, R (&d)[3]) {
              constexpr int i = decltype(ic)::value;
              R p[3], q[3];
              sm.n.get((x + CX(i)) & 3, ty + 1 + CY(i), tz + 1 + CZ(i), p);
              sm.n.get((x - CX(i)) & 3, ty + 1 - CY(i), tz + 1 - CZ(i), q);
              d[0] = p[0] - q[0]; d[1] = p[1] - q[1]; d[2] = p[2] - q[2];
            },
            nx, ny, nz);
        val = np.half_sigma * kurv * fn;
      }
      const R fx = fma(val, nx, rho * np.body[0]), fy = fma(val, ny, rho * np.body[1]),
              fz = fma(val, nz, rho * np.body[2]);
      relax<R, R>(m, rho, (m.jx + 0.5 * fx) * irho, (m.jy + 0.5 * fy) * irho, (m.jz + 0.5 * fz) * irho, fx, fy, fz, su,
                  np.s_e > 0 ? np.s_e : su, np.s_eps > 0 ? np.s_eps : su, np.s_q > 0 ? np.s_q : sq,
                  np.s_pi > 0 ? np.s_pi : su, np.s_m > 0 ? np.s_m : sq);
      from_moments<R, R>(m, f);
      // Latva-Kokko recolouring (:712-726): r_i = (rhoR/rho) f_i + beta rhoR rhoB /
      // rho w_i (n.c_i); a colour at or below EVAP_LIM empties (r_i = 0 when
      // rhoR is, r_i = f_i when rhoB is, the latter taking precedence), which the
      // two coefficients express once per node
      const bool rzero = sr <= evap, bzero = sb <= evap;
      R ratio = bzero ? 1.0 : (rzero ? 0.0 : sr * irho);
      // beta rhoR rhoB / rho times a diagonal link's weight, along each axis
      R cd = (bzero || rzero) ? 0.0 : sr * sb * irho * np.beta * (1.0 / 36.0);
      // links that come back (bit i: the push along c_i enters a solid, curve
      // :1001-1019), from a wall without velocity (flat) or from particle pp
      unsigned back = 0, flat = 0;
      R uw0 = 0, uw1 = 0, uw2 = 0;
      if (solid) {
        if (!act) {   // a solid node (or a lane outside the domain) sends nothing
          ratio = 0;
          cd = 0;
#pragma unroll
          for (int i = 0; i < 19; i++) f[i] = 0;
        }
        if (pp >= 1) {
          const int par = P.par;
          static_for<18>([&](auto kc) {   // the neighbours' masks are read together, not one per push
            constexpr int i = decltype(kc)::value + 1;
            const int wb = walls[L + (CX(i) > 0 ? oxp : (CX(i) < 0 ? oxm : 0)) +
                                 (CY(i) > 0 ? oyp : (CY(i) < 0 ? oym : 0)) + (CZ(i) > 0 ? ozp : (CZ(i) < 0 ? ozm : 0))];
            if (wb > par) flat |= 1u << i;
            else if (wb == pp) back |= 1u << i;
          });
          back |= flat;
          if (pp <= par && act) {
            // rigid-body velocity of particle pp at this node (curve :1009-1014)
            const R xr = disp(P, (double)(x + P.origin), Sp->center[0 * par + pp - 1], 0);
            const R yr = disp(P, (double)(y + P.origin), Sp->center[1 * par + pp - 1], 1);
            const R zr = disp(P, (double)(z + P.origin), Sp->center[2 * par + pp - 1], 2);
            uw0 = Sp->up[0 * par + pp - 1] + zr * Sp->rp[1 * par + pp - 1] - yr * Sp->rp[2 * par + pp - 1];
            uw1 = Sp->up[1 * par + pp - 1] + xr * Sp->rp[2 * par + pp - 1] - zr * Sp->rp[0 * par + pp - 1];
            uw2 = Sp->up[2 * par + pp - 1] + yr * Sp->rp[0 * par + pp - 1] - xr * Sp->rp[1 * par + pp - 1];
            // post-collision populations for the momentum exchange (:1241-1243),
            // read only next to particles
#pragma unroll
            for (int i = 0; i < 19; i++) ffi[(size_t)i * Ni + L] = f[i];
          }
        }
      }
      const R cnx = cd * nx, cny = cd * ny, cnz = cd * nz;
      double2* const out = reinterpret_cast<double2*>(pout_) + L;
      R sfr = 0, sfb = 0;   // links bounced back into this node
      // push along c_i: red r and blue b, as stored (0 if the link came back)
      auto push = [&](auto ic, R& r, R& b) __attribute__((always_inline)) {
        constexpr int i = decltype(ic)::value;
        if constexpr (i == 0) {
          r = ratio * f[i];
        } else if constexpr (i < 7) {
          constexpr double c = 2 * (CX(i) + CY(i) + CZ(i));   // twice the diagonal weight
          r = fma(ratio, f[i], c * (CX(i) ? cnx : (CY(i) ? cny : cnz)));
        } else {
          constexpr int s1 = CX(i) ? CX(i) : CY(i), s2 = CZ(i) ? CZ(i) : CY(i);   // the two axes of the link
          const R c1 = CX(i) ? cnx : cny, c2 = CZ(i) ? cnz : cny;
          r = fma(ratio, f[i], s1 > 0 ? (s2 > 0 ? c1 + c2 : c1 - c2) : (s2 > 0 ? c2 - c1 : -(c1 + c2)));
        }
        b = f[i] - r;
        int o = i * Ni + (CX(i) > 0 ? oxp : (CX(i) < 0 ? oxm : 0)) + (CY(i) > 0 ? oyp : (CY(i) < 0 ? oym : 0)) +
                (CZ(i) > 0 ? ozp : (CZ(i) < 0 ? ozm : 0));
        if (solid) {
          // interpolated bounce-back: the red post-collision populations of the
          // nodes next to particles, for the link update after this kernel
          if (P.bounce && pp >= 1 && pp <= P.par && act) ffi[(size_t)(19 + i) * Ni + L] = r;
          if (i > 0 && (back >> i & 1u)) {
            constexpr int j = OPC(i);
            const R star = (flat >> i & 1u) ? 0.0 : 6.0 * W(j) * (uw0 * CX(j) + uw1 * CY(j) + uw2 * CZ(j));
            const R rr = fma(sr, star, r), bb = fma(sb, star, b);
            if (act) out[j * Ni] = make_double2(rr, bb);
            sfr = sfr + rr;
            sfb = sfb + bb;
            r = b = 0;
            return;
          }
        }
        if (act) out[o] = make_double2(r, b);
      };
      // the pushes along equal (cx, cy): lane l receives the cz = +1 push of
      // lane l-1 and the cz = -1 push of lane l+1; the edge lanes' outgoing ones
      // go to the columns' exchange
      auto group = [&](auto ac, auto bc, auto i0, auto ip, auto im, R& r, R& b) __attribute__((always_inline)) {
        constexpr int a = decltype(ac)::value, g = decltype(bc)::value;
        R up[2], dn[2];
        push(i0, r, b);
        push(ip, up[0], up[1]);
        push(im, dn[0], dn[1]);
        if (ezp) { sm.zx[1][a][g][0][ty] = up[0]; sm.zx[1][a][g][1][ty] = up[1]; }
        if (ezm) { sm.zx[0][a][g][0][ty] = dn[0]; sm.zx[0][a][g][1][ty] = dn[1]; }
#pragma unroll
        for (int c = 0; c < 2; c++) {
          up[c] = __shfl_up_sync(0xffffffffu, up[c], 1);
          dn[c] = __shfl_down_sync(0xffffffffu, dn[c], 1);
        }
        if (!ezm) { r = r + up[0]; b = b + up[1]; }
        if (!ezp) { r = r + dn[0]; b = b + dn[1]; }
      };
#define SYM_I(v) std::integral_constant<int, v>{}
      R r, b;
      auto row = [&](int a, int dir) __attribute__((always_inline)) {   // to row y+1 (0) or y-1 (1) of plane x + a - 1
        sm.xch[a][dir][0][ty][tz] = r;
        sm.xch[a][dir][1][ty][tz] = b;
      };
      group(SYM_I(1), SYM_I(1), SYM_I(3), SYM_I(15), SYM_I(17), r, b); row(1, 0);
      group(SYM_I(1), SYM_I(2), SYM_I(4), SYM_I(16), SYM_I(18), r, b); row(1, 1);
      push(SYM_I(7), r, b); row(2, 0);
      push(SYM_I(9), r, b); row(2, 1);
      push(SYM_I(8), r, b); row(0, 0);
      push(SYM_I(10), r, b); row(0, 1);
      group(SYM_I(2), SYM_I(0), SYM_I(1), SYM_I(11), SYM_I(13), cen[2][0], cen[2][1]);
      group(SYM_I(0), SYM_I(0), SYM_I(2), SYM_I(12), SYM_I(14), cen[0][0], cen[0][1]);
      group(SYM_I(1), SYM_I(0), SYM_I(0), SYM_I(5), SYM_I(6), cen[1][0], cen[1][1]);
#undef SYM_I
      if (solid) {
        cen[1][0] = cen[1][0] + sfr;
        cen[1][1] = cen[1][1] + sfb;
      }
    }
    __syncthreads();
    const int om = x > xa ? -sx : oxm;
    auto fix = [&](R v) __attribute__((always_inline)) -> AT {
      fine = fine && A::ok(v);
      return A::fix(v);
    };
    if (inr) {
      AT in[3][2];
#pragma unroll
      for (int a = 0; a < 3; a++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
          R v = cen[a][c];
          if (ty > 0) v = v + sm.xch[a][0][c][ty - 1][tz];
          if (ty < ylast) v = v + sm.xch[a][1][c][ty + 1][tz];
          in[a][c] = fix(v);
        }
      // plane x-1 of this column has all its in-tile contributions (plane xa-1
      // only this plane's)
      AT* const at = n_acc + sx * x;
      atomicAdd(at + om, aPr + in[0][0]);
      atomicAdd(at + om + Ni, aPb + in[0][1]);
      aPr = aCr + in[1][0]; aPb = aCb + in[1][1];
      aCr = in[2][0]; aCb = in[2][1];
      if (x == xb - 1) {   // the end of the march: this plane's node and the one after it
        atomicAdd(at, aPr);
        atomicAdd(at + Ni, aPb);
        atomicAdd(at + oxp, aCr);
        atomicAdd(at + oxp + Ni, aCb);
      }
    }
    if (o_valid) {
      AT in[3];
#pragma unroll
      for (int a = 0; a < 3; a++) {
        R v;
        if (row_item) {
          v = sm.xch[a][o_side ? 0 : 1][o_col][o_side ? ylast : 0][tz];
        } else {
          // rows o_row (same row), o_row - 1 (its cy = +1) and o_row + 1 (cy = -1);
          // only the planes' own x has diagonal links that leave along y and z
          v = 0;
          if (o_row >= 0 && o_row <= ylast) v = sm.zx[o_side][a][0][o_col][o_row];
          if (a == 1) {
            if (o_row >= 1) v = v + sm.zx[o_side][1][1][o_col][o_row - 1];
            if (o_row < ylast) v = v + sm.zx[o_side][1][2][o_col][o_row + 1];
          }
        }
        in[a] = fix(v);
      }
      AT* const at = o_acc + sx * x;
      atomicAdd(at + om, oP + in[0]);
      oP = oC + in[1];
      oC = in[2];
      if (x == xb - 1) {
        atomicAdd(at, oP);
        atomicAdd(at + oxp, oC);
      }
    }
  };
#pragma unroll 1
  for (int x = xa - 2; x < xa; x++) {
    wait_phi(x + 2);
    compute_n(x + 1);
  }
  // the first phi load below reuses the slot of plane xa-2, read by the first turn
  __syncthreads();
#pragma unroll 1
  for (int x = xa; x < xb; x++) {
    // phi of plane x+3 on its way; normals of plane x+1 from phi planes x..x+2.
    // The slots the load overwrites (phi of plane x-2) were last read before the
    // previous plane's barriers.
    if (threadIdx.x == 0 && x + 3 <= xb + 1) load_phi(x + 3);
    if constexpr (SOLID) {
      if (near_solid(x)) {
        plane(std::true_type{}, x);
        continue;
      }
    }
    plane(std::false_type{}, x);
  }
  if (!fine) atomicOr(status, 1);
}

// Plane times a tile is charged for what comes before its first plane (five
// plane loads and the normals of two planes).  A CTA by itself spends two of
// any storage, of which others on the SM hide about half.
constexpr double kTileLead = 1.0;
// x extent of a tile whose column of x planes is nx long, at most `cap`: the
// column in equal parts
inline int split_extent(int nx, int cap) {
  cap = std::min(cap, kMaxExtent);
  const int parts = (nx + cap - 1) / cap;
  return (nx + parts - 1) / parts;
}
// The tile x extent, at most `cap`, for columns[i] columns (32 x BY
// footprints) of nx[i] planes each on `slots` resident CTAs: the one with the
// least estimated time, in planes: the work of all slots evenly shared plus
// half a tile of tail, or one whole tile when there are fewer tiles than
// slots.  A CTA needs about 6.6 us for an FP64 plane of 8 rows (6.0 FP32, 5.3
// 16-bit, 16 rows) whether the GPU is full or not, so a domain of few columns is
// bound by the length of one march.  Measured per step, extent 32 against this
// rule's: 32x32x96 FP64 243 -> 28.5 us (2 planes), FP32 205 -> 20.5 (1), 16-bit
// 184 -> 20.5 (1); 64x64x128 FP64 281 -> 102 (4), FP32 222 -> 59 (3), 16-bit
// 198 -> 51 (3); 53x53x374 FP64 263 -> 194 (6); 256x256x512 FP64 keeps 32.
inline int best_extent(const std::vector<long long>& columns, const std::vector<int>& nx, int cap, long long slots) {
  int best = 1;
  double least = 1e300;
  cap = std::min(cap, kMaxExtent);   // a caller's "no limit" may be any number
  for (int x = 1; x <= cap; x++) {
    double sum = 0.0, longest = 0.0;
    for (size_t i = 0; i < nx.size(); i++) {
      const int e = split_extent(nx[i], x);
      const int tiles = (nx[i] + e - 1) / e;
      sum += (double)columns[i] * (nx[i] + tiles * kTileLead);
      longest = std::max(longest, e + kTileLead);
    }
    const double t = std::max(longest, sum / (double)slots + 0.5 * longest);
    if (t <= least) { least = t; best = x; }
  }
  return best;
}

// ---- the fused state's side of the particle and wall work ---------------------------
// (device bodies; the batched launches are in sparse.cu)

// pin fill (derivatives :467-492): fictitious phi of solid node (x,y,z) next
// to fluid = wi-weighted mean of its fluid neighbours
template <typename R>
__device__ __forceinline__ void pinfill_node(const DevParams& P, const Pad& pd, R* phi,
                                             const int32_t* __restrict__ pin, const int32_t* __restrict__ walls_all,
                                             int x, int y, int z) {
  const long long L = lin(P, x, y, z);
  if (pin[L] <= 0) return;
  // masks and values of all neighbours are read together (one after another
  // behind its mask, each a round trip to memory)
  int wall[19];
  R ph[19];
#pragma unroll
  for (int i = 1; i < 19; i++) {
    wall[i] = walls_all[lin(P, wrapi(x + CX(i), P.nx), wrapi(y + CY(i), P.ny), wrapi(z + CZ(i), P.nz))];
    ph[i] = phi[pd.idx(x + CX(i), y + CY(i), z + CZ(i))];
  }
  R ws = R(0), v = R(0);
#pragma unroll
  for (int i = 1; i < 19; i++)
    if (wall[i] <= 0) { ws = ws + R(W(i)); v = v + R(W(i)) * ph[i]; }
  phi_store<R>(P, pd, phi, x, y, z, v / ws);
}

// particle preparation: canonical views of the fused state at a node of a
// particle box -- rho_N (this step's calmacros), rho_R/rho_B and, at nodes
// next to a particle, fi (current populations), and the previous step's
// gradient/normal (from the previous pin-filled phi): what Lagrange_points,
// momentum and refilling read.
// rr_old (16-bit storage): the reference pairs of the populations.
template <typename S>
__device__ __forceinline__ void prep_node(const DevParams& P, const Pad& pd, const sym_particles* __restrict__ Sp,
                                          const S* __restrict__ pops, const typename Codec<S>::R* __restrict__ phi_cur,
                                          const typename Codec<S>::R* __restrict__ phi_prev,
                                          const int32_t* __restrict__ walls_all, const int32_t* __restrict__ pout,
                                          double* rhoN, double* rhoR, double* rhoB, double* fi, double* gx,
                                          double* gy, double* gz, double* nxv, double* nyv, double* nzv,
                                          const Ref* __restrict__ rr_old, int x, int y, int z) {
  using R = typename Codec<S>::R;
  const long long L = lin(P, x, y, z);
  const unsigned N = (unsigned)P.N;
  // masks and populations are read together, not one behind the other
  const Ref rref = Codec<S>::kRef ? rr_old[pd.idx(x, y, z)] : Ref{};
  const int wall = walls_all[L], near = pout[L];
  R pr[19], pb[19];
  unroll19([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    Codec<S>::template load<i>(pops, N, (unsigned)L, rref, pr[i], pb[i]);
  });
  if (wall > 0) {
    rhoN[L] = 0.0;
    gx[L] = 0.0; gy[L] = 0.0; gz[L] = 0.0; nxv[L] = 0.0; nyv[L] = 0.0; nzv[L] = 0.0;
    return;
  }
  // fi is read only by the momentum exchange, at nodes with links into a
  // particle (pout > 0): written there only
  const bool links = near > 0;
  R sr = R(0), sb = R(0);
  unroll19([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    if (links) fi[(size_t)i * N + L] = (double)(pr[i] + pb[i]);
    sr = sr + pr[i];
    sb = sb + pb[i];
  });
  rhoR[L] = (double)sr; rhoB[L] = (double)sb;
  rhoN[L] = (double)phi_cur[pd.idx(x, y, z)];
  R g0 = R(0), g1 = R(0), g2 = R(0);
#pragma unroll
  for (int i = 1; i < 19; i++) {
    const R val = R(W(i)) * phi_prev[pd.idx(x + CX(i), y + CY(i), z + CZ(i))];
    if (CX(i)) g0 = g0 + val * R(CX(i));
    if (CY(i)) g1 = g1 + val * R(CY(i));
    if (CZ(i)) g2 = g2 + val * R(CZ(i));
  }
  g0 = R(3) * g0; g1 = R(3) * g1; g2 = R(3) * g2;
  const R fn = sqrt(g0 * g0 + g1 * g1 + g2 * g2);
  R n0 = R(0), n1 = R(0), n2 = R(0);
  if (fn > R(P.evap)) {
    n0 = g0 / fn; n1 = g1 / fn; n2 = g2 / fn;
    const int q = near;
    if (q >= 1) {
      wet_rotate<R>(P, Sp, q, x, y, z, n0, n1, n2);
      g0 = fn * n0; g1 = fn * n1; g2 = fn * n2;
    }
  }
  gx[L] = g0; gy[L] = g1; gz[L] = g2; nxv[L] = n0; nyv[L] = n1; nzv[L] = n2;
}

// after refilling: a refilled node's canonical populations and phi into the
// fused state, encoded with a reference pair of its own (its colour
// densities), which it records in rr_old: the references this step's collide
// decodes with
template <typename S>
__device__ __forceinline__ void refill_import_node(const DevParams& P, const Pad& pd, S* pops,
                                                   typename Codec<S>::R* phi_cur, const double* __restrict__ ri, const double* __restrict__ bi,
                                                   const double* __restrict__ rhoN, Ref* __restrict__ rr_old,
                                                   int x, int y, int z) {
  using R = typename Codec<S>::R;
  const long long L = lin(P, x, y, z);
  const unsigned N = (unsigned)P.N;
  Ref ref{};
  if constexpr (Codec<S>::kRef) {
    double sr = 0.0, sb = 0.0;
    for (int i = 0; i < 19; i++) { sr += ri[(size_t)i * N + L]; sb += bi[(size_t)i * N + L]; }
    ref = sr + sb > 0.0 ? ref_pair(float(sr), float(sb)) : ref_rest(P);
    phi_store<Ref>(P, pd, rr_old, x, y, z, ref);
  }
  unroll19([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    const R r = R(ri[(size_t)i * N + L]), b = R(bi[(size_t)i * N + L]);
    Codec<S>::template store<i>(pops, N, (unsigned)L, ref, r, r + b);
  });
  phi_store<R>(P, pd, phi_cur, x, y, z, R(rhoN[L]));
}

// whole-domain conversions between the canonical arrays and the fused state
// rr (16-bit storage, else null): receives each node's reference pair, its
// colour densities (the rest pair where both are 0: solid or empty nodes)
template <typename S>
__global__ void k_import_pops(DevParams P, Pad pd, const double* __restrict__ ri, const double* __restrict__ bi,
                              S* pops, Ref* rr, Acc::T* acc, int* status) {
  using R = typename Codec<S>::R;
  const long long L = blockIdx.x * 256LL + threadIdx.x;
  if (L >= P.N) return;
  const unsigned N = (unsigned)P.N;
  Ref ref{};
  R sr = R(0), sb = R(0);
  if constexpr (Codec<S>::kRef) {
    double dr = 0.0, db = 0.0;
    for (int i = 0; i < 19; i++) { dr += ri[(size_t)i * N + L]; db += bi[(size_t)i * N + L]; }
    ref = dr + db > 0.0 ? ref_pair(float(dr), float(db)) : ref_rest(P);
    const unsigned Lu = (unsigned)L, q = Lu / (unsigned)P.nz;
    const int z = (int)(Lu - q * (unsigned)P.nz), x = (int)(q / (unsigned)P.ny), y = (int)(q - (unsigned)x * P.ny);
    phi_store<Ref>(P, pd, rr, x, y, z, ref);
  }
  unroll19([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    const R r = R(ri[(size_t)i * N + L]), b = R(bi[(size_t)i * N + L]);
    Codec<S>::template store<i>(pops, N, (unsigned)L, ref, r, r + b);
    sr = sr + r;
    sb = sb + b;
  });
  // the accumulators the first phase field after the import reads (storages
  // that accumulate)
  if constexpr (kAccumulate<S>) {
    if (!Acc::ok(sr) || !Acc::ok(sb)) atomicOr(status, 1);
    acc[L] = Acc::ok(sr) ? Acc::fix(sr) : 0;
    acc[L + P.N] = Acc::ok(sb) ? Acc::fix(sb) : 0;
  }
}
template <typename S>
__global__ void k_export_pops(DevParams P, Pad pd, const S* __restrict__ pops, const Ref* __restrict__ rr, double* ri,
                              double* bi) {
  using R = typename Codec<S>::R;
  const long long L = blockIdx.x * 256LL + threadIdx.x;
  if (L >= P.N) return;
  const unsigned N = (unsigned)P.N;
  Ref rref{};
  if constexpr (Codec<S>::kRef) {
    const unsigned Lu = (unsigned)L, q = Lu / (unsigned)P.nz;
    const int z = (int)(Lu - q * (unsigned)P.nz), x = (int)(q / (unsigned)P.ny), y = (int)(q - (unsigned)x * P.ny);
    rref = rr[pd.idx(x, y, z)];
  }
  unroll19([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    R r, b;
    Codec<S>::template load<i>(pops, N, (unsigned)L, rref, r, b);
    ri[(size_t)i * N + L] = (double)r;
    bi[(size_t)i * N + L] = (double)b;
  });
}
// calmacros (Source1.f90:770-831) of the current fused populations without
// touching the fused state: rho, u = sum f c / rho (no force shift) and
// phi = (rhoR - rhoB) / rho on fluid nodes; phi = 0, u = 0, rho = rho0 on
// solid nodes.  rr (16-bit storage): the reference pairs of the populations.
template <typename S>
__global__ void k_macros(DevParams P, Pad pd, const S* __restrict__ pops, const Ref* __restrict__ rr,
                         const int32_t* __restrict__ walls_all, double* rho, double* ux, double* uy, double* uz,
                         double* rhoN) {
  using R = typename Codec<S>::R;
  const long long L = blockIdx.x * 256LL + threadIdx.x;
  if (L >= P.N) return;
  if (walls_all[L] >= 1) {
    rhoN[L] = 0.0; ux[L] = 0.0; uy[L] = 0.0; uz[L] = 0.0; rho[L] = P.rho0;
    return;
  }
  const unsigned N = (unsigned)P.N;
  Ref rref{};
  if constexpr (Codec<S>::kRef) {
    const unsigned Lu = (unsigned)L, q = Lu / (unsigned)P.nz;
    const int z = (int)(Lu - q * (unsigned)P.nz), x = (int)(q / (unsigned)P.ny), y = (int)(q - (unsigned)x * P.ny);
    rref = rr[pd.idx(x, y, z)];
  }
  double sr = 0.0, sb = 0.0, mx = 0.0, my = 0.0, mz = 0.0;
  unroll19([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    R r, b;
    Codec<S>::template load<i>(pops, N, (unsigned)L, rref, r, b);
    const double f = (double)r + (double)b;
    sr += (double)r;
    sb += (double)b;
    if (CX(i)) mx += f * CX(i);
    if (CY(i)) my += f * CY(i);
    if (CZ(i)) mz += f * CZ(i);
  });
  const double rh = sr + sb;
  rho[L] = rh;
  ux[L] = mx / rh; uy[L] = my / rh; uz[L] = mz / rh;
  rhoN[L] = (sr - sb) / rh;
}

template <typename R>
__global__ void k_import_phi(DevParams P, Pad pd, const double* __restrict__ rhoN, R* phi) {
  const long long L = blockIdx.x * 256LL + threadIdx.x;
  if (L >= P.N) return;
  const int z = (int)(L % P.nz), y = (int)((L / P.nz) % P.ny), x = (int)(L / ((long long)P.nz * P.ny));
  phi_store<R>(P, pd, phi, x, y, z, R(rhoN[L]));
}
template <typename R>
__global__ void k_export_phi(DevParams P, Pad pd, const R* __restrict__ phi, double* rhoN) {
  const long long L = blockIdx.x * 256LL + threadIdx.x;
  if (L >= P.N) return;
  const int z = (int)(L % P.nz), y = (int)((L / P.nz) % P.ny), x = (int)(L / ((long long)P.nz * P.ny));
  rhoN[L] = (double)phi[pd.idx(x, y, z)];
}


}  // namespace fused
}  // namespace symb200
