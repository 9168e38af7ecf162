// Real-space nonbonded pair kernel: LJ 12-6 (Lorentz-Berthelot, optional switching) plus
// Ewald-screened, reaction-field or bare Coulomb, following forces/nonbonded.rs:842-924 and
// the pair functions at nonbonded.rs:1194-1288.
//
// One warp evaluates one tile: lane l owns i-particle l of block I; the tile's 32 j-entries
// are staged in shared memory and lane l visits entry (l + k) mod 32 at step k, so every
// (i, j) pair is seen once in 32 steps with conflict-free shared-memory reads.  The force on
// each j-entry travels with the entry: it is rotated one lane per step by a warp shuffle and
// is back in lane j after 32 steps.  Self tiles (entries = block I) visit each pair from both
// sides and keep only i-forces, at half energy.  "Halves" tiles hold 16 entries for each half
// of block I (gathered against that half's smaller box): each half-warp rotates its own 16
// entries in 16 steps.  Forces are summed in `Real` within a tile and
// committed as 64-bit fixed point, so the total does not depend on tile order.
//
// Pair membership reproduces the reference exactly: pairs whose squared distance falls
// within `band` of rc^2 are re-decided from the f64 master positions with the reference's
// minimum-image and r^2 < rc^2 arithmetic (explicitly rounded, no fused multiply-add).
#include <type_traits>

#include "kernels.h"
#include "pair_math.cuh"

namespace ommb200 {
namespace {

constexpr int kPairWarps = 4;
// The tile kernels' grid in units of the engine's pair grid (8 CTAs per SM unless tuned; 5 fit):
// with more CTAs than fit, each of one or two tiles per warp, the SMs that the reciprocal chain
// leaves free take more of them.  Against one unit, with a state after each run: 23,958 particles
// 100 steps 10.45 -> 9.88 ms, 9,387 in FP64 20 steps 2.89 -> 2.65 ms; a grid of just what fits, 5
// CTAs per SM, took 5 % longer than one unit.
constexpr int kPairWaves = 4;

template <class Real, int kElec, int kTerms, bool kDump, bool kSwitch>
__global__ void __launch_bounds__(32 * kPairWarps) pair_kernel(const PairArgs<Real> a) {
  using T4 = typename V4<Real>::T4;
  using T2 = typename V4<Real>::T2;
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ T4 s_pos[kPairWarps][32];
  __shared__ T2 s_lj[kPairWarps][32];
  __shared__ int s_atom[kPairWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int warp = blockIdx.x * kPairWarps + w;
  const int nwarps = gridDim.x * kPairWarps;
  const int nt = min(*a.n_tiles, a.tile_capacity);
  const T4* posq = reinterpret_cast<const T4*>(a.posq);
  const T2* ljp = reinterpret_cast<const T2*>(a.ljp);
  const T4* entries = reinterpret_cast<const T4*>(a.entries);
  long long e_fixed = 0;
  long long w_fixed[6] = {0, 0, 0, 0, 0, 0};

  for (int t = warp; t < nt; t += nwarps) {
    const int4 tile = a.tiles[t];
    const int I = tile.x;
    const bool self = (tile.y & kTileSelf) != 0;
    if (a.block_box && !self && boxes_apart(a.block_box, I, tile.w, a.skip2)) continue;
    const bool pair_image = (tile.y & kTilePairImage) != 0;
    const bool halves = (tile.y & kTileHalves) != 0;
    const int si = 32 * I + lane;
    const T4 pi = posq[si];
    const T2 li = ljp[si];
    const int ai = a.sorted_atom[si];
    const uint32_t excl = (tile.y & kTileHasMask) ? a.masks[32 * tile.z + lane] : 0u;
    int aj = ai;
    if (self) {
      s_pos[w][lane] = pi;
      s_lj[w][lane] = li;
    } else {
      const T4 e = entries[32 * t + lane];
      int slot;
      if constexpr (sizeof(Real) == 4) slot = __float_as_int(e.w);
      else slot = (int)e.w;
      T4 pj;
      T2 lj;
      if (slot >= 0) {
        pj = posq[slot];
        lj = ljp[slot];
        aj = a.sorted_atom[slot];
      } else {
        pj.x = pj.y = pj.z = pj.w = Real(0);
        lj.x = lj.y = Real(0);
        aj = -1;
      }
      pj.x += e.x;
      pj.y += e.y;
      pj.z += e.z;
      s_pos[w][lane] = pj;
      s_lj[w][lane] = lj;
    }
    s_atom[w][lane] = aj;
    __syncwarp();
    Real fix = 0, fiy = 0, fiz = 0, fjx = 0, fjy = 0, fjz = 0;
    double e_tile = 0.0;
    double w_tile[6] = {0, 0, 0, 0, 0, 0};
    // halves tiles: lanes 0-15 (first half of block I) meet entries 0-15 in 16 steps, lanes
    // 16-31 entries 16-31; otherwise every lane meets all 32 entries.  j-forces travel one
    // lane per step within their group and are back at their entry's lane at the end.
    const int hb = halves ? (lane & 16) : 0, kmask = halves ? 15 : 31;
    const int nsteps = halves ? 16 : 32;
    const int src = hb | ((lane + 1) & kmask);
#pragma unroll 4
    for (int k = self ? 1 : 0; k < nsteps; ++k) {
      const int jl = hb | ((lane + k) & kmask);
      const T4 pj = s_pos[w][jl];
      const T2 lj = s_lj[w][jl];
      Real dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
      if (pair_image) min_image_fast(dx, dy, dz, a.box);
      Real r2 = dx * dx + dy * dy + dz * dz;
      bool use = ((excl >> jl) & 1u) == 0u;
      if (a.use_cutoff) {
        bool inside = r2 < a.cutoff2;
        if (fabs(r2 - a.cutoff2) < a.band && use) {
          const int b = s_atom[w][jl];
          inside = ai >= 0 && b >= 0 &&
                   exact_inside(a.pos, ai, b, a.periodic, a.box_exact, a.cutoff2_exact);
        }
        use = use && inside;
      }
      if (kDump && use) {
        const int b = s_atom[w][jl];
        if (ai >= 0 && b >= 0 && (!self || ai < b)) {
          const unsigned long long slot = atomicAdd(a.pair_count, 1ull);
          if ((long long)slot < a.pair_capacity) {
            a.pair_dump[2 * slot] = ai < b ? ai : b;
            a.pair_dump[2 * slot + 1] = ai < b ? b : ai;
          }
        }
      }
      Real fo, en;
      pair_terms<Real, kElec, kTerms, kSwitch>(a, use ? r2 : Real(1), pi.w * pj.w, li.x + lj.x,
                                                li.y * lj.y, fo, en);
      fo = use ? fo : Real(0);
      fix = fma(fo, dx, fix);
      fiy = fma(fo, dy, fiy);
      fiz = fma(fo, dz, fiz);
      if (kTerms && use) {
        const double scale = self ? 0.5 : 1.0;
        e_tile += scale * (double)en;
        if (kTerms > kTermsEnergy) {
          w_tile[0] -= scale * (double)(fo * dx * dx);
          w_tile[1] -= scale * (double)(fo * dy * dy);
          w_tile[2] -= scale * (double)(fo * dz * dz);
          w_tile[3] -= scale * (double)(fo * dx * dy);
          w_tile[4] -= scale * (double)(fo * dx * dz);
          w_tile[5] -= scale * (double)(fo * dy * dz);
        }
      }
      if (!self) {
        fjx = fma(-fo, dx, fjx);
        fjy = fma(-fo, dy, fjy);
        fjz = fma(-fo, dz, fjz);
        fjx = __shfl_sync(FULL, fjx, src);
        fjy = __shfl_sync(FULL, fjy, src);
        fjz = __shfl_sync(FULL, fjz, src);
      }
    }
    const Real fscale = Real(kForceScale);
    if (ai >= 0) {
      add_fixed(a.force + ai, to_fixed(fix, fscale));
      add_fixed(a.force + a.n_atoms + ai, to_fixed(fiy, fscale));
      add_fixed(a.force + 2 * a.n_atoms + ai, to_fixed(fiz, fscale));
    }
    if (!self && aj >= 0) {
      add_fixed(a.force + aj, to_fixed(fjx, fscale));
      add_fixed(a.force + a.n_atoms + aj, to_fixed(fjy, fscale));
      add_fixed(a.force + 2 * a.n_atoms + aj, to_fixed(fjz, fscale));
    }
    if (kTerms) {
      // one fixed-point rounding per tile: reduce the tile's partial sums across the warp in
      // f64 first (a fixed order, so the result stays deterministic)
      for (int off = 16; off > 0; off >>= 1) {
        e_tile += __shfl_xor_sync(FULL, e_tile, off);
        if (kTerms > kTermsEnergy)
          for (int c = 0; c < 6; ++c) w_tile[c] += __shfl_xor_sync(FULL, w_tile[c], off);
      }
      if (a.block_segment) {  // a batch: each tile's energy goes to its own system
        if (lane == 0) {
          long long* dst = a.energy + 8 * a.block_segment[I];
          add_fixed(dst, to_fixed(e_tile, kEnergyScale));
          if (kTerms > kTermsEnergy)
            for (int c = 0; c < 6; ++c) add_fixed(dst + 1 + c, to_fixed(w_tile[c], kEnergyScale));
        }
      } else {
        e_fixed += to_fixed(e_tile, kEnergyScale);
        if (kTerms > kTermsEnergy)
          for (int c = 0; c < 6; ++c) w_fixed[c] += to_fixed(w_tile[c], kEnergyScale);
      }
    }
    __syncwarp();
  }
  if (kTerms && !a.block_segment) commit_cta<kTerms>(a.energy, e_fixed, w_fixed);
}

// The 2 P i-particles of a lane, packed two by two, and their forces.
template <int P>
struct ISlots {
  float2 npx[P], npy[P], npz[P], q[P], sg[P], ep[P];  // negated positions
};
template <int P>
struct IForces {
  float2 x[P], y[P], z[P];
};
template <int P>
__device__ __forceinline__ ISlots<P> load_slots(const float4* pos, const float2* lj, int stride) {
  ISlots<P> v;
#pragma unroll
  for (int s = 0; s < P; ++s) {
    const float4 p1 = pos[2 * s * stride], p2 = pos[(2 * s + 1) * stride];
    const float2 l1 = lj[2 * s * stride], l2 = lj[(2 * s + 1) * stride];
    v.npx[s] = make_float2(-p1.x, -p2.x);
    v.npy[s] = make_float2(-p1.y, -p2.y);
    v.npz[s] = make_float2(-p1.z, -p2.z);
    v.q[s] = make_float2(p1.w, p2.w);
    v.sg[s] = make_float2(l1.x, l2.x);
    v.ep[s] = make_float2(l1.y, l2.y);
  }
  return v;
}

// The sums over the 2 P groups of G lanes that met the same i-slots: the lane of group c keeps
// i-slot c of its 2 P.  The order of the additions is fixed.
template <int P>
__device__ __forceinline__ float3 reduce_groups(const IForces<P>& f, int lane, int G) {
  constexpr unsigned FULL = 0xffffffffu;
  const bool hi = (lane & (2 * G)) != 0, odd = (lane & G) != 0;
  auto sum = [&](const float2(&v)[P]) {
    float2 t = v[0];
    if constexpr (P == 2) {
      const float2 keep = hi ? v[1] : v[0], give = hi ? v[0] : v[1];
      t = x2::add(keep, make_float2(__shfl_xor_sync(FULL, give.x, 2 * G),
                                    __shfl_xor_sync(FULL, give.y, 2 * G)));
    }
    return (odd ? t.y : t.x) + __shfl_xor_sync(FULL, odd ? t.x : t.y, G);
  };
  return make_float3(sum(f.x), sum(f.y), sum(f.z));
}

// One entry (its values duplicated into both lanes of each packed value, so a step moves no
// register) against the lane's i-particles: adds to their forces, the entry's force and the sums.
// Bit c * shift of `excluded` drops the pair with i-particle c, whose number is iatom[c * stride].
template <int P, int kElec, int kTerms, bool kDump, bool kSwitch, bool kCutoff>
__device__ __forceinline__ void pair_step(const PairArgs<float>& a, const float4 jxy, const float4 jzq,
                                          const float4 jse, uint32_t excluded, int shift, bool image,
                                          bool self, const int* jatom, const int* iatom, int stride,
                                          const ISlots<P>& q, IForces<P>& f, float& fjx, float& fjy,
                                          float& fjz, double& e_acc, double (&w_acc)[6]) {
  float2 dx[P], dy[P], dz[P], r2[P];
  bool u[2 * P];
#pragma unroll
  for (int t = 0; t < 2 * P; ++t) u[t] = ((excluded >> (t * shift)) & 1u) == 0u;
#pragma unroll
  for (int s = 0; s < P; ++s) {
    dx[s] = x2::add(make_float2(jxy.x, jxy.y), q.npx[s]);
    dy[s] = x2::add(make_float2(jxy.z, jxy.w), q.npy[s]);
    dz[s] = x2::add(make_float2(jzq.x, jzq.y), q.npz[s]);
    if (image) {
      min_image_fast(dx[s].x, dy[s].x, dz[s].x, a.box);
      min_image_fast(dx[s].y, dy[s].y, dz[s].y, a.box);
    }
    r2[s] = x2::fma(dz[s], dz[s], x2::fma(dy[s], dy[s], x2::mul(dx[s], dx[s])));
  }
  if (kCutoff) {
    const float lo = a.cutoff2 - a.band, hi = a.cutoff2 + a.band;
    bool near_cutoff = false, c[2 * P];
#pragma unroll
    for (int t = 0; t < 2 * P; ++t) {
      const float r = (t & 1) ? r2[t >> 1].y : r2[t >> 1].x;
      u[t] = u[t] && r < hi;
      c[t] = u[t] && r >= lo;
      near_cutoff = near_cutoff || c[t];
    }
    if (near_cutoff) {  // within the band: the reference's decision from the f64 positions
      const int b = *jatom;
#pragma unroll
      for (int t = 0; t < 2 * P; ++t)
        if (c[t]) {
          const int ia = iatom[t * stride];
          u[t] = ia >= 0 && b >= 0 &&
                 exact_inside(a.pos, ia, b, a.periodic, a.box_exact, a.cutoff2_exact);
        }
    }
  }
  if (kDump) {
    const int b = *jatom;
    for (int t = 0; t < 2 * P; ++t) {
      const int ia = iatom[t * stride];
      if (u[t] && ia >= 0 && b >= 0 && (!self || ia < b)) {
        const unsigned long long slot = atomicAdd(a.pair_count, 1ull);
        if ((long long)slot < a.pair_capacity) {
          a.pair_dump[2 * slot] = ia < b ? ia : b;
          a.pair_dump[2 * slot + 1] = ia < b ? b : ia;
        }
      }
    }
  }
#pragma unroll
  for (int s = 0; s < P; ++s) {
    const bool u1 = u[2 * s], u2 = u[2 * s + 1];
    float2 fo, en;
    pair_terms_x2<kElec, kTerms, kSwitch>(
        a, x2::select(u1, u2, r2[s], 1.f), x2::mul(make_float2(jzq.z, jzq.w), q.q[s]),
        x2::add(make_float2(jse.x, jse.y), q.sg[s]), x2::mul(make_float2(jse.z, jse.w), q.ep[s]), fo, en);
    fo = x2::select(u1, u2, fo, 0.f);
    f.x[s] = x2::fma(fo, dx[s], f.x[s]);
    f.y[s] = x2::fma(fo, dy[s], f.y[s]);
    f.z[s] = x2::fma(fo, dz[s], f.z[s]);
    if (kTerms) {
      const double scale = self ? 0.5 : 1.0;
      if (u1) e_acc += scale * (double)en.x;
      if (u2) e_acc += scale * (double)en.y;
      if (kTerms > kTermsEnergy) {
        const float2 fdx = x2::mul(fo, dx[s]), fdy = x2::mul(fo, dy[s]), fdz = x2::mul(fo, dz[s]);
        const float2 w[6] = {x2::mul(fdx, dx[s]), x2::mul(fdy, dy[s]), x2::mul(fdz, dz[s]),
                             x2::mul(fdx, dy[s]), x2::mul(fdx, dz[s]), x2::mul(fdy, dz[s])};
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          if (u1) w_acc[c] -= scale * (double)w[c].x;
          if (u2) w_acc[c] -= scale * (double)w[c].y;
        }
      }
    }
    if (!self) {
      fjx = fmaf(-fo.x, dx[s].x, fjx);
      fjy = fmaf(-fo.x, dy[s].x, fjy);
      fjz = fmaf(-fo.x, dz[s].x, fjz);
      fjx = fmaf(-fo.y, dx[s].y, fjx);
      fjy = fmaf(-fo.y, dy[s].y, fjy);
      fjz = fmaf(-fo.y, dz[s].y, fjz);
    }
  }
}

// The FP32 form with 2 P i-particles per lane in packed (f32x2) arithmetic.  The warp splits into
// groups of G lanes (G = 8 / P for halves tiles, 16 / P otherwise); a group owns G consecutive
// entries and the i-slots that meet them, lane m of the group holding i-slots m + c G, c < 2 P, of
// its half (halves) or of the block.  In G steps the lane meets each of the group's entries once,
// evaluating the pairs with its i-particles two by two in the lanes of packed values; the entry's
// force (all its pairs summed) rotates one lane per step within the group and is back at the
// entry's own lane after G steps.  Every i-slot is met by 2 P groups, whose partial forces are
// summed at the end, so each lane commits the i-slot equal to its lane index and the entry it
// loaded.  The cutoff (and with it the exact decision band) applies to the Ewald and
// reaction-field forms; the bare-Coulomb form is the no-cutoff method.
//
// The warps of an SM issue two instructions in three cycles; what a step does once for all its
// pairs (entry reads, force shuffles, constants moved into register pairs, the loop) is a quarter
// of it with P = 1.  P = 2 halves that share per pair and gives each warp two independent chains,
// at 120 registers (4 CTAs per SM) against 96 (5): the 23,958-particle box takes 92.5 against
// 94.3 us per step, 8,217 particles with a barostat 99 against 104.  It serves the periodic lists.
// Tiles of the whole blocks of non-periodic systems keep P = 1: with a cutoff most of them are
// skipped, which more warps in flight do faster (4,999 particles: 180 us per evaluation against
// 182).
template <int P, int kElec, int kTerms, bool kDump, bool kSwitch>
__global__ void __launch_bounds__(32 * kPairWarps, P == 2 ? 4 : 5) pair_kernel_x2(const PairArgs<float> a) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr bool kCutoff = kElec != kElecCoulomb;
  __shared__ float4 s_j[kPairWarps][3][32];  // per entry (x, x, y, y), (z, z, q, q), (s, s, e, e)
  __shared__ int s_atom[kPairWarps][32];
  __shared__ float4 s_ipos[kPairWarps][32];
  __shared__ float2 s_ilj[kPairWarps][32];
  __shared__ int s_iatom[kPairWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int warp = blockIdx.x * kPairWarps + w;
  const int nwarps = gridDim.x * kPairWarps;
  const int nt = min(*a.n_tiles, a.tile_capacity);
  const float4* posq = reinterpret_cast<const float4*>(a.posq);
  const float2* ljp = reinterpret_cast<const float2*>(a.ljp);
  const float4* entries = reinterpret_cast<const float4*>(a.entries);
  long long e_fixed = 0;
  long long w_fixed[6] = {0, 0, 0, 0, 0, 0};

  for (int t = warp; t < nt; t += nwarps) {
    const int4 tile = a.tiles[t];
    const float4 e = entries[32 * t + lane];  // unused (unwritten) for self tiles
    const int I = tile.x;
    const bool self = (tile.y & kTileSelf) != 0;
    if (a.block_box && !self && boxes_apart(a.block_box, I, tile.w, a.skip2)) continue;
    const bool pair_image = (tile.y & kTilePairImage) != 0;
    const bool halves = (tile.y & kTileHalves) != 0;
    const int si = 32 * I + lane;
    const float4 pi = posq[si];
    const float2 li = ljp[si];
    const int ai = a.sorted_atom[si];
    const uint32_t excl = (tile.y & kTileHasMask) ? a.masks[32 * tile.z + lane] : 0u;
    float4 pj = pi;
    float2 lj = li;
    int aj = ai;
    if (!self) {
      const int slot = __float_as_int(e.w);
      pj = make_float4(0.f, 0.f, 0.f, 0.f);
      lj = make_float2(0.f, 0.f);
      aj = -1;
      if (slot >= 0) {
        pj = posq[slot];
        lj = ljp[slot];
        aj = a.sorted_atom[slot];
      }
      pj.x += e.x;
      pj.y += e.y;
      pj.z += e.z;
    }
    s_j[w][0][lane] = make_float4(pj.x, pj.x, pj.y, pj.y);
    s_j[w][1][lane] = make_float4(pj.z, pj.z, pj.w, pj.w);
    s_j[w][2][lane] = make_float4(lj.x, lj.x, lj.y, lj.y);
    s_atom[w][lane] = aj;
    s_ipos[w][lane] = pi;
    s_ilj[w][lane] = li;
    s_iatom[w][lane] = ai;
    __syncwarp();
    const int G = (halves ? 8 : 16) / P, gm = G - 1;
    const int m = lane & gm, eb = lane & ~gm;
    const int i0 = (halves ? (lane & 16) : 0) + m;
    // exclusion/padding bits of the i-slots in step order: bit (16 / P) c + k of i-slot i0 + c G
    // stands for entry eb + ((m + k) mod G); a self tile also drops the diagonal
    uint32_t steps_mask = 0u;
    if (self || (tile.y & kTileHasMask)) {
      const uint32_t gmask = (1u << G) - 1u;
#pragma unroll
      for (int c = 0; c < 2 * P; ++c) {
        const int i = i0 + c * G;
        const uint32_t x = ((__shfl_sync(FULL, excl, i) | (self ? 1u << i : 0u)) >> eb) & gmask;
        steps_mask |= (((x >> m) | (x << (G - m))) & gmask) << (16 / P * c);
      }
    }
    const ISlots<P> islots = load_slots<P>(s_ipos[w] + i0, s_ilj[w] + i0, G);
    IForces<P> f = {};
    float fjx = 0.f, fjy = 0.f, fjz = 0.f;
    double e_tile = 0.0;
    double w_tile[6] = {0, 0, 0, 0, 0, 0};
    const int src = eb | ((m + 1) & gm);
    auto steps = [&](auto image_tag) {
      constexpr bool kImage = decltype(image_tag)::value;
      uint32_t sm = steps_mask;
#pragma unroll 1  // unrolled, the constants no longer stay in registers
      for (int k = 0; k < G; ++k) {
        const int jl = eb | ((m + k) & gm);
        pair_step<P, kElec, kTerms, kDump, kSwitch, kCutoff>(
            a, s_j[w][0][jl], s_j[w][1][jl], s_j[w][2][jl], sm, 16 / P, kImage, self, s_atom[w] + jl,
            s_iatom[w] + i0, G, islots, f, fjx, fjy, fjz, e_tile, w_tile);
        sm >>= 1;
        if (!self) {
          fjx = __shfl_sync(FULL, fjx, src);
          fjy = __shfl_sync(FULL, fjy, src);
          fjz = __shfl_sync(FULL, fjz, src);
        }
      }
    };
    if (pair_image)
      steps(std::true_type{});
    else
      steps(std::false_type{});
    // the groups that met the same i-slots combine; the lane commits i-slot `lane`
    const float3 fi = reduce_groups(f, lane, G);
    const float fs = float(kForceScale);
    if (ai >= 0) {
      add_fixed(a.force + ai, to_fixed(fi.x, fs));
      add_fixed(a.force + a.n_atoms + ai, to_fixed(fi.y, fs));
      add_fixed(a.force + 2 * a.n_atoms + ai, to_fixed(fi.z, fs));
    }
    if (!self && aj >= 0) {
      add_fixed(a.force + aj, to_fixed(fjx, fs));
      add_fixed(a.force + a.n_atoms + aj, to_fixed(fjy, fs));
      add_fixed(a.force + 2 * a.n_atoms + aj, to_fixed(fjz, fs));
    }
    if (kTerms) {
      for (int off = 16; off > 0; off >>= 1) {
        e_tile += __shfl_xor_sync(FULL, e_tile, off);
        if (kTerms > kTermsEnergy)
          for (int c = 0; c < 6; ++c) w_tile[c] += __shfl_xor_sync(FULL, w_tile[c], off);
      }
      if (a.block_segment) {
        if (lane == 0) {
          long long* dst = a.energy + 8 * a.block_segment[I];
          add_fixed(dst, to_fixed(e_tile, kEnergyScale));
          if (kTerms > kTermsEnergy)
            for (int c = 0; c < 6; ++c) add_fixed(dst + 1 + c, to_fixed(w_tile[c], kEnergyScale));
        }
      } else {
        e_fixed += to_fixed(e_tile, kEnergyScale);
        if (kTerms > kTermsEnergy)
          for (int c = 0; c < 6; ++c) w_fixed[c] += to_fixed(w_tile[c], kEnergyScale);
      }
    }
    __syncwarp();
  }
  if (kTerms && !a.block_segment) commit_cta<kTerms>(a.energy, e_fixed, w_fixed);
}

// ---- culling form -----------------------------------------------------------------------
// The packed FP32 form over a halves-tile list, with the entries culled at the current
// positions.  A warp takes a run of consecutive tiles of one block I (a sub-chunk: tiles
// [sub K, (sub + 1) K) of the block's range, the last sub-chunk taking the rest) and drops
// every entry that lies farther than the cutoff (plus the exact-decision band) from the
// bounding box of the current positions of its half of I: no pair of such an entry can be
// inside the cutoff, so the pair set is unchanged.  The surviving entries of each half queue in
// a ring in shared memory; whenever both halves hold 16, a round runs the halves-tile steps
// (groups of 4 lanes, four i-slots per lane) over 16 queued entries per half, and at the end of
// the sub-chunk the rest runs with dummy entries (masked for every i-slot) topping the rounds
// up.  Each round commits its entries' forces; the i-forces accumulate over the sub-chunk and
// are committed once.  Sub-chunks are fixed runs of a block's own tiles, whose order the
// builder fixes, so rounds, float sums and forces are the same run to run, whichever warp
// takes them: warps fetch sub-chunks from a counter (all blocks' first sub-chunks, then the
// second ones, ...), and the last warp to finish resets the counter for the next launch (no
// warp waits for another).  Self tiles and tiles that need a per-pair minimum image are staged
// and run directly, after the queue is drained; a self tile runs as two rounds (each half's
// i-slots with the entries of its own half, then of the other half).  Exclusion words are kept
// over all 32 i-slots of block I, an entry of a tile holding only its own half's bits.  The
// next tile's header, entry and mask word are loaded one tile ahead.
constexpr int kRing = 64;  // queued entries per half of block I, per warp (a power of two)

// 32 x 32 bit transpose across the warp: lane r holds row r (bit c = M[r][c]); the result in
// lane c is column c (bit r = M[r][c]).  Five butterfly stages of block swaps.
__device__ __forceinline__ uint32_t transpose_bits(uint32_t x, int lane) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const uint32_t lo = s == 16  ? 0x0000FFFFu
                        : s == 8 ? 0x00FF00FFu
                        : s == 4 ? 0x0F0F0F0Fu
                        : s == 2 ? 0x33333333u
                                 : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, s);
    x = (lane & s) ? ((x & ~lo) | ((y >> s) & lo)) : ((x & lo) | ((y & lo) << s));
  }
  return x;
}

struct CullRing {
  float4 j[3][2 * kRing];  // per entry (x, x, y, y), (z, z, q, q), (s, s, e, e); half h owns
                           // [h kRing, (h + 1) kRing)
  uint32_t em[2 * kRing];  // exclusion/padding bits of the entry over the 32 i-slots of I
  int at[2 * kRing];       // particle of the entry, -1 for a dummy
  float4 ipos[32];         // block I
  float2 ilj[32];
  int iatom[32];
  float4 lo[2], hi[2];     // bounding box of the real particles of each half of block I
};

__device__ __forceinline__ void ring_put(CullRing& r, int f, float4 pj, float2 lj, uint32_t em,
                                         int at) {
  r.j[0][f] = make_float4(pj.x, pj.x, pj.y, pj.y);
  r.j[1][f] = make_float4(pj.z, pj.z, pj.w, pj.w);
  r.j[2][f] = make_float4(lj.x, lj.x, lj.y, lj.y);
  r.em[f] = em;
  r.at[f] = at;
}

// Rounds of the culling kernel, in the order a warp runs them.
enum CullRound : int {
  kRoundQueue = 0,  // 16 queued entries per half from the ring heads
  kRoundImage = 1,  // a staged tile whose pairs take the minimum image
  kRoundSelf0 = 2,  // a staged self tile: each half's i-slots with its own half
  kRoundSelf1 = 3,  // ... then with the other half
};

// One round: lane m of a group of 4 lanes meets the group's 4 entries, at ring slots
// base + ((m + k) mod 4), with its four i-slots i + 4 c, in 4 steps.  The entry's force rotates
// one lane per step and ends in the lane whose m is the entry's position (self rounds keep no
// entry forces: every pair is met from both sides, at half energy).  Four i-slots per lane for the
// reasons given at the tile kernel; 255,477 particles: 398 us per launch with two, 390 with four.
template <int kElec, int kTerms, bool kDump, bool kSwitch>
__device__ __forceinline__ void cull_steps(const PairArgs<float>& a, const CullRing& r, int base,
                                           int m, int src, int i, bool image, bool self,
                                           const ISlots<2>& q, IForces<2>& f, float& fjx,
                                           float& fjy, float& fjz, double& e_acc, double (&w_acc)[6]) {
  constexpr unsigned FULL = 0xffffffffu;
#pragma unroll 1
  for (int k = 0; k < 4; ++k) {
    const int jf = base + ((m + k) & 3);
    pair_step<2, kElec, kTerms, kDump, kSwitch, true>(
        a, r.j[0][jf], r.j[1][jf], r.j[2][jf], r.em[jf] >> i, 4, image, self, r.at + jf, r.iatom + i,
        4, q, f, fjx, fjy, fjz, e_acc, w_acc);
    if (!self) {
      fjx = __shfl_sync(FULL, fjx, src);
      fjy = __shfl_sync(FULL, fjy, src);
      fjz = __shfl_sync(FULL, fjz, src);
    }
  }
}

template <int kElec, int kTerms, bool kDump, bool kSwitch>
__global__ void __launch_bounds__(32 * kPairWarps, 4) pair_kernel_cull(const PairArgs<float> a) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ CullRing s_ring[kPairWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  CullRing& rg = s_ring[w];
  const int nwarps = gridDim.x * kPairWarps;
  const int nt = min(*a.n_tiles, a.tile_capacity);
  const int per = a.cull_chunks, K = a.cull_tiles;
  const int nb = *a.n_blocks;
  const int n_items = nb * per;
  const float4* posq = reinterpret_cast<const float4*>(a.posq);
  const float2* ljp = reinterpret_cast<const float2*>(a.ljp);
  const float4* entries = reinterpret_cast<const float4*>(a.entries);
  // rounds: groups of 4 lanes (gsub: the group's first entry within its half's 16); lane m of
  // a group meets i-slots i0 + 4 c, i0 = 16 h + m, of its half h
  const int h = lane >> 4, m = lane & 3, gsub = lane & 12;
  const int i0 = (lane & 16) + m;
  const int src4 = (lane & ~3) | ((m + 1) & 3);
  const float fs = float(kForceScale);
  long long e_fixed = 0;
  long long w_fixed[6] = {0, 0, 0, 0, 0, 0};

  for (;;) {
    int it = 0;
    if (lane == 0) it = atomicAdd(a.cull_work, 1);
    it = __shfl_sync(FULL, it, 0);
    if (it >= n_items) break;
    const int sub = it / nb, I = it - sub * nb;
    const int tb = a.block_tiles[2 * I], tn = a.block_tiles[2 * I + 1];
    const int k0 = sub * K;
    if (tb < 0 || k0 >= tn) continue;  // uniform
    const int k1 = min(sub == per - 1 ? tn : min(tn, k0 + K), nt - tb);
    {
      const int si = 32 * I + lane;
      rg.ipos[lane] = posq[si];
      rg.ilj[lane] = ljp[si];
      rg.iatom[lane] = a.sorted_atom[si];
    }
    __syncwarp();
    const ISlots<2> islots = load_slots<2>(rg.ipos + i0, rg.ilj + i0, 4);
    {  // bounding box of the real particles of each half (empty: nothing is kept)
      const float4 pi = rg.ipos[lane];
      const bool real = rg.iatom[lane] >= 0;
      float lox = real ? pi.x : INFINITY, loy = real ? pi.y : INFINITY,
            loz = real ? pi.z : INFINITY;
      float hix = real ? pi.x : -INFINITY, hiy = real ? pi.y : -INFINITY,
            hiz = real ? pi.z : -INFINITY;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        lox = fminf(lox, __shfl_xor_sync(FULL, lox, o));
        loy = fminf(loy, __shfl_xor_sync(FULL, loy, o));
        loz = fminf(loz, __shfl_xor_sync(FULL, loz, o));
        hix = fmaxf(hix, __shfl_xor_sync(FULL, hix, o));
        hiy = fmaxf(hiy, __shfl_xor_sync(FULL, hiy, o));
        hiz = fmaxf(hiz, __shfl_xor_sync(FULL, hiz, o));
      }
      if ((lane & 15) == 0) {
        rg.lo[h] = make_float4(lox, loy, loz, 0.f);
        rg.hi[h] = make_float4(hix, hiy, hiz, 0.f);
      }
      __syncwarp();
    }
    IForces<2> f = {};
    double e_acc = 0.0;
    double w_acc[6] = {0, 0, 0, 0, 0, 0};
    int hd0 = 0, tl0 = 0, hd1 = 0, tl1 = 0;  // ring cursors per half (heads: multiples of 16)
    int mode = kRoundQueue;                   // the next round's kind
    int n_rounds = 0;
    bool staged_image = false;                // the staged self tile's pairs take the image
    int k = k0;
    // tile k's header, entry and exclusion word; the next tile's are fetched one tile ahead,
    // so their latency overlaps this tile's rounds
    int4 tile = make_int4(0, 0, 0, 0);
    float4 ent = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t xw = 0u;
    if (k < k1) {
      tile = a.tiles[tb + k];
      ent = entries[32 * (tb + k) + lane];
      if (tile.y & kTileHasMask) xw = a.masks[32 * tile.z + lane];
    }
    for (;;) {
      // a round is due for a staged tile, for two full halves or a nearly full ring, or to
      // empty the queue before a tile that must be staged and at the end of the sub-chunk
      const int q0 = tl0 - hd0, q1 = tl1 - hd1;
      const bool special = k < k1 && (tile.y & (kTileSelf | kTilePairImage)) != 0;
      const bool due = mode != kRoundQueue || (q0 >= 16 && q1 >= 16) || q0 > kRing - 16 ||
                       q1 > kRing - 16 || ((k >= k1 || special) && (q0 > 0 || q1 > 0));
      if (due) {
        if (mode == kRoundQueue) {  // top each half up to 16 entries with dummies
          const int hd = h ? hd1 : hd0, q = h ? q1 : q0, e = lane & 15;
          if (e >= q)
            ring_put(rg, kRing * h + ((hd + e) & (kRing - 1)), make_float4(0.f, 0.f, 0.f, 0.f),
                     make_float2(0.f, 0.f), 0xFFFFFFFFu, -1);
          __syncwarp();
        }
        const bool self = mode >= kRoundSelf0;
        const int base = mode == kRoundQueue ? kRing * h + ((h ? hd1 : hd0) & (kRing - 1)) + gsub
                                             : kRing * (h ^ (mode == kRoundSelf1)) + gsub;
        float fjx = 0.f, fjy = 0.f, fjz = 0.f;
        cull_steps<kElec, kTerms, kDump, kSwitch>(
            a, rg, base, m, src4, i0, mode == kRoundImage || (self && staged_image), self, islots, f,
            fjx, fjy, fjz, e_acc, w_acc);
        ++n_rounds;
        if (!self) {
          const int aj = rg.at[base + m];
          if (aj >= 0) {
            add_fixed(a.force + aj, to_fixed(fjx, fs));
            add_fixed(a.force + a.n_atoms + aj, to_fixed(fjy, fs));
            add_fixed(a.force + 2 * a.n_atoms + aj, to_fixed(fjz, fs));
          }
        }
        if (mode == kRoundQueue) {
          hd0 += 16;
          hd1 += 16;
          tl0 = max(tl0, hd0);
          tl1 = max(tl1, hd1);
        } else if (mode == kRoundSelf0) {
          mode = kRoundSelf1;
        } else {
          mode = kRoundQueue;
          hd0 = tl0 = hd1 = tl1 = 0;
        }
        __syncwarp();
        continue;
      }
      if (k >= k1) break;
      int4 tile_n = make_int4(0, 0, 0, 0);
      float4 ent_n = make_float4(0.f, 0.f, 0.f, 0.f);
      uint32_t xw_n = 0u;
      if (k + 1 < k1) {
        tile_n = a.tiles[tb + k + 1];
        ent_n = entries[32 * (tb + k + 1) + lane];
        if (tile_n.y & kTileHasMask) xw_n = a.masks[32 * tile_n.z + lane];
      }
      // tile k (the queue is empty if it is special)
      uint32_t col = 0u;  // exclusion bits of entry `lane` over the 32 i-slots
      if (tile.y & kTileHasMask) col = transpose_bits(xw, lane);
      if (tile.y & kTileSelf) {
        ring_put(rg, kRing * h + (lane & 15), rg.ipos[lane], rg.ilj[lane], col | (1u << lane),
                 rg.iatom[lane]);
        mode = kRoundSelf0;
        staged_image = (tile.y & kTilePairImage) != 0;
      } else {
        const float4 e = ent;
        const int slot = __float_as_int(e.w);
        float4 pj = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 lj = make_float2(0.f, 0.f);
        int aj = -1;
        if (slot >= 0) {
          pj = posq[slot];
          lj = ljp[slot];
          aj = a.sorted_atom[slot];
        }
        pj.x += e.x;
        pj.y += e.y;
        pj.z += e.z;
        const uint32_t hmask = 0xFFFFu << (lane & 16);  // the i-slots of this entry's half
        const uint32_t em = col & hmask;
        if (special) {  // a small box: every pair takes the minimum image, nothing is culled
          ring_put(rg, kRing * h + (lane & 15), pj, lj, slot >= 0 ? em : 0xFFFFFFFFu, aj);
          mode = kRoundImage;
        } else {
          // distance from the entry to its half's box with the pair distance's rounding
          // (monotone in each component, so never above any of the entry's pair r^2)
          const float4 blo = rg.lo[h], bhi = rg.hi[h];
          const float cx = fmaxf(fmaxf(blo.x - pj.x, pj.x - bhi.x), 0.f);
          const float cy = fmaxf(fmaxf(blo.y - pj.y, pj.y - bhi.y), 0.f);
          const float cz = fmaxf(fmaxf(blo.z - pj.z, pj.z - bhi.z), 0.f);
          const float d2 = fmaf(cz, cz, fmaf(cy, cy, cx * cx));
          const bool keep = slot >= 0 && d2 < a.cull2 && em != hmask;
          const unsigned kb = __ballot_sync(FULL, keep);
          if (keep) {
            const unsigned mine = (kb >> (lane & 16)) & 0xFFFFu;
            const int pos = (h ? tl1 : tl0) + __popc(mine & ((1u << (lane & 15)) - 1u));
            ring_put(rg, kRing * h + (pos & (kRing - 1)), pj, lj, em, aj);
          }
          tl0 += __popc(kb & 0xFFFFu);
          tl1 += __popc(kb >> 16);
        }
      }
      __syncwarp();
      ++k;
      tile = tile_n;
      ent = ent_n;
      xw = xw_n;
    }
    // the four groups of each half met the same i-slots; the lane commits i-slot `lane`
    const float3 fi = reduce_groups(f, lane, 4);
    if (lane == 0) atomicAdd(a.cull_rounds, (unsigned long long)n_rounds);
    const int ai = rg.iatom[lane];
    if (ai >= 0) {
      add_fixed(a.force + ai, to_fixed(fi.x, fs));
      add_fixed(a.force + a.n_atoms + ai, to_fixed(fi.y, fs));
      add_fixed(a.force + 2 * a.n_atoms + ai, to_fixed(fi.z, fs));
    }
    if (kTerms) {
      for (int off = 16; off > 0; off >>= 1) {
        e_acc += __shfl_xor_sync(FULL, e_acc, off);
        if (kTerms > kTermsEnergy)
          for (int c = 0; c < 6; ++c) w_acc[c] += __shfl_xor_sync(FULL, w_acc[c], off);
      }
      e_fixed += to_fixed(e_acc, kEnergyScale);
      if (kTerms > kTermsEnergy)
        for (int c = 0; c < 6; ++c) w_fixed[c] += to_fixed(w_acc[c], kEnergyScale);
    }
    __syncwarp();
  }
  if (kTerms) commit_cta<kTerms>(a.energy, e_fixed, w_fixed);
  // a warp counts itself only after its last fetch returned (the fetch's value decided the
  // loop's exit), so when the last warp counts itself no fetch is left and it may reset both
  // counters for the next launch
  if (lane == 0) {
    if (atomicAdd(a.cull_work + 1, 1) == nwarps - 1) {
      a.cull_work[0] = 0;
      a.cull_work[1] = 0;
    }
  }
}

// The packed particles of every slot (a rebuild packs its own, and between rebuilds the integrator
// writes those it moves: this runs for non-periodic systems and after new parameters or a
// checkpoint).
template <class Real>
__global__ void pack_kernel(int n_slots, const int* sorted_atom, const double* pos,
                            const int* image, const double* block_center, const double* qscaled,
                            const double* half_sigma, const double* two_sqrt_eps,
                            typename V4<Real>::T4* posq, typename V4<Real>::T2* ljp,
                            Box<double> b, float4* block_box) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n_slots) return;
  const int a = sorted_atom[s];
  typename V4<Real>::T4 out;
  typename V4<Real>::T2 lj;
  if (a < 0) {
    out.x = out.y = out.z = out.w = Real(0);
    lj.x = lj.y = Real(0);
  } else {
    const double x[3] = {pos[3 * a], pos[3 * a + 1], pos[3 * a + 2]};
    double r[3];
    block_local(x, image[3 * a], image[3 * a + 1], image[3 * a + 2], block_center + 3 * (s >> 5),
                b, r);
    out.x = (Real)r[0];
    out.y = (Real)r[1];
    out.z = (Real)r[2];
    out.w = (Real)qscaled[a];
    lj.x = (Real)half_sigma[a];
    lj.y = (Real)two_sqrt_eps[a];
  }
  posq[s] = out;
  ljp[s] = lj;
  if (block_box) {  // whole warps: n_slots is a multiple of 32
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    if (a >= 0) {
      lo[0] = hi[0] = (float)out.x;
      lo[1] = hi[1] = (float)out.y;
      lo[2] = hi[2] = (float)out.z;
    }
    for (int o = 16; o > 0; o >>= 1)
      for (int d = 0; d < 3; ++d) {
        lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
        hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
      }
    if ((s & 31) == 0) store_box(block_box, s >> 5, lo, hi);
  }
}

}  // namespace

template <class Real>
void launch_pair(const PairArgs<Real>& a, int elec, int terms, bool dump, int grid,
                 cudaStream_t s) {
#define OMMB200_PAIR(E, EN, D, SW)                                                  \
  if constexpr (sizeof(Real) == 4) {                                                \
    if constexpr (E != kElecCoulomb) {                                              \
      if (a.cull_tiles > 0) {                                                       \
        cudaFuncSetAttribute(pair_kernel_cull<E, EN, D, SW>,                        \
                             cudaFuncAttributePreferredSharedMemoryCarveout,        \
                             cudaSharedmemCarveoutMaxShared);                       \
        pair_kernel_cull<E, EN, D, SW><<<grid, 32 * kPairWarps, 0, s>>>(a);         \
        return;                                                                     \
      }                                                                             \
    }                                                                               \
    if (a.periodic)                                                                 \
      pair_kernel_x2<2, E, EN, D, SW><<<kPairWaves * grid, 32 * kPairWarps, 0, s>>>(a); \
    else                                                                            \
      pair_kernel_x2<1, E, EN, D, SW><<<kPairWaves * grid, 32 * kPairWarps, 0, s>>>(a); \
  } else                                                                            \
    pair_kernel<Real, E, EN, D, SW><<<kPairWaves * grid, 32 * kPairWarps, 0, s>>>(a)
#define OMMB200_PAIR_SW(E, EN, D)     \
  if (a.use_switching)                \
    OMMB200_PAIR(E, EN, D, true);     \
  else                                \
    OMMB200_PAIR(E, EN, D, false)
#define OMMB200_PAIR_E(EN, D)                                      \
  if (elec == kElecEwald) {                                        \
    OMMB200_PAIR_SW(kElecEwald, EN, D);                            \
  } else if (elec == kElecReactionField) {                         \
    OMMB200_PAIR_SW(kElecReactionField, EN, D);                    \
  } else {                                                         \
    OMMB200_PAIR_SW(kElecCoulomb, EN, D);                          \
  }
  if (dump) {
    OMMB200_PAIR_E(kTermsNone, true)
  } else if (terms == kTermsVirial) {
    OMMB200_PAIR_E(kTermsVirial, false)
  } else if (terms == kTermsEnergy) {
    OMMB200_PAIR_E(kTermsEnergy, false)
  } else {
    OMMB200_PAIR_E(kTermsNone, false)
  }
#undef OMMB200_PAIR_E
#undef OMMB200_PAIR_SW
#undef OMMB200_PAIR
}

template <class Real>
void launch_pack(int n_slots, const int* sorted_atom, const double* pos, const int* image,
                 const double* block_center, const double* qscaled, const double* half_sigma,
                 const double* two_sqrt_eps, void* posq, void* ljp, const Box<double>& box,
                 cudaStream_t s, float4* block_box) {
  pack_kernel<Real><<<ceil_div(n_slots, 256), 256, 0, s>>>(
      n_slots, sorted_atom, pos, image, block_center, qscaled, half_sigma, two_sqrt_eps,
      reinterpret_cast<typename V4<Real>::T4*>(posq), reinterpret_cast<typename V4<Real>::T2*>(ljp),
      box, block_box);
}

template void launch_pair<float>(const PairArgs<float>&, int, int, bool, int, cudaStream_t);
template void launch_pair<double>(const PairArgs<double>&, int, int, bool, int, cudaStream_t);
template void launch_pack<float>(int, const int*, const double*, const int*, const double*,
                                 const double*, const double*, const double*, void*, void*,
                                 const Box<double>&, cudaStream_t, float4*);
template void launch_pack<double>(int, const int*, const double*, const int*, const double*,
                                  const double*, const double*, const double*, void*, void*,
                                  const Box<double>&, cudaStream_t, float4*);

}  // namespace ommb200
