// cgx_tma.cuh -- prolongation tiles (device code).
//
// Separable x -> y -> z passes over a tile, the time interpolation fused, in
// CarpetLib's operation order.  A CTA marches its tile in stages of bz coarse
// planes:
//
//   * staging: the stage's coarse box (bx points, by rows, bz planes, every
//     timelevel) lies in one of two shared-memory slots.  TMA form: one
//     elected thread issues one bulk tensor copy per timelevel
//     (cp.async.bulk.tensor), completing on the slot's mbarrier; boxes may
//     start outside the array (zero fill), which only masked outputs read.
//     Plain form (arrays the tensor-copy unit cannot address): cp.async by
//     all threads.  The copies of stage s + 2 start once the x pass has read
//     stage s, and have the y/z pass of a whole stage to land;
//   * x pass: one thread per (timelevel, plane, coarse row) walks its row
//     (Line), two points per 16-byte load: by rows of an odd number of
//     16-byte units, so that the lanes of a quarter warp, which hold
//     consecutive rows, meet no bank conflict.  One item per (row, base), as
//     a window form would have it, loads 6 points per base instead of 1.6
//     and spent half of the kernel's shared-memory wavefronts;
//   * y/z pass: thread = (fine x, coarse y row) takes the window of its row
//     from the x-pass rows, both fine y, and pushes them into its z lines,
//     whose open sums stay in registers over the whole tile; threads without
//     a point compute on clamped indices and their stores are masked, so no
//     branch diverges.
//
// Two barriers per stage.  What bounds it: instruction issue and the FP64
// pipe (the exact mode's separate products and sums), not DRAM.
//
// A descriptor is staged by TMA when its source arrays can be described to
// the tensor-copy unit (16-byte aligned base, even row and plane pitches);
// the host builds one CUtensorMap per timelevel.
#pragma once
#include <cuda.h>

#include "cgx_device.cuh"

namespace cgx {

// Tile configurations the autotuner chooses between: threads per CTA, coarse
// y rows of a 16-wide tile (threads / 16: one thread per fine x and coarse
// row), the most fine z points per tile, CTAs per SM the register allocation
// must allow.  Configuration 0 is the default.  Configurations that differ
// in pz alone share their kernels (tma_kernel_cfg).  mb is that of the widest
// common case, order 5 with three timelevels (tma_blocks).
struct TmaCfg {
  int nt, pyc, pz, mb;
};
constexpr TmaCfg TMA_CFGS[] = {{256, 16, 64, 2}, {128, 8, 64, 4}, {128, 8, 32, 4}, {128, 8, 64, 5}, {128, 8, 32, 6}};
constexpr int TMA_NCFG = 5;
constexpr int tma_kernel_cfg(int c) { return c == 2 ? 1 : c; }
// the configuration of the kernels that stage by cp.async, and that of a
// single box staged by TMA
constexpr int PLAIN_CFG = 0, BOX_CFG = 1;
// mbarriers per CTA: one per stage slot
constexpr int TMA_NB = 2;

// Shared-memory geometry of a tile configuration for a stencil window of
// width W and NTL timelevels (host and device).
//   stage      bx = the coarse bases + the window + one point of
//              even-alignment shift, rounded up to an odd number of 16-byte
//              units; by = ptyc + W rows; bz planes; by * bz <= tma_rpt and
//              bx * by * bz <= tma_tls per (slot, timelevel)
//   x-pass rows  one per (timelevel, plane, row), pitch TMA_XR (two fine
//              points per coarse base, at most 9 bases): NTL * by * bz <= NT,
//              one thread each
// tma_rpt is sized for whole planes of pyc + 1 rows: three planes of three
// timelevels in 128 threads.  TMA_PMAX planes at most: more planes per stage
// mean fewer barriers, but less room for other CTAs.
constexpr int TMA_XR = PTXMAX + 2; // even: 16-byte rows
constexpr int TMA_PMAX = 4;
__host__ __device__ constexpr int tma_bx(int nbx, int W) {
  const int e = (nbx + W + 2) & ~1;
  return e / 2 % 2 ? e : e + 2;
}
__host__ __device__ constexpr int tma_rpt(int W, int nt, int pyc, int ntl, int planes) {
  const int by = pyc + W + 1, p = nt / (ntl * by);
  const int q = planes ? planes : p < 1 ? 1 : p > TMA_PMAX ? TMA_PMAX : p;
  return q * by < nt / ntl ? q * by : nt / ntl;
}
__host__ __device__ constexpr int tma_tls(int W, int nt, int pyc, int ntl, int planes) {
  return (tma_bx(PTXMAX / 2, W) * tma_rpt(W, nt, pyc, ntl, planes) + 15) / 16 * 16;
}

// Planes per stage of the one-timelevel tiles: whole turns of the phases of a
// family's z lines, so that every plane of a stage has its phase at compile
// time; 0 where the phase is carried (three timelevels: a turn of order 5
// would take 195 threads and half of the shared memory again).
__host__ __device__ constexpr int tma_planes(int phases, int ntl) { return ntl == 1 ? (3 + phases) / phases * phases : 0; }

template <class F, int NTL, int CFG> struct TSmem {
  static constexpr int W = F::HI - F::LO;
  static constexpr int NT = TMA_CFGS[CFG].nt, PYC = TMA_CFGS[CFG].pyc;
  static constexpr int P = tma_planes(F::PHASES, NTL);
  static constexpr int RPT = tma_rpt(W, NT, PYC, NTL, P); // rows per (slot, timelevel)
  static constexpr int TLS = tma_tls(W, NT, PYC, NTL, P); // doubles per (slot, timelevel)
  static constexpr int coarse = TMA_NB * NTL * TLS;
  static constexpr int total = coarse + NTL * RPT * TMA_XR; // doubles
  static_assert(NTL * RPT <= NT, "one thread per x-pass row");
};

// CTAs per SM that a variant's register allocation must allow: what its open
// z sums (two lines per timelevel) and about 48 other registers leave room
// for, and as many more as the configuration asks beyond that case's 4 of 128
// threads.
template <class F, int NTL, int TK, int CFG> constexpr int tma_blocks() {
  constexpr int line = sizeof(typename F::template Line<0, false>) / 4;
  constexpr int regs = 2 * NTL * line + 48 + (TK == T_ENO ? 16 : 0);
  constexpr int NT = TMA_CFGS[CFG].nt, extra = TMA_CFGS[CFG].mb - 512 / NT;
  constexpr int b = 65536 / (NT * regs) + extra;
  return b < 1 ? 1 : b > 1024 / NT ? 1024 / NT : b;
}

// The TMA kernels' variants: family (VC 1/3/5, CC 0-5, ENO; cell-centred ENO
// 2/3) x time interpolation (one timelevel, linear, quadratic, ENO).  The
// first TV_TUNED have a kernel per tile configuration; the cell-centred ENO
// ones run in TV_FIXED_CFG.
constexpr int TV_TUNED = 40;
constexpr int TV_FAMILIES = 12;
constexpr int TV_COUNT = 4 * TV_FAMILIES;
constexpr int TV_FIXED_CFG = 1;
constexpr int tma_cfg(int variant, int cfg) { return variant < TV_TUNED ? cfg : TV_FIXED_CFG; }
template <class D> __host__ __device__ __forceinline__ int tma_variant(const D &d) {
  int f = -1;
  if (d.kind == K_PROLONG_VC) f = d.order == 1 ? 0 : d.order == 3 ? 1 : d.order == 5 ? 2 : -1;
  else if (d.kind == K_PROLONG_CC) f = d.order >= 0 && d.order <= 5 ? 3 + d.order : -1;
  else if (d.kind == K_PROLONG_ENO) f = 9;
  else if (d.kind == K_PROLONG_CC_ENO) f = d.order == 2 ? 10 : d.order == 3 ? 11 : -1;
  if (f < 0) return -1;
  const int tv = d.ntl == 1 ? 0 : d.ntl == 2 ? 1 : d.tkind == T_ENO ? 3 : 2;
  return 4 * f + tv;
}

// ---------------------------------------------------------------- PTX
__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity) {
  unsigned ok;
  asm volatile("{\n"
               " .reg .pred p;\n"
               " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
               " selp.u32 %0, 1, 0, p;\n"
               "}\n"
               : "=r"(ok)
               : "r"(smem_u32(bar)), "r"(parity)
               : "memory");
  return ok != 0;
}
// Waits for the phase of the given parity; gives up after about 2^31 clock
// cycles (a second) and returns false.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, unsigned parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity))
    if (clock64() - t0 > (1LL << 31)) return false;
  return true;
}
// One box of a 3-d tensor map into shared memory, completing on *bar.
__device__ __forceinline__ void tma_load_3d(double *dst, const CUtensorMap *map, uint64_t *bar, int x, int y,
                                            int z) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
               " [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(smem_u32(dst)),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
               : "memory");
}

// Where a tile lies in its region: first fine point and extent.  y and z
// tiles start at even source positions: the first tile is one point short
// where the region starts at an odd one, and every tile's coarse rows and
// planes serve two fine points each.  x0: start of the x tile (d.xo).
struct TileGeo {
  int f0[3], n[3], x0;
};
__device__ __forceinline__ TileGeo tile_geo(const Desc &d, int tile) {
  const int rr = (int)div_magic((unsigned)tile, d.mg[0], d.sh[0]), tz = (int)div_magic((unsigned)rr, d.mg[1], d.sh[1]);
  const int t[3] = {tile - rr * d.tiles[0], rr - tz * d.tiles[1], tz};
  const int w[3] = {d.xw, 2 * d.ptyc, d.pz}, o[3] = {d.xo, d.soff[1] & 1, d.soff[2] & 1};
  TileGeo g;
  g.x0 = t[0] * w[0] - o[0];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    g.f0[k] = max(0, t[k] * w[k] - o[k]);
    g.n[k] = min((t[k] + 1) * w[k] - o[k] + (k == 0 ? d.xs2 : 0), d.n[k]) - g.f0[k];
  }
  return g;
}

// Staging state of one CTA.  Stages are counted over all its tiles: stage g
// uses slot g % 2, whose mbarrier phase g / 2 completes when it lands.
struct TmaRing {
  uint64_t *bars = nullptr; // TMA_NB mbarriers, arrival count 1
  unsigned g = 0;           // stages of the earlier tiles
  // failure injection for the tests of the bounded waits
  // (cgx_debug_skip_tma_plane): stage 0 is never staged, so that the wait for
  // it runs out
  bool skip = false;
};

// The x pass over one staged row: src is its first point (16-byte aligned),
// which lies xs (0 or 1) points before the window of base 0; writes the two
// fine points of bases 0 .. nbx-1 to dst.  NBX and XS give them as constants
// (NBX = 0: nbx, xs), which leaves out the sums that no base reads: 80
// instead of 120 operations for 8 bases of order 5.
template <class F, int FMA, int NBX, int XS>
__device__ __forceinline__ void x_line(const double *__restrict__ src, double *__restrict__ dst, int xs, int nbx) {
  constexpr int W = F::HI - F::LO, DD = F::D1 - F::D0;
  constexpr int QN = NBX ? (XS + NBX + W + 1) / 2 : tma_bx(PTXMAX / 2 + 1, W) / 2;
  if (NBX) nbx = NBX, xs = XS;
  typename F::template Line<FMA, true> line;
  const int nload = xs + nbx + W;
  double e[2 * QN];
  static_for<QN>([&](auto Q) {
    constexpr int q = decltype(Q)::value;
    if (NBX || 2 * q < nload) { // uniform
      const double2 v = *reinterpret_cast<const double2 *>(src + 2 * q);
      static_for<2>([&](auto K) {
        constexpr int j = 2 * q + decltype(K)::value;
        constexpr Open w{j, XS, NBX ? XS + NBX : 1 << 30};
        if (NBX && j >= XS + NBX + W) return;
        double o1 = 0.0;
        line.template push<j % F::PHASES>(j & 1 ? v.y : v.x, e[j], o1, w);
        // completes base j - W - xs
        if (j >= W && (j > W || xs == 0) && j - W - xs < nbx)
          *reinterpret_cast<double2 *>(dst + 2 * (j - W - xs)) = make_double2(e[j >= W ? j - DD : 0], o1);
      });
    }
  });
}
template <class F, int FMA>
__device__ __forceinline__ void x_row(const double *__restrict__ src, double *__restrict__ dst, int xs, int nbx) {
  constexpr int FULL = PTXMAX / 2;
  if (F::PHASES > 1 && nbx == FULL) { // uniform
    if (xs) x_line<F, FMA, FULL, 1>(src, dst, 1, FULL);
    else x_line<F, FMA, FULL, 0>(src, dst, 0, FULL);
  } else {
    x_line<F, FMA, 0, 0>(src, dst, xs, nbx);
  }
}

// fn(integral_constant<int, phase>()), phase < N uniform over the warp
template <int N, class Fn> __device__ __forceinline__ void by_phase(int phase, Fn &&fn) {
  auto one = [&](auto K) {
    if constexpr ((decltype(K)::value) < N) fn(K);
    else __builtin_unreachable();
  };
  static_assert(N <= 11, "a case per phase");
  switch (phase) {
  case 0: one(std::integral_constant<int, 0>()); break;
  case 1: one(std::integral_constant<int, 1>()); break;
  case 2: one(std::integral_constant<int, 2>()); break;
  case 3: one(std::integral_constant<int, 3>()); break;
  case 4: one(std::integral_constant<int, 4>()); break;
  case 5: one(std::integral_constant<int, 5>()); break;
  case 6: one(std::integral_constant<int, 6>()); break;
  case 7: one(std::integral_constant<int, 7>()); break;
  case 8: one(std::integral_constant<int, 8>()); break;
  case 9: one(std::integral_constant<int, 9>()); break;
  case 10: one(std::integral_constant<int, 10>()); break;
  default: __builtin_unreachable();
  }
}

// One prolongation tile.  Returns false when a wait gave up (the CTA then
// stops; the status word holds CGX_EDEVICE).  TMA: staged by tensor copies
// (maps, ring), else by cp.async from d.src.
template <class F, int FMA, int NTL, int TK, int CFG, bool TMA>
__device__ __forceinline__ bool prolong_tile(const Desc &d, const CUtensorMap *__restrict__ maps, int tile,
                                             double *sm, TmaRing &ring, int *status) {
  using S = TSmem<F, NTL, CFG>;
  constexpr int NT = S::NT, LO = F::LO, HI = F::HI, D0 = F::D0, D1 = F::D1, XR = TMA_XR;
  constexpr int BZS = tma_planes(F::PHASES, NTL); // planes per stage where fixed
  const int tid = threadIdx.x;
  const int BX = d.bx, BY = d.by, BZ = BZS ? BZS : d.bz;
  const TileGeo geo = tile_geo(d, tile);
  const int fx0 = geo.f0[0], nfx = geo.n[0], nfy = geo.n[1], nfz = geo.n[2];
  const int sx0 = d.soff[0] + fx0, sy0 = d.soff[1] + geo.f0[1], sz0 = d.soff[2] + geo.f0[2];
  const int c_first = sx0 >> 1, nbx = ((sx0 + nfx - 1) >> 1) - c_first + 1;
  // the staged boxes start at an even x coordinate (the 16-byte rule)
  const int bx0 = (c_first + LO) & ~1, xs = c_first + LO - bx0;
  const int cy0 = (sy0 >> 1) + LO, cz0 = (sz0 >> 1) + LO;
  // planes: up to the last one an output needs (the parity-0 value of the
  // last point may need one fewer than the parity-1 value)
  const int zlast = sz0 + nfz - 1;
  const int nplanes = ((zlast - (D0 < D1 && !(zlast & 1) ? 1 : 0)) >> 1) + HI - cz0 + 1;
  const int nstages = (nplanes + BZ - 1) / BZ;
  const int rows = BY * BZ; // x-pass rows per timelevel

  double *const coarse = sm;
  double *const xrows = sm + S::coarse;

  // --- staging: stage s (s = 0, 1, ...) into slot (g0 + s) % 2
  const unsigned g0 = ring.g;
  auto issue = [&](int s) { // TMA form: the elected thread
    if (ring.skip && g0 == 0 && s == 0) return; // failure injection
    const unsigned g = g0 + (unsigned)s;
    double *slot = coarse + (g & 1u) * (NTL * S::TLS);
    uint64_t *bar = &ring.bars[g & 1u];
    mbar_expect_tx(bar, (unsigned)(NTL * 8 * BX * rows));
#pragma unroll
    for (int t = 0; t < NTL; ++t) tma_load_3d(slot + t * S::TLS, maps + t, bar, bx0, cy0, cz0 + s * BZ);
  };
  auto fetch = [&](int s) { // all threads: a warp per row, a lane per point
    double *slot = coarse + ((g0 + (unsigned)s) & 1u) * (NTL * S::TLS);
    const int lane = tid & 31, gx = bx0 + lane;
    if (lane < BX)
      for (int r = tid >> 5; r < NTL * rows; r += NT / 32) {
        const int t = (r >= rows) + (NTL > 2 && r >= 2 * rows), q = r - t * rows;
        const int p = q / BY, gy = cy0 + (q - p * BY), gz = cz0 + s * BZ + p;
        double *sp = slot + t * S::TLS + q * BX + lane;
        if (gx >= 0 && gx < d.sext[0] && gy >= 0 && gy < d.sext[1] && gz >= 0 && gz < d.sext[2])
          cp_async8(sp, d.src[t] + gx + gy * d.ssy + gz * d.ssz);
        else
          *sp = 0.0; // never read by a valid output (the host checks the stencils)
      }
  };
  if constexpr (TMA) {
    if (tid == 0) {
      issue(0);
      if (nstages > 1) issue(1);
    }
  } else {
    fetch(0);
    cp_async_commit();
    if (nstages > 1) fetch(1);
    cp_async_commit();
  }

  // --- x pass: thread = (timelevel, plane, row)
  const int xt = (tid >= rows) + (NTL > 2 && tid >= 2 * rows); // timelevel, where tid < NTL * rows
  const double *const xsrc = coarse + xt * S::TLS + (tid - xt * rows) * BX;
  double *const xdst = xrows + tid * XR;

  // --- y/z owner: thread = (fine x, coarse y row) = (tid % ptx, tid / ptx);
  // threads past the ptx * ptyc owners address row ptyc - 1 and store nothing
  const int my_cyr_all = (tid * d.rpx) >> 16, my_fx = tid - my_cyr_all * d.ptx;
  const bool tact = my_cyr_all < d.ptyc;
  const int my_cyr = tact ? my_cyr_all : d.ptyc - 1;
  const bool wact = (((tid & ~31) * d.rpx) >> 16) < d.ptyc; // warp holds an owner
  const int ys0 = 2 * ((sy0 >> 1) + my_cyr);
  const long long dsy = d.dsy, dsz = d.dsz;
  int zs = 2 * (cz0 - D0) - sz0; // parity-0 point of the next plane, from the tile's first
  // what the thread stores: fine row h (of its two) in planes of parity p
  // from zs; with d.xs2, the x tile lies two points further in every other
  // row or plane (the tile 0 rows keep their first points)
  bool vst[2][2];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const int y = geo.f0[1] + ys0 + h - sy0;
      const int sh = (int)((y * dsy + (geo.f0[2] + zs + p) * dsz) & d.xs2); // 0 or 2
      const int x = fx0 + my_fx - geo.x0; // from the x tile's start
      vst[h][p] = tact && my_fx < nfx && ys0 + h >= sy0 && ys0 + h < sy0 + nfy &&
                  (d.xs2 == 0 || ((geo.x0 <= 0 || x >= sh) && x < d.xw + sh));
    }
  const double *const ycol = xrows + (my_cyr - LO) * XR + my_fx + (sx0 & 1);
  double w[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) w[k] = (NTL == 1 || (TK != T_ENO && k >= NTL)) ? 0.0 : d.w[k];
  typename F::template Line<FMA, false> zl[NTL][2];
  // store address of the parity-0 point of plane cz (base cz - D0), and from
  // there to the parity-1 point that the same plane completes (base cz - D1)
  double *oz = d.dst + (d.doff[0] + fx0 + my_fx) + (long long)(d.doff[1] + geo.f0[1] + ys0 - sy0) * dsy +
               (long long)(d.doff[2] + geo.f0[2] + zs) * dsz;
  constexpr int ODD = 1 - 2 * (D1 - D0);
  const long long odd = ODD * dsz;
  const double *col = nullptr; // of the next plane
  auto plane = [&](auto U) {   // y and z passes of a plane, U its phase
    const bool z0 = zs >= 0 && zs < nfz, z1 = zs + ODD >= 0 && zs + ODD < nfz;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      double e[NTL], o[NTL];
#pragma unroll
      for (int t = 0; t < NTL; ++t) {
        const double *c = col + t * (rows * XR);
        zl[t][h].template push<decltype(U)::value>(F::template next<FMA>(h, [&](int m) { return c[m * XR]; }), e[t],
                                                   o[t]);
      }
      const double r0 = tcombine<FMA, TK, NTL>(w, e), r1 = tcombine<FMA, TK, NTL>(w, o);
      double *const oh = h ? oz + dsy : oz;
      if (z0 && vst[h][0]) *oh = r0;
      if (z1 && vst[h][1]) oh[odd] = r1;
    }
    col += BY * XR;
    oz += 2 * dsz;
    zs += 2;
  };
  int phase = 0; // of the z lines' next push
  for (int s = 0; s < nstages; ++s) {
    const unsigned slot = (g0 + (unsigned)s) & 1u;
    const int np = min(BZ, nplanes - s * BZ);
    bool ok = true;
    if constexpr (TMA) {
      ok = mbar_wait_bounded(&ring.bars[slot], ((g0 + (unsigned)s) >> 1) & 1u);
    } else {
      cp_async_wait<1>();
      __syncthreads();
    }
    if (ok && tid < (NTL == 1 ? np * BY : NTL * rows)) x_row<F, FMA>(xsrc + slot * (NTL * S::TLS), xdst, xs, nbx);
    if constexpr (TMA) {
      if (__syncthreads_or(!ok)) { // a wait gave up
        // wait (bounded) for the next stage too, which is still in flight,
        // so that no copy lands after the CTA has left
        if (tid == 0) {
          if (status) atomicCAS(status, 0, CGX_EDEVICE);
          const unsigned g = g0 + (unsigned)s + 1u;
          if (s + 1 < nstages) mbar_wait_bounded(&ring.bars[g & 1u], (g >> 1) & 1u);
          if (!(ring.skip && g == 1u)) mbar_wait_bounded(&ring.bars[slot], ((g - 1u) >> 1) & 1u);
        }
        __syncthreads();
        return false;
      }
      if (tid == 0 && s + 2 < nstages) issue(s + 2);
    } else {
      __syncthreads();
      if (s + 2 < nstages) fetch(s + 2);
      cp_async_commit();
    }
    if (wact) { // warp-uniform
      col = ycol;
      if constexpr (BZS > 0) { // whole turns of the phases
        static_for<BZS>([&](auto P) {
          if ((decltype(P)::value) < np) plane(std::integral_constant<int, decltype(P)::value % F::PHASES>());
        });
      } else {
#pragma unroll 1
        for (int p = 0; p < np; ++p) {
          by_phase<F::PHASES>(phase, plane);
          if (++phase == F::PHASES) phase = 0;
        }
      }
    }
    if (TMA && s + 1 < nstages) __syncthreads(); // the x-pass rows are free
  }
  ring.g = g0 + (unsigned)nstages;
  if constexpr (!TMA) cp_async_wait<0>();
  __syncthreads(); // shared memory free for the next tile
  return true;
}

} // namespace cgx
