// The mixed (FP32) pressure-correction V-cycle's passes on its large levels, by
// runs of four cells.
//
// The per-cell passes (hs_mg.cuh) issue 13 scalar loads at a stride of two
// cells per update; on a large FP32 level those loads, not its bytes, set the
// time (a half-sweep of 256x128x128 alone: 21.5 us, its 101 MB at the copy
// rate 15.4 us).  Here a thread owns a column of 16-byte runs and marches a
// few planes in z: the z neighbours stay in registers, every load and store
// of an array is 16 bytes, and the two x neighbours past the run's ends are
// scalar loads that hit L1: 13.2 us.  p' solve per outer step, per-cell passes
// -> runs in one build: 256x128x128 3.16 -> 2.90 ms, 512x256x256 21.1 -> 17.3,
// 203x75x110 2.30 -> 2.22, 131x200x180 14.8 -> 14.3.  An FP64 half-sweep is bound by DRAM either way (201 MB at
// 256x128x128: 40 us per cell, 42 us by runs of two), so FP64 keeps the
// per-cell passes.  Every point update is the per-cell pass's expression term
// for term, so a level's x is theirs bit for bit.
#pragma once
#include "hs_mg.cuh"

namespace hs {
namespace run {

namespace cg = cooperative_groups;

using M = float;                 // the value type: the FP64 passes stay per cell
constexpr int W = 4, H = W / 2;  // cells of a run (16 bytes), its cells of one colour
struct Run {
  M v[W];
};
__device__ __forceinline__ Run ld(const M *p) {
  const float4 t = *reinterpret_cast<const float4 *>(p);
  return {{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ void st(M *p, const Run &r) {
  *reinterpret_cast<float4 *>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
}
// value 2 b + odd of a run; the one before and after it (l, r: the values beyond the run's ends)
__device__ __forceinline__ M sel(const Run &x, int b, int odd) {
  return odd ? x.v[2 * b + 1] : x.v[2 * b];
}
__device__ __forceinline__ M before(const Run &x, int b, int odd, M l) {
  return odd ? x.v[2 * b] : (b > 0 ? x.v[b > 0 ? 2 * b - 1 : 0] : l);
}
__device__ __forceinline__ M after(const Run &x, int b, int odd, M r) {
  return odd ? (2 * b + 2 < W ? x.v[2 * b + 2 < W ? 2 * b + 2 : 0] : r) : x.v[2 * b + 1];
}

struct Warps {
  int id, n;  // this warp, warps of the grid
};

enum { kSmooth = 0, kProlong = 1 };

// One half-sweep of colour c of level F (KIND kProlong: with the prolongation
// from C fused, as mg::prolong_smooth), in units of 32 runs x zc planes
template <int KIND>
__device__ __forceinline__ void sweep(const mg::Level<M> &F, const mg::Level<M> &C, int c, int zc,
                                      const Warps &wk) {
  const int PX = F.px, PXY = F.px * (F.ny + 2), RP = F.px / W, np = RP * F.ny;
  const int nwc = (np + 31) / 32, units = nwc * ((F.nz + zc - 1) / zc);
  const int CPX = C.px, CPXY = C.px * (C.ny + 2);
  for (int u = wk.id; u < units; u += wk.n) {
    const int z = u / nwc, e = (u - z * nwc) * 32 + (threadIdx.x & 31);
    if (e >= np) continue;
    const int j = e / RP, m = e - j * RP, i0 = W * m - 1;  // i0: the run's first cell
    const int k0 = z * zc, k1 = min(F.nz, k0 + zc);
    int q = W * m + PX * ((j + 1) + (F.ny + 2) * (k0 + 1));
    Run xm = ld(F.x + q - PXY), xc = ld(F.x + q), bl = ld(F.gz + q);
    for (int k = k0; k < k1; ++k, q += PXY) {
      const Run xp = ld(F.x + q + PXY), xs = ld(F.x + q - PX), xn = ld(F.x + q + PX);
      const M xl = F.x[q - 1], xr = F.x[q + W];
      const Run gx = ld(F.gx + q), gs = ld(F.gy + q), gn = ld(F.gy + q + PX), bh = ld(F.gz + q + PXY),
                rh = ld(F.rhs + q);
      const M gr = F.gx[q + W];
      const int pa = (i0 + j + k + c) & 1;  // the run's first cell of colour c
      Run o = xc;
#pragma unroll
      for (int b = 0; b < H; ++b) {
        const int i = i0 + 2 * b + pa;
        const bool in = i >= 0 && i < F.nx;
        M xw = before(xc, b, pa, xl), xe = after(xc, b, pa, xr), vs = sel(xs, b, pa), vn = sel(xn, b, pa),
          vb = sel(xm, b, pa), vf = sel(xp, b, pa);
        if constexpr (KIND == kProlong) {
          // neighbours x + x_coarse(parent), as mg::prolong_smooth
          const int qc = in ? mg::idx(C, (i >> 1) + 1, (j >> 1) + 1, (k >> 1) + 1) : mg::idx(C, 1, 1, 1);
          const M cp = C.x[qc], cx = C.x[(i & 1) ? qc + 1 : qc - 1], cy = C.x[(j & 1) ? qc + CPX : qc - CPX],
                  cz = C.x[(k & 1) ? qc + CPXY : qc - CPXY];
          xw = i > 0 ? xw + ((i & 1) ? cp : cx) : M(0);
          xe = i + 1 < F.nx ? xe + ((i & 1) ? cx : cp) : M(0);
          vs = j > 0 ? vs + ((j & 1) ? cp : cy) : M(0);
          vn = j + 1 < F.ny ? vn + ((j & 1) ? cy : cp) : M(0);
          vb = k > 0 ? vb + ((k & 1) ? cp : cz) : M(0);
          vf = k + 1 < F.nz ? vf + ((k & 1) ? cz : cp) : M(0);
        }
        const M gl = sel(gx, b, pa), gh = after(gx, b, pa, gr), sl = sel(gs, b, pa), sh = sel(gn, b, pa);
        const M zl = sel(bl, b, pa), zh = sel(bh, b, pa);
        M d = M(0);
        d += gl + gh;
        d += sl + sh;
        d += zl + zh;
        const M off = gl * xw + gh * xe + sl * vs + sh * vn + zl * vb + zh * vf;
        const M s = sel(rh, b, pa) + off;
        const M v = d == M(0) ? M(0) : s / d;
        if (in) {
          o.v[2 * b] = pa ? o.v[2 * b] : v;
          o.v[2 * b + 1] = pa ? v : o.v[2 * b + 1];
        }
      }
      st(F.x + q, o);
      xm = xc;
      xc = xp;
      bl = bh;
    }
  }
}

// The residuals of a run's colour-0 cells in row j, plane k, one per pair of
// values; 0 outside the level
__device__ __forceinline__ void residuals(const mg::Level<M> &F, int m, int j, int k, M (&res)[H]) {
  const int PX = F.px, PXY = F.px * (F.ny + 2);
  const bool ok = j < F.ny && k < F.nz;
  const int q = ok ? W * m + PX * ((j + 1) + (F.ny + 2) * (k + 1)) : PXY + PX;
  const Run xc = ld(F.x + q), xs = ld(F.x + q - PX), xn = ld(F.x + q + PX), xm = ld(F.x + q - PXY),
            xp = ld(F.x + q + PXY);
  const M xl = F.x[q - 1], xr = F.x[q + W];
  const Run gx = ld(F.gx + q), gs = ld(F.gy + q), gn = ld(F.gy + q + PX), bl = ld(F.gz + q), bh = ld(F.gz + q + PXY),
            rh = ld(F.rhs + q);
  const M gr = F.gx[q + W];
  const int i0 = W * m - 1, pa = (i0 + j + k) & 1;
#pragma unroll
  for (int b = 0; b < H; ++b) {
    const int i = i0 + 2 * b + pa;
    const M gl = sel(gx, b, pa), gh = after(gx, b, pa, gr), sl = sel(gs, b, pa), sh = sel(gn, b, pa);
    const M zl = sel(bl, b, pa), zh = sel(bh, b, pa);
    M d = M(0);
    d += gl + gh;
    d += sl + sh;
    d += zl + zh;
    const M off = gl * before(xc, b, pa, xl) + gh * after(xc, b, pa, xr) + sl * sel(xs, b, pa) + sh * sel(xn, b, pa) +
                  zl * sel(xm, b, pa) + zh * sel(xp, b, pa);
    const M v = sel(rh, b, pa) - (d * sel(xc, b, pa) - off);
    res[b] = ok && i >= 0 && i < F.nx ? v : M(0);
  }
}

// The restriction (mg::restrict_res: the colour-0
// children's residuals in (dk, dj) order, and the coarse seed).  A lane takes
// one fine run of a coarse row; its coarse cells begin at the odd values of
// the run, so the last one's second children are the next lane's.
__device__ __forceinline__ void restrict_level(const mg::Level<M> &F, const mg::Level<M> &C, const Warps &wk) {
  const int RP = F.px / W, np = RP * C.ny, nwc = (np + 30) / 31, units = nwc * C.nz;
  const int lane = threadIdx.x & 31;
  for (int u = wk.id; u < units; u += wk.n) {
    const int z = u / nwc, e = min((u - z * nwc) * 31 + lane, np - 1), K = z;
    const int J = e / RP, m = e - J * RP;
    const bool own = lane < 31 && (u - z * nwc) * 31 + lane < np;
    M acc[H], v[H];
    residuals(F, m, 2 * J, 2 * K, v);
#pragma unroll
    for (int b = 0; b < H; ++b) {
      acc[b] = M(0);
      acc[b] += v[b];
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      residuals(F, m, s ? 2 * J : 2 * J + 1, s ? 2 * K + 1 : 2 * K, v);
      const M nx_ = __shfl_down_sync(0xffffffffu, v[0], 1);
#pragma unroll
      for (int b = 0; b < H; ++b) acc[b] += b + 1 < H ? v[b + 1 < H ? b + 1 : 0] : nx_;
    }
    residuals(F, m, 2 * J + 1, 2 * K + 1, v);
#pragma unroll
    for (int b = 0; b < H; ++b) {
      acc[b] += v[b];
      const int I = H * m + b;
      if (!own || 2 * I >= F.nx) continue;
      const int qc = mg::idx(C, I + 1, J + 1, K + 1);
      mg::seed_store(C, qc, I, J, K, mg::unknown(C, qc) ? acc[b] : M(0), mg::seed_diag(C, qc, I, J, K, false));
    }
  }
}

// Planes a thread marches per unit on level L with nw warps: the fewest
// rounds of (planes + 1 to start a march), at most 6.  Longer marches spread
// the warps over more of the level at a time; what that costs or gains is
// small (ms per p' solve with up to 4 / 6 / 16 planes): 203x75x110 2.31 / 2.22
// / 2.22, 256x128x128 2.88 / 2.90 / 2.84, 131x200x180 14.6 / 14.3 / 13.9,
// 512x256x256 17.5 / 17.3 / 17.2
inline int pick_planes(const mg::Level<M> &L, int nw) {
  const long long nwc = ((long long)L.px / W * L.ny + 31) / 32;
  int best = 1;
  long long cost = -1;
  for (int z = 1; z <= 6; ++z) {
    const long long c = (nwc * ((L.nz + z - 1) / z) + nw - 1) / nw * (z + 1);
    if (cost < 0 || c < cost) { cost = c; best = z; }
  }
  return best;
}

// The V-cycle of mg::vcycle with levels 0..G.nrun - 1 (none of them handled by
// block 0 alone) in run passes
template <bool RO>
__device__ __forceinline__ void vcycle(const mg::Hier<M> &G, cg::grid_group &grid, int tid, int T) {
  const int nwb = blockDim.x >> 5;
  const Warps wk{(int)(blockIdx.x * nwb + (threadIdx.x >> 5)), (int)gridDim.x * nwb};
  for (int l = 0; l < G.nrun; ++l) {
    const mg::Level<M> &F = G.lv[l], &C = G.lv[l + 1];
    const int np = 2 * (l == 0 ? G.nsw : G.nswc) - 1;  // half-sweeps of colours 1, 0, 1, ...
    for (int s = 0; s < np; ++s) {
      sweep<kSmooth>(F, C, (s & 1) ^ 1, G.zc[l], wk);
      grid.sync();
    }
    restrict_level(F, C, wk);
    grid.sync();
  }
  mg::vcycle<M, double, RO>(G, false, grid, tid, T, nullptr, nullptr, G.nrun);
  for (int l = G.nrun - 1; l >= 0; --l) {
    const mg::Level<M> &F = G.lv[l], &C = G.lv[l + 1];
    const int np = 2 * (l == 0 ? G.nsw : G.nswc) - 1;  // half-sweeps 0, 1, ..., 0 after the prolongation's
    sweep<kProlong>(F, C, 1, G.zc[l], wk);
    grid.sync();
    for (int s = 0; s < np; ++s) {
      sweep<kSmooth>(F, C, s & 1, G.zc[l], wk);
      grid.sync();
    }
  }
}

}  // namespace run
}  // namespace hs
