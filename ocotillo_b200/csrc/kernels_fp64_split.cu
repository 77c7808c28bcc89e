/* kernels_fp64_split.cu -- the split FP64 block solve: few items, grey transfer (see kernels_fp64.cu). */
#include "fp64_block.h"

namespace oco {

/* ---- the split block solve ------------------------------------------------------------- */
/* With few items the persistent kernels leave most of the GPU idle while each warp walks its column
 * alone (2 us per level and warp, whatever the number of warps: 16 columns x 500 x 250 took 1.03
 * ms, 0.45 ms after the sweep's own changes).  Here everything that is independent along z runs
 * first, parallel over (warp tile, RZ levels): k_rows writes the rows' coefficients; k_chain then
 * runs the recurrences, one warp per tile, with nothing but them on its serial chain: 0.23 ms for
 * those 16 columns.  That moves ~180 B per point instead of ~75, so it is taken while there are at
 * most two tiles per SM (solve_is_split; a full wave of the persistent kernel holds 16).  Split and
 * persistent solve, plain, tiles of 32 wavelengths x levels: 64 x 512 0.17 and 0.36 ms, 296 x 512 0.35 and
 * 0.41 ms, 592 x 512 0.55 and 0.45 ms; 64 x 128 83 and 110 us, 296 x 128 112 and 110 us.  Columns
 * of 12 to 48 levels gain little or nothing (64 x 48 56 and 52-64 us, 64 x 16 48 and 32-43 us), shorter ones
 * lose (SPLIT_MIN_NZ).
 * Grey transfer takes it always: it has one wavelength per column (few items) and no opacity sums, and
 * reads rho and T directly instead of a 208-byte record per cell (16,384 columns x 512: 1.08 -> 0.41 ms).
 * Per point the operations are solve_item's, so the same bits. */
/* One cell of a grey column (grey_parameters, continuous_opacity.f90:377-390); the factors of an
 * unchanged temperature are kept. */
struct GreyCell {
  double t, p35, S;
};
template <bool STABLE>
__device__ __forceinline__ Opac opacity_grey_cell(double r, double t, double sg, bool fresh, GreyCell &k) {
  if (fresh || !same_bits(t, k.t)) {
    const double t2 = t * t;
    k.t = t;
    k.S = sigma_sb * (t2 * t2);
    k.p35 = 3.68e22 * oco_pow(t, -3.5);
  }
  const double alpha = k.p35 * r, tot = alpha + sg;
  Opac o;
  o.op = tot * r;
  o.S = k.S;
  o.num = STABLE ? alpha : sg;
  o.kr = tot;
  const double q = div_quot(o.num, tot, div_recip(tot));
  o.w = STABLE ? q : 1.0 - q;
  o.wok = div_b_ok(tot) & div_a_ok(o.num);
  o.ook = op_ok(o.op);
  return o;
}

/* The item of a lane: by_tile, wavelength tile*32 + lane of the tile's column, otherwise item
 * tile*32 + lane of the flattened list; lanes past the end repeat the last. */
__device__ __forceinline__ bool split_item(const SolveArgs &a, bool by_tile, int64_t t, int64_t &cl, int &iw) {
  const int lane = threadIdx.x & 31;
  if (by_tile) {
    const int ntiles = (a.nw + 31) / 32;
    cl = t / ntiles;
    iw = (int)(t - cl * ntiles) * 32 + lane;
    const bool on = iw < a.nw;
    if (!on) iw = a.nw - 1;
    return on;
  }
  const int64_t n = a.ncol * a.nw, i = t * 32 + lane, item = i < n ? i : n - 1;
  cl = item / a.nw;
  iw = (int)(item - cl * a.nw);
  return i < n;
}

/* Coefficient arrays of the tiles: [tile][z][32], in this order after one another; at level z0 of
 * tile t. */
struct SplitRows {
  double *aa, *xx, *cc, *dd, *kap; /* xx: diagonal (plain), its excess (stable); kap as the sweep's scratch */
  __device__ __forceinline__ SplitRows(const SolveArgs &a, int64_t tiles, int64_t t, int z0) {
    const int64_t plane = tiles * 32 * a.nz;
    aa = a.gam + t * 32 * a.nz + tile_level(z0) + (threadIdx.x & 31);
    xx = aa + plane;
    cc = xx + plane;
    dd = cc + plane;
    kap = dd + plane;
  }
};

/* by_tile: see split_item (never for grey transfer); ring: k_chain's outputs go through the ring, kappa among
 * them (both uniform, so not worth code of their own: a process pays for loading each variant at its
 * first solve). */
template <int FORM, bool GREY>
__global__ void __launch_bounds__(128, 4) k_rows(const SolveArgs a, int64_t tiles, bool by_tile, bool ring,
                                                 const ChunkInit init) {
  chunk_init(init, blockIdx.x * (int64_t)blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
  const int nch = (a.nz + RZ - 1) / RZ;
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= tiles * nch) return;
  const int64_t t = w / nch;
  const int nz = a.nz, z0 = (int)(w - t * nch) * RZ, z1 = min(z0 + RZ, nz);
  int64_t cl;
  int iw;
  const bool active = split_item(a, !GREY && by_tile, t, cl, iw);
  const BlockItem it{a, cl, iw};
  const LamR L(it, nullptr, !GREY);
  TCacheR tc;
  GreyCell gc;
  const SplitRows S(a, tiles, t, z0);
  const int zf = max(z0 - 1, 0); /* first level computed */
  auto opac = [&](int z) -> Opac {
    Opac o;
    if constexpr (GREY)
      o = opacity_grey_cell<FORM == 1>(__ldg(a.rho + cl * nz + z), __ldg(a.T + cl * nz + z), a.sigma_grey, z == zf, gc);
    else
      o = opacity_at<FORM == 1>(GlobalRec{a.pil + (cl * (int64_t)nz + z) * NF}, L, tc, z == zf);
    settle_opac<FORM == 1>(o);
    return o;
  };
  const double dz = a.dz, dz2 = a.dz2;
  double *Kb = ring || !active ? nullptr : it.K();
  const int64_t kz = it.kz();
  double kh = 1.0, yk = 1.0; /* mean opacity below the level */
  int okk = 0;
  Opac cur = opac(zf);
  auto mean = [&](const Opac &lo, const Opac &hi) {
    kh = 0.5 * (hi.op + lo.op);
    yk = div_recip(kh);
    okk = lo.ook & hi.ook & div_b_frac_ok(kh);
  };
  if (z0 > 0) {
    const Opac up = opac(z0);
    mean(cur, up);
    cur = up;
  }
  for (int j = z0; j < z1; j++) {
    const int i = (j - z0) * 32;
    const double op = cur.op, o2 = op * op;
    double o1 = div_recip(op);
    if (!cur.ook) o1 = div_call(1.0, op);
    Opac nxt{};
    if (j == 0 || j == nz - 1) { /* fill_boundary_coeffs :187-197 */
      const double zt = ((op * dz2) * cur.w) * 0.25;
      S.dd[i] = -((cur.S * zt) * o2);
      S.xx[i] = FORM == 0 ? -(((o1 + dz) + zt) * o2) : (dz + zt) * o2;
      S.aa[i] = op; /* row 0: unused */
      S.cc[i] = j == 0 ? op : 0.0;
      if (j == 0) {
        nxt = opac(1);
        mean(cur, nxt);
      }
    } else { /* fill_center_coeffs :159-165 */
      nxt = opac(j + 1);
      double aa = div_quot(o2, kh, yk);
      if (!okk) aa = div_call(o2, kh);
      mean(cur, nxt);
      double cc = div_quot(o2, kh, yk);
      if (!okk) cc = div_call(o2, kh);
      const double z3 = (dz2 * (op * (op * op))) * cur.w;
      S.aa[i] = aa;
      S.cc[i] = cc;
      S.xx[i] = FORM == 0 ? -((aa + cc) + z3) : z3;
      S.dd[i] = -(cur.S * z3);
    }
    S.kap[i] = ring ? op : o1;
    if (Kb) __stcs(&Kb[j * kz], op);
    cur = nxt;
  }
}

/* One warp per block, so that the tiles spread over the SMs.  TILE: by_tile of k_rows (as an argument it
 * costs the shortest solves 2 of 45 us: 4 columns x 16 levels x 32 wavelengths). */
template <int FORM, bool RING, bool TILE>
__global__ void __launch_bounds__(32) k_chain(const SolveArgs a, int64_t tiles) {
  __shared__ RingSmem<double> s_ring[1];
  const int64_t t = blockIdx.x;
  const int nz = a.nz;
  int64_t cl;
  int iw;
  const bool active = split_item(a, TILE, t, cl, iw);
  const BlockItem it{a, cl, iw};
  const SplitRows S(a, tiles, t, 0);
  bool bad = false;
  Chain e = chain_first<FORM>(S.xx[0], S.cc[0], S.dd[0], bad);
  S.dd[0] = e.u;
  auto step = [&](int j, double aa, double xx, double cc, double dd) {
    double g, q;
    chain_step<FORM>(e, aa, xx, cc, dd, g, q, bad);
    S.aa[tile_level(j)] = g;
    S.dd[tile_level(j)] = e.u;
    if (FORM == 1) S.xx[tile_level(j - 1)] = q; /* q_{j-1} over the excess of row j - 1 */
  };
  constexpr int G = RG_ALONE;
  struct Row {
    double a, x, c, d;
  } A[G], B[G];
  auto load = [&](Row *l, int j0) {
#pragma unroll
    for (int i = 0; i < G; i++) {
      const int64_t k = tile_level(min(j0 + i, nz - 1));
      l[i] = Row{S.aa[k], S.xx[k], S.cc[k], S.dd[k]};
    }
  };
  auto steps = [&](const Row *l, int j0) {
#pragma unroll
    for (int i = 0; i < G; i++) step(j0 + i, l[i].a, l[i].x, l[i].c, l[i].d);
  };
  int j = 1;
  load(A, 1);
#pragma unroll 1
  for (; j + 2 * G <= nz; j += 2 * G) {
    load(B, j + G);
    steps(A, j);
    load(A, j + 2 * G);
    steps(B, j + G);
  }
  Row x = A[0];
#pragma unroll 1
  for (; j < nz; j++) { /* one level loaded ahead */
    const int64_t k = tile_level(min(j + 1, nz - 1));
    const Row nx{S.aa[k], S.xx[k], S.cc[k], S.dd[k]};
    step(j, x.a, x.x, x.c, x.d);
    x = nx;
  }
  if (active && bad) {
    atomicAdd(&it.status()[0], 1ull);
    atomicMin(&it.status()[1], it.id());
  }
  __syncwarp();
  auto st = make_stores<RING ? ST_RING : ST_LANE, TILE, false>(out_ptrs(it), active, s_ring);
  solve_reverse<FORM, RG_ALONE>(it, active, e.u, S.aa, S.dd, S.kap, S.xx, st);
}

/* Outputs with z fastest from this size on go through the ring, which the single warps of k_chain wait for
 * but which writes whole runs; below it L2 joins the lanes' own stores into lines.  Which is better turns on
 * the number of tiles and the shape as much as on the size (ring / lanes, us): 16 columns x 500 x 250, 48 MB,
 * 330 / 230; grey columns x levels: 4096 x 512, 50 MB, 323 / 194; 16,384 x 512, 201 MB, 441 / 415; 25,600 x
 * 512, 315 MB, 546 / 640; 16,384 x 1024, 403 MB, 839 / 788; 65,536 x 1024, 1.6 GB, 2384 / 3104; 296 columns
 * x 32 wavelengths x 1024 levels, 233 MB, 714 / 794, x 2048 1373 / 1891; but 37 x 250 x 2048, 455 MB, 1445 /
 * 1189, and 1880 x 5 x 2048, 462 MB, 2227 / 1852. */
constexpr int64_t SPLIT_RING_BYTES = 256ll << 20;

template <int FORM, bool TILE>
static cudaError_t launch_chain(const SolveArgs &a, int64_t tiles, bool ring, cudaStream_t s) {
  if (ring)
    k_chain<FORM, true, TILE><<<(unsigned)tiles, 32, 0, s>>>(a, tiles);
  else
    k_chain<FORM, false, TILE><<<(unsigned)tiles, 32, 0, s>>>(a, tiles);
  return cudaGetLastError();
}
/* init: set up by k_rows where no record kernel comes before it (grey). */
template <int FORM>
static cudaError_t split_launch(const SolveArgs &a, int grey, const ChunkInit &init, cudaStream_t s) {
  const bool by_tile = !grey && split_by_tile(a.nw);
  const int64_t tiles = split_tiles(a.ncol, a.nw);
  const bool ring = a.layout == 0 && tiles * 32 * (int64_t)a.nz * 24 > SPLIT_RING_BYTES;
  const unsigned blocks = (unsigned)split_row_blocks(tiles, a.nz);
  if (grey)
    k_rows<FORM, true><<<blocks, 128, 0, s>>>(a, tiles, by_tile, ring, init);
  else
    k_rows<FORM, false><<<blocks, 128, 0, s>>>(a, tiles, by_tile, ring, init);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return by_tile ? launch_chain<FORM, true>(a, tiles, ring, s) : launch_chain<FORM, false>(a, tiles, ring, s);
}
cudaError_t launch_solve_split(const SolveArgs &a, int form, int grey, const ChunkInit &init, cudaStream_t s) {
  return form == 0 ? split_launch<0>(a, grey, init, s) : split_launch<1>(a, grey, init, s);
}

}  // namespace oco
