// CG on tiles of a box, the vectors on chip (sm_100a): FP64 CG of 7-point
// stencils on a box whose diagonals each hold one value, every entry of the box
// present (CsrDev::dia_box 2, dia_cst: Poisson) and every value finite, above the
// size whose values fit on chip (k_cg_chip, about 600K rows), where a tile fits
// (tile_shape: 1,440 rows of a plane, 1,920 of a face in y, 32 rows per thread and p
// in shared memory at most). That is cubes up to 128^3 and about three of four boxes
// of random edges (20 to 260) between 606K and 2.4M rows; the others, 130 x 127 x
// 129 or lines of 1,200 rows, take k_cg_onchip.
//
// A CTA owns a tile of by x bz whole lines of the box (k_cg_chip's tiles):
// p of its rows and of the lines around them in shared memory, each line
// followed by a zero (so the +-1 terms at its ends are zeros), r and x in
// tensor memory, q = A p in registers between the two grid sums of an
// iteration. A thread takes the rows of its columns (x, y) = t, t + 512, ... of
// the tile in blocks of 8 planes, so a row's place in p is the last one's plus a
// constant and p[z - 1], p[z] stay in registers. The rows of a block are computed
// without branches, those past the tile's last plane on its place and then
// dropped: with a branch per row the FP64 chains of a product run one after
// another (128^3: 13,400 clocks per product, without 10,000). An iteration executes
// 123 instructions per row. (Rows t + 512 j with their places computed one by one:
// 156, of which 120 were index arithmetic.)
// k_cg_onchip's runs of consecutive rows read two planes of p through L2 per
// product (128^3: 32,768 rows for a CTA's 14,176); a tile reads the 2 (by + bz)
// lines of its faces (8 x 15 lines: 5,888 rows for 15,360) once, into shared memory.
//
// r crosses between CTAs in the shadow of the (r, r) sum: the rows in another
// CTA's halo are stored to R, then (behind the barrier of the sum's post) a
// thread of warp 1 releases the CTA's flag, acquires the neighbours' and lets
// warps 1 .. 15 load the halo; warp 0 meanwhile waits for the sum. Tags with
// every value, as k_cg_chip has, cost 50-60 clocks per warp access (an earlier form
// of this kernel at 128^3, tiles of 10 x 12 lines: 22.8 us per iteration with tags,
// 20.9 with flags), and flags acquired by all 16 warps more still: the polls of 148
// CTAs delay the stores.
//
// The matrix is the kernel's parameters: an iteration moves nothing but the
// halo. (The same kernel with the values of other matrices read from L2 in every
// product was slower than k_cg_onchip: log-normal 128^3 42 against 36 us per
// iteration, FP32 inner CG 160^3 55 against 26: 512 threads keep too few bytes in
// flight.) Element operations and the order of a row's terms are k_cg_onchip's;
// an absent entry's term is a zero added to a sum that starts at +0.
//
// What bounds an iteration: shared memory (5 reads of 8 bytes per row in A, 1 and
// 2 in the updates: 128^3, 15,360 rows per CTA, 7,700 of 30,700 clocks), the FP64
// pipe (19 % busy) and its latency, and the two grid sums (3,200 each). Measured, us
// per iteration, k_cg_onchip / k_cg_tile: 100^3 20.9 / 10.6, 128^3 35.7 (26.3 with
// the diagonals as parameters) / 15.6. Where a block's loads in p = beta p + r were not
// issued before its stores: 128^3 16.8.
#pragma once

#include "ks_chip_cg.cuh"

namespace ks {

// k / d = quot(k, magic(d)) for k, d < 2^16 (d = 1: 2^32 does not fit).
__device__ __forceinline__ unsigned tile_magic(int d) { return d > 1 ? 0xffffffffu / (unsigned)d + 1u : 0u; }
__device__ __forceinline__ int tile_quot(int k, unsigned m) { return m ? (int)__umulhi((unsigned)k, m) : k; }

// The tile of one CTA.
struct TileRows {
  int nx, ty, tz, plane, row0, up, lp, zp, gy;  // up: rows of a plane of the box; lp, zp: a line's and a plane's pitch in p
  int nb, blocks;  // blocks of a column, of a thread
  unsigned m_nx;
  bool y0, y1, z0, z1;  // faces with a neighbour
  __device__ __forceinline__ explicit TileRows(const ChipArgs &a) {
    const int cy = blockIdx.x % a.gy, cz = blockIdx.x / a.gy;
    gy = a.gy;
    nx = a.nx;
    ty = min(a.by, a.ny - cy * a.by);
    tz = min(a.bz, a.nz - cz * a.bz);
    plane = nx * ty;
    up = nx * a.ny;
    row0 = cy * a.by * nx + cz * a.bz * up;
    lp = nx + 1;
    zp = lp * (ty + 2);
    m_nx = tile_magic(nx);
    nb = (tz + 7) / 8;
    blocks = (plane + kChipThreads - 1) / kChipThreads * nb;
    y0 = cy > 0;
    y1 = cy * a.by + ty < a.ny;
    z0 = cz > 0;
    z1 = cz * a.bz + tz < a.nz;
  }
  __device__ __forceinline__ int cta(int i) const {  // the neighbours, i < 4 (-1: none)
    const int b = blockIdx.x;
    return i == 0 ? (y0 ? b - 1 : -1) : i == 1 ? (y1 ? b + 1 : -1) : i == 2 ? (z0 ? b - gy : -1) : (z1 ? b + gy : -1);
  }
};

constexpr int kTileChunk = 8;  // rows of a block: one TMEM access

// Block c of a thread's rows: planes z0 .. z0 + 7 (those below tz) of one of its
// columns. pos, row: place in p and row in the matrix of plane z0; in: the
// column exists (else that of the tile's first row, never stored); face: it lies
// in a neighbour's halo through its y.
struct TileBlock {
  int z0, pos, row;
  bool in, face;
  __device__ __forceinline__ TileBlock(const TileRows &R, int c) {
    const int s = c / R.nb;
    z0 = kTileChunk * (c - s * R.nb);
    int col = threadIdx.x + kChipThreads * s;
    // opaque: the compiler otherwise computes every block's place once, before
    // the iterations, and spills them all
    asm volatile("" : "+r"(col));
    in = col < R.plane;
    col = in ? col : 0;
    const int y = tile_quot(col, R.m_nx);
    pos = 1 + col + y + R.lp + R.zp * (z0 + 1);
    row = R.row0 + col + R.up * z0;
    face = in && ((R.y0 && y == 0) || (R.y1 && y == R.ty - 1));
  }
};

__device__ __forceinline__ void tile_halo_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kTileHaloThreads) : "memory"); }

struct TileDiag {  // the diagonals' values
  double v[7];
};

__global__ void __launch_bounds__(kChipThreads, 1)
    k_cg_tile(const __grid_constant__ ChipArgs a, const __grid_constant__ TileDiag D) {
  constexpr int RJ = kTileRows, C = kTileChunk, HZ = kTileHaloZ, HY = kTileHaloY;
  using CV = ChipVals<double, C>;
  extern __shared__ __align__(16) unsigned char ir_smem_raw[];
  __shared__ uint32_t s_tmem;
  __shared__ ChipScalars S;
  const int t = threadIdx.x;
  DevState *st = a.st;
  // as k_cg_onchip: the same value in every CTA, so all return together
  if (*(volatile const int *)&st->k.done != kRunning) return;
  if (t < 32) {
    tm_alloc(&s_tmem, kIrTmemCols);
    tm_relinquish();
    tm_fence_before();
  }
  __syncthreads();
  tm_fence_after();
  const uint32_t w = t >> 5;
  const uint32_t tr = s_tmem + ((32u * (w & 3u)) << 16) + 128u * (w >> 2), tx = tr + 64;
  const TileRows rows(a);
  const bool lead = blockIdx.x == 0 && t == 0;  // keeps the method's state (whole solve)
  double *const sp = reinterpret_cast<double *>(ir_smem_raw);
  const double *const rin = (const double *)a.rin;
  const double eps = st->k.s[S_EPS];
  const long long maxloop = st->k.aux[A_MAXLOOP];
  // the history, written by the lead without reading the state again
  double *hist_err = nullptr;
  long long *hist_it = nullptr;
  long long hcap = 0, hlen = 0;
  if (lead && st->k.aux[A_RECORD]) {
    hist_err = st->k.hist_err;
    hist_it = st->k.hist_it;
    hcap = st->k.hcap;
  }
  // the stopping test at the top of iteration l (check_top); its code
  auto check = [&](long long l, double err) {
    if (l > maxloop) return (int)kMaxLoop;
    if (lead && hist_err) {
      if (hlen < hcap) {
        hist_err[hlen] = err;
        hist_it[hlen] = l;
      }
      hlen++;
    }
    return err <= eps ? (int)kConverged : (err != err ? (int)kNaN : (int)kRunning);
  };

  for (int i = t; i < a.smem_elems; i += kChipThreads) sp[i] = 0.0;
  __syncthreads();
  // start: r = b, p = r (own rows and halo), x = 0
  double acc = 0.0;
#pragma unroll 1
  for (int c = 0; c < rows.blocks; c++) {
    const TileBlock k(rows, c);
    double v[C], z[C];
#pragma unroll
    for (int u = 0; u < C; u++) {
      v[u] = z[u] = 0.0;
      if (k.z0 + u < rows.tz && k.in) {
        v[u] = __ldcg(rin + k.row + u * rows.up);
        sp[k.pos + u * rows.zp] = v[u];
        acc = add_rn(acc, mul_rn(v[u], v[u]));
      }
    }
    CV::put(tr + CV::W * c, v);
    CV::put(tx + CV::W * c, z);
  }
  // The halo: the tile's columns in the planes below and above, then the lines
  // before and after each plane's. f(u, side, place in p, row) for each of the
  // thread's (those of thread i of m).
  auto halo_z = [&](int i, int m, auto &&f) {
#pragma unroll
    for (int u = 0; u < HZ; u++) {
      int c = i + m * u;
      asm volatile("" : "+r"(c));  // opaque, as in TileBlock
      if (c < rows.plane) {
        const int p = 1 + c + tile_quot(c, rows.m_nx) + rows.lp, g = rows.row0 + c;
        if (rows.z0) f(u, 0, p, g - rows.up);
        if (rows.z1) f(u, 1, p + (rows.tz + 1) * rows.zp, g + rows.tz * rows.up);
      }
    }
  };
  auto halo_y = [&](int i, int m, auto &&f) {
#pragma unroll
    for (int u = 0; u < HY; u++) {
      int k = i + m * u;
      asm volatile("" : "+r"(k));
      if (k < rows.nx * rows.tz) {
        const int z = tile_quot(k, rows.m_nx), x = k - z * rows.nx;
        const int p = 1 + x + (z + 1) * rows.zp, g = rows.row0 + x + z * rows.up;
        if (rows.y0) f(u, 0, p, g - rows.nx);
        if (rows.y1) f(u, 1, p + (rows.ty + 1) * rows.lp, g + rows.plane);
      }
    }
  };
  if (t >= 32) {
    auto first = [&](int, int, int p, int g) { sp[p] = __ldcg(rin + g); };
    halo_z(t - 32, kTileHaloThreads, first);
    halo_y(t - 32, kTileHaloThreads, first);
  }
  tm_wait_st();
  if (t == 0) {
    S.alpha = S.beta = 0.0;
    S.code = kRunning;
    S.fail = 0;
  }
  unsigned long long gen = 0;
  bool ok = true;  // no wait ran out
  long long L = 1, top = 1;    // top: the last iteration whose stopping test ran
  // |b| and the stopping test at the top of iteration 1 (NormBOp, StartZeroOp)
  chip_post(a, ++gen, acc);
  ok = chip_wait(a, gen, [&](double s) {
    const double bn = sqrt(s);
    const int code = check(1, sqrt(s) / bn);
    if (t == 0) {
      S.rr = s;
      S.bnorm = bn;
      S.code = code;
    }
    if (lead) {
      st->k.s[S_BNORM] = bn;
      st->k.s[S_RR] = s;
    }
  });
  if (ok && S.code == kRunning) {
    const int sb = rows.lp, sc = rows.zp;  // distances of the diagonals +-b and +-c in p
    for (; L <= maxloop; L++) {
      // A: q = A p, (p, q)
      double q[RJ];
      acc = 0.0;
      {
        double pm = 0.0, pc = 0.0;  // p of the plane below and of this one
#pragma unroll
        for (int c = 0; c < RJ / C; c++) {
          if (c >= rows.blocks) break;
          const TileBlock k(rows, c);
          const double *pp = sp + k.pos;
          if (k.z0 == 0) {
            pm = pp[-sc];
            pc = pp[0];
          }
#pragma unroll
          for (int u = 0; u < C; u++) {
            const double pn = pp[sc];
            const double pv[7] = {pm, pp[-sb], pp[-1], pc, pp[1], pp[sb], pn};
            double y = 0.0;
#pragma unroll
            for (int d = 0; d < 7; d++) y = add_rn(y, mul_rn(D.v[d], pv[d]));
            q[C * c + u] = y;
            const double w = add_rn(acc, mul_rn(pc, y));
            acc = k.in && k.z0 + u < rows.tz ? w : acc;
            pm = pc;
            pc = pn;
            pp += k.z0 + u + 1 < rows.tz ? sc : 0;
          }
        }
      }
      chip_post(a, ++gen, acc);
      // alpha = rr / (p, q)   (rdiv: a zero denominator is a breakdown)
      ok = chip_wait(a, gen, [&](double s) {
        const double al = s == 0.0 ? 0.0 : div_rn(S.rr, s);
        if (t == 0) {
          S.alpha = al;
          S.code = s == 0.0 ? kBreakdown : (isfinite(al) ? kRunning : kNaN);
        }
      });
      if (!ok || S.code != kRunning) break;
      // B: r -= alpha q, published where another CTA reads it; (r, r) posted
      const double av = S.alpha;
      acc = 0.0;
#pragma unroll
      for (int c = 0; c < RJ / C; c++) {
        if (c >= rows.blocks) break;
        const TileBlock k(rows, c);
        double r[C];
        CV::get(tr + CV::W * c, r);
        double *R = (double *)a.P + k.row;
#pragma unroll
        for (int u = 0; u < C; u++) {
          r[u] = add_rn(mul_rn(-av, q[C * c + u]), r[u]);
          const double w = add_rn(acc, mul_rn(r[u], r[u]));
          const bool in = k.in && k.z0 + u < rows.tz;
          acc = in ? w : acc;
          const bool zf = (rows.z0 && k.z0 + u == 0) || (rows.z1 && k.z0 + u == rows.tz - 1);
          if (in && (k.face || zf)) __stcg(R + u * rows.up, r[u]);
        }
        CV::put(tr + CV::W * c, r);
      }
      tm_wait_st();
      chip_post(a, ++gen, acc);
      if (t == 32) st_release_u64(tile_flag(a.sync, blockIdx.x), (unsigned long long)L);
      // x += alpha p while the other CTAs arrive
#pragma unroll 1
      for (int c = 0; c < rows.blocks; c++) {
        const TileBlock k(rows, c);
        const double *pp = sp + k.pos;
        double x[C];
        CV::get(tx + CV::W * c, x);
#pragma unroll
        for (int u = 0; u < C; u++) {
          x[u] = add_rn(mul_rn(av, *pp), x[u]);
          pp += k.z0 + u + 1 < rows.tz ? sc : 0;
        }
        CV::put(tx + CV::W * c, x);
      }
      tm_wait_st();
      // the halo's r (warps 1 .. 15)
      double hz[HZ][2], hy[HY][2];
      if (t >= 32) {
        if (t < 36) {
          const int q = rows.cta(t - 32);
          ChipClock clk;
          bool good = true;
          while (good && q >= 0 && ld_acquire_u64(tile_flag(a.sync, q)) < (unsigned long long)L) good = clk.go_on(a.wait_ns);
          if (!good) {
            S.fail = 1;
            atomicExch(a.err, 1);
          }
        }
        tile_halo_barrier();
        halo_z(t - 32, kTileHaloThreads, [&](int u, int side, int, int g) { hz[u][side] = __ldcg((const double *)a.P + g); });
        halo_y(t - 32, kTileHaloThreads, [&](int u, int side, int, int g) { hy[u][side] = __ldcg((const double *)a.P + g); });
      }
      // beta = (r, r)_new / (r, r); then the stopping test at the top of
      // iteration L + 1 (check_top), whose verdict overrides beta's
      ok = chip_wait(a, gen, [&](double s) {
        const double rr = S.rr;
        const double be = rr == 0.0 ? 0.0 : div_rn(s, rr);
        const int bcode = rr == 0.0 ? kBreakdown : (isfinite(be) ? kRunning : kNaN);
        const int code = check(L + 1, sqrt(s) / S.bnorm);
        __syncwarp();
        if (t == 0) {
          S.rr = s;
          S.beta = be;
          S.code = code != kRunning ? code : bcode;
        }
      });
      if (ok) top = L + 1;
      if (!ok || S.code != kRunning) break;
      // C: p = beta p + r, own rows and halo
      const double bv = S.beta;
#pragma unroll 1
      for (int c = 0; c < rows.blocks; c++) {
        const TileBlock k(rows, c);
        double *pp = sp + k.pos;
        double r[C], p[C];
        CV::get(tr + CV::W * c, r);
        // planes past the tile's last one read that one, as in A: p holds one plane
        // behind it, and a block reaches up to seven
#pragma unroll
        for (int u = 0, o = 0; u < C; u++) {
          p[u] = pp[o];
          o += k.z0 + u + 1 < rows.tz ? sc : 0;
        }
#pragma unroll
        for (int u = 0; u < C; u++)
          if (k.in && k.z0 + u < rows.tz) pp[u * sc] = add_rn(mul_rn(bv, p[u]), r[u]);
      }
      if (t >= 32) {
        halo_z(t - 32, kTileHaloThreads, [&](int u, int side, int p, int) { sp[p] = add_rn(mul_rn(bv, sp[p]), hz[u][side]); });
        halo_y(t - 32, kTileHaloThreads, [&](int u, int side, int p, int) { sp[p] = add_rn(mul_rn(bv, sp[p]), hy[u][side]); });
      }
      __syncthreads();
      if (S.fail) {
        ok = false;
        break;
      }
    }
  }
  if (ok) {
    const int code = S.code;
    double *xo = (double *)a.x;
    {
#pragma unroll 1
      for (int c = 0; c < rows.blocks; c++) {
        const TileBlock k(rows, c);
        double x[C];
        CV::get(tx + CV::W * c, x);
#pragma unroll
        for (int u = 0; u < C; u++)
          if (k.z0 + u < rows.tz && k.in) __stcg(xo + k.row + u * rows.up, x[u]);
      }
    }
    if (lead) {
      st->k.s[S_ALPHA] = S.alpha;
      st->k.s[S_BETA] = S.beta;
      st->k.s[S_RR] = S.rr;
      st->k.loop = top;
      st->k.hlen = hlen;
      set_done(st, code == kRunning ? kMaxLoop : code);
    }
  }
  // every thread's TMEM accesses are complete (each waited on its own)
  tm_fence_before();
  __syncthreads();
  if (t < 32) {
    tm_fence_after();
    tm_dealloc(s_tmem, kIrTmemCols);
  }
}

}  // namespace ks
