// CG of an unstructured matrix, the vectors on chip (sm_100a): FP64 CG of
// matrices without a diagonal copy, 8K to about 600K rows, whose columns lie
// within about 12,000 rows of the row (meshes in a banded order).
//
// Kernel by kernel such a solve takes three launches per iteration on a system
// that fits in L2: 250K rows of 14 entries, 42 us, of them 17 for the product, 12
// for the vector passes, the rest between the kernels. Here a CTA owns a run
// of rpc consecutive rows, thread t its rows t + NT j: r, x and q = A p in
// registers, p of the run and of every row within the matrix's offsets of it
// (the window) in shared memory, so a row's columns are gathered there and
// never from L2. The matrix is read from L2 in every product, from a copy of
// the CSR arrays in slices of 32 rows (CsrDev::sell_*): entry k of a slice's 32
// rows lies in 32 consecutive places, so a warp's loads are full lines; places
// past a row's end are not read. Entries stay in the row's order, so q is the
// CSR kernel's, bit for bit.
//
// Per iteration as in k_cg_tile (ks_tile_cg.cuh): two grid sums; r is stored to R
// and, behind a flag per CTA, fetched by all warps but the first while the (r, r)
// sum travels. What bounds it: the L2 reads of the matrix (35 MB of values and
// offsets here), the bank conflicts of the gathers, and the two grid sums. Measured,
// us per iteration, one kernel per step (up to 32K rows: one cluster) / k_cg_csr:
// 9,000 rows of 14 entries 11.5 / 6.1, 20K 28 / 8.0, 40K 18 / 10.0, 60K 20 / 12.2, 100K
// of 20 39 / 11.0, 250K of 14 41 / 13.9, of 50 107 / 54, 600K of 7 44 / 20.4, of 27
// 162 / 50 (the matrices of 250K x 50 and 600K x 27 do not fit in L2).
#pragma once

#include "ks_chip_cg.cuh"

namespace ks {

// NT threads per CTA: 512 of 128 registers up to 4 rows per thread, 1,024 of 64
// above (us per iteration, 512 / 1,024: 100K rows 11.0 / 11.5, 250K 13.9 / 15.7,
// 400K 23.8 / 19.8). a.wl, a.wu: window rows before and after the run (the
// matrix's largest offsets).
template <int NT, int RJ>
__global__ void __launch_bounds__(NT, 1) k_cg_csr(const __grid_constant__ CsrCgArgs a) {
  constexpr int U = 8;                   // entries of a row in flight
  constexpr int HN = NT == 512 ? 12 : 6;  // window rows per thread fetched while (r, r) travels
  extern __shared__ __align__(16) unsigned char ir_smem_raw[];
  __shared__ ChipScalars S;
  const int t = threadIdx.x;
  DevState *st = a.st;
  if (*(volatile const int *)&st->k.done != kRunning) return;  // the same value in every CTA
  const int r0 = blockIdx.x * a.rpc, nr = min(a.rpc, a.n - r0);  // >= 1 (csr_shape)
  const bool lead = blockIdx.x == 0 && t == 0;                   // keeps the method's state
  double *const sp = reinterpret_cast<double *>(ir_smem_raw) + a.wl;  // p of local rows -wl .. nr + wu - 1
  const int nh = a.wl + a.wu;
  const int bl = max(r0 - a.wl, 0) / a.rpc, bh = min(r0 + nr - 1 + a.wu, a.n - 1) / a.rpc;  // CTAs in the window
  double *const R = (double *)a.P;
  const double *const rin = (const double *)a.rin;
  const double eps = st->k.s[S_EPS];
  const long long maxloop = st->k.aux[A_MAXLOOP];
  double *hist_err = nullptr;  // the history, written by the lead without reading the state again
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
  // window row k (of nh): its local row
  auto win = [&](int k) { return k < a.wl ? k - a.wl : nr + k - a.wl; };

  // start: r = b, p = r (own rows and window), x = 0
  double r[RJ], x[RJ], q[RJ];
  int len[RJ];
  int first[RJ];  // first entry of the row's slice, this lane's place
  double acc = 0.0;
#pragma unroll
  for (int j = 0; j < RJ; j++) {
    const int li = t + NT * j;
    r[j] = x[j] = q[j] = 0.0;
    len[j] = 0;
    first[j] = 0;
    if (li < nr) {
      r[j] = __ldcg(rin + r0 + li);
      sp[li] = r[j];
      acc = add_rn(acc, mul_rn(r[j], r[j]));
      const int i = r0 + li;
      len[j] = __ldg(a.ptr + i + 1) - __ldg(a.ptr + i);
      first[j] = 32 * __ldg(a.slice + i / 32) + (t & 31);  // rpc and r0 are multiples of 32
    }
  }
  for (int k = t; k < nh; k += NT) {
    const int li = win(k), c = r0 + li;
    sp[li] = c >= 0 && c < a.n ? __ldcg(rin + c) : 0.0;
  }
  if (t == 0) {
    S.alpha = S.beta = 0.0;
    S.code = kRunning;
    S.fail = 0;
  }
  unsigned long long gen = 0;
  long long L = 1, top = 1;  // top: the last iteration whose stopping test ran
  // |b| and the stopping test at the top of iteration 1 (NormBOp, StartZeroOp)
  chip_post<NT>(a, ++gen, acc);
  bool ok = chip_wait(a, gen, [&](double s) {
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
    for (; L <= maxloop; L++) {
      // A: q = A p, (p, q)
      acc = 0.0;
#pragma unroll
      for (int j = 0; j < RJ; j++) {
        if (NT * j >= nr) break;
        const int li = t + NT * j;
        const double *pp = sp + li;
        double y = 0.0;
        int e = first[j];
#pragma unroll 1
        for (int k0 = 0; __any_sync(0xffffffffu, k0 < len[j]); k0 += U, e += 32 * U) {
          double v[U];
          int o[U];
#pragma unroll
          for (int u = 0; u < U; u++) {
            v[u] = 0.0;
            o[u] = 0;
            if (k0 + u < len[j]) {
              v[u] = __ldg(a.val + e + 32 * u);
              o[u] = __ldg(a.off + e + 32 * u);
            }
          }
#pragma unroll
          for (int u = 0; u < U; u++) {
            if (k0 + u < len[j]) y = add_rn(y, mul_rn(v[u], pp[o[u]]));
          }
        }
        q[j] = y;
        if (li < nr) acc = add_rn(acc, mul_rn(*pp, y));
      }
      chip_post<NT>(a, ++gen, acc);
      // alpha = rr / (p, q)   (rdiv: a zero denominator is a breakdown)
      ok = chip_wait(a, gen, [&](double s) {
        const double al = s == 0.0 ? 0.0 : div_rn(S.rr, s);
        if (t == 0) {
          S.alpha = al;
          S.code = s == 0.0 ? kBreakdown : (isfinite(al) ? kRunning : kNaN);
        }
      });
      if (!ok || S.code != kRunning) break;
      // B: r -= alpha q, stored to R; (r, r) posted; x += alpha p and the
      // window's r while the other CTAs arrive
      const double av = S.alpha;
      acc = 0.0;
#pragma unroll
      for (int j = 0; j < RJ; j++) {
        const int li = t + NT * j;
        if (li < nr) {
          r[j] = add_rn(mul_rn(-av, q[j]), r[j]);
          __stcg(R + r0 + li, r[j]);
          acc = add_rn(acc, mul_rn(r[j], r[j]));
        }
      }
      chip_post<NT>(a, ++gen, acc);
      if (t == 32) st_release_u64(tile_flag(a.sync, blockIdx.x), (unsigned long long)L);
#pragma unroll
      for (int j = 0; j < RJ; j++) {
        const int li = t + NT * j;
        if (li < nr) x[j] = add_rn(mul_rn(av, sp[li]), x[j]);
      }
      constexpr int T = NT - 32;
      double h[HN];
      if (t >= 32) {
        if (t < 64) {
          for (int c = bl + t - 32; c <= bh; c += 32) {
            ChipClock clk;
            bool good = true;
            while (good && c != (int)blockIdx.x && ld_acquire_u64(tile_flag(a.sync, c)) < (unsigned long long)L)
              good = clk.go_on(a.wait_ns);
            if (!good) {
              S.fail = 1;
              atomicExch(a.err, 1);
            }
          }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(NT - 32) : "memory");
#pragma unroll
        for (int u = 0; u < HN; u++) {
          const int k = t - 32 + T * u, c = r0 + win(k);
          h[u] = k < nh && c >= 0 && c < a.n ? __ldcg(R + c) : 0.0;
        }
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
      // C: p = beta p + r, own rows and window
      const double bv = S.beta;
#pragma unroll
      for (int j = 0; j < RJ; j++) {
        const int li = t + NT * j;
        if (li < nr) sp[li] = add_rn(mul_rn(bv, sp[li]), r[j]);
      }
      if (t >= 32) {
        auto upd = [&](int k, double hk) {
          const int li = win(k), c = r0 + li;
          if (k < nh && c >= 0 && c < a.n) sp[li] = add_rn(mul_rn(bv, sp[li]), hk);
        };
#pragma unroll
        for (int u = 0; u < HN; u++) upd(t - 32 + T * u, h[u]);
        for (int k0 = t - 32 + T * HN; k0 < nh; k0 += 4 * T) {
          double w[4];
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int k = k0 + T * u, c = r0 + win(k);
            w[u] = k < nh && c >= 0 && c < a.n ? __ldcg(R + c) : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 4; u++) upd(k0 + T * u, w[u]);
        }
      }
      __syncthreads();
      if (S.fail) {
        ok = false;
        break;
      }
    }
  }
  if (ok) {
    double *xo = (double *)a.x;
#pragma unroll
    for (int j = 0; j < RJ; j++) {
      const int li = t + NT * j;
      if (li < nr) __stcg(xo + r0 + li, x[j]);
    }
    if (lead) {
      st->k.s[S_ALPHA] = S.alpha;
      st->k.s[S_BETA] = S.beta;
      st->k.s[S_RR] = S.rr;
      st->k.loop = top;
      st->k.hlen = hlen;
      set_done(st, S.code == kRunning ? kMaxLoop : S.code);
    }
  }
}

}  // namespace ks
