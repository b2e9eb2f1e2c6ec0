// CG with the matrix on chip (sm_100a).
//
// k_cg_onchip (ks_inner_resident.cuh) keeps a CG solve's vectors on chip and
// reads the matrix from L2 in every iteration. Where the system leaves a
// thread no more than 8 (FP64) or 16 (FP32) rows, the diagonal copy fits on
// chip too: up to 8 diagonals of 8 doubles or 16 floats are the 128 words of
// tensor memory a thread reaches (TMEM, 256 KB per SM, used as a register
// file). k_cg_chip loads it there once per launch and runs the whole solve
// (FP64 CG up to about 600K rows; the FP32 / BF16-valued inner CG of the VP
// methods up to about 1.2M rows) with one vector, r, crossing between CTAs.
//
// Which rows a CTA owns. A 7-point stencil on a box (CsrDev::dia_box): a tile
// of by x bz whole lines of the box, so that the rows around it which its
// rows read, its halo, are the 2 (by + bz) lines of its four faces (99^3: 34
// lines of 99 rows; a run of consecutive rows would read two planes, 198
// lines). Any other matrix: a run of rpc consecutive rows. Thread t of the
// CTA takes its local rows t + 512 j (j < RJ), so a warp's accesses to
// shared memory are consecutive at any offset (odd grid edges included) and
// no alignment rule applies. Matrix values in TMEM (warp w: lanes 32 (w % 4)
// .. +31, columns 128 (w / 4) .. +127; diagonal d in words d W .. +W-1), r
// and q = A p in registers, x in the TMEM words the matrix leaves or in
// registers, p of the own rows and of the halo, and a table of the halo's rows,
// in shared memory.
//
// Per iteration (cg.cpp:184-240):
//   A: q = A p, (p, q) summed over the grid -> alpha;
//   B: r -= alpha q; rows in another CTA's halo are published; (r, r)
//      summed over the grid; while it travels x += alpha p, and the halo's r
//      is fetched -> beta, stopping test;
//   C: p = beta p + r for the own rows and the halo.
// Every CTA forms the halo's p with the owner's operations on the owner's
// values, so it holds the owner's bits, and the third grid-wide wait of
// k_cg_onchip (the publication of p) is gone. r is published value by value
// with the iteration's tag in one store (16 bytes in FP64, 8 in FP32): a
// reader takes a value with its tag and needs no fence and no flag, so the
// halo arrives in the shadow of the (r, r) reduction. Tags differ from one
// launch to the next on the same array (ChipArgs::tag0). With one or two rows per
// thread r crosses behind a flag per CTA instead, acquired by warp 1 while warp 0
// waits for the sum (us per iteration, tags / flags: 128^2 3.46 / 3.10, 333^2 4.74 /
// 4.56; with more rows per thread the flags' kernel spills: 700^2 6.7 / 8.0, 99^3
// FP32 11.4 / 12.3). Element operations
// and the order of a row's terms are k_cg_onchip's; only the dot products add
// their terms in another order. An entry a row does not have is a stored zero
// and its term a zero added to a sum that starts at +0: no mask is looked at (p
// is finite; one that is not ends the method as kNaN either way). A column
// outside the matrix has p = 0.
//
// What bounds an iteration: latency, the two grid reductions before all (1.2
// to 1.6 us each; 333^2: of 4.6 us per iteration about 3.3). Measured, us per
// iteration, k_cg_onchip or the kernel it replaces / k_cg_chip: FP64 CG 128^2
// 4.39 / 3.10, 333^2 14.5 / 4.56, 512^2 11.8 / 5.11, 64^3 13.3 / 5.8, 81^3 17.5
// / 8.0; FP32 inner CG 24^3 17.9 / 3.8, 64^3 13.3 / 5.7, 99^3 (BF16 values)
// 18.3 / 11.4. The largest systems are bound by the instructions per row (7
// products from shared memory, FP64 sums of FP32 rows).
#pragma once

#include <cmath>

#include "ks_inner_resident.cuh"

namespace ks {

// 512 threads of 128 registers: with 1,024 threads of 64 the kernels that hold
// the most rows per thread spill (99^3 FP32 inner CG, 7 rows of 1,024
// threads: 14.0 us per iteration)
constexpr int kChipThreads = 512;
constexpr int kChipWords = 128;  // TMEM words of a thread
constexpr unsigned kChipMaxGrid = 160;  // CTAs a reduction takes (one per SM)

// The CTAs' slots of a reduction of generation gen (two sets, by parity).
__device__ __forceinline__ ulonglong2 *ir_slots(IrSync *s, unsigned G, unsigned long long gen) {
  ulonglong2 *base = reinterpret_cast<ulonglong2 *>(reinterpret_cast<unsigned long long *>(s + 1) + ((G + 1) & ~1u));
  return base + (size_t)(gen & 1) * G;
}

// The publication flag of CTA q, 32 bytes apart, behind the reductions' slots.
__device__ __forceinline__ unsigned long long *tile_flag(IrSync *s, int q) {
  return reinterpret_cast<unsigned long long *>(ir_slots(s, gridDim.x, 0) + 2 * gridDim.x) + 4 * q;
}


// A value and its tag as one 16-byte access (single-copy atomic).
__device__ __forceinline__ void chip_slot_st(ulonglong2 *q, double v, unsigned long long tag) {
  const unsigned long long lo = (unsigned long long)__double_as_longlong(v);
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(q), "l"(lo),
               "l"(tag)
               : "memory");
}
__device__ __forceinline__ void chip_slot_ld(const ulonglong2 *q, double &v, unsigned long long &tag) {
  unsigned long long lo;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
               : "=l"(lo), "=l"(tag)
               : "l"(q)
               : "memory");
  v = __longlong_as_double((long long)lo);
}
__device__ __forceinline__ void red_relaxed_add_u64(unsigned long long *p, unsigned long long v) {
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// A bounded wait's clock, started before the first poll; go_on() after a
// failed poll is false once the limit has passed. It looks at the global
// timer at the first polls and then at every 32nd (a read of the timer costs
// about as much as a poll).
struct ChipClock {
  unsigned long long t0 = global_ns();
  unsigned it = 0;
  __device__ __forceinline__ bool go_on(unsigned long long limit_ns) {
    const unsigned i = it++;
    if (i >= 8 && (i & 31u) != 0) return true;
    return global_ns() - t0 <= limit_ns;
  }
};

// Grid-wide sums, the same in every CTA, in two halves so that work which
// does not need the sum runs while the other CTAs arrive: chip_post adds the
// CTA's values (a block-wide step: every thread calls it) and posts the sum;
// chip_wait (every thread) waits for all CTAs and adds the sums in one fixed
// order.
//
// A post is one 16-byte store of value and generation per sum, plus (above
// kChipDirect CTAs) a relaxed count of arrivals: nothing waits for a store to
// complete before the next one, as a release would. One lane polls the count,
// then the warp reads the slots and takes a value only with its tag, again
// where a slot's store is still on its way. Up to kChipDirect CTAs the slots
// themselves are polled: one round trip less, but above that the CTAs' polls
// of the same lines slow the stores down. Measured (B200, 1,024 threads,
// microseconds per reduction, release-add and plain partials / this):
// 148 CTAs 2.24 / 1.64, 64 CTAs 2.21 / 1.51, 16 CTAs 1.97 / 1.23 (counted:
// 1.49), 2 CTAs 1.67 / 0.93; slots polled by 148 CTAs 3.4, by 64 CTAs 2.0-2.2.
//
// The reduction orders no other memory: what else crosses between CTAs
// carries tags of its own. Two generations of slots: a CTA writes generation g + 2's only after every
// CTA has posted g + 1, i.e. after every CTA has read generation g's.
constexpr unsigned kChipDirect = 32;

template <int kThreadsPerCta = kChipThreads>
__device__ __forceinline__ void chip_post(const IrArgs &a, unsigned long long gen, double v) {
  constexpr int kWarps = kThreadsPerCta / 32;
  __shared__ double sh[kWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    const unsigned G = gridDim.x;
    v = warp_sum(lane < kWarps ? sh[lane & (kWarps - 1)] : 0.0);
    if (lane == 0) {
      chip_slot_st(ir_slots(a.sync, G, gen) + blockIdx.x, v, gen);
      if (G > kChipDirect) red_relaxed_add_u64(&a.sync->count, 1ull);
    }
  }
}

// The tagged values of all CTAs, U loads per lane in flight (lanes past the
// last CTA read its slot and drop the value), again until every tag is there.
template <int U>
__device__ __forceinline__ bool chip_gather(const ulonglong2 *sl, unsigned G, unsigned long long gen,
                                          unsigned long long limit_ns, ChipClock &clk, double &sum) {
  const unsigned lane = threadIdx.x;
  double pv[U];
  unsigned long long tag[U];
  for (;;) {
#pragma unroll
    for (int u = 0; u < U; u++) chip_slot_ld(sl + min(lane + 32u * u, G - 1), pv[u], tag[u]);
    bool late = false;
#pragma unroll
    for (int u = 0; u < U; u++) late |= tag[u] != gen;
    if (!__any_sync(0xffffffffu, late)) break;
    if (!__all_sync(0xffffffffu, clk.go_on(limit_ns))) return false;
  }
  sum = 0.0;
#pragma unroll
  for (int u = 0; u < U; u++) sum += lane + 32u * u < G ? pv[u] : 0.0;
  return true;
}

// Waits for the sum; warp 0 then runs f(sum) (all 32 lanes, the same value)
// before the other threads pass the barrier at the end: scalar steps done once
// and handed on through shared memory, not by all warps, which share one FP64
// pipe. Returns false when the wait ran out (the timeout flag is then set; f
// has not run).
template <class F>
__device__ __forceinline__ bool chip_wait(const IrArgs &a, unsigned long long gen, F &&f) {
  __shared__ int s_ok;
  const unsigned G = gridDim.x;
  if (threadIdx.x < 32) {
    const unsigned lane = threadIdx.x;
    ChipClock clk;
    bool good = true;
    if (G > kChipDirect) {
      if (lane == 0) {
        const unsigned long long want = gen * (unsigned long long)G;
        while (good && ld_relaxed_u64(&a.sync->count) < want) good = clk.go_on(a.wait_ns);
      }
      good = __shfl_sync(0xffffffffu, (int)good, 0) != 0;
    }
    double s = 0.0;
    const ulonglong2 *sl = ir_slots(a.sync, G, gen);
    if (good)
      good = G > kChipDirect ? chip_gather<kChipMaxGrid / 32>(sl, G, gen, a.wait_ns, clk, s)
                             : chip_gather<1>(sl, G, gen, a.wait_ns, clk, s);
    s = warp_sum(s);
    if (good) f(s);
    if (lane == 0) {
      s_ok = good ? 1 : 0;
      if (!good) atomicExch(a.err, 1);
    }
  }
  __syncthreads();
  return s_ok != 0;
}

// N words per thread to / from TMEM (N = 1, 2, 4, 8, 16).
template <int N>
__device__ __forceinline__ void tmw_st(uint32_t ta, const uint32_t (&w)[N]) {
  static_assert(N == 1 || N == 2 || N == 4 || N == 8 || N == 16, "words");
  if constexpr (N == 1)
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(ta), "r"(w[0]) : "memory");
  else if constexpr (N == 2)
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(ta), "r"(w[0]), "r"(w[1]) : "memory");
  else if constexpr (N == 4)
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(ta), "r"(w[0]), "r"(w[1]),
                 "r"(w[2]), "r"(w[3])
                 : "memory");
  else if constexpr (N == 16)
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16};" ::"r"(ta),
        "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]),
        "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15])
        : "memory");
  else
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(ta), "r"(w[0]),
                 "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}
// Loaded registers are valid only behind the wait, which they pass through.
template <int N>
__device__ __forceinline__ void tmw_ld(uint32_t ta, uint32_t (&w)[N]) {
  static_assert(N == 1 || N == 2 || N == 4 || N == 8 || N == 16, "words");
  if constexpr (N == 1) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(w[0]) : "r"(ta) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(w[0])::"memory");
  } else if constexpr (N == 2) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(ta) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(w[0]), "+r"(w[1])::"memory");
  } else if constexpr (N == 4) {
    tm_ld4(ta, w);
    tm_wait_ld4(w);
  } else if constexpr (N == 16) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]), "=r"(w[8]),
          "=r"(w[9]), "=r"(w[10]), "=r"(w[11]), "=r"(w[12]), "=r"(w[13]), "=r"(w[14]), "=r"(w[15])
        : "r"(ta)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3]), "+r"(w[4]), "+r"(w[5]), "+r"(w[6]), "+r"(w[7]),
                   "+r"(w[8]), "+r"(w[9]), "+r"(w[10]), "+r"(w[11]), "+r"(w[12]), "+r"(w[13]), "+r"(w[14]), "+r"(w[15])::
                     "memory");
  } else {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                 : "r"(ta)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3]), "+r"(w[4]), "+r"(w[5]), "+r"(w[6]), "+r"(w[7])::
                     "memory");
  }
}

// A thread's RJ values of one diagonal in TMEM.
template <class VT, int RJ>
struct ChipVals {
  static constexpr int W = RJ * (int)sizeof(VT) / 4;
  __device__ __forceinline__ static void put(uint32_t ta, const VT (&v)[RJ]) {
    uint32_t w[W];
#pragma unroll
    for (int j = 0; j < RJ; j++) {
      if constexpr (sizeof(VT) == 4) {
        w[j] = __float_as_uint(v[j]);
      } else {
        const unsigned long long u = (unsigned long long)__double_as_longlong(v[j]);
        w[2 * j] = (uint32_t)u;
        w[2 * j + 1] = (uint32_t)(u >> 32);
      }
    }
    tmw_st<W>(ta, w);
  }
  __device__ __forceinline__ static void get(uint32_t ta, VT (&v)[RJ]) {
    uint32_t w[W];
    tmw_ld<W>(ta, w);
#pragma unroll
    for (int j = 0; j < RJ; j++) {
      if constexpr (sizeof(VT) == 4)
        v[j] = __uint_as_float(w[j]);
      else
        v[j] = __longlong_as_double((long long)(((unsigned long long)w[2 * j + 1] << 32) | w[2 * j]));
    }
  }
};

// A published value with its tag, one access.
__device__ __forceinline__ void chip_pub(void *R, long long i, double v, unsigned long long tag) {
  chip_slot_st((ulonglong2 *)R + i, v, tag);
}
__device__ __forceinline__ bool chip_take(const void *R, long long i, double &v, unsigned long long tag) {
  unsigned long long t;
  chip_slot_ld((const ulonglong2 *)R + i, v, t);
  return t == tag;
}
__device__ __forceinline__ void chip_pub(void *R, long long i, float v, unsigned long long tag) {
  const unsigned long long u = (tag << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"((unsigned long long *)R + i), "l"(u) : "memory");
}
__device__ __forceinline__ bool chip_take(const void *R, long long i, float &v, unsigned long long tag) {
  const unsigned long long u = ld_relaxed_u64((const unsigned long long *)R + i);
  v = __uint_as_float((unsigned)u);
  return (unsigned)(u >> 32) == (unsigned)tag;
}

struct ChipArgs : IrArgs {  // P is the array R of published r, zeroed before the first launch on it
  const void *vb[kMaxDiag];  // DiaT's values
  int vs[kMaxDiag];
  int nd;
  int off[kMaxDiag];
  int bf16;    // values are BF16 (VT = float)
  int smem_elems;  // p with its halo
  unsigned long long tag0;  // iteration L publishes r with tag0 + L
  // runs of rows: halo rows below and above the own ones, and the part of
  // them next to the own rows that is read whole (the second largest offset)
  int hl, hu, hl2, hu2;
  // tiles of lines
  int nx, ny, nz, by, bz, gy;
};

// The rows of one CTA and where they and their halo sit in shared memory.
// Local row li of the own rows: pos(li), row(li); halo row k < halo(): its
// position and row, row < 0 where there is none.
template <bool kTile>
struct ChipRows;

template <>
struct ChipRows<false> {
  int r0, nr, n, hl, hu, lo_far, n_lo, hl2, hi_far, n_hi, hu2;
  __device__ __forceinline__ explicit ChipRows(const ChipArgs &a) {
    r0 = blockIdx.x * a.rpc;
    n = a.n;
    nr = min(a.rpc, n - r0);  // >= 1 (chip_shape)
    hl = a.hl, hu = a.hu, hl2 = a.hl2, hu2 = a.hu2;
    // below: the columns of the largest offset [-hl, nr - hl) and the rows
    // [-hl2, 0), in which every other offset's columns lie; above likewise
    lo_far = hl2 < hl ? min(nr, hl - hl2) : 0;
    n_lo = lo_far + hl2;
    hi_far = hu2 < hu ? min(nr, hu - hu2) : 0;
    n_hi = hi_far + hu2;
    bl = max(r0 - hl, 0) / a.rpc;
    nb = min(r0 + nr - 1 + hu, n - 1) / a.rpc - bl + 1;
  }
  __device__ __forceinline__ int pos(int li) const { return hl + li; }
  __device__ __forceinline__ int row(int li) const { return r0 + li; }
  __device__ __forceinline__ bool shared(int li) const { return li < hu || li >= nr - hl; }
  __device__ __forceinline__ int shift(int, int off) const { return off; }
  __device__ __forceinline__ int halo() const { return n_lo + n_hi; }
  int bl, nb;  // the CTAs that own halo rows
  __device__ __forceinline__ int ctas() const { return nb; }
  __device__ __forceinline__ int cta(int i) const { return bl + i == (int)blockIdx.x ? -1 : bl + i; }
  __device__ __forceinline__ void halo_row(int k, int &p, int &g) const {
    int li;
    if (k < n_lo) {
      li = k < lo_far ? k - hl : k - lo_far - hl2;
    } else {
      k -= n_lo;
      li = k < hu2 ? nr + k : nr + hu - hi_far + (k - hu2);
    }
    p = hl + li;
    g = r0 + li;
    if (g < 0 || g >= n) g = -1;
  }
};

template <>
struct ChipRows<true> {
  int nx, ty, tz, plane, nr, row0, up, pitch, gy;  // up: rows of a plane of the box; pitch: of a plane in shared memory
  float inv_plane, inv_nx;
  bool y0, y1, z0, z1;  // faces with a neighbour
  __device__ __forceinline__ explicit ChipRows(const ChipArgs &a) {
    const int cy = blockIdx.x % a.gy, cz = blockIdx.x / a.gy;
    gy = a.gy;
    nx = a.nx;
    ty = min(a.by, a.ny - cy * a.by);
    tz = min(a.bz, a.nz - cz * a.bz);
    plane = nx * ty;
    nr = plane * tz;
    up = nx * a.ny;
    row0 = cy * a.by * nx + cz * a.bz * up;
    pitch = plane + 2 * nx;
    inv_plane = 1.0f / (float)plane;
    inv_nx = 1.0f / (float)nx;
    y0 = cy > 0;
    y1 = cy * a.by + ty < a.ny;
    z0 = cz > 0;
    z1 = cz * a.bz + tz < a.nz;
  }
  // k / d for k < 2^14 (the error of the product stays below half a divisor's step)
  __device__ __forceinline__ static int quot(int k, float inv) { return (int)(((float)k + 0.5f) * inv); }
  __device__ __forceinline__ int pos(int li) const { return 1 + pitch + nx + li + quot(li, inv_plane) * 2 * nx; }
  __device__ __forceinline__ int row(int li) const { return row0 + li + quot(li, inv_plane) * (up - plane); }
  __device__ __forceinline__ bool shared(int li) const {
    const int lz = quot(li, inv_plane), l = li - lz * plane;
    return (y0 && l < nx) || (y1 && l >= plane - nx) || (z0 && lz == 0) || (z1 && lz == tz - 1);
  }
  __device__ __forceinline__ int shift(int d, int) const {  // diagonals -c, -b, -1, 0, 1, b, c
    const int e = d < 3 ? 3 - d : d - 3, s = e == 0 ? 0 : e == 1 ? 1 : e == 2 ? nx : pitch;
    return d < 3 ? -s : s;
  }
  __device__ __forceinline__ int halo() const { return 2 * nx * tz + 2 * plane; }
  __device__ __forceinline__ int ctas() const { return 4; }
  __device__ __forceinline__ int cta(int i) const {  // the neighbours (-1: none)
    const int b = blockIdx.x;
    return i == 0 ? (y0 ? b - 1 : -1) : i == 1 ? (y1 ? b + 1 : -1) : i == 2 ? (z0 ? b - gy : -1) : (z1 ? b + gy : -1);
  }
  __device__ __forceinline__ void halo_row(int k, int &p, int &g) const {
    if (k < 2 * plane) {  // z faces: whole planes of the tile
      const bool hi = k >= plane;
      if (hi) k -= plane;
      p = 1 + nx + k + (hi ? (tz + 1) * pitch : 0);
      g = (hi ? z1 : z0) ? row0 + k + (hi ? tz * up : -up) : -1;
    } else {  // y faces: one line of each plane
      k -= 2 * plane;
      const bool hi = k >= nx * tz;
      if (hi) k -= nx * tz;
      const int lz = quot(k, inv_nx), lx = k - lz * nx;
      p = 1 + (lz + 1) * pitch + lx + (hi ? nx + plane : 0);
      g = (hi ? y1 : y0) ? row0 + lz * up + lx + (hi ? plane : -nx) : -1;
    }
  }
};

// The method's scalars, computed once per CTA (warp 0) and handed on here.
struct ChipScalars {
  double alpha, beta, rr, bnorm;
  int code;
  int fail;  // a halo wait ran out
};

constexpr int kChipHalo = 8;  // halo rows per thread at most

template <class VT, int NDG, int RJ, bool kTile>
__global__ void __launch_bounds__(kChipThreads, 1) k_cg_chip(const __grid_constant__ ChipArgs a) {
  using CV = ChipVals<VT, RJ>;
  constexpr int KD = NDG > 0 ? NDG : kMaxDiag;
  constexpr bool kFlags = RJ <= 2;  // how r crosses between CTAs
  constexpr bool kXT = (KD + 1) * CV::W <= kChipWords;  // x in TMEM behind the matrix
  static_assert(KD * CV::W <= kChipWords, "the matrix fits a thread's TMEM words");
  static_assert(!kTile || NDG == 7, "tiles are those of a 7-point stencil");
  extern __shared__ __align__(16) unsigned char ir_smem_raw[];
  __shared__ uint32_t s_tmem;
  __shared__ ChipScalars S;
  const int t = threadIdx.x;
  DevState *st = a.st;
  // as k_cg_onchip: the same values in every CTA, so all return together
  if (a.outer_done && *(volatile const int *)a.outer_done) return;
  if (*(volatile const int *)&st->k.done != kRunning) return;
  if (t < 32) {
    tm_alloc(&s_tmem, kIrTmemCols);
    tm_relinquish();
    tm_fence_before();
  }
  __syncthreads();
  tm_fence_after();
  const uint32_t w = t >> 5;
  const uint32_t tm = s_tmem + ((32u * (w & 3u)) << 16) + 128u * (w >> 2);
  const uint32_t tx = tm + CV::W * KD;  // x, if kXT
  const int nd = NDG > 0 ? NDG : a.nd;
  const ChipRows<kTile> rows(a);
  const int nr = rows.nr, nh = rows.halo();
  // the thread's halo rows hk0 + hstep u (flags: none of warp 0, whose hk0 stays
  // negative for all u)
  constexpr int hstep = kFlags ? kChipThreads - 32 : kChipThreads;
  const int hk0 = kFlags ? (t < 32 ? -(1 << 24) : t - 32) : t;
  const bool lead = blockIdx.x == 0 && t == 0;  // keeps the method's state (whole solve)
  // the halo's rows (-1: none) and byte positions, then p with its halo
  int2 *const sh = reinterpret_cast<int2 *>(ir_smem_raw);
  char *const sp = reinterpret_cast<char *>(sh + nh);
  auto P = [&](int o) -> VT & { return *reinterpret_cast<VT *>(sp + o); };
  const VT *const rin = (const VT *)a.rin;
  const double eps = st->k.s[S_EPS];
  const long long maxloop = st->k.aux[A_MAXLOOP];
  // the history, written by the lead without reading the state again
  double *hist_err = nullptr;
  long long *hist_it = nullptr;
  long long hcap = 0, hlen = 0;
  if (lead && a.whole && st->k.aux[A_RECORD]) {
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

  // the thread's rows, their byte positions in p (rows past the CTA's: those
  // of row 0, with zero values) and which of them are published
  unsigned pub = 0;
  int pos[RJ], row[RJ];
#pragma unroll
  for (int j = 0; j < RJ; j++) {
    const int li = t + kChipThreads * j, l = li < nr ? li : 0;
    pos[j] = rows.pos(l) * (int)sizeof(VT);
    row[j] = rows.row(l);
    if (li < nr && rows.shared(li)) pub |= 1u << j;
  }
  // the matrix into TMEM
#pragma unroll
  for (int d = 0; d < KD; d++) {
    if (NDG > 0 || d < nd) {
      VT v[RJ];
#pragma unroll
      for (int j = 0; j < RJ; j++) {
        const int li = t + kChipThreads * j;
        v[j] = (VT)0;
        if (li < nr) {
          const long long i = (long long)row[j] + a.vs[d];
          if constexpr (sizeof(VT) == 8)
            v[j] = __ldg((const double *)a.vb[d] + i);
          else
            v[j] = a.bf16 ? __uint_as_float((unsigned)__ldg((const unsigned short *)a.vb[d] + i) << 16)
                          : __ldg((const float *)a.vb[d] + i);
        }
      }
      CV::put(tm + CV::W * d, v);
    }
  }
  for (int i = t; i < a.smem_elems; i += kChipThreads) P(i * (int)sizeof(VT)) = (VT)0;
  __syncthreads();
  // start: r = b, p = r (own rows and halo), x = 0
  VT r[RJ], q[RJ];
  VT x[kXT ? 1 : RJ];
  double acc = 0.0;
#pragma unroll
  for (int j = 0; j < RJ; j++) {
    const int li = t + kChipThreads * j;
    r[j] = q[j] = (VT)0;
    if constexpr (!kXT) x[j] = (VT)0;
    if (li < nr) {
      r[j] = __ldcg(rin + row[j]);
      P(pos[j]) = r[j];
      acc = add_rn(acc, mul_rn(widen(r[j]), widen(r[j])));
    }
  }
  if constexpr (kXT) CV::put(tx, q);
  for (int k = t; k < nh; k += kChipThreads) {
    int p, g;
    rows.halo_row(k, p, g);
    p *= (int)sizeof(VT);
    sh[k] = make_int2(g, p);
    if (g >= 0) P(p) = __ldcg(rin + g);
  }
  tm_wait_st();
  if (t == 0) {
    S.alpha = S.beta = 0.0;
    S.code = kRunning;
    S.fail = 0;
    if (!a.whole) {
      S.rr = st->k.s[S_RR];
      S.bnorm = st->k.s[S_BNORM];
    }
  }
  unsigned long long gen = 0;
  bool ok = true, xw = false;  // no wait ran out; x was updated
  long long L = 1, top = 1;  // top: the last iteration whose stopping test ran
  if (a.whole) {
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
  } else {
    __syncthreads();  // p's halo and the scalars are in place
  }
  if (ok && S.code == kRunning) {
    for (; L <= maxloop; L++) {
      // A: q = A p, (p, q)
#pragma unroll
      for (int j = 0; j < RJ; j++) q[j] = (VT)0;
#pragma unroll(RJ >= 8 ? 1 : KD)  // with many rows per thread the unrolled loop spills
      for (int d = 0; d < KD; d++) {
        if (NDG > 0 || d < nd) {
          VT av[RJ];
          CV::get(tm + CV::W * d, av);
          const int o = rows.shift(d, a.off[d]) * (int)sizeof(VT);
#pragma unroll
          for (int j = 0; j < RJ; j++)
            if (j == 0 || kChipThreads * j < nr) q[j] = add_rn(q[j], mul_rn(av[j], P(pos[j] + o)));
        }
      }
      acc = 0.0;
#pragma unroll
      for (int j = 0; j < RJ; j++)
        if (t + kChipThreads * j < nr) acc = add_rn(acc, mul_rn(widen(P(pos[j])), widen(q[j])));
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
      // B: r -= alpha q, published where another CTA reads it; (r, r) posted;
      // x += alpha p and the halo's r while the other CTAs arrive
      const VT av = (VT)S.alpha;
      const unsigned long long tag = a.tag0 + (unsigned long long)L;
      acc = 0.0;
#pragma unroll
      for (int j = 0; j < RJ; j++) {
        const int li = t + kChipThreads * j;
        if (li < nr) {
          r[j] = add_rn(mul_rn((VT)(-av), q[j]), r[j]);
          if ((pub >> j) & 1u) {
            if constexpr (kFlags)
              __stcg((VT *)a.P + row[j], r[j]);
            else
              chip_pub(a.P, row[j], r[j], tag);
          }
          acc = add_rn(acc, mul_rn(widen(r[j]), widen(r[j])));
        }
      }
      chip_post(a, ++gen, acc);
      if (kFlags && t == 32) st_release_u64(tile_flag(a.sync, blockIdx.x), (unsigned long long)L);
      if constexpr (kXT) {
        VT xv[RJ];
        CV::get(tx, xv);
#pragma unroll
        for (int j = 0; j < RJ; j++) xv[j] = add_rn(mul_rn(av, P(pos[j])), xv[j]);
        CV::put(tx, xv);
        tm_wait_st();
      } else {
#pragma unroll
        for (int j = 0; j < RJ; j++) x[j] = add_rn(mul_rn(av, P(pos[j])), x[j]);
      }
      xw = true;
      // the halo's r. Flags: a warp other than the first, which waits for the sum,
      // acquires the neighbours' and lets the others load. Tags: every row's load
      // issued, then those whose tag is not this iteration's yet read again
      // (bounded either way)
      VT h[kChipHalo];
      unsigned late = 0;
      if constexpr (kFlags) {
        if (t >= 32) {
          if (t < 64) {
            for (int i = t - 32; i < rows.ctas(); i += 32) {
              const int q = rows.cta(i);
              ChipClock clk;
              bool good = true;
              while (good && q >= 0 && ld_acquire_u64(tile_flag(a.sync, q)) < (unsigned long long)L)
                good = clk.go_on(a.wait_ns);
              if (!good) {
                S.fail = 1;
                atomicExch(a.err, 1);
              }
            }
          }
          asm volatile("bar.sync 1, %0;" ::"n"(kChipThreads - 32) : "memory");
#pragma unroll
          for (int u = 0; u < kChipHalo; u++) {
            const int k = hk0 + hstep * u;
            h[u] = (VT)0;
            if (hstep * u < nh && k < nh) {
              const int g = sh[k].x;
              if (g >= 0) h[u] = __ldcg((const VT *)a.P + g);
            }
          }
        }
      } else {
#pragma unroll
        for (int u = 0; u < kChipHalo; u++) {
          const int k = hk0 + hstep * u;
          h[u] = (VT)0;
          if (hstep * u < nh && k < nh) {
            const int g = sh[k].x;
            if (g >= 0 && !chip_take(a.P, g, h[u], tag)) late |= 1u << u;
          }
        }
      }
      if (late) {
        ChipClock clk;
        do {
#pragma unroll
          for (int u = 0; u < kChipHalo; u++)
            if ((late >> u) & 1u)
              if (chip_take(a.P, sh[hk0 + hstep * u].x, h[u], tag)) late &= ~(1u << u);
          if (late && !clk.go_on(a.wait_ns)) {
            S.fail = 1;
            atomicExch(a.err, 1);
            break;
          }
        } while (late);
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
      const VT bv = (VT)S.beta;
#pragma unroll
      for (int j = 0; j < RJ; j++)
        if (t + kChipThreads * j < nr) P(pos[j]) = add_rn(mul_rn(bv, P(pos[j])), r[j]);
#pragma unroll
      for (int u = 0; u < kChipHalo; u++) {
        const int k = hk0 + hstep * u;
        if (hstep * u < nh && k >= 0 && k < nh) {
          const int2 e = sh[k];
          if (e.x >= 0) P(e.y) = add_rn(mul_rn(bv, P(e.y)), h[u]);
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
    const int code = S.code;
    VT *xo = (VT *)a.x;
    if (xw || a.whole) {
      VT xv[RJ];
      if constexpr (kXT) {
        CV::get(tx, xv);
      } else {
#pragma unroll
        for (int j = 0; j < RJ; j++) xv[j] = x[j];
      }
#pragma unroll
      for (int j = 0; j < RJ; j++) {
        const int li = t + kChipThreads * j;
        if (li < nr) __stcg(xo + row[j], xv[j]);
      }
    }
    if (lead) {
      st->k.s[S_ALPHA] = S.alpha;
      st->k.s[S_BETA] = S.beta;
      st->k.s[S_RR] = S.rr;
      if (a.whole) {
        st->k.loop = top;
        st->k.hlen = hlen;
        set_done(st, code == kRunning ? kMaxLoop : code);
      } else {  // the state the kernel-per-step inner loop leaves (nothing pending)
        st->k.done = code == kRunning ? kMaxLoop : code;
        st->k.loop = code == kBreakdown || code == kNaN ? L : L + 1;
        st->k.aux[A_PENDING] = 0;
        st->k.aux[A_XZERO] = xw ? 0 : 1;
      }
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

// Launch shape: RJ rows per thread (a power of two, 8 in FP64 and 16 in FP32
// at most) on as many CTAs as the rows keep busy. Up to kChipDirect CTAs the
// grid reductions poll their slots directly and are 0.3-0.4 us cheaper each:
// 512 rows per CTA until that many are in use, then more rows on the same
// number up to 2,048 (65,536 rows), then one CTA per SM. Measured, us per CG
// iteration (FP64, r always with tags): 112^2 on 13 / 25 / 49 CTAs 3.57 / 3.39 / 4.17, 150^2 on 22
// / 30 / 44 3.52 / 3.52 / 4.30, 256^2 on 32 / 64 / 128 3.91 / 4.51 / 4.29,
// 333^2 on 55 / 109 / 148 5.07 / 4.66 / 4.72.
inline long long chip_ctas(long long n, long long sms) {
  long long G = (n + kChipThreads - 1) / kChipThreads;
  if (G > (long long)kChipDirect) G = n <= 2048LL * kChipDirect ? (long long)kChipDirect : sms;
  return std::max<long long>(1, std::min(G, sms));
}

struct ChipShape {
  int G = 0, rpc = 0, rj = 0, tile = 0;
  int hl = 0, hu = 0, hl2 = 0, hu2 = 0;
  int nx = 0, ny = 0, nz = 0, by = 0, bz = 0, gy = 0;
  int elems = 0;
  size_t smem = 0;
};

// False where the matrix or p with its halo does not fit on chip.
template <class VT>
inline bool chip_shape(const ks_ctx *ctx, const CsrDev &A, long long n, ChipShape *s) {
  constexpr int kMaxRows = (sizeof(VT) == 8 ? 8 : 16) * kChipThreads;
  const long long sms = std::min(ctx->num_sms, (int)kChipMaxGrid);
  if (n < 1 || !A.dia_nd || A.dia_cmin != 0 || A.dia_cmax != n || n > sms * kMaxRows) return false;
  int optin = 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  *s = ChipShape{};
  const long long G0 = chip_ctas(n, sms);
  long long rows = 0;
  if (A.dia_box) {
    // the tile with the least work: its rows, plus half a row for each of the
    // halo's (fetched in the shadow of a reduction). Only heights that leave no more
    // than G0 tiles in y and whose plane fits: the lines of a long box can be many
    s->nx = A.dia_off[5];
    s->ny = A.dia_off[6] / s->nx;
    s->nz = (int)(n / A.dia_off[6]);
    double best = 0.0;
    const int top = std::min(s->ny, kMaxRows / s->nx);
    for (int by = (int)((s->ny + G0 - 1) / G0); by <= top; by++) {
      const int gy = (s->ny + by - 1) / by;
      const int bz = (int)((s->nz + G0 / gy - 1) / (G0 / gy));
      const double cost = (double)s->nx * ((double)by * bz + (by + bz));
      if ((long long)s->nx * by * bz > kMaxRows || (best > 0.0 && cost >= best)) continue;
      best = cost;
      s->by = by;
      s->bz = bz;
      s->gy = gy;
    }
    if (best > 0.0) {
      s->tile = 1;
      s->G = s->gy * ((s->nz + s->bz - 1) / s->bz);
      rows = (long long)s->nx * s->by * s->bz;
      s->rpc = (int)rows;
      s->elems = 2 + s->nx * (s->by + 2) * (s->bz + 2);
    }
  }
  if (!s->tile) {
    rows = ((n + G0 - 1) / G0 + 31) / 32 * 32;
    s->rpc = (int)rows;
    s->G = (int)((n + rows - 1) / rows);
    for (int k = 0; k < A.dia_nd; k++) {  // ascending offsets
      const int o = A.dia_off[k];
      if (o < 0) {
        if (k == 0) s->hl = -o;
        if (k == 1) s->hl2 = -o;
      } else if (o > 0) {
        s->hu2 = s->hu;
        s->hu = o;
      }
    }
  }
  s->rj = 1;
  while ((long long)s->rj * kChipThreads < rows) s->rj *= 2;
  if (s->rj * kChipThreads > kMaxRows) return false;
  long long halo = 0;  // ChipRows::halo() at most
  if (s->tile) {
    halo = 2LL * s->nx * (s->by + s->bz);
  } else {
    halo = (s->hl2 < s->hl ? std::min<long long>(rows, s->hl - s->hl2) : 0) + s->hl2 +
           (s->hu2 < s->hu ? std::min<long long>(rows, s->hu - s->hu2) : 0) + s->hu2;
    s->elems = s->hl + (int)rows + s->hu;
  }
  if (halo > kChipHalo * kChipThreads) return false;
  if (s->rj <= 2 && halo > kChipHalo * (kChipThreads - 32)) return false;
  s->smem = sizeof(VT) * (size_t)s->elems + sizeof(int2) * (size_t)halo;
  return s->smem + 2048 <= (size_t)optin;  // + the static arrays
}

// Bytes of R, the published r with its tags.
template <class VT>
inline size_t chip_r_bytes(long long n) {
  return 2 * sizeof(VT) * (size_t)n;
}

template <class VT, class MT>
inline ChipArgs chip_args(const CsrDev &A, const IrArgs &ir, const ChipShape &sh, unsigned long long tag0) {
  ChipArgs a{};
  static_cast<IrArgs &>(a) = ir;
  a.n = A.n;
  a.rpc = sh.rpc;
  const DiaT<MT> D = dview<MT>(A);
  for (int k = 0; k < kMaxDiag; k++) {
    a.vb[k] = D.vb[k];
    a.vs[k] = D.vs[k];
    a.off[k] = D.off[k];
  }
  a.nd = D.nd;
  a.bf16 = std::is_same<MT, __nv_bfloat16>::value ? 1 : 0;
  a.smem_elems = sh.elems;
  a.tag0 = tag0;
  a.hl = sh.hl, a.hu = sh.hu, a.hl2 = sh.hl2, a.hu2 = sh.hu2;
  a.nx = sh.nx, a.ny = sh.ny, a.nz = sh.nz, a.by = sh.by, a.bz = sh.bz, a.gy = sh.gy;
  return a;
}

// One launch (`probe`: only check that the grid can be co-resident, *fits);
// `cls`: its class in a profiled solve. ks_chip_cg.cu.
cudaError_t chip_launch_f64(ks_ctx *ctx, const ChipArgs &a, const ChipShape &sh, bool probe, bool *fits, int cls);
cudaError_t chip_launch_f32(ks_ctx *ctx, const ChipArgs &a, const ChipShape &sh, bool probe, bool *fits, int cls);
template <class VT>
inline cudaError_t chip_launch(ks_ctx *ctx, const ChipArgs &a, const ChipShape &sh, bool probe, bool *fits, int cls) {
  return sizeof(VT) == 8 ? chip_launch_f64(ctx, a, sh, probe, fits, cls) : chip_launch_f32(ctx, a, sh, probe, fits, cls);
}

// ---------------------------------------------------------------- CG on tiles
// Shape and launch of k_cg_tile (ks_tile_cg.cuh).
constexpr int kTileRows = 32;  // rows per thread: 64 words of TMEM each for r and x
constexpr int kTileHaloThreads = kChipThreads - 32;  // warps 1 .. 15
constexpr int kTileHaloZ = 3, kTileHaloY = 4;  // columns of a z face, rows of a y face per thread of them at most

// The tile with the least work (the rows its threads walk, plus half a row for
// each of the halo's) on at most one CTA per SM; false where none fits on chip or a
// value is not finite.
inline bool tile_shape(const ks_ctx *ctx, const CsrDev &A, long long n, ChipShape *s) {
  const long long sms = std::min(ctx->num_sms, (int)kChipMaxGrid);
  if (A.dia_box < 2 || !A.dia_cst || A.dia_cmin != 0 || A.dia_cmax != n || n > sms * kTileRows * kChipThreads) return false;
  // an absent entry's term is its diagonal's value times a zero: NaN where the value is not finite
  for (int k = 0; k < 7; k++)
    if (!std::isfinite(A.dia_cv[k])) return false;
  int optin = 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  *s = ChipShape{};
  s->tile = 1;
  s->nx = A.dia_off[5];
  s->ny = A.dia_off[6] / s->nx;
  s->nz = (int)(n / A.dia_off[6]);
  double best = 0.0;
  const int top = std::min(s->ny, kTileHaloZ * kTileHaloThreads / s->nx);  // as chip_shape
  for (int by = (int)((s->ny + sms - 1) / sms); by <= top; by++) {
    const long long gy = (s->ny + by - 1) / by;
    const long long bz = (s->nz + sms / gy - 1) / (sms / gy);
    const long long elems = 2 + (long long)(s->nx + 1) * (by + 2) * (bz + 2);
    const long long halo = 2LL * s->nx * (by + bz), cols = ((long long)s->nx * by + kChipThreads - 1) / kChipThreads;
    const double cost = (double)(cols * ((bz + 7) / 8 * 8)) * kChipThreads + 0.5 * (double)halo;
    if (cols * ((bz + 7) / 8 * 8) > kTileRows || s->nx * bz > kTileHaloY * kTileHaloThreads || elems > (1 << 20) ||
        sizeof(double) * (size_t)elems + 2048 > (size_t)optin || (best > 0.0 && cost >= best))
      continue;
    best = cost;
    s->by = by;
    s->bz = (int)bz;
    s->gy = (int)gy;
    s->elems = (int)elems;
    s->smem = sizeof(double) * (size_t)elems;
  }
  if (best == 0.0) return false;
  s->G = s->gy * ((s->nz + s->bz - 1) / s->bz);
  return true;
}

// One launch (`probe`: only check that the grid can be co-resident, *fits);
// `cls`: its class in a profiled solve. ks_chip_cg.cu.
cudaError_t tile_launch(ks_ctx *ctx, const CsrDev &A, const ChipArgs &a, const ChipShape &sh, bool probe, bool *fits,
                        int cls);

// ---------------------------------------------------------------- CG, CSR
// Shape and launch of k_cg_csr (ks_csr_cg.cuh).
constexpr int kCsrRows = 4;  // rows per thread at most (of 512 threads, above 2,048 rows per CTA of 1,024)

struct CsrCgArgs : IrArgs {  // P is the array R of published r
  const int *ptr, *slice;
  const double *val;
  const short *off;
  int wl, wu;
};

struct CsrShape : ChipShape {
  int threads = 0;
  int wl = 0, wu = 0;
};

// The CTAs of chip_ctas, whose steps were measured with the matrix in TMEM; here more
// CTAs below 65,536 rows would pay too (rows of 14 entries, us per iteration: 65,000
// rows on 32 CTAs 12.5, 66,000 on 148 7.6). lo, hi: the matrix's largest offsets.
// False where the window does not fit.
inline bool csr_shape(const ks_ctx *ctx, long long n, int lo, int hi, CsrShape *s) {
  const long long sms = std::min(ctx->num_sms, (int)kChipMaxGrid);
  if (n < 1 || n > sms * kCsrRows * 1024) return false;
  int optin = 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  *s = CsrShape{};
  const long long G = chip_ctas(n, sms);
  s->rpc = (int)(((n + G - 1) / G + 31) / 32 * 32);
  s->G = (int)((n + s->rpc - 1) / s->rpc);
  s->rj = 1;
  s->threads = s->rpc <= kCsrRows * 512 ? 512 : 1024;
  while (s->rj * s->threads < s->rpc) s->rj *= 2;
  s->wl = lo;
  s->wu = hi;
  s->smem = sizeof(double) * ((size_t)s->rpc + s->wl + s->wu);
  return s->rj <= kCsrRows && s->smem + 2048 <= (size_t)optin;
}

cudaError_t csr_launch(ks_ctx *ctx, const CsrCgArgs &a, const CsrShape &sh, bool probe, bool *fits, int cls);

}  // namespace ks
