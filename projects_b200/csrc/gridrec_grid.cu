// Gridding for chunks of several slice pairs (sm_100a): the 4 x 4 sub-tile kernel, its
// tap records and the reduction of split sub-tiles.  The tile kernel for one or two
// pairs and the tensor-core kernel are in gridrec_kernels.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "gr_device.cuh"
#include "gr_internal.h"

namespace gr {

// ------------------------------------------------------------------ gridding by groups of pairs
// The same gather as grid_kernel -- the work-list geometry, tap set and
// nearest-neighbour weights of gridrec.cu:546-566 -- for chunks of a few slice pairs.
// A work item is one kWideRows x kWideCols (4 x 8) sub-tile of H and the samples whose
// taps reach it.  A warp grids for G pairs either a bundle of Q = 32 / (G RS) items of similar
// length at once -- RS lanes hold pair p's cells of item q in registers, 4 / RS rows each --
// or one long item, lane q * G + p holding pair p's G cells q * G .. of it:
// * no shared-memory read-modify-write, no atomics, no idle lanes for few pairs; per sample
//   a tap adds w_c (w_r value) by packed FMAs over pairs of columns, real and imaginary
//   parts apart, so that the column weights are used as they lie in shared memory.
// * a bundle reads a sample's weights once for 32 cells of its lane (RS = 1), a long item once for
//   G cells: about a quarter slower per sample at G = 8, but a long item's samples pass 3 to
//   4 times as fast, and no warp holds one when the others have ended.
// * the geometry depends on the plan only: tap_record_kernel computes, once per work list, a
//   32-byte record per (sub-tile, sample) that has a tap there: the 12 table indices and the
//   sample's place in the spectra.  A warp loads 32 records at once (a batch ahead), looks
//   the weights up in a shared copy of the table and leaves them in shared memory (the lanes
//   of a group broadcast).
// * the spectra lie as [direction][j / 4][pair][j % 4]; the lanes copy their samples' values
//   to shared memory by cp.async, a batch ahead.
// Positions, indices and rounding of a tap are those of grid_kernel, and a cell sums its
// taps in the order of the list the records are made from, split items included: with
// the tile kernel's list the results are that kernel's bit for bit, with the 16-pair
// kernel's list that one's.
// Bound by the FMA issue (16 packed FMAs of 2 cycles per pair, sub-tile and sample) for 8
// pairs, more and more by the table lookups for fewer.  Gridding at 2048 x 1500 (7.1 M
// records, 32 MB of spectra a pair): 35.3 us a pair for 8 pairs, 71.0 with the 16-pair
// kernel; at 512 x 360 36 us for one pair, 84 with the tile kernel, whose longest tile (a
// chain of 2048 samples) ends long after the others.

constexpr int kGrpWarps = 4;
constexpr int kGrpRow = 48;                        // a sample's 12 weights
constexpr int kGrpZeroRow = 32;                    // a row of zero weights (items that have ended)
constexpr int kGrpWtBytes = (kGrpZeroRow + 1) * kGrpRow;
// the weights, then two batches of values
template <int G>
__host__ __device__ constexpr int grp_warp_bytes() {
  return kGrpWtBytes + 2 * G * 32 * 8;  // the weights, then two batches of values
}
static_assert(kWideRows == 4 && kWideCols == 8, "record layout");

__host__ __device__ constexpr int grp_table_bytes(int ltbl) { return ((ltbl + 2) * 4 + 15) & ~15; }

__device__ __forceinline__ void cp_async8(void* dst_smem, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_u32(dst_smem)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}
// 32 bytes (32-byte aligned, read-only for the kernel) in one load
__device__ __forceinline__ void ldg256(unsigned (&v)[8], const void* p) {
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
      : "l"(p));
}

// Sub-tile `sub` of list tile `tile`: its index among the 4 x 8 tiles, or -1 outside H.
__device__ __forceinline__ int sub_tile(const GridArgs& a, int tile, int sub, int subs) {
  if (subs == 1) return tile;
  const int tu = tile / a.tiles_v, tv = tile - (tile / a.tiles_v) * a.tiles_v;
  constexpr int kSubRows = kTile / kWideRows, kSubCols = kTile / kWideCols;
  const int p = tu * kSubRows + sub / kSubCols, q = tv * kSubCols + sub % kSubCols;
  return p * kWideRows < a.M && q * kWideCols < a.M ? p * (a.M / kWideCols) + q : -1;
}

// The records of a work list (once per list): a.items and a.runs are its items and runs,
// over 32 x 32 tiles (subs = 32, one warp per sub-tile of an item) or 4 x 8 tiles (subs =
// 1).  The samples of a run are taken in the order in which grid_kernel takes them with
// spw samples per step (spw = 32 and run.P = 1: ascending), and kept where a tap falls
// inside the sub-tile.  With rec null it only counts (counts[item * subs + sub], -1
// outside H), else it writes the records at base[...].
__global__ void __launch_bounds__(128) tap_record_kernel(GridArgs a, int subs, int spw, int* counts,
                                                         const int* base, TapRec* rec) {
  const int id = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (id >= a.n_items * subs) return;
  const Item it = a.items[id / subs];
  const int tile = sub_tile(a, it.tile, id % subs, subs);
  if (tile < 0) {
    if (!rec && lane == 0) counts[id] = -1;
    return;
  }
  const int tiles_v = a.M / kWideCols;
  const int p0 = tile / tiles_v * kWideRows, q0 = (tile - tile / tiles_v * tiles_v) * kWideCols;
  // positions as grid_kernel forms them (FP64, relative to the enclosing 32 x 32
  // tile), moved to the sub-tile by an integer
  const double offu = (double)(a.M / 2 - (p0 & ~(kTile - 1))), subu = (double)(p0 & (kTile - 1));
  const double offv = (double)(a.M / 2 - (q0 & ~(kTile - 1))), subv = (double)(q0 & (kTile - 1));
  const double L2d = a.L2, tsd = a.tblspcg;
  const unsigned zero = (unsigned)(a.ltbl + 1);
  const int phs = 32 / spw;  // steps taken at once: lane ph * spw + slot
  const int lph = lane / spw, lslot = lane - lph * spw;
  int at = rec ? base[id] : 0;
  for (int r = it.run_begin; r < it.run_end; ++r) {
    const Run run = a.runs[r];
    const double2 d = a.dir[run.dir];
    // the run's samples lie between its ends: skip it where they pass the sub-tile by
    const double ua = fma((double)run.jlo, d.x, offu) - subu, ub = fma((double)run.jhi, d.x, offu) - subu;
    const double va = fma((double)run.jlo, d.y, offv) - subv, vb = fma((double)run.jhi, d.y, offv) - subv;
    if (fmax(ua, ub) < -L2d || fmin(ua, ub) > kWideRows - 1 + L2d || fmax(va, vb) < -L2d ||
        fmin(va, vb) > kWideCols - 1 + L2d)
      continue;
    for (int blk = run.jlo; blk <= run.jhi; blk += spw * run.P) {
      for (int ph = 0; ph < run.P && blk + ph <= run.jhi; ph += phs) {
        const int j = blk + ph + lph + run.P * lslot;
        unsigned ix[kWideRows + kWideCols];
        bool row = false, col = false;
        const double u = fma((double)j, d.x, offu) - subu, v = fma((double)j, d.y, offv) - subv;
#pragma unroll
        for (int k = 0; k < kWideRows; ++k) {
          const double dd = fabs(u - (double)k);
          row = row || dd <= L2d;
          ix[k] = dd <= L2d ? (unsigned)min(table_index64(dd, tsd), a.ltbl) : zero;
        }
#pragma unroll
        for (int k = 0; k < kWideCols; ++k) {
          const double dd = fabs(v - (double)k);
          col = col || dd <= L2d;
          ix[kWideRows + k] = dd <= L2d ? (unsigned)min(table_index64(dd, tsd), a.ltbl) : zero;
        }
        const bool keep = lph < phs && ph + lph < run.P && j <= run.jhi && row && col;
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (rec && keep) {
          const unsigned place = (unsigned)(run.dir * (a.J >> 2) + (j >> 2)) * 4u + (unsigned)(j & 3);
          uint4* o = reinterpret_cast<uint4*>(rec + at + __popc(m & ((1u << lane) - 1u)));
          o[0] = make_uint4(ix[0] | ix[1] << 16, ix[2] | ix[3] << 16, ix[4] | ix[5] << 16, ix[6] | ix[7] << 16);
          o[1] = make_uint4(ix[8] | ix[9] << 16, ix[10] | ix[11] << 16, place, 0u);
        }
        at += __popc(m);
      }
    }
  }
  if (!rec && lane == 0) counts[id] = at;
}

// Four complex cells: 32 bytes, one sector.
__device__ __forceinline__ void stg256(void* p, float2 c0, float2 c1, float2 c2, float2 c3) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(c0.x), "f"(c0.y),
               "f"(c1.x), "f"(c1.y), "f"(c2.x), "f"(c2.y), "f"(c3.x), "f"(c3.y)
               : "memory");
}

// A pair of columns of one row: (re, re), (im, im) of cells 2 c2 and 2 c2 + 1.
struct GrpCell2 {
  float2 re, im;
};

// One sample on this lane's R rows: x_r = w_r * value, then acc += w_c x_r; wts: the weights
// of rows 0..3, then columns 0..7; row0: the first of the lane's rows.
template <int R>
__device__ __forceinline__ void grp_apply(GrpCell2 (&acc)[R][kWideCols / 2], float2 v,
                                          const unsigned char* wts, int row0) {
  const float4* d = reinterpret_cast<const float4*>(wts);
  float wr[4];
  if (R == 4) {
    const float4 rw = d[0];
    wr[0] = rw.x, wr[1] = rw.y, wr[2] = rw.z, wr[3] = rw.w;
  } else {
    wr[0] = reinterpret_cast<const float*>(wts)[row0];
  }
  const float4 c0 = d[1], c1 = d[2];
  const float2 wc[4] = {make_float2(c0.x, c0.y), make_float2(c0.z, c0.w), make_float2(c1.x, c1.y),
                        make_float2(c1.z, c1.w)};
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float xr = __fmul_rn(wr[r], v.x), xi = __fmul_rn(wr[r], v.y);
    const float2 x2 = make_float2(xr, xr), y2 = make_float2(xi, xi);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      acc[r][c].re = __ffma2_rn(wc[c], x2, acc[r][c].re);
      acc[r][c].im = __ffma2_rn(wc[c], y2, acc[r][c].im);
    }
  }
}

// One sample of a long item: this lane's G cells (a row, half a row, a pair or a cell).
template <int G>
__device__ __forceinline__ void grp_apply_cells(float2 (&re)[(G + 1) / 2], float2 (&im)[(G + 1) / 2],
                                                float2 v, float wr, const float* wc) {
  const float xr = __fmul_rn(wr, v.x), xi = __fmul_rn(wr, v.y);
  if (G == 1) {
    re[0].x = __fmaf_rn(wc[0], xr, re[0].x);
    im[0].x = __fmaf_rn(wc[0], xi, im[0].x);
    return;
  }
  float w[G];
  if (G >= 4) {
#pragma unroll
    for (int c = 0; c < G; c += 4) {
      const float4 t = *reinterpret_cast<const float4*>(wc + c);
      w[c] = t.x, w[(c + 1) % G] = t.y, w[(c + 2) % G] = t.z, w[(c + 3) % G] = t.w;
    }
  } else {
    const float2 t = *reinterpret_cast<const float2*>(wc);
    w[0] = t.x, w[1 % G] = t.y;
  }
#pragma unroll
  for (int c = 0; c < G / 2; ++c) {
    const float2 wp = make_float2(w[2 * c], w[2 * c + 1]);
    re[c] = __ffma2_rn(wp, make_float2(xr, xr), re[c]);
    im[c] = __ffma2_rn(wp, make_float2(xi, xi), im[c]);
  }
}

// Writes the N complex cells from column q0 of row `row` of H at `o`; row and column 0
// of H stay zero.
template <int N>
__device__ __forceinline__ void grp_store(float2* o, int row, int q0, const float2* re, const float2* im) {
  float2 c[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    c[k] = k & 1 ? make_float2(re[k / 2].y, im[k / 2].y) : make_float2(re[k / 2].x, im[k / 2].x);
    if (row == 0 || (k == 0 && q0 == 0)) c[k] = make_float2(0.f, 0.f);
  }
  if (N >= 4) {
#pragma unroll
    for (int k = 0; k + 3 < N; k += 4) stg256(o + k, c[k], c[k + 1], c[k + 2], c[k + 3]);
  } else if (N == 2) {
    *reinterpret_cast<float4*>(o) = make_float4(c[0].x, c[0].y, c[N - 1].x, c[N - 1].y);
  } else {
    *o = c[0];
  }
}

template <int G, int RS>
__global__ void __launch_bounds__(kGrpWarps * 32, kGrpMinBlocks) grid_group_kernel(GridArgs a) {
  constexpr int TR = kWideRows, TC = kWideCols;
  constexpr int LI = G * RS, Q = 32 / LI, R = TR / RS;  // lanes per item of a bundle, items, rows per lane
  constexpr int S1 = LI;                                // steps of a bundle's batch
  extern __shared__ __align__(16) unsigned char smg[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* tbl = reinterpret_cast<float*>(smg);  // the table, then a zero
  unsigned char* wb = smg + grp_table_bytes(a.ltbl) + warp * grp_warp_bytes<G>();
  for (int i = threadIdx.x; i <= a.ltbl; i += blockDim.x) tbl[i] = __ldg(&a.wtbl[i]);
  if (threadIdx.x == 0) tbl[a.ltbl + 1] = 0.f;
  if (lane < kGrpRow / 16)
    *reinterpret_cast<uint4*>(wb + kGrpZeroRow * kGrpRow + lane * 16) = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const int p = lane & (G - 1), q = lane / LI;   // this lane's pair and item
  const int row0 = lane / G % RS * R;            // and the first of its rows
  const int rq = lane % Q, rt = lane / Q;        // item and step whose record it expands
  const int crow = lane / G / (TC / G), ccol = lane / G % (TC / G) * G;  // its cells of a long item
  // the list begins with the n_long long items
  const unsigned total = (unsigned)a.n_long + (unsigned)(a.n_items - a.n_long + Q - 1) / Q;
  const unsigned char* spec = reinterpret_cast<const unsigned char*>(a.spec) + p * 32;
  const size_t MM = (size_t)a.M * a.M;
  // Warps take a long item or a bundle of Q items from a queue: the next one is read and
  // the entry after it requested while the current one is gridded, and the first records
  // and values of the next batch (of this bundle or the next) while the current batch is
  // applied.
  unsigned wreq = 0;
  auto request = [&]() {
    if (lane == 0) wreq = atomicAdd(a.queue, 1u);
  };
  // this lane's item; 0: none left, 1: a bundle, 2: a long item
  auto take = [&](Item& it) -> int {
    const unsigned w = __shfl_sync(0xffffffffu, wreq, 0);
    it = Item{0, 0, 0, -2};
    if (w >= total) return 0;
    request();
    const bool lng = w < (unsigned)a.n_long;
    const unsigned i = lng ? w : a.n_long + (w - a.n_long) * Q + q;
    if (i < (unsigned)a.n_items) it = a.items[i];
    return lng ? 2 : 1;
  };
  unsigned rec[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};  // this lane's record of the next batch
  float2* vals = reinterpret_cast<float2*>(wb + kGrpWtBytes);
  int vbuf = 0;  // which of the two value buffers holds the next batch
  // A batch is S1 steps of the items of a bundle, or 32 samples of a long item: 32 records.
  // rb, rn: first record and count of the item whose record this lane expands (the long
  // item, or item rq).
  auto load_rec = [&](int kind, int rb, int rn, int tb) {
    const int t = tb + (kind == 2 ? lane : rt);
    if (t < rn) ldg256(rec, a.rec + rb + t);
  };
  // pair p of the samples whose records lanes lane / G, 32 / G + lane / G, ... hold: step i / Q
  // of item i % Q for the record of lane i, or sample i of a long item
  auto load_values = [&](int kind, int cnt, int tb) {
    const int n = RS == 1 ? cnt : __shfl_sync(0xffffffffu, cnt, lane / G % Q * LI);
#pragma unroll
    for (int k = 0; k < G; ++k) {
      const int i = k * (32 / G) + lane / G;
      const unsigned pl = __shfl_sync(0xffffffffu, rec[6], i);
      if (tb + (kind == 2 ? i : i / Q) < n)
        cp_async8(vals + (vbuf * G + k) * 32 + lane, spec + (size_t)(pl >> 2) * (G * 32) + (pl & 3u) * 8);
    }
    cp_async_commit();
  };
  request();
  Item it, nit;
  int kind = take(it);
  if (kind == 0) return;
  int cnt = it.run_end - it.run_begin;
  int rb = __shfl_sync(0xffffffffu, it.run_begin, rq * LI), rn = __shfl_sync(0xffffffffu, cnt, rq * LI);
  load_rec(kind, rb, rn, 0);
  load_values(kind, cnt, 0);
  for (;;) {
    const int nkind = take(nit);
    const int tile = it.tile, slot = it.slot;
    const int ncnt = nit.run_end - nit.run_begin;
    // A sub-tile that no sample reaches has an empty item: its cells are written as zeros.
    const int nt = max(1, __reduce_max_sync(0xffffffffu, cnt));
    const int S = kind == 2 ? 32 : S1;
    // start of a batch: this batch's weights (lane i expands the record it holds), the
    // next batch's records; its values, later, when those are there
    auto begin = [&](int tb) {
      cp_async_wait_all();  // this lane's values of the batch
      if (tb + (kind == 2 ? lane : rt) < rn) {
        float wt[12];
#pragma unroll
        for (int e = 0; e < 12; ++e) wt[e] = tbl[(e & 1) ? rec[e >> 1] >> 16 : rec[e >> 1] & 0xffffu];
        float4* o = reinterpret_cast<float4*>(wb + lane * kGrpRow);
#pragma unroll
        for (int e = 0; e < 3; ++e) o[e] = make_float4(wt[4 * e], wt[4 * e + 1], wt[4 * e + 2], wt[4 * e + 3]);
      }
      const bool last = tb + S >= nt;
      if (last) {  // the next batch is the next bundle's first
        rb = __shfl_sync(0xffffffffu, nit.run_begin, rq * LI);
        rn = __shfl_sync(0xffffffffu, ncnt, rq * LI);
      }
      load_rec(last ? nkind : kind, rb, rn, last ? 0 : tb + S);
      __syncwarp();
      vbuf ^= 1;
    };
    auto middle = [&](int tb) {
      const bool last = tb + S >= nt;
      load_values(last ? nkind : kind, last ? ncnt : cnt, last ? 0 : tb + S);
    };
    const int tu = tile / a.tiles_v, tv = tile - (tile / a.tiles_v) * a.tiles_v;
    float2* Ht = a.H + (size_t)p * MM + (size_t)(tu * TR) * a.M + tv * TC;  // this lane's pair
    // partial sub-tile of a split one: [cell][pair], summed by split_reduce_group_kernel
    float2* part = reinterpret_cast<float2*>(a.scratch) + (size_t)max(slot, 0) * (TR * TC * G) + p;
    if (kind == 2) {
      float2 re[(G + 1) / 2], im[(G + 1) / 2];
#pragma unroll
      for (int c = 0; c < (G + 1) / 2; ++c) re[c] = im[c] = make_float2(0.f, 0.f);
      for (int tb = 0; tb < nt; tb += 32) {
        begin(tb);
        const float2* vv = vals + (vbuf ^ 1) * G * 32 + p;
        const float* w = reinterpret_cast<const float*>(wb);
        const int n = min(32, cnt - tb), half = n >> 1;
#pragma unroll 4
        for (int t = 0; t < half; ++t)
          grp_apply_cells<G>(re, im, vv[t * G], w[t * (kGrpRow / 4) + crow], w + t * (kGrpRow / 4) + TR + ccol);
        middle(tb);
#pragma unroll 4
        for (int t = half; t < n; ++t)
          grp_apply_cells<G>(re, im, vv[t * G], w[t * (kGrpRow / 4) + crow], w + t * (kGrpRow / 4) + TR + ccol);
        __syncwarp();  // weights and values are read before they are replaced
      }
      if (slot >= 0) {
#pragma unroll
        for (int c = 0; c < G; ++c)
          part[(crow * TC + ccol + c) * G] = c & 1 ? make_float2(re[c / 2].y, im[c / 2].y)
                                                   : make_float2(re[c / 2].x, im[c / 2].x);
      } else if (p < a.pairs) {
        grp_store<G>(Ht + (size_t)crow * a.M + ccol, tu * TR + crow, tv * TC + ccol, re, im);
      }
    } else {
      GrpCell2 acc[R][TC / 2];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < TC / 2; ++c) acc[r][c].re = acc[r][c].im = make_float2(0.f, 0.f);
      for (int tb = 0; tb < nt; tb += S1) {
        begin(tb);
        const float2* vv = vals + (vbuf ^ 1) * G * 32 + q * G + p;
        const unsigned char* d = wb + q * kGrpRow;
        const int n = min(S1, nt - tb), half = n >> 1;
        auto step = [&](int t) {
          const bool in = tb + t < cnt;
          grp_apply<R>(acc, in ? vv[t * Q * G] : make_float2(0.f, 0.f),
                       in ? d + t * Q * kGrpRow : wb + kGrpZeroRow * kGrpRow, row0);
        };
        for (int t = 0; t < half; ++t) step(t);
        middle(tb);
        for (int t = half; t < n; ++t) step(t);
        __syncwarp();  // weights and values are read before they are replaced
      }
      if (slot >= 0) {
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = 0; c < TC / 2; ++c) {
            part[((row0 + r) * TC + 2 * c) * G] = make_float2(acc[r][c].re.x, acc[r][c].im.x);
            part[((row0 + r) * TC + 2 * c + 1) * G] = make_float2(acc[r][c].re.y, acc[r][c].im.y);
          }
      } else if (slot == -1 && p < a.pairs) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float2 re[TC / 2], im[TC / 2];
#pragma unroll
          for (int c = 0; c < TC / 2; ++c) re[c] = acc[r][c].re, im[c] = acc[r][c].im;
          grp_store<TC>(Ht + (size_t)(row0 + r) * a.M, tu * TR + row0 + r, tv * TC, re, im);
        }
      }
    }
    if (nkind == 0) break;
    it = nit;
    kind = nkind;
    cnt = ncnt;
  }
  cp_async_wait_all();
}

// Sums the partial sub-tiles of every split sub-tile in slot order and writes H.
// Grid: (split sub-tiles, groups of G pairs); 256 threads over (cell, pair).
__global__ void __launch_bounds__(256) split_reduce_group_kernel(GridArgs a, int G) {
  const int4 sp = a.split_list[blockIdx.x];  // (tile, slot0, nsplit, slots apart)
  const int tu = sp.x / a.tiles_v, tv = sp.x - (sp.x / a.tiles_v) * a.tiles_v;
  const int p0 = tu * kWideRows, q0 = tv * kWideCols;
  const int n = kWideRows * kWideCols * G;
  const float2* base = reinterpret_cast<const float2*>(a.scratch) + (size_t)sp.y * n;
  const size_t MM = (size_t)a.M * a.M;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int cell = i / G, l = i - (i / G) * G;
    if (l >= a.pairs) continue;
    float2 sum = make_float2(0.f, 0.f);
    for (int k = 0; k < sp.z; ++k) {
      const float2 v = __ldg(&base[(size_t)k * sp.w * n + i]);
      sum.x += v.x;
      sum.y += v.y;
    }
    const int p = p0 + cell / kWideCols, q = q0 + cell % kWideCols;
    if (p == 0 || q == 0) sum = make_float2(0.f, 0.f);
    a.H[(size_t)l * MM + (size_t)p * a.M + q] = sum;
  }
}

cudaError_t launch_tap_records(const GridArgs& a, int subs, int spw, int* counts, const int* base,
                               TapRec* rec, cudaStream_t s) {
  if (a.n_items == 0) return cudaSuccess;
  tap_record_kernel<<<(a.n_items * subs + 3) / 4, 128, 0, s>>>(a, subs, spw, counts, base, rec);
  return cudaGetLastError();
}

// The kernels whose shared memory may exceed the default limit (init_kernel_attributes).
void add_grid_kernels(std::vector<const void*>& f) {
  f.push_back((const void*)grid_group_kernel<8, grp_row_split(8)>);
  f.push_back((const void*)grid_group_kernel<4, grp_row_split(4)>);
  f.push_back((const void*)grid_group_kernel<2, grp_row_split(2)>);
  f.push_back((const void*)grid_group_kernel<1, grp_row_split(1)>);
}

template <int G>
static cudaError_t launch_grid_group_g(const GridArgs& a, cudaStream_t s) {
  constexpr int RS = grp_row_split(G), Q = 32 / (G * RS);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int smem = grp_table_bytes(a.ltbl) + kGrpWarps * grp_warp_bytes<G>();
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, grid_group_kernel<G, RS>, kGrpWarps * 32, smem);
  const long bundles = a.n_long + (a.n_items - a.n_long + Q - 1) / Q;
  const long want = (bundles + kGrpWarps - 1) / kGrpWarps;
  const int blocks = (int)std::min<long>(want, (long)std::max(per_sm, 1) * sms);
  grid_group_kernel<G, RS><<<blocks, kGrpWarps * 32, smem, s>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || a.n_split_tiles == 0) return e;
  split_reduce_group_kernel<<<a.n_split_tiles, 32 * G, 0, s>>>(a, G);
  return cudaGetLastError();
}

cudaError_t launch_grid_group(const GridArgs& a, int G, cudaStream_t s) {
  if (a.n_items == 0) return cudaSuccess;
  if (a.pairs > G) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(a.queue, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  switch (G) {
    case 8: return launch_grid_group_g<8>(a, s);
    case 4: return launch_grid_group_g<4>(a, s);
    case 2: return launch_grid_group_g<2>(a, s);
    case 1: return launch_grid_group_g<1>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gr
