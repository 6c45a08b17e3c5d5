// Sparse x dense: C += A * B, for one tile (spmm_wrapper,
// bcl/containers/algorithms/spgemm.hpp:80-96 and 140-149) and for the whole
// tile loop of BCL::gemm(SPMatrix, DMatrix, DMatrix&) (spgemm.hpp:153-179) in
// one launch.
//
// Layout: one warp per (group of 1, 2 or 4 rows of one C tile, column panel
// of 32 16-byte vectors: 128 FP32 / 256 BF16 columns); lane l owns one
// vector.  The group's A entries are flattened over rows and stages and put
// 32 at a time into a per-warp shared-memory table (B-row address, value,
// row); every lane then issues its 16-byte loads of the B rows (the warp
// reads whole 512-byte row segments), UNROLL entries' loads in flight before
// their multiply-adds are applied.  Rows with thousands of entries run in
// k_spmm_long beside it.
//
// Order: per output element the multiply-adds run in stored A-row order, and
// over the C tile's stages k = (k_ + i + j) mod G in that order, starting
// from the C value already stored (beta = 1, in place) — the reference's
// sequence, so FP32 results are bit-identical.  BF16 storage keeps the chain
// in FP32 registers and rounds each C element once when it is stored.
#include "common.cuh"

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <type_traits>
#include <vector>

namespace bclx {

constexpr int kSpmmWarps = 8;

template <typename ST>
struct Vec;

template <>
struct Vec<float> {
  static constexpr int N = 4;
  __device__ __forceinline__ static void load(const float* p, float* out) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
  }
  __device__ __forceinline__ static void load_c(const float* p, float* out) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
  }
  __device__ __forceinline__ static void store(float* p, const float* in) {
    *reinterpret_cast<float4*>(p) = make_float4(in[0], in[1], in[2], in[3]);
  }
  __device__ __forceinline__ static float to_f(float x) { return x; }
  __device__ __forceinline__ static float from_f(float x) { return x; }
  __device__ __forceinline__ static void unpack_raw(uint4 v, float* out) {
    out[0] = __uint_as_float(v.x); out[1] = __uint_as_float(v.y);
    out[2] = __uint_as_float(v.z); out[3] = __uint_as_float(v.w);
  }
};

template <>
struct Vec<__nv_bfloat16> {
  static constexpr int N = 8;
  __device__ __forceinline__ static void unpack(uint4 v, float* out) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
      out[2 * i] = __uint_as_float(w[i] << 16);
      out[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
  __device__ __forceinline__ static void load(const __nv_bfloat16* p, float* out) {
    unpack(__ldg(reinterpret_cast<const uint4*>(p)), out);
  }
  __device__ __forceinline__ static void load_c(const __nv_bfloat16* p, float* out) {
    unpack(*reinterpret_cast<const uint4*>(p), out);
  }
  __device__ __forceinline__ static void store(__nv_bfloat16* p, const float* in) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t lo = __bfloat16_as_ushort(__float2bfloat16_rn(in[2 * i]));
      const uint32_t hi = __bfloat16_as_ushort(__float2bfloat16_rn(in[2 * i + 1]));
      w[i] = lo | (hi << 16);
    }
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  __device__ __forceinline__ static float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
  __device__ __forceinline__ static __nv_bfloat16 from_f(float x) { return __float2bfloat16_rn(x); }
  __device__ __forceinline__ static void unpack_raw(uint4 v, float* out) { unpack(v, out); }
};

constexpr int kSpmmUnroll = 4;  // B-row loads in flight per lane (with 32 warps per SM)

constexpr int kSpmmMaxRows = 4;  // rows of one C tile a warp walks together

// A row that a warp walks alone asks L2 for the slices of its next 32 entries from
// kSpmmAhead entries (of up to 32 stages) on, where B is of kSpmmAheadBytes or more:
// its chain waits for each group of loads, and there are few such rows (asked for by
// every row they thrash L2, see spmm_rows).  R-MAT of 400,000 x 256 on 40 x 40 tiles,
// whose long rows have no kernel of their own, FP32 3.29 -> 2.74 ms, BF16 on 33 x 33
// 2.91 -> 2.60; R-MAT of 60,000 x 256 FP32 (61 MB) 626 -> 604 us, BF16 (31 MB, in L2 as
// it is) 549 -> 591.
constexpr int kSpmmAhead = 256;
constexpr int64_t kSpmmAheadBytes = 48 << 20;

// Per-warp shared memory of the walk:
//  * the entry table of a chunk of 32 entries: (B-row address, A value, row) of
//    each, read back with broadcast 16-byte loads;
//  * C staging: the C row slices the item updates (one 16-byte vector per
//    lane and row), copied by cp.async while the A and B loads are in flight.
__shared__ uint4 spmm_tables[kSpmmWarps * 32];
__shared__ uint4 spmm_cstage[kSpmmWarps * kSpmmMaxRows * 32];

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

// Copies without a compiler memory barrier, for the pipelined loops:
// there every earlier access to the target shared memory is ordered before the
// copy by a __syncwarp, and every later one after it by a wait (which is a
// barrier), so the loads around the copies may be scheduled freely.
__device__ __forceinline__ void cp_async16_nb(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}

__device__ __forceinline__ void cp_async4_nb(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem));
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// One stage of one row of C tile (ti, tj): for stage slot kk of the
// reference's rotated order k = (k_ + ti + tj) mod gk, the A-row segment of
// row r in tile (ti, k) and the B tile (k, tj).  Empty when !valid.
template <typename ST>
struct StageLane {
  int32_t alen;
  const int32_t* acol;
  const float* aval;
  const ST* bt;
};

template <typename ST, bool SUB>
__device__ __forceinline__ StageLane<ST> stage_lane(const SpGridView& A, const DGridView& B, int64_t ti, int64_t tj,
                                                    int64_t r, int64_t kk, bool valid) {
  StageLane<ST> s{0, nullptr, nullptr, nullptr};
  const int64_t gk = A.gn;
  if (valid && kk < gk) {
    // (tile and stage counts are below 2^31: a 32-bit division)
    const uint32_t rot = SUB ? (uint32_t)__ldg(B.rot_i + ti) + (uint32_t)__ldg(B.rot_j + tj) : (uint32_t)(ti + tj);
    const int64_t k = B.natural_order ? kk : ((uint32_t)kk + rot) % (uint32_t)gk;
    const bclx_csr_t At = A.tile(ti, k);
    const int32_t as = __ldg(At.row_ptr + r);
    s.alen = __ldg(At.row_ptr + r + 1) - as;
    s.acol = At.col_ind + as;
    s.aval = reinterpret_cast<const float*>(At.vals) + as;
    s.bt = reinterpret_cast<const ST*>(B.tile(k, tj));
  }
  return s;
}

// C tile (ti, tj) and every B tile of its column start on 16 bytes.
__device__ __forceinline__ bool tiles_aligned(const DGridView& B, const DGridView& C, int64_t ti, int64_t tj) {
  bool ok = (reinterpret_cast<uintptr_t>(C.tile(ti, tj)) & 15) == 0;
  for (int64_t k = lane_id(); k < B.gm; k += 32) ok &= (reinterpret_cast<uintptr_t>(B.tile(k, tj)) & 15) == 0;
  return __all_sync(kFull, ok);
}

// One warp per (R consecutive rows of C tile (ti, tj) from r0, panel of 32
// 16-byte vectors from column c0).  The A entries of the rows' stages are
// flattened (row by row, each row's stages in rotated order) and taken in
// chunks of 32, one entry per lane: each lane turns its entry into a table entry
// (B-row address, value, row) and loads its entry of the next chunk; the warp
// reads the table UNROLL entries at a time, so that many B-row loads (raw
// 16-byte vectors) are in flight before their multiply-adds are applied in
// entry order.  The loads in flight are what the registers of 32 warps per SM
// hold, 10 MB over the GPU, which is enough for DRAM.  Asking L2 for the B-row
// slices of the next two chunks as well put 155 MB in flight, more than L2: the
// lines were evicted before their use.  Without it, and without the A entries'
// staging through shared memory, uniform matrix of 1,000,000 rows x 256 BF16
// 1.66 -> 1.31 ms, of 300,000 x 256 FP32 885 -> 703 us, stencil of 512,000 x 128 574
// -> 496, R-MAT s21 x 256 FP32 (with k_spmm_long) 4.11 -> 3.52 ms.
// A row's chain starts from its C
// value, staged in shared memory by cp.async once the row is known to have
// entries; rows without entries are not touched.  R > 1 needs R * gk <= 32
// (one lane per (row, stage)); R == 1 takes the stages 32 at a time.
// GROUP = false compiles the one-row walk alone (R == 1, no row changes to
// test for inside the unrolled loop).  `skip` (or null): rows flagged there
// are left to another kernel.  MET (at most 32 stages): so are rows of long_row
// entries or more, and their mask is returned.  `vec`: every B and C row slice of this tile
// pair is 16-byte aligned; otherwise element-wise access.
// There a lane's columns are every 32nd, so that the warp's loads of an entry are
// of neighbouring words, and EU entries' loads are in flight: with a lane's
// columns side by side and each entry's loads waited for (EU = 0), uniform
// 186,581 x 150 FP32 270 us, now 201, stencil of 262,144 x 185 BF16 799, now 587,
// R-MAT of 273,612 x 118 FP32 765, now 524; tiles whose bases lie off 16 bytes,
// uniform 300,000 x 256 FP32 1834, now 927.
template <typename ST, bool GROUP, bool SUB, int EU, bool MET = false, int XN = Vec<ST>::N, int UNROLL = kSpmmUnroll>
__device__ __forceinline__ unsigned spmm_rows(const SpGridView& A, const DGridView& B, const DGridView& C, int64_t ti,
                                              int64_t tj, int64_t r0, int R, int c0, int W, bool vec,
                                              const uint8_t* __restrict__ skip, int long_row = INT_MAX,
                                              int ahead = INT_MAX) {
  if (!GROUP) R = 1;
  using V = Vec<ST>;
  constexpr int VN = V::N;
  const int lane = lane_id();
  const int64_t nrows = min((int64_t)R, C.rows_of(ti) - r0);
  ST* __restrict__ crow0 = reinterpret_cast<ST*>(C.tile(ti, tj)) + r0 * C.ld;
  constexpr int S = EU > 0 ? 32 : 1;  // distance of an element-wise lane's columns
  const int col = c0 + (vec || EU == 0 ? lane * VN : lane);
  const bool own = col < W;
  const int bcol = own ? col : 0;  // lanes past the tile edge load column 0 (in bounds) and store nothing
  const int wib = threadIdx.x >> 5;
  uint4* tb = spmm_tables + wib * 32;
  uint4* cs = spmm_cstage + wib * (kSpmmMaxRows * 32);
  const int gk = (int)A.gn;
  float acc[VN];
  int cur = -1;  // row whose chain is in acc
  bool staged = false;
  unsigned left = 0u;
  auto flush = [&]() {
    if (cur < 0 || !own) return;
    ST* p = crow0 + cur * C.ld;
    if (vec) {
      V::store(p + col, acc);
    } else {
#pragma unroll
      for (int x = 0; x < XN; x++)
        if (col + S * x < W) p[col + S * x] = V::from_f(acc[x]);
    }
  };
  auto enter = [&](int q) {
    flush();
    cur = q;
    if (!own) return;
    if (vec) {
      cp_async_wait_all();
      V::unpack_raw(cs[q * 32 + lane], acc);
    } else {
      const ST* p = crow0 + q * C.ld;
#pragma unroll
      for (int x = 0; x < XN; x++) acc[x] = (col + S * x < W) ? V::to_f(p[col + S * x]) : 0.f;
    }
  };
  for (int64_t g0 = 0; g0 < gk; g0 += 32) {
    const int ql = GROUP ? lane / gk : 0;
    const int64_t kk = GROUP ? lane - ql * gk : g0 + lane;
    bool valid = ql < nrows;
    if (valid && skip) valid = skip[ti * C.tm + r0 + ql] == 0;
    StageLane<ST> sl = stage_lane<ST, SUB>(A, B, ti, tj, r0 + ql, kk, valid);
    int32_t aincl = warp_inclusive_scan(sl.alen);
    if (MET) {
      const int last = GROUP ? min(ql * gk + gk - 1, 31) : 31, first = GROUP ? min(ql * gk, 31) : 0;
      const int32_t through = __shfl_sync(kFull, aincl, last), from = __shfl_sync(kFull, aincl - sl.alen, first);
      const bool lng = valid && through - from >= long_row;
      left = __reduce_or_sync(kFull, lng ? 1u << ql : 0u);
      if (left) {
        if (lng) sl.alen = 0;
        aincl = warp_inclusive_scan(sl.alen);
      }
    }
    const int32_t atot = __shfl_sync(kFull, aincl, 31);
    if (atot == 0) continue;
    const int32_t aexcl = aincl - sl.alen;
    // stage the C slices of the rows that have entries
    if (!GROUP) {
      if (vec && !staged) {
        if (own) cp_async16(cs + lane, crow0 + col);
        staged = true;
      }
    } else {
      for (int q = 0; q < R; q++) {
        const int32_t hi = __shfl_sync(kFull, aincl, q * gk + gk - 1);
        const int32_t lo = __shfl_sync(kFull, aexcl, q * gk);
        if (vec && own && hi > lo) cp_async16(cs + q * 32 + lane, crow0 + q * C.ld + col);
      }
    }
    // each lane's entry of chunk e0 / 32, loaded while the chunk before is
    // applied (past the end: none)
    int32_t nkc = 0;
    float nval = 0.f;
    int nsrc = 0;
    auto fetch = [&](int32_t e0) {
      const int32_t e = e0 + lane;
      int src = 0;
#pragma unroll
      for (int step = 16; step >= 1; step >>= 1) {
        const int32_t t = __shfl_sync(kFull, aincl, src + step - 1);
        if (t <= e) src += step;
      }
      nsrc = src;
      const int32_t off = e - __shfl_sync(kFull, aexcl, src);
      const int32_t* sacol = reinterpret_cast<const int32_t*>(
          __shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.acol), src));
      const float* saval = reinterpret_cast<const float*>(
          __shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.aval), src));
      if (e < atot) {
        nkc = __ldg(sacol + off);
        nval = __ldg(saval + off);
      }
    };
    fetch(0);
    if (!GROUP && cur < 0) enter(0);
    for (int32_t e0 = 0; e0 < atot; e0 += 32) {
      const int ne = min(32, atot - e0);
      // the chunk's table.  Entries past the end point at the last entry's B
      // row (an in-bounds load whose product is never applied).
      const ST* brow = reinterpret_cast<const ST*>(
                           __shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.bt), nsrc)) +
                       (int64_t)nkc * B.ld;
      const uint64_t pa = __shfl_sync(kFull, reinterpret_cast<unsigned long long>(brow), min(lane, ne - 1));
      const int row = GROUP ? nsrc / gk : 0;
      tb[lane] = make_uint4((uint32_t)pa, (uint32_t)(pa >> 32), __float_as_uint(nval), (uint32_t)row);
      // entries that begin a row
      unsigned heads = 0;
      if (GROUP) {
        const int before = __shfl_up_sync(kFull, row, 1);
        heads = __ballot_sync(kFull, row != (lane == 0 ? cur : before));
      }
      __syncwarp();
      if (e0 + 32 < atot) fetch(e0 + 32);
      const uint4* t = tb;
      if (vec) {
        for (int u0 = 0; u0 < ne; u0 += UNROLL) {
          uint4 ent[UNROLL];
          uint4 raw[UNROLL];
#pragma unroll
          for (int u = 0; u < UNROLL; u++) ent[u] = t[(u0 + u) & 31];
#pragma unroll
          for (int u = 0; u < UNROLL; u++) {
            const ST* rp = reinterpret_cast<const ST*>((uint64_t)ent[u].x | ((uint64_t)ent[u].y << 32));
            raw[u] = __ldg(reinterpret_cast<const uint4*>(rp + bcol));
          }
          auto apply = [&](int u) {
            float b[VN];
            V::unpack_raw(raw[u], b);
            const float vs = __uint_as_float(ent[u].z);
#pragma unroll
            for (int x = 0; x < VN; x++) acc[x] = __fmaf_rn(vs, b[x], acc[x]);
          };
          if (u0 + UNROLL <= ne && ((heads >> u0) & ((1u << UNROLL) - 1u)) == 0u) {
            // a whole group of one row: no test between the loads and their use
#pragma unroll
            for (int u = 0; u < UNROLL; u++) apply(u);
          } else {
#pragma unroll
            for (int u = 0; u < UNROLL; u++)
              if (u0 + u < ne) {
                if (GROUP && ((heads >> (u0 + u)) & 1u)) enter((int)t[u0 + u].w);
                apply(u);
              }
          }
        }
      } else {
        if constexpr (EU == 0) {
          for (int u = 0; u < ne; u++) {
            const uint4 en = t[u];
            if (GROUP && (int)en.w != cur) enter((int)en.w);
            const ST* rp = reinterpret_cast<const ST*>((uint64_t)en.x | ((uint64_t)en.y << 32));
            const float vs = __uint_as_float(en.z);
#pragma unroll
            for (int x = 0; x < VN; x++)
              if (col + x < W) acc[x] = __fmaf_rn(vs, V::to_f(rp[col + x]), acc[x]);
          }
        }
        for (int u0 = 0; EU > 0 && u0 < ne; u0 += EU) {
          ST raw[EU > 0 ? EU : 1][XN];
          float vs[EU > 0 ? EU : 1];
#pragma unroll
          for (int u = 0; u < EU; u++) {
            const uint4 en = t[(u0 + u) & 31];
            const ST* rp = reinterpret_cast<const ST*>((uint64_t)en.x | ((uint64_t)en.y << 32));
            vs[u] = __uint_as_float(en.z);
#pragma unroll
            for (int x = 0; x < XN; x++)
              if (col + S * x < W) raw[u][x] = rp[col + S * x];
          }
#pragma unroll
          for (int u = 0; u < EU; u++)
            if (u0 + u < ne) {
              if (GROUP && ((heads >> (u0 + u)) & 1u)) enter((int)t[u0 + u].w);
#pragma unroll
              for (int x = 0; x < XN; x++)
                if (col + S * x < W) acc[x] = __fmaf_rn(vs[u], V::to_f(raw[u][x]), acc[x]);
            }
        }
      }
      __syncwarp();
      if (!GROUP && !MET && EU == 0 && e0 + 32 < atot && atot >= ahead) {
        // a long row's next chunk: its B-row slices, asked for together
        const char* p = reinterpret_cast<const char*>(
            reinterpret_cast<const ST*>(__shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.bt), nsrc)) +
            (int64_t)nkc * B.ld + c0);
        const int bytes = min(W - c0, 32 * VN) * (int)sizeof(ST);
        if (e0 + 32 + lane < atot)
          for (int o = 0; o < bytes; o += 128) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p + o));
      }
    }
  }
  flush();
  return left;
}

// Rows that a kernel of short rows lists and leaves to k_spmm_chain: from `most`
// entries, or from `least` and four times the mean of their tile row.  (Which
// rows are long depends on A alone: the first tile column's items list them.)
struct MetRows {
  int64_t* list;   // or null: they are listed already
  int32_t* count;
  int most, least;
};
// The bound in tile row ti (at most 32 tiles along k where least < most).
__device__ __forceinline__ int met_bound(const MetRows& met, const SpGridView& A, const DGridView& C, int64_t ti) {
  if (met.least >= met.most) return met.most;
  const float nnz = warp_sum(lane_id() < A.gn ? (float)A.tile(ti, lane_id()).nnz : 0.f);
  return min(met.most, max(met.least, (int)min(4.f * nnz / (float)C.rows_of(ti), 1e9f)));
}
// Rows x0 + (bits of left), a lane each, or one lane's loop over the bits.  The loop
// makes k_spmm_narrow spill (50 to 150 bytes), a lane each does not: R-MAT 169,343 x
// 47 FP32 274 -> 257 us, BF16 of 300,000 x 64 R-MAT 275 -> 255, uniform 114 -> 91.  But
// FP32 on 16 bytes: R-MAT of 300,000 x 16 207 with the loop, 223 a lane each, x 64 322
// and 353, of 4,000 x 16 31 and 37 (uniform 300,000 x 16 87 and 81).
template <bool LOOP>
__device__ __forceinline__ void list_met(const MetRows& met, int64_t x0, unsigned left) {
  if (LOOP) {
    if (lane_id() == 0)
      for (; left; left &= left - 1) met.list[atomicAdd(met.count, 1)] = x0 + __ffs(left) - 1;
  } else if ((left >> lane_id()) & 1u) {
    met.list[atomicAdd(met.count, 1)] = x0 + lane_id();
  }
}

// Tile columns [0, tjn) (k_spmm_narrow takes the others).  Warp items come
// from a device counter (one grab per item, the next grab in
// flight while the current item runs), so warps that draw short rows take
// more of them: the cost of a (row group, panel) item varies by orders of
// magnitude on power-law matrices.
// MET: with at most 32 tiles along k, long rows are listed and left out.
// all_long: every row flagged long is k_spmm_chain's; otherwise k_spmm_long
// takes them on aligned tiles.
// ELEM: every tile element by element (rows off 16 bytes), ELEM columns a lane.  Otherwise the tiles
// whose bases lie off 16 bytes are, with as many loads in flight as cost the
// vector walk no registers (with 16, R-MAT s21 x 256 FP32 3.94 -> 4.26 ms; in BF16
// a second copy of the walk costs it as much: 2.10 -> 2.22 ms; with MET, uniform
// 60,000 x 16 FP32 on 20 x 20 tiles 90 -> 96 us).
template <typename ST, bool GROUP, bool SUB, int ELEM, bool MET = false>
__global__ void __launch_bounds__(kSpmmWarps * 32, 4)
    k_spmm(SpGridView A, DGridView B, DGridView C, int tjn, int64_t n_items, int npanels, int R, int64_t ngroups,
           int row_align_ok, int panel_major, const uint8_t* __restrict__ long_flag, bool all_long,
           MetRows met, unsigned long long* __restrict__ next_item) {
  constexpr int PW = 32 * (ELEM ? ELEM : Vec<ST>::N);
  const int lane = lane_id();
  unsigned long long it = 0;
  if (lane == 0) it = atomicAdd(next_item, 1ULL);
  it = __shfl_sync(kFull, it, 0);
  // item numbers and their parts: 32-bit divisions where they all fit (a 64-bit
  // one is some 70 instructions)
  const bool small = n_items <= UINT32_MAX;
  auto divide = [small](int64_t a, int64_t b) { return small ? (int64_t)((uint32_t)a / (uint32_t)b) : a / b; };
  int64_t at = -1;  // the C tile `aligned` and `bound` are for
  bool aligned = false;
  int bound = INT_MAX;
  const int ahead = B.m * B.ld * (int64_t)sizeof(ST) >= kSpmmAheadBytes ? kSpmmAhead : INT_MAX;
  while (it < (unsigned long long)n_items) {
    unsigned long long nx = 0;
    if (lane == 0) nx = atomicAdd(next_item, 1ULL);
    const int64_t item = (int64_t)it;
    int64_t rg;
    int panel;
    if (panel_major) {  // all row groups of panel 0, then of panel 1, ...
      const int64_t n_rg = divide(n_items, npanels);
      panel = (int)divide(item, n_rg);
      rg = item - panel * n_rg;
    } else {  // the panels of a row group one after another
      rg = divide(item, npanels);
      panel = (int)(item - rg * npanels);
    }
    const int64_t t = divide(rg, ngroups);
    const int64_t r0 = (rg - t * ngroups) * R;
    const int64_t ti = divide(t, tjn), tj = t - ti * tjn;
    const int W = (int)C.cols_of(tj);
    const int c0 = panel * PW;
    if (r0 < C.rows_of(ti) && c0 < W) {
      if ((!ELEM || MET) && t != at) {
        at = t;
        if (!ELEM) aligned = row_align_ok && (W % Vec<ST>::N) == 0 && tiles_aligned(B, C, ti, tj);
        if (MET) bound = met_bound(met, A, C, ti);
      }
      unsigned left;
      if (ELEM)
        left = spmm_rows<ST, GROUP, SUB, 16 / (ELEM ? ELEM : 1), MET, ELEM ? ELEM : 1>(A, B, C, ti, tj, r0, R, c0, W, false, long_flag, bound);
      else if (sizeof(ST) == 2 || MET)
        left = spmm_rows<ST, GROUP, SUB, 0, MET>(A, B, C, ti, tj, r0, R, c0, W, aligned,
                                                 aligned || all_long ? long_flag : nullptr, bound, ahead);
      else if (aligned)
        left = spmm_rows<ST, GROUP, SUB, 0, MET>(A, B, C, ti, tj, r0, R, c0, W, true, long_flag, bound, ahead);
      else
        left = spmm_rows<ST, GROUP, SUB, 2, MET>(A, B, C, ti, tj, r0, R, c0, W, false, all_long ? long_flag : nullptr,
                                                 bound);
      if (MET && left && tj == 0 && panel == 0) list_met<false>(met, ti * A.tm + r0, left);
    }
    it = __shfl_sync(kFull, nx, 0);
  }
  // launched as k_spmm_long's programmatic dependent: finish only after it
  // (a normal launch returns here at once)
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// ---- long rows ----------------------------------------------------------------
//
// A row with thousands of entries is one chain of multiply-adds per output
// element (the reference's order): it cannot be split, only fed faster.  Such
// rows are found first (k_spmm_find_long), skipped by k_spmm and run by
// k_spmm_long on the context's side stream at the same time, a pair of warps per
// (row, C tile column, panel), with the B-row slices themselves copied into
// shared memory by cp.async two chunks (64 entries) ahead: the loads in
// flight cost no registers, and a chunk's multiply-adds read shared memory.
// Rows of 8 times the long-row threshold or more are listed first, so that
// the longest chains start first.

constexpr int kLongPairs = 4;   // pairs of warps per block
constexpr int kLongBSlots = 3;  // chunks of B slices per warp: applied, in flight, being issued
constexpr int kLongTSlots = 3;  // chunks of table entries per warp (with the B slices)
constexpr int kLongASlots = 6;  // chunks of staged A entries per warp
// A row is long from BCLX_TUNE_SPMM_LONG_ROW entries over all stages (512 by
// default).
constexpr int64_t kSpmmLongMinRows = 65536;  // smaller products do not use the long-row path

struct LongSmem {
  uint4 b[kLongBSlots][32][32];  // [chunk slot][entry][lane]: each lane's 16 bytes of the entry's B row
  uint4 tab[kLongTSlots][32];    // [chunk slot][entry]: B-row address, A value
  uint2 a[kLongASlots][32];      // [chunk slot][entry]: staged A (column, value)
  uint8_t src[kLongASlots][32];  // the entry's stage lane
  unsigned long long next;       // the pair's next item
};

// The two warps of a pair (a producer and a consumer) meet.
__device__ __forceinline__ void pair_sync(int pair) {
  __syncwarp();
  asm volatile("bar.sync %0, 64;\n" ::"r"(pair + 1) : "memory");
}

// Thread per A row (ti, r): entries over all stages; rows with at least
// long_row are flagged and listed: very long rows from list[0] up
// (count[0]), the others from list[rows-1] down (count[1]).
__global__ void k_spmm_find_long(SpGridView A, int long_row, int very_long_row, uint8_t* __restrict__ flag,
                                 int64_t* __restrict__ list, int32_t* __restrict__ count) {
  const int64_t rows = A.gm * A.tm;
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < rows; x += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ti = x / A.tm, r = x - ti * A.tm;
    int64_t tot = 0;
    if (r < A.rows_of(ti))
      for (int64_t k = 0; k < A.gn; k++) {
        const int32_t* rp = A.tile(ti, k).row_ptr;
        tot += __ldg(rp + r + 1) - __ldg(rp + r);
      }
    const bool lng = tot >= long_row;
    flag[x] = lng ? 1 : 0;
    if (lng) {
      if (tot >= very_long_row)
        list[atomicAdd(count, 1)] = x;
      else
        list[rows - 1 - atomicAdd(count + 1, 1)] = x;
    }
  }
}

// One long row r of C tile (ti, tj), panel from column c0 (16-byte aligned
// access: the caller checked), by a pair of warps.  In step c (a chunk of 32
// entries, one per lane when staged or built)
//   * the consumer applies chunk c: the multiply-adds in entry order from
//     shared memory;
//   * the producer stages A of chunk c + 6 (cp.async, 8 bytes per lane),
//     builds chunk c + 2 (each lane's entry -> table: B-row address, value),
//     copies its B rows into the slot that chunk c - 1 left (cp.async, every
//     lane 16 bytes of each row) and waits for chunk c + 1's;
// and the two meet.  One commit group per step holds A(c+6) and B(c+2).  The
// stages are at most 32 (one lane each).  The row's chain sets the time of
// these products: one warp doing both parts took some 60 cycles per entry, on
// an SM to itself as well. 
// Now a pair takes the SM's share of L2 traffic: R-MAT of 1,000,000 rows x 256
// BF16 1.56 -> 1.13 ms, of 300,000 x 128 FP32 551 -> 388 us, of 100,000 x 128 274 ->
// 188, s21 x 256 BF16 2.19 -> 1.91 ms.
template <typename ST, bool SUB>
__device__ __forceinline__ void spmm_long_row(LongSmem& S, int pair, bool producer, const SpGridView& A,
                                              const DGridView& B, const DGridView& C, int64_t ti, int64_t tj, int64_t r,
                                              int c0, int W) {
  using V = Vec<ST>;
  constexpr int VN = V::N;
  const int lane = lane_id();
  ST* __restrict__ crow = reinterpret_cast<ST*>(C.tile(ti, tj)) + r * C.ld;
  const int col = c0 + lane * VN;
  const bool own = col < W;
  const StageLane<ST> sl = stage_lane<ST, SUB>(A, B, ti, tj, r, lane, true);
  const int32_t aincl = warp_inclusive_scan(sl.alen);
  const int32_t atot = __shfl_sync(kFull, aincl, 31);
  const int32_t aexcl = aincl - sl.alen;
  const int32_t nch = (atot + 31) >> 5;
  if (!producer) {
    float acc[VN];
    if (own) V::load_c(crow + col, acc);
    pair_sync(pair);  // chunk 0 is there
    for (int32_t c = 0; c < nch; c++) {
      const int ne = min(32, atot - c * 32);
      const int bslot = c % kLongBSlots, tslot = c % kLongTSlots;
      auto apply = [&](int u) {
        float b[VN];
        V::unpack_raw(S.b[bslot][u][lane], b);
        const float vs = __uint_as_float(S.tab[tslot][u].z);
#pragma unroll
        for (int x = 0; x < VN; x++) acc[x] = __fmaf_rn(vs, b[x], acc[x]);
      };
      if (own) {
        if (ne == 32) {
#pragma unroll 16
          for (int u = 0; u < 32; u++) apply(u);
        } else {
          for (int u = 0; u < ne; u++) apply(u);
        }
      }
      pair_sync(pair);
    }
    if (own) V::store(crow + col, acc);
    return;
  }
  auto issue_a = [&](int32_t x) {
    if (x >= nch) return;
    const int32_t e = x * 32 + lane;
    int src = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
      const int32_t t = __shfl_sync(kFull, aincl, src + step - 1);
      if (t <= e) src += step;
    }
    src = min(src, 31);
    const int32_t off = e - __shfl_sync(kFull, aexcl, src);
    const int32_t* sacol = reinterpret_cast<const int32_t*>(
        __shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.acol), src));
    const float* saval = reinterpret_cast<const float*>(
        __shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.aval), src));
    const int slot = x % kLongASlots;
    S.src[slot][lane] = (uint8_t)src;
    if (e < atot) {
      cp_async4_nb(&S.a[slot][lane].x, sacol + off);
      cp_async4_nb(&S.a[slot][lane].y, saval + off);
    }
  };
  auto build = [&](int32_t x) {  // A(x) has landed
    if (x >= nch) return;
    const int slot = x % kLongASlots;
    const int src = S.src[slot][lane];
    const ST* sbt = reinterpret_cast<const ST*>(__shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.bt), src));
    const int32_t e = x * 32 + lane;
    if (e < atot) {
      const uint2 a = S.a[slot][lane];
      const uint64_t pa = reinterpret_cast<uint64_t>(sbt + (int64_t)(int32_t)a.x * B.ld);
      S.tab[x % kLongTSlots][lane] = make_uint4((uint32_t)pa, (uint32_t)(pa >> 32), a.y, 0u);
    }
  };
  auto issue_b = [&](int32_t x) {  // table of chunk x built, then a __syncwarp
    if (x >= nch || !own) return;
    const int ne = min(32, atot - x * 32);
    const int bslot = x % kLongBSlots, tslot = x % kLongTSlots;
    auto copy = [&](int u, const uint4& t) {
      const ST* rp = reinterpret_cast<const ST*>((uint64_t)t.x | ((uint64_t)t.y << 32));
      cp_async16_nb(&S.b[bslot][u][lane], rp + col);
    };
    if (ne == 32) {
#pragma unroll
      for (int u0 = 0; u0 < 32; u0 += 8) {
        uint4 t[8];
#pragma unroll
        for (int k = 0; k < 8; k++) t[k] = S.tab[tslot][u0 + k];
#pragma unroll
        for (int k = 0; k < 8; k++) copy(u0 + k, t[k]);
      }
    } else {
      for (int u = 0; u < ne; u++) copy(u, S.tab[tslot][u]);
    }
  };
  // fill: A(0..5) staged, chunks 0 and 1 built and their B slices asked for
  issue_a(0);
  issue_a(1);
  cp_async_commit();
  issue_a(2);
  issue_a(3);
  cp_async_commit();
  cp_async_wait_group<1>();
  build(0);
  build(1);
  __syncwarp();
  issue_b(0);
  issue_a(4);
  cp_async_commit();
  issue_b(1);
  issue_a(5);
  cp_async_commit();
  cp_async_wait_group<1>();  // B(0) and A(4) have landed
  pair_sync(pair);
  for (int32_t c = 0; c < nch; c++) {
    issue_a(c + 6);
    build(c + 2);
    __syncwarp();
    issue_b(c + 2);
    cp_async_commit();
    cp_async_wait_group<1>();  // B(c + 1) and A(c + 5) have landed
    pair_sync(pair);
  }
  cp_async_wait_all();
}

// Items (listed row, C tile column, panel), a row's items consecutive, taken
// from a device counter in list order.  Every block, once placed, lets a
// programmatic dependent (k_spmm under the dependent-launch schedule) launch.
template <typename ST, bool SUB>
__global__ void __launch_bounds__(kLongPairs * 64)
    k_spmm_long(SpGridView A, DGridView B, DGridView C, int tjn, const int64_t* __restrict__ list,
                const int32_t* __restrict__ count, int npanels, int row_align_ok,
                unsigned long long* __restrict__ next_item) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  extern __shared__ __align__(16) unsigned char long_smem[];
  const int pair = threadIdx.x >> 6;
  const bool producer = (threadIdx.x >> 5) & 1;
  LongSmem& S = reinterpret_cast<LongSmem*>(long_smem)[pair];
  constexpr int PW = 32 * Vec<ST>::N;
  const int lane = lane_id();
  const int64_t rows = A.gm * A.tm;
  const int64_t nv = count[0];
  const int64_t nl = nv + count[1];
  const int64_t per_row = (int64_t)tjn * npanels;
  const unsigned long long n = (unsigned long long)(nl * per_row);
  // the first items, dealt to the blocks in turn: neighbouring rows, which the
  // longest are, go to different SMs
  unsigned long long it = (unsigned long long)pair * gridDim.x + blockIdx.x;
  const unsigned long long dealt = (unsigned long long)gridDim.x * kLongPairs;
  while (it < n) {
    unsigned long long nx = 0;
    if (producer && lane == 0) nx = dealt + atomicAdd(next_item, 1ULL);
    const int64_t li = (int64_t)it / per_row;
    const int64_t pt = (int64_t)it - li * per_row;
    const int panel = (int)(pt % npanels);
    const int64_t tj = pt / npanels;
    const int64_t x = li < nv ? list[li] : list[rows - 1 - (li - nv)];
    const int64_t ti = x / A.tm, r = x - ti * A.tm;
    const int W = (int)C.cols_of(tj);
    if (panel * PW < W) {
      const bool vec = row_align_ok && (W % Vec<ST>::N) == 0 && tiles_aligned(B, C, ti, tj);
      // (otherwise k_spmm does it element-wise)
      if (vec) spmm_long_row<ST, SUB>(S, pair, producer, A, B, C, ti, tj, r, panel * PW, W);
    }
    if (producer && lane == 0) S.next = nx;
    pair_sync(pair);
    it = *reinterpret_cast<volatile unsigned long long*>(&S.next);
    pair_sync(pair);
  }
}

// ---- narrow and unaligned tiles ------------------------------------------------
//
// k_spmm gives a B-row slice of 512 bytes to a warp's 32 lanes.  A tile of a
// few columns leaves most of those lanes idle, and one whose rows do not
// start on 16 bytes would be read element by element, each load waited for.
// Two kernels take those tiles:
//  * k_spmm_narrow, the short rows: a group of L lanes per row (8 to 32), so
//    that a warp walks 32 / L rows at once, each lane owning NV units of the
//    row (16-byte vectors, or 4- or 2-byte words where rows start on no more);
//  * k_spmm_chain, the long rows (32 L entries or more, over all stages): one
//    chain of multiply-adds per column that cannot be split, only fed.  A
//    block takes one: producer warps copy the B-row slices of the next entries
//    into shared memory (cp.async, three buffers), one consumer warp runs 32
//    words' chains from there and does nothing else.
// Products with many rows list their long rows first (k_spmm_find_long) and
// run both at once: k_spmm_narrow is launched as k_spmm_chain's programmatic
// dependent, starts once every chain block has, and ends after it.  With
// fewer rows (where the extra launch would show) k_spmm_narrow lists the long
// rows it meets and k_spmm_chain follows.  Rows that take all 32 lanes go to
// k_spmm in place of k_spmm_narrow (see launch_narrow_nv).
// Bound: the short rows by instruction issue (60-66 % of the slots; a third of a
// warp's groups wait for its longest row) and by the latency of their loads
// (A entry, then B row), hidden by 32 warps per SM; a long row by its chain,
// 4.5 ns per entry (k_spmm_long: 25).  FP32 products, k_spmm before -> now:
// R-MAT 169,343 x 47 columns (rows on 4 bytes) 3.51 -> 0.27 ms; R-MAT 400,001 x
// 16 0.64 -> 0.27; R-MAT 300,000 x 64 0.51 -> 0.32; uniform 100,000 x 32 90 ->
// 54 us; BF16, R-MAT 50,000 x 135 (rows on 2 bytes) 2.5 -> 0.37 ms.
constexpr int kNarrowWarps = 8;
constexpr int kNarrowUnroll = 4;          // entries per lane group whose loads are in flight
// A row is long from this many steps of L entries (or BCLX_TUNE_SPMM_LONG_ROW):
// fewer make k_spmm_chain's set-up per row (3.5 us of a block) show, more leave
// a warp its longest row (R-MAT 50,000 x 8: 82 us with 16 steps, 83 with 32, 111
// with 64; R-MAT 300,000 x 32 BF16: 284, 264, 289).
constexpr int kNarrowLongSteps = 32;
// In products of few rows (not listed, see launch_narrow_nv), where a warp has
// an item or two and waits for its longest row, also a row of this many entries and
// of four times its tile row's mean (rows that are all alike stay with their
// warps): R-MAT 2,412 x 119 FP32 60 -> 39 us, 4,313 x 72 BF16 82 -> 42, 20,000 x 47
// FP32 106 -> 80, 40,000 x 90 152 -> 123.
constexpr int kNarrowFewLong = 128;
// Widest row of an aligned tile that k_spmm_narrow takes: two 128-byte lines
// (one warp then walks two rows).  At 256 bytes: R-MAT 300,000 x 64 FP32 0.32
// ms against 0.51 with k_spmm, uniform 100,000 x 128 BF16 93 us against 108.
constexpr int64_t kNarrowMaxBytes = 256;
constexpr int kChainWarps = 8;            // one applies, the others copy
constexpr int kChainPanelWords = 32;      // words of a long row that a block takes at once: one per consumer lane
constexpr int kChainBuffers = 3;
constexpr int kChainEach = 32;            // entries of a batch per copying warp: one per lane
// Shared memory for slices of `stride` words and their values.
constexpr size_t chain_bytes(int stride) {
  return 4 * (size_t)(kChainBuffers * (kChainWarps - 1) * kChainEach * (stride + 1) + kChainPanelWords);
}
static_assert(chain_bytes(kChainPanelWords) <= 92 * 1024, "two blocks per SM");

// First lane whose inclusive prefix exceeds e (32 when none does).
__device__ __forceinline__ int warp_search_lanes(int32_t incl, int32_t e) {
  int src = 0;
#pragma unroll
  for (int step = 16; step >= 1; step >>= 1) {
    const int32_t t = __shfl_sync(kFull, incl, src + step - 1);
    if (t <= e) src += step;
  }
  return src;
}

// A unit of U bytes of a row of ST: load, store and the chain step.
template <typename ST, int U>
struct Unit {
  static constexpr int N = U / (int)sizeof(ST);  // columns
  using R = std::conditional_t<U == 16, uint4, std::conditional_t<U == 4, uint32_t, uint16_t>>;
  __device__ __forceinline__ static R load(const ST* p, int u) { return __ldg(reinterpret_cast<const R*>(p) + u); }
  __device__ __forceinline__ static R load_c(const ST* p, int u) { return reinterpret_cast<const R*>(p)[u]; }
  __device__ __forceinline__ static void store(ST* p, int u, R v) { reinterpret_cast<R*>(p)[u] = v; }
  __device__ __forceinline__ static void unpack(R v, float* o) {
    if constexpr (U == 16) {
      Vec<ST>::unpack_raw(v, o);
    } else if constexpr (sizeof(ST) == 4) {
      o[0] = __uint_as_float(v);
    } else {
      o[0] = __uint_as_float((uint32_t)v << 16);
      if constexpr (U == 4) o[1] = __uint_as_float(v & 0xffff0000u);
    }
  }
  __device__ __forceinline__ static uint32_t bf16_bits(float x) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x));
  }
  __device__ __forceinline__ static R pack(const float* i) {
    if constexpr (U == 16 && sizeof(ST) == 4) {
      return make_uint4(__float_as_uint(i[0]), __float_as_uint(i[1]), __float_as_uint(i[2]), __float_as_uint(i[3]));
    } else if constexpr (U == 16) {
      return make_uint4(bf16_bits(i[0]) | bf16_bits(i[1]) << 16, bf16_bits(i[2]) | bf16_bits(i[3]) << 16,
                        bf16_bits(i[4]) | bf16_bits(i[5]) << 16, bf16_bits(i[6]) | bf16_bits(i[7]) << 16);
    } else if constexpr (sizeof(ST) == 4) {
      return __float_as_uint(i[0]);
    } else if constexpr (U == 4) {
      return bf16_bits(i[0]) | bf16_bits(i[1]) << 16;
    } else {
      return (uint16_t)bf16_bits(i[0]);
    }
  }
};

// Every row slice of C tile (ti, tj) and of its B tiles starts on U bytes and
// is a whole number of them.
template <typename ST, int U>
__device__ __forceinline__ bool tile_on(const DGridView& B, const DGridView& C, int64_t ti, int64_t tj, int W) {
  uint32_t low = (uint32_t)reinterpret_cast<uintptr_t>(C.tile(ti, tj)) | (uint32_t)(B.ld * sizeof(ST)) |
                 (uint32_t)(C.ld * sizeof(ST)) | (uint32_t)(W * sizeof(ST));
  for (int64_t k = lane_id(); k < B.gm; k += 32) low |= (uint32_t)reinterpret_cast<uintptr_t>(B.tile(k, tj));
  return __reduce_or_sync(kFull, low & (uint32_t)(U - 1)) == 0u;
}

// Rows [r0, r0 + 32/L) of C tile (ti, tj), columns [c0, c0 + W): the group of
// L lanes g walks row r0 + g, L entries at a time: each lane finds and loads
// one A entry (the next L are in flight meanwhile) and the group's lanes then
// take the B rows kNarrowUnroll at a time.  32/L * gk <= 32: one lane per
// (row, stage) holds that segment; with L == 32 the stages go 32 at a time.
// Rows of long_row entries or more are left out; their mask (by group) is
// returned.
template <typename ST, int U, int NV, bool SUB>
__device__ __forceinline__ unsigned narrow_rows(const SpGridView& A, const DGridView& B, const DGridView& C,
                                                int64_t ti, int64_t tj, int64_t r0, int L, int c0, int W,
                                                int long_row) {
  using UN = Unit<ST, U>;
  constexpr int N = UN::N;
  const int lane = lane_id();
  const int gk = (int)A.gn;
  const int grp = lane / L, li = lane & (L - 1);
  const int rows = 32 / L;
  const int64_t nrows = min((int64_t)rows, C.rows_of(ti) - r0);
  ST* __restrict__ crow = reinterpret_cast<ST*>(C.tile(ti, tj)) + (r0 + grp) * C.ld + c0;
  const int units = W / N;
  float acc[NV][N];
  bool have = false;  // the row's chain is in acc
  unsigned left = 0u;
  for (int g0 = 0; g0 < gk; g0 += 32) {
    const int sq = L == 32 ? 0 : lane / gk;
    const int64_t kk = L == 32 ? g0 + lane : lane - sq * gk;
    const StageLane<ST> sl = stage_lane<ST, SUB>(A, B, ti, tj, r0 + sq, kk, sq < nrows);
    const int32_t aincl = warp_inclusive_scan(sl.alen);
    const int32_t aexcl = aincl - sl.alen;
    const int f = L == 32 ? 0 : grp * gk, l = L == 32 ? 31 : min(grp * gk + gk - 1, 31);
    const int32_t first = __shfl_sync(kFull, aexcl, min(f, 31));
    int32_t T = __shfl_sync(kFull, aincl, l) - first;  // this group's entries
    if (grp >= nrows) T = 0;
    if (T >= long_row) {
      left = 1u << grp;
      T = 0;
    }
    const int32_t most = __reduce_max_sync(kFull, T);
    if (most == 0) continue;
    if (T > 0 && !have) {
      have = true;
#pragma unroll
      for (int i = 0; i < NV; i++)
        if (li + L * i < units) UN::unpack(UN::load_c(crow, li + L * i), acc[i]);
    }
    int32_t nc = 0;
    float nv = 0.f;
    const ST* nbt = nullptr;
    auto fetch = [&](int32_t p) {  // A entry p + li of the group's row
      const int32_t e = first + p + li;
      const int src = min(warp_search_lanes(aincl, e), 31);
      const int32_t off = e - __shfl_sync(kFull, aexcl, src);
      const int32_t* sacol = reinterpret_cast<const int32_t*>(
          __shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.acol), src));
      const float* saval = reinterpret_cast<const float*>(
          __shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.aval), src));
      nbt = reinterpret_cast<const ST*>(__shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.bt), src));
      if (p + li < T) {
        nc = __ldg(sacol + off);
        nv = __ldg(saval + off);
      }
    };
    fetch(0);
    for (int32_t p = 0; p < most; p += L) {
      const float v = nv;
      const unsigned long long baddr = reinterpret_cast<unsigned long long>(nbt + (int64_t)nc * B.ld + c0);
      if (p + L < most) fetch(p + L);
      const int here = min(L, most - p);  // (uniform)
      for (int u0 = 0; u0 < here; u0 += kNarrowUnroll) {
        float vs[kNarrowUnroll];
        const ST* br[kNarrowUnroll];
#pragma unroll
        for (int k = 0; k < kNarrowUnroll; k++) {
          br[k] = reinterpret_cast<const ST*>(__shfl_sync(kFull, baddr, u0 + k, L));
          vs[k] = __shfl_sync(kFull, v, u0 + k, L);
        }
        typename UN::R raw[kNarrowUnroll][NV];
#pragma unroll
        for (int k = 0; k < kNarrowUnroll; k++)
#pragma unroll
          for (int i = 0; i < NV; i++)
            if (p + u0 + k < T && li + L * i < units) raw[k][i] = UN::load(br[k], li + L * i);
#pragma unroll
        for (int k = 0; k < kNarrowUnroll; k++)
          if (p + u0 + k < T) {
#pragma unroll
            for (int i = 0; i < NV; i++) {
              float b[N];
              UN::unpack(raw[k][i], b);
#pragma unroll
              for (int x = 0; x < N; x++) acc[i][x] = __fmaf_rn(vs[k], b[x], acc[i][x]);
            }
          }
      }
    }
  }
  if (have) {
#pragma unroll
    for (int i = 0; i < NV; i++)
      if (li + L * i < units) UN::store(crow, li + L * i, UN::pack(acc[i]));
  }
  return __reduce_or_sync(kFull, left);
}

// Rows [r0, r1) of C tile (ti, tj), columns [c0, c1), one column per lane and
// one entry at a time: tiles whose base is off the launch's unit (the host
// sees their leading dimensions and widths, not the device array of bases).
// Rows of long_row entries or more are left out; their mask is returned.
template <typename ST, bool SUB>
__device__ __forceinline__ unsigned elem_rows(const SpGridView& A, const DGridView& B, const DGridView& C, int64_t ti,
                                              int64_t tj, int64_t r0, int64_t r1, int c0, int c1, int long_row) {
  unsigned left = 0u;
  for (int64_t r = r0; r < r1; r++) {
    int64_t total = 0;
    for (int64_t k = 0; k < A.gn; k++) {
      const int32_t* rp = A.tile(ti, k).row_ptr + r;
      total += __ldg(rp + 1) - __ldg(rp);
    }
    if (total >= long_row) left |= 1u << (r - r0);
    if (total == 0 || total >= long_row) continue;
    ST* crow = reinterpret_cast<ST*>(C.tile(ti, tj)) + r * C.ld;
    for (int c = c0 + lane_id(); c < c1; c += 32) {
      float acc = Vec<ST>::to_f(crow[c]);
      for (int64_t kk = 0; kk < A.gn; kk++) {
        const StageLane<ST> sl = stage_lane<ST, SUB>(A, B, ti, tj, r, kk, true);
        for (int32_t e = 0; e < sl.alen; e++)
          acc = __fmaf_rn(__ldg(sl.aval + e), Vec<ST>::to_f(sl.bt[(int64_t)__ldg(sl.acol + e) * B.ld + c]), acc);
      }
      crow[c] = Vec<ST>::from_f(acc);
    }
  }
  return left;
}

// The chains of n entries in a buffer: this lane's word of each slice at `sw`
// (slices STRIDE words apart), the A values at `sv`.  The next eight entries'
// words are loaded before the current eight are applied, so that a chain step
// waits for its multiply-add alone.
template <typename ST, int STRIDE>
__device__ __forceinline__ void chain_apply(const uint32_t* sw, const float* sv, int n, float* acc) {
  constexpr int CN = 4 / (int)sizeof(ST);
  struct Eight {
    uint32_t x[8];
    float v[8];
  };
  auto load = [&](Eight& t, int u) {
#pragma unroll
    for (int k = 0; k < 8; k++) t.x[k] = sw[(u + k) * STRIDE];
    const float4 a = *reinterpret_cast<const float4*>(sv + u), b = *reinterpret_cast<const float4*>(sv + u + 4);
    t.v[0] = a.x; t.v[1] = a.y; t.v[2] = a.z; t.v[3] = a.w;
    t.v[4] = b.x; t.v[5] = b.y; t.v[6] = b.z; t.v[7] = b.w;
  };
  auto step = [&](uint32_t x, float v) {
    float o[CN];
    Unit<ST, 4>::unpack(x, o);
#pragma unroll
    for (int c = 0; c < CN; c++) acc[c] = __fmaf_rn(v, o[c], acc[c]);
  };
  auto apply = [&](const Eight& t) {
#pragma unroll
    for (int k = 0; k < 8; k++) step(t.x[k], t.v[k]);
  };
  int u = 0;
  if (n >= 8) {
    Eight t0, t1;
    load(t0, 0);
    for (; u + 24 <= n; u += 16) {
      load(t1, u + 8);
      apply(t0);
      load(t0, u + 16);
      apply(t1);
    }
    if (u + 16 <= n) {
      load(t1, u + 8);
      apply(t0);
      apply(t1);
      u += 16;
    } else {
      apply(t0);
      u += 8;
    }
  }
  for (; u < n; u++) step(sw[u * STRIDE], sv[u]);
}

// One long row r of C tile (ti, tj), columns [c0, c0 + W) (at most
// kChainPanelWords words), by the whole block: warp 0 applies, the others
// copy, kChainEach entries of a batch per producer warp.  While batch b is
// applied from its buffer, batches b + 1 and b + 2 are in flight.  One barrier
// per batch: past it batch b has landed (each producer waited for its own
// copies) and batch b - 1, whose buffer batch b + 2 overwrites, has been
// applied.  MANY: more than 32 stages, 32 at a time (the loop's registers cost the
// others 1 %).  Buffers: slices of `stride` words, then the
// values.
template <typename ST, bool SUB, bool MANY>
__device__ __forceinline__ void chain_row(uint32_t* slices, float* vals, int stride, const SpGridView& A,
                                          const DGridView& B, const DGridView& C, int64_t ti, int64_t tj, int64_t r,
                                          int c0, int W, int unit) {
  constexpr int CN = 4 / (int)sizeof(ST);  // columns per word
  const int lane = lane_id();
  const int prod = (int)(threadIdx.x >> 5) - 1;  // producer number; -1: the consumer
  const int nw = (W * (int)sizeof(ST) + 3) >> 2;
  constexpr int each = kChainEach, batch = each * (kChainWarps - 1);
  ST* __restrict__ crow = reinterpret_cast<ST*>(C.tile(ti, tj)) + r * C.ld + c0;
  // the lane's columns 2 lane and 2 lane + 1 (BF16) or lane (FP32)
  float acc[CN];
  if (prod < 0) {
#pragma unroll
    for (int x = 0; x < CN; x++) acc[x] = lane < nw && lane * CN + x < W ? Vec<ST>::to_f(crow[lane * CN + x]) : 0.f;
  }
  for (int g0 = 0; g0 == 0 || (MANY && g0 < (int)A.gn); g0 += 32) {  // the stages, a lane each
    const StageLane<ST> sl = stage_lane<ST, SUB>(A, B, ti, tj, r, g0 + lane, true);
    const int32_t aincl = warp_inclusive_scan(sl.alen);
    const int32_t atot = __shfl_sync(kFull, aincl, 31);
    if (MANY && atot == 0) continue;  // (the same for every warp)
    const int32_t aexcl = aincl - sl.alen;
    const int32_t nb = (atot + batch - 1) / batch;
    if (prod < 0) {
      for (int32_t b = 0; b < nb; b++) {
        __syncthreads();
        const int n = min(batch, atot - b * batch);
        const int base = (b % kChainBuffers) * batch;
        const uint32_t* sw = slices + base * stride + lane;
        const float* sv = vals + base;
        if (stride == 4) chain_apply<ST, 4>(sw, sv, n, acc);
        else if (stride == 8) chain_apply<ST, 8>(sw, sv, n, acc);
        else if (stride == 16) chain_apply<ST, 16>(sw, sv, n, acc);
        else chain_apply<ST, 32>(sw, sv, n, acc);
      }
    } else {
      const int n_unit = W * (int)sizeof(ST) / unit;  // copies per slice
      const int trips = (each * n_unit + 31) >> 5;
      const int u_first = lane / n_unit, q_first = lane - u_first * n_unit;
      const int u_step = 32 / n_unit, q_step = 32 - u_step * n_unit;
      int32_t nc = 0;  // the pending A entry: its column, value and B tile
      float nv = 0.f;
      const ST* nbt = nullptr;
      auto fetch = [&](int32_t x) {
        if (x >= nb) return;
        const int32_t e = x * batch + prod * each + lane;
        const int src = min(warp_search_lanes(aincl, e), 31);
        const int32_t off = e - __shfl_sync(kFull, aexcl, src);
        const int32_t* sacol = reinterpret_cast<const int32_t*>(
            __shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.acol), src));
        const float* saval = reinterpret_cast<const float*>(
            __shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.aval), src));
        nbt = reinterpret_cast<const ST*>(__shfl_sync(kFull, reinterpret_cast<unsigned long long>(sl.bt), src));
        if (lane < each && e < atot) {
          nc = __ldg(sacol + off);
          nv = __ldg(saval + off);
        }
      };
      auto issue = [&](int32_t x) {  // batch x: its A entries are in nc, nv, nbt
        if (x < nb) {
          const int base = (x % kChainBuffers) * batch + prod * each;
          const int left = min(each, atot - x * batch - prod * each);  // entries of this warp (or none)
          const unsigned long long addr = reinterpret_cast<unsigned long long>(nbt + (int64_t)nc * B.ld + c0);
          if (lane < each) vals[base + lane] = nv;
          char* to = reinterpret_cast<char*>(slices + base * stride);
          int u = u_first, q = q_first;
          auto next = [&]() {
            u += u_step;
            q += q_step;
            if (q >= n_unit) {
              q -= n_unit;
              u++;
            }
          };
          if (left <= 0) {
          } else if (unit != 2) {
#pragma unroll 4
            for (int i = 0; i < trips; i++) {
              const char* from = reinterpret_cast<const char*>(__shfl_sync(kFull, addr, u & 31)) + q * unit;
              char* dst = to + u * stride * 4 + q * unit;
              if (u < left) {
                if (unit == 16) cp_async16_nb(dst, from);
                else cp_async4_nb(dst, from);
              }
              next();
            }
          } else {  // no asynchronous copy of 2 bytes: eight loads in flight
            for (int i0 = 0; i0 < trips; i0 += 8) {
              uint16_t h[8];
              int at[8];
#pragma unroll
              for (int k = 0; k < 8; k++) {
                const uint16_t* from = reinterpret_cast<const uint16_t*>(__shfl_sync(kFull, addr, u & 31)) + q;
                at[k] = u < left ? u * stride * 2 + q : -1;
                if (at[k] >= 0) h[k] = __ldg(from);
                next();
              }
#pragma unroll
              for (int k = 0; k < 8; k++)
                if (at[k] >= 0) reinterpret_cast<uint16_t*>(to)[at[k]] = h[k];
            }
          }
        }
        cp_async_commit();
      };
      fetch(0);
      issue(0);
      fetch(1);
      issue(1);
      fetch(2);
      for (int32_t b = 0; b < nb; b++) {
        cp_async_wait_group<1>();  // this warp's part of batch b has landed
        __syncthreads();
        issue(b + 2);
        fetch(b + 3);
      }
      cp_async_wait_all();
    }
    __syncthreads();  // the buffers are free again
  }
  if (prod < 0) {
#pragma unroll
    for (int x = 0; x < CN; x++)
      if (lane < nw && lane * CN + x < W) crow[lane * CN + x] = Vec<ST>::from_f(acc[x]);
  }
}

// Long rows of tile columns [tj0, tj0 + tjn), a block per (row, tile column,
// panel).  `met`: list[0, count[0]) holds the rows that k_spmm_narrow met (its
// programmatic dependent: it waits for it);
// otherwise the rows k_spmm_find_long listed, and k_spmm_narrow may start.
template <typename ST, bool SUB, bool MANY>
__global__ void __launch_bounds__(kChainWarps * 32, 2)
    k_spmm_chain(SpGridView A, DGridView B, DGridView C, int tj0, int tjn, int npanels, int stride, bool met,
                 const int64_t* __restrict__ list, const int32_t* __restrict__ count,
                 unsigned long long* __restrict__ next_item) {
  if (met) asm volatile("griddepcontrol.wait;\n" ::: "memory");
  else asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  extern __shared__ __align__(16) unsigned char chain_smem[];
  __shared__ int64_t item[2], row[2];
  uint32_t* slices = reinterpret_cast<uint32_t*>(chain_smem);
  float* vals = reinterpret_cast<float*>(slices + kChainBuffers * (kChainWarps - 1) * kChainEach * stride + kChainPanelWords);
  constexpr int PW = kChainPanelWords * 4 / (int)sizeof(ST);
  const int64_t rows = A.gm * A.tm;
  const int64_t nv = count[0], nl = nv + (met ? 0 : count[1]);
  const int64_t per = tjn * (int64_t)npanels;
  const int64_t n = nl * per;
  // thread 0 takes an item and reads its row ahead, while the block works on
  // the one before
  auto take = [&](int slot) {
    const int64_t it = (int64_t)atomicAdd(next_item, 1ULL);
    item[slot] = it < n ? it : -1;
    if (it < n) {
      const int64_t q = it / per;
      row[slot] = q < nv ? list[q] : list[rows - 1 - (q - nv)];
    }
  };
  if (threadIdx.x == 0) take(0);
  __syncthreads();
  for (int slot = 0;; slot ^= 1) {
    const int64_t it = item[slot];
    if (it < 0) break;
    const int64_t x = row[slot];  // over all tile rows
    const int64_t pt = it % per;
    const int64_t tj = tj0 + pt / npanels;
    const int64_t ti = x / A.tm;
    const int W = (int)C.cols_of(tj), c0 = (int)(pt % npanels) * PW;
    if (threadIdx.x == 0) take(slot ^ 1);
    if (c0 < W) {
      const int unit = tile_on<ST, 16>(B, C, ti, tj, W) ? 16 : (tile_on<ST, 4>(B, C, ti, tj, W) ? 4 : 2);
      chain_row<ST, SUB, MANY>(slices, vals, stride, A, B, C, ti, tj, x - ti * A.tm, c0, min(PW, W - c0), unit);
    } else {
      __syncthreads();  // (chain_row ends with a barrier)
    }
  }
}

// Short rows of tile columns [tj0, tj0 + tjn); the long rows are left to
// k_spmm_chain, and listed for it (MetRows) unless they are listed already.
template <typename ST, int U, int NV, bool SUB>
__global__ void __launch_bounds__(kNarrowWarps * 32, NV == 4 ? 3 : 4)
    k_spmm_narrow(SpGridView A, DGridView B, DGridView C, int tj0, int tjn, int L, int npanels, int64_t n_items,
                  int64_t ngroups, MetRows met, unsigned long long* __restrict__ next_item) {
  constexpr int PW = 32 * NV * Unit<ST, U>::N;  // columns of a panel
  const int lane = lane_id();
  unsigned long long it = 0;
  if (lane == 0) it = atomicAdd(next_item, 1ULL);
  it = __shfl_sync(kFull, it, 0);
  int64_t at = -1, ti = 0, tj = 0;  // the C tile of the last item
  bool on = false;
  int long_row = met.most;
  while ((int64_t)it < n_items) {
    unsigned long long nx = 0;
    if (lane == 0) nx = atomicAdd(next_item, 1ULL);
    const int64_t rg = npanels == 1 ? (int64_t)it : (int64_t)it / npanels;
    const int panel = (int)((int64_t)it - rg * npanels);
    const int64_t t = rg / ngroups;
    const int64_t r0 = (rg - t * ngroups) * (32 / L);
    if (t != at) {
      at = t;
      ti = t / tjn;
      tj = tj0 + (t - ti * tjn);
      on = tile_on<ST, U>(B, C, ti, tj, (int)C.cols_of(tj));
      long_row = met_bound(met, A, C, ti);
    }
    const int W = (int)C.cols_of(tj);
    const int c0 = panel * PW;
    if (r0 < C.rows_of(ti) && c0 < W) {
      const int c1 = min(W, c0 + PW);
      unsigned left;
      if (on) left = narrow_rows<ST, U, NV, SUB>(A, B, C, ti, tj, r0, L, c0, c1 - c0, long_row);
      else left = elem_rows<ST, SUB>(A, B, C, ti, tj, r0, min(r0 + 32 / L, C.rows_of(ti)), c0, c1, long_row);
      if (left && met.list && tj == tj0 && panel == 0)
        list_met<sizeof(ST) == 4 && U == 16>(met, ti * A.tm + r0, left);
    }
    it = __shfl_sync(kFull, nx, 0);
  }
  // launched as k_spmm_chain's programmatic dependent: finish only after it
  // (a normal launch returns here at once)
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// Launch delay of the short-row kernel under the side-stream schedule: a
// one-warp kernel on the main stream that returns after `ns` (global timer,
// bounded by an iteration cap; it waits for nothing), so that the long-row
// blocks, which each need a whole SM's shared memory, are placed first.
constexpr unsigned kLongHeadStartNs = 4000;

__global__ void k_spmm_launch_delay(unsigned ns) {
  uint64_t t0;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (int i = 0; i < 4096; i++) {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t - t0 >= ns) break;
    __nanosleep(256);
  }
}

// Blocks of k_spmm_long (one per SM: its shared memory fills the SM); the
// other SMs run k_spmm.  By default five twelfths of the SMs (61): with 49, 62
// and 74, R-MAT s21 x 256 FP32 3.84, 3.52 and 3.69 ms, BF16 2.02, 1.91 and 1.93;
// R-MAT of 1,000,000 rows x 256 FP32 2.03, 1.67 and 1.64, BF16 1.17, 1.13 and
// 1.16; of 300,000 x 128 FP32 401, 388 and 386 us.  BCLX_TUNE_SPMM_LONG_BLOCKS
// sets the count.
static int spmm_long_blocks(const Context* ctx) {
  int b = (int)tuning(ctx, BCLX_TUNE_SPMM_LONG_BLOCKS);
  if (b <= 0) b = ctx->num_sms * 5 / 12;
  return std::max(1, std::min(b, ctx->num_sms));
}

static int64_t spmm_long_min_rows() {
  const char* e = std::getenv("BCLX_SPMM_LONG_MIN_ROWS");
  return e && *e ? std::strtoll(e, nullptr, 10) : kSpmmLongMinRows;
}

// Rows per k_spmm warp item: grouping short rows shares one prologue (tile
// descriptors, row pointers, A loads) among them, while the items still
// cover every resident warp.  BCLX_TUNE_SPMM_ROWS (1, 2, 4) overrides.
static int spmm_rows_per_item(const Context* ctx, const DGridView& C, int64_t tjn, int64_t gk, int npanels) {
  auto fits = [&](int r) { return r <= kSpmmMaxRows && r * gk <= 32; };
  const int want = (int)tuning(ctx, BCLX_TUNE_SPMM_ROWS);
  if ((want == 1 || want == 2 || want == 4) && fits(want)) return want;
  const int64_t resident = (int64_t)ctx->num_sms * 4 * kSpmmWarps;
  int r = 1;
  while (fits(2 * r) && C.gm * tjn * ceil_div(C.tm, (int64_t)(2 * r)) * npanels >= resident) r *= 2;
  return r;
}

// Two schedules of the long-row and short-row kernels (BCLX_TUNE_SPMM_SCHEDULE):
//  0 (default): the long rows on the context's side stream at the highest
//    priority; k_spmm on the main stream after the list is ready and a
//    4-microsecond launch delay, so the long-row blocks take their SMs first;
//  1: one stream; k_spmm launched as k_spmm_long's programmatic dependent
//    (it launches once every long-row block has started, and finishes only
//    after k_spmm_long).
// Measured on R-MAT s21 x 256 (one B200): schedule 0 3.46 ms FP32 / 1.89 ms
// BF16, schedule 1 3.63 / 1.90 ms.  Also measured, with one warp for both parts
// of a long row (4.14 and 2.45 ms), and slower: one-warp
// long-row blocks small enough to share every SM with four k_spmm blocks
// (k_spmm capped at 56 registers, both kernels at the largest shared-memory
// carveout): 5.08 / 3.91 ms, k_spmm alone losing 15 % to the smaller L1;
// and one cp.async.bulk copy per 512-byte B slice, completing on an
// mbarrier, in place of the per-lane copies: 6.8 ms for k_spmm_long alone
// against 1.9.
template <typename ST, bool SUB>
static int launch_wide(Context* ctx, const SpGridView& A, const DGridView& B, const DGridView& C, int tjn, int align_ok) {
  constexpr int VN = Vec<ST>::N;
  const int npanels = (int)ceil_div(C.tn, 32 * VN);
  const int R = spmm_rows_per_item(ctx, C, tjn, A.gn, npanels);
  const int64_t ngroups = ceil_div(C.tm, (int64_t)R);
  const int64_t n_items = C.gm * tjn * ngroups * npanels;
  if (n_items == 0) return BCLX_OK;
  const int64_t want = ceil_div(n_items, kSpmmWarps);
  const int64_t cap = (int64_t)ctx->num_sms * 4;  // resident blocks: warps take items from a counter
  const int64_t arows = A.gm * A.tm;
  const bool long_path = align_ok && A.gn <= 32 && arows >= spmm_long_min_rows();
  // rows of at least long_row entries go to the long-row kernel: by default
  // 512 (R-MAT s21 x 256: FP32 3.52 against 3.81 ms with 1024, BF16 1.91 against
  // 2.05; of 300,000 rows x 256 BF16 425 against 528 us)
  int long_row = (int)tuning(ctx, BCLX_TUNE_SPMM_LONG_ROW);
  if (long_row <= 0) long_row = 512;
  const bool dependent = tuning(ctx, BCLX_TUNE_SPMM_SCHEDULE) == 1;
  // counters: [0] k_spmm items, [1] k_spmm_long items, [2] listed very long / other long rows (2 x int32)
  unsigned long long* ctr = nullptr;
  BCLX_TRY(scratch_alloc_n(ctx, &ctr, 3));
  BCLX_CK(cudaMemsetAsync(ctr, 0, 3 * sizeof(unsigned long long), ctx->stream));
  int32_t* cnt = reinterpret_cast<int32_t*>(ctr + 2);
  uint8_t* flag = nullptr;
  int64_t* list = nullptr;
  if (long_path) {
    BCLX_TRY(scratch_alloc_n(ctx, &flag, (size_t)arows));
    BCLX_TRY(scratch_alloc_n(ctx, &list, (size_t)arows));
    cudaStream_t ls = ctx->stream;
    if (!dependent) {
      BCLX_TRY(ensure_side_stream(ctx));
      BCLX_CK(cudaEventRecord(ctx->fork_ev, ctx->stream));
      BCLX_CK(cudaStreamWaitEvent(ctx->side, ctx->fork_ev, 0));
      ls = ctx->side;
    }
    k_spmm_find_long<<<(unsigned)std::min<int64_t>(ceil_div(arows, 256), (int64_t)ctx->num_sms * 16), 256, 0,
                       ls>>>(A, long_row, long_row * 8, flag, list, cnt);
    note_launch();
    BCLX_CK_LAUNCH();
    if (!dependent) BCLX_CK(cudaEventRecord(ctx->fork2_ev, ctx->side));
    const size_t lsmem = sizeof(LongSmem) * kLongPairs;
    BCLX_CK(cudaFuncSetAttribute(k_spmm_long<ST, SUB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lsmem));
    k_spmm_long<ST, SUB><<<(unsigned)spmm_long_blocks(ctx), kLongPairs * 64, lsmem, ls>>>(A, B, C, tjn, list, cnt, npanels,
                                                                                    align_ok, ctr + 1);
    note_launch();
    BCLX_CK_LAUNCH();
    if (!dependent) {
      BCLX_CK(cudaEventRecord(ctx->join_ev, ctx->side));
      BCLX_CK(cudaStreamWaitEvent(ctx->stream, ctx->fork2_ev, 0));
      k_spmm_launch_delay<<<1, 32, 0, ctx->stream>>>(kLongHeadStartNs);
      note_launch();
      BCLX_CK_LAUNCH();
    }
  }
  const unsigned grid = (unsigned)(want < cap ? want : cap);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kSpmmWarps * 32);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (long_path && dependent) ? 1 : 0;
  const uint8_t* lflag = flag;
  const int pmajor = (int)tuning(ctx, BCLX_TUNE_SPMM_PANEL_MAJOR);
  if (R > 1)
    BCLX_CK(cudaLaunchKernelEx(&cfg, k_spmm<ST, true, SUB, 0>, A, B, C, tjn, n_items, npanels, R, ngroups, align_ok, pmajor, lflag,
                               false, MetRows{}, ctr));
  else
    BCLX_CK(cudaLaunchKernelEx(&cfg, k_spmm<ST, false, SUB, 0>, A, B, C, tjn, n_items, npanels, 1, ngroups, align_ok, pmajor, lflag,
                               false, MetRows{}, ctr));
  note_launch();
  BCLX_CK_LAUNCH();
  if (long_path) {
    if (!dependent) BCLX_CK(cudaStreamWaitEvent(ctx->stream, ctx->join_ev, 0));
    scratch_free(ctx, flag);
    scratch_free(ctx, list);
  }
  scratch_free(ctx, ctr);
  return BCLX_OK;
}

// Launch `kern` so that it may start before the kernel ahead of it in the
// stream has finished (`early`; not inside a capture, where launches stay in
// plain order).
template <typename... KP, typename... AP>
static int launch_after(Context* ctx, bool early, unsigned grid, unsigned threads, size_t smem, void (*kern)(KP...),
                        AP... args) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (early) BCLX_CK(cudaStreamIsCapturing(ctx->stream, &cap));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early && cap == cudaStreamCaptureStatusNone ? 1 : 0;
  BCLX_CK(cudaLaunchKernelEx(&cfg, kern, KP(args)...));
  note_launch();
  return BCLX_OK;
}

// k_spmm_narrow and k_spmm_chain over tile columns [tj0, tj0 + tjn), `width`
// columns each (the last may have fewer), rows on U bytes.
template <typename ST, int U, int NV, bool SUB>
static int launch_narrow_nv(Context* ctx, const SpGridView& A, const DGridView& B, const DGridView& C, int tj0,
                            int tjn, int64_t width, int L, bool wide_rows) {
  constexpr int PW = 32 * NV * Unit<ST, U>::N;
  const int npanels = (int)ceil_div(width, PW);
  const int64_t ngroups = ceil_div(C.tm, (int64_t)(32 / L));
  const int64_t n_items = C.gm * tjn * ngroups * npanels;
  if (n_items == 0) return BCLX_OK;
  // long rows: slices a power of two of words apart
  int stride = 4;
  while (stride < kChainPanelWords && stride * 4 < width * (int64_t)sizeof(ST)) stride *= 2;
  const size_t smem = chain_bytes(stride);
  const int64_t arows = A.gm * A.tm;
  // (the kernels of short rows tell a long row by its first 32 stages at most, or by its flag, which k_spmm reads)
  const bool listed = arows >= spmm_long_min_rows() && (A.gn <= 32 || wide_rows);
  const bool chains = A.gn <= 32 || listed;
  int long_row = (int)tuning(ctx, BCLX_TUNE_SPMM_LONG_ROW);
  const bool few = chains && !listed && long_row <= 0;
  if (long_row <= 0) long_row = std::min(kNarrowLongSteps * L, listed && wide_rows ? 512 : INT_MAX);
  if (!chains) long_row = INT_MAX;
  const int long_least = few ? std::min(kNarrowFewLong, long_row) : long_row;
  // one scratch block: counters ([0] row groups taken, [1] long rows taken, [2] listed very long / other long rows,
  // 2 x int32), the list of long rows, and their flags where they are listed first
  unsigned long long* ctr = nullptr;
  BCLX_TRY(scratch_alloc(ctx, reinterpret_cast<void**>(&ctr),
                         sizeof(int64_t) * (size_t)(3 + (chains ? arows : 0)) + (size_t)(listed ? arows : 0)));
  BCLX_CK(cudaMemsetAsync(ctr, 0, 3 * sizeof(unsigned long long), ctx->stream));
  int32_t* cnt = reinterpret_cast<int32_t*>(ctr + 2);
  int64_t* list = chains ? reinterpret_cast<int64_t*>(ctr + 3) : nullptr;
  uint8_t* flag = listed ? reinterpret_cast<uint8_t*>(list + arows) : nullptr;
  const MetRows met{listed ? nullptr : list, cnt, long_row, long_least};
  if (listed) {
    k_spmm_find_long<<<(unsigned)std::min<int64_t>(ceil_div(arows, 256), (int64_t)ctx->num_sms * 16), 256, 0,
                       ctx->stream>>>(A, long_row, (int)std::min<int64_t>((int64_t)long_row * 8, INT32_MAX), flag, list, cnt);
    note_launch();
    BCLX_CK_LAUNCH();
  }
  auto narrow = [&]() {
    const int64_t blocks = std::min(ceil_div(n_items, kNarrowWarps), (int64_t)ctx->num_sms * 4);
    return launch_after(ctx, listed, (unsigned)blocks, kNarrowWarps * 32, 0, k_spmm_narrow<ST, U, NV, SUB>, A, B, C,
                        tj0, tjn, L, npanels, n_items, ngroups, met, ctr);
  };
  // A lane group of 32 takes one row; k_spmm shares a warp's set-up among up to
  // four, and a panel of its lanes is 512 bytes.  So it takes the short rows there:
  // k_spmm_narrow against k_spmm, uniform 186,581 x 150 FP32, 5 entries a row, 438
  // and 201 us; stencil of 262,144 x 185 BF16 1041 and 587; uniform 8,069 x 201 43
  // and 35; R-MAT FP32 of 273,612 x 118 570 and 524, of 300,000 x 201 1184 and 1001,
  // of 1,432,750 x 87 2467 and 2360, of 20,000 x 201 on 20 x 20 tiles 161 and 139 (long
  // rows listed and met: from 512 entries, or see kNarrowFewLong).  With 17 tiles along
  // k and more every row takes 32 lanes, and k_spmm has the lighter set-up for one as
  // well (by 16-byte vectors where the rows lie on 16 bytes): R-MAT of 400,000 on 20 x
  // 20 tiles, x 16 FP32 488 and 410 us (k_spmm with its own long rows, as launch_wide
  // runs it: 640), x 64 572 and 495 (650), x 64 BF16 649 and 479 (798), x 17 FP32 577
  // and 420, x 47 597 and 528; uniform 20,000 x 64 BF16 49 and 43; on 33 x 33 tiles, where
  // k_spmm_narrow had no chains, R-MAT of 400,000 x 16 FP32 1865 and 502, x 47 2469 and 627,
  // x 64 BF16 3306 and 575.  Rows of fewer units stay with k_spmm_narrow: R-MAT of
  // 100,000 x 47 177 and 250.
  auto wide = [&]() {
    constexpr int VN = Vec<ST>::N;
    // rows of 64 columns and fewer (here for the stages' sake): two columns a lane, eight entries' loads in flight
    const bool two = U != 16 && width <= 64;
    const int wp = (int)ceil_div(width, 32 * (two ? 2 : VN));
    const int R = two ? 1 : spmm_rows_per_item(ctx, C, tjn, A.gn, wp);
    const int64_t groups = ceil_div(C.tm, (int64_t)R), items = C.gm * tjn * groups * wp;
    const int64_t blocks = std::min(ceil_div(items, kSpmmWarps), (int64_t)ctx->num_sms * 4);
    const uint8_t* skip = flag;
    auto go = [&](auto kern) {
      return launch_after(ctx, listed, (unsigned)blocks, kSpmmWarps * 32, 0, kern, A, B, C, tjn, items, wp, R, groups, 1,
                          0, skip, true, met, ctr);
    };
    if constexpr (U == 16) {  // (only for 17 and more tiles along k: R is 1)
      return met.list ? go(k_spmm<ST, false, SUB, 0, true>) : go(k_spmm<ST, false, SUB, 0>);
    } else {
      if (two) return met.list ? go(k_spmm<ST, false, SUB, 2, true>) : go(k_spmm<ST, false, SUB, 2>);
      if (met.list) return R > 1 ? go(k_spmm<ST, true, SUB, VN, true>) : go(k_spmm<ST, false, SUB, VN, true>);
      return R > 1 ? go(k_spmm<ST, true, SUB, VN>) : go(k_spmm<ST, false, SUB, VN>);
    }
  };
  if (!listed) BCLX_TRY(wide_rows ? wide() : narrow());
  if (chains) {
    auto kern = A.gn <= 32 ? k_spmm_chain<ST, SUB, false> : k_spmm_chain<ST, SUB, true>;
    BCLX_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // one block per SM beside k_spmm_narrow, two where it has finished
    const int64_t blocks = std::min<int64_t>(arows * tjn, (int64_t)ctx->num_sms * (listed ? 1 : 2));
    BCLX_TRY(launch_after(ctx, !listed, (unsigned)blocks, kChainWarps * 32, smem, kern, A, B, C, tj0, tjn,
                          (int)ceil_div(width * (int64_t)sizeof(ST), 4 * kChainPanelWords), stride, !listed, list,
                          cnt, ctr + 1));
  }
  if (listed) BCLX_TRY(wide_rows ? wide() : narrow());
  scratch_free(ctx, ctr);
  return BCLX_OK;
}

// Lanes per row: one 16-byte vector per lane, or up to four words (each lane
// then loads as many bytes); at least as many as stages, so that a warp's
// (row, stage) segments fit its lanes.
template <typename ST, int U, bool SUB>
static int launch_narrow_u(Context* ctx, const SpGridView& A, const DGridView& B, const DGridView& C, int64_t tj0,
                           int64_t tjn, int64_t width) {
  const int64_t units = ceil_div(width * (int64_t)sizeof(ST), U);
  const int per = U == 16 ? 1 : 4;
  int L = 8;
  while (L < 32 && (L * per < units || L < A.gn)) L *= 2;
  const int64_t nv = ceil_div(std::min<int64_t>(units, 32 * per), L);
  // rows that take all 32 lanes, for their width or for the stages' sake (k_spmm
  // starts at tile column 0): see `wide` in launch_narrow_nv.  Not BF16 rows off 16
  // bytes where they are few: R-MAT of 54,871 x 178 209 us with k_spmm_narrow, 233 with
  // k_spmm (uniform 8,069 x 252 36 and 34).
  const bool wide_rows = L == 32 && tj0 == 0 && (sizeof(ST) == 4 || A.gn > 16 || A.gm * A.tm >= spmm_long_min_rows());
  if constexpr (U != 16) {
    if (nv > 2) return launch_narrow_nv<ST, U, 4, SUB>(ctx, A, B, C, (int)tj0, (int)tjn, width, L, wide_rows);
    if (nv > 1) return launch_narrow_nv<ST, U, 2, SUB>(ctx, A, B, C, (int)tj0, (int)tjn, width, L, wide_rows);
  }
  return launch_narrow_nv<ST, U, 1, SUB>(ctx, A, B, C, (int)tj0, (int)tjn, width, L, wide_rows);
}

template <typename ST, bool SUB>
static int launch_narrow(Context* ctx, const SpGridView& A, const DGridView& B, const DGridView& C, int64_t tj0,
                         int64_t tjn, int64_t width) {
  const int64_t es = (int64_t)sizeof(ST);
  const int64_t low = (B.ld * es) | (C.ld * es) | (width * es) |
                      (B.tiles ? 0 : (int64_t)(reinterpret_cast<uintptr_t>(B.single) | reinterpret_cast<uintptr_t>(C.single)));
  if (low % 16 == 0) return launch_narrow_u<ST, 16, SUB>(ctx, A, B, C, tj0, tjn, width);
  if constexpr (sizeof(ST) == 2) {
    if (low % 4 != 0) return launch_narrow_u<ST, 2, SUB>(ctx, A, B, C, tj0, tjn, width);
  }
  return launch_narrow_u<ST, 4, SUB>(ctx, A, B, C, tj0, tjn, width);
}

// Which kernel takes which tile columns: k_spmm_narrow those whose rows are
// narrow (at most kNarrowMaxBytes) or not whole 16-byte vectors, k_spmm (with
// k_spmm_long) the others.  The last tile column may be narrower than the rest.
template <typename ST, bool SUB>
static int launch_spmm(Context* ctx, const SpGridView& A, const DGridView& B, const DGridView& C, int align_ok) {
  if (C.gn == 0 || C.gm == 0) return BCLX_OK;
  const int64_t last = C.n - (C.gn - 1) * C.tn;
  const bool narrow = !align_ok || C.tn * (int64_t)sizeof(ST) <= kNarrowMaxBytes;
  const bool split = C.gn > 1 ? last % Vec<ST>::N != 0 : false;
  if (C.gn == 1) {
    if (narrow || last % Vec<ST>::N != 0) return launch_narrow<ST, SUB>(ctx, A, B, C, 0, 1, last);
    return launch_wide<ST, SUB>(ctx, A, B, C, 1, align_ok);
  }
  const int64_t tjn = split ? C.gn - 1 : C.gn;
  if (narrow) BCLX_TRY((launch_narrow<ST, SUB>(ctx, A, B, C, 0, tjn, C.tn)));
  else BCLX_TRY((launch_wide<ST, SUB>(ctx, A, B, C, (int)tjn, align_ok)));
  return split ? launch_narrow<ST, SUB>(ctx, A, B, C, tjn, 1, last) : BCLX_OK;
}

static int run_spmm(Context* ctx, const SpGridView& A, const DGridView& B, const DGridView& C, int dtype) {
  const int es = dtype == BCLX_F32 ? 4 : 2;
  const int align_ok = ((B.ld * es) % 16 == 0) && ((C.ld * es) % 16 == 0);
  if (B.rot_i) {  // a sub-grid (bclx_spmm_grid_sub): stage maps
    if (dtype == BCLX_F32) return launch_spmm<float, true>(ctx, A, B, C, align_ok);
    return launch_spmm<__nv_bfloat16, true>(ctx, A, B, C, align_ok);
  }
  if (dtype == BCLX_F32) return launch_spmm<float, false>(ctx, A, B, C, align_ok);
  return launch_spmm<__nv_bfloat16, false>(ctx, A, B, C, align_ok);
}

}  // namespace bclx

using namespace bclx;

extern "C" {

int bclx_spmm_tile(bclx_context_t c, int64_t m, int64_t n, int64_t k, int64_t nnz, void* cp, const void* bp,
                   const float* a_values, const int32_t* a_rowptr, const int32_t* a_colind, int64_t ldb,
                   int64_t ldc, int32_t bc_dtype) {
  Context* ctx = reinterpret_cast<Context*>(c);
  if (!ctx || m < 0 || n < 0 || k < 0 || nnz < 0) return BCLX_ERR_INVALID;
  if (bc_dtype != BCLX_F32 && bc_dtype != BCLX_BF16) return BCLX_ERR_DTYPE;
  if (m == 0 || n == 0) return BCLX_OK;
  if (!cp || !bp || !a_rowptr || (nnz > 0 && (!a_values || !a_colind)) || ldb < n || ldc < n)
    return BCLX_ERR_INVALID;
  if (n > INT32_MAX || m > INT32_MAX) return BCLX_ERR_INDEX_OVERFLOW;
  BCLX_CK(cudaSetDevice(ctx->device));
  SpGridView A{};
  A.tiles = nullptr;
  A.single.m = m; A.single.n = k; A.single.nnz = nnz;
  A.single.row_ptr = const_cast<int32_t*>(a_rowptr);
  A.single.col_ind = const_cast<int32_t*>(a_colind);
  A.single.vals = const_cast<float*>(a_values);
  A.single.dtype = BCLX_F32;
  A.m = m; A.n = k > 0 ? k : 1; A.tm = m; A.tn = A.n; A.gm = 1; A.gn = 1;
  DGridView B{};
  B.tiles = nullptr; B.single = const_cast<void*>(bp);
  B.m = A.n; B.n = n; B.tm = A.n; B.tn = n; B.gm = 1; B.gn = 1; B.ld = ldb;
  DGridView C{};
  C.tiles = nullptr; C.single = cp;
  C.m = m; C.n = n; C.tm = m; C.tn = n; C.gm = 1; C.gn = 1; C.ld = ldc;
  return run_spmm(ctx, A, B, C, bc_dtype);
}

static int spmm_grid_impl(bclx_context_t c, const bclx_spgrid_t* a, const bclx_dgrid_t* b, const bclx_dgrid_t* cg,
                          int natural_order, const int64_t* tile_rows = nullptr,
                          const int64_t* tile_cols = nullptr) {
  Context* ctx = reinterpret_cast<Context*>(c);
  if (!ctx || !a || !b || !cg || !a->tiles || !b->tiles || !cg->tiles) return BCLX_ERR_INVALID;
  if (a->dtype != BCLX_F32) return BCLX_ERR_DTYPE;
  if (b->dtype != cg->dtype || (b->dtype != BCLX_F32 && b->dtype != BCLX_BF16)) return BCLX_ERR_DTYPE;
  auto grid_ok = [](int64_t m, int64_t n, int64_t tm, int64_t tn, int64_t gm, int64_t gn) {
    return m >= 0 && n >= 0 && tm > 0 && tn > 0 && gm == ceil_div(m, tm) && gn == ceil_div(n, tn);
  };
  if (!grid_ok(a->m, a->n, a->tile_m, a->tile_n, a->grid_m, a->grid_n) ||
      !grid_ok(b->m, b->n, b->tile_m, b->tile_n, b->grid_m, b->grid_n) ||
      !grid_ok(cg->m, cg->n, cg->tile_m, cg->tile_n, cg->grid_m, cg->grid_n))
    return BCLX_ERR_INVALID;
  if (a->m != cg->m || a->n != b->m || b->n != cg->n) return BCLX_ERR_INVALID;
  if (a->tile_m != cg->tile_m || a->tile_n != b->tile_m || b->tile_n != cg->tile_n) return BCLX_ERR_INVALID;
  if (cg->tile_n > INT32_MAX) return BCLX_ERR_INDEX_OVERFLOW;
  BCLX_CK(cudaSetDevice(ctx->device));
  SpGridView A = make_view(*a);
  DGridView B{};
  B.tiles = b->tiles; B.m = b->m; B.n = b->n; B.tm = b->tile_m; B.tn = b->tile_n; B.gm = b->grid_m;
  B.gn = b->grid_n; B.ld = b->tile_n;
  B.natural_order = natural_order;
  DGridView C{};
  C.tiles = cg->tiles; C.m = cg->m; C.n = cg->n; C.tm = cg->tile_m; C.tn = cg->tile_n; C.gm = cg->grid_m;
  C.gn = cg->grid_n; C.ld = cg->tile_n;
  if (!tile_rows || a->grid_n == 0 || cg->grid_m == 0 || cg->grid_n == 0) return run_spmm(ctx, A, B, C, b->dtype);
  // sub-grid: the stage maps, on the device for the launch
  std::vector<int32_t> maps((size_t)(cg->grid_m + cg->grid_n));
  for (int64_t i = 0; i < cg->grid_m; i++) maps[(size_t)i] = (int32_t)(tile_rows[i] % a->grid_n);
  for (int64_t j = 0; j < cg->grid_n; j++) maps[(size_t)(cg->grid_m + j)] = (int32_t)(tile_cols[j] % a->grid_n);
  int32_t* dmaps = nullptr;
  BCLX_TRY(scratch_alloc_n(ctx, &dmaps, maps.size()));
  cudaError_t e = cudaMemcpyAsync(dmaps, maps.data(), sizeof(int32_t) * maps.size(), cudaMemcpyHostToDevice,
                                  ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);  // the host vector goes out of scope
  if (e != cudaSuccess) {
    scratch_free(ctx, dmaps);
    set_last_error(std::string("stage maps: ") + cudaGetErrorString(e));
    return BCLX_ERR_CUDA;
  }
  B.rot_i = dmaps;
  B.rot_j = dmaps + cg->grid_m;
  const int rc = run_spmm(ctx, A, B, C, b->dtype);
  scratch_free(ctx, dmaps);  // stream-ordered: after the launches (the side stream is joined)
  return rc;
}

int bclx_spmm_grid(bclx_context_t c, const bclx_spgrid_t* a, const bclx_dgrid_t* b, const bclx_dgrid_t* cg) {
  return spmm_grid_impl(c, a, b, cg, 0);
}

int bclx_spmm_grid_rowwise(bclx_context_t c, const bclx_spgrid_t* a, const bclx_dgrid_t* b, const bclx_dgrid_t* cg) {
  return spmm_grid_impl(c, a, b, cg, 1);
}

int bclx_spmm_grid_sub(bclx_context_t c, const bclx_spgrid_t* a, const bclx_dgrid_t* b, const bclx_dgrid_t* cg,
                       const int64_t* tile_rows, const int64_t* tile_cols) {
  if (!cg || !tile_rows || !tile_cols) return BCLX_ERR_INVALID;
  // global tile indices increasing (so only the last may be a ragged edge tile)
  for (int64_t i = 0; i < cg->grid_m; i++)
    if (tile_rows[i] < 0 || tile_rows[i] >= INT32_MAX || (i > 0 && tile_rows[i] <= tile_rows[i - 1]))
      return BCLX_ERR_INVALID;
  for (int64_t j = 0; j < cg->grid_n; j++)
    if (tile_cols[j] < 0 || tile_cols[j] >= INT32_MAX || (j > 0 && tile_cols[j] <= tile_cols[j - 1]))
      return BCLX_ERR_INVALID;
  return spmm_grid_impl(c, a, b, cg, 0, tile_rows, tile_cols);
}

}  // extern "C"
