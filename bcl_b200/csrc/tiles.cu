// Whole matrix <-> tile grid on the device: the slicing of a CSR matrix into
// the packed SPMatrix tile layout (what the SPMatrix(fname, blocking)
// constructor does on the host, SPMatrix.hpp:194-271 with
// CSRMatrix::get_slice_impl_, CSRMatrix.hpp:238-276), and its inverse, the
// gather of every tile back into one CSR matrix (SPMatrix::get,
// SPMatrix.hpp:516-546).  Both are byte moves:
//
//   tiling   1. every entry: check (columns ascending and in range) and count
//               the entries of each (row, tile column) run;
//            2. one exclusive scan over all counts gives every entry's tile
//               offset and local row pointer at once;
//            3. every entry goes to its tile at start(tile, row) + (position -
//               start of its run), unless 1. found a bad row.
//   gather   1. thread per row: the row's length over its tile columns;
//            2. scan -> row_ptr;  3. every entry from its run, the runs of a
//               row in tile column order, columns shifted to global.
//
// The passes over the entries give each warp kChunk rows and entries together,
// whatever rows they belong to, so that neither a hub row of a power-law
// graph nor a thousand near-empty ones are one warp's serial walk.
// Bound: the latency of the dependent loads (row pointer, entry, scattered
// offsets), all from L2.  R-MAT s19, 8.3M entries on 8x8 tiles, a warp per row
// before -> now: check and count 598 -> 97 us, scatter 1430 -> 119, gather 427 ->
// 123 (33, 134 and 134 MB of entries in and out: 5, 20 and 20 us at the HBM
// rate).
#include "common.cuh"

#include <algorithm>
#include <climits>
#include <string>

namespace bclx {

constexpr int kChunk = 512;  // rows and entries of a warp, together

// Largest row r with (rp[r] - p0) + r <= d: the row that the walk over rows and
// entries is in at its position d (at entry p0 + d - r).
template <typename T>
__device__ __forceinline__ int64_t row_at(const T* __restrict__ rp, int64_t m, int64_t p0, int64_t d) {
  int64_t lo = 0, hi = m - 1;
  while (lo < hi) {
    const int64_t mid = lo + ((hi - lo + 1) >> 1);
    if ((int64_t)__ldg(rp + mid) - p0 + mid <= d) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Walk the CSR entries, each warp kChunk rows and entries together, 32
// entries at a time: f(on, bad, p, c, slot, start, lead) on every lane,
// warp-uniformly: entry p (when `on`) goes to (tile, local row) slot `slot` as
// tile column c, begins its run when `start`, and is the first of the batch
// or of its run when `lead`; `bad`: its column is outside [0, n) or not above
// the one before it in the row.  chunk(r, c0, p) comes before a chunk's first
// batch with that entry's row, first column of its tile and position.
// `marks` (shared, kChunk per warp): at each row's first entry in the chunk,
// the row; a running maximum then gives every entry's row.
template <typename FC, typename F>
__device__ __forceinline__ void walk_entries(int64_t m, int64_t n, const int32_t* __restrict__ rp,
                                             const int32_t* __restrict__ ci, int64_t tm, int64_t tn, int64_t gn,
                                             uint16_t* marks, FC&& chunk, F&& f) {
  const int lane = lane_id();
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t p0 = __ldg(rp), p1 = __ldg(rp + m);
  for (int64_t D = warp * kChunk; D < p1 - p0 + m; D += nwarps * kChunk) {
    const int64_t ra = row_at(rp, m, p0, D), rb = row_at(rp, m, p0, D + kChunk);
    const int64_t P = max(p0 + D - ra, p0), E = min(min(p0 + D + kChunk - rb, P + kChunk), p1);
    if (P >= E) continue;
    __syncwarp();
    for (int i = lane; i < kChunk / 8; i += 32) reinterpret_cast<uint4*>(marks)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    const int64_t rl = min(min(rb, ra + kChunk), m - 1);
    for (int64_t r = ra + lane; r <= rl; r += 32) {
      const int64_t s = __ldg(rp + r);
      if (s < __ldg(rp + r + 1) && s >= P && s < E) marks[s - P] = (uint16_t)(r - ra + 1);
    }
    __syncwarp();
    int last = 1;  // the row of the entry before the batch, less ra, plus 1
    for (int64_t b = P; b < E; b += 32) {
      const int64_t p = b + lane;
      const bool on = p < E;
      const int mark = on ? marks[p - P] : 0;
      int row = mark;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(kFull, row, d);
        if (lane >= d) row = max(row, o);
      }
      row = max(row, last);
      last = __shfl_sync(kFull, row, 31);
      const int64_t r = ra + row - 1;
      const int32_t c = on ? __ldg(ci + p) : 0;
      int32_t before = __shfl_up_sync(kFull, c, 1);
      if (lane == 0 && mark == 0) before = __ldg(ci + p - 1);
      const bool inside = c >= 0 && c < n;
      const bool bad = on && (!inside || (mark == 0 && before >= c));
      const uint32_t tj = inside ? (uint32_t)c / (uint32_t)tn : 0u;
      const bool start = on && (mark != 0 || before < 0 || (uint32_t)before / (uint32_t)tn != tj);
      const int64_t ti = r / tm;
      const int64_t slot = (ti * gn + tj) * (tm + 1) + (r - ti * tm);
      if (b == P) chunk(__shfl_sync(kFull, r, 0), (int32_t)(__shfl_sync(kFull, tj, 0) * (uint32_t)tn), P);
      f(on, bad, p, c - (int32_t)(tj * (uint32_t)tn), slot, start, start || (on && lane == 0));
    }
  }
}

// Check and count.  cnt has (tm+1) slots per tile (the last stays 0, so that
// one scan yields the tile's row pointer including its end).  A row pointer
// that descends or a bad entry sets *bad; what is counted then is not used.
__global__ void __launch_bounds__(256) k_tile_count(int64_t m, int64_t n, const int32_t* __restrict__ rp,
                                                    const int32_t* __restrict__ ci, int64_t tm, int64_t tn, int64_t gn,
                                                    int32_t* __restrict__ cnt, int32_t* __restrict__ bad) {
  __shared__ __align__(16) uint16_t marks[8][kChunk];
  const int lane = lane_id();
  bool wrong = false;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m; r += (int64_t)gridDim.x * blockDim.x)
    wrong |= __ldg(rp + r) > __ldg(rp + r + 1);
  walk_entries(
      m, n, rp, ci, tm, tn, gn, marks[threadIdx.x >> 5], [](int64_t, int32_t, int64_t) {},
      [&](bool on, bool bad_here, int64_t, int32_t, int64_t slot, bool, bool lead) {
        wrong |= bad_here;
        const unsigned leads = __ballot_sync(kFull, lead);
        const int ons = __popc(__ballot_sync(kFull, on));
        if (lead) {
          const unsigned after = lane == 31 ? 0u : leads >> (lane + 1);
          atomicAdd(cnt + slot, after ? __ffs(after) : ons - lane);
        }
      });
  if (__any_sync(kFull, wrong) && lane == 0) atomicExch(bad, 1);
}

// Local row pointers and tile offsets from the scanned counts E (nothing where *bad).
__global__ void k_tile_ptrs(const int64_t* __restrict__ E, int64_t ntiles, int64_t tm, const int32_t* __restrict__ bad,
                            int32_t* __restrict__ trp, int64_t* __restrict__ toff) {
  if (*bad) return;
  const int64_t total = ntiles * (tm + 1);
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < total; x += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = x / (tm + 1), lr = x - t * (tm + 1);
    const int64_t base = __ldg(E + t * (tm + 1));
    trp[x] = (int32_t)(E[x] - base);
    if (lr == 0) toff[t] = base;
    if (x == total - 1) toff[ntiles] = E[total];
  }
}

// Every entry to its tile (nothing where *bad).
template <typename VT>
__global__ void __launch_bounds__(256) k_tile_scatter(int64_t m, int64_t n, const int32_t* __restrict__ rp,
                                                      const int32_t* __restrict__ ci, const VT* __restrict__ va,
                                                      int64_t tm, int64_t tn, int64_t gn,
                                                      const int64_t* __restrict__ E, const int32_t* __restrict__ bad,
                                                      int32_t* __restrict__ oci, VT* __restrict__ ova) {
  __shared__ __align__(16) uint16_t marks[8][kChunk];
  if (*bad) return;
  int32_t carry = 0;  // start of the run the previous batch ended in
  walk_entries(
      m, n, rp, ci, tm, tn, gn, marks[threadIdx.x >> 5],
      [&](int64_t r, int32_t c0, int64_t p) { carry = lower_bound_i32(ci, __ldg(rp + r), (int32_t)p, c0); },
      [&](bool on, bool, int64_t p, int32_t c, int64_t slot, bool start, bool) {
        // start of this entry's run: the latest run start at or before it
        int32_t s = start ? (int32_t)p : -1;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int32_t o = __shfl_up_sync(kFull, s, d);
          if (lane_id() >= d) s = max(s, o);
        }
        if (s < 0) s = carry;
        carry = __shfl_sync(kFull, s, 31);
        if (on) {
          const int64_t dst = __ldg(E + slot) + ((int32_t)p - s);
          oci[dst] = c;
          ova[dst] = __ldg(va + p);
        }
      });
}

// Thread per global row: entries over the row's tiles.
__global__ void k_gather_len(SpGridView g, int32_t* __restrict__ len) {
  const int64_t m = g.m;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m; r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ti = r / g.tm, lr = r - ti * g.tm;
    int64_t tot = 0;
    for (int64_t tj = 0; tj < g.gn; tj++) {
      const int32_t* trp = g.tile(ti, tj).row_ptr;
      tot += __ldg(trp + lr + 1) - __ldg(trp + lr);
    }
    len[r] = (int32_t)tot;
  }
}

// (nothing where the entries exceed `most`: an int32 row pointer, or the arrays that the caller gave)
__global__ void k_rowptr32(const int64_t* __restrict__ off, int64_t m, int64_t most, int32_t* __restrict__ rp) {
  if (__ldg(off + m) > most) return;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r <= m; r += (int64_t)gridDim.x * blockDim.x)
    rp[r] = (int32_t)off[r];
}

// A value as SPMatrix::get returns it: the reference gathers through
// SparseHashAccumulator, which adds each value to a zero-initialised slot
// (SparseHashAccumulator.hpp:50-53) on the host, so -0.0 comes back as +0.0
// and a signalling NaN comes back quiet (its payload kept); every other
// value is unchanged.  int32 values pass through.
__device__ __forceinline__ int32_t gathered(int32_t v) { return v; }
__device__ __forceinline__ float gathered(float v) {
  uint32_t b = __float_as_uint(v);
  if (b == 0x80000000u) b = 0u;
  else if ((b & 0x7f800000u) == 0x7f800000u && (b & 0x007fffffu)) b |= 0x00400000u;
  return __uint_as_float(b);
}

// Each warp takes kChunk rows and entries together (row_at).  Of 32 rows at a time, lanes hold the runs of the non-empty
// ones' tile columns (32 / gn rows at once; 32 tile columns of one row on
// finer grids); flattened, the runs are the output's order, so that output q
// comes from seg + q of the run that holds it: the run is the number of runs
// that begin at or before q, from a warp-wide or of their first positions.
template <typename VT>
__global__ void __launch_bounds__(256) k_gather_rows(SpGridView g, const int64_t* __restrict__ off,
                                                     int32_t* __restrict__ oci, VT* __restrict__ ova) {
  __shared__ ulonglong2 seg_all[8][32];
  __shared__ int32_t shift_all[8][32];
  __shared__ int64_t off_all[8][32];
  __shared__ uint8_t row_all[8][32];
  const int wid = threadIdx.x >> 5;
  ulonglong2* seg = seg_all[wid];
  int32_t* shift = shift_all[wid];
  const int lane = lane_id();
  const unsigned below = (1u << lane) - 1u, upto = below | (1u << lane);
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t nnz = __ldg(off + g.m);
  if (nnz > INT32_MAX) return;
  const int gn = (int)g.gn;
  const int R = gn <= 32 ? 32 / gn : 1;
  const int rr = gn <= 32 ? lane / gn : 0;
  for (int64_t D = warp * kChunk; D < nnz + g.m; D += nwarps * kChunk) {
    const int64_t ra = row_at(off, g.m, 0, D), rb = row_at(off, g.m, 0, D + kChunk);
    const int64_t P = D - ra, end = min(D + kChunk - rb, nnz);
    for (int64_t r = ra; r <= rb; r += 32) {
      __syncwarp();
      int n_rows = 0;
      {
        const int64_t row = r + lane;
        const int64_t lo = row < g.m ? __ldg(off + row) : nnz, hi = row < g.m ? __ldg(off + row + 1) : nnz;
        const bool on = row <= rb && lo < hi && lo < end && hi > P;
        const unsigned some = __ballot_sync(kFull, on);
        if (on) {
          const int at = __popc(some & below);
          row_all[wid][at] = (uint8_t)lane;
          off_all[wid][at] = lo;
        }
        n_rows = __popc(some);
        __syncwarp();
      }
      for (int i = 0; i < n_rows; i += R) {
        int64_t base = off_all[wid][i];
        for (int t0 = 0; t0 < gn; t0 += 32) {
          const int tj = gn <= 32 ? lane - rr * gn : t0 + lane;
          int32_t s = 0, len = 0;
          const int32_t* tc = nullptr;
          const VT* tv = nullptr;
          if (rr < R && i + rr < n_rows && tj < gn) {
            const int64_t row = r + row_all[wid][i + rr];
            const int64_t ti = row / g.tm;
            const int64_t lr = row - ti * g.tm;
            const bclx_csr_t t = g.tile(ti, tj);
            s = __ldg(t.row_ptr + lr);
            len = __ldg(t.row_ptr + lr + 1) - s;
            tc = t.col_ind + s;
            tv = reinterpret_cast<const VT*>(t.vals) + s;
          }
          const unsigned full = __ballot_sync(kFull, len > 0);
          const int32_t incl = warp_inclusive_scan(len);
          const int32_t total = __shfl_sync(kFull, incl, 31);
          const int32_t excl = incl - len;
          const int32_t lo = (int32_t)(P > base ? (P - base < total ? P - base : total) : 0);
          const int32_t hi = (int32_t)(end - base < total ? end - base : total);
          if (lo < hi) {
            if (len > 0) {
              const int at = __popc(full & below);
              seg[at] = make_ulonglong2(reinterpret_cast<unsigned long long>(tc) - 4ull * (unsigned)excl,
                                        reinterpret_cast<unsigned long long>(tv) - 4ull * (unsigned)excl);
              shift[at] = (int32_t)(tj * g.tn);
            }
            __syncwarp();
            int ahead = __popc(__ballot_sync(kFull, len > 0 && excl < lo)) - 1;  // runs begun before lo, less one
            for (int32_t b = lo; b < hi; b += 32) {
              const int32_t d = excl - b;
              const unsigned heads = __reduce_or_sync(kFull, len > 0 && (unsigned)d < 32u ? 1u << d : 0u);
              const int src = ahead + __popc(heads & upto);
              ahead += __popc(heads);
              const int32_t q = b + lane;
              if (q < hi) {
                const ulonglong2 from = seg[src];
                oci[base + q] = __ldg(reinterpret_cast<const int32_t*>(from.x + 4ull * (unsigned)q)) + shift[src];
                ova[base + q] = gathered(__ldg(reinterpret_cast<const VT*>(from.y + 4ull * (unsigned)q)));
              }
            }
            __syncwarp();
          }
          base += total;
          if (base >= end) break;
        }
      }
    }
  }
}

// A tile's descriptor from the packed arrays, one thread per tile.
__global__ void k_describe(bclx_spgrid_out_t g, bclx_csr_t* __restrict__ desc) {
  const int64_t nt = g.grid_m * g.grid_n;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ti = t / g.grid_n, tj = t - ti * g.grid_n;
    const int64_t lo = g.tile_offset[t];
    bclx_csr_t d;
    d.m = min(g.tile_m, g.m - ti * g.tile_m);
    d.n = min(g.tile_n, g.n - tj * g.tile_n);
    d.nnz = g.tile_offset[t + 1] - lo;
    d.row_ptr = g.tile_row_ptr + t * (g.tile_m + 1);
    d.col_ind = g.col_ind + lo;
    d.vals = reinterpret_cast<char*>(g.vals) + 4 * lo;
    d.dtype = g.dtype;
    d.pad_ = 0;
    desc[t] = d;
  }
}

static unsigned blocks_for(Context* ctx, int64_t work, int per_block) {
  int64_t b = ceil_div(work > 0 ? work : 1, per_block);
  const int64_t cap = (int64_t)ctx->num_sms * 16;
  return (unsigned)(b < cap ? b : cap);
}

}  // namespace bclx

using namespace bclx;

extern "C" {

int bclx_csr_to_tiles(bclx_context_t c, const bclx_csr_t* a, bclx_spgrid_out_t* out) {
  Context* ctx = reinterpret_cast<Context*>(c);
  if (!ctx || !a || !out) return BCLX_ERR_INVALID;
  if (a->dtype != BCLX_F32 && a->dtype != BCLX_I32) return BCLX_ERR_DTYPE;
  const int64_t m = a->m, n = a->n, tm = out->tile_m, tn = out->tile_n;
  if (m < 0 || n < 0 || tm <= 0 || tn <= 0 || out->m != m || out->n != n || out->grid_m != ceil_div(m, tm) ||
      out->grid_n != ceil_div(n, tn) || !out->tile_row_ptr || !out->tile_offset) {
    set_last_error("bclx_csr_to_tiles: output grid does not match the matrix and tile shape");
    return BCLX_ERR_INVALID;
  }
  if (n > INT32_MAX || (a->nnz > 0 && (!a->row_ptr || !a->col_ind || !a->vals || !out->col_ind || !out->vals))) {
    set_last_error("bclx_csr_to_tiles: missing arrays");
    return BCLX_ERR_INVALID;
  }
  BCLX_CK(cudaSetDevice(ctx->device));
  const int64_t gm = out->grid_m, gn = out->grid_n, ntiles = gm * gn;
  const int64_t tc = tn < INT32_MAX ? tn : INT32_MAX;  // (columns are below 2^31: 32-bit divisions by the tile width)
  const int64_t slots = ntiles * (tm + 1);
  if (slots == 0) return BCLX_OK;
  // one scratch block: E [slots + 1], the scan's block sums, cnt [slots], bad
  const int64_t sums_len = exclusive_scan_sums_len(slots);
  int64_t* E = nullptr;
  BCLX_TRY(scratch_alloc(ctx, reinterpret_cast<void**>(&E),
                         sizeof(int64_t) * (size_t)(slots + 1 + sums_len) + sizeof(int32_t) * (size_t)(slots + 1)));
  int64_t* sums = E + slots + 1;
  int32_t* cnt = reinterpret_cast<int32_t*>(sums + sums_len);
  int32_t* bad = cnt + slots;
  int32_t hbad = 0;
  const int rc = [&]() -> int {
    BCLX_CK(cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (size_t)(slots + 1), ctx->stream));
    const unsigned walkers = blocks_for(ctx, ceil_div(a->nnz + m, kChunk), 8);
    if (m > 0) {
      k_tile_count<<<walkers, 256, 0, ctx->stream>>>(m, n, a->row_ptr, a->col_ind, tm, tc, gn, cnt, bad);
      note_launch();
      BCLX_CK_LAUNCH();
    }
    BCLX_TRY(exclusive_scan_i32_buf(ctx, cnt, E, slots, sums));
    k_tile_ptrs<<<blocks_for(ctx, slots, 256), 256, 0, ctx->stream>>>(E, ntiles, tm, bad, out->tile_row_ptr,
                                                                      out->tile_offset);
    note_launch();
    BCLX_CK_LAUNCH();
    if (m == 0) return BCLX_OK;
    if (a->nnz > 0) {
      if (a->dtype == BCLX_F32)
        k_tile_scatter<float><<<walkers, 256, 0, ctx->stream>>>(m, n, a->row_ptr, a->col_ind,
                                                                reinterpret_cast<const float*>(a->vals), tm, tc, gn, E,
                                                                bad, out->col_ind, reinterpret_cast<float*>(out->vals));
      else
        k_tile_scatter<int32_t><<<walkers, 256, 0, ctx->stream>>>(
            m, n, a->row_ptr, a->col_ind, reinterpret_cast<const int32_t*>(a->vals), tm, tc, gn, E, bad, out->col_ind,
            reinterpret_cast<int32_t*>(out->vals));
      note_launch();
      BCLX_CK_LAUNCH();
    }
    BCLX_CK(cudaMemcpyAsync(&hbad, bad, sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
    BCLX_CK(cudaStreamSynchronize(ctx->stream));
    return BCLX_OK;
  }();
  scratch_free(ctx, E);
  if (rc == BCLX_OK && hbad) {
    set_last_error("bclx_csr_to_tiles: column indices must be ascending and within [0, n) in every row");
    return BCLX_ERR_INVALID;
  }
  return rc;
}

int bclx_spgrid_describe(bclx_context_t c, const bclx_spgrid_out_t* g, bclx_csr_t* desc) {
  Context* ctx = reinterpret_cast<Context*>(c);
  if (!ctx || !g || g->tile_m <= 0 || g->tile_n <= 0 || g->grid_m != ceil_div(g->m, g->tile_m) ||
      g->grid_n != ceil_div(g->n, g->tile_n))
    return BCLX_ERR_INVALID;
  if (g->dtype != BCLX_F32 && g->dtype != BCLX_I32) return BCLX_ERR_DTYPE;
  const int64_t nt = g->grid_m * g->grid_n;
  if (nt <= 0) return BCLX_OK;  // (no rows or no columns: arrays of no tiles, which may be null)
  if (!g->tile_row_ptr || !g->tile_offset || !desc) return BCLX_ERR_INVALID;
  BCLX_CK(cudaSetDevice(ctx->device));
  k_describe<<<blocks_for(ctx, nt, 256), 256, 0, ctx->stream>>>(*g, desc);
  note_launch();
  BCLX_CK_LAUNCH();
  return BCLX_OK;
}

int bclx_tiles_to_csr(bclx_context_t c, const bclx_spgrid_t* g, int32_t* row_ptr, int32_t* col_ind, void* vals) {
  Context* ctx = reinterpret_cast<Context*>(c);
  if (!ctx || !g || !row_ptr || !g->tiles) return BCLX_ERR_INVALID;
  if (g->dtype != BCLX_F32 && g->dtype != BCLX_I32) return BCLX_ERR_DTYPE;
  if (g->m < 0 || g->n < 0 || g->tile_m <= 0 || g->tile_n <= 0 || g->grid_m != ceil_div(g->m, g->tile_m) ||
      g->grid_n != ceil_div(g->n, g->tile_n)) {
    set_last_error("bclx_tiles_to_csr: inconsistent tile grid");
    return BCLX_ERR_INVALID;
  }
  BCLX_CK(cudaSetDevice(ctx->device));
  const SpGridView v = make_view(*g);
  const int64_t m = g->m;
  // one scratch block: off [m + 1], the scan's block sums, len [m]
  const int64_t sums_len = exclusive_scan_sums_len(m);
  int64_t* off = nullptr;
  BCLX_TRY(scratch_alloc(ctx, reinterpret_cast<void**>(&off),
                         sizeof(int64_t) * (size_t)(m + 1 + sums_len) + sizeof(int32_t) * (size_t)(m + 1)));
  int64_t* sums = off + m + 1;
  int32_t* len = reinterpret_cast<int32_t*>(sums + sums_len);
  int64_t nnz = 0;
  const int rc = [&]() -> int {
    if (m > 0) {
      k_gather_len<<<blocks_for(ctx, m, 256), 256, 0, ctx->stream>>>(v, len);
      note_launch();
      BCLX_CK_LAUNCH();
    }
    BCLX_TRY(exclusive_scan_i32_buf(ctx, len, off, m, sums));
    k_rowptr32<<<blocks_for(ctx, m + 1, 256), 256, 0, ctx->stream>>>(off, m, col_ind && vals ? (int64_t)INT32_MAX : 0, row_ptr);
    note_launch();
    BCLX_CK_LAUNCH();
    if (m > 0 && g->n > 0 && col_ind && vals) {
      // (the entries' number is on the device: a full grid strides over them)
      const unsigned blocks = (unsigned)(ctx->num_sms * 8);
      if (g->dtype == BCLX_F32)
        k_gather_rows<float><<<blocks, 256, 0, ctx->stream>>>(v, off, col_ind, reinterpret_cast<float*>(vals));
      else
        k_gather_rows<int32_t><<<blocks, 256, 0, ctx->stream>>>(v, off, col_ind, reinterpret_cast<int32_t*>(vals));
      note_launch();
      BCLX_CK_LAUNCH();
    }
    BCLX_CK(cudaMemcpyAsync(&nnz, off + m, sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream));
    BCLX_CK(cudaStreamSynchronize(ctx->stream));
    return BCLX_OK;
  }();
  scratch_free(ctx, off);
  if (rc != BCLX_OK) return rc;
  if (nnz > INT32_MAX) {
    set_last_error("bclx_tiles_to_csr: more than 2^31-1 entries do not fit an int32 row_ptr");
    return BCLX_ERR_INDEX_OVERFLOW;
  }
  return nnz > 0 && (!col_ind || !vals) ? BCLX_ERR_INVALID : BCLX_OK;
}

}  // extern "C"
