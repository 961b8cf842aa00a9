// tf_icc.cuh -- incomplete-Cholesky preconditioning by level scheduling.
//
// Prec_Form.f90:68-78 and Prec_Solve.f90:64-92 are sequential recurrences
// over rows.  Row i depends only on its lower neighbours k < i (forward
// sweep, and the d(k) of Prec_Form) or on its upper neighbours k > i
// (backward sweep).  Rows are grouped into levels such that every
// dependency of a row lies in an earlier level; the rows of a level are
// then computed in parallel, each with exactly the reference's arithmetic in
// exactly its order, so d, d_inv and z are the reference's bits given the
// same inputs.  Requires the diagonal-first, ascending-column layout
// Create_Matrix produces (the reference's ICC relies on it too,
// Prec_Form.f90:55-66).
//
// Two forms of the same recurrences:
//   * one CTA walks all levels of both sweeps (k_icc_apply), streaming the
//     matrix in level order through shared memory -- the path of matrices
//     whose levels are narrow, where the chain of levels is the bound and a
//     kernel per level would be launch latency and nothing else;
//   * one kernel per level (k_icc_fwd_level, k_icc_bwd_level) where levels
//     are so wide that one SM's bandwidth would be the bound (tf_icc.cu has
//     the rule).
#pragma once
#include "../../include/tf_krylov.h"
#include "tf_common.cuh"
#include "tf_icc_plan.h"

namespace tf {

// ---------------------------------------------------------------------------
// One kernel per level
// ---------------------------------------------------------------------------
// Prec_Form.f90:69-78 for the rows of one level.
static __global__ void __launch_bounds__(256) k_icc_form_level(IccLevelArgs a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.count) return;
  const int i = a.rows[t];
  const int js = a.row[i], je = a.row[i + 1];
  double sum = a.val[js];                       // diagonal entry (first)
  for (int j = js + 1; j < je; ++j) {
    const int k = a.col[j];
    if (k > i) break;
    const double v = a.val[j];
    sum = __dsub_rn(sum, __dmul_rn(__dmul_rn(a.d[k], v), v));
  }
  a.d_inv[i] = sum;
  a.d[i] = __ddiv_rn(1.0, sum);
}

// Forward substitution (Prec_Solve.f90:67-75) for one level; also applies
// the diagonal scaling of :77-81 into z, keeping the unscaled y for the
// rows of later levels.
static __global__ void __launch_bounds__(256) k_icc_fwd_level(IccLevelArgs a) {
  if (a.st && a.st->done) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.count) return;
  const int i = a.rows[t];
  const int js = a.row[i], je = a.row[i + 1];
  double sum = a.r[i];
  for (int j = js + 1; j < je; ++j) {
    const int k = a.col[j];
    if (k > i) break;
    sum = __dsub_rn(sum, __dmul_rn(a.val[j], a.y[k]));
  }
  const double yi = __dmul_rn(sum, a.d[i]);
  a.y[i] = yi;
  a.z[i] = __dmul_rn(yi, a.d_inv[i]);
}

// Backward substitution (Prec_Solve.f90:84-92) for one level.
static __global__ void __launch_bounds__(256) k_icc_bwd_level(IccLevelArgs a) {
  if (a.st && a.st->done) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.count) return;
  const int i = a.rows[t];
  const int js = a.row[i], je = a.row[i + 1];
  double sum = a.z[i];
  for (int j = je - 1; j >= js + 1; --j) {
    const int k = a.col[j];
    if (k < i) break;
    if (k < a.ni) sum = __dsub_rn(sum, __dmul_rn(a.val[j], a.z[k]));
  }
  a.z[i] = __dmul_rn(sum, a.d[i]);
}

// rho = z.r (Cg.f90:150-156) after an ICC solve.  At iteration 1 it is the
// first rho; later it shifts rho into rho_old first (Cg.f90:222).
static __global__ void __launch_bounds__(256) k_icc_rho(int ni, const double* z, const double* r,
                                                 double* part, SolveState* st) {
  __shared__ double scratch[32];
  if (st->done) return;
  double s = 0.0;
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ni; i += stride)
    s = __dadd_rn(s, __dmul_rn(z[i], r[i]));
  double v[1] = {block_red<kSum>(s, scratch)};
  const int ops[1] = {kSum};
  if (grid_reduce_last<1>(v, ops, part, &st->counter[kCntZ], scratch) && threadIdx.x == 0) {
    if (st->iter > 1) st->rho_old = st->rho;
    st->rho = v[0];
  }
}

// ---------------------------------------------------------------------------
// Packing, once per matrix
// ---------------------------------------------------------------------------
// Calls f(j) for the entries of row i the sweep visits, in its order, from
// the `skip`-th visited one on, until f returns false.
template <int DIR, class F>
__device__ __forceinline__ void icc_visit(const int* row, const int* col, int ni, int i, int skip,
                                          F&& f) {
  const int js = row[i], je = row[i + 1];
  int seen = 0;
  if (DIR == kIccFwd) {                    // Prec_Solve.f90:69-74
    for (int j = js + 1; j < je; ++j) {
      if (col[j] > i) break;
      if (seen++ >= skip && !f(j)) break;
    }
  } else {                                 // Prec_Solve.f90:85-91
    for (int j = je - 1; j >= js + 1; --j) {
      const int k = col[j];
      if (k < i) break;
      if (k >= ni) continue;               // buffer cells
      if (seen++ >= skip && !f(j)) break;
    }
  }
}

// Width of every slice (one warp each) and the widest of all.
template <int DIR>
static __global__ void __launch_bounds__(256) k_icc_widths(const int* row, const int* col, int ni,
                                                           const int* ord, int4* meta,
                                                           int nslices, int* widest) {
  const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (s >= nslices) return;
  const int4 m = meta[s];
  int len = 0;
  if (lane < m.y)
    icc_visit<DIR>(row, col, ni, ord[m.x + lane], 0, [&](int) { return ++len < kIccWidth; });
  len = __reduce_max_sync(0xffffffffu, len);
  if (lane == 0) {
    meta[s].y = m.y | len << 8;
    atomicMax(widest, len);
  }
}

// Packed entries of a slice and rows of a chunk, rounded up so that every part
// of a record starts on a 16-byte boundary.
__host__ __device__ __forceinline__ int icc_slice_entries(int rows, int width) {
  return (rows * width + 3) & ~3;
}
__host__ __device__ __forceinline__ int icc_chunk_rows(int rows) { return (rows + 3) & ~3; }
__host__ __device__ __forceinline__ int icc_record_bytes(int np, int ne) {
  return kIccMetaBytes + np * 28 + ne * 12;
}

// Per chunk: its slices' widths rounded up to the batch, size of its record.
static __global__ void __launch_bounds__(256) k_icc_chunks(int4* slice, int nslices, int batch,
                                                           int2* chunk) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, s0 = c * kIccChunk;
  if (s0 >= nslices) return;
  int ne = 0, rows = 0;
  for (int s = s0; s < min(s0 + kIccChunk, nslices); ++s) {
    const int w = slice[s].y >> 8, y = (slice[s].y & 255) | (w + batch - 1) / batch * batch << 8;
    slice[s].y = y;
    ne += icc_slice_entries(y & 255, y >> 8);
    rows += y & 255;
  }
  chunk[c] = make_int2(0, icc_record_bytes(icc_chunk_rows(rows), ne));
}

// Exclusive sum of get(i) over i < n, handed to put(i, sum); returns the
// total.  One CTA of 1024 threads.
template <class GET, class PUT>
__device__ long long icc_scan(int n, GET get, PUT put) {
  __shared__ int warp_sum_sh[32];
  __shared__ long long base_sh;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (threadIdx.x == 0) base_sh = 0;
  __syncthreads();
  for (int s0 = 0; s0 < n; s0 += 1024) {
    const int s = s0 + (int)threadIdx.x;
    const int mine = s < n ? get(s) : 0;
    int inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) warp_sum_sh[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      int w = warp_sum_sh[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
      }
      warp_sum_sh[lane] = w;
    }
    __syncthreads();
    const long long base = base_sh + (warp ? warp_sum_sh[warp - 1] : 0);
    if (s < n) put(s, base + inc - mine);
    __syncthreads();
    if (threadIdx.x == 1023) base_sh = base + inc;
    __syncthreads();
  }
  return base_sh;
}

// Offsets of the slices' entries in src and of the chunks' records (16-byte
// units); total[0] = entries, total[1] = record bytes / 16.
static __global__ void __launch_bounds__(1024) k_icc_offsets(int4* slice, int nslices,
                                                             int2* chunk, int nchunks,
                                                             long long* total) {
  const long long e = icc_scan(
      nslices, [&](int s) { return icc_slice_entries(slice[s].y & 255, slice[s].y >> 8); },
      [&](int s, long long at) { slice[s].z = (int)at; });
  const long long b = icc_scan(nchunks, [&](int c) { return chunk[c].y / 16; },
                               [&](int c, long long at) { chunk[c].x = (int)at; });
  if (threadIdx.x == 0) {
    total[0] = e;
    total[1] = b;
  }
}

// Rows' places: pos[row] = position in level order, idx[row] = index (in
// doubles) of its right-hand side in the records.
static __global__ void __launch_bounds__(256) k_icc_places(const int* ord, const int4* slice,
                                                           const int2* chunk, int nslices,
                                                           int* pos, int* idx) {
  const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (s >= nslices) return;
  const int4 m = slice[s];
  if (lane >= (m.y & 255)) return;
  const int p = m.x + lane, i = ord[p], c = s / kIccChunk;
  pos[i] = p;
  idx[i] = 2 * chunk[c].x + kIccMetaBytes / 8 + 3 * (p - slice[c * kIccChunk].x);
}

// The records' constant parts, one warp per slice, and whether any entry lies
// outside the ring.  An entry whose row was computed at most `ring` positions
// before the end of the reader's level is read from the ring (slot = position
// & (ring - 1): no position of the reader's level or before it has
// overwritten the slot); an older one from global memory.
template <int DIR>
static __global__ void __launch_bounds__(256) k_icc_fill(
    const int* row, const int* col, int ni, const int* ord, const int* pos, const int* lev_ptr,
    const int* lev_slice, const int4* slice, const int2* chunk, int nslices, int ring,
    const int* other_idx, int* src, unsigned char* rec_all, int* far_any) {
  const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (s >= nslices) return;
  const int c = s / kIccChunk, s0 = c * kIccChunk, s1 = min(s0 + kIccChunk, nslices) - 1;
  const int4 m = slice[s], first = slice[s0], last = slice[s1];
  const int rows = m.y & 255, width = m.y >> 8;
  const int np = icc_chunk_rows(last.x + (last.y & 255) - first.x);
  const int ne = last.z + icc_slice_entries(last.y & 255, last.y >> 8) - first.z;
  const int r0 = m.x - first.x, e0 = m.z - first.z;
  unsigned char* rec = rec_all + (size_t)chunk[c].x * 16;
  const int out_at = kIccMetaBytes + np * 24, val_at = out_at + np * 4;
  bool far = false, longer = false;
  if (lane < rows) {
    int* out = reinterpret_cast<int*>(rec + out_at);
    int* pcol = reinterpret_cast<int*>(rec + val_at + (size_t)ne * 8);
    const int end = lev_ptr[m.w + 1], i = ord[m.x + lane];
    out[r0 + lane] = DIR == kIccFwd ? other_idx[i] : i;
    int at = lane, left = width;
    icc_visit<DIR>(row, col, ni, i, 0, [&](int j) {
      if (left == 0) {
        longer = true;
        return false;
      }
      const int k = col[j], pk = pos[k];
      const bool near = end - pk <= ring;
      far = far || !near;
      src[m.z + at] = j;
      pcol[e0 + at] = near ? (pk & (ring - 1)) : -1 - k;
      at += rows;
      --left;
      return true;
    });
    for (; left > 0; --left, at += rows) {
      src[m.z + at] = -1;
      pcol[e0 + at] = ring;   // the slot that holds +0
    }
  }
  far = __any_sync(0xffffffffu, far);
  longer = __any_sync(0xffffffffu, longer);
  if (lane == 0) {
    IccSlice t;
    t.pos = m.x;
    t.rows = rows;
    t.val = val_at + e0 * 8;
    t.col = val_at + ne * 8 + e0 * 4;
    t.row = kIccMetaBytes + r0 * 24;
    t.out = out_at + r0 * 4;
    t.first = lev_slice[m.w];
    t.width = width | (far ? kIccFar : 0) | (longer ? kIccLong : 0);
    reinterpret_cast<IccSlice*>(rec)[s - s0] = t;
    if (far || longer) *far_any = 1;
  }
}

// Values of the scaled matrix into both directions' records, and its diagonal
// into the forward right-hand side (where k_icc_form reads it), once per
// solve.
static __global__ void __launch_bounds__(256) k_icc_pack(IccArgs a) {
  const int warps = (gridDim.x * blockDim.x) >> 5, lane = threadIdx.x & 31;
  const int w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  for (int w = w0; w < a.f.nslices + a.b.nslices; w += warps) {
    const IccDir& g = w < a.f.nslices ? a.f : a.b;
    const int s = w < a.f.nslices ? w : w - a.f.nslices, c = s / kIccChunk;
    const int4 m = g.slice[s];
    unsigned char* rec = g.rec + (size_t)g.chunk[c].x * 16;
    const IccSlice t = reinterpret_cast<const IccSlice*>(rec)[s - c * kIccChunk];
    double* val = reinterpret_cast<double*>(rec + t.val);
    if (lane < t.rows)
      for (int k = 0; k < (t.width & 255); ++k) {
        const int j = g.src[m.z + k * t.rows + lane];
        val[k * t.rows + lane] = j >= 0 ? a.val[j] : 0.0;
      }
  }
  double* rec = reinterpret_cast<double*>(a.f.rec);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.ni; i += gridDim.x * blockDim.x)
    rec[a.f.idx[i]] = a.adiag[i];
}

// Shared memory of the sweeping CTA at most.
constexpr int kIccSmemBytes = 225 * 1024;
// Up to how many rows and entries a level, on average, one CTA walks the levels.
// One CTA pays 0.3 to 1.3 us for 1,000 entries (the more neighbours lie far
// back, the more), a kernel per level 5 to 14 us a level whatever it holds.  One
// Cg iteration, us, a kernel per level / one CTA, at rows and entries a level:
//   hex 57x43x53    860  2,500   1259 /  361   polyhedral 100 k  232  1,560   6239 /   884
//   hex 64^3      1,380  4,070   1826 /  713   400 k             578  3,950  15275 /  6567
//   hex 76^3      1,942  5,750   2481 / 1796   1.0 M           1,067  7,340  25489 / 17707
//   hex 92^3      2,842  8,430   4089 / 3907   1.4 M           1,319  9,090  29612 / 23660
//   hex 100^3     3,356  9,970   4664 / 5689   2.0 M           1,674 11,560  33927 / 34502
// The lines lie below both kinds' crossing (hex 2,900 rows, polyhedral 11,300
// entries); short rows of other numberings were measured up to 2,000 a level.
constexpr long long kIccOneRows = 2000, kIccOneEntries = 11000;
// ... and where more than an eighth of the levels hold a row with more entries
// than are packed (kIccWidth): such a row is summed from global memory, about as
// long as a kernel per level takes for its level, so everything else of the level
// comes on top.  Levels of rows of 7 entries, one in a hundred of 22: 300 rows
// (2,110 entries) 858 / 480, 800 (5,630) 880 / 967, 1,600 (11,250) 903 / 1724;
// Delaunay duals (0.3 % of the rows) of 150,000 cells, 1,770 entries, 12673 / 5200.
constexpr long long kIccOneLongEntries = 4000;

// ---------------------------------------------------------------------------
// All levels in one CTA
// ---------------------------------------------------------------------------
// A level costs a chain of dependent steps: see that the level before it is
// complete, gather its results from shared memory, the row's FP64 sum, store
// the result, report.  Everything else -- entries, right-hand side, d --
// streams ahead of that chain: a producer lane copies chunks of kIccChunk
// slices (1D bulk copies) into a ring of stages, and each consumer warp loads
// its next slice into registers after it has reported the current one.
// Consumer warp w of W takes slices w, w + W, ...; `progress` counts finished
// slices, and a slice starts when all slices of earlier levels are finished
// (progress >= first slice of its level: slices of its own level or later
// ones cannot have been counted before).
//
// Measured (57x43x53 hex, 302 levels of 27 slices): 329 us for both sweeps, 160
// instructions a slice, the SM's issue slots 52 % and its shared-memory pipe
// 64 % busy; a level alone takes about 0.5 us (poll, gather, sum,
// store, report).  Copying a chunk's arrays one by one, with divisions in the
// producer's loop, made it 740 us: a bulk copy costs its issuing lane some
// 150 cycles whatever its size.
//
// No deadlock: slices are numbered in level order, so the unfinished slice
// with the smallest number never waits for another slice's result; its warp
// waits at most for its chunk, whose stage is free once the chunk `stages`
// earlier is finished, all slices of which have smaller numbers.
enum IccKind { kIccForm = 0, kIccForward = 1, kIccBackward = 2 };

// Shared-memory layout for the widest slice `width`, `stages` stages, `ring`
// slots.
struct IccLayout {
  int stage, ring_at, bar_at, total;   // a stage's size; byte offsets
  __host__ __device__ IccLayout(int width, int stages, int ring) {
    stage = (icc_record_bytes(32 * kIccChunk, 32 * kIccChunk * width) + 127) & ~127;
    ring_at = stages * stage;
    bar_at = ring_at + ring * 8 + 16;   // and the slot that holds +0
    total = bar_at + stages * 16 + 16;   // full, empty; progress, abort
  }
};

// Finished slices: counted up with release, read with acquire semantics (the
// results in the ring are stored before and gathered after).
__device__ __forceinline__ void icc_report(int* progress) {
  asm volatile("red.release.cta.shared::cta.add.u32 [%0], 1;" ::"r"(smem_u32(progress))
               : "memory");
}
__device__ __forceinline__ int icc_progress(const int* progress) {
  int v;
  asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];"
               : "=r"(v)
               : "r"(smem_u32(progress))
               : "memory");
  return v;
}

// A sweep's blocked waits: each may last `limit` ns (from its first look, to
// within a few us), so a sweep of many levels takes as long as it takes.  The
// limit counts within a wait, and nothing of it is held between waits (counting
// from the last finished slice cost 1 to 4 % of an iteration, reading the timer
// at every wait 3 %).
struct IccPatience {
  unsigned long long limit, until;
  long long look;                    // SM clock at which to read the timer again
  __device__ __forceinline__ explicit IccPatience(unsigned long long limit_ns)
      : limit(limit_ns), until(0), look(0) {}
  __device__ __forceinline__ bool over(bool first) {
    const long long c = clock64();
    if (!first && c < look) return false;
    look = c + Deadline::kLookCycles;
    if (first) until = deadline_after(limit);
    return globaltimer_ns() > until;
  }
};
// False at the limit, or once *abort_flag is set.
__device__ __forceinline__ bool icc_wait(uint64_t* bar, unsigned parity, volatile int* abort_flag,
                                         unsigned long long limit) {
  IccPatience patience(limit);
  for (bool first = true; !mbar_try_wait(bar, parity); first = false)
    if (*abort_flag || patience.over(first)) return false;
  return true;
}

// One sweep.  `it0` chunks have gone through the stages before it (returned
// count: after it).  K entries of a row, in batches of B, are loaded ahead,
// the rest of its packed width is read from the stage, and what is longer
// from the matrix.  rho accumulates z_i r_i (kIccBackward).
template <int KIND, int K, int B, int W>
__device__ __forceinline__ int icc_sweep(const IccArgs& a, unsigned char* smem,
                                         const IccLayout& L, int it0, bool& ok,
                                         unsigned long long limit, double& rho) {
  static_assert(W % kIccChunk == 0, "a warp's slices lie whole chunks apart");
  const IccDir& g = KIND == kIccBackward ? a.b : a.f;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int stages = a.stages, ring_mask = a.ring - 1;
  double* ring = reinterpret_cast<double*>(smem + L.ring_at);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.bar_at);
  uint64_t* empty = full + stages;
  int* progress = reinterpret_cast<int*>(empty + stages);
  volatile int* abort_flag = progress + 1;
  const int nchunks = (g.nslices + kIccChunk - 1) / kIccChunk;
  auto stage_of = [&](int s) { return smem + (size_t)s * L.stage; };

  if (warp >= W) {
    // ---- producers: two lanes take the chunks in turn (a lone one is bound
    // by its own instructions, about 300 cycles a chunk) when the stages are
    // even, else the first takes all ----
    const int step = (stages & 1) ? 1 : kIccProducers;
    if (lane == 0 && warp - W < step) {
      const int m0 = warp - W;
      int stage = (it0 + m0) % stages, armed = 0;
      unsigned par = (unsigned)((it0 + m0) / stages + 1) & 1u;   // of the phase to wait for
      int2 c = m0 < nchunks ? __ldg(g.chunk + m0) : make_int2(0, 0);
      int2 nxt = m0 + step < nchunks ? __ldg(g.chunk + m0 + step) : c;
      for (int m = m0; m < nchunks; m += step) {
        const int2 nxt2 = m + 2 * step < nchunks ? __ldg(g.chunk + m + 2 * step) : c;
        if (it0 + m >= stages) {
          if (!icc_wait(&empty[stage], par, abort_flag, limit)) {
            ok = false;
            *abort_flag = 1;
            break;
          }
          fence_proxy_async_smem();
        }
        mbar_arrive_expect_tx(&full[stage], (unsigned)c.y);
        bulk_g2s(stage_of(stage), g.rec + (size_t)c.x * 16, (unsigned)c.y, &full[stage]);
        if (m == nchunks - 1)   // slices there are none of
          for (int q = g.nslices - m * kIccChunk; q < kIccChunk; ++q) mbar_arrive(&empty[stage]);
        armed = m + 1;
        stage += step;
        if (stage >= stages) {
          stage -= stages;
          par ^= 1u;
        }
        c = nxt;
        nxt = nxt2;
      }
      // Every copy this lane armed has landed before the sweep ends.
      for (int m = armed - 1; m >= m0 && m >= armed - stages; m -= step)
        mbar_drain(&full[(it0 + m) % stages], (unsigned)((it0 + m) / stages) & 1u);
    }
  } else {
    // ---- consumers ----
    // What a slice costs is its instructions (an SM issues four a cycle to
    // all its warps), hence byte offsets ready in the record and rows padded
    // to whole batches instead of tests per entry.
    const double* far = KIND == kIccForm ? a.d : KIND == kIccForward ? a.y : a.z;
    double* rec_b = reinterpret_cast<double*>(a.b.rec);
    auto accumulate = [&](double sum, double v, double yk) {
      if (KIND == kIccForm) return __dsub_rn(sum, __dmul_rn(__dmul_rn(yk, v), v));
      return __dsub_rn(sum, __dmul_rn(v, yk));
    };
    // The next slice's stage and its parity.  W / kIccChunk chunks lie between
    // a warp's slices and the stages are a multiple of that, so the warp has
    // seen the chunk before in the same stage land: the parity is never two
    // phases off.
    const int ld = it0 + warp / kIccChunk;
    int stage = ld % stages;
    unsigned par = (unsigned)(ld / stages) & 1u;
    for (int s = warp; s < g.nslices; s += W) {
      // What does not depend on other rows.
      bool here = mbar_try_wait(&full[stage], par) ||
                  icc_wait(&full[stage], par, abort_flag, limit);
      if (!__all_sync(0xffffffffu, here)) {
        ok = false;
        *abort_flag = 1;
        break;
      }
      const unsigned char* st = stage_of(stage);
      const IccSlice m = reinterpret_cast<const IccSlice*>(st)[s % kIccChunk];
      const int width = m.width & 255;
      const bool mine = lane < m.rows;
      const double* sv = reinterpret_cast<const double*>(st + m.val) + lane;
      const int* sc = reinterpret_cast<const int*>(st + m.col) + lane;
      int c[K], out = 0;
      double v[K], rhs = 0.0, dd = 0.0, di = 0.0;
      if (mine) {
        const double* srow = reinterpret_cast<const double*>(st + m.row) + 3 * lane;
        rhs = srow[0];
        dd = srow[1];
        di = srow[2];
        out = reinterpret_cast<const int*>(st + m.out)[lane];
#pragma unroll
        for (int b = 0; b < K; b += B)
          if (b < width) {
#pragma unroll
            for (int k = b; k < b + B; ++k) {
              c[k] = sc[k * m.rows];
              v[k] = sv[k * m.rows];
            }
          }
      }
      // The earlier levels.
      IccPatience patience(limit);
      for (int spin = 0; icc_progress(progress) < m.first; ++spin)
        if ((spin & 63) == 63 && (*abort_flag || patience.over(spin == 63))) {
          here = false;
          break;
        }
      if (!__all_sync(0xffffffffu, here)) {
        ok = false;
        *abort_flag = 1;
        break;
      }
      const int pos = m.pos + lane;
      double sum = rhs, res = 0.0;
      if (mine) {
        if (!(m.width & (kIccFar | kIccLong))) {
#pragma unroll
          for (int b = 0; b < K; b += B)
            if (b < width) {
              double yk[B];
#pragma unroll
              for (int k = 0; k < B; ++k) yk[k] = ring[c[b + k]];
#pragma unroll
              for (int k = 0; k < B; ++k) sum = accumulate(sum, v[b + k], yk[k]);
            }
          for (int k = K; k < width; ++k)
            sum = accumulate(sum, sv[k * m.rows], ring[sc[k * m.rows]]);
        } else {
          for (int k = 0; k < width; ++k) {
            const int ck = sc[k * m.rows];
            sum = accumulate(sum, sv[k * m.rows], ck >= 0 ? ring[ck] : far[-1 - ck]);
          }
          if (m.width & kIccLong)
            icc_visit < KIND == kIccBackward
                ? kIccBwd
                : kIccFwd > (a.row, a.col, a.ni, g.ord[pos], width, [&](int j) {
                    sum = accumulate(sum, a.val[j], far[a.col[j]]);
                    return true;
                  });
        }
        // Prec_Form.f90:77, Prec_Solve.f90:75 and :91
        res = KIND == kIccForm ? __ddiv_rn(1.0, sum) : __dmul_rn(sum, dd);
        ring[pos & ring_mask] = res;
        if (g.far_any) {   // before the report: a later level may read it there
          if (KIND == kIccForm) a.d[g.ord[pos]] = res;
          if (KIND == kIccForward) a.y[g.ord[pos]] = res;
          if (KIND == kIccBackward) a.z[out] = res;
        }
      }
      __syncwarp();
      if (lane == 0) icc_report(progress);
      if (mine) {
        if (KIND == kIccForm) {
          double* rec_f = reinterpret_cast<double*>(a.f.rec) + a.f.idx[g.ord[pos]];
          rec_f[1] = res;
          rec_f[2] = sum;
          rec_b[out + 1] = res;
        } else if (KIND == kIccForward) {
          rec_b[out] = __dmul_rn(res, di);   // Prec_Solve.f90:77-81
        } else {
          if (!g.far_any) a.z[out] = res;
          rho = __dadd_rn(rho, __dmul_rn(res, di));   // di: r in the backward order
        }
      }
      if (lane == 0) mbar_arrive(&empty[stage]);
      stage += W / kIccChunk;
      if (stage >= stages) {
        stage -= stages;
        par ^= 1u;
      }
    }
  }
  return it0 + nchunks;
}

__device__ __forceinline__ void icc_init(const IccArgs& a, unsigned char* smem,
                                         const IccLayout& L) {
  if (threadIdx.x == 0) {
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.bar_at);
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&full[a.stages + s], kIccChunk);
    }
    int* progress = reinterpret_cast<int*>(full + 2 * a.stages);
    progress[0] = progress[1] = 0;
    reinterpret_cast<double*>(smem + L.ring_at)[a.ring] = 0.0;
    mbar_fence_init();
  }
  __syncthreads();
}

// Prec_Form on the scaled matrix.  One CTA.
template <int K, int B, int W>
static __global__ void __launch_bounds__(32 * (W + kIccProducers), 1) k_icc_form(IccArgs a) {
  extern __shared__ __align__(128) unsigned char tf_icc_smem[];
  const IccLayout L(a.width, a.stages, a.ring);
  icc_init(a, tf_icc_smem, L);
  bool ok = true;
  double none = 0.0;
  const unsigned long long limit = wait_limit(a.prm);
  icc_sweep<kIccForm, K, B, W>(a, tf_icc_smem, L, 0, ok, limit, none);
  if (!ok) atomicExch(&a.st->status, (int)TF_ERR_TIMEOUT);
}

// z = M^-1 r (both sweeps) and rho = z.r (Cg.f90:150-156); at iteration 1 it
// is the first rho, later it shifts rho into rho_old first (Cg.f90:222).
// One CTA.
template <int K, int B, int W>
static __global__ void __launch_bounds__(32 * (W + kIccProducers), 1) k_icc_apply(IccArgs a) {
  extern __shared__ __align__(128) unsigned char tf_icc_smem[];
  __shared__ double scratch[32];
  SolveState* st = a.st;
  if (st->done) return;
  const IccLayout L(a.width, a.stages, a.ring);
  icc_init(a, tf_icc_smem, L);
  const unsigned long long limit = wait_limit(a.prm);
  bool ok = true;
  double rho = 0.0;
  int it = icc_sweep<kIccForward, K, B, W>(a, tf_icc_smem, L, 0, ok, limit, rho);
  // the backward sweep's bulk copies read what these threads have stored
  asm volatile("fence.proxy.async;" ::: "memory");
  ok = !__syncthreads_or(!ok);
  if (threadIdx.x == 0)
    *reinterpret_cast<int*>(tf_icc_smem + L.bar_at + 16 * a.stages) = 0;   // progress
  __syncthreads();
  if (ok) icc_sweep<kIccBackward, K, B, W>(a, tf_icc_smem, L, it, ok, limit, rho);
  if (!ok) atomicExch(&st->status, (int)TF_ERR_TIMEOUT);
  rho = block_red<kSum>(rho, scratch);
  if (threadIdx.x == 0) {
    if (st->iter > 1) st->rho_old = st->rho;
    st->rho = rho;
  }
}

}  // namespace tf
