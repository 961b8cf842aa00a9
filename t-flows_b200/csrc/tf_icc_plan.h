// tf_icc_plan.h -- what a solve needs to launch the incomplete-Cholesky
// kernels of tf_icc.cuh.
#pragma once
#include <vector>

#include "tf_common.cuh"

namespace tf {

// Entries of a row kept in the packed slices; a longer row's remaining ones
// are read from the matrix itself.
constexpr int kIccWidth = 16;
constexpr int kIccChunk = 8;       // slices per bulk-copied chunk
constexpr int kIccProducers = 2;   // warps that issue the copies

enum IccDirection { kIccFwd = 0, kIccBwd = 1 };

// One direction of the sweeps.  The rows, in level order, are cut into slices
// of at most 32 rows of one level, one lane each; kIccChunk slices make a
// chunk.  Everything a sweep reads of a chunk is one record, copied to shared
// memory in one piece (a copy costs its issue: seven copies of a chunk's
// arrays took 0.68 us, 25 GB/s):
//   meta[kIccChunk]   two int4 per slice (IccSlice)
//   row[np]           three doubles: right-hand side, Prec_Form's d, and d_inv
//                     (forward) or r (backward)
//   out[np]           where the result goes: forward, the index of the row's
//                     right-hand side in the backward records (doubles);
//                     backward, the row
//   val[ne], col[ne]  entry k of lane t of a slice at its offset + k * rows +
//                     t, in the order the reference's loop visits it; column
//                     codes: >= 0 the result's slot in the shared-memory
//                     ring, < 0 row -1 - code, read from global memory.  A
//                     slice's width is a multiple of `batch`: shorter rows
//                     end in entries of value +0 that read a slot holding
//                     +0, which leave every sum as it is (x - (+0) is x, of
//                     either sign and for NaN)
// np and ne are multiples of 4.
struct IccDir {
  const int* ord;        // level order -> row
  const int4* slice;     // per slice, as built: first position, rows | width << 8,
                         // offset of its entries in src, level
  const int2* chunk;     // per chunk: offset of its record (16-byte units), bytes
  const int* src;        // packed entry -> entry of the matrix
  unsigned char* rec;    // the records
  const int* idx;        // row -> index of its right-hand side in rec (doubles)
  int nslices;
  int far_any;           // results are read from global memory too
};
constexpr int kIccMetaBytes = kIccChunk * 32;

// What a sweep reads of a slice before its rows: byte offsets in the record.
struct __align__(16) IccSlice {
  int pos;     // position of the first row
  int rows;
  int val, col;
  int row, out;
  int first;   // first slice of its level
  int width;   // | kIccFar: an entry is read from global memory; | kIccLong:
               // a row may have entries beyond the packed ones
};
constexpr int kIccFar = 1 << 8, kIccLong = 1 << 9;

struct IccArgs {
  const int* row;        // 0-based CSR
  const int* col;
  const double* val;     // scaled matrix
  const double* adiag;   // its diagonal
  int ni;
  double* d;             // by row, where far_any asks for them: Prec_Form's d
  double* y;             // ... and the forward sweep's values
  double* z;             // by row: the result
  SolveState* st;
  const SolveParams* prm;
  IccDir f, b;           // forward and backward
  int width, stages, ring;
};

// One level's rows (one kernel per level).
struct IccLevelArgs {
  const int* row;      // 0-based CSR
  const int* col;
  const double* val;   // scaled matrix
  const int* rows;     // rows of this level
  int count;           // rows in this level
  int ni;
  double* d;           // Prec_Form's d (1/pivot)
  double* d_inv;       // Prec_Form's d_inv (pivot)
  const double* r;     // right-hand side of the solve (r1)
  double* y;           // forward-sweep values
  double* z;           // result
  const SolveState* st;
};

}  // namespace tf

// A launch of the preconditioner: kernel, grid, block, shared memory and
// the arguments (owned by the plan).
struct tf_icc_launch {
  const void* fn = nullptr;
  int grid = 1, threads = 256;
  size_t smem = 0;
  std::vector<void*> args;
};

// The launches that form the preconditioner on the scaled matrix and those
// that apply it (z = M^-1 r, rho = z.r), in order.  Keeps its own arguments:
// not to be copied.
struct tf_icc_plan {
  tf::IccArgs one{};
  std::vector<tf::IccLevelArgs> level;
  struct {
    int ni;
    const double* z;
    const double* r;
    double* part;
    tf::SolveState* st;
  } rho{};
  std::vector<tf_icc_launch> form, apply;
  tf_icc_plan() = default;
  tf_icc_plan(const tf_icc_plan&) = delete;
  tf_icc_plan& operator=(const tf_icc_plan&) = delete;
};
struct tf_matrix_s;
int tf_icc_make_plan(tf_matrix_s* m, tf_icc_plan* p);
