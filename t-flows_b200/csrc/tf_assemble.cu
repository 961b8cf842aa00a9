// tf_assemble.cu -- the pressure and momentum matrices assembled on the
// device from face data, through Matrix_Type's pos(1:2, face) map.
//
// Process assembles A % val on the host every outer iteration
// (Compute_Pressure.f90, Rhie_And_Chow.f90:183-205, Compute_Momentum.f90:
// 270-297) and the drop-in then uploads it; with the face data already on
// the device the upload disappears.  Results are bit-identical to the
// reference's face loops:
//
//   * off-diagonals: the reference's assignment (pressure: -a12) or
//     accumulation from the zeroed matrix (momentum: 0 - m12);
//   * diagonals: one thread per cell adds its faces' contributions in
//     ascending face order -- the order in which the reference's sequential
//     face loop reaches that cell -- starting from 0.0, then the terms of
//     the later loops (pressure boundary faces; the inertial term).
//
// Every product and sum is issued as the reference writes it, rounded
// (__dmul_rn, __dadd_rn, ...), with no FMA contraction.
#include <cuda_runtime.h>
#include <limits.h>

#include <algorithm>
#include <memory>
#include <vector>

#include "tf_internal.h"

namespace tf {

__device__ __forceinline__ double fmin_ref(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double fmax_ref(double a, double b) { return (b > a) ? b : a; }

// a12 of Rhie_And_Chow.f90: fc * (fs * v_m(c1) + (1 - fs) * v_m(c2))
__device__ __forceinline__ double p_coef(const double* fc, const double* fw, const double* vm,
                                         int s, int c1, int c2) {
  const double fs = fw[s];
  const double v1 = vm ? vm[c1] : 1.0, v2 = vm ? vm[c2] : 1.0;
  const double t = __dadd_rn(__dmul_rn(fs, v1), __dmul_rn(__dsub_rn(1.0, fs), v2));
  return __dmul_rn(fc[s], t);
}

// ---------------------------------------------------------------------------
// Rows assembled cell by cell.  A CTA takes kAsmCells consecutive cells, whose
// entries are contiguous: it zeroes them in shared memory, every thread walks
// its cell's faces in ascending order -- both cells of a face form its
// coefficient, with the same bits -- storing its own row's entry and adding to
// its diagonal, and the tile goes out in whole lines.  One pass instead of a
// zeroing pass, a face pass that scatters two entries a face and a cell pass
// that reads the faces again.  The faces of 32 consecutive cells are listed
// lane by lane (AsmLists), so the lists are read coalesced.  Bound by the
// loads of a tile's dependent lists and face data: 1.01 M hex cells 95 -> 53 us
// a matrix (2.4 TB/s of what it cannot do without; 64 us with one visit's loads
// at a time, 61 with 12-byte lists).
// ---------------------------------------------------------------------------
constexpr int kAsmCells = 128;
constexpr int kAsmBatch = 6;        // a hex cell's faces
constexpr int kAsmEntries = 4096;   // largest tile kept in shared memory
constexpr int kAsmPlaces = 1 << 20; // places of the lists that are always granted

// Visit v of lane t of the slice of cells 32 s .. 32 s + 31 is at ptr[s] +
// 32 v + t: face | flags, or -1; its other cell; its entry, counted from the
// row's first.
struct AsmLists {
  const int* ptr;
  const int* face;
  const int* other;
  const unsigned short* entry;
};
constexpr int kAsmSecond = 1 << 30;     // the cell is the face's c2
constexpr int kAsmBoundary = 1 << 29;
constexpr int kAsmFace = kAsmBoundary - 1;

// k: AsmPressure or AsmMomentum.
template <class K>
__global__ void __launch_bounds__(kAsmCells, 10) k_asm_rows(int n, const int* __restrict__ row,
                                                        const int* __restrict__ dia, AsmLists L,
                                                        K k, int cap,
                                                        double* __restrict__ val) {
  extern __shared__ double tf_asm_tile[];
  const int c0 = blockIdx.x * kAsmCells, c1 = min(n, c0 + kAsmCells), t = threadIdx.x;
  const int j0 = row[c0], j1 = row[c1], ne = j1 - j0;
  const bool staged = ne <= cap;
  double* tile = staged ? tf_asm_tile : val + j0;
  for (int e = t; e < ne; e += kAsmCells) tile[e] = 0.0;
  __syncthreads();
  const int c = c0 + t;
  if (c < n) {
    double d = 0.0;
    const int s = c >> 5, v0 = L.ptr[s], v1 = L.ptr[s + 1], jc = row[c] - j0;
    bool boundary = false;
    // kAsmBatch visits' loads in flight, then their sums in order
    for (int v = v0 + (c & 31); v < v1; v += 32 * kAsmBatch) {
      int f[kAsmBatch], e[kAsmBatch], o[kAsmBatch];
      double a[kAsmBatch];
#pragma unroll
      for (int u = 0; u < kAsmBatch; ++u) {
        const bool in = v + 32 * u < v1;
        f[u] = in ? L.face[v + 32 * u] : -1;
        e[u] = in ? L.entry[v + 32 * u] : 0;
        if (K::kOther) o[u] = in ? L.other[v + 32 * u] : 0;
      }
#pragma unroll
      for (int u = 0; u < kAsmBatch; ++u)
        a[u] = f[u] >= 0 && !(f[u] & kAsmBoundary)
                   ? k.interior(f[u] & kAsmFace, f[u] & kAsmSecond, c, K::kOther ? o[u] : 0)
                   : 0.0;
#pragma unroll
      for (int u = 0; u < kAsmBatch; ++u) {
        if (f[u] < 0) continue;
        if (!(f[u] & kAsmBoundary)) {
          tile[jc + e[u]] = k.entry(a[u]);
          d = __dadd_rn(d, a[u]);
        } else {
          boundary = true;
          d = k.boundary(d, f[u] & kAsmFace);
        }
      }
    }
    if (boundary && k.late())   // faces of a later loop
      for (int v = v0 + (c & 31); v < v1; v += 32) {
        const int f = L.face[v];
        if (f < 0) break;
        if (f & kAsmBoundary) d = k.late_boundary(d, f & kAsmFace, c);
      }
    tile[dia[c] - j0] = k.done(d, c);
  }
  if (!staged) return;
  __syncthreads();
  for (int e = t; e < ne; e += kAsmCells) val[j0 + e] = tile[e];
}

// Whether every entry of pos (1-based) lies in the row of its face's cell.
__global__ void __launch_bounds__(256) k_asm_own(int nf, const int* __restrict__ faces,
                                                 const int* __restrict__ pos,
                                                 const int* __restrict__ row, int* foreign) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nf; s += gridDim.x * blockDim.x) {
    if (faces[2 * s + 1] <= 0) continue;
    for (int k = 0; k < 2; ++k) {
      const int c = faces[2 * s + k] - 1, p = pos[2 * s + k] - 1;
      if (p < row[c] || p >= row[c + 1]) *foreign = 1;
    }
  }
}

// The other cells and the entries of the listed faces, a thread a cell.
__global__ void __launch_bounds__(256) k_asm_lists(int n, const int* __restrict__ faces,
                                                   const int* __restrict__ pos,
                                                   const int* __restrict__ row,
                                                   const int* __restrict__ ptr,
                                                   const int* __restrict__ face, int* other,
                                                   unsigned short* entry) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  for (int v = ptr[c >> 5] + (c & 31); v < ptr[(c >> 5) + 1]; v += 32) {
    const int f = face[v];
    if (f < 0) break;
    if (f & kAsmBoundary) continue;
    const int s = f & kAsmFace, k = f & kAsmSecond ? 1 : 0;
    other[v] = faces[2 * s + 1 - k] - 1;
    entry[v] = (unsigned short)(pos[2 * s + k] - 1 - row[c]);
  }
}

// Pressure: interior faces (Rhie_And_Chow.f90:183-205), then the open
// boundary faces (Compute_Pressure.f90:140-160).
struct AsmPressure {
  static constexpr bool kOther = true;
  const double* fc;
  const double* fw;
  const double* vm;
  const int* open;
  __device__ __forceinline__ double interior(int s, bool second, int c, int o) const {
    return second ? p_coef(fc, fw, vm, s, o, c) : p_coef(fc, fw, vm, s, c, o);
  }
  __device__ __forceinline__ double entry(double a) const { return -a; }
  __device__ __forceinline__ double boundary(double d, int) const { return d; }
  __device__ __forceinline__ bool late() const { return open != nullptr; }
  __device__ __forceinline__ double late_boundary(double d, int s, int c) const {
    return open[s] ? __dadd_rn(d, __dmul_rn(fc[s], vm ? vm[c] : 1.0)) : d;
  }
  __device__ __forceinline__ double done(double d, int) const { return d; }
};

// ---------------------------------------------------------------------------
// Face by face, for a pos map that leaves the cells' own rows
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_asm_p_off(int nf, const int* __restrict__ fcell,
                                                   const int* __restrict__ fpos,
                                                   const double* __restrict__ fc,
                                                   const double* __restrict__ fw,
                                                   const double* __restrict__ vm,
                                                   double* __restrict__ val) {
  const int stride = gridDim.x * blockDim.x;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nf; s += stride) {
    const int c1 = fcell[2 * s], c2 = fcell[2 * s + 1];
    if (c2 < 0) continue;
    const double a12 = p_coef(fc, fw, vm, s, c1, c2);
    val[fpos[2 * s]] = -a12;
    val[fpos[2 * s + 1]] = -a12;
  }
}

__global__ void __launch_bounds__(256) k_asm_p_diag(int n, const int* __restrict__ cf_ptr,
                                                    const int* __restrict__ cf,
                                                    const int* __restrict__ fcell,
                                                    const int* __restrict__ dia,
                                                    const double* __restrict__ fc,
                                                    const double* __restrict__ fw,
                                                    const double* __restrict__ vm,
                                                    const int* __restrict__ bnd_open,
                                                    double* __restrict__ val) {
  const int stride = gridDim.x * blockDim.x;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += stride) {
    double d = 0.0;
    const int e0 = cf_ptr[c], e1 = cf_ptr[c + 1];
    for (int e = e0; e < e1; ++e) {   // interior faces (Rhie_And_Chow.f90:183-205)
      const int s = cf[e] >> 1;
      const int c1 = fcell[2 * s], c2 = fcell[2 * s + 1];
      if (c2 >= 0) d = __dadd_rn(d, p_coef(fc, fw, vm, s, c1, c2));
    }
    if (bnd_open) {                   // boundary faces (Compute_Pressure.f90:140-160)
      for (int e = e0; e < e1; ++e) {
        const int s = cf[e] >> 1;
        if (fcell[2 * s + 1] < 0 && bnd_open[s])
          d = __dadd_rn(d, __dmul_rn(fc[s], vm ? vm[c] : 1.0));
      }
    }
    val[dia[c]] = d;
  }
}

struct MomCoef {
  double m12, m21;
};
// Compute_Momentum.f90:270-297 with blend_matrix: upwind-blended m12, m21
__device__ __forceinline__ MomCoef m_coef(const double* fc, const double* flux, double vis,
                                          double rho, int s) {
  const double m0 = __dmul_rn(vis, fc[s]);
  const double f = flux[s];
  MomCoef k;
  k.m12 = __dsub_rn(m0, __dmul_rn(fmin_ref(f, 0.0), rho));
  k.m21 = __dadd_rn(m0, __dmul_rn(fmax_ref(f, 0.0), rho));
  return k;
}

__global__ void __launch_bounds__(256) k_asm_m_off(int nf, const int* __restrict__ fcell,
                                                   const int* __restrict__ fpos,
                                                   const double* __restrict__ fc,
                                                   const double* __restrict__ flux,
                                                   double vis, double rho,
                                                   double* __restrict__ val) {
  const int stride = gridDim.x * blockDim.x;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nf; s += stride) {
    if (fcell[2 * s + 1] < 0) continue;
    const MomCoef k = m_coef(fc, flux, vis, rho, s);
    val[fpos[2 * s]] = __dsub_rn(0.0, k.m12);
    val[fpos[2 * s + 1]] = __dsub_rn(0.0, k.m21);
  }
}

__global__ void __launch_bounds__(256) k_asm_m_diag(int n, const int* __restrict__ cf_ptr,
                                                    const int* __restrict__ cf,
                                                    const int* __restrict__ fcell,
                                                    const int* __restrict__ dia,
                                                    const double* __restrict__ fc,
                                                    const double* __restrict__ flux,
                                                    const int* __restrict__ bnd_wall,
                                                    double vis, double rho,
                                                    const double* __restrict__ vol, double dt,
                                                    double* __restrict__ val) {
  const int stride = gridDim.x * blockDim.x;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += stride) {
    double d = 0.0;
    for (int e = cf_ptr[c]; e < cf_ptr[c + 1]; ++e) {
      const int s = cf[e] >> 1, second = cf[e] & 1;
      const bool interior = fcell[2 * s + 1] >= 0;
      if (!interior && !(bnd_wall && bnd_wall[s])) continue;
      const MomCoef k = m_coef(fc, flux, vis, rho, s);
      d = __dadd_rn(d, second ? k.m21 : k.m12);
    }
    // Inertial_Term.f90 (linear): a0 = rho * vol / dt
    d = __dadd_rn(d, __ddiv_rn(__dmul_rn(rho, vol[c]), dt));
    val[dia[c]] = d;
  }
}

// Momentum: the faces in their order, wall faces among them, then
// Inertial_Term.f90 (linear): a0 = rho * vol / dt.
struct AsmMomentum {
  static constexpr bool kOther = false;
  const double* fc;
  const double* flux;
  const int* wall;
  double vis, rho;
  const double* vol;
  double dt;
  __device__ __forceinline__ double interior(int s, bool second, int, int) const {
    const MomCoef k = m_coef(fc, flux, vis, rho, s);
    return second ? k.m21 : k.m12;
  }
  __device__ __forceinline__ double entry(double a) const { return __dsub_rn(0.0, a); }
  __device__ __forceinline__ double boundary(double d, int s) const {
    return wall && wall[s] ? __dadd_rn(d, m_coef(fc, flux, vis, rho, s).m12) : d;
  }
  __device__ __forceinline__ bool late() const { return false; }
  __device__ __forceinline__ double late_boundary(double d, int, int) const { return d; }
  __device__ __forceinline__ double done(double d, int c) const {
    return __dadd_rn(d, __ddiv_rn(__dmul_rn(rho, vol[c]), dt));
  }
};

}  // namespace tf

using namespace tf;

namespace {

void faces_free(tf_matrix_s* m) {
  tf_dev_free(m->ctx, m->face_block);
  m->face_block = nullptr;
  m->d_face_cell = m->d_face_pos = m->d_cf_ptr = m->d_cf = m->d_cf_other = nullptr;
  m->d_cf_entry = nullptr;
  m->n_faces = 0;
}

size_t place_bytes(size_t count, size_t size) { return (count * size + 127) & ~(size_t)127; }

// Cuts `count` T off the block at p.
template <class T>
T* cut(unsigned char*& p, size_t count) {
  T* t = reinterpret_cast<T*>(p);
  p += place_bytes(count, sizeof(T));
  return t;
}

int upload(tf_ctx_s* ctx, int* d, const int* h, size_t count) {
  if (count > 0)
    TF_CUDA_TRY(cudaMemcpyAsync(d, h, count * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
  return TF_OK;
}

// The lists of the assembly by rows; cnt: faces a cell.  TF_ERR_OOM when there
// is no room for them, *took = 0 when they are not for these faces.
int row_lists(tf_matrix_s* m, int n_faces, const int* faces_c, const int* pos,
              const std::vector<int>& cnt, int* took) {
  const int n = m->nt;
  *took = 0;
  if (n_faces >= kAsmBoundary || m->max_row_len > 65536) return TF_OK;
  // Padded to the longest of 32 cells: not where a few cells with many faces
  // would make them several times the faces (10 bytes a place).
  std::vector<int> sptr((size_t)(n + 31) / 32 + 1, 0);
  long long places = 0, visits = 0;
  for (int c0 = 0; c0 < n; c0 += 32) {
    int w = 0;
    for (int c = c0; c < std::min(n, c0 + 32); ++c) {
      w = std::max(w, cnt[c]);
      visits += cnt[c];
    }
    places += 32LL * w;
    if (places > INT_MAX - 32) return TF_OK;
    sptr[c0 / 32 + 1] = (int)places;
  }
  if (places > std::max(4 * visits, (long long)kAsmPlaces)) return TF_OK;
  // Every cell's faces in ascending order, next[c]: the place of its next one.
  std::unique_ptr<int[]> face(new int[places + 32]);
  std::vector<int> next(n);
  for (int c = 0; c < n; ++c) next[c] = sptr[c >> 5] + (c & 31);
  auto put = [&](int c, int f) {
    face[next[c]] = f;
    next[c] += 32;
  };
  for (int s = 0; s < n_faces; ++s) {
    const int c2 = faces_c[2 * s + 1];
    put(faces_c[2 * s] - 1, s | (c2 > 0 ? 0 : kAsmBoundary));
    if (c2 > 0) put(c2 - 1, s | kAsmSecond);
  }
  for (int c = 0; c < n; ++c)
    for (int v = next[c]; v < sptr[(c >> 5) + 1]; v += 32) face[v] = -1;
  // The rest is looked up on the device.
  tf_ctx_s* ctx = m->ctx;
  cudaStream_t s = ctx->stream;
  const size_t words = (size_t)2 * n_faces, np = (size_t)places + 32;
  // A flag, the faces, pos: in the values' workspace, which holds nothing between
  // solves, unless boundary faces make them longer (an allocation and its
  // release are a third of the call on 27,000 cells).
  int *own = nullptr, *given = reinterpret_cast<int*>(m->d_val), foreign = 0;
  auto build = [&]() -> int {
    int st = TF_OK;
    if (1 + 2 * words > (size_t)m->nnz * 2) {
      st = tf_dev_alloc_bytes(ctx, (void**)&own, (1 + 2 * words) * sizeof(int));
      given = own;
    }
    if (st == TF_OK)
      st = tf_dev_alloc_bytes(ctx, &m->face_block, place_bytes(sptr.size(), 4) +
                                                       2 * place_bytes(np, 4) + place_bytes(np, 2));
    if (st != TF_OK) return st;
    unsigned char* p = static_cast<unsigned char*>(m->face_block);
    m->d_cf_ptr = cut<int>(p, sptr.size());
    m->d_cf = cut<int>(p, np);
    m->d_cf_other = cut<int>(p, np);
    m->d_cf_entry = cut<unsigned short>(p, np);
    int *d_faces = given + 1, *d_pos = d_faces + words;
    TF_CUDA_TRY(cudaMemsetAsync(given, 0, sizeof(int), s));
    st = upload(ctx, d_faces, faces_c, words);
    if (st == TF_OK) st = upload(ctx, d_pos, pos, words);
    if (st == TF_OK) st = upload(ctx, m->d_cf_ptr, sptr.data(), sptr.size());
    if (st == TF_OK) st = upload(ctx, m->d_cf, face.get(), (size_t)places);
    if (st != TF_OK) return st;
    k_asm_own<<<ctx->sm_count * 8, 256, 0, s>>>(n_faces, d_faces, d_pos, m->d_row, given);
    k_asm_lists<<<std::max(1, (n + 255) / 256), 256, 0, s>>>(n, d_faces, d_pos, m->d_row,
                                                             m->d_cf_ptr, m->d_cf,
                                                             m->d_cf_other, m->d_cf_entry);
    TF_CUDA_TRY(cudaGetLastError());
    TF_CUDA_TRY(cudaMemcpyAsync(&foreign, given, sizeof(int), cudaMemcpyDeviceToHost, s));
    return TF_OK;
  };
  int st = build();
  const cudaError_t e = cudaStreamSynchronize(s);   // the arrays copied from are still here
  tf_dev_free(ctx, own);
  if (st == TF_OK) TF_CUDA_TRY(e);
  *took = !foreign;
  return st;
}

// The lists of the assembly face by face.
int face_lists(tf_matrix_s* m, int n_faces, const int* faces_c, const int* pos,
               const std::vector<int>& cnt) {
  const int n = m->nt;
  std::vector<int> fcell((size_t)2 * n_faces + 2), fpos((size_t)2 * n_faces + 2);
  for (int s = 0; s < n_faces; ++s) {
    const int c2 = faces_c[2 * s + 1];
    fcell[2 * s] = faces_c[2 * s] - 1;
    fcell[2 * s + 1] = c2 > 0 ? c2 - 1 : -1;
    fpos[2 * s] = c2 > 0 ? pos[2 * s] - 1 : -1;
    fpos[2 * s + 1] = c2 > 0 ? pos[2 * s + 1] - 1 : -1;
  }
  // cell -> faces in ascending face order; bit 0: the cell is the face's c2
  std::vector<int> ptr((size_t)n + 1, 0);
  for (int c = 0; c < n; ++c) ptr[c + 1] = ptr[c] + cnt[c];
  std::vector<int> cf((size_t)ptr[n] + 1), fill(ptr.begin(), ptr.end() - 1);
  for (int s = 0; s < n_faces; ++s) {
    cf[fill[fcell[2 * s]]++] = s << 1;
    if (fcell[2 * s + 1] >= 0) cf[fill[fcell[2 * s + 1]]++] = (s << 1) | 1;
  }
  int st = tf_dev_alloc_bytes(m->ctx, &m->face_block,
                              place_bytes(fcell.size(), 4) + place_bytes(fpos.size(), 4) +
                                  place_bytes(ptr.size(), 4) + place_bytes(cf.size(), 4));
  if (st != TF_OK) return st;
  unsigned char* p = static_cast<unsigned char*>(m->face_block);
  m->d_face_cell = cut<int>(p, fcell.size());
  m->d_face_pos = cut<int>(p, fpos.size());
  m->d_cf_ptr = cut<int>(p, ptr.size());
  m->d_cf = cut<int>(p, cf.size());
  st = upload(m->ctx, m->d_face_cell, fcell.data(), fcell.size());
  if (st == TF_OK) st = upload(m->ctx, m->d_face_pos, fpos.data(), fpos.size());
  if (st == TF_OK) st = upload(m->ctx, m->d_cf_ptr, ptr.data(), ptr.size());
  if (st == TF_OK) st = upload(m->ctx, m->d_cf, cf.data(), cf.size());
  TF_CUDA_TRY(cudaStreamSynchronize(m->ctx->stream));
  return st;
}

}  // namespace

extern "C" int tf_faces_register(tf_ctx ctx, tf_matrix m, int n_faces, const int* faces_c,
                                 const int* pos) {
  TF_API_BEGIN
  if (!ctx || !m || m->ctx != ctx || n_faces < 0 || (n_faces > 0 && (!faces_c || !pos)))
    return TF_ERR_ARG;
  const int n = m->nt;
  std::vector<int> cnt((size_t)n + 1, 0);
  for (int s = 0; s < n_faces; ++s) {
    const int c1 = faces_c[2 * s], c2 = faces_c[2 * s + 1];
    if (c1 < 1 || c1 > n || c2 > n) return TF_ERR_LAYOUT;
    ++cnt[c1 - 1];
    if (c2 > 0) {
      const int p1 = pos[2 * s], p2 = pos[2 * s + 1];
      if (p1 < 1 || p1 > m->nnz || p2 < 1 || p2 > m->nnz) return TF_ERR_LAYOUT;
      ++cnt[c2 - 1];
    }
  }
  std::lock_guard<std::mutex> lk(m->mu);
  TF_CUDA_TRY(cudaSetDevice(ctx->device));
  faces_free(m);
  // Every entry in its own cell's row (as Create_Matrix builds pos): the rows
  // are assembled cell by cell.
  int took = 0;
  int st = row_lists(m, n_faces, faces_c, pos, cnt, &took);
  if (st == TF_ERR_OOM || (st == TF_OK && !took)) {
    faces_free(m);
    cudaGetLastError();
    st = face_lists(m, n_faces, faces_c, pos, cnt);
  }
  // Half a list is none: tf_assemble_* refuses the matrix.
  if (st != TF_OK) faces_free(m);
  else m->n_faces = n_faces;
  return st;
  TF_API_END
}

namespace {
int grid_for(tf_matrix_s* m, int items) {
  return std::max(1, std::min(m->ctx->sm_count * 8, (items + 255) / 256));
}

template <class K>
int assemble_rows(tf_matrix_s* m, const K& k, double* d_val) {
  const AsmLists lists{m->d_cf_ptr, m->d_cf, m->d_cf_other, m->d_cf_entry};
  // (a longer tile is assembled in global memory)
  const int cap = (int)std::min<long long>(kAsmEntries, (long long)m->max_row_len * kAsmCells);
  if (m->nt > 0)
    k_asm_rows<K><<<(m->nt + kAsmCells - 1) / kAsmCells, kAsmCells, cap * sizeof(double),
                    m->ctx->stream>>>(m->nt, m->d_row, m->d_dia, lists, k, cap, d_val);
  TF_CUDA_TRY(cudaGetLastError());
  return TF_OK;
}
}  // namespace

extern "C" int tf_assemble_pressure(tf_ctx ctx, tf_matrix m, const double* d_fc,
                                    const double* d_fw, const double* d_vm,
                                    const int* d_bnd_open, double* d_val) {
  TF_API_BEGIN
  if (!ctx || !m || m->ctx != ctx || !m->d_cf_ptr || !d_fc || !d_fw || !d_val)
    return TF_ERR_ARG;
  std::lock_guard<std::mutex> lk(m->mu);
  TF_CUDA_TRY(cudaSetDevice(ctx->device));
  cudaStream_t s = ctx->stream;
  if (m->d_cf_other) return assemble_rows(m, AsmPressure{d_fc, d_fw, d_vm, d_bnd_open}, d_val);
  TF_CUDA_TRY(cudaMemsetAsync(d_val, 0, (size_t)m->nnz * sizeof(double), s));
  if (m->n_faces > 0)
    k_asm_p_off<<<grid_for(m, m->n_faces), 256, 0, s>>>(m->n_faces, m->d_face_cell,
                                                         m->d_face_pos, d_fc, d_fw, d_vm, d_val);
  k_asm_p_diag<<<grid_for(m, m->nt), 256, 0, s>>>(m->nt, m->d_cf_ptr, m->d_cf, m->d_face_cell,
                                                   m->d_dia, d_fc, d_fw, d_vm, d_bnd_open,
                                                   d_val);
  TF_CUDA_TRY(cudaGetLastError());
  return TF_OK;
  TF_API_END
}

extern "C" int tf_assemble_momentum(tf_ctx ctx, tf_matrix m, const double* d_fc,
                                    const double* d_flux, const int* d_bnd_wall, double vis,
                                    double rho, const double* d_vol, double dt, double* d_val) {
  TF_API_BEGIN
  if (!ctx || !m || m->ctx != ctx || !m->d_cf_ptr || !d_fc || !d_flux || !d_vol || !d_val)
    return TF_ERR_ARG;
  std::lock_guard<std::mutex> lk(m->mu);
  TF_CUDA_TRY(cudaSetDevice(ctx->device));
  cudaStream_t s = ctx->stream;
  if (m->d_cf_other)
    return assemble_rows(m, AsmMomentum{d_fc, d_flux, d_bnd_wall, vis, rho, d_vol, dt}, d_val);
  TF_CUDA_TRY(cudaMemsetAsync(d_val, 0, (size_t)m->nnz * sizeof(double), s));
  if (m->n_faces > 0)
    k_asm_m_off<<<grid_for(m, m->n_faces), 256, 0, s>>>(m->n_faces, m->d_face_cell,
                                                         m->d_face_pos, d_fc, d_flux, vis, rho,
                                                         d_val);
  k_asm_m_diag<<<grid_for(m, m->nt), 256, 0, s>>>(m->nt, m->d_cf_ptr, m->d_cf, m->d_face_cell,
                                                   m->d_dia, d_fc, d_flux, d_bnd_wall, vis, rho,
                                                   d_vol, dt, d_val);
  TF_CUDA_TRY(cudaGetLastError());
  return TF_OK;
  TF_API_END
}
