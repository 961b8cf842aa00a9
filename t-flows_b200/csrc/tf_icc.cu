// tf_icc.cu -- host side of the level-scheduled incomplete Cholesky:
// level sets of the forward and backward sweeps, computed once per matrix
// from its structure.
#include <limits.h>
#include <stdlib.h>

#include <algorithm>
#include <vector>

#include "tf_icc.cuh"
#include "tf_internal.h"

using namespace tf;

namespace {

// Counting sort of rows by level: rows[ptr[l] .. ptr[l+1]) are level l.
void bucket(const std::vector<int>& lev, int nlev, std::vector<int>& ptr,
            std::vector<int>& rows) {
  ptr.assign(nlev + 1, 0);
  for (int v : lev) ptr[v + 1]++;
  for (int l = 0; l < nlev; ++l) ptr[l + 1] += ptr[l];
  rows.resize(lev.size());
  std::vector<int> fill(ptr.begin(), ptr.end() - 1);
  for (int i = 0; i < (int)lev.size(); ++i) rows[fill[lev[i]]++] = i;
}

}  // namespace

// Levels of the sweeps in Prec_Form.f90:69-78 / Prec_Solve.f90:67-92.
// Forward: row i waits for the lower entries visited by `do j = a_row(i)+1,
// ...; if(k > i) exit`; backward: for the upper entries visited from the
// row's end down to `if(k < i) exit`, owned rows only (k <= ni).
int tf_icc_build(tf_matrix_s* m, const int* row0, const int* col0) {
  if (const char* form = getenv("TF_ICC_SWEEPS"))   // "one" CTA, or a kernel per level
    m->icc_form = form[0] == 'o' ? 1 : -1;
  const int ni = m->ni;
  std::vector<int> levf(ni, 0), levb(ni, 0);
  int nf = 0, nb = 0;
  // Entries the sweeps visit (with buffer cells'), and the levels of rows longer
  // than is packed.
  long long entries = 0;
  std::vector<int> longf, longb;
  for (int i = 0; i < ni; ++i) {
    int l = 0, j = row0[i] + 1;
    for (; j < row0[i + 1]; ++j) {
      const int k = col0[j];
      if (k > i) break;
      l = std::max(l, levf[k] + 1);
    }
    levf[i] = l;
    nf = std::max(nf, l + 1);
    const int len = j - row0[i] - 1;
    entries += len;
    if (len > kIccWidth) longf.push_back(l);
  }
  for (int i = ni - 1; i >= 0; --i) {
    int l = 0, j = row0[i + 1] - 1;
    for (; j >= row0[i] + 1; --j) {
      const int k = col0[j];
      if (k < i) break;
      if (k < ni) l = std::max(l, levb[k] + 1);
    }
    levb[i] = l;
    nb = std::max(nb, l + 1);
    const int len = row0[i + 1] - 1 - j;
    entries += len;
    if (len > kIccWidth) longb.push_back(l);
  }
  m->icc_entries = entries;
  m->icc_long_levels = 0;
  for (auto* lev : {&longf, &longb}) {
    std::sort(lev->begin(), lev->end());
    m->icc_long_levels += (int)(std::unique(lev->begin(), lev->end()) - lev->begin());
  }
  std::vector<int> rf, rb;
  bucket(levf, nf, m->h_levf_ptr, rf);
  bucket(levb, nb, m->h_levb_ptr, rb);
  const size_t nv = (size_t)m->nt + 8;
  void* p = nullptr;
  int st = tf_dev_alloc_bytes(m->ctx, &p, std::max<size_t>(rf.size(), 1) * sizeof(int));
  m->d_levf_rows = (int*)p;
  if (st == TF_OK) st = tf_dev_alloc_bytes(m->ctx, &p, std::max<size_t>(rb.size(), 1) * sizeof(int));
  m->d_levb_rows = (int*)p;
  if (st == TF_OK) st = tf_dev_alloc_bytes(m->ctx, &p, nv * sizeof(double));
  m->d_z = (double*)p;
  if (st == TF_OK) st = tf_dev_alloc_bytes(m->ctx, &p, nv * sizeof(double));
  m->d_icc_d = (double*)p;
  if (st == TF_OK) st = tf_dev_alloc_bytes(m->ctx, &p, nv * sizeof(double));
  m->d_icc_dinv = (double*)p;
  if (st != TF_OK) return st;
  // From pageable memory these return once the source has been staged.
  TF_CUDA_TRY(cudaMemcpyAsync(m->d_levf_rows, rf.data(), rf.size() * sizeof(int),
                              cudaMemcpyHostToDevice, m->ctx->stream));
  TF_CUDA_TRY(cudaMemcpyAsync(m->d_levb_rows, rb.data(), rb.size() * sizeof(int),
                              cudaMemcpyHostToDevice, m->ctx->stream));
  if (!m->ctx->async_alloc) TF_CUDA_TRY(cudaStreamSynchronize(m->ctx->stream));
  m->icc_ready = 1;
  return TF_OK;
}

namespace {

// Slices of at most 32 rows of one level: meta = {first position, rows, 0,
// level}.
void cut_slices(const std::vector<int>& ptr, std::vector<int4>& meta, std::vector<int>& first) {
  for (size_t l = 0; l + 1 < ptr.size(); ++l) {
    first.push_back((int)meta.size());
    for (int p = ptr[l]; p < ptr[l + 1]; p += 32)
      meta.push_back(make_int4(p, std::min(32, ptr[l + 1] - p), 0, (int)l));
  }
}

// An array of the records, within what the matrix may hold beside its own.
template <class T>
int dev_array(tf_matrix_s* m, T** p, size_t count) {
  const size_t bytes = (count + 8) * sizeof(T);
  if (m->extra_bytes + m->icc_bytes + bytes > m->extra_limit) return TF_ERR_OOM;
  void* v = nullptr;
  const int st = tf_dev_alloc_bytes(m->ctx, &v, bytes);
  *p = static_cast<T*>(v);
  if (st == TF_OK) m->icc_bytes += bytes;
  return st;
}

// Whether one CTA walks the levels: by rows and entries a level, on average over
// both sweeps (kIccOneRows and what follows it).
bool narrow_levels(const tf_matrix_s* m) {
  if (m->icc_form != 0) return m->icc_form > 0;
  const long long levels = (long long)(m->h_levf_ptr.size() + m->h_levb_ptr.size()) - 2;
  const bool long_rows = 8LL * m->icc_long_levels > levels;
  return 2LL * m->ni <= kIccOneRows * levels &&
         m->icc_entries <= (long_rows ? kIccOneLongEntries : kIccOneEntries) * levels;
}

// Batch, packed width, consumer warps, stages and ring slots for the widest
// row (kIccWidth at most).  The stages are a multiple of the chunks the warps
// work on at a time (icc_sweep).
void choose_layout(tf_matrix_s* m, int widest) {
  m->icc_batch = widest <= 3 ? 3 : 4;   // a hex row has 3 entries either way
  const int w = m->icc_width = std::max(1, (widest + m->icc_batch - 1) / m->icc_batch) * m->icc_batch;
  m->icc_warps = w <= 4 ? 24 : 16;
  m->icc_stages = w <= 4 ? 6 : 4;
  m->icc_ring = 8192;
  if (IccLayout(w, m->icc_stages, m->icc_ring).total > kIccSmemBytes) m->icc_stages = 2;
}

// The records of both sweeps, made on the device before the first ICC solve
// of a matrix (a matrix that is never solved with ICC carries none).
int pack(tf_matrix_s* m) {
  cudaStream_t s = m->ctx->stream;
  const std::vector<int>* ptrs[2] = {&m->h_levf_ptr, &m->h_levb_ptr};
  const int* rows[2] = {m->d_levf_rows, m->d_levb_rows};
  struct Info {
    int widest[2], far_any[2];
    long long total[2][2];   // entries, record bytes / 16
  } info{};
  int* d_info = nullptr;
  int* d_ptr[2] = {nullptr, nullptr};      // first position of every level
  int* d_first[2] = {nullptr, nullptr};    // first slice of every level
  int* d_pos[2] = {nullptr, nullptr};
  std::vector<int4> slices[2];
  std::vector<int> first[2];
  auto grid = [](long long threads) { return (int)((threads + 255) / 256); };
  auto build = [&]() -> int {
    int st = dev_array(m, &d_info, sizeof(Info) / sizeof(int));
    if (st != TF_OK) return st;
    for (int k = 0; k < 2; ++k) {
      tf_icc_dir_s& g = m->icc_dir[k];
      cut_slices(*ptrs[k], slices[k], first[k]);
      g.nslices = (int)slices[k].size();
      const int nchunks = (g.nslices + kIccChunk - 1) / kIccChunk;
      st = dev_array(m, &g.slice, slices[k].size());
      if (st == TF_OK) st = dev_array(m, &g.chunk, nchunks);
      if (st == TF_OK) st = dev_array(m, &g.idx, m->ni);
      if (st == TF_OK) st = dev_array(m, &d_pos[k], m->ni);
      if (st == TF_OK) st = dev_array(m, &d_ptr[k], ptrs[k]->size());
      if (st == TF_OK) st = dev_array(m, &d_first[k], first[k].size());
      if (st != TF_OK) return st;
      TF_CUDA_TRY(cudaMemcpyAsync(g.slice, slices[k].data(), slices[k].size() * sizeof(int4),
                                  cudaMemcpyHostToDevice, s));
      TF_CUDA_TRY(cudaMemcpyAsync(d_ptr[k], ptrs[k]->data(), ptrs[k]->size() * sizeof(int),
                                  cudaMemcpyHostToDevice, s));
      TF_CUDA_TRY(cudaMemcpyAsync(d_first[k], first[k].data(), first[k].size() * sizeof(int),
                                  cudaMemcpyHostToDevice, s));
      const int gs = grid((long long)g.nslices * 32);
      if (k == 0)
        k_icc_widths<kIccFwd><<<gs, 256, 0, s>>>(m->d_row, m->d_col, m->ni, rows[k], g.slice,
                                                 g.nslices, d_info + k);
      else
        k_icc_widths<kIccBwd><<<gs, 256, 0, s>>>(m->d_row, m->d_col, m->ni, rows[k], g.slice,
                                                 g.nslices, d_info + k);
      TF_CUDA_TRY(cudaGetLastError());
    }
    TF_CUDA_TRY(cudaMemcpyAsync(&info, d_info, sizeof info, cudaMemcpyDeviceToHost, s));
    TF_CUDA_TRY(cudaStreamSynchronize(s));
    choose_layout(m, std::max(info.widest[0], info.widest[1]));
    for (int k = 0; k < 2; ++k) {
      tf_icc_dir_s& g = m->icc_dir[k];
      const int nchunks = (g.nslices + kIccChunk - 1) / kIccChunk;
      const int gs = grid((long long)g.nslices * 32);
      k_icc_chunks<<<grid(nchunks), 256, 0, s>>>(g.slice, g.nslices, m->icc_batch, g.chunk);
      k_icc_offsets<<<1, 1024, 0, s>>>(g.slice, g.nslices, g.chunk, nchunks,
                                       reinterpret_cast<long long*>(d_info + 4) + 2 * k);
      k_icc_places<<<gs, 256, 0, s>>>(rows[k], g.slice, g.chunk, g.nslices, d_pos[k], g.idx);
      TF_CUDA_TRY(cudaGetLastError());
    }
    TF_CUDA_TRY(cudaMemcpyAsync(&info, d_info, sizeof info, cudaMemcpyDeviceToHost, s));
    TF_CUDA_TRY(cudaStreamSynchronize(s));
    for (int k = 0; k < 2; ++k) {
      tf_icc_dir_s& g = m->icc_dir[k];
      // 32-bit indices: entries, and doubles in the records
      if (info.total[k][0] > INT_MAX - 64 || info.total[k][1] > INT_MAX / 2 - 64)
        return TF_ERR_OOM;
      st = dev_array(m, &g.src, (size_t)info.total[k][0]);
      if (st == TF_OK) st = dev_array(m, &g.rec, (size_t)info.total[k][1] * 16);
      if (st != TF_OK) return st;
      const int gs = grid((long long)g.nslices * 32);
      if (k == 0)
        k_icc_fill<kIccFwd><<<gs, 256, 0, s>>>(
            m->d_row, m->d_col, m->ni, rows[k], d_pos[k], d_ptr[k], d_first[k], g.slice, g.chunk,
            g.nslices, m->icc_ring, m->icc_dir[1].idx, g.src, g.rec, d_info + 2 + k);
      else
        k_icc_fill<kIccBwd><<<gs, 256, 0, s>>>(
            m->d_row, m->d_col, m->ni, rows[k], d_pos[k], d_ptr[k], d_first[k], g.slice, g.chunk,
            g.nslices, m->icc_ring, m->icc_dir[0].idx, g.src, g.rec, d_info + 2 + k);
      TF_CUDA_TRY(cudaGetLastError());
    }
    TF_CUDA_TRY(cudaMemcpyAsync(&info, d_info, sizeof info, cudaMemcpyDeviceToHost, s));
    TF_CUDA_TRY(cudaStreamSynchronize(s));
    for (int k = 0; k < 2; ++k) m->icc_dir[k].far_any = info.far_any[k];
    return TF_OK;
  };
  tf_icc_free(m);   // an earlier attempt's
  const int st = build();
  for (int* q : {d_info, d_ptr[0], d_ptr[1], d_first[0], d_first[1], d_pos[0], d_pos[1]})
    tf_dev_free(m->ctx, q);
  return st;
}

IccDir dir_args(const tf_icc_dir_s& g, const int* rows) {
  IccDir d{};
  d.ord = rows;
  d.slice = g.slice;
  d.chunk = g.chunk;
  d.src = g.src;
  d.rec = g.rec;
  d.idx = g.idx;
  d.nslices = g.nslices;
  d.far_any = g.far_any;
  return d;
}

template <int K, int B, int W>
int plan_one(tf_matrix_s* m, tf_icc_plan* p) {
  const int smem = IccLayout(m->icc_width, m->icc_stages, m->icc_ring).total;
  const void* form = (const void*)k_icc_form<K, B, W>;
  const void* apply = (const void*)k_icc_apply<K, B, W>;
  for (const void* f : {form, apply})
    TF_CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  p->form = {{(const void*)k_icc_pack, m->vec_grid, 256, 0, {&p->one}},
             {form, 1, 32 * (W + kIccProducers), (size_t)smem, {&p->one}}};
  p->apply = {{apply, 1, 32 * (W + kIccProducers), (size_t)smem, {&p->one}}};
  return TF_OK;
}

void plan_levels(tf_matrix_s* m, tf_icc_plan* p) {
  IccLevelArgs base{};
  base.row = m->d_row;
  base.col = m->d_col;
  base.val = m->d_val;
  base.ni = m->ni;
  base.d = m->d_icc_d;
  base.d_inv = m->d_icc_dinv;
  base.r = m->d_r;
  base.y = m->d_q;   // q is free between k_update and the next SpMV
  base.z = m->d_z;
  const size_t nf = m->h_levf_ptr.size() - 1, nb = m->h_levb_ptr.size() - 1;
  p->level.reserve(2 * nf + nb);   // the launches point into it
  auto add = [&](const void* fn, const int* rows, const std::vector<int>& ptr, size_t l,
                 SolveState* st, std::vector<tf_icc_launch>& to) {
    IccLevelArgs a = base;
    a.rows = rows + ptr[l];
    a.count = ptr[l + 1] - ptr[l];
    a.st = st;
    p->level.push_back(a);
    to.push_back({fn, std::max(1, (a.count + 255) / 256), 256, 0, {&p->level.back()}});
  };
  for (size_t l = 0; l < nf; ++l)
    add((const void*)k_icc_form_level, m->d_levf_rows, m->h_levf_ptr, l, nullptr, p->form);
  for (size_t l = 0; l < nf; ++l)
    add((const void*)k_icc_fwd_level, m->d_levf_rows, m->h_levf_ptr, l, m->d_state, p->apply);
  for (size_t l = 0; l < nb; ++l)
    add((const void*)k_icc_bwd_level, m->d_levb_rows, m->h_levb_ptr, l, m->d_state, p->apply);
  p->rho = {m->ni, m->d_z, m->d_r, m->d_part, m->d_state};
  p->apply.push_back({(const void*)k_icc_rho, m->vec_grid, 256, 0,
                      {&p->rho.ni, &p->rho.z, &p->rho.r, &p->rho.part, &p->rho.st}});
}

}  // namespace

// Where k_residual and k_update store r for the one-CTA sweeps.
IccResid tf_icc_resid(const tf_matrix_s* m) {
  IccResid r{};
  if (m->icc_packed > 0) {
    r.idx_f = m->icc_dir[0].idx;
    r.idx_b = m->icc_dir[1].idx;
    r.rec_f = reinterpret_cast<double*>(m->icc_dir[0].rec);
    r.rec_b = reinterpret_cast<double*>(m->icc_dir[1].rec);
  }
  return r;
}

// Entries padded to twice their number, and all that a row takes in both
// directions where every level, and so every slice, is one row.
size_t tf_icc_bytes(int n, int64_t nnz) {
  return (size_t)nnz * 32 + (size_t)n * 256 + ((size_t)1 << 16);
}

// Without room for the records (or with more entries than their 32-bit indices
// name) the matrix keeps one kernel per level, which needs none.
int tf_icc_prepare(tf_matrix_s* m) {
  if (m->icc_packed != 0 || !narrow_levels(m)) return TF_OK;
  int st = pack(m);
  m->icc_packed = st == TF_OK ? 1 : -1;
  if (st == TF_ERR_OOM) {
    tf_icc_free(m);
    cudaGetLastError();   // not to be found by the next launch
    st = TF_OK;
  }
  return st;
}

void tf_icc_free(tf_matrix_s* m) {
  for (auto& g : m->icc_dir) {
    for (void* q : {(void*)g.slice, (void*)g.chunk, (void*)g.src, (void*)g.idx, (void*)g.rec})
      tf_dev_free(m->ctx, q);
    g = tf_icc_dir_s();
  }
  m->icc_bytes = 0;
}

int tf_icc_kernels(const tf_matrix_s* m) {
  if (!m->icc_ready) return 0;
  const bool one = m->icc_packed > 0 || (m->icc_packed == 0 && narrow_levels(m));
  return one ? 1 : (int)(m->h_levf_ptr.size() + m->h_levb_ptr.size()) - 2 + 1;
}

int tf_icc_make_plan(tf_matrix_s* m, tf_icc_plan* p) {
  if (m->icc_packed <= 0) {
    plan_levels(m, p);
    return TF_OK;
  }
  IccArgs& a = p->one;
  a.row = m->d_row;
  a.col = m->d_col;
  a.val = m->d_val;
  a.adiag = m->d_adiag;
  a.ni = m->ni;
  a.d = m->d_icc_d;
  a.y = m->d_q;   // q is free between k_update and the next SpMV
  a.z = m->d_z;
  a.st = m->d_state;
  a.prm = m->d_params;
  a.f = dir_args(m->icc_dir[0], m->d_levf_rows);
  a.b = dir_args(m->icc_dir[1], m->d_levb_rows);
  a.width = m->icc_width;
  a.stages = m->icc_stages;
  a.ring = m->icc_ring;
  if (m->icc_batch == 3) return plan_one<3, 3, 24>(m, p);
  if (m->icc_warps == 24) return plan_one<4, 4, 24>(m, p);
  return plan_one<12, 4, 16>(m, p);
}
