// tf_vec.cu -- vector kernels for callers that run their own Krylov loop
// (the row-block solve of one system over several GPUs): the updates and
// partial sums of Native_Mod/Cg.f90 on device vectors, each expression
// rounded as the reference's loop rounds it, and deterministic sums (fixed
// grid, per-block partials combined in block order by the last block).
#include <cuda_runtime.h>

#include <algorithm>

#include "tf_internal.h"

namespace tf {

constexpr int kVecThreads = 256;

struct VecRed {
  double* part;        // kVecMaxBlocks * 2 partials
  unsigned* counter;
  double* out;
};

// The kernels walk the entries in pairs, kPairs pairs of every array loaded
// before the first is used.  Pair j is entries 2 j and 2 j + 1: one 16-byte
// access when every array allows it (VEC), two of 8 bytes otherwise -- the same
// entries in the same thread either way, so sums do not depend on alignment.
constexpr int kPairs = 4;

template <bool VEC>
__device__ __forceinline__ double2 get2(const double* x, int j) {
  if (VEC) return reinterpret_cast<const double2*>(x)[j];
  return make_double2(x[2 * j], x[2 * j + 1]);
}
template <bool VEC>
__device__ __forceinline__ void put2(double* x, int j, double2 v) {
  if (VEC) {
    reinterpret_cast<double2*>(x)[j] = v;
  } else {
    x[2 * j] = v.x;
    x[2 * j + 1] = v.y;
  }
}

// y = a x + b y (Cg.f90:166-170 p = z + beta p, :204-209 x + alfa p and
// r - alfa q); first: y = a x; a == 0: y = b y.
template <bool VEC>
__global__ void __launch_bounds__(kVecThreads) k_vec_axpby(int n, double a, const double* x,
                                                           double b, double* y, int first) {
  const int np = n >> 1, stride = gridDim.x * blockDim.x;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  auto one = [&](double xi, double yi) {
    if (first) return __dmul_rn(a, xi);
    if (a == 0.0) return __dmul_rn(b, yi);
    return __dadd_rn(__dmul_rn(a, xi), __dmul_rn(b, yi));
  };
  for (int j0 = t; j0 < np; j0 += kPairs * stride) {
    double2 xv[kPairs], yv[kPairs];
#pragma unroll
    for (int u = 0; u < kPairs; ++u) {
      const int j = j0 + u * stride;
      xv[u] = yv[u] = make_double2(0.0, 0.0);
      if (j < np) {
        if (first || a != 0.0) xv[u] = get2<VEC>(x, j);
        if (!first) yv[u] = get2<VEC>(y, j);
      }
    }
#pragma unroll
    for (int u = 0; u < kPairs; ++u) {
      const int j = j0 + u * stride;
      if (j < np) put2<VEC>(y, j, make_double2(one(xv[u].x, yv[u].x), one(xv[u].y, yv[u].y)));
    }
  }
  if ((n & 1) && t == 0) y[n - 1] = one(x[n - 1], first ? 0.0 : y[n - 1]);
}

__global__ void __launch_bounds__(kVecThreads) k_vec_gather(int n, const double* src,
                                                            const long long* idx, double* out) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = src[idx[i]];
}

__global__ void __launch_bounds__(kVecThreads) k_vec_scatter(int n, double* dst,
                                                             const long long* idx,
                                                             const double* vals) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) dst[idx[i]] = vals[i];
}

__global__ void __launch_bounds__(kVecThreads) k_vec_recip(int n, const double* x, double* out) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    out[i] = __ddiv_rn(1.0, x[i]);   // Prec_Form.f90:51 d_inv = 1.0 / d
}

// KIND 0: sum a_i b_i (b null: sum a_i); 1: sum r_i^2 / d_i^2
// (Normalized_Root_Mean_Square.f90:33-36); 2: z = r d_inv (Prec_Solve.f90:
// 44-49) and sum z_i r_i (Cg.f90:151-155); 3: min and max of x.
template <int KIND, bool VEC>
__global__ void __launch_bounds__(kVecThreads) k_vec_reduce(int n, const double* a,
                                                            const double* b, double* z,
                                                            VecRed red) {
  __shared__ double scratch[2 * (kVecThreads / 32)];
  double s0 = KIND == 3 ? red_identity<kMin>() : 0.0;
  double s1 = red_identity<kMax>();
  auto one = [&](double ai, double bi) -> double {   // returns z
    if (KIND == 0) s0 = __dadd_rn(s0, b ? __dmul_rn(ai, bi) : ai);
    if (KIND == 1) s0 = __dadd_rn(s0, nrms_term(ai, bi));
    if (KIND == 2) {
      const double zi = __dmul_rn(ai, bi);
      s0 = __dadd_rn(s0, __dmul_rn(zi, ai));
      return zi;
    }
    if (KIND == 3) {
      s0 = fmin(s0, ai);
      s1 = fmax(s1, ai);
    }
    return 0.0;
  };
  const int np = n >> 1, stride = gridDim.x * blockDim.x;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  for (int j0 = t; j0 < np; j0 += kPairs * stride) {
    double2 av[kPairs], bv[kPairs];
#pragma unroll
    for (int u = 0; u < kPairs; ++u) {
      const int j = j0 + u * stride;
      if (j < np) {
        av[u] = get2<VEC>(a, j);
        bv[u] = b ? get2<VEC>(b, j) : make_double2(0.0, 0.0);
      }
    }
#pragma unroll
    for (int u = 0; u < kPairs; ++u) {
      const int j = j0 + u * stride;
      if (j < np) {
        const double zx = one(av[u].x, bv[u].x), zy = one(av[u].y, bv[u].y);
        if (KIND == 2) put2<VEC>(z, j, make_double2(zx, zy));
      }
    }
  }
  if ((n & 1) && t == 0) {
    const double zi = one(a[n - 1], b ? b[n - 1] : 0.0);
    if (KIND == 2) z[n - 1] = zi;
  }
  if (KIND == 3) {
    double v[2] = {block_red<kMin>(s0, scratch), block_red<kMax>(s1, scratch)};
    const int ops[2] = {kMin, kMax};
    if (grid_reduce_last<2>(v, ops, red.part, red.counter, scratch) && threadIdx.x == 0) {
      red.out[0] = v[0];
      red.out[1] = v[1];
    }
  } else {
    double v[1] = {block_red<kSum>(s0, scratch)};
    const int ops[1] = {kSum};
    if (grid_reduce_last<1>(v, ops, red.part, red.counter, scratch) && threadIdx.x == 0)
      red.out[0] = v[0];
  }
}

}  // namespace tf

using namespace tf;

namespace {

constexpr int kVecMaxBlocks = 1024;

// Whether 16-byte accesses are allowed on all of the arrays (null: none).
bool pairs_aligned(const void* x, const void* y, const void* z = nullptr) {
  return (((uintptr_t)x | (uintptr_t)y | (uintptr_t)z) & 15) == 0;
}

int vec_grid(tf_ctx_s* c, int n, int per_sm = 8) {
  return std::max(1, std::min({(n + kVecThreads - 1) / kVecThreads, c->sm_count * per_sm,
                               kVecMaxBlocks}));
}

// The context's scratch for the sums (partials and a counter), on first use.
int vec_scratch(tf_ctx_s* c, VecRed* r, double* out) {
  if (!c->d_vec_scratch) {
    void* p = nullptr;
    const int st = tf_dev_alloc_bytes(c, &p, (2 * kVecMaxBlocks + 16) * sizeof(double));
    if (st != TF_OK) return st;
    c->d_vec_scratch = static_cast<double*>(p);
  }
  r->part = c->d_vec_scratch;
  r->counter = reinterpret_cast<unsigned*>(c->d_vec_scratch + 2 * kVecMaxBlocks);
  r->out = out;
  return TF_OK;
}

template <int KIND>
int vec_reduce(tf_ctx ctx, int n, const double* a, const double* b, double* z, double* out) {
  if (!ctx || n < 0 || !out || (n > 0 && !a) || (KIND >= 1 && KIND <= 2 && n > 0 && !b) ||
      (KIND == 2 && n > 0 && !z))
    return TF_ERR_ARG;
  TF_CUDA_TRY(cudaSetDevice(ctx->device));
  VecRed red;
  int st = vec_scratch(ctx, &red, out);
  if (st != TF_OK) return st;
  // A whole batch of pairs a thread where there is that much, on four CTAs an SM:
  // every CTA more is a partial sum and an atomic more for the last one to wait
  // for (2 M entries in L2, us with four / eight: dot 7.1 / 9.2, NRMS 8.3 / 10.4,
  // Jacobi 8.9 / 11.1, range 9.8 / 11.4; from HBM 10.3 / 11.8 to 11.4 / 13.2).
  const int grid = vec_grid(ctx, (n + 2 * kPairs - 1) / (2 * kPairs), 4);
  if (pairs_aligned(a, b, z))
    k_vec_reduce<KIND, true><<<grid, kVecThreads, 0, ctx->stream>>>(n, a, b, z, red);
  else
    k_vec_reduce<KIND, false><<<grid, kVecThreads, 0, ctx->stream>>>(n, a, b, z, red);
  TF_CUDA_TRY(cudaGetLastError());
  return TF_OK;
}

}  // namespace

extern "C" int tf_vec_axpby(tf_ctx ctx, int n, double a, const double* d_x, double b,
                            double* d_y, int first) {
  TF_API_BEGIN
  if (!ctx || n < 0 || (n > 0 && (!d_x || !d_y))) return TF_ERR_ARG;
  if (n == 0) return TF_OK;
  TF_CUDA_TRY(cudaSetDevice(ctx->device));
  const int grid = vec_grid(ctx, (n + 2 * kPairs - 1) / (2 * kPairs));
  if (pairs_aligned(d_x, d_y))
    k_vec_axpby<true><<<grid, kVecThreads, 0, ctx->stream>>>(n, a, d_x, b, d_y, first);
  else
    k_vec_axpby<false><<<grid, kVecThreads, 0, ctx->stream>>>(n, a, d_x, b, d_y, first);
  TF_CUDA_TRY(cudaGetLastError());
  return TF_OK;
  TF_API_END
}

extern "C" int tf_vec_gather(tf_ctx ctx, int n, const double* d_src, const int64_t* d_idx,
                             double* d_out) {
  TF_API_BEGIN
  if (!ctx || n < 0 || (n > 0 && (!d_src || !d_idx || !d_out))) return TF_ERR_ARG;
  if (n == 0) return TF_OK;
  TF_CUDA_TRY(cudaSetDevice(ctx->device));
  k_vec_gather<<<vec_grid(ctx, n), kVecThreads, 0, ctx->stream>>>(
      n, d_src, reinterpret_cast<const long long*>(d_idx), d_out);
  TF_CUDA_TRY(cudaGetLastError());
  return TF_OK;
  TF_API_END
}

extern "C" int tf_vec_scatter(tf_ctx ctx, int n, double* d_dst, const int64_t* d_idx,
                              const double* d_vals) {
  TF_API_BEGIN
  if (!ctx || n < 0 || (n > 0 && (!d_dst || !d_idx || !d_vals))) return TF_ERR_ARG;
  if (n == 0) return TF_OK;
  TF_CUDA_TRY(cudaSetDevice(ctx->device));
  k_vec_scatter<<<vec_grid(ctx, n), kVecThreads, 0, ctx->stream>>>(
      n, d_dst, reinterpret_cast<const long long*>(d_idx), d_vals);
  TF_CUDA_TRY(cudaGetLastError());
  return TF_OK;
  TF_API_END
}

extern "C" int tf_vec_recip(tf_ctx ctx, int n, const double* d_x, double* d_out) {
  TF_API_BEGIN
  if (!ctx || n < 0 || (n > 0 && (!d_x || !d_out))) return TF_ERR_ARG;
  if (n == 0) return TF_OK;
  TF_CUDA_TRY(cudaSetDevice(ctx->device));
  k_vec_recip<<<vec_grid(ctx, n), kVecThreads, 0, ctx->stream>>>(n, d_x, d_out);
  TF_CUDA_TRY(cudaGetLastError());
  return TF_OK;
  TF_API_END
}

extern "C" int tf_vec_dot(tf_ctx ctx, int n, const double* d_a, const double* d_b,
                          double* d_out) {
  TF_API_BEGIN
  return vec_reduce<0>(ctx, n, d_a, d_b, nullptr, d_out);
  TF_API_END
}

extern "C" int tf_vec_nrms_sum(tf_ctx ctx, int n, const double* d_r, const double* d_diag,
                               double* d_out) {
  TF_API_BEGIN
  return vec_reduce<1>(ctx, n, d_r, d_diag, nullptr, d_out);
  TF_API_END
}

extern "C" int tf_vec_jacobi(tf_ctx ctx, int n, const double* d_r, const double* d_dinv,
                             double* d_z, double* d_out) {
  TF_API_BEGIN
  return vec_reduce<2>(ctx, n, d_r, d_dinv, d_z, d_out);
  TF_API_END
}

extern "C" int tf_vec_minmax(tf_ctx ctx, int n, const double* d_x, double* d_out2) {
  TF_API_BEGIN
  return vec_reduce<3>(ctx, n, d_x, nullptr, nullptr, d_out2);
  TF_API_END
}
