// tf_resident.cu -- the FP64 Cg / Bicg solve (Jacobi or no preconditioning)
// of a matrix that fits the chip, as one cooperative kernel.
//
// A solve by a graph of kernels reads the matrix from L2 every iteration and
// pays three kernel boundaries and a WHILE node for it: 20 us an iteration on
// 27,000 rows, nearly all of it latency.  Here every CTA owns a run of
// consecutive rows for the whole solve: their values, column slots and p stay
// in its shared memory, x, r, q and the diagonal in its registers, and an
// iteration is two exchanges between the CTAs:
//
//   p = z + beta p      own rows, and the rows of other CTAs its own rows
//                       refer to (its halo: their z is read, their p is kept
//                       up to date here with the owner's arithmetic)
//   q = A p, p.q        from shared memory only
//   -- exchange 1: p.q -> alfa
//   x += alfa p, r -= alfa q, z = M^-1 r (stored for the neighbours), NRMS, rho
//   -- exchange 2: NRMS, rho [, range of x] -> convergence, beta
//
// Everything is rounded as the other kernels (and the reference's loops)
// round it: row sums in storage order, products and sums separately; only
// the order of the grid-wide sums differs.
//
// An exchange: each CTA stores its partial sums as words that carry the
// exchange's number in their low half and polls the words of all CTAs; each
// CTA then adds them in the same order, so all hold the same bits.  One store
// and one polled load instead of an atomic counter, a flag and the sums.  The
// neighbours' z travel in such words too: they need no fence (a fence before
// a flag cost 1850 cycles an iteration) and are polled while exchange 2 is
// under way.
#include <cuda_runtime.h>
#include <stdlib.h>

#include <algorithm>
#include <type_traits>

#include "tf_internal.h"

namespace tf {

// What one CTA owns.
struct ResCta {
  int r0, r1;       // rows
  int h0, nh;       // its halo: entries [h0, h0 + nh) of the halo list
};

struct ResArgs {
  int n;
  const int* row;
  const int* dia;
  double* val;
  double* x;
  double* b;
  unsigned long long* z;         // M^-1 r between the CTAs: two tagged words a row
  const ResCta* cta;
  const int* halo;               // rows
  const unsigned short* slot;    // per entry: place of its column in p
  unsigned long long* words;     // [2][CTAs][kResWords]
  unsigned* epoch;               // number of the last exchange on these words
  SolveState* st;
  unsigned skip;                 // numbers left to solves before it that may have given up
  double tol, norm;
  int miter, hist_cap;
  double* hist;
  unsigned long long wait_ns;
  int write_val;                 // store val back (the last solve on it)
  int cap_ne, cap_p, cap_halo;   // shared-memory capacities
};

constexpr int kResAhead = 4;              // halo entries a thread polls for during an exchange
constexpr int kResVals = 4;               // values of an exchange at most
constexpr int kResWords = 16;             // 128 bytes a CTA: a line of its own

__device__ __forceinline__ void res_store(unsigned long long* w, double v, unsigned tag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const unsigned long long hi = (b & 0xffffffff00000000ull) | tag, lo = (b << 32) | tag;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w), "l"(hi), "l"(lo)
               : "memory");
}
__device__ __forceinline__ bool res_load(const unsigned long long* w, double& v, unsigned tag) {
  unsigned long long hi, lo;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(hi), "=l"(lo) : "l"(w)
               : "memory");
  if ((unsigned)hi != tag || (unsigned)lo != tag) return false;
  v = __longlong_as_double((long long)((hi & 0xffffffff00000000ull) | (lo >> 32)));
  return true;
}

template <int T>
struct ResShared {
  double warp[kResVals][T / 32];
  double all[kResVals][8];       // per polling warp (at most 256 CTAs)
};

// One exchange of NV values (sums but for the last two of four: minimum and
// maximum): v = this thread's parts, on return the grid's.  meanwhile(): what
// every thread polls for on its own, true once it has it.  False, for the
// whole CTA, when a partner did not come within the limit since the exchange
// before.
template <int NV, int T, class F>
__device__ __forceinline__ bool res_exchange(const ResArgs& a, double (&v)[NV], unsigned& tag,
                                             ResShared<T>& sh, Deadline& deadline,
                                             F&& meanwhile) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = gridDim.x;
  ++tag;
  unsigned long long* words = a.words + (size_t)(tag & 1u) * G * kResWords;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    if (NV == 4 && q == 2) v[q] = warp_min(v[q]);
    else if (NV == 4 && q == 3) v[q] = warp_max(v[q]);
    else v[q] = warp_sum(v[q]);
    if (lane == 0) sh.warp[q][warp] = v[q];
  }
  __syncthreads();
  bool fail = deadline.passed();
  // Waits for one poll, giving up at the deadline or once another CTA has.
  auto until = [&](auto&& poll) {
    for (int spin = 0; !fail && !poll(); ++spin)
      if ((spin & 63) == 63)
        fail = deadline.passed() || *(volatile int*)&a.st->status != 0;
  };
  const int pollers = (G + 31) / 32;
  if (warp < pollers) {
    if (warp == 0) {
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        const int op = NV == 4 && q == 2 ? kMin : NV == 4 && q == 3 ? kMax : kSum;
        double w = op == kSum ? 0.0 : op == kMin ? red_identity<kMin>() : red_identity<kMax>();
        if (lane < T / 32) w = sh.warp[q][lane];
        v[q] = op == kSum ? warp_sum(w) : op == kMin ? warp_min(w) : warp_max(w);
        if (lane == 0) res_store(words + blockIdx.x * kResWords + 2 * q, v[q], tag);
      }
    }
    const int c = threadIdx.x;
#pragma unroll
    for (int q = 0; q < NV; ++q)
      v[q] = NV == 4 && q == 2 ? red_identity<kMin>()
             : NV == 4 && q == 3 ? red_identity<kMax>() : 0.0;
    if (c < G) {
      const unsigned long long* w = words + (size_t)c * kResWords;
      until([&]() {
        bool here = true;
#pragma unroll
        for (int q = 0; q < NV; ++q) here = res_load(w + 2 * q, v[q], tag) && here;
        return here;
      });
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      if (NV == 4 && q == 2) v[q] = warp_min(v[q]);
      else if (NV == 4 && q == 3) v[q] = warp_max(v[q]);
      else v[q] = warp_sum(v[q]);
      if (lane == 0) sh.all[q][warp] = v[q];
    }
  }
  until(meanwhile);
  if (__syncthreads_or(fail)) {
    if (threadIdx.x == 0) atomicExch(&a.st->status, (int)TF_ERR_TIMEOUT);
    return false;
  }
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    double r = sh.all[q][0];
    for (int w = 1; w < pollers; ++w) {
      if (NV == 4 && q == 2) r = fmin(r, sh.all[q][w]);
      else if (NV == 4 && q == 3) r = fmax(r, sh.all[q][w]);
      else r = __dadd_rn(r, sh.all[q][w]);
    }
    v[q] = r;
  }
  deadline.renew();
  return true;
}

// RPT rows a thread (row r0 + t + u T).  What bounds it: the two exchanges
// (1 to 2 us each: a store to L2 and the polls that see it) up to some
// 100,000 rows, then the shared-memory loads of the row sums.  Measured, us an
// iteration, the graph of kernels / this one: 1,000 rows 16.8 / 3.4, 27,000
// (30^3) 20.6 / 5.4, 130,000 21.9 / 6.5, 300,000 25.6 / 10.7, 21,000
// polyhedral cells 19.2 / 5.9; a solve's fixed part 105 / 70 us.
template <int PREC, bool NORM, int RPT, int T>
__global__ void __launch_bounds__(T, 1) k_resident(ResArgs a) {
  extern __shared__ __align__(16) unsigned char tf_res_smem[];
  __shared__ ResShared<T> sh;
  double* sval = reinterpret_cast<double*>(tf_res_smem);
  double* sp = sval + a.cap_ne;
  int* shalo = reinterpret_cast<int*>(sp + a.cap_p);
  unsigned short* sslot = reinterpret_cast<unsigned short*>(shalo + a.cap_halo);
  unsigned short* srow = sslot + a.cap_ne;
  const int t = threadIdx.x;
  const ResCta me = a.cta[blockIdx.x];
  const int r0 = me.r0, nr = me.r1 - me.r0, j0 = a.row[r0], ne = a.row[me.r1] - j0, nh = me.nh;
  SolveState* st = a.st;
  unsigned tag = *a.epoch + a.skip;
  Deadline deadline(a.wait_ns ? a.wait_ns : kWaitLimitNs);

  double xi[RPT], ri[RPT], ai[RPT], inv[RPT], qi[RPT];
  double s = 0.0;
#pragma unroll
  for (int u = 0; u < RPT; ++u) {
    const int l = t + u * T;
    ai[u] = 1.0;
    xi[u] = ri[u] = qi[u] = 0.0;
    if (l < nr) {
      ai[u] = a.val[a.dia[r0 + l]];
      xi[u] = a.x[r0 + l];
      ri[u] = a.b[r0 + l];   // b until the first residual
      s = __dadd_rn(s, ai[u]);
    }
  }
  for (int e = t; e < ne; e += T) {
    sval[e] = a.val[j0 + e];
    sslot[e] = a.slot[j0 + e];
  }
  for (int l = t; l <= nr; l += T) srow[l] = (unsigned short)(a.row[r0 + l] - j0);
  for (int h = t; h < nh; h += T) shalo[h] = a.halo[me.h0 + h];

  auto nothing = []() { return true; };
  // Normalisation (Cg.f90:62-84) and NRMS(b) (:95-104)
  double v1[1] = {s};
  if (!res_exchange<1, T>(a, v1, tag, sh, deadline, nothing)) return;
  const double fn = __ddiv_rn(1.0, __ddiv_rn(v1[0], (double)a.n));
  for (int e = t; e < ne; e += T) sval[e] = __dmul_rn(sval[e], fn);
  double v[NORM ? 2 : 4];
  // z of the halo entries t + u T, u < kResAhead, of the exchange under way.
  double zh[kResAhead];
  auto take = [&](int h, double& z, unsigned of) {
    return res_load(a.z + 2 * (size_t)shalo[h], z, of);
  };
  auto halo = [&]() {   // polls for the first alone, to spare L2
    if (t < nh && !take(t, zh[0], tag)) return false;
    bool here = true;
#pragma unroll
    for (int u = 1; u < kResAhead; ++u)
      if (t + u * T < nh) here = take(t + u * T, zh[u], tag) && here;
    return here;
  };
  auto reset = [&]() {
    v[0] = v[1] = 0.0;
    if constexpr (!NORM) {
      v[2] = kHuge;
      v[3] = -kHuge;
    }
  };
  auto range = [&](double x) {   // Fortran min / max (see tf_fp64.cu)
    if constexpr (!NORM) {
      v[2] = (x < v[2]) ? x : v[2];
      v[3] = (x > v[3]) ? x : v[3];
    }
  };
  auto finish = [&]() {
    if constexpr (NORM) return nrms_finish(v[0], 1, a.norm, 0.0, 0.0);
    else return nrms_finish(v[0], 0, 0.0, v[2], v[3]);
  };
  reset();
#pragma unroll
  for (int u = 0; u < RPT; ++u)
    if (t + u * T < nr) {
      ai[u] = __dmul_rn(ai[u], fn);
      ri[u] = __dmul_rn(ri[u], fn);
      inv[u] = __drcp_rn(ai[u]);
      v[0] = __dadd_rn(v[0], nrms_term(ri[u], ai[u]));
      range(xi[u]);
    }
  if (!res_exchange<NORM ? 2 : 4, T>(a, v, tag, sh, deadline, nothing)) return;
  const double bnrm2 = finish();
  double res = 0.0;
  int niter = 0;
  bool go = !(bnrm2 < a.tol);   // Cg.f90:101-104: iter = 0, res stays 0.0

  // Sum over row l of the entries with p, added to (SUB: subtracted from)
  // acc, eight entries' loads in flight.
  auto row_sum = [&](double acc, int l, auto SUB) {
    const int js = srow[l], je = srow[l + 1];
    for (int e = js; e < je; e += 8) {
      double pv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) pv[u] = e + u < je ? sp[sslot[e + u]] : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (e + u < je) {
          const double m = __dmul_rn(sval[e + u], pv[u]);
          acc = decltype(SUB)::value ? __dsub_rn(acc, m) : __dadd_rn(acc, m);
        }
    }
    return acc;
  };
  auto precond = [&](int u) { return PREC == kPrecJacobi ? __dmul_rn(ri[u], inv[u]) : ri[u]; };

  double rho = 0.0, rho_old = 0.0;
  if (go) {   // r = b - A x, NRMS(r), rho (Cg.f90:109-123, :150-156)
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (t + u * T < nr) sp[t + u * T] = xi[u];
    for (int h = t; h < nh; h += T) sp[nr + h] = a.x[shalo[h]];
    __syncthreads();
    const double xlo = NORM ? 0.0 : v[NORM ? 0 : 2], xhi = NORM ? 0.0 : v[NORM ? 0 : 3];
    reset();
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (t + u * T < nr) {
        ri[u] = row_sum(ri[u], t + u * T, std::true_type{});
        const double zi = precond(u);
        res_store(a.z + 2 * (size_t)(r0 + t + u * T), zi, tag + 1);
        v[0] = __dadd_rn(v[0], nrms_term(ri[u], ai[u]));
        v[1] = __dadd_rn(v[1], __dmul_rn(zi, ri[u]));
      }
    if constexpr (!NORM) {   // the range of x has not changed
      v[2] = xlo;
      v[3] = xhi;
    }
    if (!res_exchange<NORM ? 2 : 4, T>(a, v, tag, sh, deadline, halo)) return;
    res = finish();
    rho = v[1];
    if (blockIdx.x == 0 && t == 0 && a.hist && a.hist_cap > 0) a.hist[0] = res;
    go = !(res < a.tol) && a.miter >= 1;   // Cg.f90:120-123, or a zero-trip loop
  }
  const bool moved = go;
  for (int k = 1; go; ++k) {
    const bool first = k == 1;
    const double beta = first ? 0.0 : __ddiv_rn(rho, rho_old);
    auto direction = [&](double z, double p) {   // Cg.f90:158-171
      return first ? z : __dadd_rn(z, __dmul_rn(beta, p));
    };
#pragma unroll
    for (int u = 0; u < kResAhead; ++u) {
      const int h = t + u * T;
      if (h < nh) sp[nr + h] = direction(zh[u], sp[nr + h]);
    }
    // The rest of a large halo: exchange 2 has seen every CTA's sums, which
    // were sent after its z, so a few polls at most.  A thread that gives up
    // here goes on without its z to exchange 1, which then fails.
    for (int h = t + kResAhead * T; h < nh; h += T) {
      double z = 0.0;
      bool gone = false;
      for (int spin = 0; !take(h, z, tag) && !gone; ++spin)
        if ((spin & 63) == 63) gone = deadline.passed();
      if (gone) deadline.give_up();
      sp[nr + h] = direction(z, sp[nr + h]);
    }
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (t + u * T < nr) sp[t + u * T] = direction(precond(u), sp[t + u * T]);
    __syncthreads();
    v1[0] = 0.0;
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (t + u * T < nr) {   // Cg.f90:176-195
        qi[u] = row_sum(0.0, t + u * T, std::false_type{});
        v1[0] = __dadd_rn(v1[0], __dmul_rn(sp[t + u * T], qi[u]));
      }
    if (!res_exchange<1, T>(a, v1, tag, sh, deadline, nothing)) return;
    const double alpha = __ddiv_rn(rho, v1[0]);
    reset();
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (t + u * T < nr) {   // Cg.f90:204-209, :150-156
        xi[u] = __dadd_rn(xi[u], __dmul_rn(alpha, sp[t + u * T]));
        range(xi[u]);
        ri[u] = __dsub_rn(ri[u], __dmul_rn(alpha, qi[u]));
        const double zi = precond(u);
        res_store(a.z + 2 * (size_t)(r0 + t + u * T), zi, tag + 1);
        v[1] = __dadd_rn(v[1], __dmul_rn(zi, ri[u]));
      }
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (t + u * T < nr) v[0] = __dadd_rn(v[0], nrms_term(ri[u], ai[u]));
    if (!res_exchange<NORM ? 2 : 4, T>(a, v, tag, sh, deadline, halo)) return;
    res = finish();
    rho_old = rho;
    rho = v[1];
    if (blockIdx.x == 0 && t == 0 && a.hist && k < a.hist_cap) a.hist[k] = res;
    niter = k;
    if (res < a.tol || k >= a.miter) go = false;   // Cg.f90:220
  }

  // De-normalisation (Cg.f90:245-250)
  if (moved) {
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (t + u * T < nr) a.x[r0 + t + u * T] = xi[u];
  }
  if (a.write_val)
    for (int e = t; e < ne; e += T) a.val[j0 + e] = __ddiv_rn(sval[e], fn);
  for (int i = r0 + t; i < me.r1; i += T) a.b[i] = __ddiv_rn(__dmul_rn(a.b[i], fn), fn);
  if (blockIdx.x == 0 && t == 0) {
    *a.epoch = tag;
    st->niter = niter;
    st->res = res;
    st->bnrm2 = bnrm2;
    st->done = 1;
  }
}

// Halo and entry places of one CTA's rows, one CTA each: a bitmap of the
// columns outside its rows, and their ranks in it as places behind its own.
// The halo is in ascending order (its z is read coalesced where the matrix
// allows it).  cta[c].nh > cap: more than the list holds.
__global__ void __launch_bounds__(512) k_resident_build(const int* row, const int* col, int n,
                                                        int rows, int cap, ResCta* cta,
                                                        int* halo, unsigned short* slot,
                                                        int* largest) {
  extern __shared__ unsigned tf_res_bits[];
  __shared__ int warp_sh[16];
  const int c = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int r0 = c * rows, r1 = min(n, r0 + rows), nr = r1 - r0;
  const int j0 = row[r0], j1 = row[r1], nw = (n + 31) / 32;
  unsigned* bits = tf_res_bits;
  int* rank = reinterpret_cast<int*>(bits + nw);
  for (int w = t; w < nw; w += 512) bits[w] = 0u;
  __syncthreads();
  for (int j = j0 + t; j < j1; j += 512) {
    const int k = col[j];
    if (k < r0 || k >= r1) atomicOr(bits + (k >> 5), 1u << (k & 31));
  }
  __syncthreads();
  // Exclusive ranks of the words; a thread takes a run of them.
  const int per = (nw + 511) / 512, w0 = min(nw, t * per), w1 = min(nw, w0 + per);
  int mine = 0;
  for (int w = w0; w < w1; ++w) mine += __popc(bits[w]);
  int inc = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) warp_sh[warp] = inc;
  __syncthreads();
  int base = inc - mine;
  for (int w = 0; w < warp; ++w) base += warp_sh[w];
  for (int w = w0; w < w1; ++w) {
    rank[w] = base;
    unsigned b = bits[w];
    while (b) {
      if (halo) halo[(size_t)c * cap + base] = 32 * w + __ffs(b) - 1;
      b &= b - 1;
      ++base;
    }
  }
  if (t == 511) {
    if (halo) cta[c] = ResCta{r0, r1, c * cap, base};
    else atomicMax(largest, base);
  }
  if (!halo) return;
  __syncthreads();
  for (int j = j0 + t; j < j1; j += 512) {
    const int k = col[j], w = k >> 5;
    slot[j] = (unsigned short)(k >= r0 && k < r1
                                   ? k - r0
                                   : nr + rank[w] + __popc(bits[w] & ((1u << (k & 31)) - 1u)));
  }
}

}  // namespace tf

using namespace tf;

namespace {

struct ResShape {
  int rpt, threads;
};
constexpr ResShape kResShapes[] = {{1, 256}, {1, 512}, {2, 512}, {3, 768}};
constexpr int kResShapeCount = 4;

template <int PREC, bool NORM>
const void* res_kernel(int shape) {
  if (shape == 0) return (const void*)k_resident<PREC, NORM, 1, 256>;
  if (shape == 1) return (const void*)k_resident<PREC, NORM, 1, 512>;
  if (shape == 2) return (const void*)k_resident<PREC, NORM, 2, 512>;
  return (const void*)k_resident<PREC, NORM, 3, 768>;
}
const void* res_kernel(int prec, bool norm, int shape) {
  if (prec == kPrecJacobi)
    return norm ? res_kernel<kPrecJacobi, true>(shape) : res_kernel<kPrecJacobi, false>(shape);
  return norm ? res_kernel<kPrecNone, true>(shape) : res_kernel<kPrecNone, false>(shape);
}

size_t res_smem(int ne, int p, int halo, int rows) {
  return (size_t)ne * 8 + (size_t)p * 8 + (size_t)halo * 4 + (size_t)ne * 2 +
         ((size_t)rows + 1) * 2 + 16;
}
// k_resident_build's shared memory: a bit a row, and the words' ranks.
size_t res_bits(int n) { return (size_t)((n + 31) / 32) * 8; }
constexpr size_t kResEpochBytes = 128;
constexpr size_t kResSmemMax = 225 * 1024 - 2048;   // beside the exchange's static part

}  // namespace

namespace {

// Rows a CTA, the kernel's shape and the most entries of a CTA of a matrix that
// may fit the chip; rows = 0: it does not.  row: row pointers, from any base
// (null: entries are not looked at).
struct ResPlan {
  int rows = 0, shape = 0, cap_ne = 0;
};
ResPlan res_plan(int n, const int* row, int sms) {
  ResPlan p;
  if (n < 1 || res_bits(n) > kResSmemMax) return p;
  // Rows a CTA: 256 (one a thread) while there are SMs for that many CTAs,
  // then as many as it takes (512 at the least: us an iteration at 27,000
  // rows 5.44 / 5.56 / 5.94 with 256 / 512 / 1024 rows a CTA).
  int rows = 256;
  if ((n + rows - 1) / rows > sms) rows = std::max(512, (n + sms - 1) / sms);
  while (p.shape < kResShapeCount && kResShapes[p.shape].rpt * kResShapes[p.shape].threads < rows)
    ++p.shape;
  if (p.shape == kResShapeCount) return p;
  for (int r0 = 0; row && r0 < n; r0 += rows)
    p.cap_ne = std::max(p.cap_ne, row[std::min(n, r0 + rows)] - row[r0]);
  if (p.cap_ne > 65535 || res_smem(p.cap_ne, rows, 0, rows) > kResSmemMax) return p;
  p.cap_ne = (p.cap_ne + 7) & ~7;   // keeps what follows aligned
  p.rows = rows;
  return p;
}

// The layout's one allocation: words (sums, epoch, z), CTAs, halos, places.
struct ResBytes {
  size_t words, fixed, ctas, halo, slot;
  ResBytes(int n, int64_t nnz, int G, int largest) {
    auto up = [](size_t b) { return (b + 127) & ~size_t(127); };
    words = (size_t)2 * G * kResWords * 8;
    fixed = up(words + kResEpochBytes + (size_t)n * 16);
    ctas = up(G * sizeof(ResCta));
    halo = up((size_t)G * largest * 4 + 16);
    slot = up((size_t)nnz * 2);
  }
  size_t total() const { return fixed + ctas + halo + slot; }
};

}  // namespace

namespace {

// The CTAs' halos and the entries' places in p, made on the device from the
// matrix's row and column arrays; m->res.ctas stays 0 when they do not fit.
int res_build(tf_matrix_s* m, const ResPlan& p) {
  const int n = m->ni, sms = m->ctx->sm_count, rows = p.rows, shape = p.shape;
  const int G = (n + rows - 1) / rows, cap_ne = p.cap_ne;
  const size_t bits = res_bits(n);
  cudaStream_t s = m->ctx->stream;
  TF_CUDA_TRY(cudaFuncSetAttribute(k_resident_build, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kResSmemMax));
  int* d_largest = reinterpret_cast<int*>(m->d_part);   // free between kernels
  int largest = 0;
  TF_CUDA_TRY(cudaMemsetAsync(d_largest, 0, sizeof(int), s));
  k_resident_build<<<G, 512, bits, s>>>(m->d_row, m->d_col, n, rows, 0, nullptr, nullptr, nullptr,
                                        d_largest);
  TF_CUDA_TRY(cudaGetLastError());
  TF_CUDA_TRY(cudaMemcpyAsync(&largest, d_largest, sizeof largest, cudaMemcpyDeviceToHost, s));
  TF_CUDA_TRY(cudaStreamSynchronize(s));
  const int cap_p = rows + largest, cap_halo = (largest + 1) & ~1;
  const size_t smem = res_smem(cap_ne, cap_p, cap_halo, rows);
  if (smem > kResSmemMax || cap_p > 65535) return TF_OK;
  for (int prec : {kPrecJacobi, kPrecNone})
    for (bool norm : {false, true}) {
      const void* f = res_kernel(prec, norm, shape);
      TF_CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kResSmemMax));
      int per_sm = 0;
      TF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &per_sm, f, kResShapes[shape].threads, smem));
      if (per_sm * sms < G) return TF_OK;   // all CTAs have to be resident at once
    }
  const ResBytes bytes(n, m->nnz, G, largest);
  if (m->extra_bytes + bytes.total() > m->extra_limit) return TF_OK;
  unsigned char* d = nullptr;
  const int st = tf_dev_alloc_bytes(m->ctx, (void**)&d, bytes.total());
  if (st != TF_OK) return st;
  m->extra_bytes += bytes.total();
  m->res.block = d;
  m->res.words = reinterpret_cast<unsigned long long*>(d);
  m->res.epoch = reinterpret_cast<unsigned*>(d + bytes.words);
  m->res.z = reinterpret_cast<unsigned long long*>(d + bytes.words + kResEpochBytes);
  m->res.words_bytes = bytes.fixed;
  m->res.cta = d + bytes.fixed;
  m->res.halo = reinterpret_cast<int*>(d + bytes.fixed + bytes.ctas);
  m->res.slot = reinterpret_cast<unsigned short*>(d + bytes.fixed + bytes.ctas + bytes.halo);
  k_resident_build<<<G, 512, bits, s>>>(m->d_row, m->d_col, n, rows, largest,
                                        reinterpret_cast<ResCta*>(m->res.cta), m->res.halo,
                                        m->res.slot, nullptr);
  TF_CUDA_TRY(cudaGetLastError());
  m->res.shape = shape;
  m->res.threads = kResShapes[shape].threads;
  m->res.smem = smem;
  m->res.cap_ne = cap_ne;
  m->res.cap_p = cap_p;
  m->res.cap_halo = cap_halo;
  m->res.ctas = G;
  return TF_OK;
}

}  // namespace

// At registration, where the matrix may be solved by one kernel (row0: its row
// pointers on the host).  Without room for the layout the graph of kernels, which
// has its memory, solves the matrix.  (Made by the first solve instead, solves of
// 27,000 rows took 1 to 2 % longer on the later allocation.  TF_NO_RESIDENT keeps
// the graph, for comparisons; buffer cells are rows that no CTA would own.)
int tf_resident_prepare(tf_matrix_s* m, const int* row0) {
  if (m->nt != m->ni || getenv("TF_NO_RESIDENT")) return TF_OK;
  const ResPlan p = res_plan(m->ni, row0, m->ctx->sm_count);
  if (p.rows == 0) return TF_OK;
  int st = res_build(m, p);
  if (st == TF_ERR_OOM) {
    cudaGetLastError();   // not to be found by the next launch
    st = TF_OK;
  }
  return st;
}

// Device bytes the layout may take, for budgeting.  A CTA's halo has no more
// rows than it has entries, or than fit its shared memory (a renumbered
// matrix's entries a CTA are not known here).
size_t tf_resident_bytes(int n, int64_t nnz, const int* row, bool renumbered, int sms) {
  const ResPlan p = res_plan(n, renumbered ? nullptr : row, sms);
  if (p.rows == 0) return 0;
  const int fits = (int)(kResSmemMax / 12);
  return ResBytes(n, nnz, (n + p.rows - 1) / p.rows, renumbered ? fits : std::min(p.cap_ne, fits))
      .total();
}

bool tf_resident(const tf_matrix_s* m) {
  static const bool off = getenv("TF_NO_GRAPH") != nullptr;   // direct launches asked for
  return m->res.ctas > 0 && !off;
}

// One solve on val, x, b (device) with the parameters in *p, on m's stream;
// the state goes to *st.  queued: solves with the same parameters launched before
// it that the host has not waited for: one that gave up leaves words with numbers
// past the recorded one behind, so each leaves as many unused as it may take.
// write_val: val is scaled back into place.
int tf_resident_run(tf_matrix_s* m, int prec, const SolveParams* p, double* x, double* b,
                    SolveState* st, int queued, int write_val) {
  ResArgs a{};
  a.n = m->ni;
  a.row = m->d_row;
  a.dia = m->d_dia;
  a.val = m->d_val;
  a.x = x;
  a.b = b;
  a.z = m->res.z;
  a.cta = reinterpret_cast<const ResCta*>(m->res.cta);
  a.halo = m->res.halo;
  a.slot = m->res.slot;
  a.words = m->res.words;
  a.st = st;
  a.skip = (unsigned)queued * (2u * (unsigned)std::max(0, std::min(p->miter, 1 << 28)) + 8u);
  a.tol = p->tol;
  a.norm = p->norm;
  a.miter = p->miter;
  a.hist = p->hist;
  a.hist_cap = p->hist_cap;
  a.wait_ns = p->wait_ns;
  a.write_val = write_val;
  a.cap_ne = m->res.cap_ne;
  a.cap_p = m->res.cap_p;
  a.cap_halo = m->res.cap_halo;
  a.epoch = m->res.epoch;
  void* args[] = {&a};
  TF_CUDA_TRY(cudaLaunchCooperativeKernel(res_kernel(prec, p->has_norm != 0, m->res.shape),
                                          dim3(m->res.ctas), dim3(m->res.threads), args,
                                          m->res.smem, m->ctx->stream));
  return TF_OK;
}

// After a solve that gave up: the words of unfinished exchanges, and the recorded
// status, which a resident solve polls but does not clear.  Waited for: the
// matrix's next solve may run on another context's stream (tf_pool.cu).
int tf_resident_reset(tf_matrix_s* m) {
  cudaStream_t s = m->ctx->stream;
  if (m->res.ctas) TF_CUDA_TRY(cudaMemsetAsync(m->res.words, 0, m->res.words_bytes, s));
  TF_CUDA_TRY(cudaMemsetAsync(&m->d_state->status, 0, sizeof(int), s));
  for (auto* c : m->slices)
    if (c) TF_CUDA_TRY(cudaMemsetAsync(&c->d_state->status, 0, sizeof(int), s));
  TF_CUDA_TRY(cudaStreamSynchronize(s));
  return TF_OK;
}
