// Lanczos on the two-site effective Hamiltonian, every vector operation on the device.
//
// The reference leaves the eigensolver to its callers and gives them the BSDT vector
// primitives: Dot / Norm / Normalize / ScaleByFactor / LinearCombine on the raw buffer
// (framework/hp_numeric/blas_level1.h, complex forms :381-1080;
// tensor_manipulation/ten_linear_combine.h:186-459;
// qltensor/blk_spar_data_ten/raw_data_operations.h:225-272). Lanczos vectors all share ψ's
// block topology, so here they are plain raw buffers (FP64, or complex128 interleaved) and the
// primitives act on them directly.
//
// Step j (v_0 = ψ0 / ||ψ0||, V = [v_0 .. v_j] kept on the device):
//   w = H v_j                                   (the matvec's four contractions)
//   two passes of classical Gram-Schmidt:       c = Vᴴ w;  w -= V c;  α_j += Re c_j
//   β_{j+1} = ||w||;  v_{j+1} = w / β_{j+1}
// Full reorthogonalisation replaces the three-term recurrence (the projection on v_{j-1} is
// β_j). For a Hermitian H, α and β are real; complex dots are <x, y> = Σ conj(x) y, the
// reference's complex Dot. All of it is FP64 with deterministic reductions (fixed per-CTA
// partials summed in a fixed order), and α, β never leave the device until the caller asks
// for them. Each step is one CUDA graph (the matvec's kernels plus the vector kernels), built
// on first use.
#include <cmath>
#include <memory>
#include <type_traits>

#include "matvec.h"

using namespace qltg;

namespace {

constexpr int kVecThreads = 256;
constexpr int kVecWarps = kVecThreads / 32;
// fixed grid, deliberately independent of the device's SM count: the partial-sum order, and
// so every α and β, is the same on every run and every GPU (304 CTAs = two per SM on a
// 152-SM GB300; every CTA's sums cost it about 150 FP64 instructions, so not more)
constexpr int kVecBlocks = 304;
constexpr int kGroup = 8;   // sums formed at once: 8 real or 4 complex dots

// Scalar algebra of the two vector kinds: real FP64 (double) and complex128 (double2).
struct RealOps {
  using T = double;
  static constexpr int kParts = 1;   // doubles per dot result
  __device__ static void dot_acc(double v, double w, double* acc) { acc[0] = fma(v, w, acc[0]); }
  __device__ static double axpy_neg(const double* c, double v, double x) { return fma(-c[0], v, x); }
};
struct ComplexOps {
  using T = double2;
  static constexpr int kParts = 2;
  // acc += conj(v) w
  __device__ static void dot_acc(double2 v, double2 w, double* acc) {
    acc[0] = fma(v.x, w.x, fma(v.y, w.y, acc[0]));
    acc[1] = fma(v.x, w.y, fma(-v.y, w.x, acc[1]));
  }
  // x - c v
  __device__ static double2 axpy_neg(const double* c, double2 v, double2 x) {
    return make_double2(fma(-c[0], v.x, fma(c[1], v.y, x.x)), fma(-c[0], v.y, fma(-c[1], v.x, x.y)));
  }
};

// The sums of v[0 .. N) (N a power of two) over the warp's lanes: lane l gets the one of index
// sum_index<N>(l). Halves are exchanged while they are added, so N sums take N + 5 - log2 N - 1
// additions and not 5 N (an FP64 addition costs a warp 80 cycles here). Fixed order.
template <int N>
__device__ __forceinline__ double warp_sums(double (&v)[N], int lane) {
  int o = 16;
#pragma unroll
  for (int w = N / 2; w >= 1; w /= 2, o /= 2) {
    const bool up = lane & o;
#pragma unroll
    for (int k = 0; k < w; ++k) {
      const double send = up ? v[k] : v[k + w], keep = up ? v[k + w] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  for (; o > 0; o /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}
template <int N>
__device__ __forceinline__ int sum_index(int lane) {
  int i = 0, o = 16;
#pragma unroll
  for (int w = N / 2; w >= 1; w /= 2, o /= 2) i += lane & o ? w : 0;
  return i;
}

__host__ __device__ constexpr int pow2_up(int n) { return n <= 1 ? 1 : n <= 2 ? 2 : n <= 4 ? 4 : 8; }

// part[value * gridDim.x + CTA] = this CTA's share of conj(V_i) w for the G vectors from V (its
// elements [e0, e1), a thread's own ones). One instantiation per G: a predicated-off multiply-add
// would cost as much as an executed one.
template <class Ops, int G>
__device__ __forceinline__ void dot_group(const typename Ops::T* __restrict__ V, int64_t ld,
                                          const typename Ops::T* __restrict__ w, int64_t e0, int64_t e1,
                                          double (*red)[kGroup], double* __restrict__ part) {
  constexpr int N = G * Ops::kParts, P = pow2_up(N);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double acc[P] = {};
#pragma unroll 2
  for (int64_t e = e0 + threadIdx.x; e < e1; e += kVecThreads) {
    const typename Ops::T x = w[e];
    typename Ops::T v[G];
#pragma unroll
    for (int u = 0; u < G; ++u) v[u] = __ldg(V + (int64_t)u * ld + e);
#pragma unroll
    for (int u = 0; u < G; ++u) Ops::dot_acc(v[u], x, acc + u * Ops::kParts);
  }
  const double t = warp_sums<P>(acc, lane);
  if ((lane & (32 / P - 1)) == 0) red[warp][sum_index<P>(lane)] = t;
  __syncthreads();
  if (threadIdx.x < N) {
    double s = red[0][threadIdx.x];
#pragma unroll
    for (int q = 1; q < kVecWarps; ++q) s += red[q][threadIdx.x];
    part[(int64_t)threadIdx.x * gridDim.x + blockIdx.x] = s;
  }
  __syncthreads();
}

// x - sum over G vectors of c_i V_i, for this thread's elements.
template <class Ops, int G>
__device__ __forceinline__ void subtract_group(const typename Ops::T* __restrict__ V, int64_t ld, const double* c,
                                               typename Ops::T* __restrict__ w, int64_t e0, int64_t e1) {
  double k[G * Ops::kParts];
#pragma unroll
  for (int u = 0; u < G * Ops::kParts; ++u) k[u] = c[u];
#pragma unroll 2
  for (int64_t e = e0 + threadIdx.x; e < e1; e += kVecThreads) {
    typename Ops::T x = w[e], v[G];
#pragma unroll
    for (int u = 0; u < G; ++u) v[u] = __ldg(V + (int64_t)u * ld + e);
#pragma unroll
    for (int u = 0; u < G; ++u) x = Ops::axpy_neg(k + u * Ops::kParts, v[u], x);
    w[e] = x;
  }
}

// f.template operator()<G>(first vector) over nv vectors in groups of kGroup / kParts
template <class Ops, typename F>
__device__ __forceinline__ void by_group(int nv, F&& f) {
  constexpr int kMost = kGroup / Ops::kParts;
  int i = 0;
  for (; i + kMost <= nv; i += kMost) f(std::integral_constant<int, kMost>{}, i);
  switch (nv - i) {
    case 1: f(std::integral_constant<int, 1>{}, i); break;
    case 2: f(std::integral_constant<int, 2>{}, i); break;
    case 3: f(std::integral_constant<int, 3>{}, i); break;
    default:
      if constexpr (kMost > 4) {
        switch (nv - i) {
          case 4: f(std::integral_constant<int, 4>{}, i); break;
          case 5: f(std::integral_constant<int, 5>{}, i); break;
          case 6: f(std::integral_constant<int, 6>{}, i); break;
          case 7: f(std::integral_constant<int, 7>{}, i); break;
          default: break;
        }
      }
  }
}

// One pass of the Gram-Schmidt step over w, every CTA its own chunk of elements:
//   SUB:    w -= sum_i c[i] V_i                 (c: the dots of the pass before)
//   !NORM:  c_out[i] = <V_i, w>;  alpha[0] += Re c_out[j]
//   NORM:   c_out[0] = ||w||
// The CTA that finishes last adds the partial sums in CTA order (deterministic). A step is three
// passes - dots; subtract and dots; subtract and norm - instead of seven launches. Bound by the
// FP64 pipe (one warp instruction per 32 elements, vector and dot or subtraction).
// 8 steps on 744k real elements (one two-site vector of D = 2000), launches timed one by one:
// dots, subtractions, norms and scaling together 950 -> 520 us; the whole run with its matvecs
// 2800 -> 2400 us.
template <class Ops, bool SUB, bool NORM>
__global__ void __launch_bounds__(kVecThreads) k_gram_schmidt(const typename Ops::T* __restrict__ V, int nv, int64_t ld,
                                                              const double* __restrict__ c_in,
                                                              typename Ops::T* __restrict__ w, int64_t n,
                                                              double* __restrict__ part, int* __restrict__ arrived,
                                                              double* __restrict__ c_out, double* __restrict__ alpha,
                                                              int j) {
  using T = typename Ops::T;
  __shared__ double red[kVecWarps][kGroup];
  __shared__ int last;
  const int64_t per = (n + gridDim.x - 1) / gridDim.x;
  const int64_t e0 = (int64_t)blockIdx.x * per, e1 = min(n, e0 + per);
  if constexpr (SUB)
    by_group<Ops>(nv, [&](auto g, int i) {
      subtract_group<Ops, decltype(g)::value>(V + (int64_t)i * ld, ld, c_in + i * Ops::kParts, w, e0, e1);
    });
  // (a thread reads back only elements it wrote itself)
  int values;
  if constexpr (NORM) {
    // |z|^2 = re^2 + im^2: the real dot of the doubles with themselves
    const double* x = reinterpret_cast<const double*>(w);
    double acc[1] = {};
    for (int64_t e = e0 + threadIdx.x; e < e1; e += kVecThreads) {
#pragma unroll
      for (int r = 0; r < Ops::kParts; ++r) {
        const double v = x[e * Ops::kParts + r];
        acc[0] = fma(v, v, acc[0]);
      }
    }
    const double t = warp_sums<1>(acc, threadIdx.x & 31);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][0] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
      double s = red[0][0];
      for (int q = 1; q < kVecWarps; ++q) s += red[q][0];
      part[blockIdx.x] = s;
    }
    values = 1;
  } else {
    by_group<Ops>(nv, [&](auto g, int i) {
      dot_group<Ops, decltype(g)::value>(V + (int64_t)i * ld, ld, w, e0, e1, red,
                                         part + (int64_t)i * Ops::kParts * gridDim.x);
    });
    values = nv * Ops::kParts;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(arrived, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  if (threadIdx.x == 0) *arrived = 0;   // for the next launch
  __threadfence();
  const int lane = threadIdx.x & 31;
  for (int i = threadIdx.x >> 5; i < values; i += kVecWarps) {
    double v[1] = {};
    for (int b = lane; b < (int)gridDim.x; b += 32) v[0] += __ldcg(part + (int64_t)i * gridDim.x + b);
    const double t = warp_sums<1>(v, lane);
    if (lane == 0) {
      c_out[i] = NORM ? sqrt(t) : t;
      if (!NORM && i == j * Ops::kParts) alpha[0] += t;
    }
  }
}

__global__ void __launch_bounds__(kVecThreads) k_scale_into(const double* __restrict__ w,
                                                            const double* __restrict__ beta, double* __restrict__ v,
                                                            int64_t n) {
  const double b = beta[0];
  const double inv = b > 0.0 ? 1.0 / b : 0.0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    v[e] = w[e] * inv;
}

__global__ void k_zero(double* p, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) p[i] = 0.0;
}

}  // namespace

struct qltg_lanczos {
  qltg_matvec* mv = nullptr;
  int max_iter = 0;
  bool cplx = false;
  int64_t n = 0;          // elements of ψ
  int64_t ld = 0;         // stride between Krylov vectors in elements (n rounded up to 32)
  int steps = 0;          // steps taken since the last start
  // coef: alpha[max_iter] | beta[max_iter + 1] | c[2 (max_iter + 1)] | the second pass's c
  DevBuf V, w, part, coef, arrived;
  std::vector<cudaGraphExec_t> graphs;
  std::vector<cudaGraph_t> graph_defs;
  cudaStream_t capture = nullptr;

  int parts() const { return cplx ? 2 : 1; }
  int64_t n_doubles() const { return n * parts(); }
  double* alpha() const { return coef.as<double>(); }
  double* beta() const { return coef.as<double>() + max_iter; }
  double* cbuf(int pass) const { return coef.as<double>() + 2 * max_iter + 1 + pass * 2 * (max_iter + 1); }
  int64_t coef_doubles() const { return 2 * max_iter + 1 + 4 * (int64_t)(max_iter + 1); }
  double* vec(int i) const { return V.as<double>() + (int64_t)i * ld * parts(); }

  ~qltg_lanczos() {
    for (size_t i = 0; i < graphs.size(); ++i) {
      if (graphs[i]) cudaGraphExecDestroy(graphs[i]);
      if (graph_defs[i]) cudaGraphDestroy(graph_defs[i]);
    }
    if (capture) cudaStreamDestroy(capture);
  }

  // two passes of classical Gram-Schmidt of w against v_0 .. v_j, then beta_{j+1} = ||w||
  template <class Ops>
  void gram_schmidt(int j, cudaStream_t s) {
    using T = typename Ops::T;
    const T* Vt = V.as<T>();
    T* wt = w.as<T>();
    double* pt = part.as<double>();
    int* arr = arrived.as<int>();
    k_gram_schmidt<Ops, false, false><<<kVecBlocks, kVecThreads, 0, s>>>(Vt, j + 1, ld, nullptr, wt, n, pt, arr, cbuf(0), alpha() + j, j);
    k_gram_schmidt<Ops, true, false><<<kVecBlocks, kVecThreads, 0, s>>>(Vt, j + 1, ld, cbuf(0), wt, n, pt, arr, cbuf(1), alpha() + j, j);
    k_gram_schmidt<Ops, true, true><<<kVecBlocks, kVecThreads, 0, s>>>(Vt, j + 1, ld, cbuf(1), wt, n, pt, arr, beta() + j + 1, nullptr, 0);
  }

  // ||x|| of n_doubles() values (x is only read)
  void norm_into(const double* x, double* out, cudaStream_t s) {
    k_gram_schmidt<RealOps, false, true><<<kVecBlocks, kVecThreads, 0, s>>>(
        nullptr, 0, 0, nullptr, const_cast<double*>(x), n_doubles(), part.as<double>(), arrived.as<int>(), out, nullptr, 0);
  }

  // the kernels of step j, enqueued on s
  void enqueue_step(int j, cudaStream_t s) {
    mv->enqueue(vec(j), w.get(), s);
    if (cplx) gram_schmidt<ComplexOps>(j, s);
    else gram_schmidt<RealOps>(j, s);
    k_scale_into<<<kVecBlocks, kVecThreads, 0, s>>>(w.as<double>(), beta() + j + 1, vec(j + 1), n_doubles());
  }
};

extern "C" {

int qltg_lanczos_create(qltg_matvec* mv, int32_t max_iter, qltg_lanczos** lz) {
  return guarded([&] {
    QLTG_CHECK(mv && lz, QLTG_ERR_INVALID, "null matvec or out-pointer");
    QLTG_CHECK(max_iter >= 1 && max_iter <= 63, QLTG_ERR_INVALID, "max_iter must be 1 .. 63");
    QLTG_CUDA(cudaSetDevice(mv->ctx->device));
    auto h = std::make_unique<qltg_lanczos>();
    h->mv = mv;
    mv->frozen = true;   // the step graphs capture the matvec's current form
    h->max_iter = max_iter;
    h->cplx = mv->step[3].c.dtype == QLTG_C128;
    h->n = mv->psi_size;
    QLTG_CHECK(mv->step[3].c.size == h->n, QLTG_ERR_INVALID, "matvec result and psi differ in size");
    h->ld = (h->n + 31) / 32 * 32;
    const int64_t eb = h->cplx ? 16 : 8;
    h->V.alloc(std::max<int64_t>(1, (int64_t)(max_iter + 1) * h->ld) * eb);
    h->w.alloc(std::max<int64_t>(1, h->ld) * eb);
    h->part.alloc((int64_t)kVecBlocks * (max_iter + 1) * 2 * 8);
    h->coef.alloc(h->coef_doubles() * 8);
    h->arrived.alloc(sizeof(int));
    h->graphs.assign(max_iter, nullptr);
    h->graph_defs.assign(max_iter, nullptr);
    QLTG_CUDA(cudaStreamCreateWithFlags(&h->capture, cudaStreamNonBlocking));
    QLTG_CUDA(cudaMemsetAsync(h->arrived.get(), 0, sizeof(int), h->capture));
    QLTG_CUDA(cudaStreamSynchronize(h->capture));   // before any stream runs a step
    *lz = h.release();
  });
}

int qltg_lanczos_start(qltg_lanczos* lz, const void* psi0_dev, void* stream) {
  return guarded([&] {
    QLTG_CHECK(lz && psi0_dev, QLTG_ERR_INVALID, "null Lanczos or psi0");
    QLTG_CUDA(cudaSetDevice(lz->mv->ctx->device));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    k_zero<<<1, kVecThreads, 0, s>>>(lz->coef.as<double>(), (int)lz->coef_doubles());
    const double* x = static_cast<const double*>(psi0_dev);
    lz->norm_into(x, lz->beta(), s);   // beta_0 = ||psi0||
    k_scale_into<<<kVecBlocks, kVecThreads, 0, s>>>(x, lz->beta(), lz->vec(0), lz->n_doubles());
    QLTG_CUDA(cudaGetLastError());
    lz->steps = 0;
  });
}

int qltg_lanczos_step(qltg_lanczos* lz, void* stream) {
  return guarded([&] {
    QLTG_CHECK(lz, QLTG_ERR_INVALID, "null Lanczos");
    QLTG_CHECK(lz->steps < lz->max_iter, QLTG_ERR_INVALID, "Lanczos: max_iter steps already taken");
    QLTG_CUDA(cudaSetDevice(lz->mv->ctx->device));
    const int j = lz->steps;
    if (!lz->graphs[j]) {
      // the matvec's split-precision schedule must exist before capture (its first use builds it)
      QLTG_CUDA(cudaStreamBeginCapture(lz->capture, cudaStreamCaptureModeThreadLocal));
      try {
        lz->enqueue_step(j, lz->capture);
      } catch (...) {
        cudaGraph_t junk = nullptr;
        cudaStreamEndCapture(lz->capture, &junk);
        if (junk) cudaGraphDestroy(junk);
        throw;
      }
      QLTG_CUDA(cudaStreamEndCapture(lz->capture, &lz->graph_defs[j]));
      QLTG_CUDA(cudaGraphInstantiate(&lz->graphs[j], lz->graph_defs[j], 0));
    }
    QLTG_CUDA(cudaGraphLaunch(lz->graphs[j], static_cast<cudaStream_t>(stream)));
    lz->steps = j + 1;
  });
}

int qltg_lanczos_coeffs(qltg_lanczos* lz, int32_t* nsteps, double* alpha, double* beta, void* stream) {
  return guarded([&] {
    QLTG_CHECK(lz, QLTG_ERR_INVALID, "null Lanczos");
    QLTG_CUDA(cudaSetDevice(lz->mv->ctx->device));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int k = lz->steps;
    if (nsteps) *nsteps = k;
    if (alpha && k) QLTG_CUDA(cudaMemcpyAsync(alpha, lz->alpha(), k * sizeof(double), cudaMemcpyDeviceToHost, s));
    if (beta) QLTG_CUDA(cudaMemcpyAsync(beta, lz->beta(), (k + 1) * sizeof(double), cudaMemcpyDeviceToHost, s));
    QLTG_CUDA(cudaStreamSynchronize(s));
  });
}

int qltg_lanczos_vector(const qltg_lanczos* lz, int32_t i, const void** v_dev) {
  return guarded([&] {
    QLTG_CHECK(lz && v_dev, QLTG_ERR_INVALID, "null Lanczos or out-pointer");
    QLTG_CHECK(i >= 0 && i <= lz->steps, QLTG_ERR_INVALID, "Krylov vector index out of range");
    *v_dev = lz->vec(i);
  });
}

int qltg_lanczos_destroy(qltg_lanczos* lz) {
  delete lz;
  return QLTG_OK;
}

}  // extern "C"
