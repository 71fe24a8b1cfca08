// C-ABI entry points of libgbba (include/gbba.h): handle management, the
// solve entry, and the forward / backward projection contract that replaces
// ceres::Problem::Evaluate (3rdparty/ceres/include/ceres/problem.h:392-468)
// for the reference's reprojection functors.
#include <math_constants.h>
#include <cstring>
#include <type_traits>

#include "gbba_device.cuh"
#include "gbba_internal.h"

namespace gbba {
gbba_status solve_impl(gbba_handle* h, const gbba_problem* P, const gbba_options* o, gbba_summary* sum);
gbba_status solve_batched_impl(gbba_handle* h, const gbba_problem* probs, int32_t n, const gbba_options* o,
                               gbba_summary* sums);
// FP64 linearisation data of every camera (the solver's).
__global__ void k_cam_lin(const double* __restrict__ ext, int64_t nc, double* __restrict__ lin);

static int model_k(int m) { return m == kPinholeF ? 1 : m == kRadialK3 ? 6 : 8; }

static gbba_status check_problem(const gbba_problem* P) {
  if (!P) return GBBA_ERROR_INVALID_ARGUMENT;
  if (P->camera_model < 0 || P->camera_model > 2) return GBBA_ERROR_INVALID_ARGUMENT;
  if (P->memory != GBBA_MEMORY_HOST && P->memory != GBBA_MEMORY_DEVICE) return GBBA_ERROR_INVALID_ARGUMENT;
  if (P->num_cameras < 0 || P->num_intrinsics < 0 || P->num_points < 0 || P->num_observations < 0)
    return GBBA_ERROR_INVALID_ARGUMENT;
  if (P->num_observations > 0xFFFFFFFFLL || P->num_points >= 0xFFFFFFFFLL || P->num_cameras >= 0x7FFFFFFFLL)
    return GBBA_ERROR_TOO_LARGE;
  if (P->num_observations > 0 &&
      (!P->observations || !P->camera_index || !P->intrinsic_index || !P->point_index || !P->extrinsics ||
       !P->intrinsics || !P->points))
    return GBBA_ERROR_INVALID_ARGUMENT;
  return GBBA_SUCCESS;
}

template <typename F>
static gbba_status guarded(gbba_handle* h, void* stream, F&& f) {
  if (!h) return GBBA_ERROR_INVALID_ARGUMENT;
  try {
    GBBA_CUDA(cudaSetDevice(h->device));
    h->active = stream ? (cudaStream_t)stream : h->stream;
    return f();
  } catch (const Error& e) {
    if (std::getenv("GBBA_VERBOSE")) fprintf(stderr, "gbba: %s\n", e.what.c_str());
    cudaGetLastError();
    return e.status;
  }
}

__global__ void k_check_indices(const uint32_t* cam, const uint32_t* icam, const uint32_t* pt, int64_t no, int64_t nc,
                                int64_t ni, int64_t np, int* err) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < no; i += (int64_t)gridDim.x * blockDim.x)
    if (cam[i] >= nc || icam[i] >= ni || pt[i] >= np) atomicExch(err, 1);
}

template <int M>
__global__ void __launch_bounds__(256) k_forward(const double* ext, const double* intr, const double* pts,
                                                 const double* obs, const uint32_t* cam, const uint32_t* icam,
                                                 const uint32_t* pt, int64_t no, int loss_type, double a, double* res,
                                                 double* part) {
  constexpr int K = Model<M>::K;
  __shared__ double sh[8];
  double acc = 0.0;
  for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < no; o += (int64_t)gridDim.x * blockDim.x) {
    double E[6], Kp[K], X[3], r[2], dJe[2][6], dJk[2][K], dJx[2][3];
    for (int i = 0; i < 6; ++i) E[i] = ext[6 * (int64_t)cam[o] + i];
    for (int i = 0; i < K; ++i) Kp[i] = intr[K * (int64_t)icam[o] + i];
    for (int i = 0; i < 3; ++i) X[i] = pts[3 * (int64_t)pt[o] + i];
    residual<M, double, false>(Kp, E, X, obs[2 * o], obs[2 * o + 1], r, dJe, dJk, dJx, (double*)nullptr);
    double sr1;
    acc += robust<double>(loss_type, a, r[0] * r[0] + r[1] * r[1], &sr1);
    if (res) {
      res[2 * o] = r[0];
      res[2 * o + 1] = r[1];
    }
  }
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < 8; ++w) s += sh[w];
    part[blockIdx.x] = s;
  }
}

// Jacobian blocks and gradient of the robustified residual.  T = double is
// the plain FP64 path.  T = float is the Jacobian the mixed solve uses inside
// its Schur build (obs_jacobian<M, float, ...> in gbba_solver.cu): the FP32
// instantiation of the same hand-written adjoint, evaluated at FP32 copies of
// the parameters and observation, with the residual and the Corrector scale
// sqrt(rho') taken in FP64; the blocks are written widened to FP64.
struct BackArgs {
  const double *ext, *lin, *intr, *pts, *obs;
  const uint32_t *cam, *icam, *pt;
  int64_t no, nc, ni;
  int loss_type;
  double a;
  double *je, *jk, *jx;  // outputs, or null
  double* rc;            // corrected residuals of the stored blocks, or null
  double* grad;          // largest |term| of each entry, then its fixed-point sum, or null
  int* gexp;             // scale of each gradient entry
};

// The corrected blocks and residual of observation o.
template <int M, typename T>
__device__ __forceinline__ void back_blocks(const BackArgs& A, int64_t o, uint32_t c, uint32_t g, uint32_t p,
                                            T Je[2][6], T Jk[2][Model<M>::K], T Jx[2][3], double rc[2]) {
  constexpr int K = Model<M>::K;
  double Kp[K], X[3], r[2];
  for (int i = 0; i < K; ++i) Kp[i] = A.intr[K * (int64_t)g + i];
  for (int i = 0; i < 3; ++i) X[i] = A.pts[3 * (int64_t)p + i];
  const double ox = A.obs[2 * o], oy = A.obs[2 * o + 1];
  if constexpr (sizeof(T) == 8) {
    residual_lin<M>(Kp, A.lin + kCamLin * (int64_t)c, X, ox, oy, r, Je, Jk, Jx);
  } else {
    double E[6], dJe[2][6], dJk[2][K], dJx[2][3];
    for (int i = 0; i < 6; ++i) E[i] = A.ext[6 * (int64_t)c + i];
    residual<M, double, false>(Kp, E, X, ox, oy, r, dJe, dJk, dJx, (double*)nullptr);
    T Ef[6], Kf[K], Xf[3], rf[2];
    for (int i = 0; i < 6; ++i) Ef[i] = (T)E[i];
    for (int i = 0; i < K; ++i) Kf[i] = (T)Kp[i];
    for (int i = 0; i < 3; ++i) Xf[i] = (T)X[i];
    residual<M, T, true>(Kf, Ef, Xf, (T)ox, (T)oy, rf, Je, Jk, Jx, (T*)nullptr);
  }
  double sr1;
  robust<double>(A.loss_type, A.a, r[0] * r[0] + r[1] * r[1], &sr1);
  rc[0] = r[0] * sr1;
  rc[1] = r[1] * sr1;
  const T s = (T)sr1;
  for (int i = 0; i < 2; ++i) {
    for (int j = 0; j < 6; ++j) Je[i][j] *= s;
    for (int j = 0; j < K; ++j) Jk[i][j] *= s;
    for (int j = 0; j < 3; ++j) Jx[i][j] *= s;
  }
}

// An observation's term of a gradient entry: the same rounding wherever it is
// formed (the scale comes from the largest term as the first pass forms it).
__device__ __forceinline__ double grad_term(double j0, double j1, double r0, double r1) {
  return __fma_rn(j0, r0, __dmul_rn(j1, r1));
}

// W values per observation of a warp's 32 consecutive observations (`cnt` of
// them) to out: through shared memory, so that the stores are consecutive.
template <int W, typename T>
__device__ __forceinline__ void warp_store(double* __restrict__ out, int64_t o0, int cnt, const T* v, double* sh) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
#pragma unroll
  for (int j = 0; j < W; ++j) sh[lane * (W + 1) + j] = (double)v[j];
  __syncwarp();
  for (int e = lane; e < cnt * W; e += 32) out[o0 * W + e] = sh[(e / W) * (W + 1) + e % W];
}

// Bound by the FP64 pipe (about 250 operations an observation) and by the 272
// bytes written for it.  Before, every observation differentiated the rotation
// again, its blocks left lane by lane, a pass in front found the largest terms and
// the gradient evaluated everything a third time: 300 cameras, 1M observations
// 1673 -> 740 us for blocks, residuals and gradient (2.3x; 666 us with scales
// from the exponents of J and r alone, which left two to three bits of every
// sum unused).
// The blocks of every observation (32 consecutive ones per warp), and with a
// gradient the largest term of each of its entries.
constexpr int kBackThreads = 128;
template <int M, typename T>
__global__ void __launch_bounds__(kBackThreads) k_backward(BackArgs A) {
  constexpr int K = Model<M>::K;
  __shared__ double stage[kBackThreads / 32][32 * ((K > 6 ? 2 * K : 12) + 1)];
  const int lane = threadIdx.x & 31;
  double* sh = stage[threadIdx.x >> 5];
  const int64_t nw = (gridDim.x * (int64_t)blockDim.x) >> 5;
  for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; 32 * w < A.no; w += nw) {
    const int64_t o0 = 32 * w, o = min(o0 + lane, A.no - 1);
    const int cnt = (int)min((int64_t)32, A.no - o0);
    const uint32_t c = A.cam[o], g = A.icam[o], p = A.pt[o];
    T Je[2][6], Jk[2][K], Jx[2][3];
    double rc[2];
    back_blocks<M, T>(A, o, c, g, p, Je, Jk, Jx, rc);
    if (A.grad && lane < cnt) {
      // |term| as ordered bits; all ones for a non-finite one
      auto largest = [&](int64_t idx, T j0, T j1) {
        const double v = grad_term((double)j0, (double)j1, rc[0], rc[1]);
        const unsigned long long b = (__double2hiint(v) & 0x7ff00000) == 0x7ff00000
                                         ? ~0ull : (unsigned long long)__double_as_longlong(v) & ~(1ull << 63);
        unsigned long long* q = reinterpret_cast<unsigned long long*>(A.grad) + idx;
        if (*(volatile unsigned long long*)q < b) atomicMax(q, b);  // it only grows: a stale value costs an atomic
      };
      for (int j = 0; j < 6; ++j) largest(6 * (int64_t)c + j, Je[0][j], Je[1][j]);
      for (int j = 0; j < K; ++j) largest(6 * A.nc + K * (int64_t)g + j, Jk[0][j], Jk[1][j]);
      for (int j = 0; j < 3; ++j) largest(6 * A.nc + K * A.ni + 3 * (int64_t)p + j, Jx[0][j], Jx[1][j]);
    }
    if (A.je) warp_store<12>(A.je, o0, cnt, &Je[0][0], sh);
    if (A.jk) warp_store<2 * K>(A.jk, o0, cnt, &Jk[0][0], sh);
    if (A.jx) warp_store<6>(A.jx, o0, cnt, &Jx[0][0], sh);
    if (A.rc && lane < cnt) {
      A.rc[2 * o] = rc[0];
      A.rc[2 * o + 1] = rc[1];
    }
  }
}

// The gradient's deterministic sums (see lin_fx): every entry's terms in fixed
// point, scaled by its largest one.  kStored: from the blocks and residuals
// that k_backward wrote (256 B an observation), else evaluated again.
template <int M, typename T, bool kStored>
__global__ void __launch_bounds__(256) k_backward_sum(BackArgs A) {
  constexpr int K = Model<M>::K;
  for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < A.no; o += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t c = A.cam[o], g = A.icam[o], p = A.pt[o];
    auto put = [&](int64_t idx, double v) {
      atomicAdd(reinterpret_cast<unsigned long long*>(A.grad + idx), (unsigned long long)lin_fx(v, A.gexp[idx]));
    };
    if constexpr (kStored) {
      const double r0 = A.rc[2 * o], r1 = A.rc[2 * o + 1];
      auto block = [&](const double* __restrict__ J, int n, int64_t base) {
#pragma unroll
        for (int j = 0; j < n; ++j) put(base + j, grad_term(J[j], J[n + j], r0, r1));
      };
      block(A.je + 12 * o, 6, 6 * (int64_t)c);
      block(A.jk + 2 * K * o, K, 6 * A.nc + K * (int64_t)g);
      block(A.jx + 6 * o, 3, 6 * A.nc + K * A.ni + 3 * (int64_t)p);
    } else {
      T Je[2][6], Jk[2][K], Jx[2][3];
      double rc[2];
      back_blocks<M, T>(A, o, c, g, p, Je, Jk, Jx, rc);
      auto term = [&](T j0, T j1) { return grad_term((double)j0, (double)j1, rc[0], rc[1]); };
      for (int j = 0; j < 6; ++j) put(6 * (int64_t)c + j, term(Je[0][j], Je[1][j]));
      for (int j = 0; j < K; ++j) put(6 * A.nc + K * (int64_t)g + j, term(Jk[0][j], Jk[1][j]));
      for (int j = 0; j < 3; ++j) put(6 * A.nc + K * A.ni + 3 * (int64_t)p + j, term(Jx[0][j], Jx[1][j]));
    }
  }
}

// Between the gradient's passes: each entry's scale from its largest term, and
// the entry cleared for the fixed-point sum; after them: back to FP64 (NaN for
// an entry with a non-finite term).
__global__ void k_grad_exp(int64_t n, double nobs, double* __restrict__ grad, int* __restrict__ gexp) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    unsigned long long* q = reinterpret_cast<unsigned long long*>(grad + i);
    gexp[i] = lin_exp(*q, nobs);
    *q = 0ull;
  }
}
__global__ void k_grad_conv(int64_t n, double* __restrict__ grad, const int* __restrict__ gexp) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const long long v = __double_as_longlong(grad[i]);
    grad[i] = gexp[i] >= kFxNonFinite ? CUDART_NAN : ldexp((double)v, -gexp[i]);
  }
}

struct Staged {
  const double *ext, *intr, *pts, *obs;
  const uint32_t *cam, *icam, *pt;
};

// An array of the call in the caller's memory.
struct Span {
  const void* p;
  size_t bytes;
  bool aligned(size_t to) const { return (reinterpret_cast<uintptr_t>(p) & (to - 1)) == 0; }
  bool overlaps(const Span& o) const {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p), b = reinterpret_cast<uintptr_t>(o.p);
    return bytes && o.bytes && a < b + o.bytes && b < a + bytes;
  }
};
struct Inputs {
  Span a[7];  // extrinsics, intrinsics, points, observations, the three indices
};
static Inputs input_spans(const gbba_problem* P) {
  const size_t no = P->num_observations;
  return {{{P->extrinsics, sizeof(double) * 6 * P->num_cameras},
           {P->intrinsics, sizeof(double) * model_k(P->camera_model) * P->num_intrinsics},
           {P->points, sizeof(double) * 3 * P->num_points},
           {P->observations, sizeof(double) * 2 * no},
           {P->camera_index, sizeof(uint32_t) * no},
           {P->intrinsic_index, sizeof(uint32_t) * no},
           {P->point_index, sizeof(uint32_t) * no}}};
}
// Whether the kernels write output `o` where the caller wants it: an aligned
// array in device memory apart from everything else that the call reads or
// writes.  Other outputs are staged and copied out at the end.
static bool in_place(const gbba_problem* P, const Span& o, const Span* others = nullptr, int n = 0) {
  if (P->memory == GBBA_MEMORY_HOST || !o.aligned(sizeof(double))) return false;
  for (const Span& i : input_spans(P).a)
    if (o.overlaps(i)) return false;
  for (int i = 0; i < n; ++i)
    if (&others[i] != &o && o.overlaps(others[i])) return false;
  return true;
}

// Make the problem's arrays device-resident and check indices: the caller's
// own arrays in device memory that the kernels can read (aligned for their
// type), else copies.
static Staged stage(gbba_handle* h, const gbba_problem* P, size_t extra_bytes, char** extra) {
  const int64_t no = P->num_observations, nc = P->num_cameras, ni = P->num_intrinsics, np = P->num_points;
  const int k = model_k(P->camera_model);
  cudaStream_t st = h->active;
  Planner pl;
  pl.take<double>(6 * nc);
  pl.take<double>(k * ni);
  pl.take<double>(3 * np);
  pl.take<double>(2 * no);
  for (int i = 0; i < 3; ++i) pl.take<uint32_t>(no);
  pl.take<int>(1);
  pl.take<char>(extra_bytes);
  h->arena.reset();
  h->arena.reserve(pl.used + 4096);
  Staged s;
  const bool host = P->memory == GBBA_MEMORY_HOST;
  auto put = [&](const Span& src, size_t align) -> const void* {
    if (!host && src.aligned(align)) return src.p;
    void* d = h->arena.take<char>(src.bytes);
    if (src.bytes)
      GBBA_CUDA(cudaMemcpyAsync(d, src.p, src.bytes, host ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, st));
    return d;
  };
  const Inputs in = input_spans(P);
  s.ext = (const double*)put(in.a[0], sizeof(double));
  s.intr = (const double*)put(in.a[1], sizeof(double));
  s.pts = (const double*)put(in.a[2], sizeof(double));
  s.obs = (const double*)put(in.a[3], sizeof(double));
  s.cam = (const uint32_t*)put(in.a[4], sizeof(uint32_t));
  s.icam = (const uint32_t*)put(in.a[5], sizeof(uint32_t));
  s.pt = (const uint32_t*)put(in.a[6], sizeof(uint32_t));
  int* err = h->arena.take<int>(1);
  *extra = h->arena.take<char>(extra_bytes);
  GBBA_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
  if (no > 0) {
    const int grid = std::max(1, std::min<int>((int)ceil_div(no, 256), h->sm_count * 8));
    k_check_indices<<<grid, 256, 0, st>>>(s.cam, s.icam, s.pt, no, nc, ni, np, err);
    check_launch(h);
  }
  int herr = 0;
  GBBA_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st));
  GBBA_CUDA(cudaStreamSynchronize(st));
  GBBA_REQUIRE(herr == 0, GBBA_ERROR_INVALID_ARGUMENT, "observation index out of range");
  return s;
}

}  // namespace gbba

using namespace gbba;

extern "C" {

int gbba_abi_version(void) { return GBBA_ABI_VERSION; }

const char* gbba_status_string(gbba_status s) {
  switch (s) {
    case GBBA_SUCCESS: return "success";
    case GBBA_ERROR_INVALID_ARGUMENT: return "invalid argument";
    case GBBA_ERROR_CUDA: return "CUDA error";
    case GBBA_ERROR_OUT_OF_MEMORY: return "out of device memory";
    case GBBA_ERROR_NUMERICAL: return "non-finite cost at the initial point";
    case GBBA_ERROR_NOT_SUPPORTED: return "not supported";
    case GBBA_ERROR_TOO_LARGE: return "problem exceeds a documented limit";
    case GBBA_ERROR_NO_DEVICE: return "no CUDA device";
    case GBBA_ERROR_TIMEOUT: return "bounded device wait expired";
  }
  return "unknown status";
}

void gbba_default_options(gbba_options* o) {
  if (!o) return;
  std::memset(o, 0, sizeof(*o));
  o->max_num_iterations = 50;
  o->max_num_consecutive_invalid_steps = 5;
  o->function_tolerance = 1e-6;
  o->gradient_tolerance = 1e-10;
  o->parameter_tolerance = 1e-8;
  o->initial_trust_region_radius = 1e4;
  o->max_trust_region_radius = 1e16;
  o->min_trust_region_radius = 1e-32;
  o->min_relative_decrease = 1e-3;
  o->min_lm_diagonal = 1e-6;
  o->max_lm_diagonal = 1e32;
  o->jacobi_scaling = 1;
  o->loss_type = GBBA_LOSS_SQUARED;
  o->loss_scale = 1.0;
  o->linear_solver = GBBA_SOLVER_AUTO;
  o->precision = GBBA_PRECISION_FP64;
  o->max_linear_solver_iterations = 500;
  o->dense_schur_max_size = 16384;
  o->eta = 0.1;
  o->refinement_interval = 10;
  o->use_cuda_graphs = 1;
  o->stream = nullptr;
  o->fp64_polish_iterations = 10;
  o->schur_build = GBBA_SCHUR_BUILD_AUTO;
}

gbba_status gbba_create(int device, gbba_handle** out) {
  if (!out) return GBBA_ERROR_INVALID_ARGUMENT;
  *out = nullptr;
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
    cudaGetLastError();
    return GBBA_ERROR_NO_DEVICE;
  }
  if (device < 0 || device >= n) return GBBA_ERROR_INVALID_ARGUMENT;
  gbba_handle* h = new gbba_handle();
  h->device = device;
  try {
    GBBA_CUDA(cudaSetDevice(device));
    GBBA_CUDA(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
    int least = 0;
    GBBA_CUDA(cudaDeviceGetStreamPriorityRange(&least, &h->prio_hi));
    GBBA_CUDA(cudaStreamCreateWithPriority(&h->side, cudaStreamNonBlocking, least));
    GBBA_CUDA(cudaEventCreateWithFlags(&h->ev_main, cudaEventDisableTiming));
    GBBA_CUDA(cudaEventCreateWithFlags(&h->ev_side, cudaEventDisableTiming));
    GBBA_CUDA(cudaEventCreate(&h->ev_k0));
    GBBA_CUDA(cudaEventCreate(&h->ev_k1));
    GBBA_CUDA(cudaHostAlloc((void**)&h->pinned, 256 * sizeof(double), cudaHostAllocDefault));
    GBBA_CUDA(cudaDeviceGetAttribute(&h->sm_count, cudaDevAttrMultiProcessorCount, device));
  } catch (const Error& e) {
    delete h;
    return e.status;
  }
  *out = h;
  return GBBA_SUCCESS;
}

void gbba_destroy(gbba_handle* h) {
  if (!h) return;
  cudaSetDevice(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  h->arena.release();
  h->pair_arena.release();
  h->item_arena.release();
  if (h->pinned) cudaFreeHost(h->pinned);
  if (h->side) cudaStreamSynchronize(h->side);
  if (h->ev_main) cudaEventDestroy(h->ev_main);
  if (h->ev_side) cudaEventDestroy(h->ev_side);
  if (h->ev_k0) cudaEventDestroy(h->ev_k0);
  if (h->ev_k1) cudaEventDestroy(h->ev_k1);
  if (h->side) cudaStreamDestroy(h->side);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
}

int64_t gbba_launch_count(const gbba_handle* h) { return h ? h->launches : 0; }

gbba_status gbba_last_kernel_time(gbba_handle* h, double* seconds) {
  if (!h || !seconds) return GBBA_ERROR_INVALID_ARGUMENT;
  if (!h->kernel_timed) return GBBA_ERROR_NOT_SUPPORTED;
  if (cudaSetDevice(h->device) != cudaSuccess) {
    cudaGetLastError();
    return GBBA_ERROR_CUDA;
  }
  float ms = 0.0f;
  if (cudaEventElapsedTime(&ms, h->ev_k0, h->ev_k1) != cudaSuccess) {
    cudaGetLastError();
    return GBBA_ERROR_CUDA;
  }
  *seconds = ms * 1e-3;
  return GBBA_SUCCESS;
}

gbba_status gbba_solve(gbba_handle* h, const gbba_problem* P, const gbba_options* o, gbba_summary* sum) {
  if (!o || !sum) return GBBA_ERROR_INVALID_ARGUMENT;
  const gbba_status pc = check_problem(P);
  if (pc != GBBA_SUCCESS) return pc;
  std::memset(sum, 0, sizeof(*sum));
  return guarded(h, o->stream, [&]() { return solve_impl(h, P, o, sum); });
}

gbba_status gbba_solve_batched(gbba_handle* h, const gbba_problem* problems, int32_t num_problems,
                               const gbba_options* o, gbba_summary* summaries) {
  if (!problems || !o || !summaries || num_problems < 0) return GBBA_ERROR_INVALID_ARGUMENT;
  if (num_problems == 0) return GBBA_SUCCESS;
  for (int32_t i = 0; i < num_problems; ++i) {
    const gbba_status pc = check_problem(&problems[i]);
    if (pc != GBBA_SUCCESS) return pc;
  }
  return guarded(h, o->stream, [&]() { return solve_batched_impl(h, problems, num_problems, o, summaries); });
}

gbba_status gbba_autotune(gbba_handle* h, const gbba_problem* P, const gbba_options* o, int32_t iterations,
                          gbba_tuning* out) {
  if (!o || !out || iterations < 1) return GBBA_ERROR_INVALID_ARGUMENT;
  const gbba_status pc = check_problem(P);
  if (pc != GBBA_SUCCESS) return pc;
  std::memset(out, 0, sizeof(*out));
  return guarded(h, o->stream, [&]() -> gbba_status {
    const int k = P->camera_model == kPinholeF ? 1 : P->camera_model == kRadialK3 ? 6 : 8;
    const size_t ne = 6 * (size_t)P->num_cameras, ni = k * (size_t)P->num_intrinsics, np = 3 * (size_t)P->num_points;
    const bool dev = P->memory == GBBA_MEMORY_DEVICE;
    cudaStream_t st = h->active;
    // the parameters, restored after every trial
    std::vector<double> keep(ne + ni + np);
    auto move = [&](bool save) {
      double* arr[3] = {P->extrinsics, P->intrinsics, P->points};
      const size_t cnt[3] = {ne, ni, np};
      size_t off = 0;
      for (int a = 0; a < 3; ++a) {
        if (cnt[a]) {
          double* host = keep.data() + off;
          if (!dev) std::memcpy(save ? host : arr[a], save ? arr[a] : host, 8 * cnt[a]);
          else
            GBBA_CUDA(cudaMemcpyAsync(save ? (void*)host : (void*)arr[a], save ? (const void*)arr[a] : (const void*)host,
                                      8 * cnt[a], save ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, st));
        }
        off += cnt[a];
      }
      if (dev) GBBA_CUDA(cudaStreamSynchronize(st));
    };
    move(true);
    // fixed work per trial: exactly `iterations` LM iterations
    gbba_options t = *o;
    t.max_num_iterations = iterations;
    t.function_tolerance = 0.0;
    t.gradient_tolerance = 0.0;
    t.parameter_tolerance = 0.0;
    t.fp64_polish_iterations = 0;
    // one trial: two solves (the first warms the workspace), the second's
    // summary; the handle's choices are restored if a solve fails
    const int keep_chunk = h->pair_chunk, keep_cw = h->camera_warps;
    const bool keep_ft = h->factor_tensor;
    gbba_summary sum;
    auto trial = [&]() -> gbba_status {
      for (int rep = 0; rep < 2; ++rep) {
        std::memset(&sum, 0, sizeof(sum));
        gbba_status s = GBBA_SUCCESS;
        try {
          s = solve_impl(h, P, &t, &sum);
        } catch (...) {
          h->pair_chunk = keep_chunk;
          h->camera_warps = keep_cw;
          h->factor_tensor = keep_ft;
          throw;
        }
        move(false);
        if (s != GBBA_SUCCESS) {
          h->pair_chunk = keep_chunk;
          h->camera_warps = keep_cw;
          h->factor_tensor = keep_ft;
          return s;
        }
      }
      return GBBA_SUCCESS;
    };
    auto per_iter = [&](double total) { return sum.num_iterations > 0 ? total / sum.num_iterations : total; };
    // 1. work-item size of the camera-pair products
    const int32_t cand[3] = {32, 64, 128};
    out->num_candidates = 3;
    int best = -1;
    bool iterative = false;
    for (int c = 0; c < 3; ++c) {
      h->pair_chunk = cand[c];
      const gbba_status s = trial();
      if (s != GBBA_SUCCESS) return s;
      iterative = sum.linear_solver_iterations > 0;
      out->candidates[c] = cand[c];
      out->schur_time_s[c] = per_iter(sum.schur_kernel_time_s);
      if (best < 0 || out->schur_time_s[c] < out->schur_time_s[best]) best = c;
      if (iterative) break;  // the iterative path forms no camera-pair products
    }
    if (iterative) {
      h->pair_chunk = keep_chunk;
      out->num_candidates = 0;
      out->pair_chunk = keep_chunk;
    } else {
      h->pair_chunk = cand[best];
      out->pair_chunk = cand[best];
    }
    out->factor_tensor = -1;
    out->camera_warps = 0;
    if (!iterative && t.precision == GBBA_PRECISION_MIXED) {
      // 2. trailing-update engine of the dense FP32 factorisation
      for (int e = 0; e < 2; ++e) {
        h->factor_tensor = e == 1;
        const gbba_status s = trial();
        if (s != GBBA_SUCCESS) return s;
        out->factor_time_s[e] = per_iter(sum.factor_time_s);
      }
      h->factor_tensor = out->factor_time_s[1] <= out->factor_time_s[0];
      out->factor_tensor = h->factor_tensor ? 1 : 0;
    } else if (iterative) {
      // 3. warps per camera of the PCG camera kernels
      const int warps[3] = {2, 4, 8};
      for (int w = 0; w < 3; ++w) {
        h->camera_warps = warps[w];
        const gbba_status s = trial();
        if (s != GBBA_SUCCESS) return s;
        out->pcg_time_s[w] = per_iter(sum.linear_solver_time_s + sum.jacobian_time_s);
      }
      int wb = 0;  // the fastest, once all three are timed
      for (int w = 1; w < 3; ++w)
        if (out->pcg_time_s[w] < out->pcg_time_s[wb]) wb = w;
      h->camera_warps = warps[wb];
      out->camera_warps = warps[wb];
    }
    return GBBA_SUCCESS;
  });
}

gbba_status gbba_project_forward(gbba_handle* h, const gbba_problem* P, int32_t loss_type, double loss_scale,
                                 double* residuals, double* cost) {
  const gbba_status pc = check_problem(P);
  if (pc != GBBA_SUCCESS) return pc;
  return guarded(h, nullptr, [&]() {
    const int64_t no = P->num_observations;
    const int grid = std::max(1, std::min<int>((int)ceil_div(std::max<int64_t>(no, 1), 256), h->sm_count * 8));
    const Span out{residuals, residuals ? sizeof(double) * 2 * no : 0};
    const size_t res_bytes = in_place(P, out) ? 0 : out.bytes;
    char* extra;
    Staged s = stage(h, P, res_bytes + sizeof(double) * grid, &extra);
    double* dres = !residuals ? nullptr : res_bytes ? (double*)extra : residuals;
    double* part = (double*)(extra + res_bytes);
    cudaStream_t st = h->active;
    switch (P->camera_model) {
      case kPinholeF: k_forward<kPinholeF><<<grid, 256, 0, st>>>(s.ext, s.intr, s.pts, s.obs, s.cam, s.icam, s.pt, no, loss_type, loss_scale, dres, part); break;
      case kRadialK3: k_forward<kRadialK3><<<grid, 256, 0, st>>>(s.ext, s.intr, s.pts, s.obs, s.cam, s.icam, s.pt, no, loss_type, loss_scale, dres, part); break;
      default: k_forward<kBrownT2><<<grid, 256, 0, st>>>(s.ext, s.intr, s.pts, s.obs, s.cam, s.icam, s.pt, no, loss_type, loss_scale, dres, part); break;
    }
    check_launch(h);
    std::vector<double> hp(grid);
    GBBA_CUDA(cudaMemcpyAsync(hp.data(), part, sizeof(double) * grid, cudaMemcpyDeviceToHost, st));
    if (res_bytes) GBBA_CUDA(cudaMemcpyAsync(residuals, dres, res_bytes, cudaMemcpyDefault, st));
    GBBA_CUDA(cudaStreamSynchronize(st));
    double c = 0.0;
    for (double v : hp) c += v;
    if (cost) *cost = c;
    return GBBA_SUCCESS;
  });
}

static gbba_status project_backward(gbba_handle* h, const gbba_problem* P, int32_t loss_type, double loss_scale,
                                    bool fp32, double* jac_extrinsic, double* jac_intrinsic, double* jac_point,
                                    double* gradient) {
  const gbba_status pc = check_problem(P);
  if (pc != GBBA_SUCCESS) return pc;
  return guarded(h, nullptr, [&]() {
    const int64_t no = P->num_observations, nc = P->num_cameras, ni = P->num_intrinsics, np = P->num_points;
    const int k = model_k(P->camera_model);
    const size_t be = jac_extrinsic ? sizeof(double) * no * 12 : 0;
    const size_t bk = jac_intrinsic ? sizeof(double) * no * 2 * k : 0;
    const size_t bx = jac_point ? sizeof(double) * no * 6 : 0;
    const int64_t ng = 6 * nc + k * ni + 3 * np;
    const size_t bg = gradient ? sizeof(double) * ng : 0;
    const size_t bgx = gradient ? sizeof(int) * ng : 0;  // the gradient entries' scale exponents
    const bool stored = be && bk && bx && bg;            // the gradient is summed from the stored blocks
    const size_t brc = stored ? sizeof(double) * 2 * no : 0;
    const size_t bl = fp32 ? 0 : sizeof(double) * kCamLin * nc;
    auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
    // outputs: the caller's arrays where they can be written, else staged ones
    double* const user[4] = {jac_extrinsic, jac_intrinsic, jac_point, gradient};
    const Span outs[4] = {{jac_extrinsic, be}, {jac_intrinsic, bk}, {jac_point, bx}, {gradient, bg}};
    size_t own[4];  // bytes staged
    for (int i = 0; i < 4; ++i) own[i] = in_place(P, outs[i], outs, 4) ? 0 : al(outs[i].bytes);
    char* extra;
    Staged s = stage(h, P, own[0] + own[1] + own[2] + own[3] + al(bgx) + al(brc) + al(bl), &extra);
    auto out = [&](int i) {
      double* d = !outs[i].bytes ? nullptr : own[i] ? (double*)extra : user[i];
      extra += own[i];
      return d;
    };
    BackArgs A;
    A.je = out(0);
    A.jk = out(1);
    A.jx = out(2);
    A.grad = out(3);
    A.gexp = bgx ? (int*)extra : nullptr;
    A.rc = brc ? (double*)(extra + al(bgx)) : nullptr;
    double* lin = bl ? (double*)(extra + al(bgx) + al(brc)) : nullptr;
    A.lin = lin;
    A.ext = s.ext, A.intr = s.intr, A.pts = s.pts, A.obs = s.obs;
    A.cam = s.cam, A.icam = s.icam, A.pt = s.pt;
    A.no = no, A.nc = nc, A.ni = ni;
    A.loss_type = loss_type, A.a = loss_scale;
    cudaStream_t st = h->active;
    if (A.grad) GBBA_CUDA(cudaMemsetAsync(A.grad, 0, bg, st));
    if (lin && nc > 0) {
      k_cam_lin<<<(unsigned)ceil_div(nc, 64), 64, 0, st>>>(s.ext, nc, lin);
      check_launch(h);
    }
    const int grid = std::max(1, std::min<int>((int)ceil_div(std::max<int64_t>(no, 1), 256), h->sm_count * 8));
    const unsigned gg = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(ng, 256), 4096));
    auto run = [&](auto blocks, auto sum_stored, auto sum) {
      // the blocks and, with a gradient, its entries' largest terms; their scales;
      // the fixed-point sums; back to FP64
      if (no > 0) {
        blocks<<<(unsigned)std::min<int64_t>(ceil_div(no, kBackThreads), (int64_t)h->sm_count * 16), kBackThreads, 0, st>>>(A);
        check_launch(h);
      }
      if (!A.grad) return;
      k_grad_exp<<<gg, 256, 0, st>>>(ng, (double)std::max<int64_t>(1, no), A.grad, A.gexp);
      check_launch(h);
      if (no > 0) {
        if (stored) sum_stored<<<grid, 256, 0, st>>>(A);
        else sum<<<grid, 256, 0, st>>>(A);
        check_launch(h);
      }
      k_grad_conv<<<gg, 256, 0, st>>>(ng, A.grad, A.gexp);
      check_launch(h);
    };
    auto model = [&](auto m) {
      constexpr int M = decltype(m)::value;
      if (fp32) run(k_backward<M, float>, k_backward_sum<M, float, true>, k_backward_sum<M, float, false>);
      else run(k_backward<M, double>, k_backward_sum<M, double, true>, k_backward_sum<M, double, false>);
    };
    switch (P->camera_model) {
      case kPinholeF: model(std::integral_constant<int, kPinholeF>()); break;
      case kRadialK3: model(std::integral_constant<int, kRadialK3>()); break;
      default: model(std::integral_constant<int, kBrownT2>()); break;
    }
    const double* const written[4] = {A.je, A.jk, A.jx, A.grad};
    for (int i = 0; i < 4; ++i)
      if (own[i]) GBBA_CUDA(cudaMemcpyAsync(user[i], written[i], outs[i].bytes, cudaMemcpyDefault, st));
    GBBA_CUDA(cudaStreamSynchronize(st));
    return GBBA_SUCCESS;
  });
}

gbba_status gbba_project_backward(gbba_handle* h, const gbba_problem* P, int32_t loss_type, double loss_scale,
                                  double* jac_extrinsic, double* jac_intrinsic, double* jac_point, double* gradient) {
  return project_backward(h, P, loss_type, loss_scale, false, jac_extrinsic, jac_intrinsic, jac_point, gradient);
}

gbba_status gbba_project_backward_mixed(gbba_handle* h, const gbba_problem* P, int32_t loss_type, double loss_scale,
                                        double* jac_extrinsic, double* jac_intrinsic, double* jac_point,
                                        double* gradient) {
  return project_backward(h, P, loss_type, loss_scale, true, jac_extrinsic, jac_intrinsic, jac_point, gradient);
}

}  // extern "C"
