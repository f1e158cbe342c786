// Host side of libcps.so: contexts, device memory, launches and the C ABI
// declared in include/cps.h.
//
// Memory: one cudaMalloc'd slab per context.  The ten FP64 field planes (u, v,
// p, p', u*, v*, dE, dN, alpha, gamma) come first, each (M+1) rows x P
// doubles, P = round_up(N+1, 32); then the 25 inner-solve planes in the
// context's storage type (double for CPS_FP64, float for CPS_MIXED); then the
// grid barrier, flags, history buffer (one copy to the host per launch takes
// the two) and reduction ring.  The fields stay resident between calls; per
// outer iteration only the 8 diagnostics travel to the host.
//
// Launch, one design: the outer iterations run in one persistent kernel
// launched cooperatively (all CTAs co-resident; in clusters of 16 where one of
// them runs the PCG), synchronised by a software grid barrier whose waits are
// bounded (2 s) and report CPS_ERR_TIMEOUT instead of hanging.
//
// Launch, many designs (cps_batch_solve): one thread-block cluster per design
// at a time; clusters take designs from a device work queue, synchronise with
// the hardware cluster barrier and reduce through distributed shared memory.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <exception>
#include <mutex>
#include <new>
#include <numeric>
#include <string>
#include <thread>
#include <vector>

#include "../../include/cps.h"
#include "cps_host.h"
#include "cps_kernels.cuh"

namespace {

thread_local std::string g_create_error;

constexpr int kHistChunk = 4096;  // outer iterations per launch inside cps_solve
constexpr int kFieldPlanes = 10;  // FP64 planes: u v p pc us vs dE dN alpha gamma
constexpr int kInnerPlanes = 25;  // cU x5, cV x5, bU bV xU0 xU1 xV0 xV1 px pr pz pp0 pp1 pAp pdiag cx cy
constexpr int kMaxGridCtas = 2048;
// A context's scratch: the barrier, the flags, the history (bytes from its start), then the rest.
constexpr size_t kFlagsAt = 64, kHistAt = 256;

enum FieldPlane { kU, kV, kP, kPc, kUs, kVs, kDE, kDN, kAlpha, kGamma };

size_t round_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace

struct cps_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  int M = 0, N = 0, P = 0;
  int precision = CPS_FP64;
  cps::DesignView view{};
  char* slab = nullptr;
  size_t slab_bytes = 0;
  size_t plane_elems = 0;
  cps::GridBarrier* bar = nullptr;
  double* red = nullptr;
  int* dstatus = nullptr;
  int* dndone = nullptr;
  double* dhist = nullptr;
  double* hstage = nullptr;  // pinned, one plane of (M+1) x (N+1) doubles
  // The flags (status, n_done, pressure-drop gate) and the history lie one after
  // the other on the device and in one pinned buffer, so that a launch's outcome
  // is one copy.  A plane's metrics are written to the pinned buffer's end by
  // the kernel itself.
  int* hflags = nullptr;
  double* hhist = nullptr;   // kHistChunk * 8
  double* hplane = nullptr;  // 8
  double* dplog = nullptr;   // device, kHistChunk x 4 pressure drops of the last launch
  double* hdplog = nullptr;  // pinned copy
  double* ddphist = nullptr; // device, the pressure-drop gate's windows (cudaMalloc'd by cps_set_dp_monitor)
  double* dpseudo = nullptr; // device, the CFL controllers' state (4 doubles)
  cps::TensorMap* dtmaps = nullptr;  // device, the planes' TMA tensor maps (kTmCount), or null
  double pseudo_start = 0.0; // the controllers' starting CFL number
  int ramp_steps = 0;        // inlet velocity ramp of cps_solve (0: off)
  int iter = 0;              // outer-loop iteration index of the next iteration (monitor and gate)
  int grid = 0;
  bool cluster = false;      // the PCG may run on one thread-block cluster (cps::kCluster)
  int kernel = -1;           // grid kernel of the last launch
  unsigned ready = 0;        // bit k: grid kernel k is loaded and may use its dynamic shared memory
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  double kernel_ms = 0.0;
  long long launches = 0, outer_done = 0;
  std::string err;
};

CPS_GRID_KERNELS(extern, double)
CPS_GRID_KERNELS(extern, float)
CPS_GRID_OPTION_KERNELS(extern, double)
CPS_GRID_OPTION_KERNELS(extern, float)
CPS_GRID_MONITOR_KERNELS(extern, double)
CPS_GRID_MONITOR_KERNELS(extern, float)
CPS_BATCH_KERNELS(extern, double)
CPS_BATCH_KERNELS(extern, float)
CPS_BATCH_OPTION_KERNELS(extern, double)
CPS_BATCH_OPTION_KERNELS(extern, float)

// samplePlaneAtX (postprocessing.cpp:62-230) for one plane, one CTA: every row's
// contribution is evaluated with the reference's expressions; the five sums are
// combined in a fixed tree order.
__global__ void __launch_bounds__(cps::kThreads) cps_plane_kernel(cps::DesignView d, double xPhysical, double* out) {
  __shared__ double smem[cps::kRedWidth * 8];
  const cps::PlaneSetup ps = cps::plane_setup(d, xPhysical);
  double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // staticAreaSum, dynAreaSum, totalWeighted, area, fluxSum
  for (int i = 1 + threadIdx.x; i < d.M; i += blockDim.x) cps::plane_row(d, ps, i, acc);
  cps::block_reduce<5, 0u>(acc, smem);
  if (threadIdx.x == 0) cps::plane_metrics(acc, out);
}

namespace {

bool cuda_ok(cps_ctx* ctx, cudaError_t e, const char* what) {
  if (e == cudaSuccess) return true;
  std::string m = std::string(what) + ": " + cudaGetErrorString(e);
  if (ctx) ctx->err = m; else g_create_error = m;
  return false;
}

cps_status fail(cps_ctx* ctx, cps_status s, const std::string& msg) {
  if (ctx) ctx->err = msg; else g_create_error = msg;
  return s;
}

size_t elem_bytes(int precision) { return precision == CPS_MIXED ? sizeof(float) : sizeof(double); }

size_t footprint_bytes(int M, int N, int precision, size_t* plane_elems_out, int* P_out) {
  const int P = (int)round_up((size_t)N + 1, 32);
  const size_t plane = (size_t)(M + 1) * P;
  if (plane_elems_out) *plane_elems_out = plane;
  if (P_out) *P_out = P;
  size_t bytes = plane * sizeof(double) * kFieldPlanes;
  bytes += round_up(plane * elem_bytes(precision) * kInnerPlanes, 256);
  bytes += 256;                                                           // barrier + flags
  bytes += (size_t)(cps::kRedSlots * cps::kRedWidth + cps::kPlaneSums) * kMaxGridCtas * 8;  // reduction ring
  bytes += (size_t)kHistChunk * 8 * 8 + 64;                               // history + plane metrics
  bytes += (size_t)kHistChunk * 4 * 8;                                    // pressure-drop log
  bytes += 64;                                                            // CFL controllers' state
  bytes += 128 + sizeof(cps::TensorMap) * cps::kTmCount;                  // TMA tensor maps
  return round_up(bytes, 256);
}

// The CFL controllers' state on the device (pseudoCFL, serResidPrev,
// lsCurrentAlpha, lsBacktrackCount), written in stream order.
bool write_pseudo_state(cps_ctx* c, double cfl, double prev, double alpha, int count) {
  const double h[4] = {cfl, prev, alpha, (double)count};
  return cuda_ok(c, cudaMemcpyAsync(c->dpseudo, h, sizeof(h), cudaMemcpyHostToDevice, c->stream), "h2d") &&
         cuda_ok(c, cudaStreamSynchronize(c->stream), "h2d");
}

// ---------------------------------------------------------------------------
// TMA tensor maps of a context's planes: one 2-D map per (plane, window shape)
// the staged phases copy, over the plane's rows 0..rmax and columns 0..P-1,
// with the window's box (its shared-memory pitch x rows).  Out-of-range parts
// of a box read as zero (the phases never use them).  Built once at
// cps_create and kept in the context's slab.
// ---------------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 encode_tiled() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

template <typename E, class W>
bool encode_map(PFN_cuTensorMapEncodeTiled_v12000 fn, cps::TensorMap* out, const E* base, int P, int rows) {
  static_assert(sizeof(cps::TensorMap) == sizeof(CUtensorMap), "tensor map size");
  const cuuint64_t dims[2] = {(cuuint64_t)P, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)P * sizeof(E)};
  const cuuint32_t box[2] = {(cuuint32_t)W::kPitch, (cuuint32_t)W::kRows};
  const cuuint32_t estr[2] = {1, 1};
  static_assert(W::kPitch * sizeof(E) % 16 == 0 && W::kPitch <= 256 && W::kRows <= 256, "TMA box");
  return fn(reinterpret_cast<CUtensorMap*>(out), sizeof(E) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
            2, const_cast<E*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename T>
bool fill_maps(PFN_cuTensorMapEncodeTiled_v12000 fn, const cps::DesignView& v, const cps::Inner<T>& w, int M, int P,
               cps::TensorMap* m) {
  using LA = cps::LayoutA;
  using LC = cps::LayoutC<T>;
  using LD = cps::LayoutD<T>;
  using LB = cps::LayoutB<T>;
  const int R = M + 1;  // rows 0..M
  const long long ps = v.planeStride;
  for (int q = 0; q < 5; ++q)
    if (!encode_map<T, typename LB::WC>(fn, m + cps::kTmCU_B + q, w.cU + q * ps, P, R) ||
        !encode_map<T, typename LB::WC>(fn, m + cps::kTmCV_B + q, w.cV + q * ps, P, R))
      return false;
  if (!encode_map<T, typename LB::WC>(fn, m + cps::kTmBU_B, w.bU, P, R) ||
      !encode_map<T, typename LB::WC>(fn, m + cps::kTmBV_B, w.bV, P, R) ||
      !encode_map<T, typename LB::WX>(fn, m + cps::kTmXU0_B, w.xU0, P, R) ||
      !encode_map<T, typename LB::WX>(fn, m + cps::kTmXU1_B, w.xU1, P, R) ||
      !encode_map<T, typename LB::WX>(fn, m + cps::kTmXV0_B, w.xV0, P, R) ||
      !encode_map<T, typename LB::WX>(fn, m + cps::kTmXV1_B, w.xV1, P, R))
    return false;
  return encode_map<double, LA::WU>(fn, m + cps::kTmU_A, v.u, P, R) &&
         encode_map<double, LA::WU>(fn, m + cps::kTmV_A, v.v, P, R) &&
         encode_map<double, LA::WP>(fn, m + cps::kTmP_A, v.p, P, R) &&
         encode_map<double, LA::WA>(fn, m + cps::kTmAlpha_A, v.alpha, P, M) &&
         encode_map<T, typename LC::WUx>(fn, m + cps::kTmXU0_C, w.xU0, P, R) &&
         encode_map<T, typename LC::WUx>(fn, m + cps::kTmXU1_C, w.xU1, P, R) &&
         encode_map<double, typename LC::WUd>(fn, m + cps::kTmU_C, v.u, P, R) &&
         encode_map<double, typename LC::WUd>(fn, m + cps::kTmDE_C, v.dE, P, R) &&
         encode_map<T, typename LC::WVx>(fn, m + cps::kTmXV0_C, w.xV0, P, R) &&
         encode_map<T, typename LC::WVx>(fn, m + cps::kTmXV1_C, w.xV1, P, R) &&
         encode_map<double, typename LC::WVd>(fn, m + cps::kTmV_C, v.v, P, R) &&
         encode_map<double, typename LC::WVd>(fn, m + cps::kTmDN_C, v.dN, P, R) &&
         encode_map<double, typename LC::WG>(fn, m + cps::kTmG_C, v.gamma, P, M) &&
         encode_map<T, typename LD::WX>(fn, m + cps::kTmPX_D, w.px, P, R) &&
         encode_map<double, typename LD::WO>(fn, m + cps::kTmP_D, v.p, P, R) &&
         encode_map<double, typename LD::WO>(fn, m + cps::kTmDE_D, v.dE, P, R) &&
         encode_map<double, typename LD::WO>(fn, m + cps::kTmUS_D, v.us, P, R) &&
         encode_map<double, typename LD::WO>(fn, m + cps::kTmDN_D, v.dN, P, R) &&
         encode_map<double, typename LD::WO>(fn, m + cps::kTmVS_D, v.vs, P, R) &&
         encode_map<double, typename LD::WG>(fn, m + cps::kTmG_D, v.gamma, P, M);
}

// The context's tensor maps, or false (the staged phases then copy element by
// element): no driver entry point, an encoding refused, or CPS_STAGING=elements
// in the environment (the element-wise path, for comparisons).
bool build_tensor_maps(cps_ctx* c) {
  const char* mode = std::getenv("CPS_STAGING");
  if (mode && std::strcmp(mode, "elements") == 0) return false;
  PFN_cuTensorMapEncodeTiled_v12000 fn = encode_tiled();
  if (!fn) return false;
  cps::TensorMap h[cps::kTmCount];
  std::memset(h, 0, sizeof(h));
  const bool ok = c->precision == CPS_MIXED ? fill_maps<float>(fn, c->view, c->view.f32, c->M, c->P, h)
                                            : fill_maps<double>(fn, c->view, c->view.f64, c->M, c->P, h);
  if (!ok) return false;
  return cudaMemcpyAsync(c->dtmaps, h, sizeof(h), cudaMemcpyHostToDevice, c->stream) == cudaSuccess &&
         cudaStreamSynchronize(c->stream) == cudaSuccess;
}

cps_status validate(const cps_desc* d) {
  if (!d) return fail(nullptr, CPS_ERR_ARG, "desc is NULL");
  if (d->M < 3 || d->N < 3) return fail(nullptr, CPS_ERR_ARG, "grid too small: need M >= 3 and N >= 3");
  if ((long long)d->M * d->N > (1LL << 28)) return fail(nullptr, CPS_ERR_ARG, "grid too large");
  if (!(d->hx > 0) || !(d->hy > 0) || !(d->rho > 0) || !(d->eta > 0))
    return fail(nullptr, CPS_ERR_ARG, "hx, hy, rho and eta must be positive");
  if (!(d->uvAlpha > 0) || !(d->pAlpha >= 0)) return fail(nullptr, CPS_ERR_ARG, "bad relaxation factors");
  if (d->maxPressureIter < 0 || d->maxMomentumIter < 0) return fail(nullptr, CPS_ERR_ARG, "negative iteration cap");
  if (d->precision != CPS_FP64 && d->precision != CPS_MIXED) return fail(nullptr, CPS_ERR_ARG, "bad precision");
  if (d->layout != CPS_ROW_MAJOR && d->layout != CPS_COL_MAJOR) return fail(nullptr, CPS_ERR_ARG, "bad layout");
  if (!d->alpha || !d->gamma) return fail(nullptr, CPS_ERR_ARG, "alpha and gamma are required");
  if (d->grid_ctas < 0) return fail(nullptr, CPS_ERR_ARG, "grid_ctas < 0");
  if (d->pcg_variant != CPS_PCG_REFERENCE && d->pcg_variant != CPS_PCG_SINGLE_REDUCTION)
    return fail(nullptr, CPS_ERR_ARG, "bad pcg_variant");
  if (d->momentum_explicit != 0 && d->momentum_explicit != 1)
    return fail(nullptr, CPS_ERR_ARG, "momentum_explicit must be 0 (implicit Jacobi) or 1 (explicit)");
  return CPS_OK;
}

// Copy a host rows x cols matrix (row- or column-major) into a pitched device plane.
bool upload_plane(cps_ctx* c, double* dst, const double* src, int rows, int cols, int layout) {
  if (layout == CPS_COL_MAJOR) {
    for (int i = 0; i < rows; ++i)
      for (int j = 0; j < cols; ++j) c->hstage[(size_t)i * cols + j] = src[(size_t)j * rows + i];
  } else {
    std::memcpy(c->hstage, src, sizeof(double) * (size_t)rows * cols);
  }
  if (!cuda_ok(c, cudaMemcpy2DAsync(dst, (size_t)c->P * 8, c->hstage, (size_t)cols * 8, (size_t)cols * 8, rows,
                                    cudaMemcpyHostToDevice, c->stream), "upload"))
    return false;
  return cuda_ok(c, cudaStreamSynchronize(c->stream), "upload sync");
}

// A device plane to copy out: rows x cols of a pitched plane into a host matrix.
struct PlaneOut {
  double* dst;
  const double* src;
  int rows, cols;
};

// Rows [row, row + rows) of a plane, from the stage to the caller's memory.
void write_out(const PlaneOut& pl, int row, int rows, const double* src, int layout) {
  if (layout == CPS_COL_MAJOR) {
    for (int i = 0; i < rows; ++i)
      for (int j = 0; j < pl.cols; ++j) pl.dst[(size_t)j * pl.rows + row + i] = src[(size_t)i * pl.cols + j];
  } else {
    std::memcpy(pl.dst + (size_t)row * pl.cols, src, sizeof(double) * (size_t)rows * pl.cols);
  }
}

// Copy planes to the caller's memory through the pinned stage.  Planes below
// kPipelinedPlane go one at a time; larger ones in chunks of rows: while one
// chunk's rows are written out the next chunks are on their way.  Several
// threads write from 4 MB on: memory that the caller has just allocated (every
// call through the Python binding) takes longer to fault in than to copy, and
// columns are written element by element.  By rows into memory already in use
// each thread costs more than it saves below about 14 MB, hence the ramp.
// B200's host, us for all eight fields by rows, used / fresh memory, one plane
// at a time -> this rule (-> chunks always, eight threads from 4 MB): 40 x 24
// 85 / 92 -> 85 / 92 (116 / 122), 500 x 250 700 / 1485 -> 780 / 705 (920 / 920),
// 700 x 350 1260 / 2800 -> 1100 / 1110 (1185 / 1250), 1000 x 500 2490 / 7400 ->
// 1730 / 2070 (1710 / 1980).  Slots below kDownloadSlot spend their time in
// the calls.
constexpr size_t kPipelinedPlane = size_t(384) << 10, kDownloadSlot = size_t(64) << 10;
constexpr int kDownloadThreads = 8, kDownloadDepth = 2;

int download_threads(size_t bytes, int layout) {
  if (bytes < size_t(4) << 20) return 1;
  return layout == CPS_COL_MAJOR ? kDownloadThreads : (int)std::min<size_t>(kDownloadThreads, 2 + bytes / (size_t(5) << 19));
}

bool download_planes(cps_ctx* c, const PlaneOut* planes, int n, int layout) {
  size_t bytes = 0;
  for (int k = 0; k < n; ++k) bytes += planes[k].dst ? sizeof(double) * (size_t)planes[k].rows * planes[k].cols : 0;
  if (bytes == 0) return true;
  const size_t stage = (size_t)(c->M + 1) * (c->N + 1);
  if (stage * sizeof(double) < kPipelinedPlane) {
    for (int k = 0; k < n; ++k) {
      const PlaneOut& pl = planes[k];
      const size_t w = sizeof(double) * pl.cols;
      if (!pl.dst) continue;
      if (!cuda_ok(c, cudaMemcpy2DAsync(c->hstage, w, pl.src, (size_t)c->P * 8, w, pl.rows, cudaMemcpyDeviceToHost, c->stream),
                   "download") ||
          !cuda_ok(c, cudaStreamSynchronize(c->stream), "download sync"))
        return false;
      write_out(pl, 0, pl.rows, c->hstage, layout);
    }
    return true;
  }
  int threads = download_threads(bytes, layout);
  if (threads > 1)
    threads = std::max(1, std::min({threads, (int)std::thread::hardware_concurrency() / 2,
                                    (int)(stage * sizeof(double) / (kDownloadDepth * kDownloadSlot))}));
  // slots of at least one row each (M >= 3: four rows at least)
  int depth = threads > 1 ? kDownloadDepth : 4;
  if (threads * depth > c->M + 1) { threads = 1; depth = 4; }
  const size_t slot = stage / ((size_t)threads * depth);
  struct Chunk { int plane, row, rows; };
  std::vector<Chunk> chunks;
  try {
    for (int k = 0; k < n; ++k) {
      if (!planes[k].dst) continue;
      const int per = (int)(slot / planes[k].cols);
      for (int r = 0; r < planes[k].rows; r += per) chunks.push_back({k, r, std::min(per, planes[k].rows - r)});
    }
  } catch (const std::exception&) {
    return cuda_ok(c, cudaErrorMemoryAllocation, "download");
  }
  std::atomic<int> failed{cudaSuccess};
  auto worker = [&](int t) {
    cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
    cudaError_t e = cudaSetDevice(c->device);
    for (int q = 0; q < depth && e == cudaSuccess; ++q) e = cudaEventCreateWithFlags(&ev[q], cudaEventDisableTiming);
    auto at = [&](int q) { return c->hstage + ((size_t)t * depth + q) * slot; };
    auto issue = [&](size_t m, int q) {
      const Chunk& h = chunks[m];
      const PlaneOut& pl = planes[h.plane];
      const size_t w = sizeof(double) * pl.cols;
      e = cudaMemcpy2DAsync(at(q), w, pl.src + (size_t)h.row * c->P, (size_t)c->P * 8, w, h.rows, cudaMemcpyDeviceToHost,
                            c->stream);
      if (e == cudaSuccess) e = cudaEventRecord(ev[q], c->stream);
    };
    size_t next = t;  // the next chunk to issue; this thread's chunks are t, t + threads, ...
    for (int q = 0; q < depth && next < chunks.size() && e == cudaSuccess; ++q, next += threads) issue(next, q);
    int q = 0;
    for (size_t m = t; m < chunks.size() && e == cudaSuccess; m += threads, q = (q + 1) % depth) {
      if ((e = cudaEventSynchronize(ev[q])) != cudaSuccess) break;
      const Chunk& h = chunks[m];
      const PlaneOut& pl = planes[h.plane];
      write_out(pl, h.row, h.rows, at(q), layout);
      if (next < chunks.size()) {
        issue(next, q);
        next += threads;
      }
    }
    if (e != cudaSuccess) failed = (int)e;
    for (cudaEvent_t x : ev)
      if (x) cudaEventDestroy(x);
  };
  std::vector<std::thread> pool;
  int started = 1;
  try {
    for (; started < threads; ++started) pool.emplace_back(worker, started);
  } catch (const std::exception&) {
    // fewer threads than asked for: this one takes their chunks below
  }
  worker(0);
  for (int t = started; t < threads; ++t) worker(t);
  for (std::thread& th : pool) th.join();
  // the stage is reused: no copy may be in flight (an error leaves some issued)
  const cudaError_t end = cudaStreamSynchronize(c->stream);
  return cuda_ok(c, (cudaError_t)failed.load(), "download") && cuda_ok(c, end, "download sync");
}

double* field_ptr(cps_ctx* c, int k) { return reinterpret_cast<double*>(c->slab) + (size_t)k * c->plane_elems; }

template <typename T>
void bind_inner(cps_ctx* c, cps::Inner<T>& w) {
  T* base = reinterpret_cast<T*>(c->slab + c->plane_elems * sizeof(double) * kFieldPlanes);
  auto pl = [&](int k) { return base + (size_t)k * c->plane_elems; };
  w.cU = pl(0); w.cV = pl(5);
  w.bU = pl(10); w.bV = pl(11);
  w.xU0 = pl(12); w.xU1 = pl(13); w.xV0 = pl(14); w.xV1 = pl(15);
  w.px = pl(16); w.pr = pl(17); w.pz = pl(18); w.pp0 = pl(19); w.pp1 = pl(20); w.pAp = pl(21);
  w.pdiag = pl(22); w.cx = pl(23); w.cy = pl(24);
}

void set_step_inputs(cps_ctx* c, double Uin) {
  c->view.Uin = Uin;
  c->view.maxVel = 3.0 * std::max(std::fabs(Uin), 0.1);  // iterations.cpp:104
}

// The single-design kernels of a storage type, each with the dynamic shared
// memory it needs: one per PCG form on the default path, with every option,
// and with the monitor and every option, then the one whose PCG runs on one
// cluster (8 x 32 tiles only).  One form each: with all of them in one kernel
// (136 bytes of spills; 0, 60 and 0 for the three forms) a late outer
// iteration took, us in FP64: monitored 39.1 instead of 35.9 (256 x 128), 81.0
// instead of 76.1 (512 x 256) and 132.3 instead of 128.6 (1000 x 500); with
// the pseudo-transient term 146.5 instead of 141.5 (500 x 250 network).
struct GridKernel {
  const void* fn;
  size_t smem;
};
template <typename T, bool Monitor, bool Pseudo, int Carry>
GridKernel grid_kernel() {
  return {(const void*)cps_grid_kernel<T, Monitor, Pseudo, Carry>, cps::kernel_smem_bytes<T, Carry, Monitor>()};
}
enum GridForm : int { kGridFew, kGridMany, kGridLarge, kGridForms };
enum GridKernels : int { kGridPlain = 0, kGridOptions = kGridForms, kGridMonitor = 2 * kGridForms, kGridKernels = 3 * kGridForms, kGridCluster = kGridKernels };
template <typename T>
GridKernel grid_kernel(int k) {
  switch (k) {
    case kGridPlain + kGridFew: return grid_kernel<T, false, false, cps::kFew>();
    case kGridPlain + kGridMany: return grid_kernel<T, false, false, cps::kMany>();
    case kGridPlain + kGridLarge: return grid_kernel<T, false, false, cps::kLarge>();
    case kGridOptions + kGridFew: return grid_kernel<T, false, true, cps::kFew | cps::kOptions>();
    case kGridOptions + kGridMany: return grid_kernel<T, false, true, cps::kMany | cps::kOptions>();
    case kGridOptions + kGridLarge: return grid_kernel<T, false, true, cps::kLarge | cps::kOptions>();
    case kGridMonitor + kGridFew: return grid_kernel<T, true, true, cps::kFew | cps::kOptions>();
    case kGridMonitor + kGridMany: return grid_kernel<T, true, true, cps::kMany | cps::kOptions>();
    case kGridMonitor + kGridLarge: return grid_kernel<T, true, true, cps::kLarge | cps::kOptions>();
#if CPS_TILE_J == 32
    case kGridCluster: return grid_kernel<T, false, false, cps::kCluster>();
#endif
  }
  return {nullptr, 0};
}
GridKernel grid_kernel_of(int precision, int k) {
  return precision == CPS_MIXED ? grid_kernel<float>(k) : grid_kernel<double>(k);
}

// Whether a design needs a kernel that carries the options.
bool has_options(const cps::DesignView& v) {
  return v.pseudo != 0 || v.momExplicit != 0 || v.pcgSingleReduction != 0 || v.stageSweeps != 0;
}

// The kernel of a context's next launch; `alone`: no other launch is in flight
// on the device.  Beside another launch a design of the cluster form takes the
// grid form, two CTAs to an SM and the same bits.  B200, channel 200 x 100, 60
// outer iterations, ms per solve over 1 / 2 / 3 / 6 host threads: always the
// cluster form 5.4 / 5.3 / 5.3 / 5.3, always the grid form 6.9 / 3.6 / 2.5 /
// 2.5, this rule 5.4 / 3.5 / 2.4 / 2.4.  (A launch under way keeps its form: a
// third context may wait for it to end once.)
int grid_kernel_for(const cps_ctx* c, bool alone) {
  const bool monitor = c->view.dpMonitor != 0, options = has_options(c->view);
  if (c->cluster && alone && !monitor && !options) return kGridCluster;
  const int form = c->precision == CPS_MIXED ? cps::pcg_form<float>(c->M, c->N, c->grid)
                                             : cps::pcg_form<double>(c->M, c->N, c->grid);
  return (monitor ? kGridMonitor : options ? kGridOptions : kGridPlain) +
         (form == cps::kFew ? kGridFew : form == cps::kMany ? kGridMany : kGridLarge);
}

// Dynamic shared memory of the persistent kernels (tile staging buffers).
size_t tile_smem_for(int precision) {
  return precision == CPS_MIXED ? cps::tile_smem_bytes<float>() : cps::tile_smem_bytes<double>();
}

// Let kernel fn use `bytes` of dynamic shared memory on the current device.
bool allow_smem(cps_ctx* c, const void* fn, size_t bytes) {
  return cuda_ok(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes), "smem attribute");
}

void to_step_out(const double* h, cps_step_out* o) {
  o->residU = h[0]; o->residV = h[1]; o->residMass = h[2]; o->residMassDof = h[3]; o->err = h[4];
  o->pIters = (int)h[5]; o->uSweeps = (int)h[6]; o->vSweeps = (int)h[7];
}

// The shared memory that every grid kernel is allowed, whichever of them needs
// it: one value, so that contexts on several threads never lower each other's.
size_t grid_smem(int precision) {
  size_t most = 0;
  for (int k = 0; k < kGridKernels; ++k) most = std::max(most, grid_kernel_of(precision, k).smem);
  return most;
}

// Before a context's first launch of a kernel (which loads it); the cluster
// form's is use_cluster's to prepare.
bool ready_grid(cps_ctx* c, int k) {
  if (k == kGridCluster || (c->ready >> k & 1u)) return true;
  if (!allow_smem(c, grid_kernel_of(c->precision, k).fn, grid_smem(c->precision))) return false;
  c->ready |= 1u << k;
  return true;
}

// The persistent kernel's launch: cooperative (all CTAs co-resident), in
// clusters where its PCG runs on one.
cudaError_t launch_grid(const cps_ctx* c, int k, void** args) {
  const GridKernel kern = grid_kernel_of(c->precision, k);
  const bool cluster = k == kGridCluster;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(cluster ? (unsigned)round_up(c->grid, cps::kClusterCtas) : (unsigned)c->grid);
  cfg.blockDim = dim3(cps::kThreads);
  cfg.dynamicSmemBytes = kern.smem;
  cfg.stream = c->stream;
  cfg.attrs = attr;
  cfg.numAttrs = cluster ? 2 : 1;
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cps::kClusterCtas;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  return cudaLaunchKernelExC(&cfg, kern.fn, args);
}

// Whether a design's PCG runs on one cluster: one tile per CTA, tiles enough
// for the cluster's CTAs and no more than its warps, a cap that leaves it
// iterations to run (the form costs one more grid barrier) and that it meets
// well inside the grid barrier's time limit, and room for the launch's
// clusters at one CTA per SM (seven of 16 CTAs on B200).
bool use_cluster(const cps_ctx* c, const cps_desc* d) {
  const GridKernel kern = grid_kernel_of(c->precision, kGridCluster);
  const int tiles = cps::pcg_tiles_of(c->M, c->N);
  if (!kern.fn || c->grid != tiles || tiles < cps::kClusterCtas || tiles > cps::kClusterTiles || d->maxPressureIter < 3 ||
      d->maxPressureIter > 100000)
    return false;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3((unsigned)round_up(tiles, cps::kClusterCtas));
  cfg.blockDim = dim3(cps::kThreads);
  cfg.dynamicSmemBytes = kern.smem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cps::kClusterCtas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  int clusters = 0;
  const bool ok = cudaFuncSetAttribute(kern.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kern.smem) == cudaSuccess &&
                  cudaFuncSetAttribute(kern.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                  cudaOccupancyMaxActiveClusters(&clusters, kern.fn, &cfg) == cudaSuccess &&
                  clusters * cps::kClusterCtas >= (int)cfg.gridDim.x;
  if (!ok) cudaGetLastError();  // the other forms need none of it
  return ok;
}

cps_status run(cps_ctx* c, int n_outer, int stop_on_conv, double eps, cps_step_out* hist, int* n_done,
               double* dp_history = nullptr, int* dp_converged = nullptr, bool ramp = false) {
  int done_total = 0;
  const bool monitor = c->view.dpMonitor != 0;
  const double target = c->view.Uin;
  if (dp_converged) *dp_converged = 0;
  while (done_total < n_outer) {
    int chunk = std::min(kHistChunk, n_outer - done_total);
    if (ramp && c->ramp_steps > 0) {
      // SIMPLE.cpp:303-307: one launch per ramp iteration, each with its own inlet velocity
      if (c->iter < c->ramp_steps) {
        chunk = 1;
        set_step_inputs(c, ((double)(c->iter + 1) / c->ramp_steps) * target);
      } else {
        set_step_inputs(c, target);
      }
    }
    cps::RunControl rc{chunk, stop_on_conv, eps, c->dhist, c->dndone, c->dstatus, c->iter,
                       monitor ? c->dplog : nullptr, c->dstatus + 2, c->grid};
    // the barrier and the flags
    if (!cuda_ok(c, cudaMemsetAsync(c->bar, 0, kFlagsAt + 4 * sizeof(int), c->stream), "memset"))
      return CPS_ERR_CUDA;
    void* args[] = {&c->view, &rc, &c->bar, &c->red};
    const cps::InFlight flight(c->device);
    c->kernel = grid_kernel_for(c, flight.alone());
    if (!ready_grid(c, c->kernel) || !cuda_ok(c, cudaEventRecord(c->ev0, c->stream), "event")) return CPS_ERR_CUDA;
    if (!cuda_ok(c, launch_grid(c, c->kernel, args), "cooperative launch")) return CPS_ERR_CUDA;
    if (!cuda_ok(c, cudaEventRecord(c->ev1, c->stream), "event")) return CPS_ERR_CUDA;
    if (monitor && dp_history &&
        !cuda_ok(c, cudaMemcpyAsync(c->hdplog, c->dplog, sizeof(double) * 4 * chunk, cudaMemcpyDeviceToHost,
                                    c->stream), "d2h"))
      return CPS_ERR_CUDA;
    if (!cuda_ok(c, cudaMemcpyAsync(c->hflags, c->dstatus, kHistAt - kFlagsAt + sizeof(double) * 8 * chunk,
                                    cudaMemcpyDeviceToHost, c->stream), "d2h"))
      return CPS_ERR_CUDA;
    if (!cuda_ok(c, cudaStreamSynchronize(c->stream), "kernel")) return CPS_ERR_CUDA;
    const int status = c->hflags[0], nd = c->hflags[1];
    float ms = 0.0f;
    if (cudaEventElapsedTime(&ms, c->ev0, c->ev1) == cudaSuccess) c->kernel_ms += ms;
    c->launches += 1;
    c->outer_done += nd;
    if (hist)
      for (int k = 0; k < nd; ++k) to_step_out(c->hhist + (size_t)8 * k, &hist[done_total + k]);
    if (monitor && dp_history) std::memcpy(dp_history + (size_t)4 * done_total, c->hdplog, sizeof(double) * 4 * nd);
    if (dp_converged && c->hflags[2]) *dp_converged = 1;
    c->iter += nd;
    done_total += nd;
    if (n_done) *n_done = done_total;
    if (status != cps::kStatusOk) {
      // Reset the barrier and status so the context stays usable.
      cudaMemsetAsync(c->bar, 0, sizeof(cps::GridBarrier), c->stream);
      cudaMemsetAsync(c->dstatus, 0, sizeof(int), c->stream);
      cudaStreamSynchronize(c->stream);
      if (status == cps::kStatusTimeout) return fail(c, CPS_ERR_TIMEOUT, "device grid barrier timed out");
      return fail(c, CPS_ERR_DIVERGED, "residual is not finite (solution diverged)");
    }
    if (nd < chunk) break;  // converged
  }
  if (ramp && c->ramp_steps > 0) set_step_inputs(c, target);
  return CPS_OK;
}

// Per-device scratch of cps_batch_solve, grown on demand and reused.
struct BatchWorkspace {
  int device = -1;
  size_t cap = 0;
  cps::BatchItem* items = nullptr;
  int* order = nullptr;
  int* queue = nullptr;
  cps::BatchResult* results = nullptr;
  cps::BatchItem* h_items = nullptr;
  int* h_order = nullptr;
  cps::BatchResult* h_results = nullptr;
  cps::GridBarrier* bars = nullptr;  // group kernel: one barrier, ring and slot pair per group
  double* rings = nullptr;
  int* slots = nullptr;
  int* plan = nullptr;    // wave kernel: per wave, first[groups + 1] then which[groups]
  int* h_plan = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};
std::mutex g_batch_mutex;
std::vector<BatchWorkspace> g_batch_ws;

BatchWorkspace* batch_workspace(int device, size_t n, std::string& err) {
  BatchWorkspace* ws = nullptr;
  for (auto& w : g_batch_ws)
    if (w.device == device) ws = &w;
  if (!ws) {
    g_batch_ws.emplace_back();
    ws = &g_batch_ws.back();
    ws->device = device;
    if (cudaEventCreate(&ws->ev0) != cudaSuccess || cudaEventCreate(&ws->ev1) != cudaSuccess ||
        cudaMalloc(&ws->bars, sizeof(cps::GridBarrier) * kMaxGridCtas) != cudaSuccess ||
        cudaMalloc(&ws->rings, sizeof(double) * cps::kRedSlots * kMaxGridCtas * cps::kRedWidth) != cudaSuccess ||
        cudaMalloc(&ws->slots, sizeof(int) * 2 * kMaxGridCtas) != cudaSuccess) {
      err = "batch workspace allocation failed";
      return nullptr;
    }
  }
  if (ws->cap < n) {
    cudaFree(ws->items); cudaFree(ws->order); cudaFree(ws->queue); cudaFree(ws->results); cudaFree(ws->plan);
    cudaFreeHost(ws->h_items); cudaFreeHost(ws->h_order); cudaFreeHost(ws->h_results); cudaFreeHost(ws->h_plan);
    ws->items = nullptr; ws->order = nullptr; ws->queue = nullptr; ws->results = nullptr; ws->plan = nullptr;
    ws->h_items = nullptr; ws->h_order = nullptr; ws->h_results = nullptr; ws->h_plan = nullptr;
    ws->cap = 0;
    const size_t cap = std::max<size_t>(n, 64);
    if (cudaMalloc(&ws->items, cap * sizeof(cps::BatchItem)) != cudaSuccess ||
        cudaMalloc(&ws->order, cap * sizeof(int)) != cudaSuccess || cudaMalloc(&ws->queue, 256) != cudaSuccess ||
        cudaMalloc(&ws->results, cap * sizeof(cps::BatchResult)) != cudaSuccess ||
        cudaMalloc(&ws->plan, 3 * cap * sizeof(int)) != cudaSuccess ||
        cudaMallocHost(&ws->h_plan, 3 * cap * sizeof(int)) != cudaSuccess ||
        cudaMallocHost(&ws->h_items, cap * sizeof(cps::BatchItem)) != cudaSuccess ||
        cudaMallocHost(&ws->h_order, cap * sizeof(int)) != cudaSuccess ||
        cudaMallocHost(&ws->h_results, cap * sizeof(cps::BatchResult)) != cudaSuccess) {
      err = "batch workspace allocation failed";
      return nullptr;
    }
    ws->cap = cap;
  }
  return ws;
}

}  // namespace

// The persistent kernels' grid barrier, told to expect `expect` CTAs: with more
// than the launch has, the count it waits for is never reached and the wait
// ends only by its time limit (cps_barrier_selftest).
__global__ void __launch_bounds__(cps::kThreads) cps_barrier_selftest_kernel(cps::GridBarrier* bar, int* status,
                                                                            unsigned expect) {
  cps::GridGroup g{bar, nullptr, status, blockIdx.x, expect, 0u, 0ull};
  g.sync();
}

namespace {

// The batch kernels of a storage type, by what their designs need.
struct BatchKernels {
  const void *cluster, *group, *wave;
};
template <typename T, bool Options, int Carry>
BatchKernels batch_kernels() {
  return {(const void*)cps_cluster_kernel<T, Options, Carry>, (const void*)cps_group_kernel<T, Options, Carry>,
          (const void*)cps_wave_kernel<T, Options, Carry>};
}
// ctas[k]: the CTAs of design k.  pcg_tiles<many> serves the designs of few
// tiles too: carrying one form costs them less than carrying two (group kernel
// with both: 84 bytes of spills, with the larger one 4).
template <typename T>
BatchKernels batch_kernels(cps_ctx* const* ctxs, const std::vector<int>& ctas, bool options) {
  if (options) return batch_kernels<T, true, cps::kAll>();
  int most = cps::kFew;
  for (size_t k = 0; k < ctas.size(); ++k) most = std::max(most, cps::pcg_form<T>(ctxs[k]->M, ctxs[k]->N, ctas[k]));
  if (most == cps::kFew) return batch_kernels<T, false, cps::kFew>();
  return most == cps::kMany ? batch_kernels<T, false, cps::kMany>() : batch_kernels<T, false, cps::kForms>();
}
BatchKernels batch_kernels(cps_ctx* const* ctxs, const std::vector<int>& ctas, bool options) {
  return ctxs[0]->precision == CPS_MIXED ? batch_kernels<float>(ctxs, ctas, options)
                                         : batch_kernels<double>(ctxs, ctas, options);
}

}  // namespace

extern "C" {

const char* cps_version(void) { return "cps 0.2 (sm_100a)"; }

cps_status cps_tile_shape(int* rows, int* cols) {
  if (!rows || !cols) return fail(nullptr, CPS_ERR_ARG, "null output");
  *rows = cps::kTileI;
  *cols = cps::kTileJ;
  return CPS_OK;
}

const char* cps_last_error(const cps_ctx* ctx) { return ctx ? ctx->err.c_str() : g_create_error.c_str(); }

cps_status cps_barrier_selftest(int device, int ctas, double* kernel_ms) {
  if (ctas < 1 || ctas > 1024) return fail(nullptr, CPS_ERR_ARG, "ctas must be in 1..1024");
  if (kernel_ms) *kernel_ms = 0.0;
  if (!cuda_ok(nullptr, cudaSetDevice(device), "cudaSetDevice")) return CPS_ERR_CUDA;
  cudaStream_t st = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  char* mem = nullptr;
  int status = -1;
  float ms = 0.0f;
  // counter at [0], status at [64]
  bool ok = cuda_ok(nullptr, cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking), "stream") &&
            cuda_ok(nullptr, cudaMalloc(&mem, 128), "device allocation") &&
            cuda_ok(nullptr, cudaEventCreate(&e0), "event") && cuda_ok(nullptr, cudaEventCreate(&e1), "event") &&
            cuda_ok(nullptr, cudaMemsetAsync(mem, 0, 128, st), "memset") &&
            cuda_ok(nullptr, cudaEventRecord(e0, st), "event");
  if (ok) {
    cps_barrier_selftest_kernel<<<ctas, cps::kThreads, 0, st>>>(reinterpret_cast<cps::GridBarrier*>(mem),
                                                                 reinterpret_cast<int*>(mem + 64), (unsigned)ctas + 1u);
    ok = cuda_ok(nullptr, cudaGetLastError(), "launch") && cuda_ok(nullptr, cudaEventRecord(e1, st), "event") &&
         cuda_ok(nullptr, cudaMemcpyAsync(&status, mem + 64, sizeof(int), cudaMemcpyDeviceToHost, st), "d2h") &&
         cuda_ok(nullptr, cudaStreamSynchronize(st), "barrier self-test") &&
         cuda_ok(nullptr, cudaEventElapsedTime(&ms, e0, e1), "event time");
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (mem) cudaFree(mem);
  if (st) cudaStreamDestroy(st);
  if (!ok) return CPS_ERR_CUDA;
  if (kernel_ms) *kernel_ms = ms;
  if (status == cps::kStatusTimeout) return fail(nullptr, CPS_ERR_TIMEOUT, "device grid barrier timed out");
  if (status == cps::kStatusOk) return CPS_OK;
  return fail(nullptr, CPS_ERR_STATE, "barrier self-test: unexpected device status");
}

cps_status cps_footprint(const cps_desc* desc, unsigned long long* bytes) {
  cps_status s = validate(desc);
  if (s != CPS_OK) return s;
  if (!bytes) return fail(nullptr, CPS_ERR_ARG, "bytes is NULL");
  *bytes = footprint_bytes(desc->M, desc->N, desc->precision, nullptr, nullptr);
  return CPS_OK;
}

cps_status cps_create(const cps_desc* d, cps_ctx** out) {
  if (!out) return fail(nullptr, CPS_ERR_ARG, "out is NULL");
  *out = nullptr;
  cps_status s = validate(d);
  if (s != CPS_OK) return s;
  cps_ctx* c = new (std::nothrow) cps_ctx();
  if (!c) return fail(nullptr, CPS_ERR_OOM, "host allocation failed");
  c->device = d->device;
  c->M = d->M;
  c->N = d->N;
  c->precision = d->precision;
  c->slab_bytes = footprint_bytes(d->M, d->N, d->precision, &c->plane_elems, &c->P);
  auto bail = [&](cps_status st) {
    g_create_error = c->err;
    cps_destroy(c);
    return st;
  };
  if (!cuda_ok(c, cudaSetDevice(d->device), "cudaSetDevice")) return bail(CPS_ERR_CUDA);
  if (!cuda_ok(c, cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking), "stream")) return bail(CPS_ERR_CUDA);
  cudaError_t e = cudaMalloc(&c->slab, c->slab_bytes);
  if (e != cudaSuccess) {
    cuda_ok(c, e, "cudaMalloc");
    return bail(CPS_ERR_OOM);
  }
  if (!cuda_ok(c, cudaMemsetAsync(c->slab, 0, c->slab_bytes, c->stream), "memset")) return bail(CPS_ERR_CUDA);
  if (!cuda_ok(c, cudaEventCreate(&c->ev0), "event") || !cuda_ok(c, cudaEventCreate(&c->ev1), "event"))
    return bail(CPS_ERR_CUDA);
  const size_t stage = (size_t)(d->M + 1) * (d->N + 1);
  if (!cuda_ok(c, cudaMallocHost(&c->hstage, stage * sizeof(double)), "pinned alloc") ||
      !cuda_ok(c, cudaMallocHost(&c->hflags, kHistAt - kFlagsAt + ((size_t)kHistChunk + 1) * 8 * sizeof(double)),
               "pinned alloc") ||
      !cuda_ok(c, cudaMallocHost(&c->hdplog, sizeof(double) * 4 * kHistChunk), "pinned alloc"))
    return bail(CPS_ERR_OOM);

  char* tail = c->slab + c->plane_elems * sizeof(double) * kFieldPlanes +
               round_up(c->plane_elems * elem_bytes(d->precision) * kInnerPlanes, 256);
  c->hhist = reinterpret_cast<double*>(reinterpret_cast<char*>(c->hflags) + (kHistAt - kFlagsAt));
  c->hplane = c->hhist + (size_t)kHistChunk * 8;
  c->bar = reinterpret_cast<cps::GridBarrier*>(tail);
  c->dstatus = reinterpret_cast<int*>(tail + kFlagsAt);  // [0] status, [1] n_done
  c->dndone = c->dstatus + 1;
  c->dhist = reinterpret_cast<double*>(tail + kHistAt);
  c->red = c->dhist + (size_t)kHistChunk * 8;
  c->dplog = c->red + (size_t)(cps::kRedSlots * cps::kRedWidth + cps::kPlaneSums) * kMaxGridCtas + 8;
  c->dpseudo = c->dplog + (size_t)4 * kHistChunk;
  c->dtmaps = reinterpret_cast<cps::TensorMap*>(round_up(reinterpret_cast<size_t>(c->dpseudo + 8), 128));

  cps::DesignView& v = c->view;
  v.M = d->M; v.N = d->N; v.P = c->P;
  v.conv = d->convectionScheme; v.maxPIter = d->maxPressureIter; v.maxMomIter = d->maxMomentumIter;
  v.pcgSingleReduction = d->pcg_variant == CPS_PCG_SINGLE_REDUCTION ? 1 : 0;
  v.momExplicit = d->momentum_explicit;
  v.hx = d->hx; v.hy = d->hy; v.rho = d->rho; v.uvAlpha = d->uvAlpha; v.pAlpha = d->pAlpha; v.pTol = d->pTol;
  // Derived constants, evaluated in the reference's operation order
  // (momentum_solver.cpp:166-191, 220-222, 261; jacobi_solver.cpp:41, 63).
  v.vol = d->hx * d->hy;
  v.De = d->eta * d->hy / d->hx;
  v.Dn = d->eta * d->hx / d->hy;
  const double sinkCoeff = (d->enableTwoPointFiveD && d->Ht_channel > 0.0)
                               ? d->twoPointFiveDSinkMultiplier * (5.0 * d->eta / (2.0 * d->Ht_channel * d->Ht_channel))
                               : 0.0;
  v.sinkDiag = sinkCoeff * v.vol;
  const double convScale = d->enableConvectionScaling ? (6.0 / 7.0) : 1.0;
  v.Fcx = convScale * d->rho * d->hy;
  v.Fcy = convScale * d->rho * d->hx;
  v.relax = (1.0 - d->uvAlpha) / d->uvAlpha;
  const double tolsq = d->momentumTol * d->momentumTol;
  v.rUvAlpha = 1.0 / d->uvAlpha;
  v.pStop = cps::pcg_stop(d->pTol);
  v.thrU = tolsq * (double)((d->M - 1) * (d->N - 2));
  v.thrV = tolsq * (double)((d->M - 2) * (d->N - 1));
  v.u = field_ptr(c, kU); v.v = field_ptr(c, kV); v.p = field_ptr(c, kP); v.pc = field_ptr(c, kPc);
  v.us = field_ptr(c, kUs); v.vs = field_ptr(c, kVs); v.dE = field_ptr(c, kDE); v.dN = field_ptr(c, kDN);
  v.alpha = field_ptr(c, kAlpha); v.gamma = field_ptr(c, kGamma);
  v.planeStride = (long long)c->plane_elems;
  std::memset(&v.f64, 0, sizeof(v.f64));
  std::memset(&v.f32, 0, sizeof(v.f32));
  if (d->precision == CPS_MIXED) bind_inner<float>(c, v.f32); else bind_inner<double>(c, v.f64);
  set_step_inputs(c, 0.0);
  v.tm = build_tensor_maps(c) ? c->dtmaps : nullptr;
  {
    // The Jacobi sweeps load straight from global memory: staging their tiles
    // by TMA gave the same bits but measured 0-1.5 % slower per outer
    // iteration (the sweeps are not bound by their loads' latency).
    // CPS_STAGE_SWEEPS=1 in the environment stages them (for comparisons).
    const char* sw = std::getenv("CPS_STAGE_SWEEPS");
    v.stageSweeps = (sw && std::strcmp(sw, "1") == 0) ? 1 : 0;
  }

  if (!upload_plane(c, v.alpha, d->alpha, d->M, d->N, d->layout) ||
      !upload_plane(c, v.gamma, d->gamma, d->M, d->N, d->layout))
    return bail(CPS_ERR_CUDA);

  // Persistent grid: co-resident CTAs, at most one per tile of the design.  The
  // kernels are interchangeable within a design, so the grid is what all of
  // them allow: their launch bounds allow CPS_MIN_BLOCKS CTAs per SM, and the
  // shared memory of the largest is asked of one of them.  (Asking every kernel
  // loads every kernel: the first context of a process took 9.3 instead of
  // 7.5 ms, later ones 2.9 instead of 2.6 ms.)
  int per_sm = 0, sms = 0;
  const size_t most = grid_smem(d->precision);
  const GridKernel any = grid_kernel_of(d->precision, kGridPlain + kGridFew);
  if (!allow_smem(c, any.fn, most) ||
      !cuda_ok(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, any.fn, cps::kThreads, most), "occupancy"))
    return bail(CPS_ERR_CUDA);
  per_sm = std::min(per_sm, CPS_MIN_BLOCKS);
  if (!cuda_ok(c, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d->device), "attribute"))
    return bail(CPS_ERR_CUDA);
  if (per_sm < 1) return bail(fail(c, CPS_ERR_CUDA, "persistent kernel does not fit on an SM"));
  const int tiles = ((d->M - 1 + cps::kTileI - 1) / cps::kTileI) * ((d->N - 1 + cps::kTileJ - 1) / cps::kTileJ);
  // Default: the fewest rounds of tiles per CTA the co-resident CTAs allow,
  // with the tiles spread evenly (every CTA takes part in every barrier).
  const int cap = std::min(sms * per_sm, kMaxGridCtas);
  const int rounds = (tiles + cap - 1) / cap;
  int grid = d->grid_ctas > 0 ? d->grid_ctas : (tiles + rounds - 1) / rounds;
  grid = std::min(grid, cap);
  grid = std::max(1, std::min(grid, tiles));
  c->grid = grid;
  c->cluster = use_cluster(c, d);
  if (!ready_grid(c, grid_kernel_for(c, true))) return bail(CPS_ERR_CUDA);
  *out = c;
  return CPS_OK;
}

void cps_destroy(cps_ctx* c) {
  if (!c) return;
  if (c->stream) cudaStreamSynchronize(c->stream);
  if (c->slab) cudaFree(c->slab);
  if (c->hstage) cudaFreeHost(c->hstage);
  if (c->hflags) cudaFreeHost(c->hflags);
  if (c->hdplog) cudaFreeHost(c->hdplog);
  if (c->ddphist) cudaFree(c->ddphist);
  if (c->ev0) cudaEventDestroy(c->ev0);
  if (c->ev1) cudaEventDestroy(c->ev1);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

cps_status cps_upload_geometry(cps_ctx* c, const double* alpha, const double* gamma, int layout) {
  if (!c || !alpha || !gamma) return fail(c, CPS_ERR_ARG, "ctx, alpha and gamma are required");
  if (layout != CPS_ROW_MAJOR && layout != CPS_COL_MAJOR) return fail(c, CPS_ERR_ARG, "bad layout");
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  if (!upload_plane(c, c->view.alpha, alpha, c->M, c->N, layout) ||
      !upload_plane(c, c->view.gamma, gamma, c->M, c->N, layout))
    return CPS_ERR_CUDA;
  return CPS_OK;
}

cps_status cps_reset_fields(cps_ctx* c) {
  if (!c) return fail(nullptr, CPS_ERR_ARG, "ctx is NULL");
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  // Planes u .. dN are contiguous at the start of the slab.
  if (!cuda_ok(c, cudaMemsetAsync(c->slab, 0, c->plane_elems * sizeof(double) * (kDN + 1), c->stream), "memset"))
    return CPS_ERR_CUDA;
  c->iter = 0;
  if (c->view.pseudo && !write_pseudo_state(c, c->pseudo_start, 0.0, 1.0, 0)) return CPS_ERR_CUDA;
  return CPS_OK;
}

cps_status cps_pseudo_defaults(cps_pseudo* p, double target_velocity) {
  if (!p) return fail(nullptr, CPS_ERR_ARG, "p is NULL");
  cps_pseudo q;
  std::memset(&q, 0, sizeof(q));
  // SIMPLE.h:255-313
  q.enable = 0;
  q.use_local = 1;
  q.enable_ser = 1;
  q.enable_line_search = 1;
  q.enable_cfl_ramp = 1;
  q.ser_use_max_resid = 0;
  q.ser_min_iter = 10;
  q.ls_max_tries = 4;
  q.target_velocity = target_velocity;
  q.time_step_multiplier = 0.01;
  q.min_pseudo_speed = 0.05;
  q.pseudo_cfl = 0.1;
  q.cfl_initial = 0.1;
  q.cfl_max = 30.0;
  q.cfl_ramp_start_res = 1e-4;
  q.cfl_ramp_exponent = 0.8;
  q.cfl_ramp_smooth = 0.1;
  q.ser_cfl_min = 0.1;
  q.ser_cfl_max = 5.0;
  q.ser_smooth = 0.5;
  q.ser_max_increase = 1.1;
  q.ser_max_decrease = 0.7;
  q.ls_alpha_min = 0.1;
  q.ls_alpha_reduce = 0.3;
  q.ls_resid_increase_tol = 1.01;
  *p = q;
  return CPS_OK;
}

cps_status cps_set_pseudo(cps_ctx* c, const cps_pseudo* p) {
  if (!c) return fail(nullptr, CPS_ERR_ARG, "ctx is NULL");
  cps::DesignView& v = c->view;
  if (!p || !p->enable) {
    v.pseudo = 0;
    return CPS_OK;
  }
  const double reals[] = {p->time_step, p->target_velocity, p->time_step_multiplier, p->min_pseudo_speed, p->pseudo_cfl,
                          p->cfl_initial, p->cfl_max, p->cfl_ramp_start_res, p->cfl_ramp_exponent,
                          p->cfl_ramp_smooth, p->ser_cfl_min, p->ser_cfl_max, p->ser_smooth, p->ser_max_increase,
                          p->ser_max_decrease, p->ls_alpha_min, p->ls_alpha_reduce, p->ls_resid_increase_tol};
  for (double x : reals)
    if (!std::isfinite(x)) return fail(c, CPS_ERR_ARG, "pseudo-transient parameters must be finite");
  if (!(p->time_step_multiplier > 0.0 || p->time_step > 0.0) || p->ser_min_iter < 0 || p->ls_max_tries < 0)
    return fail(c, CPS_ERR_ARG,
                "pseudo-transient: time_step or time_step_multiplier > 0, ser_min_iter >= 0, ls_max_tries >= 0");
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  v.pseudoLocal = p->use_local ? 1 : 0;
  v.serOn = p->enable_ser ? 1 : 0;
  v.lsOn = p->enable_line_search ? 1 : 0;
  v.rampOn = p->enable_cfl_ramp ? 1 : 0;
  v.serUseMax = p->ser_use_max_resid ? 1 : 0;
  v.serMinIter = p->ser_min_iter;
  v.lsMaxTries = p->ls_max_tries;
  // SIMPLE.cpp:68-70, in the reference's operation order
  const double domainLength = c->N * v.hx;
  const double velRef = std::max(p->target_velocity, 1e-6);
  v.timeStep = p->time_step > 0.0 ? p->time_step : p->time_step_multiplier * domainLength / velRef;
  v.minPseudoSpeed = p->min_pseudo_speed;
  v.hChar = std::min(v.hx, v.hy);  // momentum_solver.cpp:190, iterations.cpp:189
  v.cflInitial = p->cfl_initial;
  v.cflMax = p->cfl_max;
  v.rampStartRes = p->cfl_ramp_start_res;
  v.rampExponent = p->cfl_ramp_exponent;
  v.rampSmooth = p->cfl_ramp_smooth;
  v.serCFLMin = p->ser_cfl_min;
  v.serCFLMax = p->ser_cfl_max;
  v.serSmooth = p->ser_smooth;
  v.serMaxIncrease = p->ser_max_increase;
  v.serMaxDecrease = p->ser_max_decrease;
  v.lsAlphaMin = p->ls_alpha_min;
  v.lsAlphaReduce = p->ls_alpha_reduce;
  v.lsTol = p->ls_resid_increase_tol;
  v.pseudoState = c->dpseudo;
  // the constructor starts the ramp at pseudoCFLInitial (SIMPLE.cpp:78-82)
  c->pseudo_start = p->enable_cfl_ramp ? p->cfl_initial : p->pseudo_cfl;
  if (!write_pseudo_state(c, c->pseudo_start, 0.0, 1.0, 0)) return CPS_ERR_CUDA;
  v.pseudo = 1;
  return CPS_OK;
}

cps_status cps_get_pseudo_state(cps_ctx* c, cps_pseudo_state* state) {
  if (!c || !state) return fail(c, CPS_ERR_ARG, "ctx and state are required");
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  double h[4];
  if (!cuda_ok(c, cudaMemcpyAsync(h, c->dpseudo, sizeof(h), cudaMemcpyDeviceToHost, c->stream), "d2h") ||
      !cuda_ok(c, cudaStreamSynchronize(c->stream), "d2h"))
    return CPS_ERR_CUDA;
  state->pseudo_cfl = h[0];
  state->ser_resid_prev = h[1];
  state->ls_alpha = h[2];
  state->ls_backtracks = (int)h[3];
  state->pad = 0;
  return CPS_OK;
}

cps_status cps_set_pseudo_state(cps_ctx* c, const cps_pseudo_state* state) {
  if (!c || !state) return fail(c, CPS_ERR_ARG, "ctx and state are required");
  if (!std::isfinite(state->pseudo_cfl) || !std::isfinite(state->ser_resid_prev) || !std::isfinite(state->ls_alpha))
    return fail(c, CPS_ERR_ARG, "pseudo state must be finite");
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  return write_pseudo_state(c, state->pseudo_cfl, state->ser_resid_prev, state->ls_alpha, state->ls_backtracks)
             ? CPS_OK
             : CPS_ERR_CUDA;
}

cps_status cps_last_pcg_form(const cps_ctx* c, int* form) {
  if (!c || !form) return fail(nullptr, CPS_ERR_ARG, "ctx and form are required");
  *form = c->kernel < 0                ? CPS_PCG_FORM_NONE
          : c->kernel == kGridCluster ? CPS_PCG_FORM_CLUSTER
                                      : CPS_PCG_FORM_FEW + c->kernel % kGridForms;
  return CPS_OK;
}

cps_status cps_get_stream(cps_ctx* c, void** stream) {
  if (!c || !stream) return fail(c, CPS_ERR_ARG, "ctx and stream are required");
  *stream = (void*)c->stream;
  return CPS_OK;
}

cps_status cps_kernel_timing(cps_ctx* c, double* kernel_ms, long long* launches, long long* outer_iterations,
                             int reset) {
  if (!c) return fail(nullptr, CPS_ERR_ARG, "ctx is NULL");
  if (kernel_ms) *kernel_ms = c->kernel_ms;
  if (launches) *launches = c->launches;
  if (outer_iterations) *outer_iterations = c->outer_done;
  if (reset) { c->kernel_ms = 0.0; c->launches = 0; c->outer_done = 0; }
  return CPS_OK;
}

cps_status cps_upload_fields(cps_ctx* c, const double* u, const double* v, const double* p, int layout) {
  if (!c) return fail(nullptr, CPS_ERR_ARG, "ctx is NULL");
  if (layout != CPS_ROW_MAJOR && layout != CPS_COL_MAJOR) return fail(c, CPS_ERR_ARG, "bad layout");
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  if (u && !upload_plane(c, c->view.u, u, c->M + 1, c->N, layout)) return CPS_ERR_CUDA;
  if (v && !upload_plane(c, c->view.v, v, c->M, c->N + 1, layout)) return CPS_ERR_CUDA;
  if (p && !upload_plane(c, c->view.p, p, c->M + 1, c->N + 1, layout)) return CPS_ERR_CUDA;
  return CPS_OK;
}

cps_status cps_step(cps_ctx* c, const cps_step_in* in, cps_step_out* out) {
  if (!c || !in) return fail(c, CPS_ERR_ARG, "ctx and in are required");
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  set_step_inputs(c, in->inletVelocity);
  int nd = 0;
  cps_step_out tmp;
  return run(c, 1, 0, 0.0, out ? out : &tmp, &nd);
}

cps_status cps_solve(cps_ctx* c, double inletVelocity, int max_outer, double eps, cps_step_out* history,
                     int* n_done) {
  if (!c) return fail(nullptr, CPS_ERR_ARG, "ctx is NULL");
  if (max_outer < 0) return fail(c, CPS_ERR_ARG, "max_outer < 0");
  if (n_done) *n_done = 0;
  if (max_outer == 0) return CPS_OK;
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  set_step_inputs(c, inletVelocity);
  return run(c, max_outer, eps > 0.0 ? 1 : 0, eps, history, n_done, nullptr, nullptr, true);
}

cps_status cps_set_inlet_ramp(cps_ctx* c, int ramp_steps) {
  if (!c) return fail(nullptr, CPS_ERR_ARG, "ctx is NULL");
  if (ramp_steps < 0) return fail(c, CPS_ERR_ARG, "ramp_steps < 0");
  c->ramp_steps = ramp_steps;
  return CPS_OK;
}

cps_status cps_set_dp_monitor(cps_ctx* c, const cps_dp_monitor* m) {
  if (!c) return fail(nullptr, CPS_ERR_ARG, "ctx is NULL");
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  c->iter = 0;
  if (!m) {
    c->view.dpMonitor = 0;
    c->view.dpGate = 0;
    return CPS_OK;
  }
  if (m->window < 1 || m->slope_window < 0 || m->ramp_steps < 0 || !(m->percent >= 0.0))
    return fail(c, CPS_ERR_ARG, "dp monitor: window >= 1, slope_window >= 0, ramp_steps >= 0, percent >= 0");
  const size_t slots = (size_t)m->window + (size_t)(m->slope_gate ? m->slope_window : 0);
  const size_t most = c->precision == CPS_MIXED ? cps::window_values<float>() : cps::window_values<double>();
  if (slots > most)
    return fail(c, CPS_ERR_ARG, "dp monitor: window + slope_window exceeds " + std::to_string(most) + " values");
  if (c->ddphist) cudaFree(c->ddphist);
  c->ddphist = nullptr;
  if (!cuda_ok(c, cudaMalloc(&c->ddphist, std::max<size_t>(slots, 1) * sizeof(double)), "cudaMalloc")) return CPS_ERR_OOM;
  if (!cuda_ok(c, cudaMemset(c->ddphist, 0, std::max<size_t>(slots, 1) * sizeof(double)), "memset")) return CPS_ERR_CUDA;
  cps::DesignView& v = c->view;
  v.dpMonitor = 1;
  v.dpGate = m->gate ? 1 : 0;
  v.dpWindow = m->window;
  v.dpSlopeGate = m->slope_gate ? 1 : 0;
  v.dpSlopeWindow = m->slope_gate ? m->slope_window : 0;
  v.dpRampSteps = m->ramp_steps;
  v.dpPercent = m->percent;
  v.dpSlopeMaxDelta = m->slope_max_delta;
  v.xPlane[0] = m->x_core_in;
  v.xPlane[1] = m->x_core_out;
  v.xPlane[2] = 0.0;
  v.xPlane[3] = (double)c->N * v.hx;  // domainXMax = N * hx (SIMPLE.cpp:250)
  v.dpHist = c->ddphist;
  return CPS_OK;
}

cps_status cps_solve_monitored(cps_ctx* c, double inletVelocity, int max_outer, double eps, cps_step_out* history,
                               double* dp_history, int* n_done, int* dp_converged) {
  if (!c) return fail(nullptr, CPS_ERR_ARG, "ctx is NULL");
  if (max_outer < 0) return fail(c, CPS_ERR_ARG, "max_outer < 0");
  if (!c->view.dpMonitor) return fail(c, CPS_ERR_ARG, "no pressure-drop monitor set (cps_set_dp_monitor)");
  if (n_done) *n_done = 0;
  if (dp_converged) *dp_converged = 0;
  if (max_outer == 0) return CPS_OK;
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  set_step_inputs(c, inletVelocity);
  return run(c, max_outer, eps > 0.0 ? 1 : 0, eps, history, n_done, dp_history, dp_converged, true);
}

cps_status cps_batch_solve(cps_ctx* const* ctxs, int n, const double* inletVelocity, const cps_batch_opts* opts,
                           cps_batch_result* results, double* kernel_ms) {
  if (!ctxs || n <= 0 || !opts || !results) return fail(nullptr, CPS_ERR_ARG, "ctxs, n > 0, opts and results required");
  if (opts->max_outer < 0) return fail(nullptr, CPS_ERR_ARG, "max_outer < 0");
  const int cl = opts->cluster_ctas > 0 ? opts->cluster_ctas : 8;
  if (cl > 16) return fail(nullptr, CPS_ERR_ARG, "cluster_ctas must be <= 16");
  cps_ctx* c0 = ctxs[0];
  for (int k = 0; k < n; ++k) {
    if (!ctxs[k]) return fail(nullptr, CPS_ERR_ARG, "NULL context in batch");
    if (ctxs[k]->device != c0->device || ctxs[k]->precision != c0->precision)
      return fail(nullptr, CPS_ERR_ARG, "a batch needs one device and one precision");
  }
  std::lock_guard<std::mutex> lock(g_batch_mutex);
  if (!cuda_ok(c0, cudaSetDevice(c0->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  const cps::InFlight flight(c0->device);
  std::string err;
  BatchWorkspace* ws = batch_workspace(c0->device, (size_t)n, err);
  if (!ws) return fail(c0, CPS_ERR_OOM, err);
  // The batch kernels carry the options (the pseudo-transient term and the CFL
  // controllers among them) only when a design of the batch has one on (a
  // separate instantiation: compiled in, they slow every batched outer
  // iteration by a quarter).
  bool options = false;
  for (int k = 0; k < n; ++k) {
    cps_ctx* c = ctxs[k];
    set_step_inputs(c, inletVelocity ? inletVelocity[k] : c->view.Uin);
    cps::BatchItem& it = ws->h_items[k];
    std::memset(&it, 0, sizeof(it));
    it.view = c->view;
    it.view.dpMonitor = 0;  // the pressure-drop monitor runs in cps_solve/cps_solve_monitored only
    it.n_outer = opts->max_outer;
    it.stop_on_conv = opts->eps > 0.0 ? 1 : 0;
    it.eps = opts->eps;
    it.hist = c->dhist;
    it.hist_cap = kHistChunk;
    it.iter0 = c->iter;
    options = options || has_options(c->view);
  }
  std::vector<int> ord(n);
  std::iota(ord.begin(), ord.end(), 0);
  if (opts->order_by_size)
    std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) {
      return (long long)ctxs[a]->M * ctxs[a]->N > (long long)ctxs[b]->M * ctxs[b]->N;
    });
  std::copy(ord.begin(), ord.end(), ws->h_order);
  cudaStream_t st = c0->stream;
  if (!cuda_ok(c0, cudaMemcpyAsync(ws->items, ws->h_items, sizeof(cps::BatchItem) * n, cudaMemcpyHostToDevice, st),
               "h2d") ||
      !cuda_ok(c0, cudaMemcpyAsync(ws->order, ws->h_order, sizeof(int) * n, cudaMemcpyHostToDevice, st), "h2d") ||
      !cuda_ok(c0, cudaMemsetAsync(ws->queue, 0, sizeof(int), st), "memset") ||
      !cuda_ok(c0, cudaMemsetAsync(ws->results, 0, sizeof(cps::BatchResult) * n, st), "memset"))
    return CPS_ERR_CUDA;
  if (opts->tiles_per_cta > 0) {
    // Groups sized to their designs, packed into waves (first fit, largest
    // first); one cooperative launch per wave, all CTAs of a wave co-resident.
    // (every batch kernel fits the SM as often as every other: they share the shared memory and launch bounds)
    const void* wk = batch_kernels(ctxs, {}, options).wave;
    int per_sm = 0, sms = 0;
    const size_t tsm = tile_smem_for(c0->precision);
    if (!allow_smem(c0, wk, tsm) ||
        !cuda_ok(c0, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, wk, cps::kThreads, tsm), "occupancy") ||
        !cuda_ok(c0, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c0->device), "attribute"))
      return CPS_ERR_CUDA;
    const int max_ctas = std::min(sms * per_sm, kMaxGridCtas);
    if (max_ctas < 1) return fail(c0, CPS_ERR_CUDA, "wave kernel does not fit on an SM");
    std::vector<int> ctas(n);
    for (int k = 0; k < n; ++k) {
      const long long tiles = (long long)((ctxs[k]->M - 1 + cps::kTileI - 1) / cps::kTileI) *
                              ((ctxs[k]->N - 1 + cps::kTileJ - 1) / cps::kTileJ);
      ctas[k] = (int)std::max(1LL, std::min<long long>(max_ctas, (tiles + opts->tiles_per_cta - 1) / opts->tiles_per_cta));
    }
    wk = batch_kernels(ctxs, ctas, options).wave;
    if (!allow_smem(c0, wk, tsm)) return CPS_ERR_CUDA;
    std::vector<int> byc(n);
    std::iota(byc.begin(), byc.end(), 0);
    std::stable_sort(byc.begin(), byc.end(), [&](int a, int b) { return ctas[a] > ctas[b]; });
    std::vector<std::vector<int>> waves;
    std::vector<int> room;
    for (int k : byc) {
      size_t w = 0;
      while (w < waves.size() && room[w] < ctas[k]) ++w;
      if (w == waves.size()) { waves.emplace_back(); room.push_back(max_ctas); }
      waves[w].push_back(k);
      room[w] -= ctas[k];
    }
    // plan: for each wave, first[G + 1] then which[G]; at most 3n ints
    std::vector<size_t> at(waves.size());
    size_t pos = 0;
    for (size_t w = 0; w < waves.size(); ++w) {
      at[w] = pos;
      int* f = ws->h_plan + pos;
      const int G = (int)waves[w].size();
      f[0] = 0;
      for (int q = 0; q < G; ++q) {
        f[q + 1] = f[q] + ctas[waves[w][q]];
        f[G + 1 + q] = waves[w][q];
      }
      pos += 2 * (size_t)G + 1;
    }
    if (!cuda_ok(c0, cudaMemcpyAsync(ws->plan, ws->h_plan, sizeof(int) * pos, cudaMemcpyHostToDevice, st), "h2d"))
      return CPS_ERR_CUDA;
    const cps::BatchItem* items = ws->items;
    cps::BatchResult* res = ws->results;
    if (!cuda_ok(c0, cudaEventRecord(ws->ev0, st), "event")) return CPS_ERR_CUDA;
    for (size_t w = 0; w < waves.size(); ++w) {
      int G = (int)waves[w].size();
      const int* first = ws->plan + at[w];
      const int* which = first + G + 1;
      const int grid = ws->h_plan[at[w] + G];
      if (!cuda_ok(c0, cudaMemsetAsync(ws->bars, 0, sizeof(cps::GridBarrier) * G, st), "memset")) return CPS_ERR_CUDA;
      void* args[] = {&items, &first, &which, &G, &res, &ws->bars, &ws->rings};
      if (!cuda_ok(c0, cudaLaunchCooperativeKernel(wk, dim3(grid), dim3(cps::kThreads), args, tsm, st),
                   "cooperative wave launch"))
        return CPS_ERR_CUDA;
    }
  } else if (opts->group_ctas > 0) {
    // Groups of CTAs in one cooperative launch (all CTAs co-resident).
    const void* gk = batch_kernels(ctxs, std::vector<int>(n, opts->group_ctas), options).group;
    int per_sm = 0, sms = 0;
    const size_t tsm = tile_smem_for(c0->precision);
    if (!allow_smem(c0, gk, tsm) ||
        !cuda_ok(c0, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gk, cps::kThreads, tsm), "occupancy") ||
        !cuda_ok(c0, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c0->device), "attribute"))
      return CPS_ERR_CUDA;
    const int K = opts->group_ctas;
    const int max_ctas = std::min(sms * per_sm, kMaxGridCtas);
    if (K > max_ctas) return fail(c0, CPS_ERR_ARG, "group_ctas exceeds the co-resident CTAs of the device");
    int groups = std::min(max_ctas / K, n);
    if (opts->max_clusters > 0) groups = std::min(groups, opts->max_clusters);
    groups = std::max(groups, 1);
    if (!cuda_ok(c0, cudaMemsetAsync(ws->bars, 0, sizeof(cps::GridBarrier) * groups, st), "memset") ||
        !cuda_ok(c0, cudaMemsetAsync(ws->slots, 0, sizeof(int) * 2 * groups, st), "memset"))
      return CPS_ERR_CUDA;
    const cps::BatchItem* items = ws->items;
    const int* order = ws->order;
    int* queue = ws->queue;
    cps::BatchResult* res = ws->results;
    int nn = n, kk = K;
    void* args[] = {&items, &order, &nn, &queue, &res, &ws->bars, &ws->rings, &ws->slots, &kk};
    if (!cuda_ok(c0, cudaEventRecord(ws->ev0, st), "event")) return CPS_ERR_CUDA;
    if (!cuda_ok(c0, cudaLaunchCooperativeKernel(gk, dim3(groups * K), dim3(cps::kThreads), args, tsm, st),
                 "cooperative group launch"))
      return CPS_ERR_CUDA;
  } else {
  const void* kern = batch_kernels(ctxs, std::vector<int>(n, cl), options).cluster;
  if (cl > 8 &&
      !cuda_ok(c0, cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), "attr"))
    return CPS_ERR_CUDA;
  if (!allow_smem(c0, kern, tile_smem_for(c0->precision))) return CPS_ERR_CUDA;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(cps::kThreads);
  cfg.dynamicSmemBytes = tile_smem_for(c0->precision);
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(cl * 64);
  int max_clusters = 0;
  if (!cuda_ok(c0, cudaOccupancyMaxActiveClusters(&max_clusters, kern, &cfg), "cluster occupancy"))
    return CPS_ERR_CUDA;
  if (max_clusters < 1) return fail(c0, CPS_ERR_CUDA, "cluster configuration does not fit");
  int clusters = std::min(max_clusters, n);
  if (opts->max_clusters > 0) clusters = std::min(clusters, opts->max_clusters);
  cfg.gridDim = dim3(cl * clusters);
  const cps::BatchItem* items = ws->items;
  const int* order = ws->order;
  int* queue = ws->queue;
  cps::BatchResult* res = ws->results;
  if (!cuda_ok(c0, cudaEventRecord(ws->ev0, st), "event")) return CPS_ERR_CUDA;
  void* args[] = {&items, &order, &n, &queue, &res};
  if (!cuda_ok(c0, cudaLaunchKernelExC(&cfg, kern, args), "cluster launch")) return CPS_ERR_CUDA;
  }
  if (!cuda_ok(c0, cudaEventRecord(ws->ev1, st), "event") ||
      !cuda_ok(c0, cudaMemcpyAsync(ws->h_results, ws->results, sizeof(cps::BatchResult) * n, cudaMemcpyDeviceToHost,
                                   st), "d2h") ||
      !cuda_ok(c0, cudaStreamSynchronize(st), "batch kernel"))
    return CPS_ERR_CUDA;
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, ws->ev0, ws->ev1);
  if (kernel_ms) *kernel_ms = ms;
  cps_status status = CPS_OK;
  for (int k = 0; k < n; ++k) {
    const cps::BatchResult& r = ws->h_results[k];
    results[k].n_done = r.n_done;
    results[k].converged = r.converged;
    results[k].status = r.status == cps::kStatusOk        ? CPS_OK
                        : r.status == cps::kStatusTimeout ? CPS_ERR_TIMEOUT
                                                          : CPS_ERR_DIVERGED;
    to_step_out(r.last, &results[k].last);
    ctxs[k]->outer_done += r.n_done;
    ctxs[k]->iter += r.n_done;
    if (r.status != cps::kStatusOk) {
      status = (cps_status)results[k].status;
      ctxs[k]->err = r.status == cps::kStatusTimeout ? "device group barrier timed out"
                                                     : "residual is not finite (solution diverged)";
    }
  }
  c0->kernel_ms += ms;
  c0->launches += 1;
  if (status != CPS_OK) g_create_error = "at least one design diverged; see results[k].status";
  return status;
}

cps_status cps_get_history(cps_ctx* c, int n, cps_step_out* history) {
  if (!c || !history || n < 0 || n > kHistChunk) return fail(c, CPS_ERR_ARG, "bad history request");
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  if (n == 0) return CPS_OK;
  if (!cuda_ok(c, cudaMemcpyAsync(c->hhist, c->dhist, sizeof(double) * 8 * n, cudaMemcpyDeviceToHost, c->stream),
               "d2h") ||
      !cuda_ok(c, cudaStreamSynchronize(c->stream), "sync"))
    return CPS_ERR_CUDA;
  for (int k = 0; k < n; ++k) to_step_out(c->hhist + (size_t)8 * k, &history[k]);
  return CPS_OK;
}

cps_status cps_sample_plane(cps_ctx* c, double x, cps_plane* out) {
  if (!c || !out) return fail(c, CPS_ERR_ARG, "ctx and out are required");
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  cps_plane_kernel<<<1, cps::kThreads, 0, c->stream>>>(c->view, x, c->hplane);
  if (!cuda_ok(c, cudaGetLastError(), "plane launch") || !cuda_ok(c, cudaStreamSynchronize(c->stream), "plane"))
    return CPS_ERR_CUDA;
  out->flowArea = c->hplane[0]; out->massFlux = c->hplane[1]; out->avgStatic = c->hplane[2];
  out->avgDynamic = c->hplane[3]; out->avgTotal = c->hplane[4]; out->valid = c->hplane[5] != 0.0;
  return CPS_OK;
}

cps_status cps_download_fields(cps_ctx* c, double* u, double* v, double* p, double* pStar, double* uStar,
                               double* vStar, double* dE, double* dN, int layout) {
  if (!c) return fail(nullptr, CPS_ERR_ARG, "ctx is NULL");
  if (layout != CPS_ROW_MAJOR && layout != CPS_COL_MAJOR) return fail(c, CPS_ERR_ARG, "bad layout");
  if (!cuda_ok(c, cudaSetDevice(c->device), "cudaSetDevice")) return CPS_ERR_CUDA;
  const int M = c->M, N = c->N;
  const cps::DesignView& w = c->view;
  const PlaneOut planes[] = {{u, w.u, M + 1, N},   {v, w.v, M, N + 1},   {p, w.p, M + 1, N + 1}, {pStar, w.pc, M + 1, N + 1},
                             {uStar, w.us, M + 1, N}, {vStar, w.vs, M, N + 1}, {dE, w.dE, M + 1, N},   {dN, w.dN, M, N + 1}};
  if (!download_planes(c, planes, 8, layout)) return CPS_ERR_CUDA;
  return CPS_OK;
}

}  // extern "C"
