// mh_noalloc.cu -- influence-matrix assembly that allocates no device memory.
//
// Some callers cannot call cudaMalloc: code that runs under a device-memory pool
// which already owns the GPU's memory (a Julia CUDA.jl session, a framework with
// its own caching allocator), or code that must not allocate once it has been
// initialised (fixed-footprint services, real-time loops).  For them this file
// provides mh_assemble_matrices_noalloc: the caller passes device buffers for the
// mesh and for S and D, and the only scratch the assembly needs -- one 256-byte
// panel record per panel (the Birk local frame, area centroid and local corners)
// -- lives in a fixed file-scope device array, so no call allocates.
//
// The array holds at most kNoAllocMaxPanels records (2 MiB); every GPU that
// loads this library keeps it until the process exits.  All calls share it and
// it keeps the previous call's contents: each call rewrites the records of its
// own panels before reading them, so nothing needs clearing, but two calls whose
// work overlaps on the GPU (different streams, or different host threads) race
// on it.
//
// Set-up: the first call in a CUDA context (per device, and again after the
// context is replaced, e.g. by cudaDeviceReset) looks up the array's device
// address with cudaGetSymbolAddress and loads the module of every kernel the
// entry point launches.  Loading a module can allocate (the 2 MiB array comes
// into being then), so that first call belongs before any stream capture and may
// fail with MH_ERR_CUDA when the pool leaves no room for the module.
#include <cuda_runtime.h>

#include <mutex>

#include "mh_internal.cuh"

namespace mh {

namespace {

constexpr int64_t kNoAllocMaxPanels = 8192;
constexpr uint32_t kNoAllocKinds = MH_GF_RANKINE | MH_GF_RANKINE_REFLECTED | MH_GF_RANKINE_REFLECTED_NEGATIVE |
                                   MH_GF_WU;
constexpr int kMaxDevices = 64;

static __device__ __align__(256) PanelRec g_noalloc_panels[kNoAllocMaxPanels];

// Host-side: the device address of g_noalloc_panels per device, valid for the CUDA
// context it was looked up in.  (In host code the symbol name is only a host-side
// stand-in for the array, not a device address.)  The context is identified by the
// driver's context id, reached through the runtime's driver entry-point query so the
// library needs no link against libcuda; without it the address is looked up on
// every call.
using CtxGetCurrentFn = int (*)(void**);
using CtxGetIdFn = int (*)(void*, unsigned long long*);

struct NoAllocSetup {
  unsigned long long ctx_id = 0;  // 0: not set up
  PanelRec* panels = nullptr;
};

std::mutex g_setup_mutex;
NoAllocSetup g_setup[kMaxDevices];
CtxGetCurrentFn g_ctx_get_current = nullptr;
CtxGetIdFn g_ctx_get_id = nullptr;
bool g_ctx_fns_resolved = false;

unsigned long long current_context_id() {
  if (!g_ctx_fns_resolved) {
    g_ctx_fns_resolved = true;
    void* f1 = nullptr;
    void* f2 = nullptr;
    cudaDriverEntryPointQueryResult q1, q2;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1) == cudaSuccess &&
        q1 == cudaDriverEntryPointSuccess &&
        cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2) == cudaSuccess &&
        q2 == cudaDriverEntryPointSuccess) {
      g_ctx_get_current = reinterpret_cast<CtxGetCurrentFn>(f1);
      g_ctx_get_id = reinterpret_cast<CtxGetIdFn>(f2);
    }
  }
  if (!g_ctx_get_current || !g_ctx_get_id) return 0;
  void* ctx = nullptr;
  unsigned long long id = 0;
  if (g_ctx_get_current(&ctx) != 0 || !ctx || g_ctx_get_id(ctx, &id) != 0) return 0;
  return id;
}

// Once per device and context, with that device current: the array's address, and every
// kernel of the entry point loaded now rather than lazily at a later (possibly captured)
// launch.
int panels_address(int device, PanelRec** out) {
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  NoAllocSetup& su = g_setup[device];
  const unsigned long long id = current_context_id();
  if (id == 0 || su.ctx_id != id) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_panels) != cudaSuccess) return MH_ERR_CUDA;
    if (load_pair_kernels() != cudaSuccess) return MH_ERR_CUDA;
    su.panels = static_cast<PanelRec*>(p);
    su.ctx_id = id;
  }
  *out = su.panels;
  return MH_OK;
}

}  // namespace

}  // namespace mh

extern "C" int mh_assemble_matrices_noalloc(void* stream, int64_t n_panels, const double* vertices,
                                            const double* centers, const double* normals, const double* areas,
                                            const double* radii, double wavenumber, uint32_t gfs, int direct,
                                            int include_identity, const double* fixed_normal, double* S, double* D) {
  using namespace mh;
  if (n_panels <= 0 || n_panels > kNoAllocMaxPanels) return MH_ERR_ARG;
  if (!vertices || !centers || !normals || !areas || !radii || !S || !D) return MH_ERR_ARG;
  if (gfs == 0 || (gfs & ~kNoAllocKinds)) return MH_ERR_UNSUPPORTED;
  if ((gfs & MH_GF_WU) && !(wavenumber > 0)) return MH_ERR_ARG;
  // an error that earlier work left pending on this thread is reported, and left pending,
  // before anything is launched, so that it is not taken for this call's own failure
  if (cudaPeekAtLastError() != cudaSuccess) return MH_ERR_CUDA;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) return MH_ERR_CUDA;
  PanelRec* panels = nullptr;
  int rc = panels_address(device, &panels);
  if (rc != MH_OK) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const LaunchCounter none{nullptr, nullptr};
  launch_panel_geometry(st, none, n_panels, vertices, centers, normals, areas, radii, panels, nullptr);
  AssemblyParams p = {};
  p.n = n_panels;
  p.P = panels;
  p.gfs = gfs;
  p.direct = direct ? 1 : 0;
  p.include_identity = include_identity ? 1 : 0;
  p.has_fixed = fixed_normal ? 1 : 0;
  for (int c = 0; c < 3; ++c) p.fixed[c] = fixed_normal ? fixed_normal[c] : 0.0;
  p.k = wavenumber;
  // the static part goes into the real parts of S and D themselves, which the wave kernel (each
  // pair's terms once for both of its entries) then reads and overwrites
  const bool has_static = (gfs & ~MH_GF_WU) != 0;
  if (has_static) launch_assemble_static(st, none, p, S, D, 2);
  if (gfs & MH_GF_WU)
    launch_assemble_wave(st, none, p, has_static ? S : nullptr, has_static ? D : nullptr, 1, nullptr, (double2*)S,
                         (double2*)D, 0, !has_static && include_identity ? 1 : 0, 2);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}
