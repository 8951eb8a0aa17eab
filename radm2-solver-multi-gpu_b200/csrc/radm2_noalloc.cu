// radm2_rosenbrock_noalloc: the integration for callers that cannot allocate device
// memory.
//
// Some callers may not call cudaMalloc while they run: a host framework that reserved all
// of the GPU's memory for its own pool at start-up (a later cudaMalloc fails or steals from
// that pool), and real-time or certified couplings whose device memory budget is fixed at
// initialisation and may not grow once the model is running.  This entry point takes device
// pointers for the inputs and outputs and keeps everything else it needs -- the solver
// kernel's per-thread scratch slots, the rate-constant table and the per-cell bookkeeping --
// in one statically sized array in this file.  It runs the same solver (radm2_wide.cuh) and
// reduction kernels as radm2_rosenbrock, on as many blocks as have a scratch slot in the array.
// Measured for 10,007 cells: 7.3 ms against 22.6 ms with the 32-thread kernel that keeps its
// working set in shared memory.
//
// The array is a __device__ object: every GPU that loads the library holds its
// RADM2_NOALLOC_BYTES until the process exits.  Host code cannot use the array's name as
// a device address (in host code it names a host-side stand-in), so the address is
// fetched with cudaGetSymbolAddress on the first call made with a given device and CUDA
// context current, and passed to the kernels.
#include <cstring>
#include <mutex>

#include "../../include/radm2.h"
#include "radm2_internal.h"
#include "gen/radm2_wide_map.h"  // the solver's scratch slot and distinct rate constants

using namespace radm2;

namespace {

constexpr size_t align256(size_t b) { return (b + 255) / 256 * 256; }

// Offsets of the carved regions (bytes): the per-cell bookkeeping, then the rate constants of the
// call's cells (only the wide solver's distinct ones), and the rest for the solver's scratch, one
// slot per block: 114 slots at 10,000 cells (which take 105 blocks), 83 for the largest batch.
constexpr int kMinBlocks = 64;
constexpr size_t kCells = RADM2_NOALLOC_MAX_CELLS;
constexpr size_t kOffNacc = 0;
constexpr size_t kOffNrej = kOffNacc + align256(sizeof(int) * kCells);
constexpr size_t kOffStatus = kOffNrej + align256(sizeof(int) * kCells);
constexpr size_t kOffHfirst = kOffStatus + align256(sizeof(int) * kCells);
constexpr size_t kOffHexit = kOffHfirst + align256(sizeof(double) * kCells);
constexpr size_t kOffTexit = kOffHexit + align256(sizeof(double) * kCells);
constexpr size_t kOffQueue = kOffTexit + align256(sizeof(double) * kCells);
constexpr size_t kOffPartials = kOffQueue + 256;
constexpr size_t kPartialsCap = 64 * 1024;
constexpr size_t kOffResult = kOffPartials + kPartialsCap;
constexpr size_t kOffRconst = kOffResult + align256(sizeof(RunResult));
constexpr size_t kSlotBytes = sizeof(double) * (size_t)RADM2_WIDE_GLOBAL_WORDS * 128;
constexpr size_t rconst_bytes(size_t ld) { return align256(sizeof(double) * RADM2_WIDE_RC_WORDS * ld); }
static_assert(kOffRconst + rconst_bytes(kCells) + kMinBlocks * kSlotBytes <= (size_t)RADM2_NOALLOC_BYTES,
              "no-alloc area too small for the largest batch");

// The statically sized device area (one per GPU that loads this library).
__device__ __align__(256) unsigned char g_noalloc_area[RADM2_NOALLOC_BYTES];

std::mutex g_setup_mutex;
// Per device: the CUDA context the address was looked up in, and the address.  A device
// reset (cudaDeviceReset) or a new primary context reloads the module at a new address, so
// the cached address is only reused while the same context is current.
struct AreaSlot {
    void *ctx;
    void *addr;
};
AreaSlot g_area[256];

using CtxGetCurrentFn = int (*)(void **);
CtxGetCurrentFn ctx_get_current()
{
    static CtxGetCurrentFn fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<CtxGetCurrentFn>(f);
    }();
    return fn;
}

// Device address of the area on the current device and context (set-up on the first call
// with that pair current; without the context query, looked up on every call).
cudaError_t area_address(int device, unsigned char **out)
{
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    void *ctx = nullptr;
    CtxGetCurrentFn get = ctx_get_current();
    const bool known_ctx = get && get(&ctx) == 0 && ctx;
    if (!known_ctx || !g_area[device].addr || g_area[device].ctx != ctx) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_area);
        if (e != cudaSuccess) return e;
        g_area[device].ctx = known_ctx ? ctx : nullptr;
        g_area[device].addr = known_ctx ? p : nullptr;
        *out = static_cast<unsigned char *>(p);
        return cudaSuccess;
    }
    *out = static_cast<unsigned char *>(g_area[device].addr);
    return cudaSuccess;
}

}  // namespace

extern "C" int radm2_rosenbrock_noalloc(int ncell, int ld, double *var, const double *fix, const double *temp,
                                        const double *rc_n2o5, const double *jv, double Tstart, double Tend,
                                        const double *AbsTol, const double *RelTol, double *RPAR, int *IPAR,
                                        int *status, void *stream)
{
    if (ncell <= 0 || ld < ncell || !var || !fix || !temp || !jv || !AbsTol || !RelTol || !RPAR || !IPAR)
        return RADM2_E_ARG;
    if ((size_t)ld > kCells) return RADM2_E_TOOBIG;  // ncell <= ld <= RADM2_NOALLOC_MAX_CELLS
    if (reduce_partials_bytes() > kPartialsCap) return RADM2_E_STATE;
    int device = 0, major = 0, nsm = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 256 ||
        cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) != cudaSuccess || major != 10 ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return RADM2_E_NODEV;
    SolveParams p;
    int autonomous = 1;
    const int ierr0 = parse_params(Tstart, Tend, AbsTol, RelTol, RPAR, IPAR, 1, &p, &autonomous);
    if (ierr0 != 1) return ierr0;
    const size_t off_scratch = kOffRconst + rconst_bytes((size_t)ld);
    const size_t slots = ((size_t)RADM2_NOALLOC_BYTES - off_scratch) / kSlotBytes;
    const WideShape shape = wide_shape(ncell, slots < (size_t)nsm ? (int)slots : nsm);

    unsigned char *area = nullptr;
    if (area_address(device, &area) != cudaSuccess) return RADM2_E_CUDA;
    cudaStream_t st = static_cast<cudaStream_t>(stream);

    double *rconst = reinterpret_cast<double *>(area + kOffRconst);
    int *queue = reinterpret_cast<int *>(area + kOffQueue);
    RunResult *d_res = reinterpret_cast<RunResult *>(area + kOffResult);
    SolveArgs a;
    std::memset(&a, 0, sizeof a);
    a.p = p;
    a.ncell = ncell;
    a.ld = ld;
    a.var = var;
    a.fix = fix;
    a.rconst = rconst;
    a.rc_words = 1;
    a.warps = shape.warps;
    a.queue = queue;
    a.scratch = reinterpret_cast<double *>(area + off_scratch);
    a.status = status ? status : reinterpret_cast<int *>(area + kOffStatus);
    a.nacc = reinterpret_cast<int *>(area + kOffNacc);
    a.nrej = reinterpret_cast<int *>(area + kOffNrej);
    a.hfirst = reinterpret_cast<double *>(area + kOffHfirst);
    a.hexit = reinterpret_cast<double *>(area + kOffHexit);
    a.texit = reinterpret_cast<double *>(area + kOffTexit);
    a.refine = 0;

    // The area keeps the previous call's contents: the work-queue counter must start at 0;
    // every other region is fully rewritten before it is read.
    if (cudaMemsetAsync(queue, 0, sizeof(int), st) != cudaSuccess) return RADM2_E_CUDA;
    if (launch_rconst_wide(ncell, ld, jv, temp, fix, rc_n2o5, rconst, st) != cudaSuccess) return RADM2_E_CUDA;
    if (launch_solver_wide(a, shape.grid, st) != cudaSuccess) return RADM2_E_CUDA;
    if (launch_reduce(ncell, a.status, a.nacc, a.nrej, a.texit, a.hexit, area + kOffPartials, d_res, st) !=
        cudaSuccess)
        return RADM2_E_CUDA;
    RunResult r;
    if (cudaMemcpyAsync(&r, d_res, sizeof r, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return RADM2_E_CUDA;

    add_step_counters(IPAR, r.nacc, r.nrej, r.nfail, autonomous);
    RPAR[10] = p.direction > 0 ? r.tmin : r.tmax;
    RPAR[11] = r.hmin;
    return r.worst;
}
