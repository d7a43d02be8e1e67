// pjg_vjp_noalloc: the J^T v evaluation without any device allocation.
//
// Some callers cannot let a library allocate device memory at call time:
// CFD and reacting-flow solvers that call the chemistry once per cell
// batch and time step from a hot loop (cudaMalloc and cudaFree can
// synchronise the whole device and stall every other stream), codes that
// must not fail for out-of-memory half-way through a simulation, and hosts
// that hand every byte of the GPU to their own pool allocator.  pjg_vjp may
// grow the mechanism's working buffer with cudaMalloc; this entry point
// instead uses a fixed scratch array that lives in this file for the life of
// the process, and calls no cudaMalloc, cudaFree or allocating library
// routine.
//
// The scratch array is kScratchDoubles doubles (16 MiB) on every device that
// loads the library, held until the process exits.  It holds the blocks'
// scratch slices (about 5 Ns doubles per state of a tile); the grid is cut to
// as many blocks as have a slice, whatever the problem's size.  A mechanism
// of which 128 states at 10 Ns doubles do not fit (more than 1,638 species) is
// rejected with PJG_ERR_ARG.
//
// Set-up: the first call on each device, with that device current, takes the
// array's device address with cudaGetSymbolAddress (a host-side name of a
// __device__ array is not a device address).  That first call should come
// before any stream capture on the device.
//
// Every call shares the one array, which keeps the contents the last call
// left there.  The kernel writes every scratch element before it reads it, so
// nothing needs clearing between calls, but calls that overlap on the GPU
// (for example on two streams) race on the array and must be serialised by
// the caller.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <mutex>

#include "../../include/pyjac_gb300.h"
#include "pjg_eval.cuh"

int pjg_internal_fail(int code, const char* msg);
int pjg_internal_vjp_args(pjg_mech* m, int64_t n, size_t scratch_doubles, EvalArgs* a, int* grid);
int pjg_internal_mech_ns(const pjg_mech* m);
int pjg_internal_check_device(const pjg_mech* m);
void pjg_internal_count_launch();

namespace {

constexpr size_t kScratchDoubles = size_t(2) << 20;  // 16 MiB
static __device__ __align__(256) double g_noalloc_scratch[kScratchDoubles];

constexpr int kMaxDevices = 64;
double* g_scratch_addr[kMaxDevices] = {};
std::mutex g_setup_mu;

int scratch_for_current_device(double** out)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return pjg_internal_fail(PJG_ERR_CUDA, "cudaGetDevice failed");
    if (dev < 0 || dev >= kMaxDevices) return pjg_internal_fail(PJG_ERR_ARG, "device index out of range");
    std::lock_guard<std::mutex> g(g_setup_mu);
    if (!g_scratch_addr[dev]) {
        double* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress((void**)&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            char msg[256];
            snprintf(msg, sizeof(msg), "cudaGetSymbolAddress of the no-alloc scratch failed: %s",
                     cudaGetErrorString(e));
            return pjg_internal_fail(PJG_ERR_CUDA, msg);
        }
        g_scratch_addr[dev] = p;
    }
    *out = g_scratch_addr[dev];
    return 0;
}

}  // namespace

extern "C" int pjg_vjp_noalloc(pjg_mech* mech, int64_t n, char order, int conp, const double* param,
                               const double* phi, const double* v, double* out, void* stream)
{
    if (!mech) return pjg_internal_fail(PJG_ERR_ARG, "null mechanism");
    if (n < 0) return pjg_internal_fail(PJG_ERR_ARG, "negative problem size");
    if (order != 'C' && order != 'F') return pjg_internal_fail(PJG_ERR_ARG, "order must be 'C' or 'F'");
    if (n == 0) return 0;
    if (!param || !phi || !v || !out) return pjg_internal_fail(PJG_ERR_ARG, "null array");
    const int ns = pjg_internal_mech_ns(mech);
    const size_t need = (size_t)10 * ns * 128;  // doubles
    if (need > kScratchDoubles) {
        char msg[256];
        snprintf(msg, sizeof(msg),
                 "pjg_vjp_noalloc: %d species need %zu bytes of scratch per 128 states, more than "
                 "the fixed %zu-byte array", ns, need * 8, kScratchDoubles * 8);
        return pjg_internal_fail(PJG_ERR_ARG, msg);
    }
    // the scratch address below is the current device's: the mechanism's
    // tables must live there too
    int rc = pjg_internal_check_device(mech);
    if (rc) return rc;
    double* scratch = nullptr;
    rc = scratch_for_current_device(&scratch);
    if (rc) return rc;
    const int NN = ns + 1;
    EvalArgs a;
    int grid = 0;
    rc = pjg_internal_vjp_args(mech, n, kScratchDoubles, &a, &grid);
    if (rc) return rc;
    a.n = n;
    a.conp = conp;
    a.param = param;
    a.phi = phi;
    a.phi_ss = order == 'F' ? 1 : NN;
    a.phi_sj = order == 'F' ? n : 1;
    a.v = v;
    a.vjp = out;
    a.scratch = scratch;
    rc = pjg_launch_tile(a, KIND_VJP, grid, stream);
    if (rc) {
        char msg[256];
        snprintf(msg, sizeof(msg), "pjg_vjp_noalloc: kernel launch failed: %s", pjg_launch_error_string());
        return pjg_internal_fail(PJG_ERR_CUDA, msg);
    }
    pjg_internal_count_launch();
    return 0;
}
