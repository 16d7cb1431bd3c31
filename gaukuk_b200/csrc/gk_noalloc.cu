// gk_noalloc.cu -- one RK2 time step on caller-owned device memory, with no
// device allocation by the library.
//
// Who needs it: callers that cannot call cudaMalloc while they run -- code
// that owns all device memory through its own pool or arena, real-time loops
// that must not allocate after start-up, and hosts whose memory budget is
// fixed when they load this library.  gk_create allocates the RK stage
// buffers and the device clock per handle; this entry point instead keeps
// them in one file-scope device array of fixed size, so the caller passes
// only the state.
//
// The scratch array (64 MiB) is part of every GPU context that loads the
// library and lives until the process exits.  In host code its name is a
// host-side stand-in, never a device address: the address used for kernel
// arguments comes from cudaGetSymbolAddress, taken once per device with that
// device current, on the first call made on the device.
//
// The stage state holds all five variable planes: the ghost fill writes the
// ghosts of every plane, MTZ included, so a grid is accepted only when
// 5 * vstride doubles fit (about 1290 x 1290 cells).
#include <atomic>
#include <cstdio>
#include <cstring>
#include <string>

#include "gaukuk_cuda.h"
#include "gk_internal.h"

int gk_internal_build_ctx(const gk_grid_desc* gd, const gk_phys_desc* pd, gk::Ctx* ctx,
                          std::string* err);

namespace {

constexpr long long kScratchDoubles = 1LL << 23;  // 64 MiB
constexpr int kMaxDevices = 64;

// Scratch: the intermediate RK stage state (5 variable planes in the device
// layout), then what a call reads back: the device clock, whether MTZ was
// non-zero, and the ticket of the call whose clock was set last.
struct NoallocResult {
    gk::DevTime clock;
    unsigned long long ticket;
    int flag;
    int flag_acc;  // the running check of one call; zero between calls
};
struct NoallocScratch {
    double stage[kScratchDoubles];
    NoallocResult res;
};

static __device__ __align__(256) NoallocScratch gk_noalloc_scratch;

// Device address of the scratch array per device, looked up on the device's
// first call.  Atomic: host threads making their first calls on one device
// at the same time each look it up and store the same value.
std::atomic<NoallocScratch*> g_scratch_addr[kMaxDevices];

// Call tickets: the begin kernel stores its call's ticket, so a call that
// finds its own ticket and step 1 in the clock knows that its launches ran
// (without reading cudaGetLastError, which would also report errors left by
// unrelated work).
std::atomic<unsigned long long> g_ticket{0};

// The CFL reduction's start value, or the zero of a scratch that no call has used.
bool is_seed(unsigned long long acc) {
    const double seed = 1e-16;
    unsigned long long bits;
    std::memcpy(&bits, &seed, sizeof(bits));
    return acc == bits || acc == 0;
}

}  // namespace

extern "C" int gk_rk2_step_noalloc(const gk_grid_desc* grid, const gk_phys_desc* phys,
                                   double* state, double dtmax, double* dt_used, void* stream) {
    if (!grid || !phys || !state) return GK_ERR_INVALID;
    gk::Ctx c{};
    std::string err;
    int rc = gk_internal_build_ctx(grid, phys, &c, &err);
    if (rc != GK_OK) {
        std::fprintf(stderr, "gk_rk2_step_noalloc: %s\n", err.c_str());
        return rc;
    }
    if (c.g.ndim != 2 || c.ph.integrator != 2 || c.ph.grav[2] != 0) {
        std::fprintf(stderr, "gk_rk2_step_noalloc: needs a 2D run with integrator 2 and gz = 0\n");
        return GK_ERR_UNSUPPORTED;
    }
    for (int side = 0; side < 6; ++side) {
        if (c.ph.bc[side] == 4) {
            // fixed sides fill their ghosts from the state at enrollment,
            // which only a handle holds (gk_set_fixed_boundary)
            std::fprintf(stderr, "gk_rk2_step_noalloc: fixed (type 4) sides need a handle\n");
            return GK_ERR_UNSUPPORTED;
        }
    }
    if (5 * c.g.vstride > kScratchDoubles) {
        std::fprintf(stderr,
                     "gk_rk2_step_noalloc: grid too large: the stage state needs %lld doubles, "
                     "the fixed scratch holds %lld (about 1290 x 1290 cells)\n",
                     5 * c.g.vstride, kScratchDoubles);
        return GK_ERR_INVALID;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return GK_ERR_CUDA;
    if (!g_scratch_addr[dev].load(std::memory_order_acquire)) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, gk_noalloc_scratch);
        if (e != cudaSuccess) {
            std::fprintf(stderr, "gk_rk2_step_noalloc: cudaGetSymbolAddress: %s\n",
                         cudaGetErrorString(e));
            return GK_ERR_CUDA;
        }
        g_scratch_addr[dev].store(static_cast<NoallocScratch*>(p), std::memory_order_release);
    }
    NoallocScratch* sc = g_scratch_addr[dev].load(std::memory_order_acquire);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    c.tm = &sc->res.clock;
    double* stage = sc->stage;

    const unsigned long long ticket = ++g_ticket;
    const bool fast = phys->mode == GK_MODE_FAST;
    auto begin = fast ? gk_fast::launch_noalloc_begin : gk_parity::launch_noalloc_begin;
    auto bc = fast ? gk_fast::launch_bc : gk_parity::launch_bc;
    auto stage2d = fast ? gk_fast::launch_stage2d : gk_parity::launch_stage2d;
    auto kick = fast ? gk_fast::launch_kick : gk_parity::launch_kick;
    // Sim::Advance for one step with dtUntilOutput = dtmax (sim.cpp:77-81):
    // one pass over the state checks that MTZ is zero and reduces cmax, and its
    // last CTA sets the clock with dt (inactive, so that nothing after it
    // runs, when MTZ is not zero); then the first gravity half kick
    // (sim.cpp:85-86) and the two RK2 stages; the last stage applies the second
    // half kick and its epilogue advances the clock.  On a grid periodic on all
    // sides the first stage writes the stage state's ghosts itself.
    begin(c, state, dtmax, &sc->res.flag_acc, &sc->res.flag, &sc->res.ticket, ticket, s);
    if (c.ph.has_grav) kick(c, state, 0, s);
    bc(c, state, s);
    gk::Ctx first = c;
    first.ph.periodic_images = c.ph.bc[0] == 1 && c.ph.bc[1] == 1 && c.ph.bc[2] == 1 && c.ph.bc[3] == 1;
    stage2d(first, state, nullptr, stage, 0, 1.0, 1.0, 0.0, s);
    if (!first.ph.periodic_images) bc(c, stage, s);
    stage2d(c, stage, state, state, 2, 0.5, 0.5, 0.5, s);
    NoallocResult r{};
    if (cudaMemcpyAsync(&r, &sc->res, sizeof(r), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return GK_ERR_CUDA;
    const gk::DevTime& t = r.clock;
    // The begin pass counts and reduces on from what the last call left, which is zero
    // and the seed unless calls overlapped.  The last of those to copy its result sees
    // what is left of them, and clears it for the calls that follow.
    if (t.done_ctas || r.flag_acc || !is_seed(t.cmax_acc)) {
        if (cudaMemsetAsync(&sc->res, 0, sizeof(sc->res), s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
            return GK_ERR_CUDA;
    }
    if (r.ticket != ticket) {
        std::fprintf(stderr, "gk_rk2_step_noalloc: a kernel of this call did not launch\n");
        return GK_ERR_CUDA;
    }
    if (r.flag) {
        std::fprintf(stderr, "gk_rk2_step_noalloc: MTZ is not zero; the fused 2D step needs vz = 0\n");
        return GK_ERR_UNSUPPORTED;
    }
    if (t.status & gk::STATUS_TMA_TIMEOUT) {
        std::fprintf(stderr, "gk_rk2_step_noalloc: a TMA row load did not complete within the "
                             "stage kernel's wait limit\n");
        return GK_ERR_CUDA;
    }
    if (t.status) return GK_ERR_NONFINITE;
    if (t.step != 1) {
        std::fprintf(stderr, "gk_rk2_step_noalloc: a kernel of this call did not launch\n");
        return GK_ERR_CUDA;
    }
    if (dt_used) *dt_used = t.t;  // one step from t = 0: t is the dt taken
    return GK_OK;
}
