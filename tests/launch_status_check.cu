// A matvec kernel whose launch is refused is reported (run on a machine without
// a device, where the runtime refuses every launch; exits 77 where there is
// one): near_status, which every entry point and every tick of the batched
// solver asks, returns it once, whatever error the caller left pending.
#include <cstdio>

#include "ctx.h"

template <typename C> static int check(int nrhs, const char *what) {
    static scd_ctx c;
    c.T = 1;
    c.n = 3;
    c.ncubes = c.ngroups = c.max_per_group = 1;
    c.max_tile_store = tile_elems(1, 1);
    // lengths without a transform: the chain launches no FFT kernel
    run_matvec(&c, (const C *)nullptr, (C *)nullptr, nrhs, nullptr);
    if (near_status(&c) != SCD_CUDA_ERROR || c.err.find("matvec launch") == std::string::npos) {
        std::printf("%s: refused launches were not reported (%s)\n", what, c.err.c_str());
        return 1;
    }
    if (c.launch_err != cudaSuccess) { std::printf("%s: the error was not cleared\n", what); return 1; }
    // the fused y-z pass alone
    c.ngroups = 0;
    c.Px = c.Py = c.Pz = 16;
    c.Nx = c.Ny = c.Nz = 8;
    c.fyz_ready = c.fyz_ready_f = true;
    run_matvec(&c, (const C *)nullptr, (C *)nullptr, nrhs, nullptr);
    if (near_status(&c) != SCD_CUDA_ERROR) { std::printf("%s: a refused y-z pass was not reported\n", what); return 1; }
    return 0;
}

int main() {
    int devices = 0;
    if (cudaGetDeviceCount(&devices) == cudaSuccess && devices > 0) return 77;
    return check<cd>(1, "FP64, 1") || check<cd>(3, "FP64, 3") || check<cd>(20, "FP64, 20") || check<cf>(1, "complex64, 1") ||
           check<cf>(20, "complex64, 20");
}
