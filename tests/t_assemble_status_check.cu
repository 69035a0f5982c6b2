// The T assembly without memory for its partial sums returns SCD_OOM and
// launches nothing (run on a machine without a device, where every allocation
// fails; exits 77 where there is one).
#include <cstdio>

#include "ctx.h"

int main() {
    int devices = 0;
    if (cudaGetDeviceCount(&devices) == cudaSuccess && devices > 0) return 77;
    scd_ctx c;
    c.n = 40000;
    const int rc = (launch_T_assemble(&c, nullptr, 100, 0, 30, nullptr, nullptr));
    if (rc != SCD_OOM || c.launches != 0) { std::printf("status %d, %lld launches\n", rc, c.launches); return 1; }
    return 0;
}
