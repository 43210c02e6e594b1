// host_cpu.cpp - says at load time that the host lacks what the other host files
// were compiled for (Makefile, HOST_ARCH), before one of their instructions ends
// the process.  Compiled for any x86-64 itself.
#include <cstdio>

#ifdef GPUQO_HOST_X86_64_V3
__attribute__((constructor)) static void check_host() {
    __builtin_cpu_init();
    if (__builtin_cpu_supports("avx2") && __builtin_cpu_supports("bmi2") && __builtin_cpu_supports("fma") &&
        __builtin_cpu_supports("popcnt"))
        return;
    std::fprintf(stderr, "gpuqo_b200: built for hosts with AVX2, BMI2, FMA and popcnt, which this one lacks: rebuild "
                         "with make -C postgres-gpuqo_b200 HOST_ARCH=\n");
}
#endif
