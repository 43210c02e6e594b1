// A stand-in for the CUDA runtime functions that the library calls, to be
// loaded ahead of the real one: device memory is host memory, a launch does
// nothing.  It fails the allocations it is told to, and a request for more shared
// memory than a block has, keeps the last error as CUDA does, and counts every
// use of a pointer that no live allocation holds: freed again, cleared, copied
// or handed to a kernel.
#include <sys/mman.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

struct dim3 {
    unsigned x, y, z;
};
struct LaunchConfig {   // the head of cudaLaunchConfig_t
    dim3 grid, block;
    size_t smem;
};

static std::map<uintptr_t, size_t> &live() {
    static auto *m = new std::map<uintptr_t, size_t>;
    return *m;
}
static std::map<const void *, std::string> &names() {
    static auto *m = new std::map<const void *, std::string>;
    return *m;
}

// dynamic shared memory that a kernel is allowed
static std::map<const void *, int> &shared_limits() {
    static auto *m = new std::map<const void *, int>;
    return *m;
}

extern "C" {
int fake_allocations, fake_fail_from = -1, fake_fail_count, fake_bad, fake_launches;
static int last_error;   // of the calls that can fail here
static int failed(int e) { return last_error = e; }

static bool held(const void *p, size_t n) {
    auto it = live().upper_bound((uintptr_t)p);
    if (p == nullptr || it == live().begin()) return false;
    --it;
    return (uintptr_t)p + n <= it->first + it->second;
}

static int allocate(void **p, size_t n) {
    const int at = fake_allocations++;
    if (fake_fail_from >= 0 && at >= fake_fail_from && at < fake_fail_from + fake_fail_count) return failed(2);
    void *m = mmap(nullptr, n ? n : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (m == MAP_FAILED) return failed(2);
    live()[(uintptr_t)m] = n;
    *p = m;
    return 0;
}

static int release(void *p) {
    if (!p) return 0;
    auto it = live().find((uintptr_t)p);
    if (it == live().end()) {
        fake_bad++;
        return failed(1);
    }
    munmap(p, it->second ? it->second : 1);
    live().erase(it);
    return 0;
}

// the pointer arguments of the kernels, by name
static int launch(const void *fn, void **args, size_t smem) {
    auto limit = shared_limits().find(fn);
    if (smem > 48 * 1024 && (limit == shared_limits().end() || smem > (size_t)limit->second)) return failed(1);
    fake_launches++;
    auto it = names().find(fn);
    const std::string name = it == names().end() ? "" : it->second;
    static const struct {
        const char *kernel;
        int pointers[12];
    } table[] = {{"5kb_dp", {0, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, -1}},
                 {"6kb_gen", {0, 3, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14}},
                 {"9k_dp_tree", {0, 2, 3, 4, 5, 6, 7, 8, 9, -1}},
                 {"7kb_init", {0, 2, 3, 4, 5, 6, -1}}};
    for (const auto &t : table) {
        if (name.find(t.kernel) == std::string::npos) continue;
        for (int i : t.pointers) {
            if (i < 0) break;
            if (!held(*(void **)args[i], 1)) fake_bad++;
        }
    }
    if (name.find("6kb_gen") != std::string::npos) {   // the overflow list: six arrays, their length
        void **list = (void **)args[15];
        const unsigned cap = *(unsigned *)(list + 6);
        const size_t size[6] = {8, 4, 4, 8, 4, 4};
        for (int i = 0; cap && i < 6; i++)
            if (!held(list[i], cap * size[i])) fake_bad++;
    }
    return 0;
}

int cudaMalloc(void **p, size_t n) { return allocate(p, n); }
int cudaHostAlloc(void **p, size_t n, unsigned) { return allocate(p, n); }
int cudaMallocHost(void **p, size_t n) { return allocate(p, n); }
int cudaFree(void *p) { return release(p); }
int cudaFreeHost(void *p) { return release(p); }
int cudaMemsetAsync(void *p, int v, size_t n, void *) {
    if (!held(p, n)) fake_bad++;
    else if (n <= (64u << 20)) memset(p, v, n);
    return 0;
}
int cudaMemcpyAsync(void *d, const void *s, size_t n, int kind, void *) {
    if (kind == 1 ? !held(d, n) : !held(s, n)) fake_bad++;
    else memcpy(d, s, n);
    return 0;
}
int cudaMemcpy(void *d, const void *s, size_t n, int kind) { return cudaMemcpyAsync(d, s, n, kind, nullptr); }
int cudaLaunchKernel(const void *fn, dim3, dim3, void **args, size_t smem, void *) { return launch(fn, args, smem); }
int cudaLaunchCooperativeKernel(const void *fn, dim3, dim3, void **args, size_t smem, void *) {
    return launch(fn, args, smem);
}
int cudaLaunchKernelExC(const LaunchConfig *c, const void *fn, void **args) { return launch(fn, args, c->smem); }

int cudaGetDevice(int *d) { return *d = 0; }
int cudaSetDevice(int) { return 0; }
int cudaGetDeviceCount(int *n) {
    *n = 1;
    return 0;
}
int cudaDeviceGetAttribute(int *v, int attr, int) {
    *v = attr == 16 ? 148 : 1;   // multiprocessors; cooperative launches
    return 0;
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
    *n = 2;
    return 0;
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 2;
    return 0;
}
int cudaFuncSetAttribute(const void *fn, int attr, int value) {
    if (attr != 8) return 0;   // dynamic shared memory of a block
    if (value > 227 * 1024) return failed(1);
    shared_limits()[fn] = value;
    return 0;
}
int cudaGetLastError() {
    const int e = last_error;
    last_error = 0;
    return e;
}
const char *cudaGetErrorString(int e) { return e ? "error" : "no error"; }
int cudaGetSymbolAddress(void **, const void *) { return 1; }
int cudaEventCreate(void **e) {
    *e = malloc(1);
    return 0;
}
int cudaEventRecord(void *, void *) { return 0; }
int cudaEventRecordWithFlags(void *, void *, unsigned) { return 0; }
int cudaEventSynchronize(void *) { return 0; }
int cudaEventElapsedTime(float *ms, void *, void *) {
    *ms = 0.f;
    return 0;
}
int cudaStreamCreateWithFlags(void **s, unsigned) {
    *s = malloc(1);
    return 0;
}
int cudaStreamSynchronize(void *) { return 0; }
int cudaStreamBeginCapture(void *, int) { return 0; }
int cudaStreamEndCapture(void *, void **g) {
    *g = malloc(1);
    return 0;
}
int cudaGraphInstantiate(void **e, void *, unsigned long long) {
    *e = malloc(1);
    return 0;
}
int cudaGraphLaunch(void *, void *) { return 0; }
int cudaGraphDestroy(void *) { return 0; }
int cudaGraphExecDestroy(void *) { return 0; }

// registration of the kernels, called by the library's initialisers; a
// <<<...>>> launch pops the configuration that it pushed
static struct {
    dim3 grid, block;
    size_t smem;
    void *stream;
} config;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void *stream) {
    config = {grid, block, smem, stream};
    return 0;
}
int __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *(void **)stream = config.stream;
    return 0;
}
void **__cudaRegisterFatBinary(void *) {
    static void *handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *, int *) {
    names()[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
}
