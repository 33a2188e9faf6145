// A CUDA runtime that launches nothing: it records what the launchers of csrc/kernels ask for, so that their rules can be tested
// without a GPU.  Linked with the kernels' objects in place of the runtime's library (tests/test_launch_rules.py).
#include <cuda.h>
#include <cuda_runtime.h>
#include <map>
#include <set>
#include <string>
#include <string.h>

namespace {
struct Launch {
    unsigned grid[3], block[3], cluster[3];
    unsigned smem, dependent;
    int device;
    char kernel[256];
};
Launch g_last;
int g_launches = 0, g_device = 0, g_occupancy_calls = 0;
int g_room[17];                                      // answer of the occupancy query by blocks of a cluster; -1: the query fails
cudaError_t g_error = cudaSuccess;
std::map<const void*, std::string> g_names;
std::map<std::pair<int, const void*>, int> g_allowed;          // (device, kernel): shared memory opted in to

CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) { return CUDA_SUCCESS; }
cudaError_t raise(cudaError_t e) { return g_error = e; }
}  // namespace

extern "C" {
void fake_room(int blocks, int clusters) { g_room[blocks] = clusters; }
void fake_device(int device) { g_device = device; }
int fake_launches() { return g_launches; }
int fake_occupancy_calls() { return g_occupancy_calls; }
void fake_last(Launch* out) { *out = g_last; }

cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int bytes) { g_allowed[{g_device, f}] = bytes; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "an error"; }
cudaError_t cudaGetLastError() { cudaError_t e = g_error; g_error = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return g_error; }
cudaError_t cudaMemcpyFromSymbol(void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *fn = (void*)encode;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void* f, void**) {
    Launch l = {{cfg->gridDim.x, cfg->gridDim.y, cfg->gridDim.z}, {cfg->blockDim.x, cfg->blockDim.y, cfg->blockDim.z}, {1, 1, 1},
                (unsigned)cfg->dynamicSmemBytes, 0, g_device, ""};
    for (unsigned i = 0; i < cfg->numAttrs; ++i) {
        const cudaLaunchAttribute& a = cfg->attrs[i];
        if (a.id == cudaLaunchAttributeClusterDimension) { l.cluster[0] = a.val.clusterDim.x; l.cluster[1] = a.val.clusterDim.y; l.cluster[2] = a.val.clusterDim.z; }
        if (a.id == cudaLaunchAttributeProgrammaticStreamSerialization) l.dependent = a.val.programmaticStreamSerializationAllowed;
    }
    strncpy(l.kernel, g_names[f].c_str(), sizeof(l.kernel) - 1);
    g_last = l;
    ++g_launches;
    // what a device does with a kernel that was not allowed this much, and with a cluster it has no room for
    auto allowed = g_allowed.find({g_device, f});
    if (l.smem > 48 * 1024 && (allowed == g_allowed.end() || (int)l.smem > allowed->second)) return raise(cudaErrorInvalidValue);
    const unsigned blocks = l.cluster[0] * l.cluster[1] * l.cluster[2];
    if (blocks > 1 && g_room[blocks] < 1) return raise(cudaErrorInvalidClusterSize);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return raise(cudaErrorNotSupported); }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* cfg) {
    ++g_occupancy_calls;
    unsigned blocks = 1;
    for (unsigned i = 0; i < cfg->numAttrs; ++i)
        if (cfg->attrs[i].id == cudaLaunchAttributeClusterDimension)
            blocks = cfg->attrs[i].val.clusterDim.x * cfg->attrs[i].val.clusterDim.y * cfg->attrs[i].val.clusterDim.z;
    if (g_room[blocks] < 0) return raise(cudaErrorInvalidClusterSize);
    *n = g_room[blocks];
    return cudaSuccess;
}

// what the objects' constructors call
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { g_names[host] = name; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 0; }
}
