/* Stand-ins for the CUDA runtime calls of a kernel launch, preloaded before the engine by test_launch_limits_cpu.py: they
 * keep per device what cudaFuncSetAttribute allowed, refuse a launch that asks for more dynamic shared memory, and
 * record the launches.  Nothing runs. */
#include <cuda_runtime_api.h>
#include <map>
#include <utility>
#include <vector>

namespace {
int g_device = 0, g_sms = 148;
std::map<std::pair<int, const void *>, int> g_limit;
struct Launch { int device, cluster, refused; };
std::vector<Launch> g_launches;

cudaError_t launch(const void *f, size_t smem, int cluster)
{
    const auto it = g_limit.find({g_device, f});
    const bool refused = smem > (size_t)(it == g_limit.end() ? 48 * 1024 : it->second);
    g_launches.push_back({g_device, cluster, refused});
    return refused ? cudaErrorInvalidValue : cudaSuccess;
}
}  // namespace

extern "C" {
void fake_use(int device, int sms) { g_device = device; g_sms = sms; g_launches.clear(); }
int fake_launches() { return (int)g_launches.size(); }
int fake_cluster(int n) { return g_launches[n].cluster; }
int fake_refused()
{
    int r = 0;
    for (const Launch &l : g_launches) r += l.refused;
    return r;
}

cudaError_t cudaGetDevice(int *d) { *d = g_device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? g_sms : 0;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v)
{
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) g_limit[{g_device, f}] = v;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **, size_t smem, cudaStream_t) { return launch(f, smem, 1); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **)
{
    int n = 1;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension)
            n = (int)(c->attrs[i].val.clusterDim.x * c->attrs[i].val.clusterDim.y * c->attrs[i].val.clusterDim.z);
    return launch(f, c->dynamicSmemBytes, n);
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}
