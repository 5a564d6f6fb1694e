// The projections (gemm_tc.cu) on a device that refuses every launch of a cluster, as a partition without room for one does.
// test_gpu_linear.py builds this as a library of its own.
#include <cuda_runtime.h>

static int g_refused = 0;
template <typename... KArgs, typename... Args>
static cudaError_t refuse_clusters(const cudaLaunchConfig_t *cfg, void (*kernel)(KArgs...), Args... args)
{
    cudaFuncAttributes attr;
    bool cluster = cudaFuncGetAttributes(&attr, (const void *)kernel) == cudaSuccess && attr.requiredClusterWidth > 1;
    for (unsigned i = 0; i < cfg->numAttrs; i++)
        cluster = cluster || (cfg->attrs[i].id == cudaLaunchAttributeClusterDimension && cfg->attrs[i].val.clusterDim.x > 1);
    if (!cluster) return cudaLaunchKernelEx(cfg, kernel, args...);
    g_refused++;
    return cudaErrorInvalidClusterSize;
}
#define cudaLaunchKernelEx refuse_clusters
#include "../sf-bert_b200/csrc/gemm_tc.cu"
#include "../sf-bert_b200/csrc/api.cu"

// bf16 operands; returns the call's own result, and the launches refused meanwhile in *refused
extern "C" int linear_refused(void *stream, void *out, const void *x, const void *w, const float *bias, const void *resid, unsigned m, unsigned n,
                              unsigned k, int act, int w_transposed, int *refused)
{
    g_refused = 0;
    const int rc = sfb::tc_linear((cudaStream_t)stream, out, x, w, bias, m, n, k, SFB_BF16, act, w_transposed != 0, resid);
    *refused = g_refused;
    return rc;
}
extern "C" int linear_status(unsigned *status) { return sfb::tc_status_gemm(status); }
