// capi.cu -- status handling and the generic C entry points of libvsmc_cuda:
// RNG word streams, the device WeightSet update, the device resampler and
// the particle gather.  The CV filter's entry points are in cv_filter.cu.
#include "call_scratch.hpp"
#include "resample_launch.cuh"
#include "weights.cuh"

#include <cstdio>
#include <cstring>
#include <string>

namespace vsmc_b200 {

static thread_local std::string g_last_error;

void set_last_error(const std::string &msg) { g_last_error = msg; }

int cuda_status(cudaError_t e, const char *what)
{
    g_last_error = std::string(what) + ": " + cudaGetErrorName(e) + " (" +
                   cudaGetErrorString(e) + ")";
    return e == cudaErrorMemoryAllocation ? VSMC_CUDA_ENOMEM : VSMC_CUDA_ECUDA;
}

// ------------------------------------------------------------ RNG words --
__device__ __forceinline__ uint4 ctr32_add(uint4 c, unsigned long long v)
{
    unsigned long long s = (unsigned long long)c.x + (v & 0xffffffffull);
    c.x = (uint32_t)s;
    unsigned long long carry = (s >> 32) + (v >> 32);
    s = (unsigned long long)c.y + (carry & 0xffffffffull);
    c.y = (uint32_t)s;
    carry = (s >> 32) + (carry >> 32);
    s = (unsigned long long)c.z + carry;
    c.z = (uint32_t)s;
    carry = s >> 32;
    c.w += (uint32_t)carry;
    return c;
}

// Thread b computes block b of the stream (word positions 4b..4b+3 relative
// to skip rounded down) and stores the words that fall in [skip, skip+n).
__global__ void k_philox_words(uint32_t k0, uint32_t k1, uint4 c0,
                               unsigned long long skip,
                               unsigned long long n, uint32_t *out)
{
    const unsigned long long b0 = skip / 4;
    const unsigned long long b =
        b0 + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned long long wend = skip + n;
    if (b * 4 >= wend)
        return;
    const uint4 r = philox4x32_10(ctr32_add(c0, b + 1), k0, k1);
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const unsigned long long pos = b * 4 + l;
        if (pos >= skip && pos < wend)
            out[pos - skip] = w[l];
    }
}

__global__ void k_threefry_words(u64x4 key, u64x4 c0, unsigned long long skip,
                                 unsigned long long n, uint64_t *out)
{
    const unsigned long long b0 = skip / 4;
    const unsigned long long b =
        b0 + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned long long wend = skip + n;
    if (b * 4 >= wend)
        return;
    const u64x4 r = threefry4x64_20(ctr64_add(c0, b + 1), key);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const unsigned long long pos = b * 4 + l;
        if (pos >= skip && pos < wend)
            out[pos - skip] = r.v[l];
    }
}

// Slot i of every column from its parent: kCopyDims columns' reads in
// flight per thread.
constexpr int kCopyDims = 4;
__global__ void __launch_bounds__(256)
k_copy_f64(long long N, unsigned dim, const double *src, double *dst,
           const int32_t *copy_from)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N)
        return;
    const long long c = copy_from[i];
    for (unsigned d = 0; d < dim; d += kCopyDims) {
        double v[kCopyDims];
#pragma unroll
        for (unsigned k = 0; k < kCopyDims; ++k)
            if (d + k < dim)
                v[k] = src[(long long)(d + k) * N + c];
#pragma unroll
        for (unsigned k = 0; k < kCopyDims; ++k)
            if (d + k < dim)
                dst[(long long)(d + k) * N + i] = v[k];
    }
}

static __global__ void k_math_eval(int fn, long long n, const double *in,
                                   double *out)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = fn == 0 ? fm::fm_log(in[i]) : fm::fm_exp(in[i]);
}

} // namespace vsmc_b200

using namespace vsmc_b200;

namespace {

size_t generic_resample_bytes(long long N)
{
    return resample_workspace_bytes(N) + align256((size_t)N * 4);
}

} // namespace

namespace {

// Sums (and for kWAdd the normalisation) of one call; the result in `h`.
template <int Kind>
cudaError_t weight_call(uint64_t N, double *lw, double *w, const double *inc,
                        cudaStream_t s, WeightCtl &h, const char *&what)
{
    CallScratch cs(s);
    const long long nt = ((long long)N + kTile - 1) / kTile;
    what = ": scratch";
    // device memory: the result when no pinned slot is free, the joined
    // sums and the tiles'
    WeightCtl *out = static_cast<WeightCtl *>(cs.slot());
    WeightCtl *ctl = nullptr;
    WAcc *tiles = nullptr;
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute at[1];
    c.stream = s;
    c.attrs = at;
    c.numAttrs = 1;
    bool cluster = false;
    if (nt <= kWcTiles) {
        int ctas = 1;
        while (ctas < nt && ctas < kWcCtas)
            ctas *= 2;
        if (ctas > 8)
            cudaFuncSetAttribute(
                k_weight_cluster<Kind>,
                cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        c.gridDim = dim3((unsigned)ctas);
        c.blockDim = dim3(kThreads);
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)ctas;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cluster = cluster_room(k_weight_cluster<Kind>, c);
    }
    cudaError_t e;
    if (out == nullptr || !cluster) {
        void *p = nullptr;
        e = cs.alloc(2 * align256(sizeof(WeightCtl)) +
                         sizeof(WAcc) * (size_t)nt,
                     &p);
        if (e != cudaSuccess)
            return e;
        char *q = static_cast<char *>(p);
        if (out == nullptr)
            out = reinterpret_cast<WeightCtl *>(q);
        ctl = reinterpret_cast<WeightCtl *>(q + align256(sizeof(WeightCtl)));
        tiles =
            reinterpret_cast<WAcc *>(q + 2 * align256(sizeof(WeightCtl)));
    }
    what = "";
    if (cluster) {
        e = cudaLaunchKernelEx(&c, k_weight_cluster<Kind>, (long long)N, lw,
                               w, inc, out);
    } else {
        k_weight_tiles<Kind><<<(unsigned)nt, kThreads, 0, s>>>(
            (long long)N, lw, static_cast<const double *>(w), inc, tiles);
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        c.gridDim = dim3(1);
        c.blockDim = dim3(kSpineThreads);
        e = cudaLaunchKernelEx(&c, k_weight_join,
                               static_cast<const WAcc *>(tiles), (int)nt, ctl,
                               out);
        if (e == cudaSuccess && Kind == kWAdd) {
            c.gridDim = dim3(
                (unsigned)(((long long)N + 4 * kThreads - 1) / (4 * kThreads)));
            c.blockDim = dim3(kThreads);
            e = cudaLaunchKernelEx(&c, k_weight_apply, (long long)N, lw, w,
                                   static_cast<const WeightCtl *>(ctl));
        }
    }
    if (e == cudaSuccess)
        e = cudaGetLastError();
    if (e == cudaSuccess && cs.slot() == nullptr)
        e = cudaMemcpyAsync(&h, out, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s);
    if (e != cudaSuccess)
        return e;
    cs.waited();
    if (cs.slot() != nullptr)
        std::memcpy(&h, cs.slot(), sizeof(h));
    return e;
}

template <int Kind>
int prospective(uint64_t N, const double *lw, const double *w,
                const double *inc, double *out, void *stream,
                const char *where)
{
    WeightCtl h;
    const char *what = "";
    const cudaError_t e = weight_call<Kind>(
        N, const_cast<double *>(lw), const_cast<double *>(w), inc,
        static_cast<cudaStream_t>(stream), h, what); // (read only)
    if (e != cudaSuccess)
        return cuda_status(e, where);
    *out = h.S1 * h.S1 / h.S2;
    // the log form needs a finite maximum and a positive sum; the plain
    // forms only finite sums (increments may be negative) and S2 > 0
    const bool bad = Kind == kWEssLog
                         ? h.error != 0
                         : !(h.S1 == h.S1 && h.S1 > -INFINITY &&
                             h.S1 < INFINITY && h.S2 < INFINITY);
    if (bad || !(h.S2 > 0.0)) {
        set_last_error(std::string(where) + ": degenerate weights");
        *out = NAN;
        return VSMC_CUDA_EDEGENERATE;
    }
    return VSMC_CUDA_OK;
}

// A resampling call's result once its stream is done: in the slot already
// (`done`), or copied from the workspace's control block.
static_assert(sizeof(ResampleCtl) <= kSlotBytes, "result fits a slot");
cudaError_t resample_result(const ResampleWorkspace &ws, CallScratch &cs,
                            bool done, cudaStream_t s, ResampleCtl &h)
{
    ResampleCtl *slot = static_cast<ResampleCtl *>(cs.slot());
    cudaError_t e = cudaSuccess;
    if (!done)
        e = cudaMemcpyAsync(slot != nullptr ? slot : &h, ws.ctl, sizeof(h),
                            cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s);
    if (e != cudaSuccess)
        return e;
    cs.waited();
    if (slot != nullptr) {
        h.error = slot->error;
        h.offset = slot->offset;
    }
    return e;
}

} // namespace

extern "C" {

const char *vsmc_cuda_status_string(int s)
{
    switch (s) {
    case VSMC_CUDA_OK:
        return "VSMC_CUDA_OK";
    case VSMC_CUDA_EINVAL:
        return "VSMC_CUDA_EINVAL";
    case VSMC_CUDA_ENOMEM:
        return "VSMC_CUDA_ENOMEM";
    case VSMC_CUDA_EDEGENERATE:
        return "VSMC_CUDA_EDEGENERATE";
    case VSMC_CUDA_ETIMEOUT:
        return "VSMC_CUDA_ETIMEOUT";
    case VSMC_CUDA_ECUDA:
        return "VSMC_CUDA_ECUDA";
    default:
        return "unknown status";
    }
}

const char *vsmc_cuda_last_error(void) { return g_last_error.c_str(); }

int vsmc_cuda_abi_version(void) { return VSMC_CUDA_ABI_VERSION; }

int vsmc_cuda_philox4x32_words(const uint32_t key[2], const uint32_t ctr[4],
                               uint64_t skip, uint64_t n, uint32_t *out,
                               void *stream)
{
    if (key == nullptr || ctr == nullptr || (out == nullptr && n > 0)) {
        set_last_error("vsmc_cuda_philox4x32_words: null pointer");
        return VSMC_CUDA_EINVAL;
    }
    if (n == 0)
        return VSMC_CUDA_OK;
    const unsigned long long blocks = (skip + n + 3) / 4 - skip / 4;
    const unsigned g = (unsigned)((blocks + 255) / 256);
    k_philox_words<<<g, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        key[0], key[1], make_uint4(ctr[0], ctr[1], ctr[2], ctr[3]), skip, n,
        out);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? VSMC_CUDA_OK
                            : cuda_status(e, "vsmc_cuda_philox4x32_words");
}

int vsmc_cuda_threefry4x64_words(const uint64_t key[4], const uint64_t ctr[4],
                                 uint64_t skip, uint64_t n, uint64_t *out,
                                 void *stream)
{
    if (key == nullptr || ctr == nullptr || (out == nullptr && n > 0)) {
        set_last_error("vsmc_cuda_threefry4x64_words: null pointer");
        return VSMC_CUDA_EINVAL;
    }
    if (n == 0)
        return VSMC_CUDA_OK;
    u64x4 k, c;
    for (int i = 0; i < 4; ++i) {
        k.v[i] = key[i];
        c.v[i] = ctr[i];
    }
    const unsigned long long blocks = (skip + n + 3) / 4 - skip / 4;
    const unsigned g = (unsigned)((blocks + 255) / 256);
    k_threefry_words<<<g, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        k, c, skip, n, out);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? VSMC_CUDA_OK
                            : cuda_status(e, "vsmc_cuda_threefry4x64_words");
}

int vsmc_cuda_weight_add_log(uint64_t N, double *lw, double *w,
                             const double *inc, double *ess, void *stream)
{
    if (N == 0 || lw == nullptr || ess == nullptr) {
        set_last_error("vsmc_cuda_weight_add_log: invalid arguments");
        return VSMC_CUDA_EINVAL;
    }
    WeightCtl h;
    const char *what = "";
    const cudaError_t e = weight_call<kWAdd>(
        N, lw, w, inc, static_cast<cudaStream_t>(stream), h, what);
    if (e != cudaSuccess)
        return cuda_status(
            e, (std::string("vsmc_cuda_weight_add_log") + what).c_str());
    if (h.error) {
        set_last_error("vsmc_cuda_weight_add_log: degenerate log-weights");
        *ess = NAN;
        return h.error;
    }
    *ess = h.S1 * h.S1 / h.S2;
    return VSMC_CUDA_OK;
}

int vsmc_cuda_weight_ess(uint64_t N, const double *log_weight,
                         const double *weight, const double *inc, int use_log,
                         double *ess, void *stream)
{
    if (N == 0 || inc == nullptr || ess == nullptr ||
        (use_log ? log_weight == nullptr : weight == nullptr)) {
        set_last_error("vsmc_cuda_weight_ess: invalid arguments");
        return VSMC_CUDA_EINVAL;
    }
    return use_log ? prospective<kWEssLog>(N, log_weight, weight, inc, ess,
                                           stream, "vsmc_cuda_weight_ess")
                   : prospective<kWEssLinear>(N, log_weight, weight, inc, ess,
                                              stream, "vsmc_cuda_weight_ess");
}

int vsmc_cuda_weight_cess(uint64_t N, const double *weight, const double *inc,
                          int use_log, double *cess, void *stream)
{
    if (N == 0 || weight == nullptr || inc == nullptr || cess == nullptr) {
        set_last_error("vsmc_cuda_weight_cess: invalid arguments");
        return VSMC_CUDA_EINVAL;
    }
    return use_log ? prospective<kWCessLog>(N, nullptr, weight, inc, cess,
                                            stream, "vsmc_cuda_weight_cess")
                   : prospective<kWCessLinear>(N, nullptr, weight, inc, cess,
                                               stream,
                                               "vsmc_cuda_weight_cess");
}

size_t vsmc_cuda_resample_workspace_size(uint64_t N)
{
    if (N == 0 || N > (1ull << 30))
        return 0;
    return generic_resample_bytes((long long)N);
}

int vsmc_cuda_resample(int scheme, uint64_t N, const double *weight,
                       const double *uniforms, uint64_t n_uniforms,
                       vsmc_cuda_threefry_state *rng, int32_t *replication,
                       int32_t *copy_from, void *workspace,
                       size_t workspace_bytes, void *stream)
{
    if (scheme < 0 || scheme > 5 || N == 0 || N > (1ull << 30) ||
        weight == nullptr || rng == nullptr || workspace == nullptr ||
        workspace_bytes < generic_resample_bytes((long long)N) ||
        (uniforms == nullptr && n_uniforms != 0) || n_uniforms > N ||
        (reinterpret_cast<uintptr_t>(workspace) & 255) != 0) {
        set_last_error("vsmc_cuda_resample: invalid arguments (scheme, N, "
                       "null pointer, or workspace too small / not "
                       "256-byte aligned)");
        return VSMC_CUDA_EINVAL;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    ResampleWorkspace ws = carve_workspace(workspace, (long long)N);
    int32_t *cf = copy_from;
    if (cf == nullptr)
        cf = reinterpret_cast<int32_t *>(static_cast<char *>(workspace) +
                                         resample_workspace_bytes((long long)N));
    ResampleCtl h;
    std::memset(&h, 0, sizeof(h));
    h.active = 1;
    h.offset = rng->offset;
    CallScratch cs(s);
    ResampleCtl *slot = static_cast<ResampleCtl *>(cs.slot());
    EngineRef eng;
    for (int i = 0; i < 4; ++i) {
        eng.key.v[i] = rng->key[i];
        eng.ctr.v[i] = rng->ctr[i];
    }
    WeightsGiven w;
    w.w = weight;
    const bool done =
        launch_resample(scheme, w, (long long)N, eng, ws, h, slot, uniforms,
                        (long long)n_uniforms, replication, cf, s);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return cuda_status(e, "vsmc_cuda_resample: launch");
    e = resample_result(ws, cs, done, s, h);
    if (e != cudaSuccess)
        return cuda_status(e, "vsmc_cuda_resample");
    if (h.error != 0) {
        set_last_error("vsmc_cuda_resample: look-back wait gave up");
        return h.error;
    }
    rng->offset = h.offset;
    return VSMC_CUDA_OK;
}

size_t vsmc_cuda_resample_mn_workspace_size(uint64_t M, uint64_t N)
{
    if (M == 0 || M > (1ull << 30) || N > (1ull << 30))
        return 0;
    const long long Nmax = (long long)(M > N ? M : N);
    return resample_workspace_bytes(Nmax) + 2 * align256((size_t)Nmax * 4);
}

int vsmc_cuda_resample_mn(int scheme, uint64_t M, uint64_t N,
                          const double *weight, const double *uniforms,
                          uint64_t n_uniforms, vsmc_cuda_threefry_state *rng,
                          int32_t *replication, int32_t *copy_from,
                          void *workspace, size_t workspace_bytes,
                          void *stream)
{
    const size_t need = vsmc_cuda_resample_mn_workspace_size(M, N);
    if (scheme < 0 || scheme > 5 || need == 0 || weight == nullptr ||
        rng == nullptr || workspace == nullptr || workspace_bytes < need ||
        (uniforms == nullptr && n_uniforms != 0) || n_uniforms > N ||
        (reinterpret_cast<uintptr_t>(workspace) & 255) != 0) {
        set_last_error("vsmc_cuda_resample_mn: invalid arguments (scheme, "
                       "M >= 1, N, null pointer, or workspace too small / "
                       "not 256-byte aligned)");
        return VSMC_CUDA_EINVAL;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool sys = scheme == VSMC_CUDA_SYSTEMATIC ||
                     scheme == VSMC_CUDA_RESIDUAL_SYSTEMATIC;
    const long long Nmax = (long long)(M > N ? M : N);
    char *wsp = static_cast<char *>(workspace);
    int32_t *cf_scratch =
        reinterpret_cast<int32_t *>(wsp + resample_workspace_bytes(Nmax));
    int32_t *rep = replication != nullptr
                       ? replication
                       : cf_scratch + align256((size_t)Nmax * 4) / 4;
    cudaError_t e = cudaSuccess;
    if (N == 0) {
        // inversion(M, 0, ...) leaves every count at zero; only the
        // systematic sequence draws its one word, in its constructor
        // (rng/u01.hpp:253-263)
        e = cudaMemsetAsync(rep, 0, M * 4, s);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(s);
        if (e != cudaSuccess)
            return cuda_status(e, "vsmc_cuda_resample_mn");
        rng->offset += sys ? 1 : 0;
        return VSMC_CUDA_OK;
    }
    if (M == N)
        return vsmc_cuda_resample(scheme, N, weight, uniforms, n_uniforms,
                                  rng, replication, copy_from, workspace,
                                  workspace_bytes, stream);
    ResampleWorkspace ws = carve_workspace(workspace, Nmax);
    ResampleCtl h;
    std::memset(&h, 0, sizeof(h));
    h.active = 1;
    h.offset = rng->offset;
    h.Nout = (long long)N;
    CallScratch cs(s);
    ResampleCtl *slot = static_cast<ResampleCtl *>(cs.slot());
    EngineRef eng;
    for (int i = 0; i < 4; ++i) {
        eng.key.v[i] = rng->key[i];
        eng.ctr.v[i] = rng->ctr[i];
    }
    WeightsGiven w;
    w.w = weight;
    const bool done =
        launch_resample(scheme, w, (long long)M, eng, ws, h, slot, uniforms,
                        (long long)n_uniforms, rep, cf_scratch, s,
                        /*cfrp=*/false);
    if (copy_from != nullptr)
        launch_resample_expand(rep, (long long)M, (long long)N, ws, copy_from, s);
    e = cudaGetLastError();
    if (e != cudaSuccess)
        return cuda_status(e, "vsmc_cuda_resample_mn: launch");
    e = resample_result(ws, cs, done, s, h);
    if (e != cudaSuccess)
        return cuda_status(e, "vsmc_cuda_resample_mn");
    if (h.error != 0) {
        set_last_error("vsmc_cuda_resample_mn: replication did not sum to N");
        return h.error;
    }
    rng->offset = h.offset;
    return VSMC_CUDA_OK;
}

int vsmc_cuda_copy_f64(uint64_t N, uint32_t dim, const double *src,
                       double *dst, const int32_t *copy_from, void *stream)
{
    if (N == 0 || src == nullptr || dst == nullptr || copy_from == nullptr ||
        src == dst) {
        set_last_error("vsmc_cuda_copy_f64: invalid arguments");
        return VSMC_CUDA_EINVAL;
    }
    k_copy_f64<<<(unsigned)((N + 255) / 256), 256, 0,
                 static_cast<cudaStream_t>(stream)>>>((long long)N, dim, src,
                                                      dst, copy_from);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? VSMC_CUDA_OK
                            : cuda_status(e, "vsmc_cuda_copy_f64");
}

int vsmc_cuda_math_eval(int fn, uint64_t n, const double *in, double *out,
                        void *stream)
{
    if ((fn != 0 && fn != 1) || n == 0 || in == nullptr || out == nullptr) {
        set_last_error("vsmc_cuda_math_eval: invalid arguments");
        return VSMC_CUDA_EINVAL;
    }
    const long long blocks = ((long long)n + 255) / 256;
    k_math_eval<<<(unsigned)(blocks < 4736 ? blocks : 4736), 256, 0,
                  static_cast<cudaStream_t>(stream)>>>(fn, (long long)n, in,
                                                       out);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? VSMC_CUDA_OK
                            : cuda_status(e, "vsmc_cuda_math_eval");
}

int vsmc_cuda_device_alloc(size_t bytes, void **ptr)
{
    if (ptr == nullptr) {
        set_last_error("vsmc_cuda_device_alloc: null pointer");
        return VSMC_CUDA_EINVAL;
    }
    *ptr = nullptr;
    if (bytes == 0)
        return VSMC_CUDA_OK;
    cudaError_t e = cudaMalloc(ptr, bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        *ptr = nullptr;
        set_last_error("vsmc_cuda_device_alloc: cudaMalloc of " +
                       std::to_string(bytes) + " bytes failed");
        return VSMC_CUDA_ENOMEM;
    }
    return VSMC_CUDA_OK;
}

int vsmc_cuda_device_free(void *ptr)
{
    if (ptr == nullptr)
        return VSMC_CUDA_OK;
    cudaError_t e = cudaFree(ptr);
    return e == cudaSuccess ? VSMC_CUDA_OK
                            : cuda_status(e, "vsmc_cuda_device_free");
}

int vsmc_cuda_memcpy(void *dst, const void *src, size_t bytes, int kind,
                     void *stream)
{
    cudaMemcpyKind k;
    switch (kind) {
    case VSMC_CUDA_HOST_TO_DEVICE:
        k = cudaMemcpyHostToDevice;
        break;
    case VSMC_CUDA_DEVICE_TO_HOST:
        k = cudaMemcpyDeviceToHost;
        break;
    case VSMC_CUDA_DEVICE_TO_DEVICE:
        k = cudaMemcpyDeviceToDevice;
        break;
    default:
        set_last_error("vsmc_cuda_memcpy: unknown direction");
        return VSMC_CUDA_EINVAL;
    }
    if (bytes == 0)
        return VSMC_CUDA_OK;
    if (dst == nullptr || src == nullptr) {
        set_last_error("vsmc_cuda_memcpy: null pointer");
        return VSMC_CUDA_EINVAL;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaMemcpyAsync(dst, src, bytes, k, s);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s);
    return e == cudaSuccess ? VSMC_CUDA_OK : cuda_status(e, "vsmc_cuda_memcpy");
}

int vsmc_cuda_stream_synchronize(void *stream)
{
    cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? VSMC_CUDA_OK
                            : cuda_status(e, "vsmc_cuda_stream_synchronize");
}

} // extern "C"
