/*
 * launch.cu -- picks and launches the encode kernels (kernels.cu) of a step or
 * a picture, and reads their counters.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "h261b_device.h"
#include "parts.h"

using namespace h261b;

namespace {

const KernelPart *const g_parts[8] = { &kernel_part_0, &kernel_part_1, &kernel_part_2, &kernel_part_3,
                                       &kernel_part_4, &kernel_part_5, &kernel_part_6, &kernel_part_7 };
/* parts a launch has used: the counters of the others are zero, and reading
 * them would load their modules */
std::atomic<bool> g_used[8];

const KernelPart &part_of(bool fmad, bool full, bool bulk)
{
    const int i = (fmad ? 4 : 0) | (full ? 2 : 0) | (bulk ? 1 : 0);
    g_used[i].store(true, std::memory_order_relaxed);
    return *g_parts[i];
}

} // namespace

extern "C" int h261b_debug_check_status(int32_t *enabled, int64_t *violations, int32_t *first_site,
                                        int32_t *first_value)
{
    if (!enabled || !violations || !first_site || !first_value)
        return H261B_ERR_ARG;
    *violations = 0;
    *first_site = *first_value = 0;
#ifdef H261B_DEBUG_CHECKS
    *enabled = 1;
    for (int i = 0; i < 8; i++) {
        unsigned long long n = 0;
        int first[2] = { 0, 0 };
        if (!g_used[i])
            continue;
        if (g_parts[i]->checks(&n, first) != H261B_OK)
            return H261B_ERR_CUDA;
        if (n && !*violations) {
            *first_site = first[0];
            *first_value = first[1];
        }
        *violations += (int64_t)n;
    }
#else
    *enabled = 0;
#endif
    return H261B_OK;
}

extern "C" int h261b_stage_status(int64_t *timeouts)
{
    if (!timeouts)
        return H261B_ERR_ARG;
    int64_t sum = 0;
    for (int i = 1; i < 8; i += 2) {   /* the bulk parts */
        unsigned int n = 0;
        if (g_used[i] && g_parts[i]->timeouts(&n) != H261B_OK)
            return H261B_ERR_CUDA;
        sum += n;
    }
    *timeouts = sum;
    return H261B_OK;
}

extern "C" int h261b_launch_step(const h261b_session_dev_t *sessions_dev, const uint32_t *work_dev,
                                 int32_t n_work, int32_t phases, int32_t warps_per_cta, int32_t max_ctas,
                                 int32_t *sched_dev, void *stream)
{
    if (n_work <= 0)
        return 0;
    if (warps_per_cta < 1 || warps_per_cta > 8)
        return (int)cudaErrorInvalidValue;
    const int fmad = (phases >> 8) & 1;
    if (phases & H261B_LAUNCH_TEAM) {
        const bool full = (phases & H261B_LAUNCH_ME_FULL) != 0, code = (phases & H261B_CODE_INLINE) != 0;
        if (phases & (H261B_ABI_OUT | H261B_STAGE_BULK | (3 << H261B_KIND_SHIFT)))
            return (int)cudaErrorInvalidValue;
        const TeamFn fn = part_of(fmad, full, 0).team(code);
        fn<<<n_work, TEAM_THREADS, 0, (cudaStream_t)stream>>>(sessions_dev, work_dev, phases & 0xFF);
        return (int)cudaGetLastError();
    }
    int kind = (phases >> H261B_KIND_SHIFT) & 3;
    /* a fused launch of every phase runs the kernel compiled for exactly that */
    const int all_phases = H261B_PHASE_ME | H261B_PHASE_MD | H261B_PHASE_ENCDEC;
    if (kind == KIND_FUSED && (phases & all_phases) == all_phases)
        kind = KIND_FULL;
    const int full = (phases & H261B_LAUNCH_ME_FULL) ? 1 : 0, abi = (phases & H261B_ABI_OUT) ? 1 : 0;
    const int bulk = (phases & H261B_STAGE_BULK) ? 1 : 0;
    const int code = (phases & H261B_CODE_INLINE) ? 1 : 0;
    const bool pdl = (phases & H261B_LAUNCH_PDL) != 0;
    const int tail_code = (phases >> H261B_TAIL_SHIFT) & 15;
    if (kind > KIND_FULL)
        return (int)cudaErrorInvalidValue;
    const int ph = phases & (0xFF | H261B_STAGE_SHORT | H261B_LAUNCH_PDL);
    const int threads = warps_per_cta * 32;
    /* the reference-layout outputs come with cp.async staging and no coding,
     * the encode kind with the reference search's part */
    const bool fused_abi = abi && kind != KIND_SEARCH && kind != KIND_ENCODE;
    const bool codes = code && kind != KIND_SEARCH && !fused_abi;
    const KernelPart &part = part_of(fmad, full && kind != KIND_ENCODE, bulk && !fused_abi);
    const size_t warp_bytes = kind == KIND_SEARCH ? part.search_bytes : codes ? part.code_bytes : part.encode_bytes;
    const size_t smem = warp_bytes * (size_t)warps_per_cta + (codes ? part.table_bytes : 0);
    const StepFn fn = part.step(kind, abi, code);
    static std::mutex mu;
    static int sms[64], resident[64][2][4][2][2][2][2][9];
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess || dev < 0 || dev >= 64)
        return (int)(err != cudaSuccess ? err : cudaErrorInvalidDevice);
    int per_sm = 0, nsm = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!sms[dev]) {
            if ((err = cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
                return (int)err;
        }
        int &r = resident[dev][fmad][kind][full][abi][bulk][code][warps_per_cta];
        if (!r) {
            /* the first launch of this instantiation.  CUDA loads a kernel when
             * it is first named: naming all 52 here took 2.5 ms of a process's
             * first launch (a QCIF stream's first 40 pictures 14.2 ms, 12.0 so) */
            err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(part.code_bytes * 8 + part.table_bytes));
            if (err != cudaSuccess)
                return (int)err;
            err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, fn, threads, smem);
            if (err != cudaSuccess)
                return (int)err;
            r = r < 1 ? 1 : r;
        }
        per_sm = r;
        nsm = sms[dev];
    }
    /* one wave of resident CTAs */
    int ctas = max_ctas > 0 ? max_ctas : nsm * per_sm;
    int chunk;
    /* a MB a warp at most: nothing to balance, and no draw (an atomic's round
     * trip before the first MB and one more after the last) */
    if (n_work <= (long long)ctas * warps_per_cta)
        sched_dev = nullptr;
    if (sched_dev) {
        /* static runs of all but about `tail` items per warp, the rest drawn
         * from the scheduler (tail_code: tail + 1, 0 for the default 2) */
        const int tail = tail_code ? tail_code - 1 : 2;
        ctas = (int)std::min<long long>(ctas, (n_work + warps_per_cta - 1) / warps_per_cta);
        const long long total_warps = (long long)ctas * warps_per_cta;
        chunk = (int)std::max<long long>(0, n_work / total_warps - tail);
    } else {
        /* contiguous runs covering every item */
        const long long total_warps = (long long)ctas * warps_per_cta;
        chunk = (int)((n_work + total_warps - 1) / total_warps);
        ctas = (n_work + chunk * warps_per_cta - 1) / (chunk * warps_per_cta);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return (int)cudaLaunchKernelEx(&cfg, fn, sessions_dev, work_dev, n_work, chunk, ph, sched_dev);
}

extern "C" int h261b_launch_team_picture(const h261b_session_dev_t *session, int32_t phases, void *stream)
{
    const bool fmad = (phases & H261B_FMAD_BIT) != 0, full = (phases & H261B_LAUNCH_ME_FULL) != 0;
    const TeamPictureFn fn = part_of(fmad, full, false).team_picture((phases & H261B_ABI_OUT) != 0);
    fn<<<session->mbw * session->mbh, TEAM_THREADS, 0, (cudaStream_t)stream>>>(*session, phases & 0xFF);
    return (int)cudaGetLastError();
}

/* ------------------------------------------------ SAD primitive peak */

namespace {

/* the motion search's inner step, on registers: one funnel shift and one
 * 4-pixel SAD per word, eight independent chains per thread */
__global__ void __launch_bounds__(256) sad_peak_kernel(const uint32_t *__restrict__ in, uint32_t *__restrict__ out,
                                                       int iters)
{
    uint32_t c[8], r[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        c[i] = in[(threadIdx.x + i) & 255];
        r[i] = in[(threadIdx.x * 7 + i) & 255];
    }
    uint32_t acc = 0;
    for (int it = 0; it < iters; it++) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            acc = sad4(c[i], r[i], acc);
            r[i] = __funnelshift_r(r[i], r[(i + 1) & 7], 8);
        }
    }
    out[blockIdx.x * blockDim.x + threadIdx.x] = acc;
}

} // namespace

extern "C" int h261b_measure_sad_peak(int32_t device, double *absdiff_per_s)
{
    if (!absdiff_per_s)
        return -1;
    int sms = 0;
    if (cudaSetDevice(device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return -2;
    const int blocks = sms * 8, threads = 256, iters = 2048;
    uint32_t *in = nullptr, *out = nullptr;
    uint32_t h[256];
    for (int i = 0; i < 256; i++)
        h[i] = (uint32_t)i * 2654435761u;
    cudaEvent_t a, b;
    float ms = 0.f;
    int rc = -2;
    if (cudaMalloc(&in, sizeof(h)) == cudaSuccess && cudaMalloc(&out, sizeof(uint32_t) * blocks * threads) == cudaSuccess &&
        cudaMemcpy(in, h, sizeof(h), cudaMemcpyHostToDevice) == cudaSuccess && cudaEventCreate(&a) == cudaSuccess &&
        cudaEventCreate(&b) == cudaSuccess) {
        sad_peak_kernel<<<blocks, threads>>>(in, out, 64);
        cudaEventRecord(a);
        sad_peak_kernel<<<blocks, threads>>>(in, out, iters);
        cudaEventRecord(b);
        if (cudaEventSynchronize(b) == cudaSuccess && cudaEventElapsedTime(&ms, a, b) == cudaSuccess && ms > 0.f) {
            *absdiff_per_s = (double)blocks * threads * iters * 8 * 4 / (ms * 1e-3);
            rc = 0;
        }
        cudaEventDestroy(a);
        cudaEventDestroy(b);
    }
    cudaFree(in);
    cudaFree(out);
    return rc;
}
