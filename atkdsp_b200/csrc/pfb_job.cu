/* The small kernels around a tile launch: the job table from launch parameters
 * or a device-held offset before it, the W2 sums after it. In a file of their
 * own, because a process's first use of a file's kernel loads all of the
 * file's: beside the kernel of every shape that was 12 ms of a handle's first
 * call, here 0.3. */
#include <cuda_runtime.h>
#include <stdint.h>
#include "internal.h"

namespace {
#include "pfb_dev.cuh"
}

/* The constants of nel device jobs (and their carries) whose int16 offset
 * lives in device memory, written into the job table after its upload and
 * before the tile kernel reads it: the tile kernel itself stays unchanged. */
__global__ void conv_from_offset_kernel(atkb_job *jobs, atkb_carry *carries, int nel) {
    /* let the tile kernel launch now: it waits for this grid's completion
     * (griddepcontrol.wait) before it reads the table */
    asm volatile("griddepcontrol.launch_dependents;");
    const int e = threadIdx.x;
    if (e >= nel || !jobs[e].doff) return;
    float cre, cim;
    doff_consts(jobs[e].doff, jobs[e].kscale, cre, cim);
    jobs[e].cre = carries[e].cre = cre;
    jobs[e].cim = carries[e].cim = cim;
}

/* A one-job table from the launch's own parameters (no host->device copy):
 * the job, its carry and the tile starts, the int16 constants derived from
 * the device-held offset when the job has one. */
__global__ void job_from_params_kernel(const atkb_job J, const atkb_carry C, int tiles, atkb_job *jobs,
                                       atkb_carry *carries, int *tile_start) {
    asm volatile("griddepcontrol.launch_dependents;");
    if (threadIdx.x != 0) return;
    atkb_job j = J;
    atkb_carry c = C;
    if (j.doff) {
        float cre, cim;
        doff_consts(j.doff, j.kscale, cre, cim);
        j.cre = c.cre = cre;
        j.cim = c.cim = cim;
    }
    jobs[0] = j;
    carries[0] = c;
    tile_start[0] = 0;
    tile_start[1] = tiles;
}

extern "C" int atkb_pfb_job_from_params(const atkb_job *J, const atkb_carry *C, int tiles, atkb_job *d_jobs,
                                        atkb_carry *d_carry, int *d_tile_start, void *stream) {
    job_from_params_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(*J, *C, tiles, d_jobs, d_carry, d_tile_start);
    return cudaGetLastError() == cudaSuccess ? ATKB_OK : ATKB_E_KERNEL;
}

extern "C" int atkb_pfb_conv_from_offset(atkb_job *d_jobs, atkb_carry *d_carry, int nel, void *stream) {
    if (nel < 1 || nel > 1024) return ATKB_E_ARG;
    conv_from_offset_kernel<<<1, nel, 0, (cudaStream_t)stream>>>(d_jobs, d_carry, nel);
    return cudaGetLastError() == cudaSuccess ? ATKB_OK : ATKB_E_KERNEL;
}

namespace {
/* the tiles' W2 partials of one single-element job, per channel: W2 power
 * (S / m), and W1 for one element (R[k] += S, counts += m), gated like
 * atkb_w12. A block of W2F_WARPS warps takes W2F_CH = 8 channels: lane l of
 * warp w reads channel l % 8 of the tiles t = s, s + 64, ... (s = 4w + l / 8,
 * 64 tile streams; sixteen loads in flight, each quarter-warp one 64-byte
 * row segment). The 64 stream sums of a channel are then added by a fixed tree
 * (eight groups of eight in stream order, then the eight group sums in
 * order), so the result is deterministic. Eight channels a block spread the
 * reads of nchan 1024 over 128 SMs. */
#define W2F_WARPS 16
#define W2F_CH 8
#define W2F_STREAMS (W2F_WARPS * 32 / W2F_CH)
__global__ void __launch_bounds__(32 * W2F_WARPS)
w2_finish_kernel(const double *__restrict__ part, int tiles, int M, long long m, const uint8_t *__restrict__ gate,
                 float2 *__restrict__ R, uint32_t *__restrict__ counts, float *__restrict__ pwr,
                 float *__restrict__ mean_pwr) {
    /* launched as a programmatic dependent of the tile kernel: wait for it */
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ double red[W2F_STREAMS][W2F_CH];
    __shared__ double grp[W2F_STREAMS / 8][W2F_CH];
    const int c = threadIdx.x % W2F_CH, sidx = threadIdx.x / W2F_CH;
    const int k = blockIdx.x * W2F_CH + c;
    double S = 0.0;
    if (k < M) {
        /* sixteen loads in flight, the ones past the last tile read as +0.0
         * (S >= +0.0, so adding it is exact and the order is unchanged) */
        for (int t = sidx; t < tiles; t += 16 * W2F_STREAMS) {
            double v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                const int r = t + u * W2F_STREAMS;
                v[u] = r < tiles ? __ldg(part + (long long)r * M + k) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 16; ++u) S += v[u];
        }
    }
    red[sidx][c] = S;
    __syncthreads();
    if (threadIdx.x < (W2F_STREAMS / 8) * W2F_CH) {
        const int g = threadIdx.x / W2F_CH;
        double G = 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) G += red[8 * g + j][c];
        grp[g][c] = G;
    }
    __syncthreads();
    if (threadIdx.x >= W2F_CH || k >= M) return;
    S = 0.0;
#pragma unroll
    for (int g = 0; g < W2F_STREAMS / 8; ++g) S += grp[g][c];
    const double inv = m ? 1.0 / (double)m : 0.0;
    if (pwr) pwr[k] = (float)(S * inv);
    if (mean_pwr) mean_pwr[k] = (float)((S * inv) / 1.0);
    if (R && counts && (!gate || gate[k])) {
        if (m > 0) {
            const float2 v = R[k];
            R[k] = make_float2((float)((double)v.x + S), (float)((double)v.y + 0.0));
        }
        counts[k] += (uint32_t)m;
    }
}
}  // namespace

extern "C" int atkb_w2_finish(const double *part, int tiles, int nchan, long long m, const uint8_t *gate, void *R,
                              uint32_t *counts, float *pwr, float *mean_pwr, void *stream) {
    /* a programmatic dependent of the tile kernel launched just before it on
     * the stream: its launch overlaps that kernel's last tiles and carries */
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((nchan + W2F_CH - 1) / W2F_CH));
    cfg.blockDim = dim3(32 * W2F_WARPS);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, w2_finish_kernel, part, tiles, nchan, m, gate, (float2 *)R,
                                             counts, pwr, mean_pwr);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? ATKB_OK : ATKB_E_KERNEL;
}
