// lbm_fieldcalc.cu -- fieldCalculate's containsNaN / spatialMean on the device.
//
// The reference's fieldCalculate reads each saved time's ten moment fields
// to the host and loops over them there (applications/fieldCalculate/
// fieldCalculate.cuh:74-170): a field "contains NaN" if any value is NaN
// (std::isnan; infinities do not count), and its spatial mean is the float
// sum of its values in global node order (x fastest, fileInput.cuh:777-820
// de-interleaves the block-tiled file into that order), added left to right
// from 0 and divided by float(nodes).  Here both run on the GPU:
//
//  * stats_kernel / stats_finish_kernel: NaN count and an FP64 sum per field,
//    a grid-wide reduction in a fixed order (repeatable bit for bit), the
//    accurate mean the solver's monitor also reports;
//  * ordered_sum_kernel: the reference's left-to-right float sum, which
//    rounds after every addition and so cannot be reassociated: one chain of
//    dependent additions per field, all fields at once.  Its printed value is
//    what the reference prints, digit for digit.
//
// The fields are copied to the device in slices of z, and a slice's additions
// run while the next slices are copied.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "lbm_b200.h"
#include "lbm_handle.hpp"

namespace {

constexpr int kStatsThreads = 256;
constexpr int kStatsBlocksPerField = 256;
constexpr int kOrderedChunk = 4096;    // values staged in shared memory at a time
constexpr int kOrderedThreads = 256;   // warp 0 adds, the warps of other schedulers fetch
constexpr int kMaxSlices = 16;
constexpr size_t kSliceBytes = size_t(8) << 20;  // of all fields, at least

__device__ __forceinline__ size_t tiled_address(int x, int y, size_t z, int nbx, int nby)
{
    const size_t tx = x & 7, ty = y & 7, tz = z & 7, bx = x >> 3, by = y >> 3, bz = z >> 3;
    return tx + 8 * (ty + 8 * (tz + 8 * (bx + size_t(nbx) * (by + size_t(nby) * bz))));
}

// grid (kStatsBlocksPerField, fields): partial FP64 sums and NaN counts per block
__global__ void __launch_bounds__(kStatsThreads) stats_kernel(const float *fields, size_t N, double *part_sum,
                                                                unsigned long long *part_nan)
{
    const float *f = fields + size_t(blockIdx.y) * N;
    double s = 0.0;
    unsigned long long nan = 0;
    for (size_t i = blockIdx.x * size_t(kStatsThreads) + threadIdx.x; i < N; i += size_t(gridDim.x) * kStatsThreads) {
        const float v = f[i];
        if (isnan(v))
            nan++;
        else
            s += double(v);
    }
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, o);
        nan += __shfl_down_sync(0xffffffffu, nan, o);
    }
    __shared__ double ws[kStatsThreads / 32];
    __shared__ unsigned long long wn[kStatsThreads / 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        ws[warp] = s;
        wn[warp] = nan;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        unsigned long long n = 0;
        for (int w = 0; w < kStatsThreads / 32; w++) {
            t += ws[w];
            n += wn[w];
        }
        part_sum[size_t(blockIdx.y) * gridDim.x + blockIdx.x] = t;
        part_nan[size_t(blockIdx.y) * gridDim.x + blockIdx.x] = n;
    }
}

// one thread per field: the blocks' partials in block order
__global__ void stats_finish_kernel(const double *part_sum, const unsigned long long *part_nan, int blocks,
                                    int fields, size_t N, double *mean, unsigned long long *nan)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= fields)
        return;
    double t = 0.0;
    unsigned long long n = 0;
    for (int b = 0; b < blocks; b++) {
        t += part_sum[size_t(k) * blocks + b];
        n += part_nan[size_t(k) * blocks + b];
    }
    mean[k] = t / double(N);
    nan[k] = n;
}

// The left-to-right float sum, in global order, of the values [g0, g1) of
// field blockIdx.x, continuing from carry[field]; the last slice (g1 == N)
// writes the mean.  What bounds it is the latency of a dependent addition:
// warp 0 does nothing but add (every lane the same chain, from shared memory
// by 16-byte broadcasts read 32 values ahead), six warps on the other three
// schedulers fetch the next chunk.  Ten fields of 192x168x176: 14.4 ms, 2.5 ns
// or 4.9 cycles per addition (one warp that fetched and added in turn: 35.1
// ms, 6.2 ns); the whole call from pageable memory 56.9 -> 23.9 ms.
__global__ void __launch_bounds__(kOrderedThreads) ordered_sum_kernel(const float *fields, size_t N, int nx, int ny,
                                                                      int tiled, size_t g0, size_t g1, float *carry,
                                                                      float *mean_ref)
{
    constexpr int kAhead = 32;  // values the adding warp reads before it needs them
    __shared__ __align__(16) float chunk[2][kOrderedChunk + kAhead];
    const float *f = fields + size_t(blockIdx.x) * N;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool adder = warp == 0, fetcher = (warp & 3) != 0;
    // fetching threads: warps 1, 2, 3, 5, 6, 7
    constexpr int kFetchers = 6 * 32;
    const int id = (warp < 4 ? warp - 1 : warp - 2) * 32 + lane;
    const size_t chunks = (g1 - g0 + kOrderedChunk - 1) / kOrderedChunk;
    auto fetch = [&](size_t c) {
        float *dst = chunk[c & 1];
        size_t g = g0 + c * kOrderedChunk + id;
        // (x, y, z) of the first value, then advanced with the index
        const size_t row = g / size_t(nx);
        int x = int(g - row * size_t(nx)), y = int(row % size_t(ny));
        size_t z = row / size_t(ny);
        for (int j = id; j < kOrderedChunk && g < g1; j += kFetchers, g += kFetchers) {
            dst[j] = __ldg(f + (tiled ? tiled_address(x, y, z, nx >> 3, ny >> 3) : g));
            if (!tiled)
                continue;
            x += kFetchers;
            while (x >= nx) {
                x -= nx;
                if (++y == ny) {
                    y = 0;
                    ++z;
                }
            }
        }
    };
    float sum = carry[blockIdx.x];
    if (fetcher && chunks > 0)
        fetch(0);
    __syncthreads();
    for (size_t c = 0; c < chunks; c++) {
        if (adder) {
            const float *v = chunk[c & 1];
            const size_t left = g1 - g0 - c * kOrderedChunk;
            const int n = left < size_t(kOrderedChunk) ? int(left) : kOrderedChunk;
            float4 cur[kAhead / 4], nxt[kAhead / 4];
            const float4 *q = reinterpret_cast<const float4 *>(v);
            auto read = [&](float4 *to, int i) {
#pragma unroll
                for (int k = 0; k < kAhead / 4; k++)
                    to[k] = q[i / 4 + k];
            };
            auto add = [&](const float4 *from) {
#pragma unroll
                for (int k = 0; k < kAhead / 4; k++) {
                    sum = __fadd_rn(sum, from[k].x);
                    sum = __fadd_rn(sum, from[k].y);
                    sum = __fadd_rn(sum, from[k].z);
                    sum = __fadd_rn(sum, from[k].w);
                }
            };
            read(cur, 0);
            int i = 0;
            for (; i + 2 * kAhead <= n; i += 2 * kAhead) {
                read(nxt, i + kAhead);
                add(cur);
                read(cur, i + 2 * kAhead);  // past the chunk's end: padding, not added
                add(nxt);
            }
            for (; i < n; i++)
                sum = __fadd_rn(sum, v[i]);
        } else if (fetcher && c + 1 < chunks) {
            fetch(c + 1);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        carry[blockIdx.x] = sum;
        if (g1 == N)
            mean_ref[blockIdx.x] = __fdiv_rn(sum, float(N));
    }
}

}  // namespace

extern "C" {

lbm_status lbm_field_statistics(int32_t device, const float *fields, int64_t nx, int64_t ny, int64_t nz,
                                int32_t nfields, lbm_order order, int32_t *nan_count, float *mean_ref,
                                double *mean)
{
    if (!fields || !nan_count || !mean_ref || !mean)
        return lbm::record_error(LBM_ERR_ARG, "lbm_field_statistics: null argument");
    if (nx <= 0 || ny <= 0 || nz <= 0 || nfields <= 0 || nfields > 65535)
        return lbm::record_error(LBM_ERR_ARG, "lbm_field_statistics: empty mesh or field count out of range");
    if (order != LBM_ORDER_GLOBAL && order != LBM_ORDER_TILED)
        return lbm::record_error(LBM_ERR_ARG, "lbm_field_statistics: unknown order");
    if (order == LBM_ORDER_TILED && (nx % 8 || ny % 8 || nz % 8))
        return lbm::record_error(LBM_ERR_ARG, "lbm_field_statistics: the tiled order needs multiples of 8");
    if (nx > (1 << 30) || ny > (1 << 30))
        return lbm::record_error(LBM_ERR_ARG, "lbm_field_statistics: mesh dimension too large");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
        return lbm::record_error(LBM_ERR_ARG, "lbm_field_statistics: device ordinal out of range");
    LBM_CUDA_RETURN(cudaSetDevice(device));
    const size_t N = size_t(nx) * size_t(ny) * size_t(nz);
    const size_t bytes = N * size_t(nfields) * sizeof(float);
    const int blocks = kStatsBlocksPerField;
    const size_t parts = size_t(blocks) * size_t(nfields);
    float *d_fields = nullptr, *d_ref = nullptr, *d_carry = nullptr;
    double *d_part = nullptr, *d_mean = nullptr;
    unsigned long long *d_pnan = nullptr, *d_nan = nullptr;
    cudaStream_t st = nullptr, cs = nullptr;  // kernels, copies
    cudaEvent_t copied[kMaxSlices] = {};
    auto release = [&]() {
        for (cudaStream_t q : {cs, st})
            if (q)
                cudaStreamSynchronize(q);
        for (cudaEvent_t v : copied)
            if (v)
                cudaEventDestroy(v);
        cudaFree(d_carry);
        cudaFree(d_fields);
        cudaFree(d_ref);
        cudaFree(d_part);
        cudaFree(d_mean);
        cudaFree(d_pnan);
        cudaFree(d_nan);
        for (cudaStream_t q : {cs, st})
            if (q)
                cudaStreamDestroy(q);
    };
    // slices of whole planes (tiled order: of whole 8-plane blocks), which are
    // contiguous in every field
    const size_t unit = size_t(nx) * size_t(ny) * (order == LBM_ORDER_TILED ? 8 : 1), units = N / unit;
    const int slices = int(std::min<size_t>({units, size_t(kMaxSlices), std::max<size_t>(1, bytes / kSliceBytes)}));
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess)
        e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
    for (int k = 0; k < slices && e == cudaSuccess; k++)
        e = cudaEventCreateWithFlags(&copied[k], cudaEventDisableTiming);
    if (e == cudaSuccess)
        e = cudaMalloc(&d_carry, size_t(nfields) * sizeof(float));
    if (e == cudaSuccess)
        e = cudaMemsetAsync(d_carry, 0, size_t(nfields) * sizeof(float), st);
    if (e == cudaSuccess)
        e = cudaMalloc(&d_fields, bytes);
    if (e == cudaSuccess)
        e = cudaMalloc(&d_ref, size_t(nfields) * sizeof(float));
    if (e == cudaSuccess)
        e = cudaMalloc(&d_part, parts * sizeof(double));
    if (e == cudaSuccess)
        e = cudaMalloc(&d_mean, size_t(nfields) * sizeof(double));
    if (e == cudaSuccess)
        e = cudaMalloc(&d_pnan, parts * sizeof(unsigned long long));
    if (e == cudaSuccess)
        e = cudaMalloc(&d_nan, size_t(nfields) * sizeof(unsigned long long));
    for (int k = 0; k < slices && e == cudaSuccess; k++) {
        const size_t g0 = units * k / slices * unit, g1 = units * (k + 1) / slices * unit;
        for (int32_t v = 0; v < nfields && e == cudaSuccess; v++)
            e = cudaMemcpyAsync(d_fields + size_t(v) * N + g0, fields + size_t(v) * N + g0, (g1 - g0) * sizeof(float),
                                cudaMemcpyHostToDevice, cs);
        if (e == cudaSuccess)
            e = cudaEventRecord(copied[k], cs);
        if (e == cudaSuccess)
            e = cudaStreamWaitEvent(st, copied[k], 0);
        if (e == cudaSuccess) {
            ordered_sum_kernel<<<unsigned(nfields), kOrderedThreads, 0, st>>>(
                d_fields, N, int(nx), int(ny), order == LBM_ORDER_TILED ? 1 : 0, g0, g1, d_carry, d_ref);
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) {
        stats_kernel<<<dim3(blocks, unsigned(nfields)), kStatsThreads, 0, st>>>(d_fields, N, d_part, d_pnan);
        stats_finish_kernel<<<(nfields + 127) / 128, 128, 0, st>>>(d_part, d_pnan, blocks, nfields, N, d_mean, d_nan);
        e = cudaGetLastError();
    }
    std::vector<unsigned long long> nan(static_cast<size_t>(nfields));
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(nan.data(), d_nan, nan.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(mean, d_mean, size_t(nfields) * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(mean_ref, d_ref, size_t(nfields) * sizeof(float), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(st);
    release();
    if (e != cudaSuccess)
        return lbm::record_error(e == cudaErrorMemoryAllocation ? LBM_ERR_NOMEM : LBM_ERR_CUDA,
                                 std::string("lbm_field_statistics: ") + cudaGetErrorString(e));
    for (int32_t k = 0; k < nfields; k++)
        nan_count[k] = nan[size_t(k)] > 0x7fffffffull ? 0x7fffffff : int32_t(nan[size_t(k)]);
    return LBM_OK;
}

}  // extern "C"
