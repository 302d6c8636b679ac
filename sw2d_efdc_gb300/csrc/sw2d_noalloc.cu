/* State measure on caller-owned device arrays that allocates nothing
 * (declared in include/sw2d_noalloc.h).
 *
 * The kernel is the measuring half of the FP64 path's prime kernel (volume
 * of the active cells and the exact CFL face-speed maxima) over the
 * reference-orientation arrays, with the partial results in a
 * file-scope device array instead of a buffer the handle allocates.  Compiled
 * with --fmad=false like the FP64 step, so the face speeds round exactly as
 * the step's own.
 */
#include "sw2d.h"
#include "sw2d_noalloc.h"

#include "sw2d_math.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>

namespace sw2d {
void set_error_message(const char* msg); /* sw2d_api.cu: the message sw2d_last_error returns */
}

namespace {

constexpr int kTile = SW2D_NOALLOC_TILE;              /* of the raster limit (sw2d_noalloc.h) */
constexpr int kMaxTiles = SW2D_NOALLOC_MAX_TILES;
constexpr int kBand = 32;                             /* most rows of a warp's task */
constexpr int kBatch = 4;                             /* of them read at once */
constexpr int kBlocksPerSm = 3;
constexpr int kBlocks = kBlocksPerSm * 152;           /* the most: GB300's SMs */
constexpr int kSlots = 3;                             /* a tile's share of the array, once its partials */
constexpr int kResult = kSlots * kMaxTiles;           /* x and y speed maxima (bits), then volume * area and speed */
constexpr int kCounter = kResult + 2;                 /* block-completion counter (low 32 bits) */
constexpr int kScratchDoubles = kCounter + 1;         /* 49,155 doubles = 393,240 bytes */

/* The scratch: the blocks' volumes (the array's size is the interface's), the
 * two maxima and then results, the counter. */
static __device__ __align__(256) double g_noalloc_scratch[kScratchDoubles];

static_assert(sizeof(double) * kScratchDoubles == 393240, "scratch size stated in sw2d_noalloc.h");
static_assert(kBlocks <= kResult && kBlocks == 456, "the blocks' volumes, as sw2d_noalloc.h states them");

/* (|velocity| + sqrt(g hm)) / spacing as the FP64 step evaluates it, raising a
 * running maximum kept as bits (non-negative doubles order like their bits).
 * A call: inlined, its binary64 instructions would be predicated, and one
 * that is predicated off still takes the FP64 pipe's 71 cycles. */
__device__ __noinline__ void raise_speed(unsigned long long* at, double q, double ha, double hb, double g, double rd) {
    const double hm = 0.50 * (ha + hb);
    const double vel = sw2d_div_rn(q, hm);
    const unsigned long long v = sw2d_f64_bits((fabs(vel) + sw2d_sqrt_rn(g * hm)) * rd);
    if (v > __ldcg(at)) atomicMax(at, v);
}
/* the same for a face whose mean depth is known by estimate only; one whose
 * mean depth is NaN has no speed */
__device__ __noinline__ void raise_speed_exact(unsigned long long* at, double q, double ha, double hb, double g, double rd,
                                               double th) {
    if (0.50 * (ha + hb) >= th) raise_speed(at, q, ha, hb, g, rd);
}
__device__ __noinline__ bool mean_ge_exact(double ha, double hb, double th) {
    return sw2d_ge_pos(0.50 * (ha + hb), th);
}
/* mean depth of a face >= th, exactly: decided from the two depths unless th
 * lies between them, then in binary32, in binary64 only within its error */
__device__ __forceinline__ bool mean_ge(double ha, double hb, float est, double th, float thf) {
    const bool a = sw2d_ge_pos(ha, th), b = sw2d_ge_pos(hb, th);
    if (a == b) return a;
    if (fabsf(est - thf) > 1e-5f * thf) return est > thf;
    return mean_ge_exact(ha, hb, th);
}

/* sum over the block in a fixed order, valid in thread 0 */
__device__ __forceinline__ double block_sum256(double v, double* sm) {
    const int tid = threadIdx.x;
    sm[tid] = v;
    __syncthreads();
    double t = 0.0;
    if (tid < 32) {
        for (int k = 0; k < 8; k++) t = __dadd_rn(t, sm[tid + 32 * k]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t = __dadd_rn(t, __shfl_down_sync(0xffffffffu, t, o));
    }
    __syncthreads();
    return t;
}

struct MeasureIn {
    const double *dem, *h, *qx, *qy;
    int R, C;
    double nodata, th, g, rdx, rdy, area;
    float thf, gf, rdxf, rdyf, est_most; /* StepParams' */
    int band; /* rows of a warp's task */
};

/* A warp takes tasks of 32 columns x `band` rows and walks down the rows, the
 * row above in registers, the column left of a lane's from its neighbour, so
 * each array is read once (plus the row above and the column left of a task);
 * kBatch rows are in flight at a time.  What it was bound by is the FP64
 * pipe, a binary64 instruction taking a warp 71 cycles: a division and a
 * square root on every face.  The face speeds are estimated in binary32
 * instead (within 2.2e-6), and only lanes within 1e-5 of the running maximum
 * are evaluated in binary64 and raise it, all lanes of a warp where an
 * estimate says nothing (est_most and above): the exact maximum in any order.
 * One binary64 addition a cell is left, the volume's.  Bounded by the latency
 * of HBM reads: 4 rows of 32-row tasks in flight at three blocks an SM
 * measured 136 us for the whole call at 4096 x 3000 (393 MB), 2 rows at four
 * or six blocks 159 and 220, 16-row tasks 186; 1320 before. */
__global__ void __launch_bounds__(256, kBlocksPerSm) k64_measure_noalloc(MeasureIn p, double* scratch) {
    __shared__ double sm[256];
    __shared__ bool last;
    const int tid = threadIdx.x, lane = tid & 31;
    const int R = p.R, C = p.C, sx_n = (C + 31) / 32;
    const int ntask = sx_n * ((R + p.band - 1) / p.band);
    const double th = p.th;
    const int64_t none = sw2d_ord(p.nodata);
    const bool any_none = p.nodata == p.nodata;
    unsigned long long* best = reinterpret_cast<unsigned long long*>(scratch + kResult);
    auto active = [&](double z) { return !(any_none && sw2d_ord(z) == none); }; /* z != nodata */
    double vol = 0.0;
    for (int task = (blockIdx.x * 256 + tid) >> 5; task < ntask; task += gridDim.x * 8) {
        const int band = task / sx_n, c = (task - band * sx_n) * 32 + lane;
        const int r0 = band * p.band, r1 = min(R, r0 + p.band);
        const bool in = c < C, left = lane == 0 && c > 0;
        bool act_n = false;
        double h_n = 0.0;
        if (in && r0 > 0) {
            const size_t i = (size_t)(r0 - 1) * C + c;
            h_n = p.h[i];
            act_n = active(p.dem[i]);
        }
        for (int r = r0; r < r1; r += kBatch) {
            double z[kBatch], h[kBatch], qx[kBatch], qy[kBatch], zl[kBatch], hl[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; k++) {
                const bool ok = in && r + k < r1;
                const size_t i = (size_t)(r + k) * C + c;
                z[k] = ok ? p.dem[i] : p.nodata;
                h[k] = ok ? p.h[i] : 0.0;
                qx[k] = ok ? p.qx[i] : 0.0;
                qy[k] = ok ? p.qy[i + r + k] : 0.0; /* rows of C + 1 */
                zl[k] = ok && left ? p.dem[i - 1] : p.nodata;
                hl[k] = ok && left ? p.h[i - 1] : 0.0;
            }
            float ex[kBatch], ey[kBatch], bx = 0.f, by = 0.f;
            double hw[kBatch], hn[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; k++) {
                const bool ok = in && r + k < r1;
                const bool act = ok && active(z[k]);
                if (act) vol = __dadd_rn(vol, h[k]);
                int aw = __shfl_up_sync(0xffffffffu, (int)act, 1);
                hw[k] = __shfl_up_sync(0xffffffffu, h[k], 1);
                if (lane == 0) {
                    aw = left && ok && active(zl[k]);
                    hw[k] = hl[k];
                }
                hn[k] = h_n;
                const float hf = sw2d_f32_est_depth(h[k]);
                const float mx = 0.5f * (hf + sw2d_f32_est_depth(h_n)), my = 0.5f * (hf + sw2d_f32_est_depth(hw[k]));
                const bool okx = act && act_n && mean_ge(h_n, h[k], mx, th, p.thf);
                const bool oky = act && aw && mean_ge(hw[k], h[k], my, th, p.thf);
                ex[k] = okx ? (fabsf(sw2d_f32_est_hi(qx[k])) * sw2d_rcp_est(mx) + sw2d_sqrt_est(p.gf * mx)) * p.rdxf : -1.f;
                ey[k] = oky ? (fabsf(sw2d_f32_est_hi(qy[k])) * sw2d_rcp_est(my) + sw2d_sqrt_est(p.gf * my)) * p.rdyf : -1.f;
                bx = fmaxf(bx, ex[k]);
                by = fmaxf(by, ey[k]);
                act_n = act;
                h_n = h[k];
            }
            const float cx = sw2d_f32_est_hi(__longlong_as_double((long long)__ldcg(best)));
            const float cy = sw2d_f32_est_hi(__longlong_as_double((long long)__ldcg(best + 1)));
            const float mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(bx)));
            const float my = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(by)));
            const float tx = fmaxf(mx, cx) * 0.99999f, ty = fmaxf(my, cy) * 0.99999f;
            if (!(mx < p.est_most && my < p.est_most)) {
                /* a negative, infinite or NaN depth or discharge, which would hide the warp's other faces: all of them */
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    if (!(ex[k] < 0.f)) raise_speed_exact(best, qx[k], h[k], hn[k], p.g, p.rdx, th);
                    if (!(ey[k] < 0.f)) raise_speed_exact(best + 1, qy[k], h[k], hw[k], p.g, p.rdy, th);
                }
                continue;
            }
            if (bx >= tx) {
#pragma unroll
                for (int k = 0; k < kBatch; k++)
                    if (ex[k] >= tx) raise_speed(best, qx[k], h[k], hn[k], p.g, p.rdx);
            }
            if (by >= ty) {
#pragma unroll
                for (int k = 0; k < kBatch; k++)
                    if (ey[k] >= ty) raise_speed(best + 1, qy[k], h[k], hw[k], p.g, p.rdy);
            }
        }
    }
    vol = block_sum256(vol, sm);
    if (tid == 0) {
        scratch[blockIdx.x] = vol;
        __threadfence();
        unsigned int* counter = reinterpret_cast<unsigned int*>(scratch + kCounter);
        last = (atomicAdd(counter, 1u) == gridDim.x - 1u);
    }
    __syncthreads();
    if (!last) return;
    /* the last block to finish combines the partials in a fixed order (every
     * block's raises come before its count) */
    __threadfence();
    double v = 0.0;
    for (unsigned k = tid; k < gridDim.x; k += 256) v = __dadd_rn(v, __ldcg(scratch + k));
    v = block_sum256(v, sm);
    if (tid == 0) {
        const double a = __longlong_as_double((long long)__ldcg(best)), w = __longlong_as_double((long long)__ldcg(best + 1));
        scratch[kResult + 0] = __dmul_rn(v, p.area);
        scratch[kResult + 1] = __dadd_rn(a, w);
    }
}

int reject(int code, const char* msg) {
    sw2d::set_error_message(msg);
    return code;
}

int cuda_fail(const char* what, cudaError_t e) {
    char buf[256];
    std::snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
    sw2d::set_error_message(buf);
    return SW2D_ERR_CUDA;
}

} // namespace

extern "C" int sw2d_measure_state_noalloc(const double* d_dem, const double* d_depth, const double* d_qx,
                                          const double* d_qy, int rows, int cols, double dx, double dy,
                                          double nodata, double th, double g, void* stream, double* volume_out,
                                          double* speed_out) {
    if (!d_dem || !d_depth || !d_qx || !d_qy || !volume_out || !speed_out)
        return reject(SW2D_ERR_INVALID, "null argument");
    if (rows < 1 || cols < 1) return reject(SW2D_ERR_INVALID, "rows and cols must be >= 1");
    if (!(dx > 0.0) || !(dy > 0.0) || !(th > 0.0) || !(g > 0.0))
        return reject(SW2D_ERR_INVALID, "dx, dy, th and g must be > 0");
    if (static_cast<long long>(rows) * cols > (1LL << 30))
        return reject(SW2D_ERR_INVALID, "rows * cols above 2^30 cells");
    const long long tiles_x = (static_cast<long long>(cols) + kTile - 1) / kTile;
    const long long tiles_y = (static_cast<long long>(rows) + kTile - 1) / kTile;
    if (tiles_x * tiles_y > kMaxTiles) {
        char buf[200];
        std::snprintf(buf, sizeof buf,
                      "raster %d x %d spans %lld tiles of 32 x 32 cells; the no-allocation measure holds at most "
                      "%d (its scratch is fixed at 393,240 bytes)",
                      rows, cols, tiles_x * tiles_y, kMaxTiles);
        return reject(SW2D_ERR_INVALID, buf);
    }
    /* The scratch array's device address belongs to the calling thread's
     * current context (one copy per device, and a fresh copy after
     * cudaDeviceReset or under another context), so it is looked up on every
     * call rather than cached.  The lookup allocates nothing; in a context
     * that has not used the library's device code yet it loads that code
     * first, which is this entry point's one-time set-up. */
    void* addr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&addr, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail("cudaGetSymbolAddress", e);
    double* scratch = static_cast<double*>(addr);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    /* the running maxima and the counter must be zero when the kernel starts */
    e = cudaMemsetAsync(scratch + kResult, 0, 3 * sizeof(double), s);
    if (e != cudaSuccess) return cuda_fail("cudaMemsetAsync", e);
    MeasureIn in;
    in.dem = d_dem;
    in.h = d_depth;
    in.qx = d_qx;
    in.qy = d_qy;
    in.R = rows;
    in.C = cols;
    in.nodata = nodata;
    in.th = th;
    in.g = g;
    in.rdx = 1.0 / dx;
    in.rdy = 1.0 / dy;
    in.area = dx * dy;
    const bool est = sw2d_est_range(th) && sw2d_est_range(g) && sw2d_est_range(dx) && sw2d_est_range(dy);
    in.thf = est ? (float)th : std::nanf("");
    in.est_most = est ? SW2D_EST_MOST : 0.f;
    in.gf = (float)g;
    in.rdxf = (float)in.rdx;
    in.rdyf = (float)in.rdy;
    /* fewer rows a task while the tasks would not reach every warp */
    const long long strips = (cols + 31LL) / 32;
    in.band = kBand;
    while (in.band > kBatch && strips * ((rows + in.band - 1) / in.band) < 8LL * kBlocks) in.band /= 2;
    const long long tasks = strips * ((rows + in.band - 1LL) / in.band);
    const int blocks = (int)std::min<long long>((tasks + 7) / 8, kBlocks);
    k64_measure_noalloc<<<blocks, 256, 0, s>>>(in, scratch);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail("k64_measure_noalloc launch", e);
    double res[2];
    e = cudaMemcpyAsync(res, scratch + kResult, sizeof res, cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) return cuda_fail("cudaMemcpyAsync", e);
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail("cudaStreamSynchronize", e);
    *volume_out = res[0];
    *speed_out = res[1];
    return SW2D_OK;
}
