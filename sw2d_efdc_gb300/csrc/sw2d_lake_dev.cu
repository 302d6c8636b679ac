/* The DEM pre-pass of a coupled run (lake_catchment_smooth,
 * SW2D-EFDC.cu:2766-2827) as a device pass on caller-owned device arrays.
 *
 * The reference sweeps the raster row by row from the last (south) row to
 * the first, each row west to east, updating in place: a catchment cell on
 * the lake edge takes the mean of its two neighbours across the edge, and
 * reads the cells south and west of it after their own update.  Only cells
 * on the mask edge change, and only edge cells south or west of one that are
 * edge cells themselves make it wait: k_lake_list appends the edge cells to a
 * list, and one CTA (k_lake_solve) keeps them in shared memory, finds each
 * one's south and west entries through a hash table and updates in rounds
 * every cell whose entries are done
 * -- as many rounds as the longest chain of edge cells, a few dozen on a
 * lake's shore, where a sweep over the anti-diagonals takes one barrier and
 * four dependent reads for each of them.  Lists longer than the table
 * (kListMax) take that sweep: numbering the anti-diagonals d = (rows-1-r) + c,
 * a cell's south and west neighbours lie on d-1 and its north and east
 * neighbours on d+1, so the cells of one diagonal are independent; the edge
 * cells are listed per diagonal (count, scan, fill), then one CTA walks the
 * diagonals in order with a barrier between non-empty ones.  Every update is
 * the reference's (a + b) / 2.0 on the same operands, so the result is
 * bit-identical to the sequential sweep.
 * Compiled with --fmad=false.
 */
#include "sw2d.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>

namespace sw2d {
void set_error_message(const char* msg); /* sw2d_api.cu */
}

namespace {

constexpr double kRefNodata = -9999.0; /* the literal the reference compares against */

__device__ __forceinline__ bool lake_edge(const int* __restrict__ m, int R, int C, int r, int c) {
    if (r < 1 || r > R - 2 || c < 1 || c > C - 2) return false;
    const size_t k = (size_t)r * C + c;
    const int v = m[k];
    return v != 1 && (v != m[k - C] || v != m[k + C] || v != m[k - 1] || v != m[k + 1]);
}

__global__ void k_lake_count(const int* __restrict__ m, int R, int C, int* __restrict__ cnt) {
    const long long n = (long long)R * C;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(k / C), c = (int)(k - (long long)r * C);
        if (lake_edge(m, R, C, r, c)) atomicAdd(&cnt[(R - 1 - r) + c], 1);
    }
}

/* exclusive scan of n counts in place (one block of 1024 threads); cnt[n]
 * receives the total */
__global__ void __launch_bounds__(1024) k_lake_scan(int* cnt, int n) {
    __shared__ int part[1024];
    const int t = threadIdx.x;
    const int per = (n + 1023) / 1024, a = min(n, t * per), b = min(n, a + per);
    int s = 0;
    for (int k = a; k < b; k++) s += cnt[k];
    part[t] = s;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) { /* inclusive scan of the chunk sums */
        const int v = t >= o ? part[t - o] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    int run = t ? part[t - 1] : 0;
    for (int k = a; k < b; k++) {
        const int v = cnt[k];
        cnt[k] = run;
        run += v;
    }
    if (t == 1023) cnt[n] = part[1023];
}

__global__ void k_lake_fill(const int* __restrict__ m, int R, int C, const int* __restrict__ start,
                            int* __restrict__ fill, int* __restrict__ list) {
    const long long n = (long long)R * C;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(k / C), c = (int)(k - (long long)r * C);
        if (!lake_edge(m, R, C, r, c)) continue;
        const int d = (R - 1 - r) + c;
        list[start[d] + atomicAdd(&fill[d], 1)] = (int)k;
    }
}

/* the wavefront: one CTA, diagonals in order; within a diagonal the cells
 * are independent (the order of the list does not matter) */
__global__ void __launch_bounds__(1024) k_lake_sweep(const int* __restrict__ m, int C, const int* __restrict__ start,
                                                     const int* __restrict__ list, int nd, double* z) {
    for (int d = 0; d < nd; d++) {
        const int a = start[d], b = start[d + 1];
        if (a == b) continue;
        for (int j = a + threadIdx.x; j < b; j += blockDim.x) {
            const size_t k = (size_t)list[j];
            const int v = m[k];
            /* across the edge with the row above, then below, then the
             * columns west and east: each test may overwrite the last
             * (SW2D-EFDC.cu:2790-2816) */
            if (v != m[k - C] && z[k + C] != kRefNodata) z[k] = (z[k - C] + z[k + C]) / 2.0;
            if (v != m[k + C] && z[k - C] != kRefNodata) z[k] = (z[k - C] + z[k + C]) / 2.0;
            if (v != m[k - 1] && z[k + 1] != kRefNodata) z[k] = (z[k - 1] + z[k + 1]) / 2.0;
            if (v != m[k + 1] && z[k - 1] != kRefNodata) z[k] = (z[k - 1] + z[k + 1]) / 2.0;
        }
        __syncthreads(); /* the diagonal's updates are read by the next one */
    }
}

constexpr int kListMax = 9216;  /* entries k_lake_solve holds */
constexpr int kHash = 32768;    /* slots of its table */
constexpr int kSolveThreads = 1024;
constexpr int kPer = kListMax / kSolveThreads;

/* The lists of the calls in flight: a list's length, then the cells.  A call
 * takes a free one for as long as it runs (it synchronises its stream before
 * it returns), so calls of several threads, streams and devices run side by
 * side; one that finds none free allocates its own.  The array is per device
 * and context; a number is taken in all of them at once. */
constexpr int kLists = 8;
__device__ int g_lake_list[kLists][1 + kListMax];
std::atomic<unsigned> lists_taken{0u};

class ListOfCall {
  public:
    ~ListOfCall() {
        if (number_ >= 0) lists_taken.fetch_and(~(1u << number_));
        if (own_) cudaFree(own_);
    }
    /* the call's list on the current device */
    cudaError_t take(int** list) {
        unsigned t = lists_taken.load();
        while (t != (1u << kLists) - 1u) {
            const unsigned free_bit = ~t & (t + 1u);
            if (!lists_taken.compare_exchange_weak(t, t | free_bit)) continue;
            while (free_bit >> ++number_ != 1u) {}
            void* base = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&base, g_lake_list);
            *list = static_cast<int*>(base) + (size_t)number_ * (1 + kListMax);
            return e;
        }
        const cudaError_t e = cudaMalloc(&own_, sizeof(int) * (1 + kListMax));
        *list = own_;
        return e;
    }

  private:
    int number_ = -1;
    int* own_ = nullptr;
};

/* edge cells in any order; count[0] their number, also past the list's end */
__global__ void k_lake_list(const int* __restrict__ m, int R, int C, int* __restrict__ count, int* __restrict__ list) {
    const long long n = (long long)R * C;
    const int lane = threadIdx.x & 31;
    for (long long k0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) - lane; k0 < n;
         k0 += (long long)gridDim.x * blockDim.x) {
        const long long k = k0 + lane;
        bool e = false;
        if (k < n) {
            const int r = (int)(k / C), c = (int)(k - (long long)r * C);
            e = lake_edge(m, R, C, r, c);
        }
        const unsigned b = __ballot_sync(0xffffffffu, e);
        if (!b) continue;
        int at = 0;
        if (lane == 0) at = atomicAdd(count, __popc(b));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(b & ((1u << lane) - 1u));
        if (e && at < kListMax) list[at] = (int)k;
    }
}

struct LakeSolve {
    double val[kListMax];     /* the cell's updated value */
    int key[kListMax];
    short dw[kListMax], ds[kListMax]; /* entries of the west and south neighbours, -1 none */
    unsigned char mode[kListMax];     /* how the cell is updated, below; kDone set when it is */
    unsigned short slot[kHash];       /* entry + 1, 0 free */
};
enum { kNone = 0, kH = 1, kHif = 2, kV = 3, kVif = 4, kDone = 128 };

__device__ __forceinline__ unsigned lake_hash(int k) { return ((unsigned)k * 2654435761u) >> 17; }

__device__ __forceinline__ int lake_find(const LakeSolve& S, int k) {
    for (unsigned h = lake_hash(k);; h = (h + 1) & (kHash - 1)) { /* at most kListMax of the slots are taken */
        const int e = S.slot[h];
        if (e == 0) return -1;
        if (S.key[e - 1] == k) return e - 1;
    }
}

/* The update of a cell (SW2D-EFDC.cu:2790-2816) is the mean across the
 * columns if the mask changes to the west and the east neighbour has data, or
 * to the east and the west one (already updated) has; else the mean across
 * the rows by the same rule with south and north for west and east; else
 * none.  kH / kV: decided at once; kHif / kVif: if the updated neighbour has
 * data. */
__global__ void __launch_bounds__(kSolveThreads) k_lake_solve(const int* __restrict__ m, int C, const int* __restrict__ count,
                                                             const int* __restrict__ list, double* z) {
    extern __shared__ __align__(16) unsigned char raw[];
    LakeSolve& S = *reinterpret_cast<LakeSolve*>(raw);
    const int t = threadIdx.x, n = *count;
    if (n > kListMax) return; /* the caller's sweep */
    for (int k = t; k < kHash; k += kSolveThreads) S.slot[k] = 0;
    for (int e = t; e < n; e += kSolveThreads) S.key[e] = list[e];
    __syncthreads();
    for (int e = t; e < n; e += kSolveThreads) {
        for (unsigned h = lake_hash(S.key[e]);; h = (h + 1) & (kHash - 1))
            if (atomicCAS(&S.slot[h], (unsigned short)0, (unsigned short)(e + 1)) == 0) break;
    }
    __syncthreads();
    unsigned open = 0u; /* the thread's entries that are not done */
    for (int q = 0; q < kPer; q++) {
        const int e = t + q * kSolveThreads;
        if (e >= n) break;
        const int k = S.key[e], v = m[k];
        const bool cn = v != m[k - C], cs = v != m[k + C], cw = v != m[k - 1], ce = v != m[k + 1];
        const double zn = z[k - C], zs = z[k + C], zw = z[k - 1], ze = z[k + 1];
        const int w = lake_find(S, k - 1), s = lake_find(S, k + C);
        int mode = kNone;
        if (cw && ze != kRefNodata) mode = kH;
        else if (ce && (w >= 0 || zw != kRefNodata)) mode = w >= 0 ? kHif : kH;
        else if (cs && zn != kRefNodata) mode = kV;
        else if (cn && (s >= 0 || zs != kRefNodata)) mode = s >= 0 ? kVif : kV;
        const bool h = mode == kH || mode == kHif;
        /* kHif may still fall back on the rows: it waits for both */
        S.dw[e] = (short)(h ? w : -1);
        S.ds[e] = (short)(mode == kV || mode == kVif || mode == kHif ? s : -1);
        S.val[e] = z[k];
        S.mode[e] = (unsigned char)mode;
        open |= 1u << q;
    }
    __syncthreads();
    volatile unsigned char* mode = S.mode;
    volatile double* val = S.val;
    /* every round finishes at least the first open cell of the sweep's order */
    for (int round = 0; round <= n; round++) {
        for (int q = 0; q < kPer; q++) {
            if (!(open >> q & 1u)) continue;
            const int e = t + q * kSolveThreads, w = S.dw[e], s = S.ds[e], md = mode[e];
            if ((w >= 0 && !(mode[w] & kDone)) || (s >= 0 && !(mode[s] & kDone))) continue;
            __threadfence_block(); /* their values after their marks */
            const int k = S.key[e];
            const bool h = md == kH || md == kHif;
            const double x = h ? z[k + 1] : z[k - C]; /* the neighbour that is updated later, if at all */
            const double y = h ? (w >= 0 ? val[w] : z[k - 1]) : (s >= 0 ? val[s] : z[k + C]);
            if (md == kH || md == kV || ((md == kHif || md == kVif) && y != kRefNodata)) {
                val[e] = (x + y) / 2.0;
            } else if (md == kHif) { /* the west neighbour lost its data: the rows' rule */
                const int v = m[k];
                const double zn = z[k - C], zs = s >= 0 ? val[s] : z[k + C];
                if ((v != m[k + C] && zn != kRefNodata) || (v != m[k - C] && zs != kRefNodata)) val[e] = (zn + zs) / 2.0;
            }
            __threadfence_block();
            mode[e] = (unsigned char)(md | kDone);
            open &= ~(1u << q);
        }
        if (!__syncthreads_or((int)open)) break;
    }
    for (int e = t; e < n; e += kSolveThreads) z[S.key[e]] = S.val[e];
}

int fail(int code, const char* what, cudaError_t e = cudaSuccess) {
    char buf[256];
    if (e != cudaSuccess)
        std::snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
    else
        std::snprintf(buf, sizeof buf, "%s", what);
    sw2d::set_error_message(buf);
    return code;
}

} // namespace

extern "C" int sw2d_lake_catchment_smooth_device(int rows, int cols, const int* d_mask, double* d_dem,
                                                 void* stream) {
    if (!d_mask || !d_dem) return fail(SW2D_ERR_INVALID, "null argument");
    if (rows < 1 || cols < 1) return fail(SW2D_ERR_INVALID, "rows and cols must be >= 1");
    if ((long long)rows * cols > (1LL << 30)) return fail(SW2D_ERR_INVALID, "rows * cols above 2^30 cells");
    if (rows < 3 || cols < 3) return SW2D_OK; /* no interior cell: nothing changes */
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const long long n = (long long)rows * cols;
    const int grid = (int)std::min<long long>((n + 255) / 256, 152 * 16);
    int total = 0;
    {
        ListOfCall mine;
        int* d_list = nullptr;
        cudaError_t e = mine.take(&d_list);
        if (e == cudaErrorMemoryAllocation) return fail(SW2D_ERR_NOMEM, "cudaMalloc", e);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_lake_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LakeSolve));
        if (e == cudaSuccess) e = cudaMemsetAsync(d_list, 0, sizeof(int), s);
        if (e == cudaSuccess) {
            k_lake_list<<<grid, 256, 0, s>>>(d_mask, rows, cols, d_list, d_list + 1);
            k_lake_solve<<<1, kSolveThreads, sizeof(LakeSolve), s>>>(d_mask, cols, d_list, d_list + 1, d_dem);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(&total, d_list, sizeof(int), cudaMemcpyDeviceToHost, s);
        const cudaError_t es = cudaStreamSynchronize(s); /* also after an error: another call may take the list next */
        if (e == cudaSuccess) e = es;
        if (e != cudaSuccess) return fail(SW2D_ERR_CUDA, "lake-edge device pass", e);
        if (total <= kListMax) return SW2D_OK;
    }
    /* more edge cells than the table holds: the sweep over the diagonals */
    const int nd = rows + cols - 1;
    int* d_cnt = nullptr;
    int* d_list = nullptr;
    cudaError_t e = cudaMalloc(&d_cnt, sizeof(int) * (size_t)(2 * nd + 2));
    if (e != cudaSuccess) return fail(SW2D_ERR_NOMEM, "cudaMalloc", e);
    int* d_fill = d_cnt + nd + 1;
    e = cudaMalloc(&d_list, sizeof(int) * (size_t)total);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_cnt, 0, sizeof(int) * (size_t)(2 * nd + 2), s);
    if (e == cudaSuccess) {
        k_lake_count<<<grid, 256, 0, s>>>(d_mask, rows, cols, d_cnt);
        k_lake_scan<<<1, 1024, 0, s>>>(d_cnt, nd);
        k_lake_fill<<<grid, 256, 0, s>>>(d_mask, rows, cols, d_cnt, d_fill, d_list);
        k_lake_sweep<<<1, 1024, 0, s>>>(d_mask, cols, d_cnt, d_list, nd, d_dem);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(d_list);
    cudaFree(d_cnt);
    if (e != cudaSuccess) return fail(SW2D_ERR_CUDA, "lake-edge device pass", e);
    return SW2D_OK;
}
