/* Host engine of the FP32 precision form (see sw2d_engine.h). */
#include "sw2d_engine.h"
#include "sw2d_threads.h"

#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <limits>

namespace sw2d {

namespace {


PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        cudaDriverEntryPointQueryResult q;
        void* p = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

bool make_map(CUtensorMap* tm, void* base, CUtensorMapDataType dt, size_t esize, uint64_t width, uint64_t height,
              uint32_t boxw, uint32_t boxh, bool nan_fill) {
    auto fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {width, height};
    cuuint64_t strides[1] = {width * esize};
    cuuint32_t box[2] = {boxw, boxh};
    cuuint32_t es[2] = {1, 1};
    return fn(tm, dt, 2, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              nan_fill ? CU_TENSOR_MAP_FLOAT_OOB_FILL_NAN_REQUEST_ZERO_FMA : CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
           CUDA_SUCCESS;
}

int pitch_of(int cols) { return ((cols + 12 + 31) / 32) * 32; }

/* f(first, last) over [0, n) on host threads, one per `grain` elements of
 * work at most (a thread costs tens of microseconds to start) */
template <typename F>
void on_threads(size_t n, size_t work, size_t grain, F f) {
    split_over_threads(n, std::min<size_t>({16, std::thread::hardware_concurrency(), n, work / grain}), f);
}

/* device arrays of a scenario in one allocation, each 256-byte aligned */
struct Carver {
    size_t at = 0, bytes = 0; /* the end of the last one; the arrays' own bytes */
    size_t take(size_t n) {
        const size_t o = at;
        bytes += n;
        at = (at + std::max<size_t>(n, 16) + 255) & ~(size_t)255;
        return o;
    }
};
constexpr size_t kNone = ~(size_t)0;
constexpr size_t kPinInputs = (size_t)8 << 20; /* inputs up to here pay for pinned staging (larger ones use it if it is there) */

/* An error is returned once: the runtime's own record of it is cleared, which
 * the next call would report as its own (what broke the context stays). */
#define ECK(call)                                                                   \
    do {                                                                            \
        cudaError_t e_ = (call);                                                    \
        if (e_ != cudaSuccess) {                                                    \
            cudaGetLastError();                                                     \
            if (err) *err = std::string(#call) + ": " + cudaGetErrorString(e_);     \
            return e_ == cudaErrorMemoryAllocation ? SW2D_ERR_NOMEM : SW2D_ERR_CUDA; \
        }                                                                           \
    } while (0)

} // namespace

Engine32::Engine32(int device) : device_(device) {}

Engine32::~Engine32() {
    cudaSetDevice(device_);
    if (stream_) cudaStreamSynchronize(stream_);
    for (auto& s : scn_) cudaFree(s->slab);
    cudaFree(d_scn_);
    cudaFree(d_work_);
    cudaFree(d_part_);
    cudaFree(d_ctl_);
    cudaFree(d_tmp_);
    cudaFree(d_stat_);
    if (ev_a_) cudaEventDestroy(ev_a_);
    if (ev_b_) cudaEventDestroy(ev_b_);
    if (ev_t0_) cudaEventDestroy(ev_t0_);
    if (ev_t1_) cudaEventDestroy(ev_t1_);
    if (stream_) cudaStreamDestroy(stream_);
    if (pin_) cudaFreeHost(pin_);
}

int Engine32::init(std::string* err) {
    ECK(cudaSetDevice(device_));
    ECK(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    ECK(cudaEventCreate(&ev_a_));
    ECK(cudaEventCreate(&ev_b_));
    ECK(cudaMalloc(&d_tmp_, fp32_volume_scratch_bytes()));
    if (fp32_configure_kernels() != 0) {
        if (err) *err = "cannot enable the FP32 kernel's shared memory";
        return SW2D_ERR_CUDA;
    }
    /* rows per work item: SW2D_SEGMENT_ROWS fixes it (else the autotuner) */
    if (seg_fixed_ == 0) {
        if (const char* e = std::getenv("SW2D_SEGMENT_ROWS")) {
            const int v = std::atoi(e);
            if (v >= 16 && v <= M_MAXSEG) seg_ = seg_fixed_ = v;
        }
    }
    ECK(cudaEventCreate(&ev_t0_));
    ECK(cudaEventCreate(&ev_t1_));
    ECK(cudaDeviceGetAttribute(&nsm_, cudaDevAttrMultiProcessorCount, device_));
    for (int k = 0; k < T32_NCLASS; k++) {
        bps_[k] = fp32_blocks_per_sm(k);
        if (bps_[k] <= 0) {
            if (err) *err = "the FP32 kernel does not fit on an SM";
            return SW2D_ERR_CUDA;
        }
    }
    if (!encode_fn()) {
        if (err) *err = "cuTensorMapEncodeTiled unavailable";
        return SW2D_ERR_CUDA;
    }
    return SW2D_OK;
}

size_t Engine32::scenario_bytes(int rows, int cols, bool rain_field, int outlet_cap) {
    const size_t P = pitch_of(cols), NR = rows + 2 * M_H;
    const size_t cells = P * NR;
    size_t b = cells * (8 * sizeof(float) + 1); /* 8 float fields + optional Manning class byte */
    if (rain_field) b += cells * sizeof(float);
    const size_t tiles = (size_t)((cols + M_CW - 1) / M_CW) * ((rows + 15) / 16);
    b += tiles * sizeof(float) + (size_t)outlet_cap * 16 + sizeof(Clock32) + 4096;
    return b;
}

size_t Engine32::bytes_in_use() const {
    size_t b = 0;
    for (auto& s : scn_) b += s->bytes;
    return b;
}

int Engine32::add(const ScenarioInput& in, long long id, std::string* err, int* index_out) {
    ECK(cudaSetDevice(device_));
    if (in.rows < 2 || in.cols < 2 || !in.dem) {
        if (err) *err = "scenario needs rows, cols >= 2 and a DEM";
        return SW2D_ERR_INVALID;
    }
    if (in.mclass && (in.ntable <= 0 || in.ntable > T32_MAXCLASS || !in.mtable)) {
        if (err) *err = "Manning table must have 1..64 entries";
        return SW2D_ERR_INVALID;
    }
    auto sp = std::make_unique<Scenario32>();
    Scenario32& S = *sp;
    S.id = id;
    const int R = in.rows, C = in.cols, P = pitch_of(C), NR = R + 2 * M_H;
    S.R = R;
    S.C = C;
    S.P = P;
    S.NR = NR;
    const size_t cells = (size_t)P * NR;
    const int tx = (C + M_CW - 1) / M_CW, nb = (R + M_DR - 1) / M_DR; /* datum tiles: strips x bands */
    /* point sources (a later source on a cell replaces an earlier one, as the
     * reference's stream_flow writes them) */
    std::vector<int> src_keep;
    if (in.nsrc > 0) {
        if (in.nsrc > T32_MAXSRC || !in.src_cells || !in.src_q || in.nq <= 0 || !(in.dtoq > 0)) {
            if (err) *err = "point sources";
            return SW2D_ERR_INVALID;
        }
        for (int k = 0; k < in.nsrc; k++) {
            if (in.src_cells[k] < 0 || in.src_cells[k] >= R * C) {
                if (err) *err = "source cell out of range";
                return SW2D_ERR_INVALID;
            }
            bool later = false;
            for (int j = k + 1; j < in.nsrc; j++) later |= in.src_cells[j] == in.src_cells[k];
            if (!later) src_keep.push_back(k);
        }
    }
    const int nu = (int)src_keep.size(), nrain = std::max(in.nrain, 1);
    const bool has_evap = in.evap && in.nevap > 0;

    /* what the host fills (contiguous in the slab and in its staging copy),
     * then what starts as zeros */
    Carver cv;
    const size_t o_z = cv.take(cells * 4), o_h = cv.take(cells * 4);
    const size_t o_cls = in.mclass ? cv.take(cells) : kNone;
    const size_t o_rw = in.rain_weight ? cv.take(cells * 4) : kNone;
    const size_t o_datum = cv.take((size_t)tx * nb * 4);
    const size_t o_rain = cv.take((size_t)(nrain + 2) * 8);
    const size_t o_evap = has_evap ? cv.take((size_t)(in.nevap + 2) * 8) : kNone;
    const size_t o_srcc = nu > 0 ? cv.take((size_t)nu * 4) : kNone;
    const size_t o_srcq = nu > 0 ? cv.take((size_t)(in.nq + 2) * nu * 8) : kNone;
    const size_t o_clk = cv.take(sizeof(Clock32));
    const size_t staged = cv.at;
    const size_t o_h1 = cv.take(cells * 4);
    const size_t o_qx[2] = {cv.take(cells * 4), cv.take(cells * 4)}, o_qy[2] = {cv.take(cells * 4), cv.take(cells * 4)};
    const size_t o_kc = cv.take(cells * 4);
    const size_t o_out = in.outlet_cap > 0 ? cv.take((size_t)in.outlet_cap * 16) : kNone;

    char* slab = nullptr;
    {
        cudaError_t e = cudaMalloc((void**)&slab, cv.at);
        if (e != cudaSuccess) {
            cudaGetLastError();
            if (err) *err = std::string("cudaMalloc: ") + cudaGetErrorString(e);
            return SW2D_ERR_NOMEM;
        }
    }
    S.slab = slab;
    S.bytes = cv.bytes;
    auto fail_free = [&](int rc) {
        cudaStreamSynchronize(stream_);
        cudaFree(slab);
        return rc;
    };
    int rc;
#define ACK(call)                                                               \
    do {                                                                        \
        cudaError_t e_ = (call);                                                \
        if (e_ != cudaSuccess) {                                                \
            cudaGetLastError();                                                 \
            if (err) *err = std::string(#call) + ": " + cudaGetErrorString(e_); \
            return fail_free(SW2D_ERR_CUDA);                                    \
        }                                                                       \
    } while (0)
    ACK(cudaMemsetAsync(slab + staged, 0, cv.at - staged, stream_));
    Scn32& d = S.d;
    auto dev = [&](size_t o) -> void* { return o == kNone ? nullptr : slab + o; };
    d.h[0] = (float*)dev(o_h);
    d.h[1] = (float*)dev(o_h1);
    for (int k = 0; k < 2; k++) {
        d.qx[k] = (float*)dev(o_qx[k]);
        d.qy[k] = (float*)dev(o_qy[k]);
    }
    d.kc = (float*)dev(o_kc);
    float* const dz = (float*)dev(o_z);
    d.z = dz;
    uint8_t* const dcls = (uint8_t*)dev(o_cls);
    d.cls = dcls;
    d.datum = (float*)dev(o_datum);
    float* const drw = (float*)dev(o_rw);
    d.rainw = drw;
    d.rain = (double*)dev(o_rain);
    d.evap = (double*)dev(o_evap);
    d.srcq = (double*)dev(o_srcq);
    d.src_cell = (int*)dev(o_srcc);
    d.outlet = (double*)dev(o_out);
    d.clk = (Clock32*)dev(o_clk);

    /* host staging: per datum tile (a
     * strip of 224 columns x a band of 64 rows) the mean active elevation
     * rounded to 1/16 m, bed offsets from it with NaN for inactive cells */
    std::vector<char> pageable;
    char* stage;
    std::string refused;
    if (staged <= std::max(kPinInputs, pin_bytes_) && reserve_pin(staged, &refused) == SW2D_OK) {
        stage = static_cast<char*>(pin_);
    } else { /* large inputs, or no pinned memory to be had */
        pageable.resize(staged);
        stage = pageable.data();
    }
    float* const zoff = (float*)(stage + o_z);
    float* const hbuf = (float*)(stage + o_h);
    uint8_t* const cls = in.mclass ? (uint8_t*)(stage + o_cls) : nullptr;
    float* const rw = in.rain_weight ? (float*)(stage + o_rw) : nullptr;
    float* const datum = (float*)(stage + o_datum);
    const float nan = std::numeric_limits<float>::quiet_NaN();
    for (int r = 0; r < NR; r++) { /* the halo: inactive, dry, class 0, weight 1 */
        const bool in_rows = r >= M_H && r < M_H + R;
        const size_t row = (size_t)r * P;
        auto blank = [&](size_t a, size_t b) {
            std::fill(zoff + row + a, zoff + row + b, nan);
            std::fill(hbuf + row + a, hbuf + row + b, 0.f);
            if (cls) std::fill(cls + row + a, cls + row + b, (uint8_t)0);
            if (rw) std::fill(rw + row + a, rw + row + b, 1.f);
        };
        if (in_rows) {
            blank(0, M_H);
            blank((size_t)(M_H + C), (size_t)P);
        } else {
            blank(0, (size_t)P);
        }
    }
    std::vector<double> band_weight((size_t)nb, 0.0); /* active cells' rain weight, band by band */
    std::atomic<bool> bad_class(false);
    on_threads((size_t)nb, (size_t)R * C, (size_t)1 << 19, [&](size_t j0, size_t j1) {
        for (size_t j = j0; j < j1; j++) {
            const int ra = (int)j * M_DR, rb = std::min(R, ra + M_DR);
            double aw = 0.0;
            for (int i = 0; i < tx; i++) {
                const int ca = i * M_CW, cb = std::min(C, ca + M_CW);
                double sum = 0;
                long n = 0;
                for (int r = ra; r < rb; r++)
                    for (int c = ca; c < cb; c++) {
                        const double z = in.dem[(size_t)r * C + c];
                        if (z != in.nodata) {
                            sum += z;
                            n++;
                        }
                    }
                const float dt = n ? (float)(std::round(sum / n * 16.0) / 16.0) : 0.f;
                datum[j * tx + i] = dt;
                const double dat = dt;
                for (int r = ra; r < rb; r++) {
                    const size_t k = (size_t)r * C, g = (size_t)(r + M_H) * P + M_H;
                    for (int c = ca; c < cb; c++) {
                        const double z = in.dem[k + c];
                        const bool act = z != in.nodata;
                        zoff[g + c] = act ? (float)(z - dat) : nan;
                        hbuf[g + c] = act && in.depth ? (float)in.depth[k + c] : 0.f;
                        if (!rw && act) aw += 1.0;
                    }
                    if (cls)
                        for (int c = ca; c < cb; c++) {
                            const uint8_t cl = in.mclass[k + c];
                            if (cl >= in.ntable) bad_class = true;
                            cls[g + c] = cl;
                        }
                    if (rw)
                        for (int c = ca; c < cb; c++) {
                            rw[g + c] = in.rain_weight[k + c];
                            if (in.dem[k + c] != in.nodata) aw += (double)in.rain_weight[k + c];
                        }
                }
            }
            band_weight[j] = aw;
        }
    });
    if (bad_class) {
        if (err) *err = "Manning class out of table range";
        return fail_free(SW2D_ERR_INVALID);
    }
    double active_weight = 0.0;
    for (double w : band_weight) active_weight += w;
    auto series = [&](size_t o, const double* v, int n, size_t total) {
        double* t = (double*)(stage + o);
        std::fill(t, t + total, 0.0);
        for (int k = 0; k < n; k++) t[k] = v[k];
    };
    series(o_rain, in.rain, in.nrain, (size_t)nrain + 2);
    if (has_evap) series(o_evap, in.evap, in.nevap, (size_t)in.nevap + 2);
    if (nu > 0) {
        int* cellv = (int*)(stage + o_srcc);
        double* q = (double*)(stage + o_srcq);
        std::fill(q, q + (size_t)(in.nq + 2) * nu, 0.0);
        for (int u = 0; u < nu; u++) {
            cellv[u] = in.src_cells[src_keep[u]];
            for (int t = 0; t < in.nq; t++) q[(size_t)t * nu + u] = in.src_q[(size_t)t * in.nsrc + src_keep[u]];
        }
    }
    {
        Clock32 c{};
        c.t = in.t0;
        c.t_end = in.t_end;
        std::memcpy(stage + o_clk, &c, sizeof c);
    }
    ACK(cudaMemcpyAsync(slab, stage, staged, cudaMemcpyHostToDevice, stream_));

    /* tensor maps: rows of 232 columns, four rows per staged block; the bed
     * reads NaN (inactive) outside the array */
    bool ok = true;
    for (int k = 0; k < 2; k++) {
        ok &= make_map(&d.tm_h[k], d.h[k], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, P, NR, M_BW, M_RB, false);
        ok &= make_map(&d.tm_qx[k], d.qx[k], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, P, NR, M_BW, M_RB, false);
        ok &= make_map(&d.tm_qy[k], d.qy[k], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, P, NR, M_BW, M_RB, false);
    }
    ok &= make_map(&d.tm_z, dz, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, P, NR, M_BW, M_RB, true);
    ok &= make_map(&d.tm_kc, d.kc, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, P, NR, M_BW, M_RB, false);
    if (dcls) ok &= make_map(&d.tm_cls, dcls, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, P, NR, M_CLSW, M_CLSR, false);
    if (drw) ok &= make_map(&d.tm_rw, drw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, P, NR, M_BW, M_RWR, false);
    if (!ok) {
        if (err) *err = "cuTensorMapEncodeTiled failed";
        return fail_free(SW2D_ERR_CUDA);
    }
    d.R = R;
    d.C = C;
    d.P = P;
    d.tiles_x = tx;
    d.bands = nb;
    d.seg = 0;     /* work items: set by rebuild */
    d.tiles_y = 0;
    d.outflow_south = in.outflow_south;
    d.series_mode = in.series_mode;
    d.dt_mode = in.dt_mode;
    d.nrain = nrain;
    d.nevap = has_evap ? in.nevap : 0;
    d.nsrc = nu;
    d.nq = nu > 0 ? in.nq : 0;
    d.dtoq = nu > 0 ? in.dtoq : 3600.0;
    d.outlet_cap = in.outlet_cap;
    d.dx = (float)in.dx;
    d.dy = (float)in.dy;
    d.rdx = (float)(1.0 / in.dx);
    d.rdy = (float)(1.0 / in.dy);
    d.th = (float)in.th;
    d.g = (float)in.g;
    const double pct_lake = 1.00 - in.frac_lwl, pct_land = 1.00 - (in.frac_int + in.frac_inf);
    d.pct_lake = (float)pct_lake;
    d.pct_land = (float)pct_land;
    d.ev_wl_min = (float)in.ev_wl_min;
    d.ledger_cells = pct_lake != pct_land || has_evap; /* evaporation acts on lake cells only */
    d.rain_static = active_weight * pct_land;
    d.dxd = in.dx;
    d.dyd = in.dy;
    d.dtrain = in.dtrain;
    d.dt_fixed = in.dt;
    d.cfl = in.cfl;
    d.dt_max = in.dt_max;
    d.area = in.dx * in.dy;
    for (int k = 0; k < T32_MAXCLASS; k++)
        d.ntab[k] = (float)(in.mclass ? (k < in.ntable ? in.mtable[k] : 0.0) : in.manning);
    S.t_end_default = in.t_end;
    /* initial volume and CFL speed into the clock, then the first slot, from
     * the scenario's own descriptor (the work lists are built when it runs) */
    const size_t idx = scn_.size();
    if ((rc = reserve_scn(idx + 1, err))) return fail_free(rc);
    ACK(cudaMemcpyAsync(d_scn_ + idx, &d, sizeof d, cudaMemcpyHostToDevice, stream_));
    fp32_launch_volume(d_scn_, (int)idx, d, d_tmp_, true, stream_);
    fp32_launch_prime(d_scn_ + idx, 1, nullptr, stream_);
    ACK(cudaStreamSynchronize(stream_)); /* the staging copy is the next scenario's */
    ACK(cudaGetLastError());
#undef ACK
    scn_.push_back(std::move(sp));
    dirty_ = true;
    if (index_out) *index_out = (int)idx;
    return SW2D_OK;
}

int Engine32::reserve_pin(size_t bytes, std::string* err) {
    if (pin_bytes_ >= bytes) return SW2D_OK;
    if (pin_) cudaFreeHost(pin_);
    pin_ = nullptr;
    pin_bytes_ = 0;
    ECK(cudaMallocHost(&pin_, bytes));
    pin_bytes_ = bytes;
    return SW2D_OK;
}

/* room for n descriptors; those on the device are lost when it grows (the
 * next rebuild uploads them all) */
int Engine32::reserve_scn(size_t n, std::string* err) {
    if (n <= d_scn_cap_) return SW2D_OK;
    const size_t cap = std::max(n, 2 * d_scn_cap_);
    cudaFree(d_scn_);
    cudaFree(d_stat_);
    d_scn_ = nullptr;
    d_stat_ = nullptr;
    d_scn_cap_ = 0;
    dirty_ = true;
    ECK(cudaMalloc(&d_scn_, cap * sizeof(Scn32)));
    ECK(cudaMalloc(&d_stat_, cap * sizeof(Status32)));
    d_scn_cap_ = cap;
    return SW2D_OK;
}

int Engine32::remove(int index) {
    if (index < 0 || index >= (int)scn_.size()) return SW2D_ERR_INVALID;
    cudaSetDevice(device_);
    cudaStreamSynchronize(stream_);
    cudaFree(scn_[index]->slab);
    scn_.erase(scn_.begin() + index);
    dirty_ = true;
    return SW2D_OK;
}

/* Rows per work item of class k: at most seg_, fewer where that leaves the
 * GPU idle.  An iteration of a class is modelled by what the persistent
 * kernel measures on a GB300: a CTA marches a row in 0.70 us when it has its
 * SM to itself, 0.95, 1.19 or 1.49 us beside one, two or three others, over
 * the item's rows and their six halo rows in whole blocks of M_RB (what goes
 * by between iterations does not depend on the choice).  One scenario's items
 * run in whole waves over the CTAs; several scenarios fill one another's
 * gaps.  Measured, us an iteration, with items of 128, 64 and 16 rows and with
 * this rule's: 200 x 310 cells 101, 56, 24 and 13.7 (2 rows); 1000^2 103, 58,
 * 32 and 28.3 (18); 2048^2 124, 85, 88 and 66.2 (46); from about 12 M cells on,
 * items of seg_ rows fill the GPU and the halo rows decide. */
int Engine32::fill_rows(int k) const {
    static const double row_us[4] = {0.70, 0.95, 1.19, 1.49};
    const int per_sm = std::max(1, cps_ > 0 ? std::min(cps_, bps_[k]) : bps_[k]);
    const int slots = per_sm * nsm_;
    std::vector<const Scn32*> in;
    for (auto& s : scn_)
        if (fp32_feature_class(s->d) == k) in.push_back(&s->d);
    int best = seg_;
    double best_us = 0.0;
    for (int n = 0;; n++) { /* 2, 6, 10, ... rows and the halo make whole blocks; and seg_ itself */
        const int seg = std::min(seg_, 2 + M_RB * n);
        long long items = 0, rows = 0;
        int longest = 0;
        for (const Scn32* d : in) {
            const int r = std::min(seg, d->R), ni = d->tiles_x * ((d->R + r - 1) / r);
            const int marched = (r + 6 + M_RB - 1) / M_RB * M_RB;
            items += ni;
            rows += (long long)ni * marched;
            longest = std::max(longest, marched);
        }
        const long long busy = std::min<long long>(items, slots);
        const double us = row_us[std::min(3, (int)((busy + nsm_ - 1) / nsm_) - 1)];
        const double waves = in.size() == 1 ? (double)longest * (double)((items + slots - 1) / slots)
                                            : std::max((double)longest, (double)rows / (double)slots);
        const double t = waves * us;
        if (n == 0 || t <= best_us) {
            best = seg;
            best_us = t;
        }
        if (seg == seg_) break;
    }
    return best;
}

int Engine32::rebuild(std::string* err) {
    if (!dirty_) return SW2D_OK;
    work_.clear();
    std::vector<Scn32> host(scn_.size());
    /* work items grouped by feature class, scenarios in order within a class;
     * .w is the item's slot in the scenario-ordered partials */
    for (int k = 0; k < T32_NCLASS; k++) {
        class_first_[k] = (int)work_.size();
        bool any = false;
        for (auto& sp : scn_) any = any || fp32_feature_class(sp->d) == k;
        const int rows = !any || seg_fixed_ > 0 ? seg_ : fill_rows(k);
        for (size_t i = 0; i < scn_.size(); i++) {
            Scn32& d = scn_[i]->d;
            if (fp32_feature_class(d) != k) continue;
            d.seg = std::min(rows, d.R);
            d.tiles_y = (d.R + d.seg - 1) / d.seg;
            d.first_work = (int)work_.size();
            for (int ty = 0; ty < d.tiles_y; ty++)
                for (int tx = 0; tx < d.tiles_x; tx++)
                    work_.push_back(make_int4((int)i, tx, ty, (int)work_.size()));
            d.nwork = (int)work_.size() - d.first_work;
            host[i] = d;
        }
        class_n_[k] = (int)work_.size() - class_first_[k];
        /* the class's longest items first in every iteration (a scenario's
         * last segment is shorter), so the tail of an iteration holds short
         * items; the order is the same in every iteration, so a scenario's
         * items of the next iteration come after its own of this one */
        auto rows_of = [&](const int4& w) {
            const Scn32& d = scn_[w.x]->d;
            return std::min(d.seg, d.R - w.z * d.seg);
        };
        std::stable_sort(work_.begin() + class_first_[k], work_.end(),
                         [&](const int4& a, const int4& b) { return rows_of(a) > rows_of(b); });
    }
    int rc = reserve_scn(host.size(), err);
    if (rc) return rc;
    if (work_.size() > d_work_cap_) {
        cudaFree(d_work_);
        cudaFree(d_part_);
        d_work_ = nullptr;
        d_part_ = nullptr;
        d_work_cap_ = std::max<size_t>(work_.size(), 2 * d_work_cap_);
        ECK(cudaMalloc(&d_work_, d_work_cap_ * sizeof(int4)));
        ECK(cudaMalloc(&d_part_, d_work_cap_ * sizeof(Part32)));
    }
    if (fp32_ctl_bytes((int)scn_.size()) > d_ctl_cap_) {
        cudaFree(d_ctl_);
        d_ctl_ = nullptr;
        d_ctl_cap_ = std::max(fp32_ctl_bytes((int)scn_.size()), 2 * d_ctl_cap_);
        ECK(cudaMalloc(&d_ctl_, d_ctl_cap_));
    }
    if (!host.empty())
        ECK(cudaMemcpyAsync(d_scn_, host.data(), host.size() * sizeof(Scn32), cudaMemcpyHostToDevice, stream_));
    if (!work_.empty())
        ECK(cudaMemcpyAsync(d_work_, work_.data(), work_.size() * sizeof(int4), cudaMemcpyHostToDevice, stream_));
    ECK(cudaStreamSynchronize(stream_));
    dirty_ = false;
    return SW2D_OK;
}

/* CTAs of class k's persistent launch: the CTAs per SM in use (at most what
 * the SM holds) on every SM, at most one per work item -- no more items than
 * that can run at a time, and CTAs that hold later iterations' tickets poll
 * the counters that the running ones release */
int Engine32::grid_of(int k) const {
    const int per_sm = cps_ > 0 ? std::min(cps_, bps_[k]) : bps_[k];
    return std::max(1, std::min(per_sm * nsm_, class_n_[k]));
}

/* niter iterations: one persistent launch per feature class present */
int Engine32::launch(int niter, std::string* err) {
    int grid[T32_NCLASS];
    for (int k = 0; k < T32_NCLASS; k++) grid[k] = grid_of(k);
    ECK(fp32_launch_chunk(d_scn_, (int)scn_.size(), d_work_, class_first_, class_n_, d_part_, d_ctl_, niter, grid,
                          stream_));
    return SW2D_OK;
}

int Engine32::tune(long long budget, std::string* err, long long* advanced) {
    *advanced = 0;
    double cells = 0;
    for (auto& sp : scn_) cells += (double)sp->R * sp->C;
    if (seg_fixed_ > 0 || cells < (1 << 20)) return SW2D_OK;
    const int bucket = (int)std::floor(std::log2(cells));
    if (bucket == bucket_) return SW2D_OK;
    int rc;
    auto use = [&](int seg, int cps) {
        if (seg != seg_ || cps != cps_) {
            seg_ = seg;
            cps_ = cps;
            dirty_ = true; /* new work items */
            return rebuild(err);
        }
        return (int)SW2D_OK;
    };
    const auto cached = tuned_.find(bucket);
    if (cached != tuned_.end()) {
        if ((rc = use(cached->second.first, cached->second.second))) return rc;
        bucket_ = bucket;
        return SW2D_OK;
    }
    int most = 0;
    for (int k = 0; k < T32_NCLASS; k++)
        if (class_n_[k] > 0) most = std::max(most, bps_[k]);
    std::vector<std::pair<int, int>> cands;
    for (int seg : {64, 128, 256, 512}) {
        cands.emplace_back(seg, 0);
        if (most > 1) cands.emplace_back(seg, most - 1);
    }
    /* iterations per candidate: one untimed (the new work split's first
     * launch), then one timed launch of up to a chunk */
    const long long per = std::min<long long>(kChunk + 1, budget / (long long)cands.size());
    if (per < 3) return SW2D_OK; /* too few iterations to tune now: a later, longer call will */
    const auto t0 = std::chrono::steady_clock::now();
    std::pair<int, int> best(seg_, cps_);
    float best_ms = 3.4e38f;
    for (const auto& cand : cands) {
        if ((rc = use(cand.first, cand.second))) return rc;
        if ((rc = launch(1, err))) return rc;
        ECK(cudaEventRecord(ev_t0_, stream_));
        if ((rc = launch((int)(per - 1), err))) return rc;
        ECK(cudaEventRecord(ev_t1_, stream_));
        ECK(cudaEventSynchronize(ev_t1_));
        float ms = 0;
        ECK(cudaEventElapsedTime(&ms, ev_t0_, ev_t1_));
        *advanced += per;
        if (ms < best_ms) {
            best_ms = ms;
            best = cand;
        }
    }
    if ((rc = use(best.first, best.second))) return rc;
    tuned_[bucket] = best;
    bucket_ = bucket;
    tuning_ms_ += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    tunings_++;
    return SW2D_OK;
}

int Engine32::tune_now(long long budget, std::string* err, long long* advanced) {
    ECK(cudaSetDevice(device_));
    *advanced = 0;
    int rc = rebuild(err);
    if (rc) return rc;
    if (scn_.empty() || budget <= 0) return SW2D_OK;
    return tune(budget, err, advanced);
}

int Engine32::set_t_end(int index, double t_end, std::string* err) {
    ECK(cudaSetDevice(device_));
    int rc = rebuild(err);
    if (rc) return rc;
    if (index >= 0)
        fp32_launch_prime(d_scn_ + index, 1, &t_end, stream_);
    else if (!scn_.empty())
        fp32_launch_prime(d_scn_, (int)scn_.size(), &t_end, stream_);
    ECK(cudaGetLastError());
    return SW2D_OK;
}

int Engine32::run(long long n, std::string* err) {
    ECK(cudaSetDevice(device_));
    int rc = rebuild(err);
    if (rc) return rc;
    if (scn_.empty() || n <= 0) return SW2D_OK;
    ECK(cudaEventRecord(ev_a_, stream_));
    long long done = 0;
    if ((rc = tune(n, err, &done))) return rc;
    for (; n - done >= kChunk; done += kChunk)
        if ((rc = launch(kChunk, err))) return rc;
    if (n > done && (rc = launch((int)(n - done), err))) return rc;
    ECK(cudaGetLastError());
    ECK(cudaEventRecord(ev_b_, stream_));
    ECK(cudaEventSynchronize(ev_b_));
    float ms = 0;
    ECK(cudaEventElapsedTime(&ms, ev_a_, ev_b_));
    last_ms_ = ms;
    last_iters_ = n;
    return SW2D_OK;
}

int Engine32::sync(std::string* err) {
    ECK(cudaStreamSynchronize(stream_));
    return SW2D_OK;
}

int Engine32::get_clock(int index, Clock32* out, std::string* err) {
    ECK(cudaMemcpyAsync(out, scn_[index]->d.clk, sizeof(Clock32), cudaMemcpyDeviceToHost, stream_));
    ECK(cudaStreamSynchronize(stream_));
    return SW2D_OK;
}

int Engine32::get_status(std::vector<Status32>* out, std::string* err) {
    out->resize(scn_.size());
    if (scn_.empty()) return SW2D_OK;
    int rc = rebuild(err);
    if (rc) return rc;
    fp32_launch_status(d_scn_, (int)scn_.size(), d_stat_, stream_);
    ECK(cudaMemcpyAsync(out->data(), d_stat_, scn_.size() * sizeof(Status32), cudaMemcpyDeviceToHost, stream_));
    ECK(cudaStreamSynchronize(stream_));
    return SW2D_OK;
}

int Engine32::get_state(int index, double* depth, double* qx, double* qy, std::string* err) {
    Scenario32& S = *scn_[index];
    Clock32 c;
    int rc = get_clock(index, &c, err);
    if (rc) return rc;
    const int cur = c.slot.cur;
    const int R = S.R, C = S.C, P = S.P;
    struct Field {
        const float* src;
        int rows, cols;
        double* dst;
    } f[3] = {{S.d.h[cur], R, C, depth}, {S.d.qx[cur], R + 1, C, qx}, {S.d.qy[cur], R, C + 1, qy}};
    /* whole padded rows into pinned staging (a copy into pageable memory runs
     * at a few GB/s), all fields of a small raster at once, then the interior
     * widened to binary64 on host threads */
    const size_t one = (size_t)(R + 1) * P * sizeof(float);
    const bool together = 3 * one <= ((size_t)16 << 20);
    if ((rc = reserve_pin(together ? 3 * one : one, err))) return rc;
    auto fetch = [&](const Field& x, char* to) {
        return cudaMemcpyAsync(to, x.src + (size_t)M_H * P, (size_t)x.rows * P * sizeof(float), cudaMemcpyDeviceToHost,
                               stream_);
    };
    auto widen = [&](const Field& x, const char* from) {
        const float* s = reinterpret_cast<const float*>(from) + M_H;
        on_threads((size_t)x.rows, (size_t)x.rows * x.cols, (size_t)1 << 18, [=](size_t a, size_t b) {
            for (size_t r = a; r < b; r++)
                for (int k = 0; k < x.cols; k++) x.dst[r * x.cols + k] = s[r * P + k];
        });
    };
    char* const base = static_cast<char*>(pin_);
    for (int k = 0; k < 3; k++) {
        if (!f[k].dst) continue;
        ECK(fetch(f[k], together ? base + k * one : base));
        if (together) continue;
        ECK(cudaStreamSynchronize(stream_));
        widen(f[k], base);
    }
    if (together) {
        ECK(cudaStreamSynchronize(stream_));
        for (int k = 0; k < 3; k++)
            if (f[k].dst) widen(f[k], base + k * one);
    }
    return SW2D_OK;
}

size_t Engine32::snapshot_bytes(int index) const {
    const Scenario32& S = *scn_[index];
    return sizeof(Clock32) + 4 * (size_t)S.P * S.NR * sizeof(float);
}

int Engine32::snapshot(int index, void* buf, std::string* err) {
    Scenario32& S = *scn_[index];
    Clock32 c;
    int rc = get_clock(index, &c, err);
    if (rc) return rc;
    char* p = static_cast<char*>(buf);
    std::memcpy(p, &c, sizeof c);
    p += sizeof c;
    const size_t n = (size_t)S.P * S.NR * sizeof(float);
    const float* src[4] = {S.d.h[c.slot.cur], S.d.qx[c.slot.cur], S.d.qy[c.slot.cur], S.d.kc};
    for (int k = 0; k < 4; k++) {
        ECK(cudaMemcpyAsync(p, src[k], n, cudaMemcpyDeviceToHost, stream_));
        p += n;
    }
    ECK(cudaStreamSynchronize(stream_));
    return SW2D_OK;
}

int Engine32::restore(int index, const void* buf, std::string* err) {
    Scenario32& S = *scn_[index];
    const char* p = static_cast<const char*>(buf);
    Clock32 c;
    std::memcpy(&c, p, sizeof c);
    p += sizeof c;
    if (c.slot.cur != 0 && c.slot.cur != 1) {
        if (err) *err = "snapshot clock is not valid";
        return SW2D_ERR_INVALID;
    }
    const size_t n = (size_t)S.P * S.NR * sizeof(float);
    float* dst[4] = {S.d.h[c.slot.cur], S.d.qx[c.slot.cur], S.d.qy[c.slot.cur], S.d.kc};
    for (int k = 0; k < 4; k++) {
        ECK(cudaMemcpyAsync(dst[k], p, n, cudaMemcpyHostToDevice, stream_));
        p += n;
    }
    ECK(cudaMemcpyAsync(S.d.clk, &c, sizeof c, cudaMemcpyHostToDevice, stream_));
    ECK(cudaStreamSynchronize(stream_));
    return SW2D_OK;
}

int Engine32::get_volume(int index, double* vol, double* smax, std::string* err) {
    int rc = rebuild(err);
    if (rc) return rc;
    fp32_launch_volume(d_scn_, index, scn_[index]->d, d_tmp_, false, stream_);
    double vs[2];
    ECK(cudaMemcpyAsync(vs, d_tmp_, 2 * sizeof(double), cudaMemcpyDeviceToHost, stream_));
    ECK(cudaStreamSynchronize(stream_));
    if (vol) *vol = vs[0];
    if (smax) *smax = vs[1];
    return SW2D_OK;
}

int Engine32::get_outlet(int index, double* t, double* q, int cap, int* count, std::string* err) {
    Scenario32& S = *scn_[index];
    Clock32 c;
    int rc = get_clock(index, &c, err);
    if (rc) return rc;
    const int oc = S.d.outlet_cap;
    long long n = std::min<long long>(c.outlet_n, oc);
    if (count) *count = (int)n;
    if (!n || (!t && !q)) return SW2D_OK;
    std::vector<double> buf((size_t)oc * 2);
    ECK(cudaMemcpyAsync(buf.data(), S.d.outlet, buf.size() * 8, cudaMemcpyDeviceToHost, stream_));
    ECK(cudaStreamSynchronize(stream_));
    long long first = c.outlet_n > oc ? c.outlet_n % oc : 0;
    for (long long k = 0; k < n && k < cap; k++) {
        long long j = (first + k) % oc;
        if (t) t[k] = buf[2 * j];
        if (q) q[k] = buf[2 * j + 1];
    }
    return SW2D_OK;
}

} // namespace sw2d
