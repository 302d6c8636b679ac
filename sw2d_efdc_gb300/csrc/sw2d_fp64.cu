/* FP64 SW2D step on sm_103a: the plain path whose results match the
 * reference's own kernels (SW2D-EFDC.cu:97-725).
 *
 * GB300's FP64 pipe runs at ~1/64 of the FP32 rate, so this path is bound by
 * FP64 instructions, not HBM: one takes a warp 71 issue cycles of its SM
 * quarter whether one lane or 32 take part.  The step is therefore split so
 * that nothing FP64 is computed twice and what is computed runs on full
 * warps, in two kernels per iteration:
 *   k64_flux   : new x/y face discharges of every face (flux, :97-353) from the
 *                stored face velocities uu1/vv1 of the previous iteration
 *                (momentum faces, weir and dry-bed faces and edge terms each
 *                packed into a list per block), and the CFL face-speed
 *                maxima of the entering state
 *   k64_update : per tile, "active and h* < th" flags of the provisional depth
 *                (continuity at t, :602-664) in shared memory, decided in
 *                binary32 wherever its error allows;
 *                treat_error (:695-725, restated per face) and the final
 *                depth at t+dt; the closed faces written back and the face
 *                velocities uu1 = qx/hm, vv1 = qy/hn of the new state
 *                (hm_hn, uu1_vv1, :362-452); partials of the ledger sums.  One
 *                extra block adds up the previous iteration's partials in a
 *                fixed order and prepares the next iteration's length and
 *                forcing beside the tiles.
 * At 4096 x 4096 (pond break) an iteration takes 1.24 ms early in the run
 * (timed apart: flux 0.82, update 0.44) and 1.32 ms at t = 600 s (0.89, 0.44),
 * against 5.17 ms with part-empty warps, a binary64 provisional depth and conversions and
 * sums predicated off beside the path taken; at 256 x 256 18.5 us against 62
 * us, most of it the clock's work at the end of the last tile's block before.
 * forward (:670-693) is a buffer swap for the depth (h[cur] -> h[nxt]); the
 * discharges keep fixed roles: qx[0]/qy[0] hold the state, k64_flux writes
 * its new faces into qx[1]/qy[1], and k64_update writes every face, closed
 * or not, back into qx[0]/qy[0] -- so no tile reads a face another tile has
 * already closed (the provisional depth needs them unclosed).
 * Compiled with --fmad=false: every expression is evaluated with the same
 * roundings as the CPU oracle (gcc -ffp-contract=off), explicit fma() only
 * where sw2d_math.h spells it.
 */
#include "sw2d_internal.h"
#include "sw2d_math.h"

#include <algorithm>
#include <climits>

namespace sw2d {

#define H SW2D_HALO

/* the entry in force at `time`: sw2d_series_index with the division on the integer pipes */
__device__ __forceinline__ int series_index(double time, double dts, int n) {
    return sw2d_series_entry(sw2d_div_rn(time, dts), n);
}

__device__ __forceinline__ double series_at(const double* v, int n, double dts, double time, int mode) {
    if (mode == 0 && time <= 1.00) return v[0] * time; /* SW2D-EFDC.cu:546-551 */
    const int it = series_index(time, dts, n);
    const double a = v[it];
    if (mode == 2) return a;
    const double b = v[it + 1], d = time - dts * (it);
    return mode == 0 ? a + sw2d_div_rn(b - a, dts * d) : a + (b - a) * sw2d_div_rn(d, dts);
}

__device__ __forceinline__ double source_at(const StepParams& p, int i, double time) {
    double q;
    const double* Q = p.srcq;
    const int ns = p.nsrc;
    if (p.series_mode == 0 && time <= 1.00) { /* stream_flow SW2D-EFDC.cu:531-538 */
        q = Q[i] * time;
    } else {
        const int it = series_index(time, p.dtoq, p.nq);
        const double a = Q[(size_t)it * ns + i];
        q = a;
        if (p.series_mode != 2) {
            const double b = Q[(size_t)(it + 1) * ns + i], d = time - p.dtoq * (it);
            q = p.series_mode == 0 ? a + sw2d_div_rn(b - a, p.dtoq * d) : a + (b - a) * sw2d_div_rn(d, p.dtoq);
        }
    }
    return sw2d_div_rn(q, p.dx * p.dy);
}

/* Length and forcing of the iteration that starts at time t, by one whole
 * warp.  FIXED: the reference's loop (:4798, :4838, :4876).  CFL:
 * min(dt_max, cfl/s), shortened to end exactly at t_end.  Every lane computes
 * the length; the quotients and series values that follow from it are
 * independent, so lane k computes the k-th of them (a binary64 operation
 * costs a warp 71 cycles however many lanes take part, and a chain of nine
 * divisions by one thread took longer than a small raster's tiles). */
__device__ __forceinline__ void prepare_slot(const StepParams& p, Slot* s, double t, double smax, double t_end) {
    const int lane = threadIdx.x & 31;
    double dt2, tm, tn;
    int active;
    if (p.dt_mode == 0) {
        double dt = p.dt_fixed;
        active = (t + dt <= t_end);
        dt2 = 2.00 * dt;
        tm = t + dt;
        tn = tm + dt;
    } else {
        active = (t < t_end);
        dt2 = smax > 0 ? fmin(p.dt_max, sw2d_div_rn(p.cfl, smax)) : p.dt_max;
        if (t + dt2 > t_end) dt2 = t_end - t;
        tm = t + 0.5 * dt2;
        tn = t + dt2;
    }
    if (lane == 0) {
        s->t = t;
        s->t_mid = tm;
        s->t_next = tn;
        s->dt2 = dt2;
        s->active = active;
    }
    if (lane < 2) (lane ? &s->dt2dy : &s->dt2dx)[0] = sw2d_div_rn(dt2, lane ? p.dy : p.dx);
    if (lane < 4) { /* rain at t and tm, then evaporation */
        const bool ev = lane >= 2;
        const double* v = ev ? p.evap : p.rain;
        double r = 0.0;
        if (v)
            r = sw2d_div_rn(series_at(v, ev ? p.nevap : p.nrain, p.dtrain, (lane & 1) ? tm : t, p.series_mode),
                            p.dtrain * 1000.0);
        (ev ? ((lane & 1) ? &s->ev2 : &s->ev1) : ((lane & 1) ? &s->rr2 : &s->rr1))[0] = r;
    }
    for (int k = lane; k < 2 * p.nsrc; k += 32) {
        const int i = k >> 1;
        ((k & 1) ? s->ql2 : s->ql1)[i] = source_at(p, i, (k & 1) ? tm : t);
    }
}

/* ------------------------------------------------------------------------ */
/* flux: SW2D-EFDC.cu:97-353                                                 */

__device__ __forceinline__ double face_manning(const StepParams& p, size_t a, size_t b) {
    if (!p.mcls) return p.manning;
    return sw2d_half(p.mtab[p.mcls[a]] + p.mtab[p.mcls[b]]);
}

/* (g n_f) n_f of the face between cells b and a: the reference's gg*rn*rn
 * (:193, :310), from the class-pair table or the uniform value when the
 * host could evaluate it once with the same operations */
__device__ __forceinline__ double friction_coef(const StepParams& p, size_t b, size_t a) {
    if (!p.mcls) return p.gnn_uni;
    if (p.gnn) return p.gnn[(int)p.mcls[b] * p.ncls + (int)p.mcls[a]];
    const double nf = face_manning(p, b, a);
    return p.g * nf * nf;
}

__device__ __forceinline__ double friction(const StepParams& p, double coef, double sq, double hm) {
    /* :193-198; the division by pow(hm, 1.333333) as a product with hm^-1.333333 */
    if (sw2d_le_pos(hm, p.th)) return 0.00;
    return (coef * sq) * sw2d_rpow_manning(hm);
}

/* a / dx for the continuity: exact scaling when dx is a power of two (the
 * constant division returns the same bits), else sw2d_div_by */
__device__ __forceinline__ double div_spacing(double a, const sw2d_divisor& d, int k) {
    if (k < 0) return sw2d_div_by(a, &d);
    return k == 0 ? a : sw2d_pow2_down(a, k, d.rd);
}

/* x is zero, or of a magnitude in [2^-400, 2^400] */
__device__ __forceinline__ bool mid_range(double x) {
    const uint32_t hi = (uint32_t)__double2hiint(x);
    return ((hi & 0x7ff00000u) - (623u << 20) <= (800u << 20)) || ((hi << 1) | (uint32_t)__double2loint(x)) == 0u;
}

/* Upwind donor-cell transport across the edge between two neighbouring
 * faces of the same orientation (the reference's umr/uml, umu/umd, vnr/vnl,
 * vnu/vnd, SW2D-EFDC.cu:171-189, :288-306):
 *     a (q1 + q0) / 2 + |a| (q0 - q1) / 2,   a = (w1 + w0) / 2,
 * with q0 the discharge of the face the edge is read from first.  The
 * reference evaluates every edge twice, once from each face beside it, with
 * the same operands in the same order (+ commutes exactly), so one
 * evaluation per edge gives bit-identical fluxes.  Halvings are exact while
 * nothing is subnormal, so with operands in the middle of the exponent range
 * the three of them are one quartering of the sum at the end. */
__device__ __noinline__ double edge_term_wide(double w, double qs, double qd) {
    const double a = sw2d_half(w);
    return sw2d_half(a * qs) + sw2d_half(fabs(a) * qd);
}
__device__ __forceinline__ double edge_term(double w1, double w0, double q0, double q1) {
    const double w = w1 + w0, qs = q1 + q0, qd = q0 - q1;
    if (mid_range(w) && mid_range(qs) && mid_range(qd)) return sw2d_quarter(w * qs + fabs(w) * qd);
    return edge_term_wide(w, qs, qd);
}

/* Kind of a face (SW2D-EFDC.cu:115-165, same tests in the same order):
 *   0 closed (an inactive side, or both sides at or below th)
 *   1 momentum (gravity, convection, friction)
 *   2 weir from side a, 3 weir from side b (a side's surface below the
 *     other side's bed), 4 / 5 dry-bed front with side b / a alone above th.
 * Side a is the north (x faces) / west (y faces) cell; ea, za its surface
 * h + z and its bed as ordered integers (sw2d_ord), ca its code.  The product
 * (hb - th) (ha - th) < 0 of the reference is decided from the two
 * comparisons with th (the differences keep the comparisons' signs and
 * their product of depths cannot underflow), and so is the front's sign.  A
 * weir from a side at or below th carries nothing: closed. */
constexpr int kActive = 1, kWet = 2, kBelow = 4; /* cell codes: active, h > th, h < th */
__device__ __forceinline__ int classify(int ca, int cb, int64_t ea, int64_t eb, int64_t za, int64_t zb) {
    if (!(ca & cb & kActive) || !((ca | cb) & kWet)) return 0;
    if (eb < za) return (ca & kWet) ? 2 : 0;
    if (ea < zb) return (cb & kWet) ? 3 : 0;
    return ((cb & kWet) && (ca & kBelow)) ? 4 : ((ca & kWet) && (cb & kBelow)) ? 5 : 1;
}

/* Discharge of a weir or dry-bed face, (c d) sqrt(G d): d the depth on the
 * weir's side, or the higher surface above the higher bed (:125-157). */
__device__ __forceinline__ double face_special(int kind, double ha, double hb, int64_t ea, int64_t eb, int64_t za,
                                               int64_t zb, double gg) {
    double d = kind == 2 ? ha : hb;
    if (kind > 3) d = sw2d_f64_of_ord(eb > ea ? eb : ea) - sw2d_f64_of_ord(zb > za ? zb : za);
    const double c = kind == 2 ? 0.5440 : kind == 3 ? -0.544 : kind == 4 ? -0.350 : 0.350;
    return c * d * sw2d_sqrt_rn((kind <= 3 ? gg : 2.00 * gg) * d);
}

/* momentum update of a face (SW2D-EFDC.cu:165-202 x, :282-319 y): along /
 * across are the face's two edge differences, already scaled. */
__device__ __forceinline__ double face_momentum(const StepParams& p, double coef, double ha, double za, double eb,
                                                double hm, double q0, double u0, double vt, double along,
                                                double across, double dt2, double dt2n) {
    const double gg = p.g;
    const double g13 = gg * hm * dt2n * (eb - ha - za);
    const double sq = sw2d_sqrt_rn(u0 * u0 + vt * vt); /* on the integer pipes, correctly rounded */
    const double ram = friction(p, coef, sq, hm);
    const double a = sw2d_half(dt2 * ram);
    /* the division on the integer pipes, correctly rounded (sw2d_div_rn) */
    return sw2d_div_rn((1.00 - a) * q0 + (-along - across - g13), 1.00 + a);
}

__device__ unsigned long long block_max_u64(unsigned long long v, unsigned long long* sm);

/* CFL speed contribution of one face of the entering state: (|velocity| +
 * sqrt(g * mean depth)) / spacing for faces between two active cells whose
 * mean depth is >= th (the oracle's cfl_speed, same operations). */
__device__ __forceinline__ double face_speed(double vel, double hm, double g, double rd) {
    return (fabs(vel) + sw2d_sqrt_rn(g * hm)) * rd;
}

#define NWARP (SW2D_BX * SW2D_BY / 32)

__device__ __forceinline__ int tid_linear() { return threadIdx.y * SW2D_BX + threadIdx.x; }

/* binary32 estimate of a face speed, from integer operations: a conversion
 * from binary64 costs a binary64 operation on this GPU */
__device__ __forceinline__ float face_speed_est(bool ok, double vel, double hm, double g, double rd) {
    return ok ? (fabsf(sw2d_f32_est_of_f64(vel)) + sqrtf(sw2d_f32_est_of_f64(g) * sw2d_f32_est_of_f64(hm))) *
                    sw2d_f32_est_of_f64(rd)
              : 0.0f;
}

/* exact block maxima of the x and the y face speeds together: binary32
 * estimates for every face, binary64 only for the faces within 1e-5 of the
 * block's binary32 maximum; both reductions share their barriers.  The
 * maxima are valid in thread 0. */
__device__ __forceinline__ void block_face_speed_max2(bool okx, double vx, double hmx, double rdx, bool oky,
                                                      double vy, double hmy, double rdy, double g, float* smf,
                                                      unsigned long long* smu, unsigned long long* sx,
                                                      unsigned long long* sy) {
    const int lane = tid_linear() & 31, warp = tid_linear() >> 5;
    const float ex = face_speed_est(okx, vx, hmx, g, rdx), ey = face_speed_est(oky, vy, hmy, g, rdy);
    float mx = ex, my = ey;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        my = fmaxf(my, __shfl_xor_sync(0xffffffffu, my, o));
    }
    if (lane == 0) {
        smf[warp] = mx;
        smf[NWARP + warp] = my;
    }
    __syncthreads();
    mx = smf[0];
    my = smf[NWARP];
#pragma unroll
    for (int k = 1; k < NWARP; k++) {
        mx = fmaxf(mx, smf[k]);
        my = fmaxf(my, smf[NWARP + k]);
    }
    unsigned long long bx = 0ull, by = 0ull;
    if (okx && ex >= mx * 0.99999f) bx = (unsigned long long)__double_as_longlong(face_speed(vx, hmx, g, rdx));
    if (oky && ey >= my * 0.99999f) by = (unsigned long long)__double_as_longlong(face_speed(vy, hmy, g, rdy));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long ux = __shfl_down_sync(0xffffffffu, bx, o), uy = __shfl_down_sync(0xffffffffu, by, o);
        bx = ux > bx ? ux : bx;
        by = uy > by ? uy : by;
    }
    if (lane == 0) {
        smu[warp] = bx;
        smu[NWARP + warp] = by;
    }
    __syncthreads();
    if (warp == 0) {
        bx = lane < NWARP ? smu[lane] : 0ull;
        by = lane < NWARP ? smu[NWARP + lane] : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long ux = __shfl_down_sync(0xffffffffu, bx, o), uy = __shfl_down_sync(0xffffffffu, by, o);
            bx = ux > bx ? ux : bx;
            by = uy > by ? uy : by;
        }
    }
    *sx = bx;
    *sy = by;
}

/* Rare binary64 work as calls: inlined, its instructions are computed ahead
 * of their branch or predicated, and one that is predicated off still takes
 * its 71 cycles. */
__device__ __noinline__ bool mean_ge_exact(double ha, double hb, double th) {
    return sw2d_ge_pos(sw2d_half(ha + hb), th);
}
/* raises a running maximum (bits of non-negative doubles) to a face's speed */
__device__ __noinline__ void raise_speed(unsigned long long* at, double vel, double ha, double hb, double g, double rd) {
    const unsigned long long v = sw2d_f64_bits(face_speed(vel, sw2d_half(ha + hb), g, rd));
    if (v <= 0x7ff0000000000000ull && v > __ldcg(at)) atomicMax(at, v);
}
/* the same for a face whose mean depth is known by estimate only */
__device__ __noinline__ void raise_speed_exact(unsigned long long* at, double vel, double ha, double hb, double g, double rd,
                                               double th) {
    if (mean_ge_exact(ha, hb, th)) raise_speed(at, vel, ha, hb, g, rd);
}

/* 8 bytes from global to shared memory past the registers; zeros when !in */
__device__ __forceinline__ void copy8_async(double* to, const double* from, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from),
                 "r"(in ? 8 : 0)
                 : "memory");
}

/* mean depth of a face >= th, exactly (true where the estimate is infinite,
 * which sends the face to raise_speed_exact): decided from the two cells'
 * codes unless th lies between their depths, then in binary32, in binary64
 * only within its error */
__device__ __forceinline__ bool mean_ge(double ha, double hb, int ca, int cb, float est, double th, float thf) {
    if (!((ca ^ cb) & kBelow)) return !(ca & kBelow);
    if (fabsf(est - thf) > 1e-5f * thf) return est > thf; /* not with thf NaN */
    return mean_ge_exact(ha, hb, th);
}

/* Every kernel of an iteration is launched with programmatic serialisation:
 * its blocks may be set up while the one before drains, and wait here for it
 * to be complete and its writes visible.  (Letting them come earlier, by an
 * explicit trigger, measured 11.1 against 11.6 us an iteration at 33 x 41 but
 * 21.1 against 19.5 at 256 x 256, where they take the place of running blocks;
 * plain launches 12.1 and 20.0.) */
__device__ __forceinline__ void after_previous() { cudaGridDependencySynchronize(); }

/* The new discharges of the faces of a 32 x BY block of cells (north and
 * west face of each), four block barriers:
 *   1  the block and a ring around it staged in shared memory; the surface
 *      h + z once per cell;
 *   2  every thread classifies its two faces; momentum faces are listed from
 *      the front of a list, weir and dry-bed faces from its back; closed faces
 *      are written at once;
 *   3  the edge terms some listed face reads are listed (from the rows'
 *      bit masks), and the weir and dry-bed faces computed;
 *   4  the edge terms, then the momentum faces, computed from their lists.
 * What bounds it: a binary64 instruction takes a warp 71 cycles on a GB300
 * whether one lane or all take part (measured), so the point of the lists is
 * that every binary64 instruction runs on full warps and that x and y faces,
 * the four kinds of edges and the three kinds of weir share one instruction
 * stream each (they differ in shared-memory offsets and selected operands).
 * CFL: face speeds estimated in binary32; a warp whose best estimate does
 * not reach the running maximum is done, else its lanes within 1e-5 of the
 * best are evaluated in binary64 and raise the maximum, all of its lanes where
 * an estimate says nothing (est_most and above): the result is the exact
 * maximum in any order.
 * PER_SM bounds the registers: 7 gives 32 of them (and 32 bytes of spills) and
 * six blocks an SM, as many as their 33 KB of shared memory let run; 6 would
 * give 40 at the same six (843 us against 820 at 4096 x 4096); 5 gives 48. */
template <int BY, int NT, int PER_SM>
__global__ void __launch_bounds__(NT, PER_SM) k64_flux(StepParams p, int cur) {
    constexpr int BX = SW2D_BX, NF = 2 * BX * BY, SW = BX + 2, NV = (BY + 2) * SW, NH = (BY + 1) * SW;
    static_assert(BX == 32, "one row per warp: its ballot is the row's bit mask");
    __shared__ double sh[NH];                         /* depth: rows -1 .. BY-1 */
    __shared__ int64_t so[2 * NH];                    /* surface h + z, then bed, as ordered integers */
    __shared__ float shf[NH];                         /* depth estimate */
    constexpr int U = 0, V = NV, QX = 2 * NV, QY = 3 * NV;
    __shared__ double sf[4 * NV];                     /* face velocities and discharges: rows -1 .. BY */
    __shared__ double sedge[4 * NH];
    __shared__ uint8_t scode[NH];
    __shared__ unsigned short flist[NF], elist[2 * NF + 2 * BX + 2 * BY];
    __shared__ unsigned rowx[BY + 1], rowy[BY + 1];
    __shared__ int cnt[3];
    const int tx = threadIdx.x, ty = threadIdx.y, t = ty * BX + tx;
    const int c0 = blockIdx.x * BX, r0 = blockIdx.y * BY;
    const int c = c0 + tx, r = r0 + ty;
    const Slot& s = p.clk->slot[cur];
    after_previous();
    const double dt2 = s.dt2, dt2dx = s.dt2dx, dt2dy = s.dt2dy;
    const int active = s.active;
    const int P = p.P, R = p.R, C = p.C;
    const size_t i = (size_t)(r + H) * P + (c + H);
    const double th = p.th;
    {
        /* velocities and discharges are first read after the second barrier:
         * copied past the registers, waited for there */
        const double* const from[4] = {p.uu1, p.vv1, p.qx[0], p.qy[0]};
        for (int k = t; k < NV; k += NT) {
            const int rr = k / SW, cc = k - rr * SW;
            const int gr = r0 - 1 + rr, gc = c0 - 1 + cc;
            const bool in = gr <= R + 1 && gc <= C + 1; /* the padded raster */
            const size_t g = in ? (size_t)(gr + H) * P + (gc + H) : 0;
#pragma unroll
            for (int f = 0; f < 4; f++) copy8_async(&sf[f * NV + k], from[f] + g, in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const double* __restrict__ h = p.h[cur];
        const double* __restrict__ z = p.z;
        const uint8_t* __restrict__ flags = p.flags;
        if (t < 3) cnt[t] = 0;
        if (t == 3) rowx[BY] = rowy[BY] = 0u;
        for (int k = t; k < NH; k += NT) {
            const int rr = k / SW, cc = k - rr * SW;
            const int gr = r0 - 1 + rr, gc = c0 - 1 + cc;
            const bool in = gr <= R + 1 && gc <= C + 1;
            const size_t g = (size_t)(gr + H) * P + (gc + H);
            const double hh = in ? h[g] : 0.0, zz = in ? z[g] : 0.0;
            sh[k] = hh;
            so[k] = sw2d_ord(hh + zz);
            so[NH + k] = sw2d_ord(zz);
            shf[k] = sw2d_f32_est_depth(hh);
            scode[k] = (uint8_t)((in ? (flags[g] & SW2D_F_ACTIVE) : 0) | (sw2d_gt_pos(hh, th) ? kWet : 0) |
                                 (sw2d_lt_pos(hh, th) ? kBelow : 0));
        }
    }
    if (!active) { /* (the whole block) nothing in flight may outlive it */
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }
    __syncthreads();
    const int s0 = (ty + 1) * SW + tx + 1;
    const bool doX = r <= R && c < C, doY = r < R && c <= C;
    if (ty < BY) {
        const int cc = scode[s0], cn = scode[s0 - SW], cw = scode[s0 - 1];
        const int64_t ec = so[s0], zc = so[NH + s0];
        int kx = 0, ky = 0;
        if (doX) {
            if (r == R && p.outflow_south) /* south edge: free overfall when open */
                kx = (cn & kActive) && (cn & kWet) ? 2 : 0;
            else
                kx = classify(cn, cc, so[s0 - SW], ec, so[NH + s0 - SW], zc);
        }
        if (doY) ky = classify(cw, cc, so[s0 - 1], ec, so[NH + s0 - 1], zc);
        if (doX && kx == 0) p.qx[1][i] = 0.0;
        if (doY && ky == 0) p.qy[1][i] = 0.0;
        const unsigned all = 0xffffffffu, lt = (1u << tx) - 1u;
        const unsigned mx = __ballot_sync(all, kx == 1), my = __ballot_sync(all, ky == 1);
        const unsigned px = __ballot_sync(all, kx > 1), py = __ballot_sync(all, ky > 1);
        int base = 0;
        if (tx == 0) {
            rowx[ty] = mx;
            rowy[ty] = my;
            base = atomicAdd(&cnt[0], __popc(mx) + __popc(my));
        } else if (tx == 1) {
            base = atomicAdd(&cnt[1], __popc(px) + __popc(py));
        }
        int mb = __shfl_sync(all, base, 0) + __popc(mx & lt);
        int pb = NF - 1 - (__shfl_sync(all, base, 1) + __popc(px & lt));
        if (kx) flist[kx == 1 ? mb : pb] = (unsigned short)(2 * t | kx << 10);
        mb = mb - __popc(mx & lt) + __popc(mx) + __popc(my & lt);
        pb = pb + __popc(px & lt) - __popc(px) - __popc(py & lt);
        if (ky) flist[ky == 1 ? mb : pb] = (unsigned short)(2 * t + 1 | ky << 10);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (ty < BY) {
        /* edges of the row: south of its cells for x and y faces (types 0,
         * 2), east of them and west of the first (1, 3); warp 0 also the
         * edges north of the block */
        const unsigned X = rowx[ty], Y = rowy[ty], m0 = X | rowx[ty + 1], m2 = Y | rowy[ty + 1];
        const unsigned m1 = X | (X >> 1), m3 = Y | (Y >> 1);
        const unsigned u0 = ty == 0 ? X : 0u, u2 = ty == 0 ? Y : 0u;
        const unsigned w1 = X & 1u, w3 = Y & 1u;
        const int n0 = __popc(m0), n1 = n0 + __popc(m1), n2 = n1 + __popc(m2), n3 = n2 + __popc(m3);
        const int n4 = n3 + __popc(u0), n5 = n4 + __popc(u2), n6 = n5 + (int)w1;
        int base = 0;
        if (tx == 0) base = atomicAdd(&cnt[2], n6 + (int)w3);
        base = __shfl_sync(0xffffffffu, base, 0);
        const unsigned lt = (1u << tx) - 1u, bit = 1u << tx;
        if (m0 & bit) elist[base + __popc(m0 & lt)] = (unsigned short)(s0 << 2);
        if (m1 & bit) elist[base + n0 + __popc(m1 & lt)] = (unsigned short)(s0 << 2 | 1);
        if (m2 & bit) elist[base + n1 + __popc(m2 & lt)] = (unsigned short)(s0 << 2 | 2);
        if (m3 & bit) elist[base + n2 + __popc(m3 & lt)] = (unsigned short)(s0 << 2 | 3);
        if (u0 & bit) elist[base + n3 + __popc(u0 & lt)] = (unsigned short)((s0 - SW) << 2);
        if (u2 & bit) elist[base + n4 + __popc(u2 & lt)] = (unsigned short)((s0 - SW) << 2 | 2);
        if (tx == 0 && w1) elist[base + n5] = (unsigned short)((s0 - 1) << 2 | 1);
        if (tx == 0 && w3) elist[base + n6] = (unsigned short)((s0 - 1) << 2 | 3);
    }
    if (p.dt_mode == 1 && ty < BY) {
        const int cc = scode[s0], cn = scode[s0 - SW], cw = scode[s0 - 1];
        const float hx = 0.5f * (shf[s0] + shf[s0 - SW]), hy = 0.5f * (shf[s0] + shf[s0 - 1]);
        const bool okx = doX && r > 0 && r < R && (cn & cc & kActive) && mean_ge(sh[s0 - SW], sh[s0], cn, cc, hx, th, p.thf);
        const bool oky = doY && c > 0 && c < C && (cw & cc & kActive) && mean_ge(sh[s0 - 1], sh[s0], cw, cc, hy, th, p.thf);
        const float ex = okx ? (fabsf(sw2d_f32_est_hi(sf[U + s0])) + sw2d_sqrt_est(p.gf * hx)) * p.rdxf : 0.f;
        const float ey = oky ? (fabsf(sw2d_f32_est_hi(sf[V + s0])) + sw2d_sqrt_est(p.gf * hy)) * p.rdyf : 0.f;
        unsigned long long* best = p.flight->smax[cur];
        const float cx = sw2d_f32_est_hi(__longlong_as_double((long long)__ldcg(best)));
        const float cy = sw2d_f32_est_hi(__longlong_as_double((long long)__ldcg(best + 1)));
        const float mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(ex)));
        const float my = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(ey)));
        if (mx < p.est_most && my < p.est_most) {
            if (okx && ex >= fmaxf(mx, cx) * 0.99999f) raise_speed(best, sf[U + s0], sh[s0], sh[s0 - SW], p.g, p.rdx);
            if (oky && ey >= fmaxf(my, cy) * 0.99999f) raise_speed(best + 1, sf[V + s0], sh[s0], sh[s0 - 1], p.g, p.rdy);
        } else { /* a negative, infinite or NaN depth or velocity, which would hide the warp's other faces: all of them */
            if (okx) raise_speed_exact(best, sf[U + s0], sh[s0], sh[s0 - SW], p.g, p.rdx, th);
            if (oky) raise_speed_exact(best + 1, sf[V + s0], sh[s0], sh[s0 - 1], p.g, p.rdy, th);
        }
    }
    for (int k = t; k < cnt[1]; k += NT) {
        const int id = flist[NF - 1 - k], ft = (id & 1023) >> 1, ly = ft / BX, lx = ft % BX;
        const int sj = (ly + 1) * SW + lx + 1, sa = (id & 1) ? sj - 1 : sj - SW;
        const double F = face_special(id >> 10, sh[sa], sh[sj], so[sa], so[sj], so[NH + sa], so[NH + sj], p.g);
        ((id & 1) ? p.qy[1] : p.qx[1])[(size_t)(r0 + ly + H) * P + (c0 + lx + H)] = F;
    }
    __syncthreads();
    for (int k = t; k < cnt[2]; k += NT) {
        const int id = elist[k], e = id >> 2;
        const int w = ((id & 1) ? V : U) + e, q = ((id & 2) ? QY : QX) + e, step = (id & 1) ? 1 : SW;
        const int back = (id & 3) == 1 ? 1 - SW : (id & 3) == 2 ? SW - 1 : 0;
        sedge[(id & 3) * NH + e] = edge_term(sf[w + step], sf[w + back], sf[q], sf[q + step]);
    }
    __syncthreads();
    for (int k = t; k < cnt[0]; k += NT) {
        const int id = flist[k], ft = (id & 1023) >> 1, ly = ft / BX, lx = ft % BX;
        const bool y = (id & 1) != 0; /* the y face west of cell j, else the x face north of it */
        const int sj = (ly + 1) * SW + lx + 1, da = y ? 1 : SW, st = y ? SW : 1;
        const size_t j = (size_t)(r0 + ly + H) * P + (c0 + lx + H);
        const int ea = (y ? 2 * NH : 0) + sj, eb = ea + NH;
        double along = dt2dx * (sedge[ea] - sedge[ea - SW]), across = dt2dy * (sedge[eb] - sedge[eb - 1]);
        if (y && r0 + ly == 0) along = 0.0;    /* the reference's edge rules (:280-284, :184-186) */
        if (!y && c0 + lx == 0) across = 0.0;
        const double hm = sw2d_half(sh[sj] + sh[sj - da]);
        const int T = (y ? U : V) + sj; /* the other direction's face velocities */
        const double vt = sw2d_quarter(sf[T] + sf[T + st] + sf[T - da] + sf[T - da + st]);
        const double F = face_momentum(p, friction_coef(p, j, j - (y ? 1 : P)), sh[sj - da],
                                       sw2d_f64_of_ord(so[NH + sj - da]), sw2d_f64_of_ord(so[sj]), hm,
                                       sf[(y ? QY : QX) + sj], sf[(y ? V : U) + sj], vt, along, across, dt2,
                                       y ? dt2dy : dt2dx);
        (y ? p.qy[1] : p.qx[1])[j] = F;
    }
}

/* ------------------------------------------------------------------------ */
/* continuity: SW2D-EFDC.cu:602-664                                          */

template <bool FULL>
__device__ __forceinline__ double continuity(const StepParams& p, size_t i, uint8_t f, double ho,
                                             double divx, double divy, double dt2, double rr,
                                             double ev, const double* ql, double* raw,
                                             double* rain_term) {
    double pct, evapo;
    if (sw2d_gt(ho, p.ev_wl_min)) {
        pct = p.pct_lake;
        evapo = ev;
    } else {
        pct = p.pct_land;
        evapo = 0.000;
    }
    const double rcell = p.rainw ? rr * sw2d_f64_of_f32(p.rainw[i]) : rr; /* exact, off the FP64 pipe */
    /* (((dqx/dx + dqy/dy) - q_src) - r pct) + e; subtracting a zero source
     * and adding a zero evaporation change no value, so they are skipped */
    double sum = div_spacing(divx, p.ddx, p.kdx) + div_spacing(divy, p.ddy, p.kdy);
    if (FULL && (f & SW2D_F_SOURCE)) {
        double qli = 0.0;
        for (int k = 0; k < p.nsrc; k++)
            if (p.src_idx[k] == (int)i) qli = ql[k];
        sum = sum - qli;
    }
    sum = sum - rcell * pct;
    if (FULL && p.evap) sum = sum + evapo;
    double hn = ho - dt2 * sum;
    *raw = hn;
    *rain_term = rcell * pct;
    hn = sw2d_max0(hn);
    if (!(f & SW2D_F_ACTIVE)) hn = 0.00;
    return hn;
}

/* ------------------------------------------------------------------------ */
/* block reductions (fixed order: deterministic for a given grid)            */


__device__ __forceinline__ double block_sum(double v, double* sm) {
    const int lane = tid_linear() & 31, warp = tid_linear() >> 5, nw = (int)(blockDim.x * blockDim.y) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) sm[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (warp == 0) {
        t = lane < nw ? sm[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    }
    return t; /* valid in thread 0 */
}

__device__ unsigned long long block_max_u64(unsigned long long v, unsigned long long* sm) {
    const int lane = tid_linear() & 31, warp = tid_linear() >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long u = __shfl_down_sync(0xffffffffu, v, o);
        v = u > v ? u : v;
    }
    __syncthreads();
    if (lane == 0) sm[warp] = v;
    __syncthreads();
    unsigned long long t = 0;
    if (warp == 0) {
        t = lane < NWARP ? sm[lane] : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            unsigned long long u = __shfl_down_sync(0xffffffffu, t, o);
            t = u > t ? u : t;
        }
    }
    return t; /* valid in thread 0 */
}

#define NPART 4 /* prime: volume, CFL bits x, y; update: weighted rain, lake cells, land cells, outlet */

/* Adds the ledger sums of the last iteration of parity `par`, if they are
 * not added yet (its tiles' partials were written by its k64_update), and its
 * outlet record; by one whole block.  last_row: the tile row that holds the
 * raster's last row. */
__device__ void settle_ledger(const StepParams& p, int par, int gx, int gy, int last_row) {
    __shared__ double smd[NWARP];
    Flight64::Sums& in = p.flight->sums[par];
    if (!__ldcg(&in.pending)) return;
    const int nt = blockDim.x, tid = threadIdx.x, tiles = gx * gy;
    const double* part = p.partials + (size_t)par * tiles * NPART;
    double vr = 0.0, ve = 0.0, vd = 0.0, vq = 0.0;
    if (p.ledger_cells) {
        for (int b = tid; b < tiles; b += nt) {
            const double* pb = part + (size_t)b * NPART;
            if (p.rainw) vr += __ldcg(pb);
            ve += __ldcg(pb + 1);
            if (!p.rainw) vd += __ldcg(pb + 2);
        }
        if (p.rainw) vr = block_sum(vr, smd);
        ve = block_sum(ve, smd);
        if (!p.rainw) vd = block_sum(vd, smd);
    }
    if (p.outflow_south) { /* the tiles that hold the last row */
        for (int b = tid; b < gx; b += nt) vq += __ldcg(part + (size_t)(last_row * gx + b) * NPART + 3);
        vq = block_sum(vq, smd);
    }
    if (tid == 0) {
        DevClock* clk = p.clk;
        const double dt2 = in.dt2, area = p.area, rr2 = in.rr2, ev2 = in.ev2, tn = in.t_next, src = in.src;
        const double l0 = clk->led[LED_RAIN], l1 = clk->led[LED_EVAP], l2 = clk->led[LED_SOURCE], l3 = clk->led[LED_OUTFLOW];
        in.pending = 0;
        const double rain = !p.ledger_cells ? rr2 * p.rain_static
                            : p.rainw       ? vr
                                            : ve * (rr2 * p.pct_lake) + vd * (rr2 * p.pct_land);
        const double qo = vq * p.dy;
        clk->led[LED_RAIN] = l0 + dt2 * rain * area;
        clk->led[LED_EVAP] = l1 + dt2 * (ve * ev2) * area;
        clk->led[LED_SOURCE] = l2 + dt2 * src * area;
        clk->led[LED_QOUT] = qo;
        clk->led[LED_OUTFLOW] = l3 + dt2 * qo;
        if (!isfinite(vq)) atomicOr(&clk->status, 1);
        if (p.outlet) {
            const long long n = clk->outlet_n, k = n % p.outlet_cap;
            p.outlet[2 * k] = tn;
            p.outlet[2 * k + 1] = qo;
            clk->outlet_n = n + 1;
        }
    }
}

/* The clock of the iteration in slot `cur`, by one warp of an extra block of
 * its k64_update, beside the tiles: the CFL speed k64_flux found and the next
 * iteration's length and forcing. */
__device__ void advance_clock(const StepParams& p, int cur) {
    if (threadIdx.x >= 32) return;
    DevClock* clk = p.clk;
    Flight64* fl = p.flight;
    const Slot& s = clk->slot[cur];
    if (!s.active) {
        const unsigned long long* from = reinterpret_cast<const unsigned long long*>(&s);
        unsigned long long* to = reinterpret_cast<unsigned long long*>(&clk->slot[cur ^ 1]);
        for (int k = threadIdx.x; k < (int)(sizeof(Slot) / 8); k += 32) to[k] = from[k];
        return;
    }
    /* of the state this iteration started from */
    const double smax = __longlong_as_double((long long)__ldcg(&fl->smax[cur][0])) +
                        __longlong_as_double((long long)__ldcg(&fl->smax[cur][1]));
    const double t = s.t_next, t_end = clk->t_end, dt2 = s.dt2, rr2 = s.rr2, ev2 = s.ev2;
    const long long iters = clk->iters + 1, lim = clk->iter_end;
    __syncwarp();
    /* past the iteration limit the next slot is inactive: t_end = t */
    prepare_slot(p, &clk->slot[cur ^ 1], t, smax, iters < lim ? t_end : t);
    if (threadIdx.x == 0) {
        fl->smax[cur][0] = fl->smax[cur][1] = 0ull;
        Flight64::Sums& o = fl->sums[cur];
        o.dt2 = dt2;
        o.rr2 = rr2;
        o.ev2 = ev2;
        o.t_next = t;
        double src = 0.0;
        for (int k = 0; k < p.nsrc; k++) /* a source overridden on its cell adds nothing */
            if (p.src_idx[k] >= 0) src += s.ql2[k];
        o.src = src;
        o.pending = 1;
        clk->led[LED_DTLAST] = dt2;
        clk->led[LED_SMAX] = smax;
        if (!isfinite(smax)) atomicOr(&clk->status, 1);
        clk->t = t;
        clk->s_max = smax;
        clk->iters = iters;
    }
}

/* ------------------------------------------------------------------------ */
/* continuity at t, treat_error, continuity at t+dt, hm_hn + uu1_vv1:         */
/* SW2D-EFDC.cu:602-664, :695-725, :362-452 in one pass                       */

/* "active and provisional depth < th" of a cell, decided from a binary32
 * estimate of the depth (sw2d_dry_est): 0 or 1, or 2 where the exact binary64
 * continuity has to decide. */
template <bool FULL>
__device__ __noinline__ bool provisional_exact(const StepParams& p, const Slot& s, size_t i, uint8_t f, double ho,
                                               double fN, double fS, double fW, double fE) {
    double raw, rt;
    return sw2d_lt_pos(continuity<FULL>(p, i, f, ho, fS - fN, fE - fW, s.dt2, s.rr1, s.ev1, s.ql1, &raw, &rt), p.th);
}
template <bool FULL>
__device__ __forceinline__ uint8_t provisional_dry(const StepParams& p, float dt2, float rl, float rd, float ev, size_t i,
                                                   uint8_t f, double ho, double fN, double fS, double fW, double fE) {
    const bool lake = sw2d_gt(ho, p.ev_wl_min);
    float src = lake ? rl : rd;
    if (p.rainw) src *= p.rainw[i];
    float mag = fabsf(src);
    if (FULL && lake) {
        src -= ev;
        mag += fabsf(ev);
    }
    const int dry = sw2d_dry_est(sw2d_f32_est_hi(ho), sw2d_f32_est_hi(fN), sw2d_f32_est_hi(fS), sw2d_f32_est_hi(fW),
                                 sw2d_f32_est_hi(fE), src, mag, dt2, p.rdxf, p.rdyf, p.thf);
    return (uint8_t)(FULL && (f & SW2D_F_SOURCE) ? 2 : dry);
}

/* FULL: evaporation, point sources or rain whose ledger is kept per cell.
 * Tile of the update kernel: TW x TH cells (and their north and west faces)
 * per block.  The dry flags are evaluated on the tile plus two rows north
 * and west and one row south and east, the new depths on the tile plus the
 * row north and the column west: the faces of the tile read both; the halo
 * is recomputed, not exchanged.  Block 0 prepares the next iteration
 * meanwhile and block 1 adds up the previous one's ledger sums (chains of
 * dependent reads, divisions and sums; at the end of the last tile they would
 * be the longest part of a small raster's iteration).
 * Bounded by the binary64 additions and products of the final depth and of
 * the face means (71 issue cycles a warp each; the flags take none) and by
 * the latencies between them: large tiles run eight blocks an SM (32
 * registers, up to 80 bytes of spills), 438 us at 4096 x 4096 against 472 and
 * 511 with six and five. */
template <int TW, int TH, int NT, bool FULL>
__global__ void __launch_bounds__(NT, TH >= 16 && !FULL ? 8 : 6) k64_update(StepParams p, int cur, int gx, int gy) {
    constexpr int DW = TW + 3, DH = TH + 3, NW = TW + 1, NH = TH + 1;
    after_previous();
    if (blockIdx.x < 2) {
        if (blockIdx.x == 0) advance_clock(p, cur);
        else settle_ledger(p, cur ^ 1, gx, gy, (p.R - 1) / TH);
        return;
    }
    __shared__ uint8_t sdry[DH][DW];   /* rows r0-2 .. r0+TH, cols c0-2 .. c0+TW */
    __shared__ double shn[NH][NW];     /* rows r0-1 .. r0+TH-1, cols c0-1 .. c0+TW-1 */
    __shared__ double smd[NWARP];
    const int tid = threadIdx.x;
    const int tile = blockIdx.x - 2, tyi = tile / gx;
    const int c0 = (tile - tyi * gx) * TW, r0 = tyi * TH;
    const int nxt = cur ^ 1;
    const Slot& s = p.clk->slot[cur];
    const int P = p.P, R = p.R, C = p.C;
    const double th = p.th;
    const double* __restrict__ fx = p.qx[1]; /* k64_flux's new discharges, read only */
    const double* __restrict__ fy = p.qy[1];
    const double* __restrict__ hc = p.h[cur];
    if (!s.active) {
        /* the loop condition failed: the iteration copies the depth */
        for (int k = tid; k < TW * TH; k += NT) {
            const int r = r0 + k / TW, c = c0 + k % TW;
            if (r < R && c < C) {
                const size_t i = (size_t)(r + H) * P + (c + H);
                p.h[nxt][i] = hc[i];
            }
        }
        return;
    }
    const double dt2 = s.dt2, rr2 = s.rr2, ev2 = s.ev2;
    {
        /* 1: provisional depth at t -> "active and h* < th" (0 outside the raster) */
        const float dt2f = sw2d_f32_est_of_f64(dt2), rr1 = sw2d_f32_est_of_f64(s.rr1);
        const float rl = rr1 * p.plf, rd = rr1 * p.pdf, ev = FULL ? sw2d_f32_est_of_f64(s.ev1) : 0.f;
        int open = 0;
        for (int k = tid; k < DH * DW; k += NT) {
            const int rr = k / DW, cc = k - rr * DW;
            const int r = r0 - 2 + rr, c = c0 - 2 + cc;
            uint8_t dflag = 0;
            if (r >= 0 && r < R && c >= 0 && c < C) {
                const size_t i = (size_t)(r + H) * P + (c + H);
                const uint8_t f = p.flags[i];
                if (f & SW2D_F_ACTIVE)
                    dflag = provisional_dry<FULL>(p, dt2f, rl, rd, ev, i, f, hc[i], fx[i], fx[i + P], fy[i], fy[i + 1]);
            }
            sdry[rr][cc] = dflag;
            open |= dflag & 2;
        }
        if (open) { /* the thread's own undecided cells */
            for (int k = tid; k < DH * DW; k += NT) {
                const int rr = k / DW, cc = k - rr * DW;
                if (sdry[rr][cc] != 2) continue;
                const size_t i = (size_t)(r0 - 2 + rr + H) * P + (c0 - 2 + cc + H);
                sdry[rr][cc] = provisional_exact<FULL>(p, s, i, p.flags[i], hc[i], fx[i], fx[i + P], fy[i], fy[i + 1]);
            }
        }
    }
    __syncthreads();
    /* 2: treat_error per face (a face carrying water out of a cell whose
     * provisional depth fell below th is closed, :704-719), final depth
     * at t+dt; written for the tile's own cells, kept in shared memory
     * for the faces */
    double vr = 0.0;
    int nlake = 0, nland = 0;
    for (int k = tid; k < NH * NW; k += NT) {
        const int rr = k / NW, cc = k - rr * NW;
        const int r = r0 - 1 + rr, c = c0 - 1 + cc;
        double hn = 0.0;
        if (r >= 0 && r < R && c >= 0 && c < C) {
            const size_t i = (size_t)(r + H) * P + (c + H);
            const uint8_t f = p.flags[i];
            const int dr = rr + 1, dc = cc + 1;
            const uint8_t dC = sdry[dr][dc];
            double fN = fx[i], fS = fx[i + P], fW = fy[i], fE = fy[i + 1];
            if ((sw2d_gt0(fN) && sdry[dr - 1][dc]) || (sw2d_lt0(fN) && dC)) fN = 0;
            if ((sw2d_gt0(fS) && dC) || (sw2d_lt0(fS) && sdry[dr + 1][dc])) fS = 0;
            if ((sw2d_gt0(fW) && sdry[dr][dc - 1]) || (sw2d_lt0(fW) && dC)) fW = 0;
            if ((sw2d_gt0(fE) && dC) || (sw2d_lt0(fE) && sdry[dr][dc + 1])) fE = 0;
            const double ho = hc[i];
            double raw, rt;
            hn = continuity<FULL>(p, i, f, ho, fS - fN, fE - fW, dt2, rr2, ev2, s.ql2, &raw, &rt);
            if (rr >= 1 && cc >= 1) { /* the tile's own cell */
                p.h[nxt][i] = hn;
                if (f & SW2D_F_ACTIVE) {
                    if (sw2d_lt0(raw)) atomicAdd(&p.clk->led[LED_CLAMP], -raw * p.area); /* max(h, 0) gain */
                    if (FULL && p.ledger_cells) {
                        if (p.rainw) vr += rt;
                        if (sw2d_gt(ho, p.ev_wl_min)) nlake++;
                        else nland++;
                    }
                }
            }
        }
        shn[rr][cc] = hn;
    }
    __syncthreads();
    /* 3: the closed faces written back and the face velocities of the new
     * state, uu1 = qx/hm and vv1 = qy/hn (hm_hn, uu1_vv1), for the
     * tile's north and west faces (the raster's south and east edge
     * faces in the last tile row / column) */
    for (int k = tid; k < TH * TW; k += NT) {
        const int rr = k / TW, cc = k - rr * TW;
        const int r = r0 + rr, c = c0 + cc;
        if (r > R || c > C) continue;
        const size_t i = (size_t)(r + H) * P + (c + H);
        const int dr = rr + 2, dc = cc + 2, nr = rr + 1, nc = cc + 1;
        if (c < C) {
            double F = fx[i];
            if ((sw2d_gt0(F) && sdry[dr - 1][dc]) || (sw2d_lt0(F) && sdry[dr][dc])) F = 0;
            p.qx[0][i] = F;
            double hm;
            if (r == 0) hm = shn[nr][nc];
            else if (r == R) hm = shn[nr - 1][nc];
            else hm = sw2d_half(shn[nr][nc] + shn[nr - 1][nc]);
            p.uu1[i] = sw2d_ge_pos(hm, th) ? sw2d_div_rn(F, hm) : 0.00;
        }
        if (r < R) {
            double F = fy[i];
            if ((sw2d_gt0(F) && sdry[dr][dc - 1]) || (sw2d_lt0(F) && sdry[dr][dc])) F = 0;
            p.qy[0][i] = F;
            double hn;
            if (c == 0) hn = shn[nr][nc];
            else if (c == C) hn = shn[nr][nc - 1];
            else hn = sw2d_half(shn[nr][nc] + shn[nr][nc - 1]);
            p.vv1[i] = sw2d_ge_pos(hn, th) ? sw2d_div_rn(F, hn) : 0.0;
        }
    }
    /* ledger sums of the tile, added up beside the next iteration's tiles */
    double* pb = p.partials + ((size_t)cur * gx * gy + tile) * NPART;
    if (FULL && p.ledger_cells) {
        if (p.rainw) vr = block_sum(vr, smd);
        /* counts as binary32-exact integers: at most TW * TH */
        nlake = __reduce_add_sync(0xffffffffu, nlake);
        nland = __reduce_add_sync(0xffffffffu, nland);
        __shared__ int sc[2];
        if (tid < 2) sc[tid] = 0;
        __syncthreads();
        if ((tid & 31) == 0) {
            atomicAdd(&sc[0], nlake);
            atomicAdd(&sc[1], nland);
        }
        __syncthreads();
        if (tid == 0) {
            pb[0] = vr;
            pb[1] = (double)sc[0];
            pb[2] = (double)sc[1];
        }
    }
    if (p.outflow_south && r0 <= R - 1 && R - 1 < r0 + TH) {
        double vq = 0.0;
        for (int cc = tid; cc < TW; cc += NT) { /* the open faces south of the last row */
            const int c = c0 + cc, dr = R - 1 - r0 + 2, dc = cc + 2;
            if (c >= C) continue;
            const size_t i = (size_t)(R - 1 + H) * P + (c + H);
            const double F = fx[i + P];
            const bool shut = (sw2d_gt0(F) && sdry[dr][dc]) || (sw2d_lt0(F) && sdry[dr + 1][dc]);
            if ((p.flags[i] & SW2D_F_ACTIVE) && !shut) vq += F;
        }
        vq = block_sum(vq, smd);
        if (tid == 0) pb[3] = vq;
    }
}

__device__ __forceinline__ void report(const StepParams& p) {
    const DevClock* clk = p.clk;
    Flight64::Report& o = p.flight->report;
    o.iters = clk->iters;
    o.t = clk->t;
    o.dt2 = clk->slot[0].dt2;
    o.active = clk->slot[0].active;
    o.status = clk->status;
}

__global__ void __launch_bounds__(SW2D_BX * SW2D_BY) k64_settle(StepParams p, int gx, int gy,
                                                                     int last_row) {
    settle_ledger(p, 0, gx, gy, last_row); /* the last iteration is of one parity; the other has nothing to add */
    settle_ledger(p, 1, gx, gy, last_row);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        p.clk->iter_end = LLONG_MAX;
        report(p);
    }
}

__global__ void __launch_bounds__(32) k64_begin(StepParams p, double t_end, long long limit) {
    DevClock* clk = p.clk;
    const long long iters = clk->iters, end = limit < 0 ? LLONG_MAX : iters + limit;
    prepare_slot(p, &clk->slot[0], clk->t, clk->s_max, iters < end ? t_end : clk->t);
    __syncwarp();
    if (threadIdx.x == 0) {
        clk->t_end = t_end;
        clk->iter_end = end;
        p.flight->report.iters0 = iters;
        report(p);
    }
}

/* Volume (sum of h over active cells) and, with full, the CFL speed of the
 * current state (face rule of k64_flux); the last block stores them and
 * prepares the next slot. */
__global__ void __launch_bounds__(SW2D_BX * SW2D_BY) k64_prime(StepParams p, int cur, int full) {
    if (!full) { /* one block: the next slot only */
        DevClock* clk = p.clk;
        if (tid_linear() < 32)
            prepare_slot(p, &clk->slot[cur], clk->t, clk->s_max, clk->iters < clk->iter_end ? clk->t_end : clk->t);
        return;
    }
    __shared__ double smd[NWARP];
    __shared__ float smf[2 * NWARP];
    __shared__ unsigned long long smu[2 * NWARP];
    __shared__ bool last;
    const int c = blockIdx.x * SW2D_BX + threadIdx.x;
    const int r = blockIdx.y * SW2D_BY + threadIdx.y;
    double vol = 0.0;
    bool okx = false, oky = false;
    double hmx = 0, hmy = 0, vx = 0, vy = 0;
    if (r < p.R && c < p.C) {
        const int P = p.P;
        const size_t i = (size_t)(r + H) * P + (c + H);
        const double* h = p.h[cur];
        const uint8_t fc = p.flags[i];
        if (fc & SW2D_F_ACTIVE) {
            vol = h[i];
            if (r > 0 && (p.flags[i - P] & SW2D_F_ACTIVE)) {
                hmx = 0.50 * (h[i] + h[i - P]);
                okx = hmx >= p.th;
                vx = p.uu1[i];
            }
            if (c > 0 && (p.flags[i - 1] & SW2D_F_ACTIVE)) {
                hmy = 0.50 * (h[i] + h[i - 1]);
                oky = hmy >= p.th;
                vy = p.vv1[i];
            }
        }
    }
    vol = block_sum(vol, smd);
    unsigned long long sx, sy;
    block_face_speed_max2(okx, vx, hmx, p.rdx, oky, vy, hmy, p.rdy, p.g, smf, smu, &sx, &sy);
    const int tid = tid_linear();
    const int b = blockIdx.y * gridDim.x + blockIdx.x;
    if (tid == 0) {
        p.partials[(size_t)b * NPART + 0] = vol;
        p.partials[(size_t)b * NPART + 1] = __longlong_as_double((long long)sx);
        p.partials[(size_t)b * NPART + 2] = __longlong_as_double((long long)sy);
    }
    __threadfence();
    if (tid == 0) last = (atomicAdd(&p.clk->counter, 1u) == gridDim.x * gridDim.y - 1);
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int nb = gridDim.x * gridDim.y;
    double v = 0.0;
    unsigned long long ux = 0ull, uy = 0ull;
    for (int bb = tid; bb < nb; bb += SW2D_BX * SW2D_BY) {
        const volatile double* pb = p.partials + (size_t)bb * NPART;
        v += pb[0];
        unsigned long long a = (unsigned long long)__double_as_longlong(pb[1]);
        unsigned long long w = (unsigned long long)__double_as_longlong(pb[2]);
        ux = a > ux ? a : ux;
        uy = w > uy ? w : uy;
    }
    v = block_sum(v, smd);
    ux = block_max_u64(ux, smu);
    uy = block_max_u64(uy, smu);
    if (tid < 32) {
        DevClock* clk = p.clk;
        /* full: 1 = volume only (the clock is left alone), 2 = initial state
         * (volume origin, CFL speed and the first slot) */
        const double vol = __shfl_sync(0xffffffffu, v, 0) * p.area;
        const double smax = __longlong_as_double((long long)__shfl_sync(0xffffffffu, ux, 0)) +
                            __longlong_as_double((long long)__shfl_sync(0xffffffffu, uy, 0));
        if (tid == 0) {
            clk->led[LED_VOLUME] = vol;
            if (full == 2) {
                clk->s_max = smax;
                clk->led[LED_SMAX] = smax;
                clk->led[LED_VOLUME0] = vol;
            }
            clk->counter = 0;
        }
        if (full == 2)
            prepare_slot(p, &clk->slot[cur], clk->t, smax, clk->iters < clk->iter_end ? clk->t_end : clk->t);
    }
}

/* ------------------------------------------------------------------------ */
/* hm_hn + uu1_vv1: SW2D-EFDC.cu:362-452, the face velocities of the current
 * state (after its depth was set or restored; the iteration's own are
 * written by k64_update) */

__global__ void __launch_bounds__(SW2D_BX * SW2D_BY) k64_facevel(StepParams p, int cur) {
    const int c = blockIdx.x * SW2D_BX + threadIdx.x;
    const int r = blockIdx.y * SW2D_BY + threadIdx.y;
    if (r > p.R || c > p.C) return;
    const int P = p.P;
    const size_t i = (size_t)(r + H) * P + (c + H);
    const double* __restrict__ h = p.h[cur];
    const double th = p.th;
    if (c < p.C) {
        const double F = p.qx[0][i];
        double hm;
        if (r == 0) hm = h[i];
        else if (r == p.R) hm = h[i - P];
        else hm = sw2d_half(h[i] + h[i - P]);
        p.uu1[i] = sw2d_ge_pos(hm, th) ? sw2d_div_rn(F, hm) : 0.00;
    }
    if (r < p.R) {
        const double F = p.qy[0][i];
        double hn;
        if (c == 0) hn = h[i];
        else if (c == p.C) hn = h[i - 1];
        else hn = sw2d_half(h[i] + h[i - 1]);
        p.vv1[i] = sw2d_ge_pos(hn, th) ? sw2d_div_rn(F, hn) : 0.0;
    }
}

/* Reference-layout velocities for output: uu_vv (:458-483), uua_vva (:489-522). */
__global__ void k64_cellvel(StepParams p, int cur, double* uu, double* vv, double* uua, double* vva) {
    const int c = blockIdx.x * SW2D_BX + threadIdx.x;
    const int r = blockIdx.y * SW2D_BY + threadIdx.y;
    if (r >= p.R || c >= p.C) return;
    const int P = p.P;
    const size_t i = (size_t)(r + H) * P + (c + H);
    const size_t k = (size_t)r * p.C + c;
    const double* u1 = p.uu1;
    const double* v1 = p.vv1;
    if (uu || vv) {
        double a = 0, b = 0;
        if (p.h[cur][i] >= p.th) {
            a = (u1[i + P] + u1[i]) / 2.00;
            b = (v1[i + 1] + v1[i]) / 2.00;
        }
        if (uu) uu[k] = a;
        if (vv) vv[k] = b;
    }
    if (uua) uua[k] = (c > 0) ? 0.250 * (u1[i] + u1[i + P] + u1[i - 1] + u1[i + P - 1]) : 0.50 * (u1[i] + u1[i + P]);
    if (vva) vva[k] = (r > 0) ? 0.250 * (v1[i] + v1[i + 1] + v1[i - P] + v1[i - P + 1]) : 0.50 * (v1[i] + v1[i + 1]);
}

/* Boundary-discharge sample (couple_BC_efdc, SW2D-EFDC.cu:728-1067): one
 * thread per boundary face.  North/south faces use uua and east/west faces
 * vva at the catchment cell, as the reference's call passes them
 * (SW2D-EFDC.cu:4909, signature :728); inflow to the lake only. */
__global__ void k_couple(StepParams p, int n, const int* __restrict__ faces, int lagged, int initial,
                         double* __restrict__ vel_prev, double* __restrict__ q) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int P = p.P;
    const int i = faces[2 * k], side = faces[2 * k + 1];
    const int r = i / P - H, c = i % P - H;
    const double* u1 = p.uu1;
    const double* v1 = p.vv1;
    double vnow;
    if (side <= 1)
        vnow = (c > 0) ? 0.250 * (u1[i] + u1[i + P] + u1[i - 1] + u1[i + P - 1]) : 0.50 * (u1[i] + u1[i + P]);
    else
        vnow = (r > 0) ? 0.250 * (v1[i] + v1[i + 1] + v1[i - P] + v1[i - P + 1]) : 0.50 * (v1[i] + v1[i + 1]);
    const double v = initial ? 0.0 : (lagged ? vel_prev[k] : vnow);
    const double hh = p.h[0][i];
    double out;
    switch (side) {
    case 1: out = (v < 0) ? -v * hh * p.dx : 0.00; break; /* south :760-767 */
    case 0: out = (v > 0) ? v * hh * p.dx : 0.00; break;  /* north :777-784 */
    case 2: out = (v < 0) ? -v * hh * p.dy : 0.00; break; /* east :794-801 */
    default: out = (v > 0) ? v * hh * p.dy : 0.00; break; /* west :812-819 */
    }
    q[k] = out;
    vel_prev[k] = vnow;
}

void launch_couple(const StepParams& p, int nfaces, const int* faces, int lagged, int initial, double* vel_prev,
                   double* q, cudaStream_t s) {
    k_couple<<<(nfaces + 127) / 128, 128, 0, s>>>(p, nfaces, faces, lagged, initial, vel_prev, q);
}

/* ------------------------------------------------------------------------ */

static dim3 grid_faces(const StepParams& p) {
    return dim3((p.C + 1 + SW2D_BX - 1) / SW2D_BX, (p.R + 1 + SW2D_BY - 1) / SW2D_BY);
}
static dim3 grid_cells(const StepParams& p) {
    return dim3((p.C + SW2D_BX - 1) / SW2D_BX, (p.R + SW2D_BY - 1) / SW2D_BY);
}

int fp64_kernels_per_iteration() { return 2; }

/* How a raster is cut into the update kernel's tiles and the flux kernel's
 * blocks: large ones for the smaller share of halo while there are many,
 * small ones so that a small raster reaches every SM (each block's chain of
 * dependent binary64 operations then holds fewer of them).  Each line lies
 * between the sizes where one side and the other is faster; measured, us an
 * iteration, plain slopes / fractal terrain with lake terms and sources:
 *   update tiles 64 x 16 against 32 x 16: 1482 / 1364 and 1510 / 1400 at
 *     4096^2, 213.6 / 204.8 and 214.5 / 205.5 at 1450^2, 192.6 / 175.9 and
 *     191.3 / 174.0 at 1361^2;
 *   32 x 16 against 32 x 8: 56.4 / 49.1 and 57.7 / 50.8 at 600^2, 48.4 / 48.0
 *     and 48.4 / 48.7 at 548^2, 35.7 / 33.9 and 34.0 / 32.4 at 400^2;
 *   32 x 8 against 32 x 4: 27.5 / 28.6 and 28.6 / 28.5 at 330^2, 23.8 / 26.1
 *     and 23.9 / 24.5 at 310^2, 21.2 / 21.7 and 20.3 / 20.1 at 256^2, 13.5 /
 *     17.8 and 12.6 / 16.4 at 33^2;
 *   flux blocks of 8 rows against 4 (256 threads each): 67.4 / 64.3 and 67.6
 *     / 68.5 at 700^2, 52.4 / 46.8 and 50.7 / 48.9 at 566^2, 47.3 / 43.6 and
 *     43.2 / 41.8 at 480^2;
 *   flux blocks with 32 registers against 48: 1482 / 1364 and 1525 / 1422 at
 *     4096^2, 118.9 / 108.2 and 119.7 / 110.2 at 1024^2, 86.5 / 80.2 and 86.6
 *     / 81.5 at 836^2, 74.9 / 69.8 and 74.6 / 69.6 at 767^2. */
struct Cut64 {
    int kind, tw, th, gx, gy;
    dim3 flux;
    int by;
    bool lean; /* the flux kernel with 32 registers */
};
static Cut64 cut_of(int R, int C) {
    Cut64 k;
    const long long cells = (long long)(R + 1) * (C + 1);
    k.kind = cells >= 2000000 ? 0 : cells >= 300000 ? 1 : cells >= 100000 ? 2 : 3;
    k.tw = k.kind == 0 ? 64 : 32;
    k.th = k.kind <= 1 ? 16 : k.kind == 2 ? 8 : 4;
    k.gx = (C + 1 + k.tw - 1) / k.tw;
    k.gy = (R + 1 + k.th - 1) / k.th;
    k.by = cells >= 320000 ? 8 : 4;
    k.lean = cells >= 700000;
    k.flux = dim3((C + 1 + SW2D_BX - 1) / SW2D_BX, (R + 1 + k.by - 1) / k.by);
    return k;
}

size_t fp64_partials(int rows, int cols) {
    const Cut64 k = cut_of(rows, cols);
    const size_t prime = (size_t)((cols + SW2D_BX - 1) / SW2D_BX) * ((rows + SW2D_BY - 1) / SW2D_BY);
    return NPART * std::max(prime, (size_t)2 * k.gx * k.gy);
}

template <typename... A>
static void chain_launch(void (*k)(A...), dim3 grid, dim3 block, cudaStream_t s, A... args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k, args...); /* an error stays for the caller's cudaGetLastError */
}

template <bool FULL>
static void launch_update(const Cut64& k, int n, const StepParams& p, int cur, cudaStream_t s) {
    if (k.kind == 0) chain_launch(k64_update<64, 16, 256, FULL>, dim3(n), dim3(256), s, p, cur, k.gx, k.gy);
    else if (k.kind == 1) chain_launch(k64_update<32, 16, 256, FULL>, dim3(n), dim3(256), s, p, cur, k.gx, k.gy);
    else if (k.kind == 2) chain_launch(k64_update<32, 8, 256, FULL>, dim3(n), dim3(256), s, p, cur, k.gx, k.gy);
    else chain_launch(k64_update<32, 4, 256, FULL>, dim3(n), dim3(256), s, p, cur, k.gx, k.gy);
}

void fp64_launch_iteration(const StepParams& p, int cur, cudaStream_t s, cudaEvent_t* ev) {
    const Cut64 k = cut_of(p.R, p.C);
    if (ev) cudaEventRecord(ev[0], s);
    const dim3 blk(SW2D_BX, 8);
    if (k.by == 4) chain_launch(k64_flux<4, 256, 5>, k.flux, blk, s, p, cur);
    else if (!k.lean) chain_launch(k64_flux<8, 256, 5>, k.flux, blk, s, p, cur);
    else chain_launch(k64_flux<8, 256, 7>, k.flux, blk, s, p, cur);
    if (ev) cudaEventRecord(ev[1], s);
    const int n = k.gx * k.gy + 2;
    const bool full = p.evap || p.nsrc > 0 || p.ledger_cells;
    if (full) launch_update<true>(k, n, p, cur, s);
    else launch_update<false>(k, n, p, cur, s);
    if (ev) cudaEventRecord(ev[2], s);
}

void fp64_launch_settle(const StepParams& p, cudaStream_t s) {
    const Cut64 k = cut_of(p.R, p.C);
    k64_settle<<<1, SW2D_BX * SW2D_BY, 0, s>>>(p, k.gx, k.gy, (p.R - 1) / k.th);
}

void fp64_launch_begin(const StepParams& p, double t_end, long long limit, cudaStream_t s) {
    k64_begin<<<1, 32, 0, s>>>(p, t_end, limit);
}

void fp64_launch_prime(const StepParams& p, int cur, int full, cudaStream_t s) {
    k64_prime<<<full ? grid_cells(p) : dim3(1, 1), dim3(SW2D_BX, SW2D_BY), 0, s>>>(p, cur, full);
}

void fp64_launch_face_velocity(const StepParams& p, int cur, cudaStream_t s) {
    k64_facevel<<<grid_faces(p), dim3(SW2D_BX, SW2D_BY), 0, s>>>(p, cur);
}

void fp64_launch_cell_velocity(const StepParams& p, int cur, double* uu, double* vv, double* uua,
                               double* vva, cudaStream_t s) {
    k64_cellvel<<<grid_cells(p), dim3(SW2D_BX, SW2D_BY), 0, s>>>(p, cur, uu, vv, uua, vva);
}

} // namespace sw2d
