// letkf_members.cu -- the caller's conversion around letkf_run on the device.
//
// Reference: run_da_parallel (code/x86/TradDA/DA/EnDNN/src/module_da_parallel.F90:163-261)
// hands letkf_run the ensemble as mean and perturbations (dnn2letkf, :184-204)
// and turns the analysis back into full members with the relaxation-to-prior
// blend and the background and analysis spreads (letkf2dnn, :214-258).
// letkf_gpu_run_members runs the three steps on the GPU, so full members go in
// and full members and spreads come out without a host pass over the state.
// With one column per cube, no overlap and no vertical blocks (and k <= 64 in
// the mixed forms; not where the FP64 form runs on the tensor cores) the steps
// are fused into the analysis (LgParams::members):
// H reads the members as they are, and the update kernels form each row's
// mean and perturbations as they read the row and write the blended members
// and both spreads, so no pass over the state is added.  Otherwise:
//   k_members_split: per state row, the mean over members (sum / real(ens))
//       and the perturbations; a NaN member stops the run (the reference
//       prints and stops, :188-193);
//   the analysis of letkf_gpu_run on the split state;
//   k_members_blend: where |grid_lat| <= polar_lat,
//       xout = gamma1 (axb + xb) + gamma2 (axa + xa),
//       spread_b = sqrt(sum xb^2 / ens), spread_a = sqrt(sum (xout - axa)^2 / ens);
//       elsewhere the background passes through (xout = xb + axb) and both
//       spreads are the background's.
// Lanes over members, shuffle sums.
#include <cmath>

#include "letkf_internal.cuh"

namespace {

constexpr int kT = 256;

// The sums over the lanes of four rows' values d[0..3], in the order of a xor tree
// from 16 down to 1 (the first two steps fold two rows into one value each):
// row i's in the lanes 8 i .. 8 i + 7.
__device__ __forceinline__ double fold4(const double *d, int lane)
{
    const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
    const double e0 = (h16 ? d[2] : d[0]) + __shfl_xor_sync(0xffffffffu, h16 ? d[0] : d[2], 16);
    const double e1 = (h16 ? d[3] : d[1]) + __shfl_xor_sync(0xffffffffu, h16 ? d[1] : d[3], 16);
    double v = (h8 ? e1 : e0) + __shfl_xor_sync(0xffffffffu, h8 ? e0 : e1, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ bool is_nan_bits(double x)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
    return u > 0x7ff0000000000000ull;
}

// Four rows per warp at a time.  The FP64 pipe bounds both passes (a warp per
// row spent most of it on the lane sums, the division and the square roots of one
// row): the sums fold rows together, and the divisions and roots are done
// for several rows at once.  4,050 columns of 97 rows, k = 64: split 0.54 -> 0.38 ms,
// blend 1.53 -> 0.63 ms.
__global__ void __launch_bounds__(kT)
k_members_split(int64_t nrows, int k, const double *__restrict__ xin, double *__restrict__ xb,
                double *__restrict__ axb, unsigned *__restrict__ status)
{
    constexpr int NE = LG_MAX_ENS / 32;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (kT / 32);
    const double fk = (double)(float)k;    // real(ens)
    for (int64_t r0 = 4 * (blockIdx.x * (int64_t)(kT / 32) + (threadIdx.x >> 5)); r0 < nrows; r0 += 4 * warps) {
        double x[4][NE], s[4];
        bool bad = false;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const double *src = xin + min(r0 + i, nrows - 1) * k;
#pragma unroll
            for (int q = 0; q < NE; q++) x[i][q] = (lane + 32 * q < k) ? src[lane + 32 * q] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            s[i] = 0.0;
#pragma unroll
            for (int q = 0; q < NE; q++)
                if (lane + 32 * q < k) {
                    bad |= is_nan_bits(x[i][q]);
                    s[i] += x[i][q];
                }
        }
        const double m = fold4(s, lane) / fk;
        if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(status, LG_ST_BAD_STATE);
        if ((lane & 7) == 0 && r0 + lane / 8 < nrows) axb[r0 + lane / 8] = m;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const double mi = __shfl_sync(0xffffffffu, m, 8 * i);
            if (r0 + i >= nrows) continue;
#pragma unroll
            for (int q = 0; q < NE; q++)
                if (lane + 32 * q < k) xb[(r0 + i) * k + lane + 32 * q] = x[i][q] - mi;
        }
    }
}

// `per` rows per warp (a multiple of 4, at most 32): row j's spreads on lane j.
__global__ void __launch_bounds__(kT)
k_members_blend(int nlat, int n, int64_t nrows, int k, int per, double gamma1, double gamma2, double polar,
                const float *__restrict__ glat, const double *__restrict__ xb, const double *__restrict__ axb,
                const double *xa, const double *__restrict__ axa, double *xout, double *__restrict__ spread_b,
                double *__restrict__ spread_a)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (kT / 32);
    const double fk = (double)(float)k;
    for (int64_t r0 = per * (blockIdx.x * (int64_t)(kT / 32) + (threadIdx.x >> 5)); r0 < nrows; r0 += per * warps) {
        const int64_t mine = r0 + lane;
        const bool on = lane < per && mine < nrows;
        const unsigned blends =
            __ballot_sync(0xffffffffu, on && fabs((double)glat[on ? mine / n % nlat : 0]) <= polar);
        const double my_ab = on ? axb[mine] : 0.0, my_aa = on ? axa[mine] : 0.0;
        double my_sb = 0.0, my_sa = 0.0;
        for (int j = 0; j < per && r0 + j < nrows; j += 4) {
            double ab[4], aa[4], sb[4], sa[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                ab[i] = __shfl_sync(0xffffffffu, my_ab, j + i);
                aa[i] = __shfl_sync(0xffffffffu, my_aa, j + i);
                sb[i] = sa[i] = 0.0;
            }
            for (int e = lane; e < k; e += 32) {
                double b[4], a[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int64_t at = min(r0 + j + i, nrows - 1) * k + e;
                    b[i] = xb[at];
                    a[i] = ((blends >> (j + i)) & 1u) ? xa[at] : 0.0;
                }
                // xout may be xa itself: each lane reads its members before writing them
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    double o, d;
                    if ((blends >> (j + i)) & 1u) {
                        o = __dadd_rn(__dmul_rn(gamma1, __dadd_rn(ab[i], b[i])),
                                      __dmul_rn(gamma2, __dadd_rn(aa[i], a[i])));
                        d = __dsub_rn(o, aa[i]);
                    } else {
                        o = __dadd_rn(b[i], ab[i]);
                        d = b[i];
                    }
                    sa[i] = __dadd_rn(sa[i], __dmul_rn(d, d));
                    sb[i] = __dadd_rn(sb[i], __dmul_rn(b[i], b[i]));
                    if (r0 + j + i < nrows) xout[(r0 + j + i) * k + e] = o;
                }
            }
            // row j + i's sums from lanes 8 i to lane j + i
            const double vb = __shfl_sync(0xffffffffu, fold4(sb, lane), 8 * (lane & 3));
            const double va = __shfl_sync(0xffffffffu, fold4(sa, lane), 8 * (lane & 3));
            if ((lane & ~3) == j) {
                my_sb = vb;
                my_sa = va;
            }
        }
        const double qb = sqrt(my_sb / fk), qa = sqrt(my_sa / fk);
        if (on) {
            spread_b[mine] = qb;
            spread_a[mine] = qa;
        }
    }
}

unsigned grid_for(int64_t nrows, int per)
{
    const int64_t want = (nrows + per * (kT / 32) - 1) / (per * (kT / 32));
    return (unsigned)(want < (1 << 20) ? want : (1 << 20));
}

// Room for the split state, as far as it is not held yet.
bool split_has_room(letkf_ctx *ctx, size_t nstate, size_t nmean, int64_t nobs)
{
    size_t grow = 0, held = 0, fr = 0, tot = 0;
    auto add = [&](const DevBuf<double> &b, size_t n) {
        if (n <= b.n) return;
        grow += n * sizeof(double);
        held += b.n * sizeof(double);
    };
    add(ctx->d_xb, nstate);
    add(ctx->d_xa, nstate);
    add(ctx->d_axb, nmean);
    add(ctx->d_axa, nmean);
    if (grow == 0) return true;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return lg_split_fits((int64_t)(fr + held), (int64_t)grow, nobs, ctx->k) != 0;
}

}  // namespace

// Whether `room` bytes hold `split` bytes of split state and what the run cannot do
// without beside it: the observations' arrays (y in k doubles, and up to 128 bytes) and
// 2 GiB, of which the list pool leaves 1 GiB and the rest serves it and the
// core's intermediates (both go in smaller pieces where memory is short).
extern "C" int lg_split_fits(int64_t room, int64_t split, int64_t nobs, int64_t k)
{
    return split + nobs * (8 * k + 128) + ((int64_t)2 << 30) <= room;
}

extern "C" int letkf_gpu_run_members(letkf_ctx *ctx, const double *xb_in, const letkf_obs *obs,
                                     const letkf_blend *blend, double *xa_out, double *spread_b,
                                     double *spread_a, int flags)
{
    if (!ctx) return LETKF_ERR_INVALID;
    if (!xb_in || !xa_out || !spread_b || !spread_a || !blend)
        return lg_set_err(ctx, LETKF_ERR_INVALID, "NULL pointer");
    if (flags != LETKF_HOST_PTRS && flags != LETKF_DEVICE_PTRS) return lg_set_err(ctx, LETKF_ERR_INVALID, "bad flags");
    if (ctx->range0 != 0 || ctx->range1 != ctx->ncubes)
        return lg_set_err(ctx, LETKF_ERR_UNSUPPORTED, "the members entry point analyses every cube");
    int rc = lg_check_run(ctx, obs);
    if (rc) return rc;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return lg_set_err(ctx, LETKF_ERR_CUDA, "cudaSetDevice");
    const bool host = flags == LETKF_HOST_PTRS;
    const int k = ctx->k, n = ctx->n;
    const int64_t nrows = ctx->ncol * n;
    const size_t nstate = (size_t)nrows * k, nmean = (size_t)nrows;
    auto cu = [&](cudaError_t e) { return e == cudaSuccess ? LETKF_OK : lg_set_err(ctx, LETKF_ERR_CUDA, cudaGetErrorString(e)); };
#define LG_TRY(x)                     \
    do {                              \
        const int rc_ = cu(x);        \
        if (rc_) return rc_;          \
    } while (0)
    LG_TRY(cudaEventRecord(ctx->ev[0], ctx->stream));
    rc = lg_reset_status(ctx);
    if (rc) return rc;
    // The split and the blend fused into the analysis (H reads the members as
    // they are, the update forms each row's mean and perturbations as it reads
    // it and writes the blended members and both spreads): no state pass of
    // its own.  Kept as separate passes where the update is not one pass over
    // one column per cube (overlapped cubes, vertical blocks) and for the
    // mixed form's wide core (k = 96, 128).
    bool fused = ctx->params.cube_n == 1 && ctx->params.overlap == 0 && !(ctx->params.vert_dist > 0.0) &&
                 !(lg_is_mixed(ctx->params.precision) && k > 64);
    // The FP64 form's tensor-core path (letkf_f64.cu) takes the split state:
    // its analysis with two passes over the state is far shorter than the
    // fused k_core_fp64 (4 degrees, k = 64, 4,050 columns: 4.9 against 81 ms
    // on the device).  Where the split state does not fit the device beside the
    // rest of the run, or the context's limit, the fused form stays.
    if (fused && !lg_is_mixed(ctx->params.precision) && lg_f64_supports(k) &&
        (ctx->scratch_limit == 0 || 16 * (nstate + nmean) <= (size_t)ctx->scratch_limit) &&
        split_has_room(ctx, nstate, nmean, obs->nobs)) {
        cudaError_t e = ctx->d_xb.reserve(nstate);
        if (e == cudaSuccess) e = ctx->d_axb.reserve(nmean);
        if (e == cudaSuccess) e = ctx->d_xa.reserve(nstate);
        if (e == cudaSuccess) e = ctx->d_axa.reserve(nmean);
        if (e == cudaSuccess) {
            fused = false;
        } else if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            ctx->d_xb.release();
            ctx->d_xa.release();
        } else {
            LG_TRY(e);
        }
    }
    if (fused) {
        LG_TRY(ctx->d_spb.reserve(nmean));
        LG_TRY(ctx->d_spa.reserve(nmean));
        const double *din = xb_in;
        double *dout = xa_out, *dsb = spread_b, *dsa = spread_a;
        if (host) {
            LG_TRY(ctx->d_xb.reserve(nstate));
            LG_TRY(ctx->d_xa.reserve(nstate));
            LG_TRY(cudaMemcpyAsync(ctx->d_xb.p, xb_in, sizeof(double) * nstate, cudaMemcpyHostToDevice, ctx->stream));
            din = ctx->d_xb.p;
            dout = ctx->d_xa.p;
            dsb = ctx->d_spb.p;
            dsa = ctx->d_spa.p;
        }
        ctx->members_on = true;
        ctx->members_g1 = blend->gamma1;
        ctx->members_g2 = blend->gamma2;
        ctx->members_polar = blend->polar_lat_deg;
        ctx->members_spb = dsb;
        ctx->members_spa = dsa;
        unsigned long long cnt[LG_CNT_N] = {};
        rc = lg_run_analysis(ctx, obs, host, din, nullptr, dout, nullptr, cnt);
        ctx->members_on = false;
        ctx->members_spb = ctx->members_spa = nullptr;
        if (rc) return rc;
        if (host) {
            LG_TRY(cudaMemcpyAsync(xa_out, dout, sizeof(double) * nstate, cudaMemcpyDeviceToHost, ctx->stream));
            LG_TRY(cudaMemcpyAsync(spread_b, dsb, sizeof(double) * nmean, cudaMemcpyDeviceToHost, ctx->stream));
            LG_TRY(cudaMemcpyAsync(spread_a, dsa, sizeof(double) * nmean, cudaMemcpyDeviceToHost, ctx->stream));
        }
        return lg_finish_run(ctx, obs, cnt);
    }
    LG_TRY(ctx->d_xb.reserve(nstate));
    LG_TRY(ctx->d_axb.reserve(nmean));
    LG_TRY(ctx->d_xa.reserve(nstate));
    LG_TRY(ctx->d_axa.reserve(nmean));
    const double *din = xb_in;
    if (host) {
        // the analysis perturbations are written to d_xa only after the split
        LG_TRY(cudaMemcpyAsync(ctx->d_xa.p, xb_in, sizeof(double) * nstate, cudaMemcpyHostToDevice, ctx->stream));
        din = ctx->d_xa.p;
    }
    lg_count_launch();
    k_members_split<<<grid_for(nrows, 4), kT, 0, ctx->stream>>>(nrows, k, din, ctx->d_xb.p, ctx->d_axb.p,
                                                             ctx->d_status.p);
    LG_TRY(cudaGetLastError());
    unsigned long long cnt[LG_CNT_N] = {};
    unsigned st = 0;
    rc = lg_read_status(ctx, st, cnt);
    if (rc) return rc;
    if (st & LG_ST_BAD_STATE) return lg_set_err(ctx, LETKF_ERR_INVALID, "a background member is NaN");
    rc = lg_run_analysis(ctx, obs, host, ctx->d_xb.p, ctx->d_axb.p, ctx->d_xa.p, ctx->d_axa.p, cnt);
    if (rc) return rc;
    double *dout = xa_out, *dsb = spread_b, *dsa = spread_a;
    if (host) {
        LG_TRY(ctx->d_spb.reserve(nmean));
        LG_TRY(ctx->d_spa.reserve(nmean));
        dout = ctx->d_xa.p;          // blended in place
        dsb = ctx->d_spb.p;
        dsa = ctx->d_spa.p;
    }
    // 32 rows per warp once that still gives every SM eight warps
    const int per = nrows >= 32 * 8 * 152 ? 32 : 4;
    lg_count_launch();
    k_members_blend<<<grid_for(nrows, per), kT, 0, ctx->stream>>>(
        ctx->nlat, n, nrows, k, per, blend->gamma1, blend->gamma2, blend->polar_lat_deg, ctx->d_glat.p, ctx->d_xb.p,
        ctx->d_axb.p, ctx->d_xa.p, ctx->d_axa.p, dout, dsb, dsa);
    LG_TRY(cudaGetLastError());
    if (host) {
        LG_TRY(cudaMemcpyAsync(xa_out, dout, sizeof(double) * nstate, cudaMemcpyDeviceToHost, ctx->stream));
        LG_TRY(cudaMemcpyAsync(spread_b, dsb, sizeof(double) * nmean, cudaMemcpyDeviceToHost, ctx->stream));
        LG_TRY(cudaMemcpyAsync(spread_a, dsa, sizeof(double) * nmean, cudaMemcpyDeviceToHost, ctx->stream));
    }
#undef LG_TRY
    return lg_finish_run(ctx, obs, cnt);
}
