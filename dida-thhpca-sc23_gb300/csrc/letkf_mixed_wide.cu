// letkf_mixed_wide.cu -- mixed-precision per-cube LETKF core for k = 96 and 128.
//
// The same analysis and precision choices as k_core_mixed (letkf_mixed.cu;
// letkf_core, code/x86/TradDA/DA/LETKF/src/letkf_core.F90:14-233, and
// xb_2_xa, letkf_compute.F90:231-301) for ensembles whose stacked hi/lo rows
// (2k) do not fit one MMA's 128 rows.  Differences of layout:
//   * A: the tile holds Yhat_lo in rows 0..k-1 (zero to 127) and Yhat_hi
//     from row 128; two MMAs per K step, lo x hi and hi x hi (N = k),
//     accumulate into two TMEM ranges (columns 0 and 256 of a 512-column
//     allocation: one CTA per SM); g and the diagonal of A are summed on the
//     FP32 pipe by the conversion threads, as in the narrow core;
//   * A = 0.5 (S + S^T) with S = HH + 2 LH staged once (no FP64 copy of A':
//     the w-bar residual adds (k-1)/rho in FP64 to the FP32 A);
//   * the update's operands (xb rows and T, k members deep) are two
//     128-byte-swizzled tiles along the member axis.
// Three launches per block of cubes, as the narrow core's at k = 64: the A build
// and the update on the tensor cores (a work queue; one CTA per SM, the update
// two at k = 96), and between them the eigenproblems (k_wide_eig), which spend their time on
// shuffles, barriers and dependent arithmetic and therefore run several CTAs
// per SM.  The FP32 Jacobi takes the hierarchical ordering over blocks of two
// columns (k = 128, lg_jacobi32b2) or three (k = 96, lg_jacobi32b3).  One
// launch with all stages, a cube at a time on 8 warps per SM, took 64.5 ms on
// 28,800 cubes of k = 96 (72% of it in the Jacobi, a third of the issue slots
// used); the three take 29.2 ms: 3.7 A build, 22.1 eigenproblems, 3.4 update.
#include <algorithm>

#include "letkf_internal.cuh"
#include "letkf_jacobi.cuh"
#include "letkf_mixed_util.cuh"
#include "letkf_umma.cuh"

#ifndef LG_MIXED_JACOBI_TOL
#define LG_MIXED_JACOBI_TOL 2e-6f
#endif
// chunks summed by the tensor cores in the scratch accumulators before the
// FP32 round-to-nearest addition to the running sums (as in letkf_mixed.cu)
#ifndef LG_ACC_FLUSH
#define LG_ACC_FLUSH 16
#endif

namespace {

constexpr int kTB = 512;         // threads of the A build (its conversions bound it)
constexpr int kTW = 256;         // threads of the update

constexpr size_t r1024(size_t b) { return (b + 1023) & ~(size_t)1023; }
constexpr size_t zmax(size_t a, size_t b) { return a > b ? a : b; }

template <int K>
struct WCfg {
    static constexpr int KB = K / 4;
    static constexpr int NLOW = KB * (KB + 1) / 2;
    static constexpr int CH = 64;                        // observations per MMA tile
    static constexpr uint32_t TMEM_COLS = 512;
    static constexpr uint32_t HI_COL = 256;              // first TMEM column of the hi accumulator
    static constexpr uint32_t ACC1 = 128;                // scratch accumulators after the running ones
    static constexpr int NB = K;                         // A-build N: Yhat_hi
    static constexpr int TROWS = (128 + NB > 256) ? 128 + NB : 256;
    static constexpr int TILE = TROWS * 128;
    static constexpr int LDS = K + 1;                    // S staging row stride
    static constexpr size_t STAGE = (size_t)CH * K * sizeof(float);
    static constexpr size_t TBSUB = (size_t)K * 128;     // one T tile along members (K rows)
    static constexpr size_t AREA_A = r1024(zmax(2 * TILE + 2 * STAGE, (size_t)K * LDS * sizeof(float)));
    static constexpr size_t SMEM_A = 1024 + AREA_A +
                                     2 * K * sizeof(double) + 3 * CH * (sizeof(int) + 2 * sizeof(float));
    // the update's operands: tiles of 64 members, hi and lo; at k = 96 the last 32
    // members of both share one tile (lo from byte 64 of a row), so two CTAs fit
    static constexpr int UT = K == 96 ? 3 : 4;
    static constexpr int PER_SM_U = K == 96 ? 2 : 1;
    __device__ static __forceinline__ int utile(int lo, int s) { return K == 96 ? (s ? 2 : lo) : 2 * lo + s; }
    __device__ static __forceinline__ int uchunk(int lo, int s, int c) { return K == 96 && s ? c + 4 * lo : c; }
    static constexpr size_t SMEM_U = 1024 + UT * TBSUB + UT * 16384 + sizeof(double) * (K + 128);
    static_assert(K > 64 && K <= 128 && K % 32 == 0, "wide form: k = 96 or 128");
    static_assert(TILE % 1024 == 0 && STAGE % 1024 == 0 && TBSUB % 1024 == 0, "1024-byte aligned tiles");
    static_assert(SMEM_A <= 227 * 1024 && SMEM_U <= 227 * 1024, "shared memory");
    static_assert(16 * K * sizeof(float) <= STAGE, "g and diagonal task sums pass through a gather stage");
    static_assert(K <= (int)ACC1 && HI_COL + ACC1 + K <= TMEM_COLS, "A-build accumulators must fit the TMEM allocation");
};

// Launch 1: A (FP32, without (k-1)/rho I) into mA and g into mg for the cubes of
// the work queue's chunks.
template <int K>
__global__ void __launch_bounds__(kTB, 1)
k_wide_build(LgParams prm, const float *__restrict__ ys32, const int32_t *__restrict__ lidx,
             const float2 *__restrict__ lmeta, const int *__restrict__ queue, int nchunks, int chunk,
             const int64_t *__restrict__ loff, const int32_t *__restrict__ lcnt, int64_t ncubes,
             float *__restrict__ mA, double *__restrict__ mg, unsigned long long *__restrict__ counters,
             unsigned *__restrict__ status, const unsigned *__restrict__ ymax)
{
    using C = WCfg<K>;
    constexpr int CH = C::CH;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *RA = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    double *misc = reinterpret_cast<double *>(RA + C::AREA_A);       // 2K
    int *mg_i = reinterpret_cast<int *>(misc + 2 * K);              // 3 x CH obs indices
    float *msq = reinterpret_cast<float *>(mg_i + 3 * CH);          // 3 x CH sqrt(rloc)
    float *me = msq + 3 * CH;                                       // 3 x CH e
    float *stage0 = reinterpret_cast<float *>(RA + 2 * C::TILE);
    float *stage1 = stage0 + CH * K;
    __shared__ uint64_t mbar[3];
    __shared__ uint32_t s_tmem;
    __shared__ int s_ok, s_chunk;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) lg_tmem_alloc(lg_smem_u32(&s_tmem), C::TMEM_COLS);
    if (tid == 0)
        for (int b = 0; b < 3; b++) lg_mbar_init(&mbar[b], 1);
    lg_tc_fence_before();
    __syncthreads();
    lg_tc_fence_after();
    const uint32_t tmem = s_tmem;
    const uint32_t idesc_a = lg_idesc_f16(128, C::NB);
    // the operands times 2^E (FP16 range), the products times 2^-2E
    const int ye = lg_f16_scale_exp(*ymax);
    const float ysc = lg_pow2f(ye), yunsc = lg_pow2f(-2 * ye);
    uint32_t ncommit[3] = {0u, 0u, 0u};
    bool pending[3] = {false, false, false};
    bool failed = false;

    // Bounded wait for the last commit on barrier b; one that runs out leaves
    // the commit pending for the drain (at most one commit per barrier is
    // outstanding, so the phase parity names it).
    auto wait_bar = [&](int b, uint32_t limit) -> bool {
        if (!pending[b]) return true;
        if (tid == 0) s_ok = lg_mbar_wait(&mbar[b], (ncommit[b] - 1u) & 1u, limit) ? 1 : 0;
        __syncthreads();
        const int ok = s_ok;
        __syncthreads();
        if (ok) pending[b] = false;
        return ok != 0;
    };

    for (;;) {
        if (tid == 0) {
            const unsigned long long q = atomicAdd(&counters[LG_CNT_QUEUE], 1ull);
            s_chunk = q < (unsigned long long)nchunks ? queue[q] : -1;
        }
        __syncthreads();
        const int ck = s_chunk;
        __syncthreads();
        if (ck < 0) break;
        // chunks are aligned to multiples of `chunk` in cube numbering; the
        // first and last chunk of a window may be partial
        const int64_t chunk_at = prm.cube0 / chunk * chunk + (int64_t)ck * chunk;
        const int cube_begin = (int)max(chunk_at, prm.cube0);
        const int cube_end = (int)min(ncubes, chunk_at + chunk);
        for (int cube = cube_begin; cube < cube_end; cube++) {
            const int64_t off = loff[cube];
            const int p = lcnt[cube];
            // rows K..127 and 128+K..TROWS-1 of both tiles stay zero
            for (int t = tid; t < 2 * C::TROWS * 8; t += kTB) {
                const int b = t / (C::TROWS * 8), rest = t % (C::TROWS * 8);
                const int r = rest / 8, c = rest % 8;
                if ((r >= K && r < 128) || r >= 128 + K)
                    *reinterpret_cast<uint4 *>(RA + b * C::TILE + lg_sw128_offset(r, c)) = make_uint4(0, 0, 0, 0);
            }
            const int nch = (p + CH - 1) / CH;
            // the FP32-pipe sums of this thread's conversion tasks (t = tid + i kTB:
            // column t % K, observations 8 (t / K) .. + 7 of every chunk)
            constexpr int NTASK = (K * 8 + kTB - 1) / kTB;
            float acc_g[NTASK], acc_d[NTASK];
#pragma unroll
            for (int i = 0; i < NTASK; i++) acc_g[i] = acc_d[i] = 0.0f;
            auto load_meta = [&](int x, int &gi, float2 &mf) {      // tid < CH
                const int o = x * CH + tid;
                if (x < nch && o < p) {
                    gi = lidx[off + o];
                    mf = lmeta[off + o];
                } else {
                    gi = -1;
                    mf = make_float2(0.0f, 0.0f);
                }
            };
            auto put_meta = [&](int x, int gi, float2 mf) {
                const int r = (x % 3) * CH + tid;
                mg_i[r] = gi;
                msq[r] = mf.x * ysc;
                me[r] = mf.y * ysc;
            };
            auto issue_rows = [&](int x) {
                float *st = (x & 1) ? stage1 : stage0;
                const int *gs = mg_i + (x % 3) * CH;
                constexpr int PPR = K / 4;
                for (int q = tid; q < CH * PPR; q += kTB) {
                    const int o = q / PPR, part = q % PPR;
                    const int gi = gs[o];
                    if (gi >= 0) cp_async16(lg_smem_u32(st + o * K + part * 4), ys32 + (int64_t)gi * K + part * 4);
                }
                cp_async_commit();
            };
            int pf_g = -1;
            float2 pf_m = make_float2(0.0f, 0.0f);
            if (nch > 0) {
                if (tid < CH) {
                    int g0, g1;
                    float2 m0, m1;
                    load_meta(0, g0, m0);
                    load_meta(1, g1, m1);
                    load_meta(2, pf_g, pf_m);
                    put_meta(0, g0, m0);
                    put_meta(1, g1, m1);
                }
                __syncthreads();
                issue_rows(0);
                issue_rows(1);
            }
            for (int ch = 0; ch < nch; ch++) {
                const int b = ch & 1;
                const float *st = b ? stage1 : stage0;
                const float *sq = msq + (ch % 3) * CH, *ev = me + (ch % 3) * CH;
                cp_async_wait<1>();
                __syncthreads();
                unsigned char *tile = RA + b * C::TILE;
                if (!wait_bar(b, prm.spin_limit)) {
                    failed = true;
                    break;
                }
                const int cnt = min(CH, p - ch * CH);
#pragma unroll
                for (int i = 0; i < NTASK; i++) {
                    const int t = tid + i * kTB;
                    if (t < K * 8) {
                        const int m = t % K, c = t / K;
                        float v[8];
                        uint4 hi, lo;
                        const float4 f0 = *reinterpret_cast<const float4 *>(sq + 8 * c);
                        const float4 f1 = *reinterpret_cast<const float4 *>(sq + 8 * c + 4);
                        const float4 e0 = *reinterpret_cast<const float4 *>(ev + 8 * c);
                        const float4 e1 = *reinterpret_cast<const float4 *>(ev + 8 * c + 4);
                        const float f[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
                        const float e[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
#pragma unroll
                        for (int j = 0; j < 8; j++) v[j] = (8 * c + j < cnt) ? st[(8 * c + j) * K + m] * f[j] : 0.0f;
                        split8_f16(v, hi, lo);
                        *reinterpret_cast<uint4 *>(tile + lg_sw128_offset(128 + m, c)) = hi;
                        *reinterpret_cast<uint4 *>(tile + lg_sw128_offset(m, c)) = lo;
                        // g and the diagonal (e is zero past the list's end)
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            acc_g[i] = fmaf(v[j], e[j], acc_g[i]);
                            acc_d[i] = fmaf(v[j], v[j], acc_d[i]);
                        }
                    }
                }
                lg_fence_async_smem();
                __syncthreads();
                if (ch > 0 && ch % LG_ACC_FLUSH == 0) {
                    // the last group's sums into the running ones in FP32 round to
                    // nearest (the first group's copied) before this chunk's
                    // products restart the scratch accumulators; chunk ch - 2's
                    // products were waited for above
                    if (!wait_bar(b ^ 1, prm.spin_limit)) {
                        failed = true;
                        break;
                    }
                    lg_tc_fence_after();
                    if (warp < 4) {
                        const uint32_t tl = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
                        for (int h = 0; h < 2; h++) {
                            const uint32_t base = tl + (h ? C::HI_COL : 0u);
#pragma unroll 1
                            for (int c0 = 0; c0 < K; c0 += 16) {
                                float v[16], u[16];
                                lg_tmem_ld16x2(base + C::ACC1 + (uint32_t)c0, base + (uint32_t)c0, v, u);
                                if (ch > LG_ACC_FLUSH) {
#pragma unroll
                                    for (int j = 0; j < 16; j++) v[j] = u[j] + v[j];
                                }
                                lg_tmem_st16(base + (uint32_t)c0, v);
                            }
                        }
                    }
                    lg_tc_fence_before();
                    __syncthreads();
                }
                if (tid == 0) {
                    lg_tc_fence_after();
                    const uint64_t dlo = lg_desc_sw128(lg_smem_u32(tile));
                    const uint64_t dhi = lg_desc_sw128(lg_smem_u32(tile + 128 * 128));   // Yhat_hi, e: A_hi and B
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {
                        const uint32_t acc = (ch % LG_ACC_FLUSH != 0 || kk > 0) ? 1u : 0u;
                        lg_umma_bf16(tmem + C::ACC1, dlo + 2 * kk, dhi + 2 * kk, idesc_a, acc);
                        lg_umma_bf16(tmem + C::HI_COL + C::ACC1, dhi + 2 * kk, dhi + 2 * kk, idesc_a, acc);
                    }
                    lg_umma_commit(&mbar[b]);
                }
                ncommit[b]++;
                pending[b] = true;
                if (tid < CH) {
                    put_meta(ch + 2, pf_g, pf_m);
                    load_meta(ch + 3, pf_g, pf_m);
                }
                __syncthreads();
                issue_rows(ch + 2);
            }
            cp_async_wait<0>();
            if (failed) break;
            // the task sums through the first gather stage (no copy in flight, its
            // rows read before the last chunk's barrier): [g | diag][task]
#pragma unroll
            for (int i = 0; i < NTASK; i++) {
                const int t = tid + i * kTB;
                if (t < K * 8) {
                    stage0[t] = acc_g[i];
                    stage0[K * 8 + t] = acc_d[i];
                }
            }
            if (!wait_bar(0, prm.spin_limit) || !wait_bar(1, prm.spin_limit)) {
                failed = true;
                break;
            }
            lg_tc_fence_after();
            __syncthreads();
            // g and diag(A) over the 8 observation groups in a fixed order, times
            // 2^-2E, in misc (before S, which overlaps the stage, is written)
            if (tid < K) {
                double sg = 0.0, sd = 0.0;
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    sg += (double)stage0[c * K + tid];
                    sd += (double)stage0[K * 8 + c * K + tid];
                }
                misc[tid] = sg * (double)yunsc;
                misc[K + tid] = sd * (double)yunsc;
            }
            __syncthreads();
            // A = 0.5 (S + S^T), S = HH + 2 LH; g
            float *S = reinterpret_cast<float *>(RA);
            if (warp < 4) {
                const int row = warp * 32 + lane;
                const uint32_t tl = tmem + ((uint32_t)(warp * 32) << 16);
                for (int c0 = 0; c0 < K; c0 += 16) {
                    float lo[16], hi[16];
                    if (p > 0) {
                        // the last group's sums, plus the running ones before it
                        float u[16];
                        lg_tmem_ld16x2(tl + C::ACC1 + (uint32_t)c0, tl + (uint32_t)c0, lo, u);
                        if (nch > LG_ACC_FLUSH) {
#pragma unroll
                            for (int j = 0; j < 16; j++) lo[j] = u[j] + lo[j];
                        }
                        lg_tmem_ld16x2(tl + C::HI_COL + C::ACC1 + (uint32_t)c0, tl + C::HI_COL + (uint32_t)c0, hi, u);
                        if (nch > LG_ACC_FLUSH) {
#pragma unroll
                            for (int j = 0; j < 16; j++) hi[j] = u[j] + hi[j];
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; j++) lo[j] = hi[j] = 0.0f;
                    }
                    if (row < K) {
#pragma unroll
                        for (int j = 0; j < 16; j++) S[row * C::LDS + c0 + j] = fmaf(2.0f, lo[j], hi[j]);
                    }
                }
            }
            lg_tc_fence_before();
            __syncthreads();
            float *Ac = mA + ((int64_t)cube - prm.cube0) * K * K;
            for (int idx = tid; idx < K * K; idx += kTB) {
                const int i = idx / K, j = idx % K;
                Ac[idx] = i == j ? (float)misc[K + i] : 0.5f * (S[i * C::LDS + j] + S[j * C::LDS + i]) * yunsc;
            }
            if (tid < K) mg[((int64_t)cube - prm.cube0) * K + tid] = misc[tid];
            __syncthreads();                                          // S is dead
        }
        if (failed) break;
    }
    if (failed && tid == 0) atomicOr(status, LG_ST_TIMEOUT);
    cp_async_wait<0>();
    // every committed MMA finishes before the TMEM is freed (at the normal
    // limit, whatever limit the run's waits had)
    bool drained = true;
    for (int b = 0; b < 3; b++) drained = wait_bar(b, LG_MBAR_SPIN_LIMIT) && drained;
    if (!drained && tid == 0) atomicOr(status, LG_ST_TIMEOUT);
    lg_tc_fence_before();
    __syncthreads();
    lg_tc_fence_after();
    if (warp == 0) lg_tmem_dealloc(tmem, C::TMEM_COLS);
}

// Launch 2: eigenpairs of A' = A + (k-1)/rho I, wbar and T for runs of LG_WARM_RUN
// cubes, a run per CTA at a time (each cube starts from the previous one's
// eigenvectors, the run's first from A' itself).  T (FP32) into mX, wbar over
// g in mg.  k = 96 on 128 threads, four CTAs per SM, or on 256, two per SM (the
// same results: lg_jacobi32b3): 128 issue fewer instructions, 256 end a run
// sooner.  Four warps per SM partition hide each other's shuffles and
// reciprocals; the matrix A stays in L2 and is read by rows.  28,800 cubes: 22.1 ms
// (35,000 cycles per problem and sweep on an SM, against 80,000 with one
// problem per SM).
template <int K, int T>
struct WECfg {
    // column strides that put the slots of a load phase on disjoint banks
    static constexpr int LDW = K == 96 && T == 256 ? K + 4 : K + 16;
    static constexpr int PER_SM = T == 128 ? 4 : 2;
    static constexpr size_t SMEM = sizeof(double) * 2 * K + sizeof(float) * ((size_t)K * LDW + 2 * K + 4 * K);
};

template <int K, int T>
__global__ void __launch_bounds__(T, WECfg<K, T>::PER_SM)
k_wide_eig(int64_t cube0, int64_t cube_end, double inflation, const float *__restrict__ mA, float *__restrict__ mX,
           double *__restrict__ mg, unsigned long long *__restrict__ counters)
{
    using C = WCfg<K>;
    constexpr int LDW = WECfg<K, T>::LDW, NW = T / 32, NCW = K / NW, NR = K / 32;
    extern __shared__ double smd[];
    double *wbar = smd, *gv = smd + K;
    float *W = reinterpret_cast<float *>(gv + K);            // columns; X after the solve
    float *il = W + K * LDW + 2 * K, *fs = il + K, *hc = fs + K, *rv = hc + K;
    __shared__ int s_rot;
    __shared__ int64_t s_run;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const double cdiag = (double)(K - 1) / inflation;
    const float cdiagf = (float)cdiag;
    const int64_t base = cube0 / LG_WARM_RUN * LG_WARM_RUN;
    const int64_t nruns = (cube_end - base + LG_WARM_RUN - 1) / LG_WARM_RUN;
    for (;;) {
        if (tid == 0) s_run = (int64_t)atomicAdd(&counters[LG_CNT_QUEUE], 1ull);
        __syncthreads();
        const int64_t run = s_run;
        __syncthreads();
        if (run >= nruns) break;
        const int64_t c0 = max(cube0, base + run * LG_WARM_RUN), c1 = min(cube_end, base + (run + 1) * LG_WARM_RUN);
        for (int64_t c = c0; c < c1; c++) {
            const float *Ac = mA + (c - cube0) * K * K;
            for (int i = tid; i < K; i += T) {
                gv[i] = mg[(c - cube0) * K + i];
                rv[i] = (float)gv[i];
            }
            if (c == c0) {
                // cold start: the Jacobi works on A' itself (symmetric: column j = row j)
                for (int idx = tid; idx < K * K; idx += T) {
                    const int j = idx / K, i = idx % K;
                    W[j * LDW + i] = Ac[idx] + (i == j ? cdiagf : 0.0f);
                }
            } else {
                // warm start: W = A' X = A X + (k-1)/rho X, NCW columns per warp, the
                // rows across the lanes
                float acc[NCW][NR];
#pragma unroll
                for (int a = 0; a < NCW; a++)
#pragma unroll
                    for (int q = 0; q < NR; q++) acc[a][q] = 0.0f;
                float *wc = W + warp * NCW * LDW;
#pragma unroll 1
                for (int l = 0; l < K; l += 4) {
                    float x[4][NR];
#pragma unroll
                    for (int e = 0; e < 4; e++)
#pragma unroll
                        for (int q = 0; q < NR; q++) x[e][q] = Ac[(l + e) * K + lane + 32 * q];
#pragma unroll
                    for (int a = 0; a < NCW; a++) {
                        const float4 y = *reinterpret_cast<const float4 *>(wc + a * LDW + l);
#pragma unroll
                        for (int q = 0; q < NR; q++) {
                            acc[a][q] = fmaf(x[0][q], y.x, acc[a][q]);
                            acc[a][q] = fmaf(x[1][q], y.y, acc[a][q]);
                            acc[a][q] = fmaf(x[2][q], y.z, acc[a][q]);
                            acc[a][q] = fmaf(x[3][q], y.w, acc[a][q]);
                        }
                    }
                }
                __syncwarp();                              // a column is read by its own warp only
#pragma unroll
                for (int a = 0; a < NCW; a++)
#pragma unroll
                    for (int q = 0; q < NR; q++) {
                        float *w = wc + a * LDW + lane + 32 * q;
                        *w = fmaf(cdiagf, *w, acc[a][q]);
                    }
            }
            // the next cube's A into L2 while this one is solved
            if (c + 1 < c1) {
                const char *nxt = reinterpret_cast<const char *>(Ac + K * K);
                for (int l = tid; l < K * K * 4 / 128; l += T)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(nxt + l * 128));
            }
            __syncthreads();
            int sw;
            if constexpr (K == 128)
                sw = lg_jacobi32b2<K, LDW, LDW>(W, W + K * LDW, &s_rot, LG_MIXED_JACOBI_TOL, 24);
            else
                sw = lg_jacobi32b3<K, LDW, LDW, T>(W, W + K * LDW, &s_rot, LG_MIXED_JACOBI_TOL, 24);
            if (tid == 0) {
                atomicMax(&counters[LG_CNT_MAXSWEEP], (unsigned long long)sw);
                atomicAdd(&counters[LG_CNT_SUMSWEEP], (unsigned long long)sw);
                if (sw > 24) atomicAdd(&counters[LG_CNT_NOTCONV], 1ull);
            }
            // lambda_j = |w_j|; x_j = w_j / lambda_j in its place
            for (int j = warp; j < K; j += NW) {
                float w[NR], s = 0.0f;
#pragma unroll
                for (int q = 0; q < NR; q++) {
                    w[q] = W[j * LDW + lane + 32 * q];
                    s = fmaf(w[q], w[q], s);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                const float lamf = sqrtf(s), inv = 1.0f / lamf;
#pragma unroll
                for (int q = 0; q < NR; q++) W[j * LDW + lane + 32 * q] = w[q] * inv;
                if (lane == 0) {
                    il[j] = inv;
                    fs[j] = sqrtf((float)(K - 1) / lamf);
                }
            }
            __syncthreads();
            if (warp == 0) {
                float lo = 3.0e38f, hi = 0.0f;
                for (int j = lane; j < K; j += 32) {
                    lo = fminf(lo, il[j]);
                    hi = fmaxf(hi, il[j]);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
                }
                if (lane == 0 && hi > 1.0e4f * lo) atomicAdd(&counters[LG_CNT_ILLCOND], 1ull);
            }
            // wbar = X diag(1/lambda) X^T g in FP32 and one refinement step
            for (int it = 0; it < 2; it++) {
                float r[NR];
#pragma unroll
                for (int q = 0; q < NR; q++) r[q] = rv[lane + 32 * q];
                for (int j = warp; j < K; j += NW) {
                    float d = 0.0f;
#pragma unroll
                    for (int q = 0; q < NR; q++) d = fmaf(W[j * LDW + lane + 32 * q], r[q], d);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
                    if (lane == 0) hc[j] = d * il[j];
                }
                __syncthreads();
                for (int i = tid; i < K; i += T) {
                    float a0 = 0.0f, a1 = 0.0f;
#pragma unroll 8
                    for (int j = 0; j < K; j += 2) {
                        a0 = fmaf(W[j * LDW + i], hc[j], a0);
                        a1 = fmaf(W[(j + 1) * LDW + i], hc[j + 1], a1);
                    }
                    wbar[i] = (it == 0 ? 0.0 : wbar[i]) + (double)(a0 + a1);
                }
                __syncthreads();
                if (it == 0) {
                    // residual g - A' wbar in FP64 (FP32 values of A converted on the
                    // integer pipe), four rows per warp at a time: the sums over the
                    // lanes fold two rows into one value per step
                    double wl[NR];
#pragma unroll
                    for (int q = 0; q < NR; q++) wl[q] = wbar[lane + 32 * q];
#pragma unroll 1
                    for (int i0 = 4 * warp; i0 < K; i0 += 4 * NW) {
                        double d[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            d[e] = 0.0;
#pragma unroll
                            for (int q = 0; q < NR; q++)
                                d[e] = fma(lg_f2d_bits(Ac[(i0 + e) * K + lane + 32 * q]), wl[q], d[e]);
                        }
                        const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
                        const double k0 = h16 ? d[2] : d[0], k1 = h16 ? d[3] : d[1];
                        const double s0 = h16 ? d[0] : d[2], s1 = h16 ? d[1] : d[3];
                        const double e0 = k0 + __shfl_xor_sync(0xffffffffu, s0, 16);
                        const double e1 = k1 + __shfl_xor_sync(0xffffffffu, s1, 16);
                        double v = (h8 ? e1 : e0) + __shfl_xor_sync(0xffffffffu, h8 ? e0 : e1, 8);
#pragma unroll
                        for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                        const int i = i0 + (h16 ? 2 : 0) + (h8 ? 1 : 0);
                        if ((lane & 7) == 0) rv[i] = (float)(gv[i] - (v + cdiag * wbar[i]));
                    }
                    __syncthreads();
                }
            }
            for (int i = tid; i < K; i += T) mg[(c - cube0) * K + i] = wbar[i];
            // T = X diag(f) X^T, 4x4 tiles of the lower triangle
            float *Tc = mX + (c - cube0) * K * K;
#pragma unroll 1
            for (int b = tid; b < C::NLOW; b += T) {
                int bi, bj;
                lg_decode_block(b, bi, bj);
                float t[4][4];
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int jj = 0; jj < 4; jj++) t[i][jj] = 0.0f;
#pragma unroll 4
                for (int j = 0; j < K; j++) {
                    const float f = fs[j];
                    const float4 av = *reinterpret_cast<const float4 *>(W + j * LDW + 4 * bi);
                    const float4 bv = *reinterpret_cast<const float4 *>(W + j * LDW + 4 * bj);
                    const float a[4] = {av.x, av.y, av.z, av.w};
                    const float bq[4] = {bv.x * f, bv.y * f, bv.z * f, bv.w * f};
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int jj = 0; jj < 4; jj++) t[i][jj] = fmaf(a[i], bq[jj], t[i][jj]);
                }
                if (bi == bj) {
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int jj = i + 1; jj < 4; jj++) t[i][jj] = t[jj][i];
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    *reinterpret_cast<float4 *>(Tc + (4 * bi + i) * K + 4 * bj) = make_float4(t[i][0], t[i][1], t[i][2], t[i][3]);
                    if (bi != bj)
                        *reinterpret_cast<float4 *>(Tc + (4 * bj + i) * K + 4 * bi) = make_float4(t[0][i], t[1][i], t[2][i], t[3][i]);
                }
            }
            __syncthreads();
        }
    }
}

// Launch 3: xa = xb^T (T + wbar 1^T) from T in mX and wbar in mg.
template <int K>
__global__ void __launch_bounds__(kTW, WCfg<K>::PER_SM_U)
k_wide_update(LgGrid g, LgParams prm, const int *__restrict__ queue, int nchunks, int chunk, int64_t ncubes,
              const double *__restrict__ xb, const double *__restrict__ axb, double *__restrict__ xa,
              double *__restrict__ axa, double *__restrict__ trans_out, double *__restrict__ w_out,
              const float *__restrict__ mX, const double *__restrict__ mg, unsigned long long *__restrict__ counters,
              unsigned *__restrict__ status)
{
    using C = WCfg<K>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *tb = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *xt = tb + C::UT * C::TBSUB;
    double *wbar = reinterpret_cast<double *>(xt + C::UT * 16384);
    double *inc = wbar + K;                                    // 128
    __shared__ uint64_t mbar[3];
    __shared__ uint32_t s_tmem;
    __shared__ int s_ok, s_chunk;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) lg_tmem_alloc(lg_smem_u32(&s_tmem), 128);
    if (tid == 0)
        for (int b = 0; b < 3; b++) lg_mbar_init(&mbar[b], 1);
    lg_tc_fence_before();
    __syncthreads();
    lg_tc_fence_after();
    const uint32_t tmem = s_tmem;
    const uint32_t idesc_u = lg_idesc_bf16(128, K);
    uint32_t ncommit[3] = {0u, 0u, 0u};
    bool pending[3] = {false, false, false};
    bool failed = false;

    // Bounded wait for the last commit on barrier b; one that runs out leaves
    // the commit pending for the drain (at most one commit per barrier is
    // outstanding, so the phase parity names it).
    auto wait_bar = [&](int b, uint32_t limit) -> bool {
        if (!pending[b]) return true;
        if (tid == 0) s_ok = lg_mbar_wait(&mbar[b], (ncommit[b] - 1u) & 1u, limit) ? 1 : 0;
        __syncthreads();
        const int ok = s_ok;
        __syncthreads();
        if (ok) pending[b] = false;
        return ok != 0;
    };

    for (;;) {
        if (tid == 0) {
            const unsigned long long q = atomicAdd(&counters[LG_CNT_QUEUE], 1ull);
            s_chunk = q < (unsigned long long)nchunks ? queue[q] : -1;
        }
        __syncthreads();
        const int ck = s_chunk;
        __syncthreads();
        if (ck < 0) break;
        // chunks are aligned to multiples of `chunk` in cube numbering; the
        // first and last chunk of a window may be partial
        const int64_t chunk_at = prm.cube0 / chunk * chunk + (int64_t)ck * chunk;
        const int cube_begin = (int)max(chunk_at, prm.cube0);
        const int cube_end = (int)min(ncubes, chunk_at + chunk);
        for (int cube = cube_begin; cube < cube_end; cube++) {
            const float *Tc = mX + ((int64_t)cube - prm.cube0) * K * K;
            const double *wb = mg + ((int64_t)cube - prm.cube0) * K;
            if (trans_out) {
                for (int idx = tid; idx < K * K; idx += kTW)
                    trans_out[(int64_t)cube * K * K + idx] = (double)Tc[idx] + wb[idx % K];     // T is symmetric
                if (tid < K) w_out[(int64_t)cube * K + tid] = wb[tid];
            }
            // the member mean of xb^T T is sqrt(rho) xbar (T 1 = sqrt(rho) 1): the
            // FP64 increment takes it, xb^T (wbar + sqrt(rho)/k 1), not the tensor
            // products (as in the narrow core)
            if (tid < K) wbar[tid] = wb[tid] + sqrt(prm.inflation) / (double)K;
            __syncthreads();
            // T tiles (B operand, N = K rows) along members: hi tiles 0, 1 then lo tiles 0, 1
            for (int t = tid; t < K * (K / 8); t += kTW) {
                const int e = t / (K / 8), cg = t % (K / 8), s = cg / 8, c = cg % 8;
                float v[8];
                *reinterpret_cast<float4 *>(v) = *reinterpret_cast<const float4 *>(Tc + e * K + 8 * cg);
                *reinterpret_cast<float4 *>(v + 4) = *reinterpret_cast<const float4 *>(Tc + e * K + 8 * cg + 4);
                uint4 hi, lo;
                split8(v, hi, lo);
                *reinterpret_cast<uint4 *>(tb + C::utile(0, s) * C::TBSUB + lg_sw128_offset(e, C::uchunk(0, s, c))) = hi;
                *reinterpret_cast<uint4 *>(tb + C::utile(1, s) * C::TBSUB + lg_sw128_offset(e, C::uchunk(1, s, c))) = lo;
            }
            const int n = g.n;
            const int bjc = (int)(cube % prm.nbj), bic = (int)(cube / prm.nbj);
            const int sj = bjc * prm.cube_n, ej = min(sj + prm.cube_n - 1, g.nlat - 1);
            const int si = bic * prm.cube_n, ei = min(si + prm.cube_n - 1, g.nlon - 1);
            for (int ii = si; ii <= ei && !failed; ii++)
                for (int jj = sj; jj <= ej && !failed; jj++) {
                    const int64_t col = jj + (int64_t)g.nlat * ii;
                    const double *xbc = xb + col * n * K;
                    double *xac = xa + col * n * K;
                    for (int r0 = 0; r0 < n; r0 += 128) {
                        const int R = min(128, n - r0);
                        for (int t = tid; t < 128 * (K / 8); t += kTW) {
                            const int r = t / (K / 8), cg = t % (K / 8), s = cg / 8, c = cg % 8;
                            float v[8];
                            if (r < R) {
                                const double2 *src =
                                    reinterpret_cast<const double2 *>(xbc + (int64_t)(r0 + r) * K + 8 * cg);
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    const double2 q = src[j];
                                    v[2 * j] = (float)q.x;
                                    v[2 * j + 1] = (float)q.y;
                                }
                            } else {
#pragma unroll
                                for (int j = 0; j < 8; j++) v[j] = 0.0f;
                            }
                            uint4 hi, lo;
                            split8(v, hi, lo);
                            *reinterpret_cast<uint4 *>(xt + C::utile(0, s) * 16384 + lg_sw128_offset(r, C::uchunk(0, s, c))) = hi;
                            *reinterpret_cast<uint4 *>(xt + C::utile(1, s) * 16384 + lg_sw128_offset(r, C::uchunk(1, s, c))) = lo;
                        }
                        for (int r = warp; r < R; r += kTW / 32) {
                            const double *src = xbc + (int64_t)(r0 + r) * K;
                            double s = 0.0;
                            for (int i = lane; i < K; i += 32) s += src[i] * wbar[i];
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                            if (lane == 0) inc[r] = s;
                        }
                        lg_fence_async_smem();
                        __syncthreads();
                        if (tid == 0) {
                            lg_tc_fence_after();
#pragma unroll
                            for (int kk = 0; kk < K / 16; kk++) {
                                const int s = kk / 4, k4 = kk % 4;
                                const int kh = k4 + C::uchunk(0, s, 0) / 2, kl = k4 + C::uchunk(1, s, 0) / 2;
                                const uint64_t dh = lg_desc_sw128(lg_smem_u32(xt + C::utile(0, s) * 16384)) + 2 * kh;
                                const uint64_t dl = lg_desc_sw128(lg_smem_u32(xt + C::utile(1, s) * 16384)) + 2 * kl;
                                const uint64_t th = lg_desc_sw128(lg_smem_u32(tb + C::utile(0, s) * C::TBSUB)) + 2 * kh;
                                const uint64_t tl = lg_desc_sw128(lg_smem_u32(tb + C::utile(1, s) * C::TBSUB)) + 2 * kl;
                                lg_umma_bf16(tmem, dh, th, idesc_u, kk > 0 ? 1u : 0u);
                                lg_umma_bf16(tmem, dh, tl, idesc_u, 1u);
                                lg_umma_bf16(tmem, dl, th, idesc_u, 1u);
                            }
                            lg_umma_commit(&mbar[2]);
                        }
                        ncommit[2]++;
                        pending[2] = true;
                        if (!wait_bar(2, prm.spin_limit)) {
                            failed = true;
                            break;
                        }
                        lg_tc_fence_after();
                        if (warp < 4) {
                            const int r = warp * 32 + lane;
                            const uint32_t tl = tmem + ((uint32_t)(warp * 32) << 16);
                            // member mean and perturbations in FP32 (the products are
                            // FP32 sums of BF16 hi/lo terms), written as FP64 with the
                            // conversion on the integer pipe
                            float part[8];
#pragma unroll
                            for (int q = 0; q < 8; q++) part[q] = 0.0f;
                            for (int c0 = 0; c0 < K; c0 += 16) {
                                float v[16];
                                lg_tmem_ld16(tl + (uint32_t)c0, v);
#pragma unroll
                                for (int e = 0; e < 16; e++) part[e & 7] += v[e];
                            }
                            const float meanf =
                                (((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]))) /
                                (float)K;
                            if (r < R) {
                                const int64_t row = col * n + r0 + r;
                                axa[row] = axb[row] + inc[r];
                            }
                            double *dst = xac + (int64_t)(r0 + r) * K;
                            for (int c0 = 0; c0 < K; c0 += 16) {
                                float v[16];
                                lg_tmem_ld16(tl + (uint32_t)c0, v);
                                if (r < R) {
#pragma unroll
                                    for (int e = 0; e < 16; e += 2)
                                        *reinterpret_cast<double2 *>(dst + c0 + e) =
                                            make_double2(lg_f2d_bits(v[e] - meanf), lg_f2d_bits(v[e + 1] - meanf));
                                }
                            }
                        }
                        lg_tc_fence_before();
                        __syncthreads();
                    }
                }
            if (failed) break;
            __syncthreads();
        }
        if (failed) break;
    }
    if (failed && tid == 0) atomicOr(status, LG_ST_TIMEOUT);
    // every committed MMA finishes before the TMEM is freed (at the normal
    // limit, whatever limit the run's waits had)
    bool drained = true;
    for (int b = 0; b < 3; b++) drained = wait_bar(b, LG_MBAR_SPIN_LIMIT) && drained;
    if (!drained && tid == 0) atomicOr(status, LG_ST_TIMEOUT);
    lg_tc_fence_before();
    __syncthreads();
    lg_tc_fence_after();
    if (warp == 0) lg_tmem_dealloc(tmem, 128);
}

// Cubes one launch sequence holds intermediates for (A and T: 8 k^2 bytes per cube),
// a multiple of every chunk; a device that cannot give that takes smaller
// blocks.
constexpr int64_t kWideCubes = 1 << 15;

template <int K, int T>
cudaError_t launch_eig(letkf_ctx *ctx, int64_t b0, int64_t b1, int64_t runs, int nsm)
{
    using E = WECfg<K, T>;
    const cudaError_t e = cudaFuncSetAttribute(k_wide_eig<K, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)E::SMEM);
    if (e != cudaSuccess) return e;
    lg_count_launch();
    k_wide_eig<K, T><<<(unsigned)std::min<int64_t>(runs, (int64_t)nsm * E::PER_SM), T, E::SMEM, ctx->stream>>>(
        b0, b1, ctx->params.inflation, ctx->d_mA.p, ctx->d_mX.p, ctx->d_mg.p, ctx->d_counters.p);
    return cudaGetLastError();
}

template <int K>
cudaError_t launch_wide(letkf_ctx *ctx, const LgGrid &g, const double *xb, const double *axb, double *xa,
                        double *axa, double *trans_out, double *w_out)
{
    using C = WCfg<K>;
    if (ctx->win1 <= ctx->win0) return cudaSuccess;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(k_wide_build<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM_A)) !=
        cudaSuccess)
        return e;
    if ((e = cudaFuncSetAttribute(k_wide_update<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM_U)) !=
        cudaSuccess)
        return e;
    const int64_t w0 = ctx->win0, w1 = ctx->win1, unit = lg_run_chunk(ctx);
    // blocks end at multiples of `step` in cube numbering, so the runs, the
    // chunks and the results do not depend on the blocking
    int64_t step = std::max(kWideCubes, unit);
    auto block_end = [&](int64_t b) { return std::min(w1, (b / step + 1) * step); };
    // larger blocks than what is held only where the device has room for them: one
    // that is short of memory keeps its buffers from run to run
    const size_t kk = (size_t)K * K, cube_bytes = 2 * kk * sizeof(float) + K * sizeof(double);
    const int64_t held = (int64_t)std::min(std::min(ctx->d_mA.n, ctx->d_mX.n) / kk, ctx->d_mg.n / K);
    size_t fr = 0, tot = 0;
    if (std::min(step, w1 - w0) > held && cudaMemGetInfo(&fr, &tot) == cudaSuccess)
        while (step > unit && std::min(step, w1 - w0) > held &&
               (size_t)std::min(step, w1 - w0) * cube_bytes > fr + (size_t)held * cube_bytes)
            step /= 2;
    for (;; step /= 2) {
        const size_t most = (size_t)std::min(step, w1 - w0);
        e = ctx->d_mA.reserve(most * K * K);
        if (e == cudaSuccess) e = ctx->d_mX.reserve(most * K * K);
        if (e == cudaSuccess) e = ctx->d_mg.reserve(most * K);
        if (e != cudaErrorMemoryAllocation || step <= unit) break;
        cudaGetLastError();
        ctx->d_mA.release();
        ctx->d_mX.release();
    }
    for (int64_t b0 = w0, b1; b0 < w1 && e == cudaSuccess; b0 = b1) {
        b1 = block_end(b0);
        ctx->win0 = b0;
        ctx->win1 = b1;
        int chunk = 0, nchunks = 0;
        if ((e = lg_build_chunk_queue(ctx, chunk, nchunks)) != cudaSuccess) break;
        // persistent grids; the CTAs take chunks (runs) with the queue cursor
        const unsigned blocks = (unsigned)(nchunks < nsm ? nchunks : nsm);
        auto rewind = [&] {
            return cudaMemsetAsync(ctx->d_counters.p + LG_CNT_QUEUE, 0, sizeof(unsigned long long), ctx->stream);
        };
        const LgParams prm = lg_params(ctx);
        if ((e = rewind()) != cudaSuccess) break;
        lg_count_launch();
        k_wide_build<K><<<blocks, kTB, C::SMEM_A, ctx->stream>>>(
            prm, ctx->d_ys32.p, ctx->d_lidx.p, ctx->d_lmeta.p, ctx->d_queue.p, nchunks, chunk, ctx->d_loff.p,
            ctx->d_lcnt.p, b1, ctx->d_mA.p, ctx->d_mg.p, ctx->d_counters.p, ctx->d_status.p, ctx->d_ymax.p);
        if ((e = cudaGetLastError()) != cudaSuccess) break;
        if ((e = rewind()) != cudaSuccess) break;
        const int64_t runs = (b1 - b0 / LG_WARM_RUN * LG_WARM_RUN + LG_WARM_RUN - 1) / LG_WARM_RUN;
        // up to two runs per SM the launch lasts as long as a run, and 256 threads
        // end it sooner (k = 96, 1,800 cubes: 4.05 against 4.55 ms, 4,050: 5.71
        // against 5.80); beyond, 128 threads (5,832 cubes: 7.15 against 8.10 ms,
        // 16,200: 13.9 against 15.9)
        if (K == 96 && runs > 2 * nsm) e = launch_eig<K, K == 96 ? 128 : 256>(ctx, b0, b1, runs, nsm);
        else e = launch_eig<K, 256>(ctx, b0, b1, runs, nsm);
        if (e != cudaSuccess) break;
        if ((e = rewind()) != cudaSuccess) break;
        lg_count_launch();
        k_wide_update<K><<<(unsigned)std::min(nchunks, C::PER_SM_U * nsm), kTW, C::SMEM_U, ctx->stream>>>(
            g, prm, ctx->d_queue.p, nchunks, chunk, b1, xb, axb, xa, axa, trans_out, w_out, ctx->d_mX.p, ctx->d_mg.p,
            ctx->d_counters.p, ctx->d_status.p);
        e = cudaGetLastError();
    }
    ctx->win0 = w0;
    ctx->win1 = w1;
    return e;
}

}  // namespace

size_t lg_wide_scratch_bytes(const letkf_ctx *ctx)
{
    if (ctx->k <= 64) return 0;
    const size_t n = (size_t)std::min<int64_t>(ctx->range1 - ctx->range0, kWideCubes) * ctx->k;
    const size_t want = n * (2 * ctx->k * sizeof(float) + sizeof(double));
    const size_t held = (ctx->d_mA.n + ctx->d_mX.n) * sizeof(float) + ctx->d_mg.n * sizeof(double);
    return want > held ? want - held : 0;
}

cudaError_t lg_launch_core_mixed_wide(letkf_ctx *ctx, const LgGrid &g, const double *xb, const double *axb,
                                      double *xa, double *axa, double *trans_out, double *w_out)
{
    switch (g.k) {
    case 96: return launch_wide<96>(ctx, g, xb, axb, xa, axa, trans_out, w_out);
    case 128: return launch_wide<128>(ctx, g, xb, axb, xa, axa, trans_out, w_out);
    default: return cudaErrorInvalidValue;
    }
}
