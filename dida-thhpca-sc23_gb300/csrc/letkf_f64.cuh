// letkf_f64.cuh -- what the kernels of the FP64 form's tensor-core path share
// (letkf_f64.cu: ensembles of 32, 48, 64; letkf_f64_wide.cu: 96 and 128).
#pragma once

#include "letkf_internal.cuh"
#include "letkf_fixed.cuh"

namespace {

constexpr int kTF = 512;                  // threads of the kernels below
constexpr int kMaxIter = 8;               // most corrections of T

// Storage size of a problem's k x k matrices between the launches.
__host__ __device__ constexpr int store_size(int k) { return k <= 32 ? 32 : k <= 64 ? 64 : k; }

// Scratch counters: the eigensolve's (LG_CNT_*), then these.
enum { F64_QUEUE = LG_CNT_N, F64_NLIST, F64_CNT_N };

}  // namespace

// One block of problems: problems q0 .. q0 + nq - 1, problem q being level
// block q % nvb of cube q / nvb; the arrays are indexed by q - q0.
struct LgF64Block {
    int64_t q0;
    int nq, nvb;
    // matrices of ks x ks and vectors of ks (store_size), zero past the ensemble
    long long *A;              // integers: A / 2^ea, later T' 2^sT
    int *ea;
    float *A32, *X, *lam;      // A, its eigenvectors (by column) and eigenvalues
    double *g;                 // g, later u
    float *amax;               // largest diagonal element of A'
    int *flag, *list;          // 1: solved by k_core_fp64; the flagged problems
    unsigned long long *cnt;   // F64_CNT_N counters
    const float *rowmax;       // largest |element| of every row of y
};

namespace {

using Block = LgF64Block;

__device__ __forceinline__ void fall_back(const Block &B, int q)
{
    if (atomicExch(&B.flag[q], 1) == 0) B.list[atomicAdd(&B.cnt[F64_NLIST], 1ull)] = q;
}

// 16-byte cp.async, zero-filled when !valid.
__device__ __forceinline__ void cp_async16_z(uint32_t dst, const void *src, bool valid)
{
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// One problem's list of observations, as the A builds read it.
struct ListSrc {
    const LgRowSrc &src;
    const float *rowmax;       // largest |element| of every row of y
    int64_t off;
    int p;
    bool vertical;             // weights times the factor of the ln-p distance
    double lnp, vert_dist;
    int gcv;
    // entry x: row of y (-1 past the end), sqrt(rdiaginv rloc) (rrloc,
    // letkf_core.F90:64-66), its product with dep, the row's largest |element|
    __device__ __forceinline__ void entry(int x, int64_t &gi, double &s, double &sd, float &rm) const
    {
        gi = -1;
        s = sd = 0.0;
        rm = 0.0f;
        if (x >= p) return;
        const int64_t li = off + x;
        gi = src.batch ? li : (int64_t)src.lidx[li];
        double rl = src.batch ? src.brloc[li] : src.lrloc[li];
        const float rd = src.batch ? src.brdi[li] : src.rinvf[gi];
        const double d = src.batch ? src.bdep[li] : src.dep[gi];
        rm = rowmax[gi];
        if (vertical) {
            const double z = fabs(lnp - src.olnp[gi]) / vert_dist;
            rl = rl * (gcv ? lg_schr2(z) : lg_schr(z));
        }
        s = sqrt((double)rd * rl);
        sd = s * d;
    }
};

// The fixed point of a list: Yhat 2^sY and e 2^sE rounded to integers, sums of
// products in units of 2^sh of level 5 (A) and 2^shG (g).
struct ListScale {
    int sY, sE, sh, shG;
    bool pairs;                // the first digits' squares over any 128 observations stay below 2^24
    bool bad;                  // not finite, or out of range
};

// Scales from bounds over the whole list: the largest |Yhat| and |e|, and the
// sums of squares of e and of the rows' largest |Yhat| over the list and over
// every group of 128 observations (what two chunks sum); thread t < first brings
// entry t, the others are read here (a vertical weight from FP32, rounded up).
// wm: 6 x 16 words of shared memory.  Called by all kTF threads.
__device__ __forceinline__ ListScale list_scale(const ListSrc &L, int first, double e_s, double e_sd, float e_rm,
                                                unsigned (*wm)[kTF / 32])
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const LgRowSrc &src = L.src;
    const float y0 = e_rm * (__double2float_ru(e_s) * 1.0001f), d0 = __double2float_ru(fabs(e_sd));
    unsigned my = __float_as_uint(y0) & 0x7fffffffu, me = __float_as_uint(d0) & 0x7fffffffu;
    auto warp_sum = [](float x) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        return x;
    };
    // a warp's 32 entries are a quarter of a group; `first` and kTF are whole
    // groups, so warps 4 g .. 4 g + 3 always share one: the largest sums of
    // each warp bound every group's
    float sq = warp_sum(y0 * y0), se = warp_sum(d0 * d0), gq = sq, ge = se;
    for (int i0 = first + 32 * warp; i0 < L.p; i0 += kTF) {
        float y = 0.0f, d = 0.0f;
        if (i0 + lane < L.p) {
            const int64_t li = L.off + i0 + lane;
            const int64_t gi = src.batch ? li : (int64_t)src.lidx[li];
            const float rd = src.batch ? src.brdi[li] : src.rinvf[gi];
            float rl = (float)(src.batch ? src.brloc[li] : src.lrloc[li]);
            if (L.vertical) {
                const float z = (float)(fabs(L.lnp - src.olnp[gi]) / L.vert_dist);
                // (FP32 next to the cut-off is good to 1e-6 of the weight at zero)
                rl *= L.gcv ? lg_schr2f(z) + 4e-6f : z > 2.0001f ? 0.0f : 1.0f;
            }
            const float s = sqrtf(rd) * sqrtf(rl) * 1.0001f;
            d = fabsf((float)(src.batch ? src.bdep[li] : src.dep[gi])) * s;
            y = L.rowmax[gi] * s;
        }
        my = max(my, __float_as_uint(y) & 0x7fffffffu);
        me = max(me, __float_as_uint(d) & 0x7fffffffu);
        const float wq = warp_sum(y * y), we = warp_sum(d * d);
        sq += wq;
        se += we;
        gq = fmaxf(gq, wq);
        ge = fmaxf(ge, we);
    }
    my = __reduce_max_sync(0xffffffffu, my);
    me = __reduce_max_sync(0xffffffffu, me);
    if (lane == 0) {
        wm[0][warp] = my;
        wm[1][warp] = me;
        wm[2][warp] = __float_as_uint(sq);
        wm[3][warp] = __float_as_uint(se);
        wm[4][warp] = __float_as_uint(gq);
        wm[5][warp] = __float_as_uint(ge);
    }
    __syncthreads();
    sq = se = gq = ge = 0.0f;
#pragma unroll
    for (int g = 0; g < kTF / 128; g++) {
        float a = 0.0f, b = 0.0f;
#pragma unroll
        for (int i = 4 * g; i < 4 * g + 4; i++) {
            my = max(my, wm[0][i]);
            me = max(me, wm[1][i]);
            sq += __uint_as_float(wm[2][i]);
            se += __uint_as_float(wm[3][i]);
            a += __uint_as_float(wm[4][i]);
            b += __uint_as_float(wm[5][i]);
        }
        gq = fmaxf(gq, a);
        ge = fmaxf(ge, b);
    }
    ListScale r;
    // the sums of squares in units of the largest (the worst case where FP32
    // cannot hold them)
    const float mf = __uint_as_float(my), mef = __uint_as_float(me), n = (float)L.p;
    auto units = [](float sum, float most, float worst) {
        const float u = 1.001f * (sum / most) / most;
        return u < worst && most >= 1e-15f ? u : worst;
    };
    const float ratio = units(sq, mf, n), ratio_e = units(se, mef, n);
    const float group = units(gq, mf, 128.0f), group_e = units(ge, mef, 128.0f);
    // first digits of at most 512; with at most 16 units in any 128 observations
    // they may have one bit more (their squares then stay below 2^24), with more
    // than 64 they are summed 64 observations at a time
    const int more = group <= 15.9f ? 1 : 0, more_e = group_e <= 15.9f ? 1 : 0;
    r.pairs = group <= 63.0f && group_e <= 63.0f;
    r.sY = 48 + more - lg_exp2f_bits(__float_as_uint(mf * 1.01f));
    r.sE = 48 + more_e - lg_exp2f_bits(__float_as_uint(mef * 1.01f));
    // A <= ratio 2^(98 + 2 more): 2 A 2^-(30 + sh) < 2^61
    r.sh = 8 + 2 * more + max(1, lg_exp2f_bits(__float_as_uint(fmaxf(ratio, 1.0f))) + 1);
    // |g| <= sqrt(ratio ratio_e) 2^(98 + more + more_e) (Cauchy-Schwarz): a few
    // strong rows among many weak ones have a small ratio of Yhat beside a large
    // one of e, and g needs more room than A's unit leaves
    const float rg = sqrtf(fmaxf(ratio, 1.0f)) * sqrtf(fmaxf(ratio_e, 1.0f)) * 1.001f;
    r.shG = 8 + more + more_e + max(1, lg_exp2f_bits(__float_as_uint(rg)) + 1);
    r.bad = my >= 0x7e000000u || me >= 0x7e000000u || r.sh > 30 || r.shG > 30;
    return r;
}

// s 2^e by the exponent (s is zero or normal, and so is s 2^e).
__device__ __forceinline__ double scale_exp(double s, int e)
{
    return s == 0.0 ? 0.0 : __hiloint2double(__double2hiint(s) + (e << 20), __double2loint(s));
}

}  // namespace

// The launches of one block of problems for ensembles of 96 and 128
// (letkf_f64_wide.cu); scratch: lg_f64w_scratch(k) 64-bit words per CTA.
size_t lg_f64w_scratch(int k);
cudaError_t lg_f64w_block(letkf_ctx *ctx, const LgGrid &g, const LgParams &prm, const LgRowSrc &src,
                          const LgF64Block &B, const int64_t *loff, const int32_t *lcnt, const double *xb,
                          const double *axb, double *xa, double *axa, double *trans_out, double *w_out, int nsm,
                          long long *scratch);
