// Balloon-Windkessel BOLD model for data assimilation: the step after the hot
// path in DA_voxel.py (voxel activity -> BOLD signal, data_assimilation/DA_voxel.py:314-331).
//
// The reference advances models/bold_model_pytorch.py:61-96 (BOLD.run) once
// per simulated step as ~20 separate tensor operations.  Here one thread owns
// one voxel's state (s, q, v, f_in) in registers for a whole window of steps:
// one launch per window, the activity streamed in and the signal streamed out
// with coalesced loads and stores.  Arithmetic follows BOLD.run in float32 and
// in its order: q, v, f_in, s are advanced in place in that order (q reads the
// old v and f_in, f_in the old s, the output the new q and v); divisions by
// parameters are correctly rounded divisions; x ** y is powf.  Parameters are
// Python floats in the reference, so every parameter expression is evaluated
// in double on the host and rounded to float32 once.
#include <cmath>

#include "dtb_engine.h"

namespace dtb {

struct BoldConst {
    float eps, tao_s, tao_f, tao_0, e0, v0, dt;
    float one_m_e0, div_alpha, div_alpha_m1, seven_e0, e0_term;
};

// Steps taken together.  A step is four recurrences of very different weight: (s, f_in) needs
// two divisions, v a power, q two powers and three divisions, and only v's and q's last
// operations wait for the step before.  One warp per scheduler is all a DA window fills (23,000
// voxels are 719 warps for 592 schedulers), so a step-by-step loop waits for each power in turn;
// kBoldSteps steps side by side keep that many of them in flight.
constexpr int kBoldSteps = 4;
constexpr int kBoldThreads = 64;    // small blocks spread a window's few warps evenly over the SMs
// Largest 1/alpha taken by products.  x^n has up to n - 1 roundings, over [0.5, 2] at most 3.3 ulp
// for n = 6, 4.5 for 8 and 10.9 for 15 and 16 (powf is documented with 4), but they do not reach the
// window: its output, q and v after 800 steps of 20,000 voxels lie as far from 64 bits with products
// as with powf for every n up to here (2.06e-7 to 2.24e-7, n = 5 2.13e-7 both, n = 16 2.15e-7 and
// 2.16e-7), the steps' own float32 sums being what sets the distance.
constexpr int kBoldMostWhole = 16;

// x^n by squaring for the whole exponent n >= 1 (uniform over the grid).
__device__ __forceinline__ float pow_whole(float x, int n) {
    float r = 1.0f, b = x;
    bool first = true;
    for (; n; n >>= 1) {
        if (n & 1) {
            r = first ? b : __fmul_rn(r, b);
            first = false;
        }
        if (n > 1) b = __fmul_rn(b, b);
    }
    return r;
}

// v^(1/alpha - 1) and v^(1/alpha).  WHOLE: 1/alpha is the whole number `whole` (5 for the default
// alpha of 0.2), up to kBoldMostWhole; the powers are then products, without the ~100 instructions
// that a powf costs the critical path.
template <bool WHOLE>
__device__ __forceinline__ void bold_powers(const BoldConst& c, int whole, float v, float& pm1, float& p) {
    if constexpr (WHOLE) {
        pm1 = whole > 1 ? pow_whole(v, whole - 1) : 1.0f;
        p = whole > 1 ? __fmul_rn(pm1, v) : v;
    } else {
        pm1 = powf(v, c.div_alpha_m1);
        p = powf(v, c.div_alpha);
    }
}

// N steps from step k on.
template <bool WHOLE, int N>
__device__ __forceinline__ void bold_steps(const BoldConst& c, int whole, uint32_t n, uint32_t i, uint32_t k,
                                           const float* __restrict__ u, float* __restrict__ out, float& s, float& q, float& v,
                                           float& f) {
    float uk[N], fk[N], fq[N], pm1[N], vn[N];
#pragma unroll
    for (int j = 0; j < N; ++j) uk[j] = __ldcs(u + static_cast<size_t>(k + j) * n + i);
    // s and f_in: d_s = epsilon * u - s / tao_s - (f_in - 1) / tao_f
#pragma unroll
    for (int j = 0; j < N; ++j) {
        fk[j] = f;
        const float d_s = __fsub_rn(__fsub_rn(__fmul_rn(c.eps, uk[j]), __fdiv_rn(s, c.tao_s)),
                                    __fdiv_rn(__fsub_rn(f, 1.0f), c.tao_f));
        f = __fadd_rn(f, __fmul_rn(s, c.dt));
        f = f > 0.0f ? f : 0.0f;
        s = __fadd_rn(s, __fmul_rn(d_s, c.dt));
    }
    // f_in * q_part / E_0, q_part = 1 - (1 - E_0) ** (1 / f_in) where f_in > 0, else 1
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const float part = fk[j] > 0.0f ? __fsub_rn(1.0f, powf(c.one_m_e0, __fdiv_rn(1.0f, fk[j]))) : 1.0f;
        fq[j] = __fdiv_rn(__fmul_rn(fk[j], part), c.e0);
    }
    // v, with the power that q takes of its old value
#pragma unroll
    for (int j = 0; j < N; ++j) {
        float p;
        bold_powers<WHOLE>(c, whole, v, pm1[j], p);
        const float dv = __fdiv_rn(__fsub_rn(fk[j], p), c.tao_0);
        v = __fadd_rn(v, __fmul_rn(dv, c.dt));
        vn[j] = v;
    }
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const float dq = __fdiv_rn(__fsub_rn(fq[j], __fmul_rn(q, pm1[j])), c.tao_0);
        q = __fadd_rn(q, __fmul_rn(dq, c.dt));
        if (out) {
            // V_0 * (7 E_0 (1 - q) + 2 (1 - q / v) + (2 E_0 - 0.2) (1 - v))
            const float a = __fmul_rn(c.seven_e0, __fsub_rn(1.0f, q));
            const float b = __fmul_rn(2.0f, __fsub_rn(1.0f, __fdiv_rn(q, vn[j])));
            const float d = __fmul_rn(c.e0_term, __fsub_rn(1.0f, vn[j]));
            out[static_cast<size_t>(k + j) * n + i] = __fmul_rn(c.v0, __fadd_rn(__fadd_rn(a, b), d));
        }
    }
}

template <bool WHOLE>
__global__ void __launch_bounds__(kBoldThreads)
bold_kernel(BoldConst c, int whole, uint32_t n, uint32_t steps, const float* __restrict__ u, float* __restrict__ state,
            float* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s = state[i], q = state[n + i], v = state[2 * n + i], f = state[3 * n + i];
    uint32_t k = 0;
    for (; k + kBoldSteps <= steps; k += kBoldSteps) bold_steps<WHOLE, kBoldSteps>(c, whole, n, i, k, u, out, s, q, v, f);
    for (; k < steps; ++k) bold_steps<WHOLE, 1>(c, whole, n, i, k, u, out, s, q, v, f);
    state[i] = s;
    state[n + i] = q;
    state[2 * n + i] = v;
    state[3 * n + i] = f;
}

}  // namespace dtb

extern "C" {

void dtb_bold_default_params(dtb_bold_params* p) {
    if (!p) return;
    // data_assimilation/DA_voxel.py:470-476
    *p = dtb_bold_params{200.0, 0.8, 0.4, 1.0, 0.2, 0.8, 0.02, 1e-3};
}

int32_t dtb_bold_run(const dtb_bold_params* p, uint32_t n, uint32_t steps, const float* u, float* state, float* out,
                     void* stream) {
    if (!p || (n && (!u || !state))) return dtb::fail(DTB_INVALID_PARAMETER, "NULL argument");
    if (!(p->alpha > 0.0) || !(p->tao_s != 0.0) || !(p->tao_f != 0.0) || !(p->tao_0 != 0.0) || !(p->E_0 != 0.0))
        return dtb::fail(DTB_INVALID_PARAMETER, "BOLD parameters: alpha > 0 and nonzero time constants and E_0");
    if (n == 0 || steps == 0) return DTB_OK;
    const double div_alpha = 1.0 / p->alpha;
    const dtb::BoldConst c{static_cast<float>(p->epsilon), static_cast<float>(p->tao_s), static_cast<float>(p->tao_f),
                           static_cast<float>(p->tao_0), static_cast<float>(p->E_0), static_cast<float>(p->V_0),
                           static_cast<float>(p->delta_t), static_cast<float>(1.0 - p->E_0),
                           static_cast<float>(div_alpha), static_cast<float>(div_alpha - 1.0),
                           static_cast<float>(7.0 * p->E_0), static_cast<float>(2.0 * p->E_0 - 0.2)};
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    // 1 / alpha as float32: a small whole number takes the products
    const bool whole = c.div_alpha >= 1.0f && c.div_alpha <= dtb::kBoldMostWhole && c.div_alpha == std::floor(c.div_alpha) &&
                       c.div_alpha_m1 == c.div_alpha - 1.0f;
    const uint32_t blocks = (n + dtb::kBoldThreads - 1) / dtb::kBoldThreads;
    if (whole)
        dtb::bold_kernel<true><<<blocks, dtb::kBoldThreads, 0, s>>>(c, static_cast<int>(c.div_alpha), n, steps, u, state, out);
    else
        dtb::bold_kernel<false><<<blocks, dtb::kBoldThreads, 0, s>>>(c, 0, n, steps, u, state, out);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return dtb::cuda_fail(e, "bold_kernel");
    return DTB_OK;
}

}  // extern "C"
