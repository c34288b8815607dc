// Ensemble Kalman update of data assimilation: DA_voxel.filter
// (data_assimilation/DA_voxel.py:289-307), the step that follows the BOLD
// model in each assimilation window.
//
// w_hat [E][V][S] holds, per ensemble member and voxel, the assimilated
// hyper-parameters, the hemodynamic state and, last, the BOLD signal.  With
// d = w_hat - mean_e(w_hat), c_v = sum_e d[e,v,S-1]^2 / (E-1) + sigma,
// T[e,v] = d[e,v,S-1] / c_v / (E-1) and the innovation
// I[e,v] = y[v] + sqrt(sigma) n[e,v] - w_hat[e,v,S-1]:
//   w = w_hat + rate * I[e,v] * sum_e' T[e',v] d[e',v,s]
//             + (1 - rate) * sum_e' G[e,e'] d[e',v,s],   G = I T^T / V.
// Three kernels: per-voxel statistics, the E x E gain G, and the update.  Everything
// accumulates in double and is rounded once, so the result is the float32 rounding of the
// exact update (the reference's float32 reductions and GEMMs agree to ~1e-7 relative).
#include <algorithm>

#include "dtb_engine.h"

namespace dtb {

constexpr int kDaThreads = 256;

// Statistics: a CTA takes `vb` consecutive voxels, whose vb x S columns are contiguous in every
// member's row, so the members' loads are coalesced (one warp per voxel read 4 bytes of 32
// different lines per load).  The 256 threads are `groups` rows of `width` lanes (width a power
// of two, at least vb x S where that fits); partial sums of a column meet in shared memory in a
// fixed order.
__global__ void __launch_bounds__(kDaThreads)
da_stats_kernel(uint32_t E, uint32_t V, uint32_t S, uint32_t vb, uint32_t width, const float* __restrict__ w,
                const float* __restrict__ y, const float* __restrict__ noise, double sigma, double* __restrict__ mean,
                double* __restrict__ temp, double* __restrict__ innov, double* __restrict__ colsum) {
    __shared__ double s_part[kDaThreads], s_mean[kDaThreads];
    const uint32_t groups = kDaThreads / width, g = threadIdx.x / width, x = threadIdx.x % width;
    const uint32_t v0 = blockIdx.x * vb, nv = min(vb, V - v0), cols = nv * S;
    const size_t row = static_cast<size_t>(V) * S;
    const double sq = sqrt(sigma);
    // sum of a column's partial sums, for every thread of lane column x
    auto meet = [&](double part) {
        __syncthreads();
        s_part[threadIdx.x] = part;
        __syncthreads();
        double sum = 0.0;
        for (uint32_t k = 0; k < groups; ++k) sum += s_part[k * width + x];
        return sum;
    };
    for (uint32_t c0 = 0; c0 < cols; c0 += width) {         // one pass unless S is wider than the CTA
        const uint32_t col = c0 + x;
        const bool in = col < cols;
        const uint32_t vl = in ? col / S : 0u, v = v0 + vl;
        const float* base = w + static_cast<size_t>(v0) * S + (in ? col : 0u);
        double acc = 0.0;
        if (in) {
#pragma unroll 4
            for (uint32_t e = g; e < E; e += groups) acc += base[e * row];
        }
        const double m = meet(acc) / E;
        // the voxel's last column: its mean and variance
        const float* last = w + static_cast<size_t>(v) * S + S - 1;
        double ml;
        if (cols <= width) {                                 // it is another lane's column of this pass
            if (in && g == 0) s_mean[x] = m;
            __syncthreads();
            ml = s_mean[in ? vl * S + S - 1 : 0u];
        } else {
            double al = 0.0;
            if (in) {
#pragma unroll 4
                for (uint32_t e = g; e < E; e += groups) al += last[e * row];
            }
            ml = meet(al) / E;
        }
        double cx = 0.0;
        if (in) {
#pragma unroll 4
            for (uint32_t e = g; e < E; e += groups) {
                const double d = last[e * row] - ml;
                cx += d * d;
            }
        }
        const double cxx = meet(cx) / (E - 1) + sigma;
        double cs = 0.0;
        if (in) {
            const bool lead = col % S == S - 1;              // the lane that writes the voxel's temp and innov
#pragma unroll 4
            for (uint32_t e = g; e < E; e += groups) {
                const double l = last[e * row];
                const double t = (l - ml) / cxx / (E - 1);
                cs += t * (base[e * row] - m);
                if (lead) {
                    temp[static_cast<size_t>(e) * V + v] = t;
                    innov[static_cast<size_t>(e) * V + v] = static_cast<double>(y[v]) + sq * noise[static_cast<size_t>(e) * V + v] - l;
                }
            }
        }
        const double sum = meet(cs);
        if (in && g == 0) {
            mean[static_cast<size_t>(v0) * S + col] = m;
            colsum[static_cast<size_t>(v0) * S + col] = sum;
        }
    }
}

// G[e][f] = sum_v I[e,v] T[f,v] / V: one warp per (e, f).  The factors are read from L2 for each of
// the E^2 products; 8 x 8 tiles of products that staged them in shared memory measured slower at
// every size (whole filter: 16 x 3000 x 6 34 against 66 us, 100 x 1000 x 10 64 against 78, 150 x
// 3000 x 16 289 against 360), each tile being a chain over all voxels on few CTAs.  Count holds E^2.
template <class Count>
__global__ void __launch_bounds__(256)
da_gain_kernel(uint32_t E, uint32_t V, const double* __restrict__ innov, const double* __restrict__ temp,
               double* __restrict__ gain) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const Count products = static_cast<Count>(E) * E;
    for (Count k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < products; k += nw) {
        const uint32_t e = static_cast<uint32_t>(k / E), f = static_cast<uint32_t>(k % E);
        double acc = 0.0;
        for (uint32_t v = lane; v < V; v += 32) acc += innov[static_cast<size_t>(e) * V + v] * temp[static_cast<size_t>(f) * V + v];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) gain[k] = acc / V;
    }
}

// Update: a thread owns one column (voxel, state) for kUpdRows members, so a deviation is read
// and widened once for kUpdRows products (one thread per output widened it for each); the
// members' gains sit in shared memory and are read as broadcasts, kUpdChunk of them at a time.
// Over 16 to 150 members, 1,000 and 3,000 voxels and 6 to 16 states ten members a thread run within
// 5 us of the better of 8 and 16 and mostly are the best (150 x 3000 x 16: 8 / 10 / 16 members 297 /
// 284 / 334 us, 97 x 3000 x 10 106 / 101 / 114, 33 x 3000 x 6 39 / 41 / 43).
constexpr int kUpdThreads = 128, kUpdChunk = 128;
template <int kUpdRows>
__global__ void __launch_bounds__(kUpdThreads)
da_update_kernel(uint32_t E, uint32_t V, uint32_t S, const float* __restrict__ w, const double* __restrict__ mean,
                 const double* __restrict__ innov, const double* __restrict__ colsum, const double* __restrict__ gain,
                 double rate, float* __restrict__ out) {
    __shared__ double s_gain[kUpdChunk][kUpdRows];
    const size_t cols = static_cast<size_t>(V) * S;
    const size_t col = static_cast<size_t>(blockIdx.x) * kUpdThreads + threadIdx.x;
    const uint32_t e0 = blockIdx.y * kUpdRows;
    const bool in = col < cols;
    const double m = in ? mean[col] : 0.0;
    double acc[kUpdRows] = {};
    for (uint32_t f0 = 0; f0 < E; f0 += kUpdChunk) {
        const uint32_t nf = min(static_cast<uint32_t>(kUpdChunk), E - f0);
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < nf * kUpdRows; k += kUpdThreads) {
            const uint32_t r = k / nf, f = k % nf;
            s_gain[f][r] = e0 + r < E ? gain[static_cast<size_t>(e0 + r) * E + f0 + f] : 0.0;
        }
        __syncthreads();
        if (in) {
#pragma unroll 4
            for (uint32_t f = 0; f < nf; ++f) {
                const double d = w[static_cast<size_t>(f0 + f) * cols + col] - m;
#pragma unroll
                for (int r = 0; r < kUpdRows; ++r) acc[r] = __fma_rn(s_gain[f][r], d, acc[r]);
            }
        }
    }
    if (!in) return;
    const uint32_t v = static_cast<uint32_t>(col / S);
    const double cs = colsum[col];
#pragma unroll
    for (int r = 0; r < kUpdRows; ++r) {
        const uint32_t e = e0 + r;
        if (e >= E) break;
        const size_t k = static_cast<size_t>(e) * cols + col;
        const double x = static_cast<double>(w[k]) + rate * innov[static_cast<size_t>(e) * V + v] * cs + (1.0 - rate) * acc[r];
        out[k] = static_cast<float>(x);
    }
}

}  // namespace dtb

extern "C" int32_t dtb_da_filter(uint32_t ensembles, uint32_t voxels, uint32_t states, const float* w_hat,
                                 const float* bold_y, const float* noise, double bold_sigma, double rate, float* w_out,
                                 void* stream) {
    if (!w_hat || !bold_y || !noise || !w_out) return dtb::fail(DTB_INVALID_PARAMETER, "NULL argument");
    if (ensembles < 2 || voxels == 0 || states == 0) return dtb::fail(DTB_INVALID_PARAMETER, "need >= 2 members, voxels and states");
    if (!(bold_sigma >= 0.0)) return dtb::fail(DTB_INVALID_PARAMETER, "bold_sigma must be >= 0");
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    const size_t E = ensembles, V = voxels, S = states;
    double* buf = nullptr;
    const size_t n_mean = V * S, n_ev = E * V;
    cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(&buf), sizeof(double) * (2 * n_mean + 2 * n_ev + E * E), s);
    if (e != cudaSuccess) return dtb::cuda_fail(e, "dtb_da_filter scratch");
    double* mean = buf;
    double* colsum = mean + n_mean;
    double* temp = colsum + n_mean;
    double* innov = temp + n_ev;
    double* gain = innov + n_ev;
    int dev = 0, sms = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) {
        cudaFreeAsync(buf, s);
        return dtb::cuda_fail(e, "dtb_da_filter");
    }
    // voxels per statistics CTA: as many as 64 columns take, fewer where that leaves an SM fewer than
    // two CTAs (a narrower CTA also walks the members in fewer turns).  Whole filter, 64 columns
    // against this: 150 x 50 x 6 60 / 40 us, 64 x 300 x 6 37 / 30, 16 x 1000 x 6 27 / 25; four or
    // eight CTAs an SM cost the last 2 and 7 us more.
    const uint32_t vb = static_cast<uint32_t>(std::max<size_t>(1, std::min<size_t>(64 / S, (V + 2 * sms - 1) / (2 * sms))));
    uint32_t width = 1;
    while (width < vb * S && width < dtb::kDaThreads) width *= 2;
    dtb::da_stats_kernel<<<static_cast<uint32_t>((V + vb - 1) / vb), dtb::kDaThreads, 0, s>>>(
        ensembles, voxels, states, vb, width, w_hat, bold_y, noise, bold_sigma, mean, temp, innov, colsum);
    const uint32_t gain_ctas = static_cast<uint32_t>(std::min<size_t>((E * E + 7) / 8, 4096));
    if (E < 65536) dtb::da_gain_kernel<uint32_t><<<gain_ctas, 256, 0, s>>>(ensembles, voxels, innov, temp, gain);
    else dtb::da_gain_kernel<unsigned long long><<<gain_ctas, 256, 0, s>>>(ensembles, voxels, innov, temp, gain);
    // ten members a thread, two where ten leave SMs without a CTA (whole filter, ten against two:
    // 40 x 50 x 10 25 / 18 us, 100 x 50 x 6 31 / 24, 16 x 300 x 10 21 / 18)
    const uint32_t col_ctas = static_cast<uint32_t>((V * S + dtb::kUpdThreads - 1) / dtb::kUpdThreads);
    auto update = [&](auto kernel, uint32_t rows) {
        kernel<<<dim3(col_ctas, (ensembles + rows - 1) / rows), dtb::kUpdThreads, 0, s>>>(ensembles, voxels, states, w_hat, mean, innov,
                                                                                      colsum, gain, rate, w_out);
    };
    if (static_cast<size_t>(col_ctas) * ((E + 9) / 10) < static_cast<size_t>(sms)) update(dtb::da_update_kernel<2>, 2);
    else update(dtb::da_update_kernel<10>, 10);
    e = cudaGetLastError();
    cudaFreeAsync(buf, s);
    if (e != cudaSuccess) return dtb::cuda_fail(e, "dtb_da_filter");
    return DTB_OK;
}
