// tc_prior_diff.cu -- derivatives of the qGGMRF prior beyond its gradient,
// for differentiating the MBIR objective and unrolled reconstructions.
//
// The prior potential whose gradient is the reference's clamped 26-neighbour
// stencil (src/gpu/cuTV2.cu:33-76 with the clamp of
// src/gpu/dev_memory.cuh:88-94) is
//   U(x) = 1/2 sum_v sum_{26 d} w_d rho(x_v - x_c(v+d)),
//   rho(delta) = u^2 / (c + u^(2-p)),  u = |delta| / sigma   (q = 2),
// with rho'(delta) = delta A(t) / sigma^2, t = u^(2-p),
//   A(t) = (2c + p t) / (c + t)^2,  A'(t) = ((p - 4) c - p t) / (c + t)^3,
//   rho''(delta) = (A + (2 - p) t A') / sigma^2   (finite at delta = 0),
// and the sigma derivatives
//   d rho / d sigma  = -delta rho'(delta) / sigma,
//   d rho' / d sigma = -(delta rho''(delta) + rho'(delta)) / sigma.
// Nothing here has a counterpart in the reference, which only evaluates the
// gradient.
#include "tc_edges.cuh"
#include "tc_plan.cuh"
#include "tc_prior.cuh"

namespace tc {

constexpr int DX = 32, DY = 8;
constexpr int DN = 3 * (DY + 2) * (DX + 2);

struct PriorTerms {
    float rho, d1, d2;  // rho, rho', rho'' (with the 1/sigma^2 factors)
};

__device__ __forceinline__ PriorTerms prior_terms(float delta, float inv_sigma, float inv_sq,
                                                  float qmp, float p) {
    const float l = fmaxf(lg2_approx(fabsf(delta) * inv_sigma), -200.0f);
    const float t = ex2_approx(qmp * l);
    const float r = rcp_approx(MRF_C + t);
    const float A = (2.0f * MRF_C + p * t) * (r * r);
    const float Ap = ((p - 4.0f) * MRF_C - p * t) * (r * r * r);
    PriorTerms o;
    o.rho = delta * delta * inv_sq * r;
    o.d1 = delta * A * inv_sq;
    o.d2 = (A + qmp * t * Ap) * inv_sq;
    return o;
}

// the clamped 3 x 10 x 34 neighbourhood of the CTA's 32 x 8 patch of slice s
__device__ __forceinline__ void load_nbhd(float *tile, const float *__restrict__ a, int s, int S,
                                          int R, int C, int r0, int c0) {
    const size_t plane = (size_t)R * C;
    for (int i = threadIdx.y * DX + threadIdx.x; i < DN; i += DX * DY) {
        const int dz = i / ((DY + 2) * (DX + 2));
        const int rem = i - dz * (DY + 2) * (DX + 2);
        const int dy = rem / (DX + 2), dx = rem - dy * (DX + 2);
        const int ss = min(max(s + dz - 1, 0), S - 1);
        const int rr = min(max(r0 + dy - 1, 0), R - 1);
        const int cc = min(max(c0 + dx - 1, 0), C - 1);
        tile[i] = a[ss * plane + (size_t)rr * C + cc];
    }
}

__device__ __forceinline__ int nb_index(int dz, int dy, int dx) {
    return (dz * (DY + 2) + threadIdx.y + dy) * (DX + 2) + threadIdx.x + dx;
}

// partials[cta] = {1/2 sum w rho, 1/2 sum w d rho / d sigma}
__global__ void k_qggmrf_value(const float *__restrict__ x, int S, int R, int C, float inv_sigma,
                               float inv_sq, float qmp, float p, double *__restrict__ partials) {
    __shared__ float tile[DN];
    const int c0 = blockIdx.x * DX, r0 = blockIdx.y * DY, s = blockIdx.z;
    load_nbhd(tile, x, s, S, R, C, r0, c0);
    __syncthreads();
    const int c = c0 + threadIdx.x, r = r0 + threadIdx.y;
    double acc[2] = {0.0, 0.0};
    if (c < C && r < R) {
        const float u = tile[nb_index(1, 1, 1)];
        float a0 = 0.0f, a1 = 0.0f;
#pragma unroll
        for (int dz = 0; dz < 3; ++dz)
#pragma unroll
            for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                for (int dx = 0; dx < 3; ++dx) {
                    if (dz == 1 && dy == 1 && dx == 1) continue;
                    const float w = c_qggmrf_w[(dz * 3 + dy) * 3 + dx];
                    const float d = u - tile[nb_index(dz, dy, dx)];
                    const PriorTerms pt = prior_terms(d, inv_sigma, inv_sq, qmp, p);
                    a0 = fmaf(w, pt.rho, a0);
                    a1 = fmaf(w, d * pt.d1, a1);
                }
        acc[0] = 0.5 * (double)a0;
        acc[1] = -0.5 * (double)a1 * (double)inv_sigma;
    }
    block_sum<2>(acc, threadIdx.y * DX + threadIdx.x, DX * DY);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        double *dst = partials + (((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * 2;
        dst[0] = acc[0];
        dst[1] = acc[1];
    }
}

// hv[u] = scale * sum_d w rho''(x_u - x_n) (v_u - v_n)   (if hv)
// partials[cta] = {sum_u v_u sum_d w rho'(delta),
//                  sum_u v_u sum_d w d rho'(delta) / d sigma}
// One voxel per thread of a 32 x 8 tile; an edge's rho' and rho'' are
// evaluated once and passed through shared memory (tc_edges.cuh).  Four
// buffers of x and v planes: a voxel's backward edges read the plane below.
// 32 slices of 768^2: 764 -> 562 us, with the two dot products 940 -> 618
// (one partial pair per run of slices instead of one per slice).  Issue bounds
// it (ncu: 78 % of the slots, L1 data pipe 58 %, FMA pipe 43 %, SFU pipe 37 %)
// at three CTAs per SM, which both 71 KB of shared memory and 80 registers set.
constexpr int HTY = 8;
struct HSmem {
    float x[4][EdgeTile<HTY>::PN], v[4][EdgeTile<HTY>::PN];
    float d1[2][9][EdgeTile<HTY>::PN], d2[2][9][EdgeTile<HTY>::PN];  // to the next slice
    float f1[4][EdgeTile<HTY>::PN], f2[4][EdgeTile<HTY>::PN];        // within the slice
};

__global__ void __launch_bounds__(ET, 3)
k_qggmrf_hvp(const float *__restrict__ x, const float *__restrict__ v, float *__restrict__ hv,
             int S, int R, int C, float inv_sigma, float inv_sq, float qmp, float p, float scale,
             double *__restrict__ partials, int zc) {
    using T = EdgeTile<HTY>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    HSmem &sm = *reinterpret_cast<HSmem *>(smem_raw);
    const int c0 = blockIdx.x * EX, r0 = blockIdx.y * HTY;
    const int z0 = blockIdx.z * zc, z1 = min(S, z0 + zc);
    const int tx = threadIdx.x % EX, ty = threadIdx.x / EX;
    const int o = (ty + 1) * EPW + tx + 1;
    const int c = c0 + tx, r = r0 + ty;
    auto load = [&](int q) {
        T::load(sm.x[(q + 4) & 3], x, q, S, R, C, r0, c0);
        T::load(sm.v[(q + 4) & 3], v, q, S, R, C, r0, c0);
    };
    // this thread's ring items, read once
    unsigned item[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int i = threadIdx.x + j * ET;
        item[j] = i < kRing<HTY>.n ? __ldg(&kRingDev<HTY>.v[i]) : ~0u;
    }
    auto ring = [&](const float *a, const float *b, int nxt, int kmax) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int pos = item[j] & 0xffff, k = item[j] >> 16;
            if (k >= kmax) continue;
            const int nb = pos + (k < 9 ? (k / 3 - 1) * EPW + k % 3 - 1 : k < 12 ? EPW + k - 10 : 1);
            const PriorTerms t = prior_terms(a[pos] - (k < 9 ? b : a)[nb], inv_sigma, inv_sq, qmp, p);
            if (k < 9) {
                sm.d1[nxt][k][pos] = t.d1;
                sm.d2[nxt][k][pos] = t.d2;
            } else {
                sm.f1[k - 9][pos] = t.d1;
                sm.f2[k - 9][pos] = t.d2;
            }
        }
    };
    load(z0 - 1);
    load(z0);
    cp_async_commit();
    load(z0 + 1);
    cp_async_commit();
    cp_async_wait_prev();
    __syncthreads();
    if (S > 1) {
        // the edges from plane z0 - 1
        const float *a = sm.x[(z0 + 3) & 3], *b = sm.x[z0 & 3];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const PriorTerms t =
                prior_terms(a[o] - b[o + e_dy(k) * EPW + e_dx(k)], inv_sigma, inv_sq, qmp, p);
            sm.d1[0][k][o] = t.d1;
            sm.d2[0][k][o] = t.d2;
        }
        ring(a, b, 0, 9);
    }
    cp_async_wait_all();
    __syncthreads();
    double acc[2] = {0.0, 0.0};
    for (int s = z0, cur = 0; s < z1; ++s, cur ^= 1) {
        if (s + 1 < z1) load(s + 2);
        cp_async_commit();
        const float *xm = sm.x[(s + 3) & 3], *xa = sm.x[s & 3], *xb = sm.x[(s + 1) & 3];
        const float *vm = sm.v[(s + 3) & 3], *va = sm.v[s & 3], *vb = sm.v[(s + 1) & 3];
        const float u = xa[o], vu = va[o];
        float o1[ENDIR], o2[ENDIR];
#pragma unroll
        for (int k = 0; k < ENDIR; ++k) {
            const PriorTerms t = prior_terms(u - (k < 9 ? xb : xa)[o + e_dy(k) * EPW + e_dx(k)],
                                             inv_sigma, inv_sq, qmp, p);
            o1[k] = t.d1;
            o2[k] = t.d2;
            if (k < 9) {
                sm.d1[cur ^ 1][k][o] = t.d1;
                sm.d2[cur ^ 1][k][o] = t.d2;
            } else {
                sm.f1[k - 9][o] = t.d1;
                sm.f2[k - 9][o] = t.d2;
            }
        }
        ring(xa, xb, cur ^ 1, ENDIR);
        __syncthreads();
        if (c < C && r < R) {
            // a single slice is its own clamped neighbour below and above
            const int low = S > 1 ? cur : cur ^ 1;
            float h = 0.0f, g1 = 0.0f, gs = 0.0f;
            auto add = [&](int k, float d, float dv, float d1, float d2) {
                const float w = e_w(k);
                h = fmaf(w * d2, dv, h);
                g1 = fmaf(w, d1, g1);
                gs = fmaf(w, fmaf(d, d2, d1), gs);
            };
            // neighbours in (dz, dy, dx) order; those before the voxel hold
            // its edge, rho' with the other sign
#pragma unroll
            for (int k = 8; k >= 0; --k) {
                const int q = o - e_dy(k) * EPW - e_dx(k);
                add(k, u - xm[q], vu - vm[q], -sm.d1[low][k][q], sm.d2[low][k][q]);
            }
#pragma unroll
            for (int k : {11, 10, 9, 12}) {
                const int q = o - e_dy(k) * EPW - e_dx(k);
                add(k, u - xa[q], vu - va[q], -sm.f1[k - 9][q], sm.f2[k - 9][q]);
            }
#pragma unroll
            for (int k : {12, 9, 10, 11}) {
                const int q = o + e_dy(k) * EPW + e_dx(k);
                add(k, u - xa[q], vu - va[q], o1[k], o2[k]);
            }
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                const int q = o + e_dy(k) * EPW + e_dx(k);
                add(k, u - xb[q], vu - vb[q], o1[k], o2[k]);
            }
            if (hv) hv[((size_t)s * R + r) * C + c] = scale * h;
            acc[0] += (double)vu * (double)g1;
            acc[1] -= (double)vu * (double)gs * (double)inv_sigma;
        }
        cp_async_wait_all();
        __syncthreads();
    }
    if (partials) {
        block_sum<2>(acc, threadIdx.x, ET);
        if (threadIdx.x == 0) {
            double *dst = partials + (((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * 2;
            dst[0] = acc[0];
            dst[1] = acc[1];
        }
    }
}

static int prior_args(int S, int R, int C, float sigma, float p) {
    if (S < 0 || R < 0 || C < 0) TC_FAIL(TC_ERR_SHAPE, "negative size");
    if (S > 65535) TC_FAIL(TC_ERR_SHAPE, "too many slices for one prior launch");
    if (!(sigma > 0) || !std::isfinite(sigma)) TC_FAIL(TC_ERR_ARG, "sigma must be > 0");
    if (!(p > 0 && p <= 2)) TC_FAIL(TC_ERR_ARG, "p must be in (0, 2]");
    return TC_OK;
}

// sum the per-CTA pairs on the device and copy the two totals to the host
static int finish_dots(double *parts, int nparts, double *a, double *b, cudaStream_t st) {
    double h[2] = {0.0, 0.0};
    TC_TRY(reduce_partials(parts, nparts, 2, parts + (size_t)nparts * 2, st));
    TC_CUDA(cudaMemcpyAsync(h, parts + (size_t)nparts * 2, 2 * sizeof(double),
                            cudaMemcpyDeviceToHost, st));
    TC_CUDA(cudaStreamSynchronize(st));
    if (a) *a = h[0];
    if (b) *b = h[1];
    return TC_OK;
}

int qggmrf_value_launch(const float *x, int S, int R, int C, float sigma, float p, double *value,
                        double *dsigma, cudaStream_t st) {
    TC_TRY(prior_args(S, R, C, sigma, p));
    if ((size_t)S * R * C == 0) {
        if (value) *value = 0.0;
        if (dsigma) *dsigma = 0.0;
        return TC_OK;
    }
    const dim3 grid(ceil_div(C, DX), ceil_div(R, DY), S);
    const int nparts = (int)(grid.x * grid.y * grid.z);
    double *parts = nullptr;
    TC_CUDA(cudaMallocAsync(&parts, ((size_t)nparts * 2 + 2) * sizeof(double), st));
    const PriorParams pp = make_prior(sigma, p, 1.0f);
    k_qggmrf_value<<<grid, dim3(DX, DY), 0, st>>>(x, S, R, C, pp.inv_sigma, pp.inv_sq, pp.qmp, p,
                                                  parts);
    cudaError_t e = cudaGetLastError();
    int rc = e == cudaSuccess ? finish_dots(parts, nparts, value, dsigma, st) : TC_ERR_CUDA;
    if (e != cudaSuccess) set_error(std::string("CUDA error: ") + cudaGetErrorString(e));
    cudaFreeAsync(parts, st);
    return rc;
}

int qggmrf_hvp_launch(const float *x, const float *v, float *hv, int S, int R, int C, float sigma,
                      float p, float scale, double *vg, double *vgs, cudaStream_t st) {
    TC_TRY(prior_args(S, R, C, sigma, p));
    if ((size_t)S * R * C == 0) {
        if (vg) *vg = 0.0;
        if (vgs) *vgs = 0.0;
        return TC_OK;
    }
    const bool dots = vg || vgs;
    int dev = 0, nsm = 0;
    TC_CUDA(cudaGetDevice(&dev));
    TC_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    TC_CUDA(cudaFuncSetAttribute(k_qggmrf_hvp, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(HSmem)));
    const int gx = ceil_div(C, EX), gy = ceil_div(R, HTY);
    const int zc = edge_run(gx * gy, S, 3 * nsm);
    const dim3 grid(gx, gy, ceil_div(S, zc));
    const int nparts = (int)(grid.x * grid.y * grid.z);
    double *parts = nullptr;
    if (dots) TC_CUDA(cudaMallocAsync(&parts, ((size_t)nparts * 2 + 2) * sizeof(double), st));
    const PriorParams pp = make_prior(sigma, p, scale);
    k_qggmrf_hvp<<<grid, ET, sizeof(HSmem), st>>>(x, v, hv, S, R, C, pp.inv_sigma, pp.inv_sq,
                                                  pp.qmp, p, scale, parts, zc);
    cudaError_t e = cudaGetLastError();
    int rc = TC_OK;
    if (e != cudaSuccess) {
        set_error(std::string("CUDA error: ") + cudaGetErrorString(e));
        rc = TC_ERR_CUDA;
    } else if (dots) {
        rc = finish_dots(parts, nparts, vg, vgs, st);
    }
    if (parts) cudaFreeAsync(parts, st);
    return rc;
}

}  // namespace tc
