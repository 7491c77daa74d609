// tc_prior.cu -- standalone qGGMRF gradient, g += scale * sum_26 w rho'(x_v - x_n)
// with clamp-to-edge boundaries (src/gpu/cuTV2.cu:33-93,
// src/gpu/dev_memory.cuh:88-94).
#include "tc_edges.cuh"
#include "tc_plan.cuh"

namespace tc {

// One voxel per thread of a 32 x 8 tile.  Evaluating all 26 edges of every
// voxel, the kernel ran at the SFU's rate (78 operations per voxel: 317 of
// its 356 us on 32 slices of 768^2); with shared edges and the ring's 11 %
// more there are 43, and it takes 272 us (16 x 2048^2: 1246 -> 918).  Now issue
// bounds it (ncu: 76 % of the slots, SFU pipe 71 %, L1 data pipe 50 %; the
// waits are for a shared-memory or SFU result), and warps per SM count: six
// CTAs of 40 registers 272 us, five 280, seven (32 registers) 293; 32 x 16
// tiles at three CTAs 362.  Volumes of a few hundred thousand voxels take as
// long as before (10 to 20 us, launch and latency); thin ones whose tiles are
// mostly padding up to 4 us longer (700 x 3 x 5: 10 -> 14 us).
constexpr int QTY = 8, QCTAS = 6;
struct QSmem {
    float plane[3][EdgeTile<QTY>::PN];
    float e1[2][9][EdgeTile<QTY>::PN];  // edges to the next slice, by producer
    float e0[4][EdgeTile<QTY>::PN];     // edges within the slice
};

__global__ void __launch_bounds__(ET, QCTAS)
k_qggmrf(const float *__restrict__ x, float *__restrict__ g, int S, int R, int C, PriorParams pp,
         int zc) {
    using T = EdgeTile<QTY>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    QSmem &sm = *reinterpret_cast<QSmem *>(smem_raw);
    const int c0 = blockIdx.x * EX, r0 = blockIdx.y * QTY;
    const int z0 = blockIdx.z * zc, z1 = min(S, z0 + zc);
    const int tx = threadIdx.x % EX, ty = threadIdx.x / EX;
    auto plane = [&](int p) { return sm.plane[(p + 3) % 3]; };
    // this thread's ring items, read once
    unsigned item[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int i = threadIdx.x + j * ET;
        item[j] = i < kRing<QTY>.n ? __ldg(&kRingDev<QTY>.v[i]) : ~0u;
    }
    auto ring = [&](const float *a, const float *b, float (*e1)[T::PN], int kmax) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int pos = item[j] & 0xffff, k = item[j] >> 16;
            if (k >= kmax) continue;
            const int nb = pos + (k < 9 ? (k / 3 - 1) * EPW + k % 3 - 1 : k < 12 ? EPW + k - 10 : 1);
            const float e = d_pot_unscaled(a[pos] - (k < 9 ? b : a)[nb], pp);
            if (k < 9) e1[k][pos] = e;
            else sm.e0[k - 9][pos] = e;
        }
    };
    const int o = (ty + 1) * EPW + tx + 1;
    const int c = c0 + tx, r = r0 + ty;
    T::load(plane(z0 - 1), x, z0 - 1, S, R, C, r0, c0);
    T::load(plane(z0), x, z0, S, R, C, r0, c0);
    cp_async_commit();
    T::load(plane(z0 + 1), x, z0 + 1, S, R, C, r0, c0);
    cp_async_commit();
    cp_async_wait_prev();
    __syncthreads();
    if (S > 1) {
        // the edges from plane z0 - 1
        const float *a = plane(z0 - 1), *b = plane(z0);
#pragma unroll
        for (int k = 0; k < 9; ++k)
            sm.e1[0][k][o] = d_pot_unscaled(a[o] - b[o + e_dy(k) * EPW + e_dx(k)], pp);
        ring(a, b, sm.e1[0], 9);
    }
    cp_async_wait_all();
    __syncthreads();
    for (int s = z0, cur = 0; s < z1; ++s, cur ^= 1) {
        if (s + 1 < z1) T::load(plane(s + 2), x, s + 2, S, R, C, r0, c0);
        cp_async_commit();
        const bool in = c < C && r < R;
        const size_t i = ((size_t)s * R + r) * C + c;
        const float g0 = in ? g[i] : 0.0f;
        const float *a = plane(s), *b = plane(s + 1);
        float own[ENDIR];
        const float u = a[o];
#pragma unroll
        for (int k = 0; k < ENDIR; ++k) {
            own[k] = d_pot_unscaled(u - (k < 9 ? b : a)[o + e_dy(k) * EPW + e_dx(k)], pp);
            if (k < 9) sm.e1[cur ^ 1][k][o] = own[k];
            else sm.e0[k - 9][o] = own[k];
        }
        ring(a, b, sm.e1[cur ^ 1], ENDIR);
        __syncthreads();
        if (in) {
            // a single slice is its own clamped neighbour below and above
            float (*below)[T::PN] = sm.e1[S > 1 ? cur : cur ^ 1];
            float acc = 0.0f;
            // neighbours in (dz, dy, dx) order: the 13 before the voxel hold
            // its edge themselves, with the other sign
#pragma unroll
            for (int k = 8; k >= 0; --k)
                acc = fmaf(e_w(k), -below[k][o - e_dy(k) * EPW - e_dx(k)], acc);
#pragma unroll
            for (int k : {11, 10, 9, 12})
                acc = fmaf(e_w(k), -sm.e0[k - 9][o - e_dy(k) * EPW - e_dx(k)], acc);
#pragma unroll
            for (int k : {12, 9, 10, 11}) acc = fmaf(e_w(k), own[k], acc);
#pragma unroll
            for (int k = 0; k < 9; ++k) acc = fmaf(e_w(k), own[k], acc);
            g[i] = g0 + (pp.scale * pp.inv_sq) * acc;
        }
        cp_async_wait_all();
        __syncthreads();
    }
}

int qggmrf_launch(const float *x, float *g, int S, int R, int C, float sigma, float p,
                  float scale, cudaStream_t st) {
    if (S > 65535) TC_FAIL(TC_ERR_SHAPE, "too many slices for one prior launch");
    int dev = 0, nsm = 0;
    TC_CUDA(cudaGetDevice(&dev));
    TC_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    static_assert(sizeof(QSmem) <= 48 * 1024, "no opt-in for more shared memory needed");
    const int gx = ceil_div(C, EX), gy = ceil_div(R, QTY);
    const int zc = edge_run(gx * gy, S, QCTAS * nsm);
    const dim3 grid(gx, gy, ceil_div(S, zc));
    k_qggmrf<<<grid, ET, sizeof(QSmem), st>>>(x, g, S, R, C, make_prior(sigma, p, scale), zc);
    TC_LAUNCH_CHECK();
    return TC_OK;
}

}  // namespace tc
