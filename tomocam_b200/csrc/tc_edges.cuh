// tc_edges.cuh -- the standalone prior kernels' march through the slices with
// every edge of the 26-neighbour stencil evaluated once.
//
// rho' is odd and rho'' even, so of a voxel's 26 edges the 13 "forward" ones
// are evaluated by the voxel and the 13 others by the neighbours they lead
// to.  A CTA of 32 x 8 threads owns a 32 x TY tile of voxels and marches
// through a run of slices; the planes it needs (with a one-voxel clamped
// ring) are copied into shared memory a step ahead, and the edges' values go
// through shared memory: those to the next slice in two alternating sets of
// nine planes, those within the slice in four planes.  The tile's ring also
// produces the edges that end inside the tile, a list built at compile time.
//
// Each voxel adds its edges in the order (dz, dy, dx) of the 26 offsets, so
// the sums are bit for bit those of a kernel that evaluates all 26.
#pragma once

#include "tc_cpasync.cuh"
#include "tc_prior.cuh"

namespace tc {

constexpr int EX = 32, EY = 8, ET = EX * EY;  // threads
constexpr int EPW = EX + 2;                   // plane row: x = -1 .. 32

// forward direction k: k < 9: dz = 1, (dy, dx) = (k / 3 - 1, k % 3 - 1); k = 9,
// 10, 11: dz = 0, dy = 1, dx = k - 10; k = 12: (0, 0, 1)
constexpr int ENDIR = 13;
__host__ __device__ constexpr int e_dy(int k) { return k < 9 ? k / 3 - 1 : (k < 12 ? 1 : 0); }
__host__ __device__ constexpr int e_dx(int k) { return k < 9 ? k % 3 - 1 : (k < 12 ? k - 10 : 1); }
__host__ __device__ constexpr float e_w(int k) {
    const int n = (k < 9) + (e_dy(k) != 0) + (e_dx(k) != 0);
    return n == 1 ? 0.0523f : (n == 2 ? 0.0370f : 0.0302f);
}

// ring producers: plane offset of the producer | direction << 16
template <int TY>
struct RingItems {
    int n;
    unsigned v[2 * ET];
};
template <int TY>
constexpr RingItems<TY> make_ring() {
    RingItems<TY> t{};
    for (int k = 0; k < ENDIR; ++k)
        for (int y = -1; y <= TY; ++y)
            for (int x = -1; x <= EX; ++x) {
                if (x >= 0 && x < EX && y >= 0 && y < TY) continue;
                const int cy = y + e_dy(k), cx = x + e_dx(k);
                if (cx < 0 || cx >= EX || cy < 0 || cy >= TY) continue;
                t.v[t.n++] = (unsigned)((y + 1) * EPW + x + 1) | ((unsigned)k << 16);
            }
    return t;
}
template <int TY>
constexpr RingItems<TY> kRing = make_ring<TY>();
static_assert(kRing<8>.n <= 2 * ET, "at most two ring items per thread");
template <int TY>
__device__ const RingItems<TY> kRingDev = make_ring<TY>();

template <int TY>
struct EdgeTile {
    static constexpr int PN = (TY + 2) * EPW;  // one plane
    // plane p of a (clamped to the volume) into dst by 4-byte asynchronous copies
    __device__ __forceinline__ static void load(float *dst, const float *__restrict__ a, int p,
                                                int S, int R, int C, int r0, int c0) {
        const float *src = a + (size_t)min(max(p, 0), S - 1) * R * C;
        for (int i = threadIdx.x; i < PN; i += ET) {
            const int y = i / EPW, x = i - y * EPW;
            const int rr = min(max(r0 + y - 1, 0), R - 1), cc = min(max(c0 + x - 1, 0), C - 1);
            cp_async4(dst + i, src + (size_t)rr * C + cc);
        }
    }
};

// slices per CTA: a run costs its planes and about one more for the plane
// below it; the run with the fewest (waves) x (planes + 1) is taken
inline int edge_run(int tiles, int S, int slots) {
    int best = S;
    double cost = 1e300;
    for (int nz = 1; nz <= (S < 1024 ? S : 1024); ++nz) {
        const int zc = ceil_div(S, nz);
        const double c = (double)ceil_div(tiles * ceil_div(S, zc), slots) * (zc + 1.0);
        if (c < cost) {
            cost = c;
            best = zc;
        }
    }
    return best;
}

}  // namespace tc
