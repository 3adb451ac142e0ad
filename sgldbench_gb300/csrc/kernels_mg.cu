// Multigrid transfer, smoothing and bookkeeping kernels on the full grid.
//
// Restriction / prolongation (reference: src/Solving_RestrictResidual.m,
// src/Solving_InterpolationDeviation.m and their MEX kernels).  The
// reference builds a per-coarse-element table of the (s+1)^3 fine nodes,
// scatters RI' r / multiplicity into the coarse nodes and averages RI x over
// the elements sharing a fine node.  Because trilinear interpolation from a
// continuous coarse field gives the same value from every element that
// contains a fine node, that operator is exactly P = trilinear interpolation
// restricted to active fine nodes and R = P'.  On the structured grid this is
// a separable tent stencil of half-width s: w(d) = (s - |d|) / s per axis.
// Inactive nodes carry zeros on every level, so no tables are needed.
//
// The additive V-cycle of the reference (src/Solving_Vcycle.m:12-50) is
//   r_l = R r_{l-1};  x_L = A_L^-1 r_L;
//   x_{l} = t_l + P x_{l+1} + t_l  with t_l = (omega r_l) ./ D_l.
// 2 omega ./ D_l is formed once per assembly, so a fine node takes one
// multiply-add, x_l = r_l (2 omega / D_l) + P x_{l+1}, which may differ from the
// reference's sum in the last bit.
#include <algorithm>

#include "sgld_internal.cuh"

namespace sgld {

template <typename T>
__global__ void k_restrict(const T *__restrict__ rf, T *__restrict__ rc, int nyc, int nxc, int nzc, int s) {
    const int NYc = nyc + 1, NXc = nxc + 1, NZc = nzc + 1;
    const int NYf = s * nyc + 1, NXf = s * nxc + 1, NZf = s * nzc + 1;
    // grid: x over the (y, x) plane of coarse nodes, y over z (32-bit index math)
    const int pl = blockIdx.x * blockDim.x + threadIdx.x;
    if (pl >= NYc * NXc) return;
    const int I = pl % NYc, J = pl / NYc, Kz = blockIdx.y;
    const int64_t n = (int64_t)pl + (int64_t)NYc * NXc * Kz;
    (void)NZc;
    const T inv = T(1) / T(s);
    T a0 = T(0), a1 = T(0), a2 = T(0);
    for (int dz = -s + 1; dz < s; ++dz) {
        const int fz = s * Kz + dz;
        if (fz < 0 || fz >= NZf) continue;
        const T wz = T(s - abs(dz)) * inv;
        for (int dx = -s + 1; dx < s; ++dx) {
            const int fx = s * J + dx;
            if (fx < 0 || fx >= NXf) continue;
            const T wxz = T(s - abs(dx)) * inv * wz;
            for (int dy = -s + 1; dy < s; ++dy) {
                const int fy = s * I + dy;
                if (fy < 0 || fy >= NYf) continue;
                const T w = T(s - abs(dy)) * inv * wxz;
                const int64_t f = (int64_t)fy + (int64_t)NYf * (fx + (int64_t)NXf * fz);
                a0 += w * rf[3 * f];
                a1 += w * rf[3 * f + 1];
                a2 += w * rf[3 * f + 2];
            }
        }
    }
    rc[3 * n] = a0;
    rc[3 * n + 1] = a1;
    rc[3 * n + 2] = a2;
}

// Span 2: lanes along y, 32-bit indices (grids below 2^31 / 3 nodes).  A coarse
// node outside the active domain (cflag) gets 0 without reading the fine grid: all
// 8 coarse elements around it are empty, so every fine node strictly inside
// their union -- the tent's support -- is inactive and holds 0.
//
// FP32: a thread per coarse node.  Taps are read at clamped positions, those past
// the grid with weight 0, so that no branch stands between the 81 loads: with one
// per tap row they went out row by row, nine memory latencies one after the other
// (384 x 192 x 192 blobs, finest level: 29.6 -> 25.0 us).  Inactive coarse nodes
// are not written: the FP32 V-cycle's coarse vectors are zeroed when allocated.
// a += the 27 taps of coarse node (I, J, K)
__device__ __forceinline__ void restrict2_taps(const float *__restrict__ rf, int I, int J, int K, int nyf, int nxf, int nzf,
                                               float (&a)[3]) {
    // offsets and weights of the three taps of each axis
    int o[3][3];
    float w[3][3];
    const int c[3] = {I, J, K}, m[3] = {nyf, nxf, nzf}, st[3] = {3, 3 * (nyf + 1), 3 * (nyf + 1) * (nxf + 1)};
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        o[ax][1] = st[ax] * 2 * c[ax];
        o[ax][0] = c[ax] > 0 ? o[ax][1] - st[ax] : o[ax][1];
        o[ax][2] = 2 * c[ax] < m[ax] ? o[ax][1] + st[ax] : o[ax][1];
        w[ax][1] = 1.f;
        w[ax][0] = c[ax] > 0 ? 0.5f : 0.f;
        w[ax][2] = 2 * c[ax] < m[ax] ? 0.5f : 0.f;
    }
#pragma unroll
    for (int dz = 0; dz < 3; ++dz) {
        float v[3][3][3];
#pragma unroll
        for (int dx = 0; dx < 3; ++dx)
#pragma unroll
            for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                for (int q = 0; q < 3; ++q) v[dx][dy][q] = rf[o[0][dy] + o[1][dx] + o[2][dz] + q];
        // y, then x, then z
        float p[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int dx = 0; dx < 3; ++dx)
#pragma unroll
            for (int q = 0; q < 3; ++q)
                p[q] += w[1][dx] * (v[dx][1][q] + (w[0][0] * v[dx][0][q] + w[0][2] * v[dx][2][q]));
#pragma unroll
        for (int q = 0; q < 3; ++q) a[q] += w[2][dz] * p[q];
    }
}

__global__ void __launch_bounds__(128) k_restrict2_f32(const float *__restrict__ rf, float *__restrict__ rc,
                                                       const uint8_t *__restrict__ cflag, int nyc, int nxc, int nzc,
                                                       int keep_zeros) {
    const int NYc = nyc + 1, NXc = nxc + 1;
    const int pl = blockIdx.x * blockDim.x + threadIdx.x;
    if (pl >= NYc * NXc) return;
    const int n = 3 * (pl + NYc * NXc * blockIdx.y);
    if (!(cflag[n / 3] & NF_ACTIVE)) {
        if (!keep_zeros) rc[n] = rc[n + 1] = rc[n + 2] = 0.f;
        return;
    }
    float a[3] = {0.f, 0.f, 0.f};
    restrict2_taps(rf, pl % NYc, pl / NYc, (int)blockIdx.y, 2 * nyc, 2 * nxc, 2 * nzc, a);
#pragma unroll
    for (int q = 0; q < 3; ++q) rc[n + q] = a[q];
}

// FP64 is bound by its operations: a thread takes zp coarse planes of a column and
// forms the sum over a fine plane's 9 taps once, as the plane between two coarse
// planes serves both: 54 operations and 18 taps per node instead of 81 and 27
// (256 x 128 x 128, finest level: 89 -> 75 us).
__global__ void __launch_bounds__(128) k_restrict2_f64(const double *__restrict__ rf, double *__restrict__ rc,
                                                       const uint8_t *__restrict__ cflag, int nyc, int nxc, int nzc,
                                                       int zp) {
    using T = double;
    const int NYc = nyc + 1, NXc = nxc + 1;
    const int NYf = 2 * nyc + 1, NXf = 2 * nxc + 1;
    const int pl = blockIdx.x * blockDim.x + threadIdx.x;
    if (pl >= NYc * NXc) return;
    const int I = pl % NYc, J = pl / NYc;
    const bool y0 = I > 0, y1 = I < nyc, x0 = J > 0, x1 = J < nxc;
    const int oy[3] = {y0 ? -3 : 0, 0, y1 ? 3 : 0}, ox[3] = {x0 ? -3 * NYf : 0, 0, x1 ? 3 * NYf : 0};
    const int base = 3 * (2 * I + NYf * 2 * J), fplane = 3 * NYf * NXf;
    // half-weighted neighbours along y and x of fine plane z
    auto plane = [&](int z, T (&p)[3]) {
        const T *r = rf + base + fplane * z;
        T v[3][3][3];
#pragma unroll
        for (int dx = 0; dx < 3; ++dx)
#pragma unroll
            for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                for (int q = 0; q < 3; ++q) v[dx][dy][q] = r[oy[dy] + ox[dx] + q];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            T s[3];
#pragma unroll
            for (int dx = 0; dx < 3; ++dx)
                s[dx] = v[dx][1][q] + T(0.5) * ((y0 ? v[dx][0][q] : T(0)) + (y1 ? v[dx][2][q] : T(0)));
            p[q] = s[1] + T(0.5) * ((x0 ? s[0] : T(0)) + (x1 ? s[2] : T(0)));
        }
    };
    const int K0 = blockIdx.y * zp, K1 = min(nzc + 1, K0 + zp);
    T lo[3] = {T(0), T(0), T(0)};
    bool have = K0 == 0;   // lo holds fine plane 2 K - 1
    for (int K = K0; K < K1; ++K) {
        const int n = 3 * (pl + NYc * NXc * K);
        if (!(cflag[n / 3] & NF_ACTIVE)) {
            rc[n] = rc[n + 1] = rc[n + 2] = T(0);
            have = false;
            continue;
        }
        T mid[3], up[3];
        if (!have && K > 0) plane(2 * K - 1, lo);
        plane(2 * K, mid);
        plane(min(2 * K + 1, 2 * nzc), up);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            if (K == nzc) up[q] = T(0);
            rc[n + q] = mid[q] + T(0.5) * ((K > 0 ? lo[q] : T(0)) + up[q]);
            lo[q] = up[q];
        }
        have = true;
    }
}

// Span 4: a warp per coarse node, whose lanes share the 7^3 taps (consecutive
// lanes along fine y).  A non-dyadic hierarchy's first coarse level has 1/64 of
// the fine nodes: a thread per coarse node left a 64 x 32 x 32 grid with 18
// CTAs, each thread walking 343 taps (71 us in FP64, 36 us in FP32 there).  With
// k_prolong_rows4 the FP64 analysis of that grid went from 23.9 to 16.0 ms, the
// mixed one from 10.5 to 6.9 ms.
template <typename T>
__global__ void __launch_bounds__(256) k_restrict4(const T *__restrict__ rf, T *__restrict__ rc,
                                                   const uint8_t *__restrict__ cflag, int nyc, int nxc, int nzc,
                                                   int keep_zeros) {
    constexpr int S = 4, W = 2 * S - 1;
    const int NYc = nyc + 1, NXc = nxc + 1;
    const int NYf = S * nyc + 1, NXf = S * nxc + 1, NZf = S * nzc + 1;
    const int pl = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (pl >= NYc * NXc) return;
    const int I = pl % NYc, J = pl / NYc, Kz = blockIdx.y, n = 3 * (pl + NYc * NXc * Kz);
    if (!(cflag[n / 3] & NF_ACTIVE)) {
        if (!keep_zeros && lane < 3) rc[n + lane] = T(0);
        return;
    }
    T a[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int k = 0; k < (W * W * W + 31) / 32; ++k) {
        const int t = lane + 32 * k, dy = t % W - (S - 1), dx = t / W % W - (S - 1), dz = t / (W * W) - (S - 1);
        const int fy = S * I + dy, fx = S * J + dx, fz = S * Kz + dz;
        if (t < W * W * W && fy >= 0 && fy < NYf && fx >= 0 && fx < NXf && fz >= 0 && fz < NZf) {
            const T w = T((S - abs(dy)) * (S - abs(dx)) * (S - abs(dz))) * (T(1) / T(S * S * S));
            const T *r = rf + 3 * (fy + NYf * (fx + NXf * fz));
#pragma unroll
            for (int c = 0; c < 3; ++c) a[c] += w * r[c];
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) a[c] += __shfl_xor_sync(0xffffffffu, a[c], o);
    if (lane < 3) rc[n + lane] = lane == 0 ? a[0] : lane == 1 ? a[1] : a[2];
}

template <typename T>
void launch_restrict(const Level &fine, const Level &coarse, const T *rf, T *rc, cudaStream_t st) {
    ++g_launches;
    const dim3 g((unsigned)(((coarse.ny + 1) * (coarse.nx + 1) + 127) / 128), (unsigned)(coarse.nz + 1));
    const bool small = 3 * (int64_t)fine.nnode < (int64_t)INT32_MAX;
    // FP32: the coarse vectors (the levels' r32) are zeroed at allocation and keep zeros at
    // inactive nodes
    const int keep = sizeof(T) == sizeof(float) && static_cast<const void *>(rc) == coarse.r32;
    if (small && coarse.span == 2) {
        if constexpr (sizeof(T) == sizeof(float)) {
            k_restrict2_f32<<<g, 128, 0, st>>>(rf, rc, coarse.nflag, coarse.ny, coarse.nx, coarse.nz, keep);
        } else {
            // 8 (else 4, 2, 1) coarse planes per CTA while that keeps 8 CTAs per SM
            int zp = 8;
            while (zp > 1 && (int64_t)g.x * ((coarse.nz + zp) / zp) < 152 * 8) zp >>= 1;
            k_restrict2_f64<<<dim3(g.x, (unsigned)((coarse.nz + zp) / zp)), 128, 0, st>>>(
                rf, rc, coarse.nflag, coarse.ny, coarse.nx, coarse.nz, zp);
        }
    } else if (small && coarse.span == 4)
        k_restrict4<T><<<dim3((unsigned)(((coarse.ny + 1) * (coarse.nx + 1) + 7) / 8), g.y), 256, 0, st>>>(
            rf, rc, coarse.nflag, coarse.ny, coarse.nx, coarse.nz, keep);
    else
        k_restrict<T><<<g, 128, 0, st>>>(rf, rc, coarse.ny, coarse.nx, coarse.nz, coarse.span);
}
template void launch_restrict<double>(const Level &, const Level &, const double *, double *, cudaStream_t);
template void launch_restrict<float>(const Level &, const Level &, const float *, float *, cudaStream_t);

// warp stage in the kernel's precision T, the warp sums added in FP64
template <typename T>
__device__ __forceinline__ double warp_block_sum(T v, double *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) red[w] = (double)v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += red[i];
    return s;
}

// x_f = r_f .* D + P x_c on active fine nodes, 0 elsewhere, where D holds 2 omega
// over the Jacobi diagonal.
// FINAL (finest level): fixed DOFs set to 0 and partial sums of x_f . r_f.
template <typename T, bool FINAL>
__global__ void k_prolong_smooth(const T *__restrict__ xc, const T *__restrict__ rf, const T *__restrict__ D,
                                 const uint8_t *__restrict__ nflag, T *__restrict__ xf, int nyc, int nxc,
                                 int nzc, int s, double *__restrict__ partial) {
    const int NYc = nyc + 1, NXc = nxc + 1;
    const int NYf = s * nyc + 1, NXf = s * nxc + 1, NZf = s * nzc + 1;
    // grid: x over the (y, x) plane of fine nodes, y over z (32-bit index math)
    const int pl = blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t n = (int64_t)pl + (int64_t)NYf * NXf * blockIdx.y;
    T dot = T(0);
    (void)NZf;
    if (pl < NYf * NXf) {
        const uint8_t f = nflag[n];
        T o0 = T(0), o1 = T(0), o2 = T(0);
        if (f & NF_ACTIVE) {
            const int iy = pl % NYf, ix = pl / NYf, iz = blockIdx.y;
            const int I = iy / s, J = ix / s, Kz = iz / s;
            const int ry = iy - s * I, rx = ix - s * J, rz = iz - s * Kz;
            const T inv = T(1) / T(s);
            const T wy[2] = {T(s - ry) * inv, T(ry) * inv};
            const T wx[2] = {T(s - rx) * inv, T(rx) * inv};
            const T wz[2] = {T(s - rz) * inv, T(rz) * inv};
            T p0 = T(0), p1 = T(0), p2 = T(0);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (c && rz == 0) continue;
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    if (b && rx == 0) continue;
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
                        if (a && ry == 0) continue;
                        const T w = wy[a] * wx[b] * wz[c];
                        const int64_t m = (int64_t)(I + a) + (int64_t)NYc * ((J + b) + (int64_t)NXc * (Kz + c));
                        p0 += w * xc[3 * m];
                        p1 += w * xc[3 * m + 1];
                        p2 += w * xc[3 * m + 2];
                    }
                }
            }
            const T r0 = rf[3 * n], r1 = rf[3 * n + 1], r2 = rf[3 * n + 2];
            o0 = r0 * D[3 * n] + p0;
            o1 = r1 * D[3 * n + 1] + p1;
            o2 = r2 * D[3 * n + 2] + p2;
            if (FINAL) {
                if (f & NF_FIXX) o0 = T(0);
                if (f & NF_FIXY) o1 = T(0);
                if (f & NF_FIXZ) o2 = T(0);
                dot = o0 * r0 + o1 * r1 + o2 * r2;
            }
        }
        xf[3 * n] = o0;
        xf[3 * n + 1] = o1;
        xf[3 * n + 2] = o2;
    }
    if (FINAL && partial) {
        __shared__ double red[8];
        const double sum = warp_block_sum<T>(dot, red);
        if (threadIdx.x == 0) partial[blockIdx.x + gridDim.x * blockIdx.y] = sum;
    }
}

// Span 2: a thread per coarse node (I, J, K) writing the fine nodes (2 I + ry, 2 J +
// rx, 2 K + rz), 0 <= ry, rx, rz < 2 (only 0 past the last coarse cell of an
// axis): the 8 coarse corners are loaded once per 8 fine nodes, the upper 4 of
// a plane are the lower 4 of the next (a CTA marches through zp planes), and the
// interpolation is sums of 1, 2, 4 or 8 corners, axis by axis, scaled once.
// Indices are 32-bit.  Same result as k_prolong_smooth up to the order of the sums.
// All of a batch's loads (r, 2 omega / D and flags of the cell's 8 fine nodes in FP32, of
// 4 in FP64) are issued before the first is used, at clamped positions for the
// nodes past the grid; with a branch around each fine node they went out node by
// node, eight memory latencies per cell.  Finest level: FP32 384 x 192 x 192 blobs 76 ->
// 53 us, FP64 (bound by its operations, 13.5 per node instead of 33) 256 x 128 x 128
// 247 -> 131 us.
// With cflag (the coarse node flags; passed for the FP32 V-cycle, whose output
// vectors are zeroed when allocated), a thread whose 8 coarse corners are all
// inactive writes nothing: every fine element touching one of its fine nodes
// lies in a coarse element sharing a corner with the cell, and an active
// coarse element makes all 8 of its corners active, so those fine nodes are
// inactive and already hold 0.
template <typename T, bool FINAL>
__global__ void __launch_bounds__(128) k_prolong_cells(const T *__restrict__ xc, const T *__restrict__ rf,
                                                       const T *__restrict__ D, const uint8_t *__restrict__ nflag,
                                                       const uint8_t *__restrict__ cflag,
                                                       T *__restrict__ xf, int nyc, int nxc, int nzc, int zp,
                                                       double *__restrict__ partial) {
    constexpr int BZ = sizeof(T) == 4 ? 2 : 1;   // fine planes per batch of loads
    const int NYc = nyc + 1, NXc = nxc + 1;
    const int NYf = 2 * nyc + 1, NXf = 2 * nxc + 1;
    const int pl = blockIdx.x * blockDim.x + threadIdx.x;
    T dot = T(0);
    if (pl < NYc * NXc) {
        const int I = pl % NYc, J = pl / NYc;
        const int ly = I < nyc, lx = J < nxc;   // the cell has fine nodes at ry = 1, rx = 1
        const int cpl = NYc * NXc, fpl = NYf * NXf;
        // coarse corners of the cell's column: index b (x) 2 + a (y)
        const int co[4] = {pl, pl + ly, pl + (lx ? NYc : 0), pl + ly + (lx ? NYc : 0)};
        auto plane_active = [&](int K) {
            bool any = false;
            if (K <= nzc)
#pragma unroll
                for (int k = 0; k < 4; ++k) any |= (cflag[co[k] + cpl * K] & NF_ACTIVE) != 0;
            return any;
        };
        const int K0 = blockIdx.y * zp, K1 = min(nzc + 1, K0 + zp);
        bool act0 = cflag ? plane_active(K0) : true, act1 = cflag ? plane_active(K0 + 1) : true;
        T c0[4][3], c1[4][3];
        bool have = false;   // c0 holds plane K
        for (int K = K0; K < K1; ++K) {
            const bool live = act0 || act1;
            act0 = act1;
            if (cflag) act1 = plane_active(K + 2);
            if (!live) {
                have = false;
                continue;
            }
            const int lz = K < nzc, up = lz ? cpl : 0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    if (!have) c0[k][q] = xc[3 * (co[k] + cpl * K) + q];
                    c1[k][q] = xc[3 * (co[k] + cpl * K + up) + q];
                }
            const int f00 = 2 * I + NYf * 2 * J + fpl * 2 * K;
#pragma unroll
            for (int z0 = 0; z0 < 2; z0 += BZ) {
                T r[BZ][2][2][3], dg[BZ][2][2][3];
                uint8_t fl[BZ][2][2];
#pragma unroll
                for (int z = 0; z < BZ; ++z)
#pragma unroll
                    for (int x = 0; x < 2; ++x)
#pragma unroll
                        for (int y = 0; y < 2; ++y) {
                            const int f = f00 + (y && ly ? 1 : 0) + (x && lx ? NYf : 0) + (z0 + z && lz ? fpl : 0);
                            fl[z][x][y] = nflag[f];
#pragma unroll
                            for (int q = 0; q < 3; ++q) {
                                r[z][x][y][q] = rf[3 * f + q];
                                dg[z][x][y][q] = D[3 * f + q];
                            }
                        }
#pragma unroll
                for (int z = 0; z < BZ; ++z) {
                    const int rz = z0 + z;
                    if (rz && !lz) break;
                    T qz[4][3];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int q = 0; q < 3; ++q) qz[k][q] = rz ? c0[k][q] + c1[k][q] : c0[k][q];
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        if (x && !lx) break;
                        T qx[2][3];
#pragma unroll
                        for (int a = 0; a < 2; ++a)
#pragma unroll
                            for (int q = 0; q < 3; ++q) qx[a][q] = x ? qz[a][q] + qz[2 + a][q] : qz[a][q];
#pragma unroll
                        for (int y = 0; y < 2; ++y) {
                            if (y && !ly) break;
                            const int f = f00 + y + NYf * x + fpl * rz;
                            const T scale = T(1) / T((1 + rz) * (1 + x) * (1 + y));
                            const bool act = (fl[z][x][y] & NF_ACTIVE) != 0;
                            T o[3];
#pragma unroll
                            for (int q = 0; q < 3; ++q) {
                                const T p = y ? qx[0][q] + qx[1][q] : qx[0][q];
                                o[q] = act ? r[z][x][y][q] * dg[z][x][y][q] + scale * p : T(0);
                                if (FINAL && (fl[z][x][y] & (NF_FIXX << q))) o[q] = T(0);
                            }
                            if (FINAL && act)
                                dot += o[0] * r[z][x][y][0] + o[1] * r[z][x][y][1] + o[2] * r[z][x][y][2];
                            // inactive nodes of an output that keeps zeros there (cflag set) are not rewritten
                            if (act || !cflag) {
#pragma unroll
                                for (int q = 0; q < 3; ++q) xf[3 * f + q] = o[q];
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int q = 0; q < 3; ++q) c0[k][q] = c1[k][q];
            have = true;
        }
    }
    if (FINAL && partial) {
        __shared__ double red[4];
        const double sum = warp_block_sum<T>(dot, red);
        if (threadIdx.x == 0) partial[blockIdx.x + gridDim.x * blockIdx.y] = sum;
    }
}

// Span 4: a thread per fine column (fx, fz) and coarse cell along y, writing
// the cell's 4 fine nodes of that column.  Same operator as k_prolong_cells, whose
// thread per coarse cell walks 64 fine nodes and left a 64 x 32 x 32 grid with 18
// CTAs (73 us in FP64, 28 us in FP32 there).
// keep_zeros: inactive nodes of xf hold 0 and are not written.
template <typename T, bool FINAL>
__global__ void __launch_bounds__(128) k_prolong_rows4(const T *__restrict__ xc, const T *__restrict__ rf,
                                                       const T *__restrict__ D, const uint8_t *__restrict__ nflag,
                                                       T *__restrict__ xf, int nyc, int nxc, int nzc,
                                                       int keep_zeros, double *__restrict__ partial) {
    constexpr int S = 4;
    const int NYc = nyc + 1, NXc = nxc + 1, NYf = S * nyc + 1, NXf = S * nxc + 1;
    const int pl = blockIdx.x * blockDim.x + threadIdx.x;
    T dot = T(0);
    if (pl < NYc * NXf) {
        const int I = pl % NYc, fx = pl / NYc, fz = blockIdx.y;
        const int J = fx / S, rx = fx % S, K = fz / S, rz = fz % S;
        const int f0 = S * I + NYf * (fx + NXf * fz), ly = I < nyc ? S : 1;
        uint8_t fl[S];
        T r[S][3], dg[S][3];
        bool any = false;
        // r and D are loaded whatever the flags say, so that they do not wait for them
#pragma unroll
        for (int k = 0; k < S; ++k) {
            fl[k] = k < ly ? nflag[f0 + k] : 0;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                r[k][q] = k < ly ? rf[3 * (f0 + k) + q] : T(0);
                dg[k][q] = k < ly ? D[3 * (f0 + k) + q] : T(0);
            }
        }
#pragma unroll
        for (int k = 0; k < S; ++k) any |= (fl[k] & NF_ACTIVE) != 0;
        T qa[2][3] = {};
        if (any) {
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    if ((c && rz == 0) || (b && rx == 0)) continue;
                    const T w = T((c ? rz : S - rz) * (b ? rx : S - rx)) * (T(1) / T(S * S));
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
                        if (a && I == nyc) continue;
                        const T *x = xc + 3 * ((I + a) + NYc * ((J + b) + NXc * (K + c)));
#pragma unroll
                        for (int q = 0; q < 3; ++q) qa[a][q] += w * x[q];
                    }
                }
        }
#pragma unroll
        for (int k = 0; k < S; ++k) {
            if (k >= ly) break;
            const bool act = (fl[k] & NF_ACTIVE) != 0;
            T o[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                o[q] = act ? r[k][q] * dg[k][q] + (T(S - k) / T(S) * qa[0][q] + T(k) / T(S) * qa[1][q]) : T(0);
                if (FINAL && (fl[k] & (NF_FIXX << q))) o[q] = T(0);
            }
            if (FINAL && act) dot += o[0] * r[k][0] + o[1] * r[k][1] + o[2] * r[k][2];
            if (act || !keep_zeros) {
#pragma unroll
                for (int q = 0; q < 3; ++q) xf[3 * (f0 + k) + q] = o[q];
            }
        }
    }
    if (FINAL && partial) {
        __shared__ double red[4];
        const double sum = warp_block_sum<T>(dot, red);
        if (threadIdx.x == 0) partial[blockIdx.x + gridDim.x * blockIdx.y] = sum;
    }
}

template <typename T>
void launch_prolong_smooth(const Level &fine, const Level &coarse, const T *xc, const T *rf, const T *diag,
                           T *xf, bool final_level, double *partial_dot, int *nblocks_out, cudaStream_t st) {
    const bool small = 3 * (int64_t)fine.nnode < (int64_t)INT32_MAX;
    // empty cells are skipped in FP32 only: the FP32 V-cycle's outputs (d_z32 and the
    // levels' x32) are zeroed at allocation, so their inactive nodes hold 0 throughout
    const bool skip_inactive = sizeof(T) == sizeof(float);
    if (small && coarse.span == 4) {
        const dim3 g((unsigned)(((coarse.ny + 1) * (int64_t)(fine.nx + 1) + 127) / 128), (unsigned)(fine.nz + 1));
        if (nblocks_out) *nblocks_out = (int)(g.x * g.y);
        ++g_launches;
        if (final_level)
            k_prolong_rows4<T, true><<<g, 128, 0, st>>>(xc, rf, diag, fine.nflag, xf, coarse.ny, coarse.nx,
                                                        coarse.nz, skip_inactive, partial_dot);
        else
            k_prolong_rows4<T, false><<<g, 128, 0, st>>>(xc, rf, diag, fine.nflag, xf, coarse.ny, coarse.nx,
                                                         coarse.nz, skip_inactive, nullptr);
        return;
    }
    if (small && coarse.span == 2) {
        // 8 (else 4) coarse planes per CTA while that keeps at least 8 CTAs per SM
        const int64_t plane_ctas = ((coarse.ny + 1) * (int64_t)(coarse.nx + 1) + 127) / 128;
        int zp = 8;
        while (zp > 1 && plane_ctas * ((coarse.nz + zp) / zp) < 152 * 8) zp >>= 1;
        const dim3 g((unsigned)plane_ctas, (unsigned)((coarse.nz + zp) / zp));
        if (nblocks_out) *nblocks_out = (int)(g.x * g.y);
        ++g_launches;
        const uint8_t *cflag = skip_inactive ? coarse.nflag : nullptr;
        if (final_level)
            k_prolong_cells<T, true><<<g, 128, 0, st>>>(xc, rf, diag, fine.nflag, cflag, xf, coarse.ny,
                                                           coarse.nx, coarse.nz, zp, partial_dot);
        else
            k_prolong_cells<T, false><<<g, 128, 0, st>>>(xc, rf, diag, fine.nflag, cflag, xf, coarse.ny,
                                                            coarse.nx, coarse.nz, zp, nullptr);
        return;
    }
    const dim3 nb((unsigned)(((fine.ny + 1) * (fine.nx + 1) + 255) / 256), (unsigned)(fine.nz + 1));
    if (nblocks_out) *nblocks_out = (int)(nb.x * nb.y);
    ++g_launches;
    if (final_level)
        k_prolong_smooth<T, true><<<nb, 256, 0, st>>>(xc, rf, diag, fine.nflag, xf, coarse.ny, coarse.nx,
                                                      coarse.nz, coarse.span, partial_dot);
    else
        k_prolong_smooth<T, false><<<nb, 256, 0, st>>>(xc, rf, diag, fine.nflag, xf, coarse.ny, coarse.nx,
                                                       coarse.nz, coarse.span, nullptr);
}
template void launch_prolong_smooth<double>(const Level &, const Level &, const double *, const double *,
                                            const double *, double *, bool, double *, int *, cudaStream_t);
template void launch_prolong_smooth<float>(const Level &, const Level &, const float *, const float *, const float *,
                                           float *, bool, double *, int *, cudaStream_t);

// ---- the FP32 V-cycle's small levels -----------------------------------------
// A launch on a level of a few thousand nodes costs a memory latency and its place in
// the chain of launches, about 4 us, whatever it computes.  The cycle is additive and
// its levels are nested by factors of 2 (4 below the finest of a non-dyadic hierarchy), so
// the chains collapse:
//   * the product of restrictions is the tent of span 4, 8, so that up to three
//     coarser residuals are formed from one level's in one launch;
//   * trilinear interpolation through the levels in between is trilinear interpolation
//     on each level's own cell, so a thread that prolongates to 8 fine nodes carries
//     the 8 corners of its cell down from the coarsest level, adding r (2 omega / D) on
//     the way; the levels in between are not written at all.
// The sums are those of the level-by-level launches in another order.  FP32 V-cycle, us:
// 96 x 48 x 48 51 -> 37, 125 x 61 x 67 blob shape 55 -> 48, 192 x 96 x 96 65 -> 50, 384 x 192 x 192
// 160 -> 140, 256 x 128 x 128 134 -> 123; non-dyadic 64 x 32 x 32 33 -> 25.

// S-fold restriction at coarse node (I, J, K) by 2 S NX threads: 2 S lanes along y (one
// idle), NX groups along x, each of which takes 2 S / NX columns through z.  Taps are read at
// clamped positions, those past the grid with weight 0; position and weight along y
// and x are formed once, so that a tap is its three loads and a few operations.  (With the
// taps numbered through and taken apart one by one, the 192 x 96 x 96 shape's launch took
// 12.3 us, now 9.5.)
template <int S, int NX>
__device__ __forceinline__ void restrict_chain_taps(const float *__restrict__ rf, int I, int J, int K, int nyf, int nxf,
                                                    int nzf, int t, float (&a)[3]) {
    constexpr int H = 2 * S / NX;
    const int dy = t % (2 * S) - (S - 1), y = S * I + dy, cy = min(max(y, 0), nyf);
    const int NYf = nyf + 1, plane = 3 * NYf * (nxf + 1);
    int off[H];
    float w[H];
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const int dx = t / (2 * S) + NX * h - (S - 1), x = S * J + dx, cx = min(max(x, 0), nxf);
        off[h] = 3 * (cy + NYf * cx);
        w[h] = cy == y && cx == x ? (float)((S - abs(dy)) * (S - abs(dx))) : 0.f;   // 0 at S as well
    }
#pragma unroll
    for (int dz = 1 - S; dz < S; ++dz) {
        const int z = S * K + dz, cz = min(max(z, 0), nzf);
        const float wz = cz == z ? (float)(S - abs(dz)) : 0.f;
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const float *r = rf + off[h] + plane * cz;
#pragma unroll
            for (int c = 0; c < 3; ++c) a[c] = fmaf(w[h] * wz, r[c], a[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) a[c] *= 1.f / (float)(S * S * S);
}

// target k is the level 2, 4, 8 times coarser than the base (k = 0, 1, 2; a base whose next
// level is 4 times coarser has no target 0); CTAs in the order 2, 1, 0 (the longest sums first)
struct RestrictChain {
    int k0, k1;                        // the first and the last target
    int ny[4], nx[4], nz[4];           // [0] the base, [1 + k] target k
    const uint8_t *flag[3];
    float *out[3];
    int first[3];                      // the target's first CTA
};

__global__ void __launch_bounds__(128) k_restrict_chain(const float *__restrict__ rf,
                                                        const __grid_constant__ RestrictChain c) {
    const int b = blockIdx.x, lane = threadIdx.x & 31;
    int k = c.k0;
    while (k < c.k1 && b < c.first[k]) ++k;
    const int per = k == 0 ? 128 : k == 1 ? 4 : 1;   // coarse nodes per CTA: a thread, a warp, a CTA for each
    const int i = (b - c.first[k]) * per + (k == 0 ? (int)threadIdx.x : k == 1 ? (int)(threadIdx.x >> 5) : 0);
    const int NY = c.ny[1 + k] + 1, NX = c.nx[1 + k] + 1;
    if (i >= NY * NX * (c.nz[1 + k] + 1)) return;
    if (!(c.flag[k][i] & NF_ACTIVE)) return;          // holds 0 since it was allocated
    const int I = i % NY, J = i / NY % NX, K = i / (NY * NX);
    float a[3] = {0.f, 0.f, 0.f};
    float *out = c.out[k] + 3 * i;
    if (k == 0) {
        restrict2_taps(rf, I, J, K, c.ny[0], c.nx[0], c.nz[0], a);
#pragma unroll
        for (int q = 0; q < 3; ++q) out[q] = a[q];
        return;
    }
    if (k == 1)
        restrict_chain_taps<4, 4>(rf, I, J, K, c.ny[0], c.nx[0], c.nz[0], lane, a);
    else
        restrict_chain_taps<8, 8>(rf, I, J, K, c.ny[0], c.nx[0], c.nz[0], (int)threadIdx.x, a);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < 3; ++q) a[q] += __shfl_xor_sync(0xffffffffu, a[q], o);
    if (k == 1) {
        if (lane < 3) out[lane] = lane == 0 ? a[0] : lane == 1 ? a[1] : a[2];
        return;
    }
    __shared__ float red[4][3];
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 3; ++q) red[threadIdx.x >> 5][q] = a[q];
    __syncthreads();
    if (threadIdx.x < 3) {
        const int q = threadIdx.x;
        out[q] = (red[0][q] + red[1][q]) + (red[2][q] + red[3][q]);
    }
}

// levels by distance from the output's: [0] the next coarser one, [M] the coarsest, whose
// solution x is given; r and D of the M levels in between
template <int M>
struct ProlongChain {
    int ny[M + 1], nx[M + 1], nz[M + 1];
    const float *r[M], *D[M], *x;
};

// corners of a cell's half along one axis: index bit `step` of v, half b
__device__ __forceinline__ void half_cell(float (&v)[8], int step, int b) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (k & step) continue;
        const float lo = v[k], hi = v[k | step], mid = 0.5f * (lo + hi);
        v[k] = b ? mid : lo;
        v[k | step] = b ? hi : mid;
    }
}

// v: x of the next coarser level at the corners of its cell (I, J, K), component q, corner
// k = y | x << 1 | z << 2; positions past the grid repeat the last node.  A corner that no
// active fine node depends on may hold anything finite.
template <int M>
__device__ __forceinline__ void chain_corners(const ProlongChain<M> &c, int I, int J, int K, float (&v)[3][8]) {
    float cr[M][8][3];
#pragma unroll
    for (int l = 0; l <= M; ++l) {
        const int y = I >> l, x = J >> l, z = K >> l, NY = c.ny[l] + 1, NP = NY * (c.nx[l] + 1);
        const int n = y + NY * x + NP * z;
        const int oy = y < c.ny[l] ? 1 : 0, ox = x < c.nx[l] ? NY : 0, oz = z < c.nz[l] ? NP : 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int m = 3 * (n + (k & 1 ? oy : 0) + (k & 2 ? ox : 0) + (k & 4 ? oz : 0));
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                if (l == M)
                    v[q][k] = c.x[m + q];
                else
                    cr[l][k][q] = c.r[l][m + q] * c.D[l][m + q];
            }
        }
    }
#pragma unroll
    for (int l = M - 1; l >= 0; --l)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            half_cell(v[q], 1, I >> l & 1);
            half_cell(v[q], 2, J >> l & 1);
            half_cell(v[q], 4, K >> l & 1);
#pragma unroll
            for (int k = 0; k < 8; ++k) v[q][k] += cr[l][k][q];
        }
}

// x_f = r_f .* D + P x_c as k_prolong_cells, a thread per node of the next coarser level
template <int M, bool FINAL>
__global__ void __launch_bounds__(128) k_prolong_chain(const __grid_constant__ ProlongChain<M> c,
                                                       const float *__restrict__ rf, const float *__restrict__ D,
                                                       const uint8_t *__restrict__ nflag, float *__restrict__ xf,
                                                       double *__restrict__ partial) {
    const int nyc = c.ny[0], nxc = c.nx[0], nzc = c.nz[0];
    const int NYc = nyc + 1, NXc = nxc + 1, NYf = 2 * nyc + 1, NXf = 2 * nxc + 1;
    const int pl = blockIdx.x * blockDim.x + threadIdx.x;
    float dot = 0.f;
    if (pl < NYc * NXc) {
        const int I = pl % NYc, J = pl / NYc, K = blockIdx.y;
        const int ly = I < nyc, lx = J < nxc, lz = K < nzc, fpl = NYf * NXf;
        const int f00 = 2 * I + NYf * 2 * J + fpl * 2 * K;
        // everything that this thread reads, before anything waits for it
        float r[8][3], dg[8][3];
        uint8_t fl[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int f = f00 + ((k & 1) && ly ? 1 : 0) + ((k & 2) && lx ? NYf : 0) + ((k & 4) && lz ? fpl : 0);
            fl[k] = nflag[f];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                r[k][q] = rf[3 * f + q];
                dg[k][q] = D[3 * f + q];
            }
        }
        float v[3][8];
        chain_corners<M>(c, I, J, K, v);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (((k & 1) && !ly) || ((k & 2) && !lx) || ((k & 4) && !lz)) continue;
            const int f = f00 + (k & 1) + (k & 2 ? NYf : 0) + (k & 4 ? fpl : 0);
            const bool act = (fl[k] & NF_ACTIVE) != 0;
            float o[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                float p = 0.f;
#pragma unroll
                for (int m = 0; m < 8; ++m)
                    if ((m & ~k) == 0) p += v[q][m];
                const float scale = 1.f / (float)((k & 1 ? 2 : 1) * (k & 2 ? 2 : 1) * (k & 4 ? 2 : 1));
                o[q] = fmaf(scale, p, r[k][q] * dg[k][q]);
                if (FINAL && (fl[k] & (NF_FIXX << q))) o[q] = 0.f;
            }
            if (act) {   // inactive nodes hold 0
                if (FINAL) dot += o[0] * r[k][0] + o[1] * r[k][1] + o[2] * r[k][2];
#pragma unroll
                for (int q = 0; q < 3; ++q) xf[3 * f + q] = o[q];
            }
        }
    }
    if (FINAL && partial) {
        __shared__ double red[4];
        const double sum = warp_block_sum<float>(dot, red);
        if (threadIdx.x == 0) partial[blockIdx.x + gridDim.x * blockIdx.y] = sum;
    }
}

// the same for a finest level 4 times finer than the next: threads as in k_prolong_rows4
template <int M>
__global__ void __launch_bounds__(128) k_prolong_chain4(const __grid_constant__ ProlongChain<M> c,
                                                        const float *__restrict__ rf, const float *__restrict__ D,
                                                        const uint8_t *__restrict__ nflag, float *__restrict__ xf,
                                                        double *__restrict__ partial) {
    constexpr int S = 4;
    const int nyc = c.ny[0], NYc = nyc + 1, NYf = S * nyc + 1, NXf = S * c.nx[0] + 1;
    const int pl = blockIdx.x * blockDim.x + threadIdx.x;
    float dot = 0.f;
    if (pl < NYc * NXf) {
        const int I = pl % NYc, fx = pl / NYc, fz = blockIdx.y, rx = fx % S, rz = fz % S;
        const int f0 = S * I + NYf * (fx + NXf * fz), ly = I < nyc ? S : 1;
        uint8_t fl[S];
        float r[S][3], dg[S][3];
#pragma unroll
        for (int k = 0; k < S; ++k) {
            const int f = f0 + (k < ly ? k : 0);
            fl[k] = nflag[f];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                r[k][q] = rf[3 * f + q];
                dg[k][q] = D[3 * f + q];
            }
        }
        float v[3][8];
        chain_corners<M>(c, I, fx / S, fz / S, v);
        float qa[2][3] = {};
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
            const float w = (float)((k & 4 ? rz : S - rz) * (k & 2 ? rx : S - rx)) * (1.f / (S * S));
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                qa[0][q] = fmaf(w, v[q][k], qa[0][q]);
                qa[1][q] = fmaf(w, v[q][k + 1], qa[1][q]);
            }
        }
#pragma unroll
        for (int k = 0; k < S; ++k) {
            if (k >= ly || !(fl[k] & NF_ACTIVE)) continue;   // inactive nodes hold 0
            float o[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                o[q] = r[k][q] * dg[k][q] + ((float)(S - k) / S * qa[0][q] + (float)k / S * qa[1][q]);
                if (fl[k] & (NF_FIXX << q)) o[q] = 0.f;
                xf[3 * (f0 + k) + q] = o[q];
            }
            dot += o[0] * r[k][0] + o[1] * r[k][1] + o[2] * r[k][2];
        }
    }
    if (partial) {
        __shared__ double red[4];
        const double sum = warp_block_sum<float>(dot, red);
        if (threadIdx.x == 0) partial[blockIdx.x + gridDim.x * blockIdx.y] = sum;
    }
}

// Nodes of the level that a chained launch starts from (restriction) or ends on
// (prolongation), at most; past them the extra taps and corners cost more than launches:
// the 192 x 96 x 96 blob shape's cycle takes 50 us chained from its second level (233,000 nodes),
// 58 from the third, 71 from the finest (1.8 million).
constexpr int64_t CHAIN_NODES = 300000;

static bool dyadic_below(const std::vector<Level> &lv, int l) {
    for (size_t k = l + 1; k < lv.size(); ++k)
        if (lv[k].span != 2) return false;
    return true;
}

// Residuals of the levels below level b from b's: returns how many levels it did (0: use launch_restrict)
int launch_restrict_chain(const std::vector<Level> &lv, int b, const float *rf, cudaStream_t st) {
    const int L = (int)lv.size();
    if (L - 1 - b < 2 || lv[b].nnode > CHAIN_NODES || !dyadic_below(lv, b + 1)) return 0;
    RestrictChain c;
    c.k0 = lv[b + 1].span == 2 ? 0 : 1;
    if (lv[b + 1].span != 2 << c.k0) return 0;
    c.k1 = std::min(2, c.k0 + L - 2 - b);
    int ctas = 0;
    for (int k = c.k1; k >= c.k0; --k) {
        const Level &l = lv[b + 1 + k - c.k0];
        const int per = k == 0 ? 128 : k == 1 ? 4 : 1;
        c.flag[k] = l.nflag;
        c.out[k] = l.r32;
        c.first[k] = ctas;
        ctas += (int)((l.nnode + per - 1) / per);
        c.ny[1 + k] = l.ny;
        c.nx[1 + k] = l.nx;
        c.nz[1 + k] = l.nz;
    }
    c.ny[0] = lv[b].ny;
    c.nx[0] = lv[b].nx;
    c.nz[0] = lv[b].nz;
    ++g_launches;
    k_restrict_chain<<<ctas, 128, 0, st>>>(rf, c);
    return c.k1 - c.k0 + 1;
}

template <int M>
static void prolong_chain(const std::vector<Level> &lv, int f, const float *rf, float *xf, double *partial, dim3 g,
                          cudaStream_t st) {
    ProlongChain<M> c;
    for (int k = 0; k <= M; ++k) {
        const Level &l = lv[f + 1 + k];
        c.ny[k] = l.ny;
        c.nx[k] = l.nx;
        c.nz[k] = l.nz;
        if (k < M) {
            c.r[k] = l.r32;
            c.D[k] = l.idiag32;
        } else {
            c.x = l.x32;
        }
    }
    if (lv[f + 1].span == 4)
        k_prolong_chain4<M><<<g, 128, 0, st>>>(c, rf, lv[f].idiag32, lv[f].nflag, xf, partial);
    else if (f == 0)
        k_prolong_chain<M, true><<<g, 128, 0, st>>>(c, rf, lv[f].idiag32, lv[f].nflag, xf, partial);
    else
        k_prolong_chain<M, false><<<g, 128, 0, st>>>(c, rf, lv[f].idiag32, lv[f].nflag, xf, nullptr);
}

// x of level f straight from the coarsest level's; false: go level by level
bool launch_prolong_chain(const std::vector<Level> &lv, int f, const float *rf, float *xf, double *partial, int *nblocks,
                          cudaStream_t st) {
    const int M = (int)lv.size() - 2 - f;
    if (M < 1 || M > 3 || lv[f].nnode > CHAIN_NODES || !dyadic_below(lv, f + 1)) return false;
    const Level &l = lv[f + 1];
    if (l.span != 2 && (l.span != 4 || f != 0)) return false;
    const dim3 g = l.span == 4 ? dim3((unsigned)(((l.ny + 1) * (lv[f].nx + 1) + 127) / 128), (unsigned)(lv[f].nz + 1))
                               : dim3((unsigned)(((l.ny + 1) * (l.nx + 1) + 127) / 128), (unsigned)(l.nz + 1));
    if (f == 0 && nblocks) *nblocks = (int)(g.x * g.y);
    ++g_launches;
    if (M == 1)
        prolong_chain<1>(lv, f, rf, xf, partial, g, st);
    else if (M == 2)
        prolong_chain<2>(lv, f, rf, xf, partial, g, st);
    else
        prolong_chain<3>(lv, f, rf, xf, partial, g, st);
    return true;
}

// ---- Jacobi diagonals (src/Solving_AssembleFEAstencil.m:82-121) -------------
// reference corner order j = 1..8 as offsets (dy, dx, dz)
__constant__ int c_cdy[8] = {1, 1, 0, 0, 1, 1, 0, 0};
__constant__ int c_cdx[8] = {0, 1, 1, 0, 0, 1, 1, 0};
__constant__ int c_cdz[8] = {0, 0, 0, 0, 1, 1, 1, 1};
__constant__ double c_dKe[24];

// UNIFORM: all 24 diagonal entries of Ke are equal, as for an isotropic cube, so the sum
// of the 8 moduli times that entry serves all three components: 9 FP64 operations per
// node instead of 24 (256 x 128 x 128: 176 -> 79 us).
template <bool UNIFORM>
__global__ void k_diag_finest(const double *__restrict__ E, const uint8_t *__restrict__ nflag, int ny, int nx, int nz,
                              double *__restrict__ D) {
    const int NY = ny + 1, NX = nx + 1, NZ = nz + 1;
    const int64_t nn = (int64_t)NY * NX * NZ;
    const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (n >= nn) return;
    double d[3] = {0.0, 0.0, 0.0};
    if (nflag[n] & NF_ACTIVE) {
        const int iy = (int)(n % NY), ix = (int)((n / NY) % NX), iz = (int)(n / ((int64_t)NY * NX));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int ey = iy - c_cdy[j], ex = ix - c_cdx[j], ez = iz - c_cdz[j];
            if (ey < 0 || ex < 0 || ez < 0 || ey >= ny || ex >= nx || ez >= nz) continue;
            const double ev = E[(int64_t)ey + (int64_t)ny * (ex + (int64_t)nx * ez)];
            if (UNIFORM) {
                d[0] += ev;
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) d[c] += c_dKe[3 * j + c] * ev;
            }
        }
        if (UNIFORM) d[0] = d[1] = d[2] = d[0] * c_dKe[0];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) D[3 * n + c] = d[c];
}

void launch_diag_finest(const Level &l0, const double *E, const double *Ke, double *diag, cudaStream_t s) {
    double dk[24], mean = 0.0;
    for (int i = 0; i < 24; ++i) {
        dk[i] = Ke[i + 24 * i];
        mean += dk[i] / 24.0;
    }
    bool uniform = true;   // to rounding
    for (int i = 0; i < 24; ++i) uniform = uniform && fabs(dk[i] - mean) <= 1e-15 * fabs(mean);
    if (uniform)
        for (int i = 0; i < 24; ++i) dk[i] = mean;
    cudaMemcpyToSymbolAsync(c_dKe, dk, sizeof dk, 0, cudaMemcpyHostToDevice, s);
    ++g_launches;
    const unsigned nb = (unsigned)((l0.nnode + 255) / 256);
    if (uniform)
        k_diag_finest<true><<<nb, 256, 0, s>>>(E, l0.nflag, l0.ny, l0.nx, l0.nz, diag);
    else
        k_diag_finest<false><<<nb, 256, 0, s>>>(E, l0.nflag, l0.ny, l0.nx, l0.nz, diag);
}

__global__ void k_diag_from_Ks(const double *__restrict__ Ks, const uint8_t *__restrict__ eact,
                               const uint8_t *__restrict__ nflag, int ny, int nx, int nz, double *__restrict__ D) {
    const int NY = ny + 1, NX = nx + 1, NZ = nz + 1;
    const int64_t nn = (int64_t)NY * NX * NZ;
    const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (n >= nn) return;
    double d0 = 0.0, d1 = 0.0, d2 = 0.0;
    if (nflag[n] & NF_ACTIVE) {
        const int iy = (int)(n % NY), ix = (int)((n / NY) % NX), iz = (int)(n / ((int64_t)NY * NX));
        for (int j = 0; j < 8; ++j) {
            const int ey = iy - c_cdy[j], ex = ix - c_cdx[j], ez = iz - c_cdz[j];
            if (ey < 0 || ex < 0 || ez < 0 || ey >= ny || ex >= nx || ez >= nz) continue;
            const int64_t e = (int64_t)ey + (int64_t)ny * (ex + (int64_t)nx * ez);
            if (!eact[e]) continue;
            const double *k = Ks + 576 * e;
            d0 += k[(3 * j) * 25];
            d1 += k[(3 * j + 1) * 25];
            d2 += k[(3 * j + 2) * 25];
        }
    }
    D[3 * n] = d0;
    D[3 * n + 1] = d1;
    D[3 * n + 2] = d2;
}

void launch_diag_from_Ks(const Level &l, double *diag, cudaStream_t s) {
    ++g_launches;
    k_diag_from_Ks<<<(unsigned)((l.nnode + 255) / 256), 256, 0, s>>>(l.Ks, l.eact, l.nflag, l.ny, l.nx, l.nz, diag);
}

// a thread per node: the finest level's three entries are equal, one division then
__global__ void k_inverse_diag(const double *__restrict__ D, const uint8_t *__restrict__ nflag, int64_t nn,
                               double omega2, double *__restrict__ iD, float *__restrict__ iD32) {
    const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (n >= nn) return;
    double v[3] = {0.0, 0.0, 0.0};
    if (nflag[n] & NF_ACTIVE) {
        const double d0 = D[3 * n], d1 = D[3 * n + 1], d2 = D[3 * n + 2];
        v[0] = v[1] = v[2] = omega2 / d0;
        if (d1 != d0) v[1] = omega2 / d1;
        if (d2 != d0) v[2] = omega2 / d2;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        iD[3 * n + c] = v[c];
        iD32[3 * n + c] = (float)v[c];
    }
}

void launch_inverse_diag(const Level &l, double omega, cudaStream_t s) {
    ++g_launches;
    k_inverse_diag<<<(unsigned)((l.nnode + 255) / 256), 256, 0, s>>>(l.diag, l.nflag, l.nnode, 2.0 * omega, l.idiag,
                                                                     l.idiag32);
}

// ---- compact <-> full conversions -------------------------------------------
__global__ void k_scatter_nodes(const int64_t *__restrict__ map, int64_t n, const double *__restrict__ src,
                                double *__restrict__ dst) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= 3 * n) return;
    const int64_t node = i / 3;
    const int c = (int)(i - 3 * node);
    dst[3 * map[node] + c] = src[i];
}
template <int PER>
__global__ void k_gather_rows(const int64_t *__restrict__ map, int64_t n, const double *__restrict__ src,
                              double *__restrict__ dst) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= PER * n) return;
    const int64_t row = i / PER;
    dst[i] = src[PER * map[row] + (i - PER * row)];
}
__global__ void k_scatter_elems(const int64_t *__restrict__ map, int64_t n, const double *__restrict__ src,
                                double *__restrict__ dst) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) dst[map[i]] = src[i];
}

void launch_scatter_nodes(const int64_t *map, int64_t n, const double *compact, double *full, cudaStream_t s) {
    if (n > 0) {
        ++g_launches;
        k_scatter_nodes<<<(unsigned)((3 * n + 255) / 256), 256, 0, s>>>(map, n, compact, full);
    }
}
void launch_gather_rows(const int64_t *map, int64_t n, int per, const double *src, double *dst, cudaStream_t s) {
    if (n <= 0) return;
    const unsigned nb = (unsigned)((per * n + 255) / 256);
    ++g_launches;
    switch (per) {
        case 1: k_gather_rows<1><<<nb, 256, 0, s>>>(map, n, src, dst); break;
        case 3: k_gather_rows<3><<<nb, 256, 0, s>>>(map, n, src, dst); break;
        case 6: k_gather_rows<6><<<nb, 256, 0, s>>>(map, n, src, dst); break;
        default: k_gather_rows<12><<<nb, 256, 0, s>>>(map, n, src, dst); break;
    }
}
void launch_gather_nodes(const int64_t *map, int64_t n, const double *full, double *compact, cudaStream_t s) {
    launch_gather_rows(map, n, 3, full, compact, s);
}
void launch_scatter_elems(const int64_t *map, int64_t n, const double *compact, double *full, cudaStream_t s) {
    if (n > 0) {
        ++g_launches;
        k_scatter_elems<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(map, n, compact, full);
    }
}
void launch_gather_elems(const int64_t *map, int64_t n, const double *full, double *compact, cudaStream_t s) {
    launch_gather_rows(map, n, 1, full, compact, s);
}

// ---- fixed-DOF bookkeeping (src/FEA_SetupVoxelBased.m:13-26) ----------------
__global__ void k_fixed_indicator(const uint8_t *__restrict__ nflag, int64_t nn, double *__restrict__ v) {
    const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const uint8_t f = nflag[n];
    v[3 * n] = (f & NF_FIXX) ? 1.0 : 0.0;
    v[3 * n + 1] = (f & NF_FIXY) ? 1.0 : 0.0;
    v[3 * n + 2] = (f & NF_FIXZ) ? 1.0 : 0.0;
}
void launch_fixed_indicator(const Level &l, double *v, cudaStream_t s) {
    ++g_launches;
    k_fixed_indicator<<<(unsigned)((l.nnode + 255) / 256), 256, 0, s>>>(l.nflag, l.nnode, v);
}
// a coarse DOF is fixed iff the restricted fixed indicator is nonzero
__global__ void k_mark_fixed(uint8_t *__restrict__ nflag, int64_t nn, const double *__restrict__ v) {
    const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (n >= nn) return;
    uint8_t f = nflag[n] & NF_ACTIVE;
    if (v[3 * n] != 0.0) f |= NF_FIXX;
    if (v[3 * n + 1] != 0.0) f |= NF_FIXY;
    if (v[3 * n + 2] != 0.0) f |= NF_FIXZ;
    nflag[n] = f;
}
void launch_mark_fixed(Level &l, const double *restricted, cudaStream_t s) {
    ++g_launches;
    k_mark_fixed<<<(unsigned)((l.nnode + 255) / 256), 256, 0, s>>>(l.nflag, l.nnode, restricted);
}

__global__ void k_mask_fixed(const uint8_t *__restrict__ nflag, int64_t nn, double *__restrict__ v) {
    const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const uint8_t f = nflag[n];
    if (f & NF_FIXX) v[3 * n] = 0.0;
    if (f & NF_FIXY) v[3 * n + 1] = 0.0;
    if (f & NF_FIXZ) v[3 * n + 2] = 0.0;
}
void launch_mask_fixed(const Level &l0, double *v, cudaStream_t s) {
    ++g_launches;
    k_mask_fixed<<<(unsigned)((l0.nnode + 255) / 256), 256, 0, s>>>(l0.nflag, l0.nnode, v);
}

}  // namespace sgld
