// Galerkin coarse-level assembly and the coarsest-level direct solve
// (reference: src/Solving_AssembleFEAstencil.m:7-135 with
// src/MEXfuncs/Solving_AssembleCmptStencilFromFinestLevel.cpp and
// src/MEXfuncs/Solving_AssembleCmptStencilFromNonFinestLevel.cpp).
//
//  * level 2:  Ks_E = sum_q E_q H_q, H_q = P_q' Ke P_q (templates built on the
//    host, q = child position, s^3 of them);
//  * level l>2: Ks_E = sum_q P_q' Ks_q P_q, P_q the trilinear interpolation from
//    the parent's corners to child q's, applied axis by axis;
//  * coarsest: dense K on the free DOFs (in a bandwidth-reducing order),
//    blocked band Cholesky K = L L' and the explicit triangular inverse
//    M = L^-1, captured once into a CUDA graph; each V-cycle applies
//    K^-1 r = M' (M r) as two dense triangular mat-vecs.  The reference
//    applies its sparse Cholesky factor with two triangular solves
//    (src/Solving_Vcycle.m:116-118); M' M gives the same numbers to rounding
//    and turns two sequential solves into parallel mat-vecs.
#include <cooperative_groups.h>
#include <math.h>

#include <atomic>
#include <utility>
#include <vector>

#include "sgld_internal.cuh"
#include "df_arith.cuh"
#include "wide_sum.cuh"

namespace sgld {

// Element matrices are symmetric: the kernels form the 300 entries of the
// upper triangle (row <= col) and mirror them.
__constant__ unsigned char c_pr[300], c_pc[300];

// The table is the same for every context; each device gets it once.
static std::atomic<bool> g_pairs_done[kMaxDevices];

static int current_device() {
    int dev = 0;
    cudaGetDevice(&dev);
    return dev;
}

void forget_asm_tables(int dev) { g_pairs_done[dev] = false; }

static void upload_pairs(cudaStream_t s) {
    std::atomic<bool> &done = g_pairs_done[current_device()];
    if (done) return;
    unsigned char pr[300], pc[300];
    int k = 0;
    for (int col = 0; col < 24; ++col)
        for (int row = 0; row <= col; ++row) {
            pr[k] = (unsigned char)row;
            pc[k] = (unsigned char)col;
            ++k;
        }
    cudaMemcpyToSymbolAsync(c_pr, pr, sizeof pr, 0, cudaMemcpyHostToDevice, s);
    cudaMemcpyToSymbolAsync(c_pc, pc, sizeof pc, 0, cudaMemcpyHostToDevice, s);
    done = true;
}

// ---- coarse element matrices straight from the finest level ------------------
// Ks_E = sum_q E_q H_q over the S^3 finest elements q inside coarse element E,
// with templates H_q = P_q' Ke P_q (P_q: trilinear interpolation from E's
// corners to q's corners; span S = 2 or 4).  Composed trilinear
// interpolation is trilinear, so S = 4 gives the same matrices as two
// Galerkin steps of span 2.  A CTA handles EB consecutive coarse elements;
// thread t owns one upper-triangle entry and keeps EB accumulators.
constexpr int EB = 16;

// The sums run in compensated double-float arithmetic (Dot2 accumulators, at
// the FP32 issue rate): in FP64 the kernel was bound by GB300's FP64 pipe
// (ncu: 99 % busy).  H2 holds the templates as (hi, lo) float pairs; E is
// split on load.
template <int NQ>
__global__ void __launch_bounds__(320) k_asm_templates_df(const double *__restrict__ E,
                                                          const uint8_t *__restrict__ eact_c,
                                                          const float2 *__restrict__ H2, int nyc, int nxc, int nzc,
                                                          double *__restrict__ Ks) {
    constexpr int S = (NQ == 8) ? 2 : 4;
    __shared__ float2 ev[EB][NQ];
    const int64_t nel = (int64_t)nyc * nxc * nzc;
    const int64_t e0 = (int64_t)blockIdx.x * EB;
    const int nyf = S * nyc, nxf = S * nxc;
    for (int idx = threadIdx.x; idx < EB * NQ; idx += blockDim.x) {
        const int k = idx / NQ, q = idx % NQ;
        const int64_t e = e0 + k;
        double v = 0.0;
        if (e < nel && eact_c[e]) {
            const int cy = (int)(e % nyc), cx = (int)((e / nyc) % nxc), cz = (int)(e / ((int64_t)nyc * nxc));
            const int oy = q % S, ox = (q / S) % S, oz = q / (S * S);
            v = E[(int64_t)(S * cy + oy) + (int64_t)nyf * ((S * cx + ox) + (int64_t)nxf * (S * cz + oz))];
        }
        const df d = df_from(v);
        ev[k][q] = make_float2(d.hi, d.lo);
    }
    __syncthreads();
    const int t = threadIdx.x;
    if (t >= 300) return;
    const int r = c_pr[t], c = c_pc[t];
    const int off = r + 24 * c, offt = c + 24 * r;
    dacc acc[EB];
    for (int q = 0; q < NQ; ++q) {
        const float2 h = H2[576 * q + off];
#pragma unroll
        for (int k = 0; k < EB; ++k) acc[k].add(ev[k][q], h);
    }
#pragma unroll
    for (int k = 0; k < EB; ++k) {
        const int64_t e = e0 + k;
        if (e < nel && eact_c[e]) {
            const double v = df_to(acc[k].value());
            Ks[576 * e + off] = v;
            Ks[576 * e + offt] = v;
        }
    }
}

void launch_asm_templates(const Level &coarse, int S, const double *E, const double *H, double *Ks, cudaStream_t s) {
    upload_pairs(s);
    const unsigned nb = (unsigned)((coarse.nel + EB - 1) / EB);
    ++g_launches;
    // the float-pair copy of every template sits (8 + 64) * 576 entries after
    // its FP64 form (setup_templates lays out FP64 span 2, span 4, then the pairs)
    const float2 *H2 = reinterpret_cast<const float2 *>(H + 72 * 576);
    if (S == 2)
        k_asm_templates_df<8><<<nb, 320, 0, s>>>(E, coarse.eact, H2, coarse.ny, coarse.nx, coarse.nz, Ks);
    else
        k_asm_templates_df<64><<<nb, 320, 0, s>>>(E, coarse.eact, H2, coarse.ny, coarse.nx, coarse.nz, Ks);
}

// Jacobi diagonal of a span-2 coarse level without its element matrices:
// diag(N, c) = sum_{coarse elements e around N} sum_q E_q H_q[(3j+c),(3j+c)]
// with j the corner of e at N.
__global__ void k_diag_templates(const double *__restrict__ E, const uint8_t *__restrict__ nflag,
                                 const double *__restrict__ H, int ny, int nx, int nz, double *__restrict__ D) {
    const int NY = ny + 1, NX = nx + 1;
    const int pl = blockIdx.x * blockDim.x + threadIdx.x;
    if (pl >= NY * NX) return;
    const int iy = pl % NY, ix = pl / NY, iz = blockIdx.y;
    const int64_t n = (int64_t)pl + (int64_t)NY * NX * iz;
    double d0 = 0.0, d1 = 0.0, d2 = 0.0;
    if (nflag[n] & NF_ACTIVE) {
        const int cdy[8] = {1, 1, 0, 0, 1, 1, 0, 0}, cdx[8] = {0, 1, 1, 0, 0, 1, 1, 0}, cdz[8] = {0, 0, 0, 0, 1, 1, 1, 1};
        const int nyf = 2 * ny, nxf = 2 * nx;
        for (int j = 0; j < 8; ++j) {
            const int ey = iy - cdy[j], ex = ix - cdx[j], ez = iz - cdz[j];
            if (ey < 0 || ex < 0 || ez < 0 || ey >= ny || ex >= nx || ez >= nz) continue;
            for (int q = 0; q < 8; ++q) {
                const int oy = q & 1, ox = (q >> 1) & 1, oz = q >> 2;
                const double ev = E[(int64_t)(2 * ey + oy) + (int64_t)nyf * ((2 * ex + ox) + (int64_t)nxf * (2 * ez + oz))];
                if (ev == 0.0) continue;
                const double *h = H + 576 * q;
                d0 += ev * h[(3 * j) * 25];
                d1 += ev * h[(3 * j + 1) * 25];
                d2 += ev * h[(3 * j + 2) * 25];
            }
        }
    }
    D[3 * n] = d0;
    D[3 * n + 1] = d1;
    D[3 * n + 2] = d2;
}

void launch_diag_templates(const Level &coarse, const double *E, const double *H2, double *diag, cudaStream_t s) {
    const dim3 g((unsigned)(((coarse.ny + 1) * (coarse.nx + 1) + 255) / 256), (unsigned)(coarse.nz + 1));
    ++g_launches;
    k_diag_templates<<<g, 256, 0, s>>>(E, coarse.nflag, H2, coarse.ny, coarse.nx, coarse.nz, diag);
}

// ---- deeper levels: P_q' Ks_q P_q ---------------------------------------------
// P_q interpolates trilinearly from the parent's corners to child q's (q = oy + 2 ox
// + 4 oz), so it is a product of three 1D steps.  Along an axis, child and parent share
// one corner ("near"); the far corners' values are f_near = a_near, f_far = (a_near +
// a_far) / 2.  Transposed and doubled, a pair gives (2 f_near + f_far, f_far): one
// operation per pair and axis, and 2^-6 at the end for both sides.
// A warp takes a child: lane = row of its symmetric matrix, the three steps along
// the row in registers, a transpose through shared memory, the three steps along
// the column; the 8 children add in a fixed order.  Bound by the FP64 pipe: 72
// operations per lane and child (the walk over W_q's nonzeros by tables in constant
// memory, read at different places by a warp's lanes, took 1.04 ms for the 8192
// elements of level 4 of 256 x 128 x 128; now 0.35).
__global__ void __launch_bounds__(256) k_asm_coarse(const double *__restrict__ Kf, const uint8_t *__restrict__ eact_f,
                                                    const uint8_t *__restrict__ eact_c, int nyc, int nxc, int nzc,
                                                    double *__restrict__ Ks) {
    const int64_t e = blockIdx.x + (int64_t)gridDim.x * blockIdx.y;
    const int64_t nel = (int64_t)nyc * nxc * nzc;
    if (e >= nel || !eact_c[e]) return;
    __shared__ double st[8][24][25];
    const int q = threadIdx.x >> 5, r = threadIdx.x & 31;
    const int o[3] = {(q >> 1) & 1, q & 1, q >> 2};   // the child's half along x, y (rows), z
    const int cy = (int)(e % nyc), cx = (int)((e / nyc) % nxc), cz = (int)(e / ((int64_t)nyc * nxc));
    const int64_t f = (int64_t)(2 * cy + o[1]) + 2 * (int64_t)nyc * ((2 * cx + o[0]) + 2 * (int64_t)nxc * (2 * cz + o[2]));
    const bool on = eact_f[f];   // the warp's child
    // corner near | far: bit 0 = x, 1 = rows, 2 = z (0 = near) -> reference corner j
    auto corner = [&](int k) {
        const int x = (k & 1) ^ o[0], y = ((k >> 1) & 1) ^ o[1], z = (k >> 2) ^ o[2];
        return 4 * z + (y ? x : 3 - x);
    };
    int dofs[8];   // first DOF of the 8 corners in that order
#pragma unroll
    for (int k = 0; k < 8; ++k) dofs[k] = 3 * corner(k);
    auto steps = [](double (&v)[24]) {
#pragma unroll
        for (int ax = 0; ax < 3; ++ax)
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (!(k >> ax & 1))
#pragma unroll
                    for (int c = 0; c < 3; ++c) v[3 * k + c] = fma(2.0, v[3 * k + c], v[3 * (k | 1 << ax) + c]);
    };
    const int mine = r < 24 ? 3 * corner(r / 3) + r % 3 : 0;   // this lane's row, and later column
    double v[24];
    if (on && r < 24) {
        const double *src = Kf + 576 * f + 24 * mine;
#pragma unroll
        for (int i = 0; i < 24; ++i) v[i] = src[dofs[i / 3] + i % 3];
        steps(v);
#pragma unroll
        for (int i = 0; i < 24; ++i) st[q][r][i] = v[i];
    }
    __syncwarp();
    if (r < 24) {
#pragma unroll
        for (int i = 0; i < 24; ++i) v[i] = on ? st[q][i][r] : 0.0;
        if (on) steps(v);
    }
    __syncwarp();
    if (r < 24)
#pragma unroll
        for (int i = 0; i < 24; ++i) st[q][dofs[i / 3] + i % 3][mine] = v[i];
    __syncthreads();
    for (int t = threadIdx.x; t < 300; t += 256) {
        const int row = c_pr[t], col = c_pc[t];
        double sum = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) sum += st[k][row][col];
        sum *= 1.0 / 64.0;
        double *out = Ks + 576 * e;
        out[row + 24 * col] = sum;
        out[col + 24 * row] = sum;
    }
}

void launch_asm_coarse(const Level &coarse, const Level &fine, double *Ks, cudaStream_t s) {
    upload_pairs(s);
    const int64_t nel = coarse.nel;
    const unsigned gx = (unsigned)(nel < 65535 ? nel : 65535);
    const unsigned gy = (unsigned)((nel + gx - 1) / gx);
    ++g_launches;
    k_asm_coarse<<<dim3(gx, gy), 256, 0, s>>>(fine.Ks, fine.eact, coarse.eact, coarse.ny, coarse.nx, coarse.nz, Ks);
}

// ---- coarsest level: dense matrix on the free DOFs ---------------------------
// pos[dof] = row of that DOF in the dense matrix or -1; rows[i] = full DOF of row i.
// A thread per row and (neighbour node, component): it adds the entries of the up to
// 8 elements that hold both nodes, so every matrix entry is written once (a thread
// per row that added its 8 elements' 24 entries one after the other in memory took
// 100 us, now 8).
__global__ void k_coarse_dense(const double *__restrict__ Ks, const uint8_t *__restrict__ eact, int ny, int nx, int nz,
                               const int *__restrict__ rows, const int *__restrict__ pos, int ncf, double *__restrict__ A) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ncf) return;
    const int d = blockIdx.y % 3, nb = blockIdx.y / 3;
    const int ny_ = nb % 3 - 1, nx_ = nb / 3 % 3 - 1, nz_ = nb / 9 - 1;   // offset of the neighbour
    const int NY = ny + 1, NX = nx + 1, NZ = nz + 1;
    const int dof = rows[i], node = dof / 3, c = dof % 3;
    const int iy = node % NY, ix = (node / NY) % NX, iz = node / (NY * NX);
    const int my = iy + ny_, mx = ix + nx_, mz = iz + nz_;
    if (my < 0 || mx < 0 || mz < 0 || my >= NY || mx >= NX || mz >= NZ) return;
    const int p = pos[3 * (my + NY * (mx + NX * mz)) + d];
    if (p < 0) return;
    // reference corner order j: offsets (dy, dx, dz), and back
    const int ady[8] = {1, 1, 0, 0, 1, 1, 0, 0}, adx[8] = {0, 1, 1, 0, 0, 1, 1, 0}, adz[8] = {0, 0, 0, 0, 1, 1, 1, 1};
    double sum = 0.0;
    bool any = false;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int ey = iy - ady[j], ex = ix - adx[j], ez = iz - adz[j];
        const int qy = ady[j] + ny_, qx = adx[j] + nx_, qz = adz[j] + nz_;   // the neighbour's corner
        if (ey < 0 || ex < 0 || ez < 0 || ey >= ny || ex >= nx || ez >= nz) continue;
        if (qy < 0 || qy > 1 || qx < 0 || qx > 1 || qz < 0 || qz > 1) continue;
        const int64_t e = (int64_t)ey + (int64_t)ny * (ex + (int64_t)nx * ez);
        if (!eact[e]) continue;
        const int kk = 4 * qz + (qy ? qx : 3 - qx);
        sum += Ks[576 * e + (3 * j + c) + 24 * (3 * kk + d)];
        any = true;
    }
    if (any) A[(int64_t)i + (int64_t)ncf * p] = sum;
}

void launch_coarse_dense(const Level &lc, int ncf, const int *rows_and_pos, double *A, cudaStream_t s) {
    const int *rows = rows_and_pos;
    const int *pos = rows_and_pos + ncf;
    if (ncf == 0) return;   // every coarsest DOF fixed: nothing to factor
    cudaMemsetAsync(A, 0, sizeof(double) * (size_t)ncf * ncf, s);
    ++g_launches;
    k_coarse_dense<<<dim3((ncf + 127) / 128, 81), 128, 0, s>>>(lc.Ks, lc.eact, lc.ny, lc.nx, lc.nz, rows, pos, ncf, A);
}

// ---- blocked band Cholesky, NB x NB tiles, column-major n x n ------------------
constexpr int NB = 32;

// 1/sqrt(d) in double-float: FP32 seed, two Newton steps y += y (1 - d y^2) / 2
__device__ __forceinline__ df df_rsqrt(df d) {
    df y = {rsqrtf(d.hi), 0.f};
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const df h = df_sub({1.f, 0.f}, df_mul(df_mul(d, y), y));
        y = df_add(y, df_mul(df_mul(y, {0.5f, 0.f}), h));
    }
    return y;
}

// 1/d in double-float: FP32 reciprocal y and its Newton correction y (1 - d y), whose
// factor 1 - d y (about 2^-24) is needed to FP32 accuracy only
__device__ __forceinline__ df df_rcp(df d) {
    const float y = __frcp_rn(d.hi);
    return quick_two_sum(y, __fmul_rn(y, __fmaf_rn(-d.lo, y, __fmaf_rn(-d.hi, y, 1.f))));
}

// One block column of the band Cholesky (4 warps per CTA), in double-float
// arithmetic: GB300's FP64 pipe would serialise the pivot chain (a warp-wide
// FP64 instruction occupies its sub-partition for many cycles).  The matrix
// stays FP64 in memory; tiles are split into (hi, lo) on load.
//   * every CTA factors the 32 x 32 diagonal tile as L D L': row = lane, column
//     4 k + w in register k of warp w.  A step's only exchange is the pivot column,
//     through shared memory: its owner updates the next pivot column first and
//     publishes it, then one barrier.  The registers move down by one every four
//     steps, so the loop stays rolled (unrolled, its code is read once and from
//     far away: 51 us a launch).  A step's serial chain is a reciprocal and two
//     products; the square roots that turn L D L' into the Cholesky factor are
//     taken for all columns at once afterwards.  (With the tile in shared memory, a
//     square root in the chain, branches around the updates and two barriers a step
//     the launch took 30 us; now 15);
//   * CTA 0 writes the factored tile back, unless other CTAs of the launch still have to
//     read the tile as it was (they may start late, beside another stream's work): then it
//     goes to `diag`, and the trailing update's launch puts it in its place;
//   * CTA b > 0 solves CP_RS rows of the band below against it (X = A L^-T):
//     16 lanes per row, two columns per lane in registers, x_q broadcast by a
//     16-wide shuffle.
constexpr int CP_THREADS = 128;
constexpr int CP_RS = 8;

__global__ void __launch_bounds__(CP_THREADS) k_chol_panel(double *A, int n, int k0, int rend, double *diag, int *info) {
    __shared__ float2 T[NB][NB + 1];     // the factor
    __shared__ float2 rd[NB], ld[NB];    // 1 / L[j][j], L[j][j]
    const int t = threadIdx.x, r = t & 31, w = t >> 5;
    const int m = min(NB, n - k0);
    auto get = [](float2 v) -> df { return {v.x, v.y}; };
    df a[NB / 4];
#pragma unroll
    for (int k = 0; k < NB / 4; ++k) {
        const int c = 4 * k + w;
        a[k] = (r < m && c < m && c <= r) ? df_from(A[(int64_t)(k0 + r) + (int64_t)n * (k0 + c)])
                                          : df{r == c ? 1.f : 0.f, 0.f};
    }
    if (w == 0) T[r][0] = make_float2(a[0].hi, a[0].lo);
    __syncthreads();
#pragma unroll 1
    for (int j0 = 0; j0 < NB; j0 += 4) {
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
            const int j = j0 + jj;
            df d = get(T[j][j]);
            const bool bad = !(d.hi > 0.f);
            if (bad) d = {1.f, 0.f};
            if (bad && t == 0 && blockIdx.x == 0 && info) atomicExch(info, k0 + j + 1);
            // row r's multiplier; its column q loses f * (column j's row q)
            const df f = df_mul(get(T[r][j]), df_rcp(d));
            // no condition on q: columns that are done and rows above the diagonal take values
            // that nothing reads, and the eight updates run side by side
            auto update = [&](int k) {
                a[k] = df_sub(a[k], df_mul(f, get(T[min(j0 + 4 * k + w, NB - 1)][j])));
            };
            const int kn = jj < 3 ? 0 : 1;   // the next pivot column's register, in warp (jj + 1) & 3
            update(kn);
            if (w == ((jj + 1) & 3) && j + 1 < NB) T[r][j + 1] = make_float2(a[kn].hi, a[kn].lo);
#pragma unroll
            for (int k = 0; k < NB / 4; ++k)
                if (k != kn) update(k);
            __syncthreads();
        }
#pragma unroll
        for (int k = 0; k + 1 < NB / 4; ++k) a[k] = a[k + 1];
    }
    // L = (L D) D^-1/2, columns over the warps
    df y = {0.f, 0.f}, d = get(T[r][r]);
    if (!(d.hi > 0.f)) d = {1.f, 0.f};
    y = df_rsqrt(d);
    if (w == 0) {
        const df l = df_mul(d, y);
        rd[r] = make_float2(y.hi, y.lo);
        ld[r] = make_float2(l.hi, l.lo);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NB / 4; ++k) {
        const int c = 4 * k + w;
        const df x = df_mul(get(T[r][c]), get(rd[c]));
        T[r][c] = make_float2(x.hi, x.lo);
    }
    __syncthreads();
    if (blockIdx.x == 0) {
        for (int idx = t; idx < NB * NB; idx += CP_THREADS) {
            const int rr = idx & 31, cc = idx >> 5;
            const double v = rr > cc ? df_to(get(T[rr][cc])) : (rr == cc ? df_to(get(ld[rr])) : 0.0);
            if (gridDim.x > 1)
                diag[idx] = v;
            else if (rr < m && cc < m)
                A[(int64_t)(k0 + rr) + (int64_t)n * (k0 + cc)] = v;
        }
        return;
    }
    const int rr = t >> 4, g = t & 15;
    const int row = k0 + NB + (blockIdx.x - 1) * CP_RS + rr;
    const bool live = row < rend;
    df a0 = {0.f, 0.f}, a1 = {0.f, 0.f};
    if (live) {
        if (g < m) a0 = df_from(A[(int64_t)row + (int64_t)n * (k0 + g)]);
        if (g + 16 < m) a1 = df_from(A[(int64_t)row + (int64_t)n * (k0 + g + 16)]);
    }
#pragma unroll 4
    for (int q = 0; q < NB; ++q) {
        const df xq = df_shfl(df_mul(q < 16 ? a0 : a1, get(rd[q])), q & 15, 16);
        // selects, so that no branch stands in the chain
        const df b0 = df_sub(a0, df_mul(xq, get(T[g][q]))), b1 = df_sub(a1, df_mul(xq, get(T[g + 16][q])));
        a0 = g > q ? b0 : (g == q ? xq : a0);
        a1 = g + 16 > q ? b1 : (g + 16 == q ? xq : a1);
    }
    if (live) {
        if (g < m) A[(int64_t)row + (int64_t)n * (k0 + g)] = df_to(a0);
        if (g + 16 < m) A[(int64_t)row + (int64_t)n * (k0 + g + 16)] = df_to(a1);
    }
}


// trailing update A[i,j] -= sum_k A[i,k] A[j,k] over the panel's columns k for
// the band tiles below it: blockIdx.x = tile pair (ii >= jj), blockIdx.y =
// SY_RS-row slice of tile ii (slices spread one pair's work over SMs).  The
// products are summed in double-float; A stays FP64.
constexpr int SY_RS = 8;

__global__ void __launch_bounds__(256) k_syrk_update(double *A, int n, int k0, int jb0, int nbt,
                                                     const double *__restrict__ diag) {
    if (blockIdx.x == 0 && blockIdx.y == 0)   // the panel's diagonal tile, which this launch does not read
        for (int idx = threadIdx.x; idx < NB * NB; idx += 256)
            A[(int64_t)(k0 + (idx & 31)) + (int64_t)n * (k0 + (idx >> 5))] = diag[idx];
    int p = blockIdx.x, ii = 0;
    while (p > ii) {
        p -= ii + 1;
        ++ii;
    }
    const int jj = p;
    const int i0 = (jb0 + ii) * NB + blockIdx.y * SY_RS, j0 = (jb0 + jj) * NB;
    __shared__ float2 Ai[SY_RS][NB + 1], Aj[NB][NB + 1];
    const int t = threadIdx.x;
    const int m = min(NB, n - k0);
    for (int idx = t; idx < NB * NB; idx += 256) {
        const int r = idx & 31, c = idx >> 5;
        const df v = df_from((j0 + r < n && c < m) ? A[(int64_t)(j0 + r) + (int64_t)n * (k0 + c)] : 0.0);
        Aj[r][c] = make_float2(v.hi, v.lo);
    }
    {
        const int r = t & (SY_RS - 1), c = t / SY_RS;
        const df v = df_from((i0 + r < n && c < m) ? A[(int64_t)(i0 + r) + (int64_t)n * (k0 + c)] : 0.0);
        Ai[r][c] = make_float2(v.hi, v.lo);
    }
    __syncthreads();
    const int r = t & (SY_RS - 1), c = t / SY_RS;
    const int gi = i0 + r, gj = j0 + c;
    if (gi >= n || gj >= n || gj > gi) return;
    dacc v;
#pragma unroll
    for (int q = 0; q < NB; ++q) v.add(Ai[r][q], Aj[c][q]);
    A[(int64_t)gi + (int64_t)n * gj] -= df_to(v.value());
}

// Band of L by columns in double-float form: LB[k*(b+1) + j] = L[k+j, k]
// (j = 0..b, zero past n), so that the rows of one column are contiguous;
// rd[i] = 1 / L[i,i].
__global__ void k_band_cols(const double *__restrict__ L, int n, int b, float2 *__restrict__ LB,
                            float2 *__restrict__ rd) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < n) {
        const df r = df_from(1.0 / L[t + (int64_t)n * t]);
        rd[t] = make_float2(r.hi, r.lo);
    }
    if (t >= (int64_t)n * (b + 1)) return;
    const int k = (int)(t / (b + 1)), j = (int)(t % (b + 1));
    const df v = df_from(k + j < n ? L[(int64_t)(k + j) + (int64_t)n * k] : 0.0);
    LB[t] = make_float2(v.hi, v.lo);
}

__device__ __forceinline__ float2 band_at(const float2 *__restrict__ LB, int b, int i, int k) {
    return LB[(int64_t)k * (b + 1) + (i - k)];   // requires 0 <= i - k <= b
}

// Inverses of the aligned 32 x 32 diagonal blocks of L (double-float),
// column-major per block: D[kb*1024 + t*32 + r] = (L_kb^-1)[r, t].  One warp
// per block, lane t forms column t by forward substitution (rows past n are
// treated as identity rows).
__global__ void __launch_bounds__(32) k_block_inverse(const float2 *__restrict__ LB, const float2 *__restrict__ rd,
                                                      int n, int b, float2 *__restrict__ D) {
    __shared__ float2 Ls[32][33];   // L_kb[r][k], k < r
    __shared__ float2 X[32][33];    // X[r][t] = column t of the inverse
    const int t = threadIdx.x, i0 = blockIdx.x * 32;
    for (int r = 0; r < 32; ++r) {
        const int i = i0 + r, k = i0 + t;
        Ls[r][t] = (t < r && i < n && i - k <= b) ? band_at(LB, b, i, k) : make_float2(0.f, 0.f);
    }
    __syncwarp();
    auto rdiag = [&](int r) -> df {
        const int i = i0 + r;
        return i < n ? df{rd[i].x, rd[i].y} : df{1.f, 0.f};
    };
    for (int r = 0; r < 32; ++r) {
        df x = {0.f, 0.f};
        if (r == t) {
            x = rdiag(r);
        } else if (r > t) {
            df s = {0.f, 0.f};
            for (int k = t; k < r; ++k) s = df_add(s, df_mul({Ls[r][k].x, Ls[r][k].y}, {X[k][t].x, X[k][t].y}));
            x = df_mul(df_neg(s), rdiag(r));
        }
        X[r][t] = make_float2(x.hi, x.lo);
    }
    __syncwarp();
    for (int tt = 0; tt < 32; ++tt) D[(int64_t)blockIdx.x * 1024 + tt * 32 + t] = X[t][tt];
}

// M = L^-1 in double-float arithmetic, a CTA per group of TI_G columns
// c0..c0+TI_G-1 walking down aligned 32-row blocks i0 (GB300's FP64 issue
// rate would bound the n^2 b / 2 multiply-adds):
//   1. S = L[i0:i0+32, i0-b:i0] * M[i0-b:i0, group]: the band tile is staged
//      in shared memory by TI_KC-column chunks, the group's earlier rows of M
//      sit in a shared ring of R >= b + 32 rows; thread (row r = lane, column
//      pair of its warp) accumulates two entries with no masking (the band
//      tile and the ring hold zeros where L or M vanish);
//   2. M[i0:i0+32, group] = D_blk (E - S) with the block's precomputed
//      inverse, E the identity columns of the group.
// Writes M in FP64 (hi + lo) and in FP32 (the FP32 V-cycle's copy).
// A group is TI_G = 16 columns (8 warps) when the ring fits in shared memory,
// else 8, 4 or 2 (wide coarsest bands, e.g. the reference's default hierarchy).
constexpr int TI_KC = 64;

template <int TI_G>
__global__ void __launch_bounds__(16 * TI_G) k_trinv_tiles(const float2 *__restrict__ LB,
                                                           const float2 *__restrict__ D, int n, int b, int R,
                                                           double *__restrict__ M, float *__restrict__ M32) {
    constexpr int TI_THREADS = 16 * TI_G;
    extern __shared__ float2 tsm[];
    float2 *ring = tsm;                       // [R][TI_G]
    float2 *Lt = ring + (int64_t)R * TI_G;    // [32][TI_KC + 1]
    float2 *rhs = Lt + 32 * (TI_KC + 1);      // [32][TI_G]
    const int t = threadIdx.x, r = t & 31, gp = (t >> 5) * 2;
    const int c0 = blockIdx.x * TI_G;
    for (int idx = t; idx < R * TI_G; idx += TI_THREADS) ring[idx] = make_float2(0.f, 0.f);
    __syncthreads();
    for (int i0 = c0 & ~31; i0 < n; i0 += 32) {
        dacc a0, a1;
        const int kbeg = max(0, i0 - b);
        for (int kc = kbeg; kc < i0; kc += TI_KC) {
            const int kn = min(TI_KC, i0 - kc);
            for (int idx = t; idx < 32 * TI_KC; idx += TI_THREADS) {
                const int rr = idx & 31, kk = idx >> 5, i = i0 + rr, k = kc + kk;
                Lt[rr * (TI_KC + 1) + kk] =
                    (kk < kn && i < n && i - k <= b) ? band_at(LB, b, i, k) : make_float2(0.f, 0.f);
            }
            __syncthreads();
#pragma unroll 4
            for (int kk = 0; kk < kn; ++kk) {
                const float2 l = Lt[r * (TI_KC + 1) + kk];
                const float2 *m = ring + (int64_t)((kc + kk) & (R - 1)) * TI_G + gp;
                a0.add(l, m[0]);
                a1.add(l, m[1]);
            }
            __syncthreads();
        }
        const int i = i0 + r;
        {
            df e0 = df_neg(a0.value()), e1 = df_neg(a1.value());
            if (i == c0 + gp) e0 = df_add(e0, {1.f, 0.f});
            if (i == c0 + gp + 1) e1 = df_add(e1, {1.f, 0.f});
            rhs[r * TI_G + gp] = make_float2(e0.hi, e0.lo);
            rhs[r * TI_G + gp + 1] = make_float2(e1.hi, e1.lo);
        }
        __syncthreads();
        dacc v0, v1;
        const float2 *dblk = D + (int64_t)(i0 >> 5) * 1024 + r;
#pragma unroll 8
        for (int q = 0; q < 32; ++q) {
            const float2 d = q <= r ? dblk[q * 32] : make_float2(0.f, 0.f);
            v0.add(d, rhs[q * TI_G + gp]);
            v1.add(d, rhs[q * TI_G + gp + 1]);
        }
        const df x0 = v0.value(), x1 = v1.value();
        float2 *slot = ring + (int64_t)(i & (R - 1)) * TI_G + gp;
        // rows above a column's start come out as exact zeros
        slot[0] = make_float2(x0.hi, x0.lo);
        slot[1] = make_float2(x1.hi, x1.lo);
        if (i < n) {
            const int ca = c0 + gp, cb = ca + 1;
            if (ca < n && i >= ca) {
                M[(int64_t)i + (int64_t)n * ca] = df_to(x0);
                if (M32) M32[(int64_t)i + (int64_t)n * ca] = x0.hi;
            }
            if (cb < n && i >= cb) {
                M[(int64_t)i + (int64_t)n * cb] = df_to(x1);
                if (M32) M32[(int64_t)i + (int64_t)n * cb] = x1.hi;
            }
        }
        // the transpose into the upper triangle (M^T, column-major), staged
        // through shared memory so that the stores run along the group's columns
        __syncthreads();
        rhs[r * TI_G + gp] = make_float2(x0.hi, x0.lo);
        rhs[r * TI_G + gp + 1] = make_float2(x1.hi, x1.lo);
        __syncthreads();
        for (int idx = t; idx < 32 * TI_G; idx += TI_THREADS) {
            const int g = idx % TI_G, rr = idx / TI_G;
            const int cc = c0 + g, ii = i0 + rr;
            if (ii < n && cc < n && ii > cc) {
                const float2 v = rhs[rr * TI_G + g];
                M[(int64_t)cc + (int64_t)n * ii] = (double)v.x + (double)v.y;
                if (M32) M32[(int64_t)cc + (int64_t)n * ii] = v.x;
            }
        }
        __syncthreads();
    }
}

size_t trinv_smem_bytes(int R, int G) { return sizeof(float2) * ((size_t)R * G + 32 * (TI_KC + 1) + 32 * G); }

constexpr int TI_LP = TI_KC + 4, TI_DP = 36;   // padded rows, 16-byte aligned, of the FP32 sweep's tiles

// The same column sweep in FP32 (the hi words of the double-float band and
// block inverses, FP32 FMA accumulation), writing only the FP32 copy M32 that
// the FP32 V-cycle of the mixed-precision solves applies.  Its rounding error
// only perturbs that preconditioner: the coarse apply M32' (M32 r) stays
// symmetric positive semi-definite for any M32, and the outer solve still
// converges on the FP64 residual.
//
// The sweep is a chain of small steps, so their loads run ahead: while a chunk of the
// band is multiplied, the next one (of this row block or the first of the next) is on
// its way in registers, and so is the row block's inverse.  Rows above the group's
// first column are not read: M is zero there.  (Each chunk loaded when it was
// needed: 1.37 ms for 3888 rows of half band 287; now 0.83.)
template <int TI_G>
__global__ void __launch_bounds__(16 * TI_G) k_trinv_tiles32(const float2 *__restrict__ LB,
                                                             const float2 *__restrict__ D, int n, int b, int R,
                                                             float *__restrict__ M32) {
    constexpr int TI_THREADS = 16 * TI_G;
    constexpr int NL = 32 * TI_KC / TI_THREADS, ND = 1024 / TI_THREADS;
    extern __shared__ __align__(16) float tsm32[];
    float *ring = tsm32;                      // [TI_G][R]: column g's rows, row i in slot i mod R
    float *Lt = ring + (int64_t)R * TI_G;     // [32][TI_LP]
    float *Dt = Lt + 32 * TI_LP;              // [32][TI_DP]: (inverse of the diagonal block)[r][q]
    float *rhs = Dt + 32 * TI_DP;             // [TI_G][TI_DP]
    const int t = threadIdx.x, r = t & 31, gp = (t >> 5) * 2;
    const int c0 = blockIdx.x * TI_G, first = c0 & ~31;
    for (int idx = t; idx < R * TI_G; idx += TI_THREADS) ring[idx] = 0.f;
    // a row block's first band column, rounded down to a group of 4 (the band is zero there)
    auto kbegin = [&](int i0) { return max(first, (i0 - b) & ~3); };
    float lreg[NL], dreg[ND];
    auto fetch_band = [&](int i0, int kc) {   // chunk kc .. of row block i0
        const int kn = min(TI_KC, i0 - kc);
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            const int idx = t + k * TI_THREADS, rr = idx & 31, kk = idx >> 5, i = i0 + rr, kcol = kc + kk;
            lreg[k] = (kk < kn && i < n && i - kcol <= b) ? band_at(LB, b, i, kcol).x : 0.f;
        }
    };
    auto fetch_inverse = [&](int i0) {
#pragma unroll
        for (int k = 0; k < ND; ++k) dreg[k] = D[(int64_t)(i0 >> 5) * 1024 + t + k * TI_THREADS].x;
    };
    auto fma4x = [](const float4 l, const float4 m, float acc) {
        return fmaf(l.w, m.w, fmaf(l.z, m.z, fmaf(l.y, m.y, fmaf(l.x, m.x, acc))));
    };
    auto at4 = [](const float *p) { return *reinterpret_cast<const float4 *>(p); };
    fetch_inverse(first);
    for (int i0 = first; i0 < n; i0 += 32) {
        float a0 = 0.f, a1 = 0.f;
        const bool more = i0 + 32 < n;
        __syncthreads();   // the last block's Dt, rhs and ring rows
#pragma unroll
        for (int k = 0; k < ND; ++k) {
            const int idx = t + k * TI_THREADS, rr = idx & 31, q = idx >> 5;
            Dt[rr * TI_DP + q] = q <= rr ? dreg[k] : 0.f;
        }
        if (more) fetch_inverse(i0 + 32);
        for (int kc = kbegin(i0); kc < i0; kc += TI_KC) {
            const int kn = min(TI_KC, i0 - kc);   // a multiple of 4
#pragma unroll
            for (int k = 0; k < NL; ++k) {
                const int idx = t + k * TI_THREADS;
                Lt[(idx & 31) * TI_LP + (idx >> 5)] = lreg[k];
            }
            __syncthreads();
            if (kc + TI_KC < i0)
                fetch_band(i0, kc + TI_KC);
            else if (more)
                fetch_band(i0 + 32, kbegin(i0 + 32));
            // four columns of the band a step; R is a power of two, so four slots never wrap
#pragma unroll 4
            for (int kk = 0; kk < kn; kk += 4) {
                const float4 l = at4(Lt + r * TI_LP + kk);
                const float *m = ring + gp * R + ((kc + kk) & (R - 1));
                a0 = fma4x(l, at4(m), a0);
                a1 = fma4x(l, at4(m + R), a1);
            }
            __syncthreads();
        }
        if (i0 == first && more) fetch_band(i0 + 32, kbegin(i0 + 32));   // no chunk before it
        const int i = i0 + r;
        rhs[gp * TI_DP + r] = (i == c0 + gp ? 1.f : 0.f) - a0;
        rhs[(gp + 1) * TI_DP + r] = (i == c0 + gp + 1 ? 1.f : 0.f) - a1;
        __syncthreads();
        float x0 = 0.f, x1 = 0.f;
#pragma unroll
        for (int q = 0; q < 32; q += 4) {
            const float4 d = at4(Dt + r * TI_DP + q);
            x0 = fma4x(d, at4(rhs + gp * TI_DP + q), x0);
            x1 = fma4x(d, at4(rhs + (gp + 1) * TI_DP + q), x1);
        }
        ring[gp * R + (i & (R - 1))] = x0;
        ring[(gp + 1) * R + (i & (R - 1))] = x1;
        if (i < n) {
            const int ca = c0 + gp, cb = ca + 1;
            if (ca < n && i >= ca) M32[(int64_t)i + (int64_t)n * ca] = x0;
            if (cb < n && i >= cb) M32[(int64_t)i + (int64_t)n * cb] = x1;
        }
        // the transpose into the upper triangle, so that the stores run along the columns
        __syncthreads();
        for (int idx = t; idx < 32 * TI_G; idx += TI_THREADS) {
            const int g = idx % TI_G, rr = idx / TI_G;
            const int cc = c0 + g, ii = i0 + rr;
            if (ii < n && cc < n && ii > cc) M32[(int64_t)cc + (int64_t)n * ii] = ring[g * R + (ii & (R - 1))];
        }
    }
}

size_t trinv32_smem_bytes(int R, int G) {
    return sizeof(float) * ((size_t)R * G + 32 * TI_LP + 32 * TI_DP + G * TI_DP);
}

// launches of the two sweeps for the context's column-group width
template <int G>
static void trinv32_launch(const Ctx &c, const float2 *LB, const float2 *D, int n, int b) {
    k_trinv_tiles32<G><<<(n + G - 1) / G, 16 * G, trinv32_smem_bytes(c.trinv_ring, G), c.stream>>>(
        LB, D, n, b, c.trinv_ring, c.d_Ainv32);
}
template <int G>
static void trinv64_launch(const Ctx &c, const float2 *LB, const float2 *D, int n, int b) {
    k_trinv_tiles<G><<<(n + G - 1) / G, 16 * G, trinv_smem_bytes(c.trinv_ring, G), c.stream>>>(
        LB, D, n, b, c.trinv_ring, c.d_Ainv, nullptr);
}
template <int G>
static void trinv_attributes(int R) {
    cudaFuncSetAttribute(k_trinv_tiles<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)trinv_smem_bytes(R, G));
    cudaFuncSetAttribute(k_trinv_tiles32<G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)trinv32_smem_bytes(R, G));
}

// Enqueues the whole factorization (band Cholesky, L^-1, FP32 copy); no host
// synchronisation, so the sequence is captured once into a CUDA graph.
static void factor_enqueue(Ctx &c, int *d_info) {
    const int n = c.ncf;
    const int nblk = (n + NB - 1) / NB;
    const int bw = (c.cband + NB - 1) / NB + 1;   // band in tiles (safety margin of one)
    double *A = c.d_Ac;
    cudaMemsetAsync(d_info, 0, sizeof(int), c.stream);
    for (int kb = 0; kb < nblk; ++kb) {
        const int k0 = kb * NB;
        const int kend = min(nblk - 1, kb + bw);
        const int nbelow = kend - kb;
        const int rend = min(n, (kend + 1) * NB);
        const int ntrsm = rend > k0 + NB ? (rend - k0 - NB + CP_RS - 1) / CP_RS : 0;
        ++g_launches;
        k_chol_panel<<<1 + ntrsm, CP_THREADS, 0, c.stream>>>(A, n, k0, rend, c.d_LB, d_info);   // d_LB: scratch until the factor is done
        if (nbelow > 0) {
            const int npairs = nbelow * (nbelow + 1) / 2;
            ++g_launches;
            k_syrk_update<<<dim3(npairs, NB / SY_RS), 256, 0, c.stream>>>(A, n, k0, kb + 1, nbelow, c.d_LB);
        }
    }
    const int b = c.cband;
    // d_LB (n (b+1) + n + nblk 1024 doubles) holds, as float pairs, the band
    // by columns, 1/diag and the diagonal-block inverses
    float2 *LB = reinterpret_cast<float2 *>(c.d_LB), *rd = LB + (int64_t)n * (b + 1), *D = rd + n;
    ++g_launches;
    k_band_cols<<<(unsigned)(((int64_t)n * (b + 1) + 255) / 256), 256, 0, c.stream>>>(A, n, b, LB, rd);
    ++g_launches;
    k_block_inverse<<<nblk, 32, 0, c.stream>>>(LB, rd, n, b, D);
    cudaMemsetAsync(c.d_Ainv32, 0, sizeof(float) * (size_t)n * n, c.stream);
    ++g_launches;
    switch (c.trinv_g) {
        case 16: trinv32_launch<16>(c, LB, D, n, b); break;
        case 8: trinv32_launch<8>(c, LB, D, n, b); break;
        case 4: trinv32_launch<4>(c, LB, D, n, b); break;
        default: trinv32_launch<2>(c, LB, D, n, b); break;
    }
}

// The FP64 copy M of L^-1 (double-float sweep), for the FP64 V-cycle; made on
// first use after each factorization.
int ensure_coarse_m64(Ctx &c) {
    if (c.m64_valid || c.ncf == 0) return 0;
    const int n = c.ncf, b = c.cband;
    const int nblk = (n + NB - 1) / NB;
    const float2 *LB = reinterpret_cast<const float2 *>(c.d_LB), *D = LB + (int64_t)n * (b + 1) + n;
    (void)nblk;
    if (cudaMemsetAsync(c.d_Ainv, 0, sizeof(double) * (size_t)n * n, c.stream) != cudaSuccess) return -1;
    ++g_launches;
    switch (c.trinv_g) {
        case 16: trinv64_launch<16>(c, LB, D, n, b); break;
        case 8: trinv64_launch<8>(c, LB, D, n, b); break;
        case 4: trinv64_launch<4>(c, LB, D, n, b); break;
        default: trinv64_launch<2>(c, LB, D, n, b); break;
    }
    if (cudaGetLastError() != cudaSuccess) return -1;
    c.m64_valid = true;
    return 0;
}

// Cholesky of the dense coarsest matrix in d_Ac (lower, in place) and
// M = L^-1 in d_Ainv / d_Ainv32.  Returns 0, the 1-based failing pivot, -1 on
// a CUDA error or -2 when the band is too wide for the shared ring.
int coarse_factor_invert(Ctx &c) {
    const int n = c.ncf;
    if (n == 0) return 0;
    int *d_info = c.d_iflag + 8;
    if (!c.factor_graph) {
        int R = 32;
        while (R < c.cband + 32) R <<= 1;
        int G = 16;   // the widest column group whose ring fits
        while (G > 2 && trinv_smem_bytes(R, G) > 220 * 1024) G >>= 1;
        const size_t smem = trinv_smem_bytes(R, G);
        if (smem > 220 * 1024) return -2;
        switch (G) {
            case 16: trinv_attributes<16>(R); break;
            case 8: trinv_attributes<8>(R); break;
            case 4: trinv_attributes<4>(R); break;
            default: trinv_attributes<2>(R); break;
        }
        c.trinv_ring = R;
        c.trinv_g = G;
        c.trinv_smem = smem;
        const int64_t before = g_launches;
        cudaGraph_t g = nullptr;
        if (cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return -1;
        factor_enqueue(c, d_info);
        if (cudaStreamEndCapture(c.stream, &g) != cudaSuccess) return -1;
        c.factor_graph_launches = g_launches - before;
        g_launches = before;
        if (cudaGraphInstantiate(&c.factor_graph, g, 0) != cudaSuccess) {
            cudaGraphDestroy(g);
            return -1;
        }
        cudaGraphDestroy(g);
    }
    if (cudaGraphLaunch(c.factor_graph, c.stream) != cudaSuccess) return -1;
    g_launches += c.factor_graph_launches;
    c.m64_valid = false;
    int info = 0;
    cudaMemcpyAsync(&info, d_info, sizeof(int), cudaMemcpyDeviceToHost, c.stream);
    cudaStreamSynchronize(c.stream);
    return info;
}

// ---- coarse apply: x_L[free] = A^-1 r_L[free] = M' (M r) -------------------------
// The inverse factor is stored square: M (lower triangle, column-major) and
// its transpose in the upper triangle, so that both products are column-major
// GEMVs with coalesced loads.
//   lower (UPPER = false): y_i = sum_{j <= i} M[i + n j] v[rows[j]]
//   upper (UPPER = true):  x[rows[j]] = sum_{i >= j} M[j + n i] v[i]   (= (M' v)_j)
// A cluster of CL_CTAS CTAs covers 32 output rows.  Their columns are dealt to the
// cluster's 32 warps in blocks of 32, so the triangle's short and long rows
// load all of them alike; lane l holds row i0 + l, and the 32 loads of a block
// (one coalesced row segment per column) are in flight together.  The warps' sums
// meet in shared memory, the CTAs' sums in the first CTA's through distributed
// shared memory, where they are added in a fixed order.  Chunk partials in global
// memory cost two more launches and a memset of x per apply: the FP32 V-cycle of
// 384 x 192 x 192 blobs (1300 rows) went from 214 to 193 us, of 256 x 128 x 128
// (3888 rows) from 151 to 136, of 96 x 48 x 48 from 63 to 53.  An apply of a few thousand rows
// is a chain of latencies: 4 CTAs per cluster are better than 8 (96 x 48 x 48: 3.5 us less
// a cycle, 256 x 128 x 128: 2) and than 2, or 1 to 4 of 16 or 32 warps (4 to 6 less on 96 x 48 x 48).
constexpr int CL_WARPS = 8, CL_CTAS = 4;

template <typename T, bool UPPER>
__global__ void __cluster_dims__(1, CL_CTAS, 1) __launch_bounds__(32 * CL_WARPS)
    k_coarse_gemv(const T *__restrict__ M, const int *__restrict__ rows, const int *__restrict__ pos, int ndof,
                  const T *__restrict__ v, int n, T *__restrict__ y) {
    namespace cg = cooperative_groups;
    using S = WideSum<T>;
    __shared__ S red[CL_WARPS][32];
    __shared__ S sums[CL_CTAS][32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i0 = blockIdx.x * 32, i = i0 + lane, ii = min(i, n - 1);
    auto cluster = cg::this_cluster();
    auto started = cluster.barrier_arrive();   // every CTA of the cluster runs before its memory is written
    const int first = UPPER ? i0 : 0, last = UPPER ? n : min(n, i0 + 32);
    S acc = {};
    for (int jb = first + 32 * (w + CL_WARPS * (int)blockIdx.y); jb < last; jb += 32 * CL_WARPS * CL_CTAS) {
        const int jl = jb + lane;
        const T vl = (jl < n) ? (UPPER ? v[jl] : v[rows[jl]]) : T(0);
        T m[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) m[q] = (jb + q < n) ? M[(int64_t)(jb + q) * n + ii] : T(0);
        T a[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
        for (int q = 0; q < 32; ++q) {
            const T vq = __shfl_sync(0xffffffffu, vl, q);
            // the other triangle holds the transpose
            if (UPPER ? jb + q >= i : jb + q <= i) a[q & 3] += m[q] * vq;
        }
        acc.add((a[0] + a[1]) + (a[2] + a[3]));
    }
    red[w][lane] = acc;
    __syncthreads();
    cluster.barrier_wait(std::move(started));
    if (w == 0) {
        S t[CL_WARPS];
#pragma unroll
        for (int k = 0; k < CL_WARPS; ++k) t[k] = red[k][lane];
        cluster.map_shared_rank(&sums[0][0], 0)[32 * blockIdx.y + lane] =
            ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
    }
    cluster.sync();
    if (blockIdx.y == 0 && w == 0 && i < n)
        y[UPPER ? rows[i] : i] = ((sums[0][lane] + sums[1][lane]) + (sums[2][lane] + sums[3][lane])).value();
    // x is zero off the free DOFs
    if (UPPER && blockIdx.x == 0 && blockIdx.y == 1)
        for (int d = threadIdx.x; d < ndof; d += 32 * CL_WARPS)
            if (pos[d] < 0) y[d] = T(0);
}

template <typename T>
static void coarse_apply(const Ctx &c, const T *M, const T *rc, T *xc, T *ybuf, cudaStream_t s) {
    const int ndof = (int)(3 * c.lv[c.L - 1].nnode);
    if (c.ncf == 0) {
        cudaMemsetAsync(xc, 0, sizeof(T) * ndof, s);
        return;
    }
    const dim3 g((c.ncf + 31) / 32, CL_CTAS);
    const int *pos = c.d_cfree + c.ncf;
    g_launches += 2;
    k_coarse_gemv<T, false><<<g, 32 * CL_WARPS, 0, s>>>(M, c.d_cfree, pos, ndof, rc, c.ncf, ybuf);
    k_coarse_gemv<T, true><<<g, 32 * CL_WARPS, 0, s>>>(M, c.d_cfree, pos, ndof, ybuf, c.ncf, xc);
}

void launch_coarse_apply_f64(const Ctx &c, const double *rc, double *xc, cudaStream_t s) {
    coarse_apply<double>(c, c.d_Ainv, rc, xc, c.d_cy, s);
}

void launch_coarse_apply_f32(const Ctx &c, const float *rc, float *xc, cudaStream_t s) {
    coarse_apply<float>(c, c.d_Ainv32, rc, xc, reinterpret_cast<float *>(c.d_cy + c.ncf), s);
}

}  // namespace sgld
