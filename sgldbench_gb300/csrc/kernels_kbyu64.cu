// FP64 and double-float matrix-free K*u of the finest level in sum-factorised Hadamard form
// (reference: src/MEXfuncs/Solving_KbyU_MatrixFree_mex.cpp:53-138).
//
// GB300 issues about two FP64 operations per clock and SM, so the operator is
// bound by the number of FP64 instructions and by nothing else: 238 MB of
// vectors on the 256 x 128 x 128 grid take 35 us of HBM time, 137 operations
// per element 0.94 ms of FP64 time.  The kernel therefore forms every partial
// result once and lets the elements around it share it through shared memory:
//   * the y butterfly of an edge along y (4 elements share it): 6 operations;
//   * the x butterfly of a face in a node layer (2 elements): 12;
//   * per element the z butterfly (21: the three rigid translations are not
//     needed), E * Kh in the 8-value form of a cubic-symmetric element matrix
//     (8 + 33), the z butterfly undone and added to what the element layer
//     below carried up (30), the x butterfly undone (12);
//   * the two faces of an edge add (6), the y butterfly is undone (6) and the
//     two edges of a node add (3).
// The form before it applied the three butterflies per element: 234
// operations, on a fixed 32 x 8 tile whose halo and ragged edges made 1.43
// threads per node of that grid.  sgld_kbyu_device (with its scatter and
// gather) went from 2.85 to 1.52 ms on 256 x 128 x 128 and from 302 to 71 us on
// 64 x 32 x 32, where the fixed tile filled 60 of 152 SMs.
//
// Double-float (the outer loop of the mixed-precision solve): the same kernel on pairs hi +
// lo of FP32 numbers with 48 significant bits (df_arith.cuh: Knuth's TwoSum, the FMA form
// of Dekker's product; 11 FP32 operations per add, 7 per multiply), as GB300 issues 64
// FP32 operations in the time of one FP64 operation.  The result is within a few units of
// 2^-48 of the FP64 operator (tests compare to 1e-12), enough for the FP64 residual
// recurrence and the true residual at exit.  The data stay FP64 in HBM: a staged word is split
// in place by the thread that copied it, a node's sum is joined when it is stored, and
// the dot product is FP64 on the words of u themselves.  115 adds and 34 multiplies
// make about 1500 FP32 operations per element; the form that applied the whole
// transform per element needed 2570, on a fixed 32 x 8 tile: 740 us on 256 x 128 x 128,
// now 523, 262 us on the 192 x 96 x 96 blob shape, now 145, and 106 us on 64 x 32 x 32, now 34.
//
// A CTA owns (ye-1) x (xe-1) node columns and marches through zc node layers;
// thread t handles the element column t % ye, t / ye of its ye x xe element
// tile.  Any ye and xe will do, as both exchanges go through shared memory, so
// the tile is chosen to fit the grid (kbyu64_pick_tile).
#include "sgld_internal.cuh"
#include "df_arith.cuh"

namespace sgld {

// Hadamard-basis element matrix (sgld_internal.cuh), and its 8-value form
// A-B, B, C, D, E, F-G, G, H (KH_CLASS in kernels_stencil.cu), in both arithmetics
__constant__ double c_kh64[KH_NNZ];
__constant__ double c_kc64[8];
__constant__ float2 c_khdf[KH_NNZ];
__constant__ float2 c_kcdf[8];

void upload_kh64(const double *Kh, const double *kc, cudaStream_t s) {
    cudaMemcpyToSymbolAsync(c_kh64, Kh, sizeof(double) * KH_NNZ, 0, cudaMemcpyHostToDevice, s);
    cudaMemcpyToSymbolAsync(c_kc64, kc, sizeof(double) * 8, 0, cudaMemcpyHostToDevice, s);
    float2 p[KH_NNZ + 8];
    for (int i = 0; i < KH_NNZ + 8; ++i) {
        const double v = i < KH_NNZ ? Kh[i] : kc[i - KH_NNZ];
        const float hi = (float)v;
        p[i] = make_float2(hi, (float)(v - (double)hi));
    }
    cudaMemcpyToSymbolAsync(c_khdf, p, sizeof(float2) * KH_NNZ, 0, cudaMemcpyHostToDevice, s);
    cudaMemcpyToSymbolAsync(c_kcdf, p + KH_NNZ, sizeof(float2) * 8, 0, cudaMemcpyHostToDevice, s);
}

namespace k64 {
constexpr int MAX_THREADS = 384;   // at 168 registers a thread
constexpr int STAGE = 5;           // staged words per thread and node layer, at most
constexpr int SLOTS = 4;           // node layers in shared memory

__host__ __device__ constexpr int threads(int ye, int xe) { return (ye * xe + 31) & ~31; }
constexpr int node_words(int ye, int xe) { return 3 * (ye + 1) * (xe + 1); }
constexpr size_t smem(int ye, int xe) {   // node ring, edge, face and node exchanges
    return sizeof(double) * ((size_t)SLOTS * node_words(ye, xe) + 6 * ye * (xe + 1) + 9 * ye * xe);
}
}  // namespace k64

// the arithmetic of a value: FP64, or double-float
struct A64 {
    using V = double;
    __device__ __forceinline__ static V from(double a) { return a; }
    __device__ __forceinline__ static double to(V a) { return a; }
    __device__ __forceinline__ static V add(V a, V b) { return a + b; }
    __device__ __forceinline__ static V sub(V a, V b) { return a - b; }
    __device__ __forceinline__ static V mul(V a, V b) { return a * b; }
    __device__ __forceinline__ static V fma(V a, V b, V c) { return ::fma(a, b, c); }
    __device__ __forceinline__ static V kh(int i) { return c_kh64[i]; }
    __device__ __forceinline__ static V kc(int i) { return c_kc64[i]; }
    __device__ __forceinline__ static V load(const double *p) { return *p; }
    __device__ __forceinline__ static void store(double *p, V v) { *p = v; }
    static constexpr bool SPLIT = false;
};
struct ADF {
    using V = df;
    __device__ __forceinline__ static V from(double a) { return df_from(a); }
    __device__ __forceinline__ static double to(V a) { return df_to(a); }
    __device__ __forceinline__ static V add(V a, V b) { return df_add(a, b); }
    __device__ __forceinline__ static V sub(V a, V b) { return df_sub(a, b); }
    __device__ __forceinline__ static V mul(V a, V b) { return df_mul(a, b); }
    __device__ __forceinline__ static V fma(V a, V b, V c) { return df_add(df_mul(a, b), c); }
    __device__ __forceinline__ static V kh(int i) { return {c_khdf[i].x, c_khdf[i].y}; }
    __device__ __forceinline__ static V kc(int i) { return {c_kcdf[i].x, c_kcdf[i].y}; }
    // a value takes the 8 bytes of the word it came from
    __device__ __forceinline__ static V load(const double *p) {
        const float2 t = *reinterpret_cast<const float2 *>(p);
        return {t.x, t.y};
    }
    __device__ __forceinline__ static void store(double *p, V v) { *reinterpret_cast<float2 *>(p) = make_float2(v.hi, v.lo); }
    static constexpr bool SPLIT = true;
};

// h <- E Kh h without the translations h[0..2]; k holds E times the 8 values
template <typename A>
__device__ __forceinline__ void kh_cubic_f64(typename A::V (&h)[24], const typename A::V (&k)[8]) {
    using V = typename A::V;
#define Y3(i, j, l, a, b)                                                 \
    {                                                                     \
        const V t = A::mul(k[b], A::add(A::add(h[i], h[j]), h[l]));       \
        h[i] = A::fma(k[a], h[i], t);                                     \
        h[j] = A::fma(k[a], h[j], t);                                     \
        h[l] = A::fma(k[a], h[l], t);                                     \
    }
#define YC(i, j) h[i] = h[j] = A::mul(k[2], A::add(h[i], h[j]));
#define YD(i, j)                                      \
    {                                                 \
        const V a = h[i], b = h[j];                   \
        h[i] = A::fma(k[4], b, A::mul(k[3], a));      \
        h[j] = A::fma(k[4], a, A::mul(k[3], b));      \
    }
    Y3(3, 7, 14, 0, 1)
    YC(4, 6)
    YC(5, 12)
    YC(8, 13)
    YD(9, 20)
    YD(10, 17)
    Y3(11, 16, 18, 5, 6)
    YD(15, 19)
    h[21] = A::mul(h[21], k[7]);
    h[22] = A::mul(h[22], k[7]);
    h[23] = A::mul(h[23], k[7]);
#undef Y3
#undef YC
#undef YD
}

// the same for any element matrix with the hexahedral block pattern
template <typename A>
__device__ __forceinline__ void kh_general_f64(typename A::V (&h)[24], typename A::V e) {
    using V = typename A::V;
#define Z3(i, j, l, o)                                                                                       \
    {                                                                                                        \
        const V a = A::mul(e, h[i]), b = A::mul(e, h[j]), d = A::mul(e, h[l]);                               \
        h[i] = A::fma(A::kh(o + 2), d, A::fma(A::kh(o + 1), b, A::mul(A::kh(o), a)));                        \
        h[j] = A::fma(A::kh(o + 5), d, A::fma(A::kh(o + 4), b, A::mul(A::kh(o + 3), a)));                    \
        h[l] = A::fma(A::kh(o + 8), d, A::fma(A::kh(o + 7), b, A::mul(A::kh(o + 6), a)));                    \
    }
#define Z2(i, j, o)                                                      \
    {                                                                    \
        const V a = A::mul(e, h[i]), b = A::mul(e, h[j]);                \
        h[i] = A::fma(A::kh(o + 1), b, A::mul(A::kh(o), a));             \
        h[j] = A::fma(A::kh(o + 3), b, A::mul(A::kh(o + 2), a));         \
    }
    Z3(3, 7, 14, 0)
    Z2(4, 6, 9)
    Z2(5, 12, 13)
    Z2(8, 13, 17)
    Z2(9, 20, 21)
    Z2(10, 17, 25)
    Z3(11, 16, 18, 29)
    Z2(15, 19, 38)
    h[21] = A::mul(h[21], A::mul(A::kh(42), e));
    h[22] = A::mul(h[22], A::mul(A::kh(43), e));
    h[23] = A::mul(h[23], A::mul(A::kh(44), e));
#undef Z3
#undef Z2
}

__device__ __forceinline__ void copy_word(double *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

// y = K u on the full grid; y is 0 at fixed DOFs and at inactive nodes.  When
// DOT, also writes sum(u .* y) of this CTA's nodes to partial[block].
// tiles: the CTAs' activity map for this tile (0: no active element in the
// CTA's box, so all it owns is zero), or null.
template <typename A, bool DOT, bool CUBIC>
__global__ void __launch_bounds__(k64::MAX_THREADS, 1)
    k_kbyu64(const double *__restrict__ u, double *__restrict__ y, const double *__restrict__ E,
             const uint8_t *__restrict__ nflag, int ny, int nx, int nz, int ye, int xe, int zc,
             double *__restrict__ partial, const uint8_t *__restrict__ tiles) {
    using V = typename A::V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, nt = blockDim.x;
    const int tn = ye * xe, te = ye * (xe + 1), nw = k64::node_words(ye, xe);
    double *su = reinterpret_cast<double *>(smem_raw);   // [SLOTS][nw] node layers
    double *se = su + k64::SLOTS * nw;                   // [6][te] y butterflies of the edges of a node layer
    double *sl = se + 6 * te;                            // [6][tn] left face shares of the edges
    double *sn = sl + 6 * tn;                            // [3][tn] upper shares of the nodes
    const int ly = tid % ye, lx = tid / ye;
    const bool elem = tid < tn;
    const int NY = ny + 1, NX = nx + 1, NZ = nz + 1;
    const int y0 = blockIdx.x * (ye - 1), x0 = blockIdx.y * (xe - 1), z0 = blockIdx.z * zc;
    const int zend = min(z0 + zc, NZ);
    const int gy = y0 + ly, gx = x0 + lx;   // the node this thread completes: local (ly+1, lx+1)
    const bool owner = elem && ly < ye - 1 && lx < xe - 1 && gy < NY && gx < NX;
    const int64_t plane = (int64_t)NY * NX, slot = blockIdx.x + gridDim.x * (blockIdx.y + (int64_t)gridDim.y * blockIdx.z);
    if (tiles && !tiles[slot]) {
        if (owner)
            for (int z = z0; z < zend; ++z) {
                double *o = y + 3 * (gy + (int64_t)NY * gx + plane * z);
                o[0] = o[1] = o[2] = 0.0;
            }
        if (DOT && tid == 0) partial[slot] = 0.0;
        return;
    }
    // this thread's words of a node layer: offsets in the layer, -1 past the grid, -2 none
    int off[k64::STAGE];
#pragma unroll
    for (int k = 0; k < k64::STAGE; ++k) {
        const int i = tid + k * nt;
        off[k] = -2;
        if (i < nw) {
            const int node = i / 3, c = i - 3 * node, ny_ = node % (ye + 1), nx_ = node / (ye + 1);
            const int py = y0 - 1 + ny_, px = x0 - 1 + nx_;
            off[k] = (py >= 0 && py < NY && px >= 0 && px < NX) ? 3 * (py + NY * px) + c : -1;
        }
    }
    auto stage = [&](int z) {   // node layer z into its slot
        double *dst = su + ((z + k64::SLOTS) % k64::SLOTS) * nw;
        const double *src = u + 3 * plane * z;
        const bool zin = z >= 0 && z < NZ;
#pragma unroll
        for (int k = 0; k < k64::STAGE; ++k) {
            const int i = tid + k * nt;
            if (off[k] == -2) continue;
            if (zin && off[k] >= 0)
                copy_word(dst + i, src + off[k]);
            else
                dst[i] = 0.0;
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    // after this thread's copies have landed: its words of node layer z as values
    auto landed = [&](int z) {
        if (!A::SPLIT) return;
        double *dst = su + ((z + k64::SLOTS) % k64::SLOTS) * nw;
#pragma unroll
        for (int k = 0; k < k64::STAGE; ++k)
            if (off[k] != -2) A::store(dst + tid + k * nt, A::from(dst[tid + k * nt]));
    };
    // y butterflies of the edges of node layer z: sum and u(ly) - u(ly+1)
    auto edges = [&](int z) {
        if (!elem) return;
        const double *p = su + ((z + k64::SLOTS) % k64::SLOTS) * nw + 3 * (ly + (ye + 1) * lx);
        for (int x = lx;; ++x, p += 3 * (ye + 1)) {   // the last column's threads also form the column past it
            double *o = se + ly + ye * x;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const V lo = A::load(p + c), hi = A::load(p + 3 + c);
                A::store(o + c * te, A::add(lo, hi));
                A::store(o + (3 + c) * te, A::sub(lo, hi));
            }
            if (lx < xe - 1 || x == xe) break;
        }
    };
    // the 12 face coefficients (index 3 (bx | by << 1) + c) of this element column
    auto faces = [&](V (&F)[12]) {
        const double *p = se + tid;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const V a = A::load(p + i * te), b = A::load(p + i * te + ye);
            const int k = i < 3 ? i : i + 3;   // by = 0: 0..2, by = 1: 6..8
            F[k] = A::add(a, b);
            F[k + 3] = A::sub(b, a);
        }
    };
    const int ey = y0 - 1 + ly, ex = x0 - 1 + lx;
    const bool ein = elem && ey >= 0 && ey < ny && ex >= 0 && ex < nx;
    const double *ep = E + ey + (int64_t)ny * ex;
    const int64_t eplane = (int64_t)ny * nx;
    auto modulus = [&](int z) { return ein && z >= 0 && z < nz ? ep[eplane * z] : 0.0; };

    const V zero = A::from(0.0);
    V Fp[12], carry[12];
    double dot = 0.0;
    bool live = false;   // carry is not zero
#pragma unroll
    for (int i = 0; i < 12; ++i) Fp[i] = carry[i] = zero;
    stage(z0 - 1);
    stage(z0);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    landed(z0 - 1);
    landed(z0);
    __syncthreads();
    edges(z0 - 1);
    __syncthreads();
    double ev = modulus(z0 - 1), en = modulus(z0);
    if (elem && ev != 0.0) faces(Fp);
    __syncthreads();
    edges(z0);
    // node layer ez, one barrier after its shares were written; its flags, and for the dot
    // product of split words u itself, were loaded a layer ahead
    V lo[3] = {zero, zero, zero};
    uint8_t fl = 0;
    double un[3] = {0.0, 0.0, 0.0};
    int64_t node = gy + (int64_t)NY * gx + plane * (z0 - 1);
    auto ahead = [&](int ez) {
        if (!owner || ez < z0) return;
        fl = nflag[node];
        if (DOT && A::SPLIT)
#pragma unroll
            for (int c = 0; c < 3; ++c) un[c] = u[3 * node + c];
    };
    auto output = [&](int ez) {
        if (!owner || ez < z0) return;
        const double *us = su + ((ez + k64::SLOTS) % k64::SLOTS) * nw + 3 * (ly + 1 + (ye + 1) * (lx + 1));
        double *yo = y + 3 * (node - plane);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double o = (fl & (NF_FIXX << c)) ? 0.0 : A::to(A::add(lo[c], A::load(sn + c * tn + tid + 1)));
            yo[c] = o;
            if (DOT) dot = fma(A::SPLIT ? un[c] : us[c], o, dot);
        }
    };
    // two barriers per element layer: the edges of the next node layer are formed with the
    // undone edges of this one, a node layer is written a barrier later
    for (int ez = z0 - 1; ez < zend; ++ez) {
        // element layer ez between node layers ez (faces Fp) and ez + 1
        __syncthreads();
        output(ez - 1);
        ahead(ez);
        node += plane;
        if (ez + 2 <= zend) stage(ez + 2);
        V rp[6];
        if (elem) {
            V Ft[12];
            // the faces of layer ez + 1 are needed by the elements below and above them
            if (ev != 0.0 || en != 0.0) faces(Ft);
            V phi[12];
            live |= ev != 0.0;
            if (ev != 0.0) {
                V h[24];
#pragma unroll
                for (int i = 0; i < 12; ++i) {
                    h[i] = i < 3 ? zero : A::add(Fp[i], Ft[i]);
                    h[12 + i] = A::sub(Ft[i], Fp[i]);
                }
                const V e = A::from(ev);
                if constexpr (CUBIC) {
                    V k[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) k[i] = A::mul(A::kc(i), e);
                    kh_cubic_f64<A>(h, k);
                } else {
                    kh_general_f64<A>(h, e);
                }
#pragma unroll
                for (int i = 0; i < 12; ++i) {
                    phi[i] = i < 3 ? A::sub(carry[i], h[12 + i]) : A::add(carry[i], A::sub(h[i], h[12 + i]));
                    carry[i] = i < 3 ? h[12 + i] : A::add(h[i], h[12 + i]);
                }
            } else {   // void: nothing is read from its nodes, whatever they hold
#pragma unroll
                for (int i = 0; i < 12; ++i) {
                    phi[i] = carry[i];
                    carry[i] = zero;
                }
            }
            // x butterfly undone: column lx gets phi0 - phi1, column lx + 1 phi0 + phi1
            if (live) {
#pragma unroll
                for (int i = 0; i < 6; ++i) {
                    const int k = i < 3 ? i : i + 3;
                    A::store(sl + i * tn + tid, A::sub(phi[k], phi[k + 3]));
                    rp[i] = A::add(phi[k], phi[k + 3]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 6; ++i) {
                    sl[i * tn + tid] = 0.0;
                    rp[i] = zero;
                }
            }
            live = ev != 0.0;   // carried up
            if (en != 0.0) {
#pragma unroll
                for (int i = 0; i < 12; ++i) Fp[i] = Ft[i];
            }
            ev = en;
            en = modulus(ez + 2);
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        if (ez + 2 <= zend) landed(ez + 2);
        __syncthreads();
        // edge of column lx + 1: this element's right part and the next column's left part; y
        // butterfly undone: node ly + 1 gets t0 - t1, node ly gets t0 + t1
        if (elem && lx < xe - 1) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const V t0 = A::add(rp[c], A::load(sl + c * tn + tid + ye));
                const V t1 = A::add(rp[3 + c], A::load(sl + (3 + c) * tn + tid + ye));
                lo[c] = A::sub(t0, t1);
                A::store(sn + c * tn + tid, A::add(t0, t1));
            }
        }
        if (ez + 1 < zend) edges(ez + 2);
    }
    __syncthreads();
    output(zend - 1);
    if (DOT) {
        __shared__ double red[k64::MAX_THREADS / 32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_down_sync(0xffffffffu, dot, o);
        if ((tid & 31) == 0) red[tid >> 5] = dot;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int i = 0; i < nt / 32; ++i) s += red[i];
            partial[slot] = s;
        }
    }
}

// The tile for a grid, by the FP64 work of the busiest SM.  Its CTAs, (CTAs / 152
// rounded up), run as many at a time as fit into 384 threads; each of the SM's four
// schedulers takes a quarter of their warps, rounded up, and needs 64 clocks per
// FP64 instruction and warp, 137 instructions per element layer; a layer costs
// about 2000 clocks of latency and barriers besides, a CTA's start 6000.  Small grids
// get many small CTAs that fill the SMs, large ones tiles whose ragged edge and
// halo are small.  On a grid with void regions the CTAs' work differs from tile to
// tile, and the last one to start decides: there the cost is the active share of
// the work, spread evenly, plus one whole CTA.  (With the solid grid's rule the 384 x
// 192 x 192 blob shape took 3.69 ms, with this one 2.01; the fixed 32 x 8 x 16 tile
// 3.28.)  The double-float form takes the same tile and map, although latency binds it rather
// than the FP64 pipe: the rule's choice is the best of a sweep for it too on 256 x 128 x 128 (523 us),
// on the 384 x 192 x 192 blob shape another tile would be 10 % faster (18 x 7 x 13: 850 us, the choice
// 16 x 12 x 15: 951).  At most SGLD_NOALLOC_MAX_CTAS CTAs, the scratch of the allocation-free
// call, where the grid allows it.
void kbyu64_pick_tile(Level &l) {
    const int NY = l.ny + 1, NX = l.nx + 1, NZ = l.nz + 1;
    constexpr int SMS = 152, MAX_CTAS = 32768;
    const double fill = (double)l.nnode_active / (double)l.nnode;
    const bool solid = fill > 0.85;
    double best = 0.0;
    l.k64_ye = 0;
    for (int ty = 1; ty <= NY; ++ty) {   // tiles along y: the smallest ye that needs no more of them
        const int ye = (NY + ty - 1) / ty + 1;
        if ((NY + ye - 2) / (ye - 1) != ty) continue;
        if (ye < 4 && ty > 1) break;
        if (ye * 2 > k64::MAX_THREADS) continue;
        for (int tx = 1; tx <= NX; ++tx) {
            const int xe = (NX + tx - 1) / tx + 1;
            if ((NX + xe - 2) / (xe - 1) != tx) continue;
            if (xe < 4 && tx > 1) break;
            const int nt = k64::threads(ye, xe);
            if (nt > k64::MAX_THREADS || k64::node_words(ye, xe) > k64::STAGE * nt) continue;
            for (int tz = 1; tz <= NZ; ++tz) {
                const int zc = (NZ + tz - 1) / tz;
                if ((NZ + zc - 1) / zc != tz) continue;
                if (zc < 2 && tz > 1) break;
                const int64_t n = (int64_t)ty * tx * tz;
                // clocks per layer of k CTAs together, and of a CTA's share of that
                const int w = nt / 32, fit = k64::MAX_THREADS / nt;
                auto layer = [&](int k) { return (k * w + 3) / 4 * 64.0 * 137.0 + 2000.0; };
                auto clocks = [&](double per_layer) { return (zc + 1) * per_layer + 6000.0; };
                double cost;
                if (solid) {
                    const int64_t r = (n + SMS - 1) / SMS;   // CTAs of the busiest SM
                    cost = (double)(r / fit) * clocks(layer(fit)) + (r % fit ? clocks(layer((int)(r % fit))) : 0.0);
                } else {
                    cost = (fill * (double)n / SMS + 1.0) * clocks(layer(fit) / fit);
                }
                if (n > MAX_CTAS) cost *= 1e6;
                if (!l.k64_ye || cost < best) {
                    best = cost;
                    l.k64_ye = ye;
                    l.k64_xe = xe;
                    l.k64_zc = zc;
                }
            }
        }
    }
}

dim3 kbyu64_grid(const Level &l) {
    return dim3((l.ny + l.k64_ye - 1) / (l.k64_ye - 1), (l.nx + l.k64_xe - 1) / (l.k64_xe - 1),
                (l.nz + l.k64_zc) / l.k64_zc);
}

template <typename A, bool DOT, bool CUBIC>
static void attributes(size_t smem) {
    cudaFuncSetAttribute(k_kbyu64<A, DOT, CUBIC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

void init_kbyu64_attributes() {
    // the widest node ring any tile asks for
    size_t most = 0;
    for (int ye = 2; ye <= k64::MAX_THREADS / 2; ++ye)
        for (int xe = 2; ye * xe <= k64::MAX_THREADS; ++xe)
            if (k64::node_words(ye, xe) <= k64::STAGE * k64::threads(ye, xe) && k64::smem(ye, xe) > most)
                most = k64::smem(ye, xe);
    attributes<A64, true, true>(most);
    attributes<A64, true, false>(most);
    attributes<A64, false, true>(most);
    attributes<A64, false, false>(most);
    attributes<ADF, true, true>(most);
    attributes<ADF, true, false>(most);
    attributes<ADF, false, true>(most);
    attributes<ADF, false, false>(most);
}

template <typename A>
static void launch(const Level &l0, const double *E, const double *u, double *y, double *partial, int *nblocks,
                   cudaStream_t s) {
    const int ye = l0.k64_ye, xe = l0.k64_xe;
    const dim3 g = kbyu64_grid(l0);
    if (nblocks) *nblocks = (int)(g.x * g.y * g.z);
    const auto k = partial ? (l0.kh_cubic64 ? k_kbyu64<A, true, true> : k_kbyu64<A, true, false>)
                           : (l0.kh_cubic64 ? k_kbyu64<A, false, true> : k_kbyu64<A, false, false>);
    ++g_launches;
    k<<<g, k64::threads(ye, xe), k64::smem(ye, xe), s>>>(u, y, E, l0.nflag, l0.ny, l0.nx, l0.nz, ye, xe, l0.k64_zc,
                                                         partial, l0.tiles64);
}

void launch_kbyu_f64(const Level &l0, const double *E, const double *u, double *y, double *partial_dot,
                     int *nblocks_out, cudaStream_t s) {
    launch<A64>(l0, E, u, y, partial_dot, nblocks_out, s);
}

void launch_kbyu_df(const Level &l0, const double *E, const double *u, double *y, double *partial_dot,
                    int *nblocks_out, cudaStream_t s) {
    launch<ADF>(l0, E, u, y, partial_dot, nblocks_out, s);
}

}  // namespace sgld
