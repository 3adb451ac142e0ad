// Kernels of the mixed-precision solve (SGLD_PREC_MIXED).
//
// The outer loop is the reference's PCG in FP64 made flexible (Polak-Ribiere
// beta = -lambda z_new'q / z'r), so that the preconditioner may change from
// one application to the next.  The preconditioner is a fixed number of FP32
// CG iterations on K e = r, each preconditioned by the reference's additive
// V-cycle in FP32.  The inner loop runs entirely on the device (scalars in
// device memory) and is captured once into a CUDA graph.
#include "sgld_internal.cuh"

namespace sgld {

constexpr int MB = 256;

__device__ __forceinline__ double mblock_reduce(double v) {
    __shared__ double red[MB / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int i = 0; i < MB / 32; ++i) s += red[i];
    return s;
}

// four independent accumulators per thread, so that four loads are in flight
// (a K*u launch on a large grid leaves tens of thousands of partials)
__device__ double msum_partials(const double *__restrict__ part, int nb) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int i = threadIdx.x;
    for (; i + 3 * MB < nb; i += 4 * MB) {
        s0 += part[i];
        s1 += part[i + MB];
        s2 += part[i + 2 * MB];
        s3 += part[i + 3 * MB];
    }
    for (; i < nb; i += MB) s0 += part[i];
    return mblock_reduce((s0 + s1) + (s2 + s3));
}

// The vector updates of the inner CG sum up to FUSE_PARTS partials themselves (usum_partials).
constexpr int UB = 512;   // threads of an update
constexpr int UGRID = 152 * 2;

// inner scalars (FP64 storage): rho = z.s of the last iteration, alpha, beta,
// r0 = s.s at entry, the iteration count of this inner solve, the current
// iteration cap, whether the last inner solve stopped at that cap short of
// its tolerance, and (slot 8) the total over the outer solve (reset by the
// host at the start of each solve)
enum { IS_RHO = 0, IS_ALPHA = 1, IS_BETA = 2, IS_R0 = 3, IS_IT = 4, IS_KCAP = 5, IS_CAPHIT = 6, IS_ZS = 7, IS_TOT = 8 };

// alpha and beta of the inner CG.  z.s of an iteration goes to IS_ZS with beta and
// to IS_RHO with alpha, so that no launch writes a scalar that another of its CTAs
// may still have to read.
__device__ __forceinline__ double icg_beta(double rho, double zs) { return rho != 0.0 ? zs / rho : 0.0; }
__device__ __forceinline__ double icg_alpha(double zs, double dt) { return dt != 0.0 ? zs / dt : 0.0; }

// op 0 (entry of an inner solve): r0 = sum, rho = 0, it = 0, and the cap:
// kbase at the first inner solve of an outer solve, doubled (up to klimit)
// after an inner solve that hit its cap without reaching its tolerance;
// op 1: alpha = z.s / sum, rho = z.s;  op 2: beta = sum / rho (0 on the first
// iteration, rho = 0), z.s = sum
__global__ void k_icg_scalar(int op, double *__restrict__ sc, const double *__restrict__ part, int nb, int kbase,
                             int klimit) {
    const double s = msum_partials(part, nb);
    if (threadIdx.x != 0) return;
    if (op == 0) {
        if (sc[IS_TOT] == 0.0) {
            sc[IS_KCAP] = (double)kbase;
        } else if (sc[IS_CAPHIT] != 0.0) {
            sc[IS_KCAP] = fmin(2.0 * sc[IS_KCAP], (double)klimit);
        }
        sc[IS_CAPHIT] = 0.0;
        sc[IS_R0] = s;
        sc[IS_RHO] = 0.0;
        sc[IS_IT] = 0.0;
        sc[IS_ALPHA] = 0.0;   // the first d update adds alpha * d = 0 to e
    } else if (op == 1) {
        const double zs = sc[IS_ZS];
        sc[IS_ALPHA] = icg_alpha(zs, s);
        sc[IS_RHO] = zs;
    } else {
        sc[IS_BETA] = icg_beta(sc[IS_RHO], s);
        sc[IS_ZS] = s;
    }
}

// alpha (OP 1) or beta (OP 2) for all threads of a CTA, from the nsum partials of its
// denominator or numerator, or as k_icg_scalar left it (nsum = 0)
template <int OP>
__device__ __forceinline__ float icg_coefficient(double *__restrict__ sc, const double *__restrict__ sum, int nsum) {
    if (nsum == 0) return (float)sc[OP == 1 ? IS_ALPHA : IS_BETA];
    const double other = sc[OP == 1 ? IS_ZS : IS_RHO];
    const double s = usum_partials(sum, nsum);
    __shared__ float coef;
    if (threadIdx.x == 0) {
        const double v = OP == 1 ? icg_alpha(other, s) : icg_beta(other, s);
        if (blockIdx.x == 0) {
            sc[OP == 1 ? IS_ALPHA : IS_BETA] = v;
            sc[OP == 1 ? IS_RHO : IS_ZS] = OP == 1 ? other : s;
        }
        coef = (float)v;
    }
    __syncthreads();
    return coef;
}

// end of an inner iteration: count it and keep iterating while it < kmax and
// ||s|| > eta ||s_0||, eta = max(eta_min, tol / (2 relres)) with the outer
// solve's tolerance and current relative residual (outer[15], outer[3]): the
// inner solve of the last outer step only goes as far as the outer tolerance
// needs.  eta_min <= 0: exactly kmax iterations.  For thread 0: whether to go on.
// The threshold is formed beside the sum, by a thread of a warp that takes no part in it:
// a launch of one CTA is all latency, and its FP64 division alone a good part of it.
__device__ __forceinline__ bool icg_more(double *__restrict__ sc, const double *__restrict__ part, int nb, int kmax,
                                         double eta_min, const double *__restrict__ outer, double *__restrict__ total) {
    __shared__ double limit;
    __shared__ int below;   // under the cap
    if (threadIdx.x == 128) {
        const double it = sc[IS_IT] + 1.0, cap = eta_min > 0.0 ? sc[IS_KCAP] : (double)kmax;
        double l = 0.0;
        if (eta_min > 0.0) {
            const double relres = outer[3], tol = outer[15];
            const double eta = (relres > 0.0) ? fmax(eta_min, 0.5 * tol / relres) : eta_min;
            l = eta * eta * sc[IS_R0];
        }
        sc[IS_IT] = it;
        *total += 1.0;
        limit = l;
        below = it < cap;
    }
    const double ss = usum_partials(part, nb);   // ends with a barrier
    if (threadIdx.x != 0) return false;
    bool more = below != 0;
    if (eta_min > 0.0) {
        const bool above = ss > limit;
        if (!more && above) sc[IS_CAPHIT] = 1.0;
        more = more && above;
    }
    return more;
}

// sets the condition of the graph's while node
__global__ void k_icg_cond(cudaGraphConditionalHandle h, double *__restrict__ sc, const double *__restrict__ part,
                           int nb, int kmax, double eta_min, const double *__restrict__ outer,
                           double *__restrict__ total) {
    const bool more = icg_more(sc, part, nb, kmax, eta_min, outer, total);
    if (threadIdx.x == 0) cudaGraphSetConditional(h, more ? 1u : 0u);
}

// sets a conditional handle: a handle's default value is applied when the
// top-level graph is launched, not when a conditional body containing its
// node runs again, so a loop nested in another loop's body is re-armed with
// this kernel before each entry
__global__ void k_set_cond(cudaGraphConditionalHandle h, unsigned v) {
    if (threadIdx.x == 0) cudaGraphSetConditional(h, v);
}

void launch_set_cond(cudaGraphConditionalHandle h, unsigned v, cudaStream_t s) {
    ++g_launches;
    k_set_cond<<<1, 32, 0, s>>>(h, v);
}

// after the outer residual test: keep the outer while loop going and apply
// the preconditioner (the if node) unless the solve stopped (iflag[2])
__global__ void k_outer_cond(cudaGraphConditionalHandle hw, cudaGraphConditionalHandle hi,
                             const int *__restrict__ iflag) {
    if (threadIdx.x != 0) return;
    const unsigned go = iflag[2] ? 0u : 1u;
    cudaGraphSetConditional(hw, go);
    cudaGraphSetConditional(hi, go);
}

void launch_outer_cond(cudaGraphConditionalHandle hw, cudaGraphConditionalHandle hi, const int *iflag,
                       cudaStream_t s) {
    ++g_launches;
    k_outer_cond<<<1, 32, 0, s>>>(hw, hi, iflag);
}

// the same decision written to *flag for a host-driven loop (profiling: the
// kernels of a conditional graph body do not appear in a profiler's launch list)
__global__ void k_icg_cond_flag(int *flag, double *__restrict__ sc, const double *__restrict__ part, int nb,
                                int kmax, double eta_min, const double *__restrict__ outer,
                                double *__restrict__ total) {
    const bool more = icg_more(sc, part, nb, kmax, eta_min, outer, total);
    if (threadIdx.x == 0) *flag = more ? 1 : 0;
}

void launch_icg_cond_flag(int *flag, double *sc, const double *part, int nb, int kmax, double eta_min,
                          const double *outer, double *total, cudaStream_t s) {
    ++g_launches;
    k_icg_cond_flag<<<1, MB, 0, s>>>(flag, sc, part, nb, kmax, eta_min, outer, total);
}

void launch_icg_cond(cudaGraphConditionalHandle h, double *sc, const double *part, int nb, int kmax,
                     double eta_min, const double *outer, double *total, cudaStream_t s) {
    ++g_launches;
    k_icg_cond<<<1, MB, 0, s>>>(h, sc, part, nb, kmax, eta_min, outer, total);
}

// s = r, e = 0, d = 0 and partial sums of s.s (entry of an inner solve)
__global__ void k_icg_init(const float *__restrict__ r, float *__restrict__ s, float *__restrict__ e,
                           float *__restrict__ d, int64_t n, double *__restrict__ part) {
    float acc = 0.f;
    for (int64_t i = blockIdx.x * (int64_t)MB + threadIdx.x; i < n; i += (int64_t)gridDim.x * MB) {
        const float v = r[i];
        s[i] = v;
        e[i] = 0.f;
        d[i] = 0.f;
        acc = fmaf(v, v, acc);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    __shared__ double wred[MB / 32];
    if ((threadIdx.x & 31) == 0) wred[threadIdx.x >> 5] = (double)acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int i = 0; i < MB / 32; ++i) t += wred[i];
        part[blockIdx.x] = t;
    }
}

int launch_icg_init(const float *r, float *s, float *e, float *d, int64_t n, double *part, cudaStream_t st) {
    ++g_launches;
    const int nb = reduce_blocks(n);
    k_icg_init<<<nb, MB, 0, st>>>(r, s, e, d, n, part);
    return nb;
}

void launch_icg_scalar(int op, double *sc, const double *part, int nb, cudaStream_t s, int kbase, int klimit) {
    ++g_launches;
    k_icg_scalar<<<1, MB, 0, s>>>(op, sc, part, nb, kbase, klimit);
}

// The FP32 vectors are separate allocations (256-byte aligned), so the
// streaming kernels below move them as float4 and finish the n % 4 tail
// element-wise.
__device__ __forceinline__ float4 fma4(float a, float4 x, float4 y) {
    return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}

// s -= alpha t; partial sums of s.s (new s).  The matching e += alpha d is deferred to
// the next d update (k_icg_dupdate), or, after the last iteration, to k_widen_dots: d is
// read there anyway, which saves one pass over e and d per iteration.  Bound by the
// vectors' traffic on large grids and by latency on small ones, so a thread's first
// words are on their way while its CTA sums the partials.
__device__ __forceinline__ float sq4(float4 v, float acc) {
    return fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, acc))));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// v: lane 0's is the warp's
__device__ __forceinline__ void store_partial(double v, double *__restrict__ part) {
    __shared__ double wred[UB / 32];
    if ((threadIdx.x & 31) == 0) wred[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < UB / 32; ++k) t += wred[k];
        part[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(UB, 4) k_icg_update(float *__restrict__ s, const float *__restrict__ t, int64_t n,
                                                   double *__restrict__ sc, const double *__restrict__ sum, int nsum,
                                                   double *__restrict__ part) {
    const int64_t n4 = n >> 2, stride = (int64_t)gridDim.x * UB, i0 = blockIdx.x * (int64_t)UB + threadIdx.x;
    float4 *s4 = reinterpret_cast<float4 *>(s);
    const float4 *t4 = reinterpret_cast<const float4 *>(t);
    float4 sv = make_float4(0.f, 0.f, 0.f, 0.f), tv = sv;
    if (i0 < n4) {
        sv = s4[i0];
        tv = t4[i0];
    }
    const float a = icg_coefficient<1>(sc, sum, nsum);
    float acc = 0.f;
    if (i0 < n4) {
        sv = fma4(-a, tv, sv);
        s4[i0] = sv;
        acc = sq4(sv, acc);
    }
#pragma unroll 2
    for (int64_t i = i0 + stride; i < n4; i += stride) {
        const float4 v = fma4(-a, t4[i], s4[i]);
        s4[i] = v;
        acc = sq4(v, acc);
    }
    const int64_t i = 4 * n4 + i0;
    if (i < n) {
        const float v = fmaf(-a, t[i], s[i]);
        s[i] = v;
        acc = fmaf(v, v, acc);
    }
    store_partial((double)warp_sum(acc), part);
}

// e += alpha d (the previous iteration's step, alpha still in place); then d = w + beta d
__global__ void __launch_bounds__(UB, 4) k_icg_dupdate(float *__restrict__ e, float *__restrict__ d,
                                                    const float *__restrict__ w, int64_t n, double *__restrict__ sc,
                                                    const double *__restrict__ sum, int nsum) {
    const int64_t n4 = n >> 2, stride = (int64_t)gridDim.x * UB, i0 = blockIdx.x * (int64_t)UB + threadIdx.x;
    float4 *e4 = reinterpret_cast<float4 *>(e), *d4 = reinterpret_cast<float4 *>(d);
    const float4 *w4 = reinterpret_cast<const float4 *>(w);
    float4 ev = make_float4(0.f, 0.f, 0.f, 0.f), dv = ev, wv = ev;
    if (i0 < n4) {
        dv = d4[i0];
        ev = e4[i0];
        wv = w4[i0];
    }
    const float a = (float)sc[IS_ALPHA], b = icg_coefficient<2>(sc, sum, nsum);
    if (i0 < n4) {
        e4[i0] = fma4(a, dv, ev);
        d4[i0] = fma4(b, dv, wv);
    }
#pragma unroll 2
    for (int64_t i = i0 + stride; i < n4; i += stride) {
        const float4 v = d4[i];
        e4[i] = fma4(a, v, e4[i]);
        d4[i] = fma4(b, v, w4[i]);
    }
    const int64_t i = 4 * n4 + i0;
    if (i < n) {
        const float v = d[i];
        e[i] = fmaf(a, v, e[i]);
        d[i] = fmaf(b, v, w[i]);
    }
}

// ---- the same two updates over the active runs only -------------------------
// On a grid with inactive regions the inner CG's vectors are exactly zero at
// inactive nodes: the inner solve's entry kernel writes every node, K*u and
// the V-cycle leave zeros there, and these updates keep zeros zero.  So the
// updates may visit only the active nodes' words.
// The active y-runs (merged where they touch or lie a few nodes apart) are
// cut into chunks of at most 2048 floats, each cut on a 16-byte boundary
// (runs[i] = first DOF | floats << 40).  A warp takes a chunk: float4 groups, and
// the words before the first and after the last 16-byte boundary one by one.  A
// chunk is mostly one or two groups a lane, so its time is the latency of its
// loads: the single words and the first RUN_BATCH groups are loaded together, those of
// the warp's first chunk before the partials are summed.  (Head words, groups
// and tail words each with their own loads and stores: 58 and 37 us for the d and s update
// of the 384 x 192 x 192 blob shape, now 49 and 28; 18.5 and 16.5 us on 192 x 96 x 96, now
// 13 and 12.)  Sums visit the chunks in a fixed order.
constexpr int RUN_SHIFT = 40;
constexpr int64_t RUN_MASK = (int64_t(1) << RUN_SHIFT) - 1;
constexpr int RUN_BATCH = 4, RUN_BATCH3 = 3;   // groups a lane loads at once, of two and of three vectors

// a warp's chunk: word `single` of this lane (-1: none), n4 groups from group g4
struct RunChunk {
    int64_t single = -1, g4 = 0;
    int n4 = 0;
    __device__ __forceinline__ void take(int64_t rv, int lane) {
        const int64_t b = rv & RUN_MASK;
        const int len = (int)(rv >> RUN_SHIFT), head = min((int)((4 - (b & 3)) & 3), len);
        g4 = (b + head) >> 2;
        n4 = (len - head) >> 2;
        const int rest = len - head - 4 * n4;
        single = lane < head ? b + lane : lane >= 4 && lane < 4 + rest ? b + head + 4 * (int64_t)n4 + (lane - 4) : -1;
    }
};

// NV vectors' words of a chunk: the single word and a batch of groups
template <int NV, int Q>
struct RunWords {
    float one[NV];
    float4 four[Q][NV];
    __device__ __forceinline__ void load(const RunChunk &c, int k0, const float *const (&v)[NV]) {
#pragma unroll
        for (int j = 0; j < NV; ++j) one[j] = k0 < 32 && c.single >= 0 ? v[j][c.single] : 0.f;
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int j = 0; j < NV; ++j)
                four[q][j] = k0 + 32 * q < c.n4 ? reinterpret_cast<const float4 *>(v[j])[c.g4 + k0 + 32 * q]
                                                : make_float4(0.f, 0.f, 0.f, 0.f);
    }
};

__global__ void __launch_bounds__(UB, 2) k_icg_update_runs(float *s, const float *t, const int64_t *__restrict__ runs,
                                                        int64_t nruns, double *__restrict__ sc,
                                                        const double *__restrict__ sum, int nsum,
                                                        double *__restrict__ part) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = (int64_t)blockIdx.x * (UB / 32) + (threadIdx.x >> 5), nw = (int64_t)gridDim.x * (UB / 32);
    const float *const src[2] = {s, t};
    RunChunk c;
    RunWords<2, RUN_BATCH> x;
    if (w0 < nruns) {
        c.take(runs[w0], lane);
        x.load(c, lane, src);
    }
    const float a = icg_coefficient<1>(sc, sum, nsum);
    // a warp's even and odd chunks apart: 9728 sums over the grid, as long a chain in FP32 as with
    // twice the warps
    float acc = 0.f, other = 0.f;
    for (int64_t r = w0; r < nruns;) {
        const int64_t rv = runs[min(r + nw, nruns - 1)];
        if (c.single >= 0) {
            const float v = fmaf(-a, x.one[1], x.one[0]);
            s[c.single] = v;
            acc = fmaf(v, v, acc);
        }
        for (int k0 = lane;;) {
#pragma unroll
            for (int q = 0; q < RUN_BATCH; ++q)
                if (k0 + 32 * q < c.n4) {
                    const float4 v = fma4(-a, x.four[q][1], x.four[q][0]);
                    reinterpret_cast<float4 *>(s)[c.g4 + k0 + 32 * q] = v;
                    acc = sq4(v, acc);
                }
            k0 += 32 * RUN_BATCH;
            if (k0 - lane >= c.n4) break;
            x.load(c, k0, src);
        }
        const float last = acc;
        acc = other;
        other = last;
        if ((r += nw) >= nruns) break;
        c.take(rv, lane);
        x.load(c, lane, src);
    }
    store_partial((double)warp_sum(acc) + (double)warp_sum(other), part);
}

__global__ void __launch_bounds__(UB, 2) k_icg_dupdate_runs(float *e, float *d, const float *w,
                                                         const int64_t *__restrict__ runs, int64_t nruns,
                                                         double *__restrict__ sc, const double *__restrict__ sum,
                                                         int nsum) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = (int64_t)blockIdx.x * (UB / 32) + (threadIdx.x >> 5), nw = (int64_t)gridDim.x * (UB / 32);
    const float *const src[3] = {e, d, w};
    RunChunk c;
    RunWords<3, RUN_BATCH3> x;
    if (w0 < nruns) {
        c.take(runs[w0], lane);
        x.load(c, lane, src);
    }
    const float a = (float)sc[IS_ALPHA], b = icg_coefficient<2>(sc, sum, nsum);
    for (int64_t r = w0; r < nruns;) {
        const int64_t rv = runs[min(r + nw, nruns - 1)];
        if (c.single >= 0) {
            e[c.single] = fmaf(a, x.one[1], x.one[0]);
            d[c.single] = fmaf(b, x.one[1], x.one[2]);
        }
        for (int k0 = lane;;) {
#pragma unroll
            for (int q = 0; q < RUN_BATCH3; ++q)
                if (k0 + 32 * q < c.n4) {
                    reinterpret_cast<float4 *>(e)[c.g4 + k0 + 32 * q] = fma4(a, x.four[q][1], x.four[q][0]);
                    reinterpret_cast<float4 *>(d)[c.g4 + k0 + 32 * q] = fma4(b, x.four[q][1], x.four[q][2]);
                }
            k0 += 32 * RUN_BATCH3;
            if (k0 - lane >= c.n4) break;
            x.load(c, k0, src);
        }
        if ((r += nw) >= nruns) break;
        c.take(rv, lane);
        x.load(c, lane, src);
    }
}

// CTAs over the chunks, a warp each, at most `most`: the s update runs best as the two CTAs
// that an SM holds (384 x 192 x 192 blob shape: 28 us, 32 with 8 per SM), the d update,
// whose traffic is 2.5 times that, with more, which the SMs take as they finish (49 us, 70 with two)
static int run_blocks(int64_t nruns, int most) {
    const int64_t b = (nruns + UB / 32 - 1) / (UB / 32);
    return (int)(b < most ? (b > 0 ? b : 1) : most);
}
static int update_blocks(int64_t n) {
    const int64_t b = (n / 4 + UB - 1) / UB;
    return (int)(b < 2 * UGRID ? (b > 0 ? b : 1) : 2 * UGRID);
}

// the scalar of an update from nb partials: by the update itself, or by a launch before it
static int icg_sum(int op, double *sc, const double *sum, int nb, cudaStream_t st) {
    if (nb <= FUSE_PARTS) return nb;
    launch_icg_scalar(op, sc, sum, nb, st, 0, 0);
    return 0;
}

void launch_icg_dupdate(float *e, float *d, const float *w, const Level &l0, double *sc, const double *sum, int nb,
                        cudaStream_t st) {
    const int nsum = icg_sum(2, sc, sum, nb, st);
    ++g_launches;
    if (l0.runs) {
        k_icg_dupdate_runs<<<run_blocks(l0.nruns, 152 * 8), UB, 0, st>>>(e, d, w, l0.runs, l0.nruns, sc, sum, nsum);
    } else {
        const int64_t n = 3 * l0.nnode;
        k_icg_dupdate<<<update_blocks(n), UB, 0, st>>>(e, d, w, n, sc, sum, nsum);
    }
}

int launch_icg_update(float *s, const float *t, const Level &l0, double *sc, const double *sum, int nb, double *part,
                      cudaStream_t st) {
    const int nsum = icg_sum(1, sc, sum, nb, st);
    ++g_launches;
    const int64_t n = 3 * l0.nnode;
    const int g = l0.runs ? run_blocks(l0.nruns, UGRID) : update_blocks(n);
    if (l0.runs)
        k_icg_update_runs<<<g, UB, 0, st>>>(s, t, l0.runs, l0.nruns, sc, sum, nsum, part);
    else
        k_icg_update<<<g, UB, 0, st>>>(s, t, n, sc, sum, nsum, part);
    return g;
}

// z64 = e32 + alpha d32 (the last iteration's deferred step; masked at fixed
// DOFs by construction), partials of z.r and z.q
__global__ void k_widen_dots(const float *__restrict__ e, const float *__restrict__ d,
                             const double *__restrict__ sc, double *__restrict__ z, const double *__restrict__ r,
                             const double *__restrict__ q, int64_t n, double *__restrict__ p1,
                             double *__restrict__ p2) {
    const float al = (float)sc[IS_ALPHA];
    double a = 0.0, b = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)MB + threadIdx.x; i < n; i += (int64_t)gridDim.x * MB) {
        const double zi = (double)fmaf(al, d[i], e[i]);
        z[i] = zi;
        a += zi * r[i];
        b += zi * q[i];
    }
    a = mblock_reduce(a);
    b = mblock_reduce(b);
    if (threadIdx.x == 0) {
        p1[blockIdx.x] = a;
        p2[blockIdx.x] = b;
    }
}

void launch_widen_dots(const float *e, const float *d, const double *sc, double *z, const double *r,
                       const double *q, int64_t n, double *p1, double *p2, int nb, cudaStream_t st) {
    ++g_launches;
    k_widen_dots<<<nb, MB, 0, st>>>(e, d, sc, z, r, q, n, p1, p2);
}

// outer flexible-PCG scalars after the preconditioner: beta = -lambda zq / x1, x1 = zr
// (slots as in kernels_vec.cu: S_X1 = 1, S_LAM = 2, S_BETA = 4)
__global__ void k_flex_beta(double *__restrict__ scal, const int *__restrict__ iflag, const double *__restrict__ p1,
                            const double *__restrict__ p2, int nb, int first) {
    const double zr = msum_partials(p1, nb);
    const double zq = msum_partials(p2, nb);
    if (threadIdx.x != 0) return;
    if (first) {
        scal[1] = zr;
        return;
    }
    if (iflag[2]) return;
    scal[4] = -scal[2] * zq / scal[1];
    scal[1] = zr;
}

void launch_flex_beta(double *scal, const int *iflag, const double *p1, const double *p2, int nb, int first,
                      cudaStream_t st) {
    ++g_launches;
    k_flex_beta<<<1, MB, 0, st>>>(scal, iflag, p1, p2, nb, first);
}

// r32 = (float) r64
__global__ void k_narrow(const double *__restrict__ a, float *__restrict__ b, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)MB + threadIdx.x; i < n; i += (int64_t)gridDim.x * MB) b[i] = (float)a[i];
}

void launch_narrow(const double *a, float *b, int64_t n, cudaStream_t st) {
    ++g_launches;
    k_narrow<<<reduce_blocks(n), MB, 0, st>>>(a, b, n);
}

// r64 = (double) r32
__global__ void k_widen(const float *__restrict__ a, double *__restrict__ b, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)MB + threadIdx.x; i < n; i += (int64_t)gridDim.x * MB) b[i] = (double)a[i];
}

void launch_widen(const float *a, double *b, int64_t n, cudaStream_t st) {
    ++g_launches;
    k_widen<<<reduce_blocks(n), MB, 0, st>>>(a, b, n);
}

}  // namespace sgld
