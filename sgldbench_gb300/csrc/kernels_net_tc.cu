// The U-Net's 3x3x3 convolutions (forward, data gradient and weight gradient)
// on the tensor cores: tcgen05.mma on BF16 operands with FP32 accumulation in
// tensor memory.  Same operands and epilogues as the CUDA-core convolutions
// (kernels_net.cu): BF16 activations and weights, FP32 gradients rounded to BF16
// as operands (once per gradient, by the caller).
//
// Forward and data gradient: an implicit GEMM per CTA of 128 output voxels x all
// output channels, reduced over 27 taps x input channels.  Per tap t a CTA of 4 warps
//   * copies A = the 128 voxels' neighbours at tap t (cin channels each, zero
//     outside the grid or past cin) into shared memory in the MMA's K-major
//     core-matrix layout, one 16-byte cp.async per 8 channels,
//   * copies B = the tap's weight image (cout rows x cin, the same layout,
//     prepared once per pass for all convolutions by k_wimages),
//   * and one thread issues cin/16 MMAs of 128 x cout x 16 into the TMEM
//     accumulator, then commits them to the buffer's mbarrier.
// A tap's work is a memory latency and little else, and the coarse levels have
// only a few CTAs, so the copies run three taps ahead of the MMAs in a ring of four
// buffers; a buffer is refilled once the commit of the tap that last used it has
// arrived (bounded waits).  (Gathered in registers and stored when they came, one tap
// at a time, a launch of the 65 x 33 x 33 network took 66 to 134 us on its two coarsest
// levels, now 23 to 25, and 49 to 72 us on the others, now 19 to 28.)
// The epilogue reads the accumulator with tcgen05.ld (warp w holds voxel rows 32w ..
// 32w+31) and stores 4 channels at a time.
#include <cuda_bf16.h>

#include <algorithm>

#include "sgld_net.cuh"
#include "tc_ptx.cuh"

namespace sgld {

namespace {
constexpr int TC_BM = 128;   // output voxels per CTA (the MMA's M)
constexpr int TC_CMAX = 64;  // channels on either side (K and N padded to 16)

__device__ __forceinline__ uint16_t bf16_bits(bf16 v) { return __bfloat16_as_ushort(v); }

// 16 bytes global -> shared, asynchronously; bytes past n (0 or 16) are zeros
__device__ __forceinline__ void copy16(uint32_t dst, const void *src, uint32_t n) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {   // all but the last N groups have landed
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// the C channels of a voxel's row src as 16-byte chunks 128 bytes apart at dst, KP channels
// in all; zeros past C and everywhere unless on.  vec: rows are 16-byte aligned, and
// the copies are asynchronous.
__device__ __forceinline__ void stage_row(uint32_t dst, const bf16 *src, bool on, int C, int KP, bool vec) {
    if (vec) {
        const uint32_t n = on ? 16u : 0u;
#pragma unroll 4
        for (int c = 0; c < C; c += 8) copy16(dst + 16 * c, src + c, n);
        for (int c = C; c < KP; c += 8) copy16(dst + 16 * c, src, 0u);
    } else {
        for (int c = 0; c < KP; c += 8) {
            uint32_t h[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t lo = on && c + 2 * j < C ? bf16_bits(src[c + 2 * j]) : 0u;
                const uint32_t hi = on && c + 2 * j + 1 < C ? bf16_bits(src[c + 2 * j + 1]) : 0u;
                h[j] = lo | hi << 16;
            }
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(dst + 16 * c), "r"(h[0]), "r"(h[1]),
                         "r"(h[2]), "r"(h[3])
                         : "memory");
        }
    }
}

// Bit t of the mask: the neighbour at tap t = (dy+1) + 3(dx+1) + 9(dz+1) is in the grid.
// Computed once per voxel, so that a tap costs a bit test and an offset that all threads share.
__device__ __forceinline__ uint32_t tap_mask(int y, int x, int z, int taps, int ny, int nx, int nz) {
    if (taps == 1) return 1u;
    const uint32_t my = (y > 0 ? 1u : 0u) | 2u | (y + 1 < ny ? 4u : 0u);
    const uint32_t mx = (x > 0 ? my : 0u) | my << 3 | (x + 1 < nx ? my << 6 : 0u);
    return (z > 0 ? mx : 0u) | mx << 9 | (z + 1 < nz ? mx << 18 : 0u);
}
__device__ __forceinline__ int64_t tap_offset(int t, int taps, int ny, int nx) {
    return taps == 1 ? 0 : (t % 3 - 1) + (int64_t)ny * ((t / 3) % 3 - 1 + (int64_t)nx * (t / 9 - 1));
}
}  // namespace

// Weight images of all convolutions, one launch: img[t] = the B operand of tap t (NP x
// KP, K-major core matrices).  Forward: row n, column k holds W[t][k][n] (K = cin, N =
// cout).  flip (data gradient): W[taps-1-t][n][k] (K = cout, N = cin).  Zero elsewhere.
__global__ void k_wimages(const bf16 *__restrict__ w, const __grid_constant__ NetImages im, int flip,
                          bf16 *__restrict__ out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= im.at[im.n]) return;
    int c = 0;
    while (i >= im.at[c + 1]) ++c;
    const int taps = im.taps[c], cin = im.cin[c], cout = im.cout[c], K = flip ? cout : cin, N = flip ? cin : cout;
    const int KP = (K + 15) & ~15, NP = (N + 15) & ~15;
    const int64_t per = (int64_t)NP * KP, j = i - im.at[c];
    const int t = (int)(j / per), rem = (int)(j - t * per), n = rem / KP, k = rem - n * KP;
    const bf16 *W = w + im.w[c];
    bf16 v = __float2bfloat16_rn(0.f);
    if (k < K && n < N) v = flip ? W[((int64_t)(taps - 1 - t) * cin + n) * cout + k] : W[((int64_t)t * cin + k) * cout + n];
    out[im.at[c] + t * per + tc::canon_off(n, k, KP) / 2] = v;
}

constexpr int TC_NS = 4;   // buffers of the convolution's ring

// MODE 0: BF16 out = relu(. + bias)     MODE 1: FP32 out = . + bias (linear head)
// MODE 2: FP32 out (=/+=) mask(.)      (gradient of a ReLU output when mask != null)
template <int MODE>
__global__ void __launch_bounds__(TC_BM) k_conv_tc(const bf16 *__restrict__ in, int cin, const bf16 *__restrict__ wimg,
                                                   int KP, int NP, const float *__restrict__ bias, int cout, int taps,
                                                   int ny, int nx, int nz, void *__restrict__ outp,
                                                   const bf16 *__restrict__ mask, int accumulate,
                                                   int *__restrict__ err) {
    extern __shared__ __align__(128) unsigned char tsm[];
    const int abytes = TC_BM * KP * 2, bbytes = NP * KP * 2;
    unsigned char *Abuf = tsm;                      // [TC_NS][abytes]
    unsigned char *Bbuf = tsm + TC_NS * abytes;     // [TC_NS][bbytes]
    uint64_t *bars = reinterpret_cast<uint64_t *>(tsm + TC_NS * (abytes + bbytes));
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bars + TC_NS);
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t ncols = NP <= 32 ? 32u : 64u;
    const int64_t V = (int64_t)ny * nx * nz;
    const int64_t v = (int64_t)blockIdx.x * TC_BM + tid;   // this thread's voxel = row tid of A
    int y = 0, x = 0, z = 0;
    if (v < V) {
        y = (int)(v % ny);
        x = (int)((v / ny) % nx);
        z = (int)(v / ((int64_t)ny * nx));
    }
    const bool vec = (cin & 7) == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0;
    const uint32_t there = v < V ? tap_mask(y, x, z, taps, ny, nx, nz) : 0u;
    const bf16 *row = in + (v < V ? v : 0) * cin;
    const uint32_t arow = tc::saddr(Abuf + tc::canon_off(tid, 0, KP)), brow = tc::saddr(Bbuf + 16 * tid);
    auto stage = [&](int t) {   // tap t into buffer t mod TC_NS
        if (t < taps) {
            const bool on = there >> t & 1;
            stage_row(arow + t % TC_NS * abytes, on ? row + tap_offset(t, taps, ny, nx) * cin : in, on, cin, KP, vec);
            const unsigned char *src = reinterpret_cast<const unsigned char *>(wimg) + (int64_t)t * bbytes;
#pragma unroll 4
            for (int i = 16 * tid; i < bbytes; i += 16 * TC_BM) copy16(brow + t % TC_NS * bbytes + i - 16 * tid, src + i, 16u);
        }
        copies_commit();
    };
    for (int t = 0; t < TC_NS - 1; ++t) stage(t);
    if (warp == 0) {
        tc::tmem_alloc(tc::saddr(tslot), ncols);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        for (int i = 0; i < TC_NS; ++i) tc::mbar_init(tc::saddr(bars + i), 1);
        tc::mbar_init_fence();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t taddr = *tslot;
    const uint32_t idesc = tc::idesc_bf16(TC_BM, NP);
    const uint32_t lbo = 128, sbo = (uint32_t)(KP / 8) * 128;
    bool ok = true;
    for (int t = 0; t < taps; ++t) {
        const int buf = t % TC_NS;
        copies_wait<TC_NS - 2>();   // this thread's copies of tap t
        tc::fence_proxy_async();
        __syncthreads();
        if (tid == 0) {
            tc::tc_fence_after();
            const uint32_t a0 = tc::saddr(Abuf + buf * abytes), b0 = tc::saddr(Bbuf + buf * bbytes);
            for (int kk = 0; kk < KP / 16; ++kk)
                tc::mma_bf16(taddr, tc::smem_desc(a0 + 256 * kk, lbo, sbo), tc::smem_desc(b0 + 256 * kk, lbo, sbo),
                             idesc, (t > 0 || kk > 0) ? 1u : 0u);
            tc::mma_commit(tc::saddr(bars + buf));
        }
        // the next tap to fetch takes the buffer of tap t-1: wait for its MMAs
        const int u = t - 1;
        if (t > 0 && t + TC_NS - 1 < taps) ok = tc::mbar_wait(tc::saddr(bars + u % TC_NS), (u / TC_NS) & 1) && ok;
        stage(t + TC_NS - 1);
    }
    copies_wait<0>();
    // the last commit covers every MMA issued before it
    const int lu = taps - 1;
    ok = tc::mbar_wait(tc::saddr(bars + lu % TC_NS), (uint32_t)((lu / TC_NS) & 1)) && ok;
    tc::tc_fence_after();
    if (__syncthreads_or(!ok)) {
        // a wait gave up: wait once more (bounded) so that no MMA is in flight, free TMEM, flag it
        tc::mbar_wait(tc::saddr(bars + lu % TC_NS), (uint32_t)((lu / TC_NS) & 1));
        tc::tc_fence_before();
        __syncthreads();
        if (warp == 0) tc::tmem_dealloc(taddr, ncols);
        if (tid == 0 && err) atomicExch(err, 1);
        return;
    }
    const bool quads = (cout & 3) == 0;   // rows of whole 4-channel groups: 8- and 16-byte accesses
    for (int c0 = 0; c0 < NP; c0 += 16) {
        float r[16];
        tc::tmem_ld16(taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, r);
        if (v >= V) continue;
        if (quads) {
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
                if (c0 + j >= cout) continue;
                const int64_t o = v * cout + c0 + j;
                float val[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) val[k] = r[j + k] + ((MODE != 2 && bias) ? bias[c0 + j + k] : 0.f);
                if (MODE == 0) {
                    uint32_t h[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        h[k] = (uint32_t)bf16_bits(__float2bfloat16_rn(fmaxf(val[2 * k], 0.f))) |
                               (uint32_t)bf16_bits(__float2bfloat16_rn(fmaxf(val[2 * k + 1], 0.f))) << 16;
                    *reinterpret_cast<uint2 *>(static_cast<bf16 *>(outp) + o) = make_uint2(h[0], h[1]);
                } else {
                    float4 *out = reinterpret_cast<float4 *>(static_cast<float *>(outp) + o);
                    if (MODE == 2) {
                        if (mask) {
                            const uint2 m = *reinterpret_cast<const uint2 *>(mask + o);
                            const uint32_t mb[2] = {m.x, m.y};
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                if (!(__bfloat162float(__ushort_as_bfloat16((uint16_t)(mb[k >> 1] >> (16 * (k & 1))))) > 0.f))
                                    val[k] = 0.f;
                        }
                        if (accumulate) {
                            const float4 old = *out;
                            val[0] = old.x + val[0];
                            val[1] = old.y + val[1];
                            val[2] = old.z + val[2];
                            val[3] = old.w + val[3];
                        }
                    }
                    *out = make_float4(val[0], val[1], val[2], val[3]);
                }
            }
            continue;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int co = c0 + j;
            if (co >= cout) continue;
            const int64_t o = v * cout + co;
            float val = r[j] + ((MODE != 2 && bias) ? bias[co] : 0.f);
            if (MODE == 0) {
                static_cast<bf16 *>(outp)[o] = __float2bfloat16_rn(fmaxf(val, 0.f));
            } else if (MODE == 1) {
                static_cast<float *>(outp)[o] = val;
            } else {
                if (mask && !(__bfloat162float(mask[o]) > 0.f)) val = 0.f;
                float *out = static_cast<float *>(outp);
                out[o] = accumulate ? out[o] + val : val;
            }
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(taddr, ncols);
}

// Weight and bias gradients of one convolution on the tensor cores, split over
// voxel ranges like the FP32-pipe k_conv_wgrad:
//   part[s][t][ci][co] = sum_{v in range s} in[nb(v,t)][ci] * g[v][co]
//   part[s][taps*cin*cout + co] = sum_{v in range s} g[v][co]     (the bias)
// as D = A B^T, K = the voxels of the CTA's range, 128 per block, all accumulated in
// one TMEM tile.  A's 128 rows are the channels at TG taps (as many as fit: row tl CP
// + ci for tap blockIdx.x TG + tl, CP = cin rounded up to 8) and, for the group with
// the centre tap, one row of ones after them, so that D's row there is the bias
// sum; B's rows are the cout gradient channels (BF16).
// Both operands are channels-last in memory, which is the MMA's MN-major layout: 8
// channels of a voxel are the 16 contiguous bytes of a core-matrix row, so they are
// copied as they are (16-byte cp.async, two blocks ahead in a ring of three) and the
// instruction reads them transposed.  (K-major, the copy transposed them 2 bytes at a
// time, and a CTA did one tap: 31 to 101 us a launch, now 9 to 47, and 65 for the 34
// ranges of the 8-channel input.)
constexpr int WG_NS = 3;

__global__ void __launch_bounds__(TC_BM) k_conv_wgrad_tc(const bf16 *__restrict__ in, int cin,
                                                         const bf16 *__restrict__ g, int cout, int NP, int taps, int TG,
                                                         int ny, int nx, int nz, int64_t vchunk,
                                                         float *__restrict__ part, int64_t pstride,
                                                         int *__restrict__ err) {
    extern __shared__ __align__(128) unsigned char tsm[];
    constexpr int KB = TC_BM;                     // voxels per block (the K of 8 MMAs)
    // MN-major core matrices: 8 channels x 8 voxels of 128 bytes; blocks along the channels
    // adjacent (128 bytes), blocks of 8 voxels alb / blb bytes apart
    const int alb = TC_BM / 8 * 128, blb = NP / 8 * 128;
    const int abytes = TC_BM * KB * 2, bbytes = NP * KB * 2;
    unsigned char *Abuf = tsm, *Bbuf = tsm + WG_NS * abytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(tsm + WG_NS * (abytes + bbytes));
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bars + WG_NS);
    const int tid = threadIdx.x, warp = tid >> 5;
    const int t0 = blockIdx.x * TG, s = blockIdx.y;
    const int CP = (cin + 7) & ~7, ones = TG * CP;   // the row of ones
    const int centre = taps == 1 ? 0 : 13;
    const bool bias = t0 <= centre && centre < t0 + TG;
    const uint32_t ncols = NP <= 32 ? 32u : 64u;
    // rows that no tap fills stay zero: clear the buffers once
    for (int i = tid; i < WG_NS * abytes / 16; i += TC_BM) reinterpret_cast<uint4 *>(Abuf)[i] = make_uint4(0, 0, 0, 0);
    if (warp == 0) {
        tc::tmem_alloc(tc::saddr(tslot), ncols);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        for (int i = 0; i < WG_NS; ++i) tc::mbar_init(tc::saddr(bars + i), 1);
        tc::mbar_init_fence();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t taddr = *tslot;
    const int64_t V = (int64_t)ny * nx * nz;
    const int64_t vb = (int64_t)s * vchunk, ve = min(V, vb + vchunk);
    const int nblk = ve > vb ? (int)((ve - vb + KB - 1) / KB) : 0;
    const uint32_t idesc = tc::idesc_bf16(TC_BM, NP) | tc::IDESC_MN_MAJOR;
    const bool vec_in = (cin & 7) == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0;
    const bool vec_g = (cout & 7) == 0 && (reinterpret_cast<uintptr_t>(g) & 15) == 0;
    auto stage = [&](int b) {   // voxel block b into buffer b mod WG_NS; column tid of both operands
        if (b < nblk) {
            const uint32_t A = tc::saddr(Abuf + b % WG_NS * abytes + (tid >> 3) * alb + (tid & 7) * 16);
            const uint32_t B = tc::saddr(Bbuf + b % WG_NS * bbytes + (tid >> 3) * blb + (tid & 7) * 16);
            const int64_t v = vb + (int64_t)b * KB + tid;
            const bool valid = v < ve;
            const unsigned vu = valid ? (unsigned)v : 0u, col = vu / ny;
            const uint32_t there =
                valid ? tap_mask((int)(vu - col * ny), (int)(col % nx), (int)(col / nx), taps, ny, nx, nz) : 0u;
            const bf16 *row = in + (int64_t)vu * cin;
            const int tn = min(TG, taps - t0);
            for (int tl = 0; tl < tn; ++tl) {
                const bool on = there >> (t0 + tl) & 1;
                stage_row(A + tl * CP * 16, on ? row + tap_offset(t0 + tl, taps, ny, nx) * cin : in, on, cin, CP, vec_in);
            }
            if (bias)
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %2, %2};\n" ::"r"(A + ones * 16),
                             "r"(valid ? (uint32_t)bf16_bits(__float2bfloat16_rn(1.f)) : 0u), "r"(0)
                             : "memory");
            stage_row(B, valid ? g + v * cout : g, valid, cout, NP, vec_g);
        }
        copies_commit();
    };
    for (int b = 0; b < WG_NS - 1; ++b) stage(b);
    bool ok = true;
    for (int b = 0; b < nblk; ++b) {
        const int buf = b % WG_NS;
        copies_wait<WG_NS - 2>();
        tc::fence_proxy_async();
        __syncthreads();
        if (tid == 0) {
            tc::tc_fence_after();
            const uint32_t a0 = tc::saddr(Abuf + buf * abytes), b0 = tc::saddr(Bbuf + buf * bbytes);
            for (int kk = 0; kk < KB / 16; ++kk)
                tc::mma_bf16(taddr, tc::smem_desc(a0 + 2 * alb * kk, alb, 128), tc::smem_desc(b0 + 2 * blb * kk, blb, 128),
                             idesc, (b > 0 || kk > 0) ? 1u : 0u);
            tc::mma_commit(tc::saddr(bars + buf));
        }
        const int u = b - 1;
        if (b > 0 && b + WG_NS - 1 < nblk) ok = tc::mbar_wait(tc::saddr(bars + u % WG_NS), (u / WG_NS) & 1) && ok;
        stage(b + WG_NS - 1);
    }
    copies_wait<0>();
    const int lu = nblk - 1;
    if (nblk > 0) ok = tc::mbar_wait(tc::saddr(bars + lu % WG_NS), (uint32_t)((lu / WG_NS) & 1)) && ok;
    tc::tc_fence_after();
    if (__syncthreads_or(!ok)) {
        if (nblk > 0) tc::mbar_wait(tc::saddr(bars + lu % WG_NS), (uint32_t)((lu / WG_NS) & 1));
        tc::tc_fence_before();
        __syncthreads();
        if (warp == 0) tc::tmem_dealloc(taddr, ncols);
        if (tid == 0 && err) atomicExch(err, 1);
        return;
    }
    // TMEM lane = row (warp w holds rows 32w .. 32w+31)
    const int tl = tid / CP, ci = tid - tl * CP, t = t0 + tl;
    float *out = nullptr;
    if (tl < TG && t < taps && ci < cin)
        out = part + (int64_t)s * pstride + ((int64_t)t * cin + ci) * cout;
    else if (bias && tid == ones)
        out = part + (int64_t)s * pstride + (int64_t)taps * cin * cout;
    for (int c0 = 0; c0 < NP; c0 += 16) {
        float r[16];
        tc::tmem_ld16(taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, r);
        if (!out) continue;
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (c0 + j < cout) out[c0 + j] = nblk > 0 ? r[j] : 0.f;
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(taddr, ncols);
}

static inline int pad16(int c) { return (c + 15) & ~15; }
static inline int nblk_tc(int64_t n, int b) { return (int)((n + b - 1) / b); }
static size_t tc_smem(int KP, int NP) { return TC_NS * ((size_t)TC_BM * KP * 2 + (size_t)NP * KP * 2) + 8 * TC_NS + 16; }

bool net_conv_tc_fits(int cin, int cout) { return cin <= TC_CMAX && cout <= TC_CMAX; }

static size_t tc_wgrad_smem(int NP) {
    return WG_NS * ((size_t)TC_BM * TC_BM * 2 + (size_t)NP * TC_BM * 2) + 8 * WG_NS + 16;
}

bool net_wgrad_tc_fits(int cin, int cout) { return cin < TC_BM - 8 && cout <= TC_CMAX; }

void net_conv_wgrad_tc(const bf16 *in, int cin, const bf16 *gout, int cout, int taps, int ny, int nx, int nz, int S,
                       int64_t vchunk, float *part, int64_t pstride, int *err, cudaStream_t s) {
    const int NP = pad16(cout), CP = (cin + 7) & ~7;
    const int TG = std::min(taps, (TC_BM - 1) / CP);   // taps per CTA, a row left for the ones
    ++g_launches;
    k_conv_wgrad_tc<<<dim3((taps + TG - 1) / TG, S), TC_BM, tc_wgrad_smem(NP), s>>>(in, cin, gout, cout, NP, taps, TG, ny,
                                                                                    nx, nz, vchunk, part, pstride, err);
}

void net_tc_init_attributes() {
    cudaFuncSetAttribute(k_conv_wgrad_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc_wgrad_smem(TC_CMAX));
    const int mx = (int)tc_smem(TC_CMAX, TC_CMAX);
    cudaFuncSetAttribute(k_conv_tc<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
    cudaFuncSetAttribute(k_conv_tc<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
    cudaFuncSetAttribute(k_conv_tc<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
}

void net_weight_images(const bf16 *w, const NetImages &im, bool flip, bf16 *out, cudaStream_t s) {
    ++g_launches;
    k_wimages<<<nblk_tc(im.at[im.n], 256), 256, 0, s>>>(w, im, flip ? 1 : 0, out);
}

void net_conv_fwd_tc(const bf16 *in, int cin, const bf16 *wimg, const float *b, int cout, int taps, int ny, int nx,
                     int nz, bool relu_bf16_out, void *out, int *err, cudaStream_t s) {
    const int64_t V = (int64_t)ny * nx * nz;
    const int KP = pad16(cin), NP = pad16(cout);
    ++g_launches;
    if (relu_bf16_out)
        k_conv_tc<0><<<nblk_tc(V, TC_BM), TC_BM, tc_smem(KP, NP), s>>>(in, cin, wimg, KP, NP, b, cout, taps, ny, nx, nz,
                                                                       out, nullptr, 0, err);
    else
        k_conv_tc<1><<<nblk_tc(V, TC_BM), TC_BM, tc_smem(KP, NP), s>>>(in, cin, wimg, KP, NP, b, cout, taps, ny, nx, nz,
                                                                       out, nullptr, 0, err);
}

// data gradient: gin (=/+=) mask(conv(gout, flipped w)), wimg the flipped images, i.e. K =
// cout input channels and N = cin output channels
void net_conv_bwd_data_tc(const bf16 *gout, int cout, const bf16 *wimg, int cin, int taps, int ny, int nx, int nz,
                          const bf16 *mask, float *gin, bool accumulate, int *err, cudaStream_t s) {
    const int64_t V = (int64_t)ny * nx * nz;
    const int KP = pad16(cout), NP = pad16(cin);
    ++g_launches;
    k_conv_tc<2><<<nblk_tc(V, TC_BM), TC_BM, tc_smem(KP, NP), s>>>(gout, cout, wimg, KP, NP, nullptr, cin, taps, ny, nx,
                                                                   nz, gin, mask, accumulate ? 1 : 0, err);
}

}  // namespace sgld
