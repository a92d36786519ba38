// One training step of the learned proposal's network on the tcgen05 tensor
// cores, in two launches:
//
//   k_lp_step_tc   forward, loss, backward and the weight gradients' partial
//                  sums of a block of rows per CTA
//   k_lp_update    the partial sums added in a fixed order, the bias
//                  gradients, the loss and (training) Adam and the BF16 copies
//
// What bounds it: latency.  A step of 4096 rows is 0.5 GFLOP and 6 MB of
// traffic, but a chain of six dependent matrix products per row; as separate
// launches (three forward GEMMs, the loss in one block, five backward GEMMs
// with their sums, three column sums, Adam, conversion) it took 441 us on a
// GB300, most of it launches that filled a fraction of the GPU; in these two
// it takes 34 us.  Here a row's
// activations and gradients never leave shared memory: every operand is
// stored once, as 8 x 8 core matrices, and read by the tensor cores as K-major
// in the layer products and as MN-major (the same bytes, transposed) where
// rows are the contraction, in dZ = dY W and in the weight gradients.
//
// The split of the batch (k_per rows a CTA, at most kLpSteps CTAs), the order
// of every sum and the rounding of every intermediate are those of separate
// GEMMs with the weight gradients split along the batch.
#include <cuda_bf16.h>

#include "esp_learned.h"
#include "esp_lp_tc.cuh"
#include "esp_tc.cuh"

namespace esp {

namespace {

constexpr int kStepThreads = 256;
constexpr int kStepRows = 128;       // rows in flight per CTA (tensor-memory lanes)
constexpr uint32_t kColsD = 0, kColsW2 = 128, kColsW3 = 256, kColsW1 = 384;   // tensor-memory columns

struct alignas(128) LpStepSmem {
    __nv_bfloat16 w1[kMlpHid * kMlpInPad], w2[kMlpHid * kMlpHid], w3[kMlpOutPad * kMlpHid];
    __nv_bfloat16 x[kStepRows * kMlpInPad], h1[kStepRows * kMlpHid], h2[kStepRows * kMlpHid];
    __nv_bfloat16 dz2[kStepRows * kMlpHid], dz1[kStepRows * kMlpHid];
    __nv_bfloat16 d_o[kStepRows * kMlpOutPad];
    __nv_bfloat16 past_d_o[kStepRows * kMlpOutPad];   // read (and ignored) as rows 32..127 of dO^T
    float b1[kMlpHid], b2[kMlpHid], b3[kMlpOutPad];
    unsigned long long bar;
    uint32_t tmem;
    int stop;
};

// Descriptor of a matrix of C columns (kmajor_offset) whose columns are the
// contraction, from column 16 kk, or whose rows are, from row 16 kk.
__device__ __forceinline__ uint64_t desc_k(uint32_t base, int C, int kk)
{
    return smem_desc(base + 256u * kk, 128u, (uint32_t)(C / 8) * 128u);
}
__device__ __forceinline__ uint64_t desc_mn(uint32_t base, int C, int kk)
{
    const uint32_t group = (uint32_t)(C / 8) * 128u;   // 8 rows
    return smem_desc(base + 2u * group * kk, group, 128u);
}
constexpr uint32_t kIdescAT = 1u << 15, kIdescBT = 1u << 16;   // A, B MN-major

__global__ void __launch_bounds__(kStepThreads, 1) k_lp_step_tc(const LpStepArgs a)
{
    extern __shared__ __align__(128) unsigned char smem_step[];
    LpStepSmem &s = *reinterpret_cast<LpStepSmem *>(smem_step);
    const int t = threadIdx.x, row = t & (kStepRows - 1), half = t >> 7;   // columns 64 half ..
    const int z = blockIdx.x, kb = z * a.k_per, ke = min(a.rows, kb + a.k_per);

    auto stage = [&](const __nv_bfloat16 *src, __nv_bfloat16 *dst, int rows, int C) {
        for (int i = t; i < rows * (C / 8); i += kStepThreads) {
            const int r = i / (C / 8), c = (i % (C / 8)) * 8;
            *reinterpret_cast<uint4 *>(reinterpret_cast<unsigned char *>(dst) + kmajor_offset(r, c, C)) =
                __ldg(reinterpret_cast<const uint4 *>(src + (size_t)r * C + c));
        }
    };
    stage(a.w.w1, s.w1, kMlpHid, kMlpInPad);
    stage(a.w.w2, s.w2, kMlpHid, kMlpHid);
    stage(a.w.w3, s.w3, kMlpOutPad, kMlpHid);
    for (int i = t; i < kMlpHid; i += kStepThreads) { s.b1[i] = __ldg(a.w.b1 + i); s.b2[i] = __ldg(a.w.b2 + i); }
    if (t < kMlpOutPad) s.b3[t] = __ldg(a.w.b3 + t);
    for (int i = t; i < kStepRows * kMlpOutPad / 8; i += kStepThreads)
        reinterpret_cast<uint4 *>(s.past_d_o)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (t == 0) {
        mbar_init(smem_u32(&s.bar), 1);
        s.stop = 0;
    }
    if (t < 32) {
        tmem_alloc(smem_u32(&s.tmem), 512);
        tmem_relinquish();
    }
    const uint32_t x = smem_u32(s.x), h1 = smem_u32(s.h1), h2 = smem_u32(s.h2), d_o = smem_u32(s.d_o);
    const uint32_t dz2 = smem_u32(s.dz2), dz1 = smem_u32(s.dz1), bar = smem_u32(&s.bar);
    const uint32_t w1 = smem_u32(s.w1), w2 = smem_u32(s.w2), w3 = smem_u32(s.w3);

    // Operand writes of every thread -> tensor cores, the issuing thread's
    // MMAs, and their completion seen by every thread.  false (for the whole
    // CTA) when the wait gave up; `pending` then says whether no thread saw
    // the MMAs complete.
    uint32_t phase = 0;
    bool pending = false;
    auto run = [&](auto &&issue) -> bool {
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (t == 0) {
            issue();
            tc_commit(bar);
        }
        const bool seen = mbar_wait(bar, phase, kTcWaitLimit);
        if (__syncthreads_or(!seen)) {
            pending = __syncthreads_or(seen) == 0;
            if (!pending) phase ^= 1u;
            return false;
        }
        phase ^= 1u;
        tc_fence_after();
        return true;
    };
    auto put8 = [&](__nv_bfloat16 *dst, int C, int c, const uint4 &v) {
        *reinterpret_cast<uint4 *>(reinterpret_cast<unsigned char *>(dst) + kmajor_offset(row, c, C)) = v;
    };
    auto pack8 = [&](const float *v) -> uint4 {
        return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
    };

    bool ok = true;
    for (int r0 = kb; r0 < ke && ok; r0 += kStepRows) {
        const int nv = min(kStepRows, ke - r0), gr = r0 + row;
        const bool live = row < nv;
        const bool first = r0 == kb;
        const int ksteps = (nv + 15) / 16;
        // ---- rows: features (and, below, targets) of the batch -------------
        long long src = gr;
        if (live && a.n_all > 0) {
            // random row of the training set, with replacement
            const Philox4 p = philox4x32_10((uint32_t)gr, a.s_lo, a.s_hi, 0x7EA1u, a.k0, a.k1);
            src = (long long)__umul64hi(((unsigned long long)p.x << 32) | p.y, (unsigned long long)a.n_all);
        }
        if (half == 0) {
            uint4 v0 = make_uint4(0u, 0u, 0u, 0u), v1 = v0;
            if (live) {
                const uint4 *xs = reinterpret_cast<const uint4 *>(a.x + (size_t)src * kMlpInPad);
                v0 = __ldg(xs); v1 = __ldg(xs + 1);
            }
            put8(s.x, kMlpInPad, 0, v0);
            put8(s.x, kMlpInPad, 8, v1);
        }
        float4 tv = make_float4(0.f, 0.f, 1.f, 1.f);
        if (half == 0 && live) tv = __ldg(reinterpret_cast<const float4 *>(a.t) + src);
        // the tensor memory is allocated (and its address known) after the
        // barrier in the first product
        uint32_t lane = 0;
        auto D = [&]() { return s.tmem + kColsD; };
        // H = relu(D + b)
        auto hidden = [&](__nv_bfloat16 *h, const float *bias) {
#pragma unroll 1
            for (int c0 = 64 * half; c0 < 64 * half + 64; c0 += 16) {
                float v[16];
                tmem_ld16(lane + (uint32_t)c0, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = fmaxf(v[j] + bias[c0 + j], 0.f);
                put8(h, kMlpHid, c0, pack8(v));
                put8(h, kMlpHid, c0 + 8, pack8(v + 8));
            }
        };
        // dZ = D where H > 0, to shared memory and (for the bias gradient) rows in global memory
        auto masked = [&](__nv_bfloat16 *dz, const __nv_bfloat16 *h, __nv_bfloat16 *out) {
#pragma unroll 1
            for (int c0 = 64 * half; c0 < 64 * half + 64; c0 += 8) {
                if ((c0 & 8) == 0) {
                    float v[16];
                    tmem_ld16(lane + (uint32_t)c0, v);
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const uint4 hv = *reinterpret_cast<const uint4 *>(reinterpret_cast<const unsigned char *>(h) +
                                                                          kmajor_offset(row, c0 + 8 * q, kMlpHid));
                        const __nv_bfloat16 *hb = reinterpret_cast<const __nv_bfloat16 *>(&hv);
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (!(__bfloat162float(hb[j]) > 0.f)) v[8 * q + j] = 0.f;
                        const uint4 p = pack8(v + 8 * q);
                        put8(dz, kMlpHid, c0 + 8 * q, p);
                        if (live) *reinterpret_cast<uint4 *>(out + (size_t)gr * kMlpHid + c0 + 8 * q) = p;
                    }
                }
            }
        };
        // ---- forward: H1 = relu(X W1^T + b1), H2 = relu(H1 W2^T + b2), O = H2 W3^T + b3
        if (!(ok = run([&]() { tc_mma(D(), desc_k(x, kMlpInPad, 0), desc_k(w1, kMlpInPad, 0), idesc_bf16_f32(128, kMlpHid), 0u); })))
            break;
        lane = s.tmem + ((uint32_t)(row & ~31) << 16);
        hidden(s.h1, s.b1);
        if (!(ok = run([&]() {
                  for (int kk = 0; kk < kMlpHid / 16; ++kk)
                      tc_mma(D(), desc_k(h1, kMlpHid, kk), desc_k(w2, kMlpHid, kk), idesc_bf16_f32(128, kMlpHid), kk > 0);
              })))
            break;
        hidden(s.h2, s.b2);
        if (!(ok = run([&]() {
                  for (int kk = 0; kk < kMlpHid / 16; ++kk)
                      tc_mma(D(), desc_k(h2, kMlpHid, kk), desc_k(w3, kMlpHid, kk), idesc_bf16_f32(128, kMlpOutPad), kk > 0);
              })))
            break;
        // ---- loss -log q of the row and its gradient dO ---------------------
        if (half == 0) {
            float o[kMlpOutPad], d[kMlpOutPad];
            tmem_ld16(lane, o);
            tmem_ld16(lane + 16u, o + 16);
#pragma unroll
            for (int k = 0; k < kMlpOutPad; ++k) {
                o[k] += s.b3[k];
                d[k] = 0.f;
            }
            if (live) {
                float lq = 0.f;
                if (gr < a.n_real) {
                    VmfMix mix;
                    vmf_params(o, tv.w, mix);
                    lq = vmf_logpdf_grad(mix, tv.x, tv.y, tv.z, d);
                }
                a.lq[gr] = lq;
            }
#pragma unroll
            for (int k = 0; k < kMlpOut; ++k) d[k] *= -a.scale;
#pragma unroll
            for (int c = 0; c < kMlpOutPad; c += 8) {
                const uint4 p = pack8(d + c);
                put8(s.d_o, kMlpOutPad, c, p);
                if (live) *reinterpret_cast<uint4 *>(a.d_o + (size_t)gr * kMlpOutPad + c) = p;
            }
        }
        // ---- dZ2 = (dO W3) . [H2 > 0]; dW3 += dO^T H2 -----------------------
        if (!(ok = run([&]() {
                  for (int kk = 0; kk < kMlpOutPad / 16; ++kk)
                      tc_mma(D(), desc_k(d_o, kMlpOutPad, kk), desc_mn(w3, kMlpHid, kk),
                             idesc_bf16_f32(128, kMlpHid) | kIdescBT, kk > 0);
                  for (int kk = 0; kk < ksteps; ++kk)
                      tc_mma(s.tmem + kColsW3, desc_mn(d_o, kMlpOutPad, kk), desc_mn(h2, kMlpHid, kk),
                             idesc_bf16_f32(128, kMlpHid) | kIdescAT | kIdescBT, !first || kk > 0);
              })))
            break;
        masked(s.dz2, s.h2, a.dz2);
        // ---- dZ1 = (dZ2 W2) . [H1 > 0]; dW2 += dZ2^T H1 ---------------------
        if (!(ok = run([&]() {
                  for (int kk = 0; kk < kMlpHid / 16; ++kk)
                      tc_mma(D(), desc_k(dz2, kMlpHid, kk), desc_mn(w2, kMlpHid, kk),
                             idesc_bf16_f32(128, kMlpHid) | kIdescBT, kk > 0);
                  for (int kk = 0; kk < ksteps; ++kk)
                      tc_mma(s.tmem + kColsW2, desc_mn(dz2, kMlpHid, kk), desc_mn(h1, kMlpHid, kk),
                             idesc_bf16_f32(128, kMlpHid) | kIdescAT | kIdescBT, !first || kk > 0);
              })))
            break;
        masked(s.dz1, s.h1, a.dz1);
        // ---- dW1 += dZ1^T X --------------------------------------------------
        if (!(ok = run([&]() {
                  for (int kk = 0; kk < ksteps; ++kk)
                      tc_mma(s.tmem + kColsW1, desc_mn(dz1, kMlpHid, kk), desc_mn(x, kMlpInPad, kk),
                             idesc_bf16_f32(128, kMlpInPad) | kIdescAT | kIdescBT, !first || kk > 0);
              })))
            break;
    }
    if (ok && kb < ke) {
        // ---- this CTA's partial weight gradients ------------------------------
        const uint32_t lane = s.tmem + ((uint32_t)(row & ~31) << 16);
        float *part = a.part + (size_t)z * kLpStepPart;
        auto store = [&](uint32_t cols, float *dst, bool take) {
            float v[16];
            tmem_ld16(lane + cols, v);
            if (take)
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                    *reinterpret_cast<float4 *>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        };
        for (int c0 = 64 * half; c0 < 64 * half + 64; c0 += 16) {
            store(kColsW2 + (uint32_t)c0, part + kLpPartW2 + row * kMlpHid + c0, true);
            if (row < 32) store(kColsW3 + (uint32_t)c0, part + kLpPartW3 + row * kMlpHid + c0, true);
        }
        if (half == 0) store(kColsW1, part + kLpPartW1 + row * kMlpInPad, true);
    }
    if (!ok && t == 0) atomicExch(a.err, 1);
    // a give-up with MMAs possibly still running: wait for them once more
    // (bounded) before the tensor memory is freed
    if (pending && t == 0) mbar_wait(bar, phase, kTcWaitLimit);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (t < 32) tmem_dealloc(s.tmem, 512);
}

// Adam (Kingma & Ba, 2015) with bias correction; every rounding spelled out,
// the same as k_adam (esp_learned.cu) takes
__device__ __forceinline__ float adam(const LpUpdateArgs &a, int i, float gi)
{
    const float mi = fmaf(1.f - a.b1, gi, __fmul_rn(a.b1, a.m[i]));
    const float vi = fmaf(__fmul_rn(1.f - a.b2, gi), gi, __fmul_rn(a.b2, a.v[i]));
    a.m[i] = mi; a.v[i] = vi;
    const float p = __fsub_rn(a.p[i], __fmul_rn(a.lr, mi / a.c1) / __fadd_rn(sqrtf(vi / a.c2), a.eps));
    a.p[i] = p;
    return p;
}

constexpr int kUpThreads = 256;
constexpr int kUpWeights = kMlpHid * kMlpInPad + kMlpHid * kMlpHid + kMlpOutPad * kMlpHid;
constexpr int kUpWeightBlocks = kUpWeights / kUpThreads;
constexpr int kUpBiasBlocks = (kMlpHid + kMlpHid + kMlpOutPad) / 32;
constexpr int kUpTile = 256;   // rows of a column-sum tile
static_assert(kUpWeights % kUpThreads == 0 && kLpPartW1 % 4 == 0, "block roles");

// Blocks [0, kUpWeightBlocks): a weight per thread, its partial sums in split
// order.  Then 32 columns of a bias gradient each: thread (x, y) adds rows y,
// y + 8, ... of column x in order, the eight sums in order.  Last: the loss.
__global__ void __launch_bounds__(kUpThreads) k_lp_update(const LpUpdateArgs a)
{
    __shared__ __align__(16) unsigned char smem[kUpTile * 64];
    const int t = threadIdx.x;
    if (blockIdx.x < kUpWeightBlocks) {
        const int i = blockIdx.x * kUpThreads + t;   // W2, W3, W1 as in the partials
        float g = 0.f;
#pragma unroll 16
        for (int z = 0; z < a.splits; ++z) g += __ldg(a.part + (size_t)z * kLpStepPart + i);
        int pi, wi;
        __nv_bfloat16 *w;
        if (i < kLpPartW3) { wi = i; pi = kPadW2 + wi; w = a.w2; }
        else if (i < kLpPartW1) { wi = i - kLpPartW3; pi = kPadW3 + wi; w = a.w3; }
        else { wi = i - kLpPartW1; pi = kPadW1 + wi; w = a.w1; }
        a.g[pi] = g;
        if (a.train) w[wi] = __float2bfloat16_rn(adam(a, pi, g));
    } else if (blockIdx.x < kUpWeightBlocks + kUpBiasBlocks) {
        const int b = blockIdx.x - kUpWeightBlocks;   // 0..3 dZ1, 4..7 dZ2, 8 dO
        const __nv_bfloat16 *src = b < 4 ? a.dz1 : (b < 8 ? a.dz2 : a.d_o);
        const int ld = b < 8 ? kMlpHid : kMlpOutPad, c0 = b < 8 ? 32 * (b & 3) : 0;
        const int pi = (b < 4 ? kPadB1 : (b < 8 ? kPadB2 : kPadB3)) + c0;
        const int cx = t & 31, cy = t >> 5;
        float acc = 0.f;
        // tiles of kUpTile rows x 64 bytes through shared memory, the next
        // one in flight while this one is added
        uint4 nxt[4];
        auto fetch = [&](int r0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int k = t + q * kUpThreads, r = r0 + (k >> 2);
                nxt[q] = make_uint4(0u, 0u, 0u, 0u);
                if (r < a.rows) nxt[q] = __ldg(reinterpret_cast<const uint4 *>(src + (size_t)r * ld + c0) + (k & 3));
            }
        };
        fetch(0);
        for (int r0 = 0; r0 < a.rows; r0 += kUpTile) {
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 4; ++q) reinterpret_cast<uint4 *>(smem)[t + q * kUpThreads] = nxt[q];
            __syncthreads();
            if (r0 + kUpTile < a.rows) fetch(r0 + kUpTile);
            const __nv_bfloat16 *tile = reinterpret_cast<const __nv_bfloat16 *>(smem) + cx;
            const int n = min(kUpTile, a.rows - r0);
#pragma unroll 8
            for (int r = cy; r < n; r += 8) acc += __bfloat162float(tile[r * 32]);
        }
        __syncthreads();
        float *sum = reinterpret_cast<float *>(smem);
        sum[cy * 33 + cx] = acc;
        __syncthreads();
        if (cy == 0) {
            float v = 0.f;
            for (int k = 0; k < 8; ++k) v += sum[k * 33 + cx];
            a.g[pi + cx] = v;
            if (a.train) adam(a, pi + cx, v);
        }
    } else {
        double *sum = reinterpret_cast<double *>(smem);
        double acc = 0.0;
        for (int i = t; i < a.n_real; i += kUpThreads) acc += -(double)__ldg(a.lq + i);
        sum[t] = acc;
        __syncthreads();
        for (int w = kUpThreads / 2; w > 0; w >>= 1) {
            if (t < w) sum[t] += sum[t + w];
            __syncthreads();
        }
        if (t == 0) *a.loss = sum[0] * (double)a.scale;
    }
}

}  // namespace

cudaError_t lp_step_configure()
{
    static_assert(sizeof(LpStepSmem) <= 227 * 1024, "shared memory of a training step");
    return cudaFuncSetAttribute(k_lp_step_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LpStepSmem));
}

// Rows of a CTA: the batch in at most kLpSteps parts of whole chunks of 64.
int lp_step_rows(int rows)
{
    int n = (rows + 63) / 64;
    if (n > kLpSteps) n = kLpSteps;
    const int per = (rows + n - 1) / n;
    return (per + 63) / 64 * 64;
}

cudaError_t launch_lp_step(const LpStepArgs &a, const LpUpdateArgs &u0, cudaStream_t st)
{
    if (a.rows <= 0 || (a.rows & 7) || a.k_per <= 0 || (a.k_per & 63)) return cudaErrorInvalidValue;
    LpUpdateArgs u = u0;
    u.splits = (a.rows + a.k_per - 1) / a.k_per;
    if (u.splits > kLpSteps) return cudaErrorInvalidValue;
    k_lp_step_tc<<<u.splits, kStepThreads, sizeof(LpStepSmem), st>>>(a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_lp_update<<<kUpWeightBlocks + kUpBiasBlocks + 1, kUpThreads, 0, st>>>(u);
    return cudaGetLastError();
}

}  // namespace esp
