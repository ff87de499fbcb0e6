// radiance_cache.cu — the learned radiance cache: a small MLP trained
// online on the path tracer's own radiance samples, on the tensor cores.
//
// Network: 10 inputs (position normalised to the scene bounds, incoming
// direction, normal, roughness) → 12-band frequency encoding (sin and cos of
// 2^b·π·x, b = 0..11, for every input: 240 features) + the 10 raw inputs + a
// constant 1 + 5 zeros = 256 features → 5 hidden layers of 64 (ReLU) → 3
// outputs (RGB radiance; padded to 16 for the MMA).  No biases (the constant
// feature gives layer 1 one).  33,792 weights.
//
// Precision: forward (inference and training) in FP16 with FP32 accumulation
// in TMEM; backward in BF16 (gradients need BF16's range) with FP32
// accumulation; FP32 master weights, FP32 Adam.
//
// Every GEMM is a tcgen05.mma with M = 128 rows (a tile of 128 samples, two
// threads per sample, a group of 8 warps per tile in flight) and operands in
// shared memory (tc_mma.cuh):
//   rc_forward      X·W1ᵀ → ReLU → ·W2ᵀ … → ·W6ᵀ, activations kept in shared
//                   memory between layers, three tiles in flight per CTA;
//                   training also stores H1..H5 and the relative-L2 loss
//                   gradient dZ6 and goes on with dZ6·W6 ⊙ [H5>0] = dZ5, …
//                   down to dZ1 (BF16).
//   rc_wgrad        dWlᵀ = Σ_tiles H(l-1)ᵀ·dZl: both operands MN-major
//                   (each sample's features are stored as they come, 16
//                   bytes at a time), accumulated across sample tiles in
//                   TMEM, then added to the FP32 gradient.
//   rc_adam         Adam on the FP32 master weights; rewrites the FP16
//                   forward and BF16 backward operand copies in the K-major
//                   layout so kernels copy them to shared memory verbatim.
// All mbarrier waits are bounded (tc::mbar_wait); a timeout sets a status
// bit, the CTA waits once more for its MMAs, frees its TMEM and returns.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "rc_kernels.h"
#include "tc_mma.cuh"

namespace orn {
namespace rc {

__device__ __forceinline__ uint16_t f2h(float x) { return __half_as_ushort(__float2half_rn(x)); }
__device__ __forceinline__ uint16_t f2b(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }

// The encoding of one sample's 10 inputs, produced 8 features at a time:
// emit8(f0, v) receives features f0..f0+7.  Input j gives features
// 24j + 2b (sin 2^b·π·x) and 24j + 2b + 1 (cos), b = 0..11, by angle
// doubling from one sincospi: sin 2a = 2 sin a cos a, cos 2a = (cos a - sin a)
// (cos a + sin a); the absolute error after 11 doublings stays below 2e-4,
// under the FP16 rounding of the features.  Features 240..249 are the raw
// inputs, 250 is 1 (the bias of layer 1), 251..255 are 0.
// PART q: features 64 q..64 q + 63 only (an input may have features in two
// parts); emit8 gets 8 features at a time.
template <int PART, class F>
__device__ __forceinline__ void encode_part(const float* in, F&& emit8) {
    constexpr int kLo = 64 * PART, kHi = kLo + 64 < kEncoded ? kLo + 64 : kEncoded;
    float g[8];
#pragma unroll
    for (int j = kLo / 24; j < (kHi + 23) / 24; ++j) {
        float s, c;
        sincospif(in[j], &s, &c);
#pragma unroll
        for (int b = 0; b < kBands; ++b) {
            g[(2 * b) & 7] = s;
            g[(2 * b + 1) & 7] = c;
            const int f0 = 24 * j + 2 * b - 6;
            if ((b & 3) == 3 && f0 >= kLo && f0 < kHi) emit8(f0, g);
            const float s2 = 2.0f * s * c, c2 = (c - s) * (c + s);
            s = s2;
            c = c2;
        }
    }
    if constexpr (PART == 3) {
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] = in[j];
        emit8(kEncoded, g);
        g[0] = in[8];
        g[1] = in[9];
        g[2] = 1.0f;
#pragma unroll
        for (int j = 3; j < 8; ++j) g[j] = 0.0f;
        emit8(kEncoded + 8, g);
    }
}
// The part of features 128 HALF..128 HALF + 127 that belongs to the sample's
// thread `sub` (0 or 1).
template <int HALF, class F>
__device__ __forceinline__ void encode(uint32_t sub, const float* in, F&& emit8) {
    if (sub == 0) encode_part<2 * HALF>(in, emit8);
    else encode_part<2 * HALF + 1>(in, emit8);
}

// 8 values rounded to FP16 / BF16, two per instruction.
__device__ __forceinline__ uint32_t h2(float a, float b) {
    const __half2 r = __floats2half2_rn(a, b);
    return *(const uint32_t*)&r;
}
__device__ __forceinline__ uint32_t b2(float a, float b) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(a, b);
    return *(const uint32_t*)&r;
}
__device__ __forceinline__ uint4 half8(const float* v) {
    return make_uint4(h2(v[0], v[1]), h2(v[2], v[3]), h2(v[4], v[5]), h2(v[6], v[7]));
}
__device__ __forceinline__ uint4 bf8(const float* v) {
    return make_uint4(b2(v[0], v[1]), b2(v[2], v[3]), b2(v[4], v[5]), b2(v[6], v[7]));
}
__device__ __forceinline__ uint32_t half_to_bf(uint32_t h) {
    const float2 f = __half22float2(*(const __half2*)&h);
    return b2(f.x, f.y);
}

// Offset (in elements) of layer l's backward operand inside the BF16 copy:
// layers 6, 5, 4, 3, 2 in that order (the order in which training goes back).
__host__ __device__ constexpr uint32_t bwd_offset(int l) {
    uint32_t o = 0;
    for (int i = kLayers - 1; i > l; --i) o += rc_layer_in(i) * rc_layer_out(i);
    return o;
}

// The 256 threads of a tile's group, two per sample (row): the first 128 and
// the last 128 split a row's features and columns.
constexpr uint32_t kGroup = 256;

// A group's threads meet at named barrier `id` (1 + the group; barrier 0 is
// __syncthreads'); the second form also returns whether `v` holds for all of
// them.
__device__ __forceinline__ void group_bar(uint32_t id) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kGroup) : "memory");
}
__device__ __forceinline__ bool group_bar_and(uint32_t id, bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "bar.red.and.pred p, %2, %3, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"(v ? 1u : 0u), "r"(id), "n"(kGroup)
        : "memory");
    return r != 0;
}

// A tile group's synchronisation state for its MMA rounds: its mbarrier,
// the phase it waits for next, whether every wait so far completed, and its
// named barrier.
struct Sync {
    uint64_t* mbar;
    uint32_t phase;
    bool ok;
    uint32_t bar;
};

// Issues D(TMEM) = A · Bᵀ (+ D when `accumulate`), A: 128 x K at `a`, B:
// N x K at `b` (columns of an operand of `b_cols` columns), both K-major (or
// both MN-major when `mn_major`): makes the group's shared-memory writes
// visible to the tensor core, then the group's first thread issues the K/16
// MMAs and commits them to the group's mbarrier.  Every thread of the group
// calls.
__device__ __forceinline__ void gemm_issue(Sync& s, uint32_t tmem, const unsigned char* a, const unsigned char* b,
                                           uint32_t K, uint32_t b_cols, uint32_t N, bool bf16, bool accumulate,
                                           bool mn_major = false) {
    tc::fence_async_smem();
    tc::fence_before_sync();
    group_bar(s.bar);
    tc::fence_after_sync();
    if ((threadIdx.x & (kGroup - 1)) == 0 && s.ok) {
        const uint32_t idesc = tc::idesc_f16(128, N, bf16, mn_major);
        const uint32_t sbo = (K / 8u) * 128u, b_sbo = (b_cols / 8u) * 128u;
        for (uint32_t ks = 0; ks < K / 16u; ++ks) {
            const uint64_t ad = tc::smem_desc(tc::smem_addr(a) + ks * 256u, 128u, sbo);
            const uint64_t bd = tc::smem_desc(tc::smem_addr(b) + ks * 256u, 128u, b_sbo);
            tc::mma_f16(tmem, ad, bd, idesc, accumulate || ks > 0);
        }
        tc::mma_commit(s.mbar);
    }
}

// Waits (bounded) for the group's issued MMAs; all its threads agree on
// s.ok afterwards.
__device__ __forceinline__ void gemm_wait(Sync& s) {
    const bool ok = s.ok && tc::mbar_wait(s.mbar, s.phase, 2000000000ull);
    s.ok = group_bar_and(s.bar, ok);
    // on failure s.phase stays the phase of the round still in flight
    if (s.ok) s.phase ^= 1u;
    tc::fence_after_sync();
}

__device__ __forceinline__ void gemm_round(Sync& s, uint32_t tmem, const unsigned char* a, const unsigned char* b,
                                           uint32_t K, uint32_t b_cols, uint32_t N, bool bf16, bool accumulate) {
    gemm_issue(s, tmem, a, b, K, b_cols, N, bf16, accumulate);
    gemm_wait(s);
}

// `N` FP32 columns of this thread's TMEM lane (its row of the tile; a warp
// reads the 32 lanes of its index modulo 4).
template <uint32_t N>
__device__ __forceinline__ void read_row(uint32_t tmem, float* v) {
    const uint32_t lane_base = (32u * ((threadIdx.x >> 5) & 3u)) << 16;
#pragma unroll
    for (uint32_t c = 0; c < N; c += 16) tc::tmem_ld16(tmem + lane_base + c, v + c);
    tc::tmem_ld_wait();
}

// Allocates `ncols` TMEM columns (warp 0) and initialises `nbar` mbarriers.
__device__ __forceinline__ uint32_t cta_setup(uint32_t* tmem_slot, uint64_t* mbar, uint32_t nbar, uint32_t ncols) {
    if (threadIdx.x < 32) {
        tc::tmem_alloc(tmem_slot, ncols);
        tc::tmem_relinquish();
    }
    if (threadIdx.x == 0)
        for (uint32_t i = 0; i < nbar; ++i) tc::mbar_init(mbar + i, 1);
    tc::fence_async_smem();   // (weights that any thread of the CTA has written)
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    return *tmem_slot;
}

// After a timed-out wait: give the group's MMAs in flight one more bounded
// wait, record the failure, then free the CTA's TMEM columns (on every
// path; `tmem_base` is the allocation's first column).  Freeing while an
// MMA might still write them is only reached when both waits (3 s) ran
// out; a CTA that exited holding its columns would instead leave them
// allocated for every later CTA on that SM, whose tcgen05.alloc could then
// wait forever, so the columns are always returned.
__device__ __forceinline__ void cta_teardown(Sync& s, uint32_t tmem_base, uint32_t ncols, uint32_t* status) {
    if (!s.ok) {
        tc::mbar_wait(s.mbar, s.phase, 1000000000ull);
        if ((threadIdx.x & (kGroup - 1)) == 0) atomicOr(status, 4u);   // ERR_MMA
    }
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) tc::tmem_dealloc(tmem_base, ncols);
}

// ---- forward (and, in training, back through layers 6..2) ---------------------------
// What bounds it: a tile is a serial chain (encode, MMA, wait, ReLU and
// repack, MMA, ...) on a few warps, so the chip is filled with chains and each
// is kept short.  Three groups per CTA, each with a tile in flight (its own X
// buffer, mbarrier, named barrier and 64 TMEM columns); two threads per sample
// halve a row's encoding and its repacking.  Group g takes tiles blockIdx.x +
// g * gridDim.x, then every 3 * gridDim.x-th, so that a small call spreads over
// the SMs first.
// Shared memory: the six FP16 weight operands (67,584 B), in training the five
// BF16 backward operands (34,816 B), and per group half of X (128 x 128 FP16:
// layer 1 runs in two halves of its inputs, accumulated in TMEM in the order
// of one MMA over all of them).  A layer's activations, later gradients,
// overwrite the start of X: the MMA that read it has completed by then.
// Training goes back through the layers in the same kernel, the ReLU masks
// being a word per layer in the thread that made them.
// Measured (GB300, device time): inference of 100,003 samples 37 us with two
// groups, one thread per sample and a whole X each, 31 us with four groups on
// halves of X, 22 us with three of two threads.  Training forward and backward
// of 16,384 samples 32 us as two kernels, 27 us as one, 21 us with two threads.
constexpr uint32_t kWfBytes = kWeightCount * 2;
constexpr uint32_t kWbBytes = kBackwardWeightCount * 2;
constexpr uint32_t kHalf = kFeatures / 2;
constexpr uint32_t kXBytes = 128 * kHalf * 2;
constexpr uint32_t kCols = kHidden / 2;   // a thread's columns of a row
constexpr uint32_t kTiles = 3;            // groups per CTA, a tile each
constexpr uint32_t kFwdCols = 256;        // a power of two, 64 per group
constexpr uint32_t forward_smem(bool train) { return kWfBytes + (train ? kWbBytes : 0u) + kTiles * kXBytes; }
static_assert(forward_smem(true) <= 227u * 1024u && kTiles * kHidden <= kFwdCols, "forward shared and tensor memory");

template <bool TRAIN>
__global__ void __launch_bounds__(kGroup * kTiles, 1)
rc_forward(RcForward p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar[kTiles];
    __shared__ uint32_t tmem_slot;
    const uint32_t grp = threadIdx.x / kGroup, sub = (threadIdx.x >> 7) & 1u, t = threadIdx.x & 127u;
    const uint32_t col = sub * kCols;   // this thread's first column of row t
    unsigned char* W = smem;
    unsigned char* Wb = smem + kWfBytes;   // (training) the backward operands of layers 6..2
    unsigned char* X = smem + kWfBytes + (TRAIN ? kWbBytes : 0u) + grp * kXBytes;
    const uint32_t n = p.n_dev ? min(*p.n_dev, p.n) : p.n;
    const uint32_t tiles = (n + 127) / 128;
    if (blockIdx.x >= tiles) return;
    for (uint32_t i = threadIdx.x; i < kWfBytes / 16; i += blockDim.x)
        ((uint4*)W)[i] = __ldg((const uint4*)p.weights_f16 + i);
    if (TRAIN)
        for (uint32_t i = threadIdx.x; i < kWbBytes / 16; i += blockDim.x)
            ((uint4*)Wb)[i] = __ldg((const uint4*)p.weights_bf16 + i);
    const uint32_t tmem_base = cta_setup(&tmem_slot, mbar, kTiles, kFwdCols);
    const uint32_t tmem = tmem_base + grp * kHidden;
    Sync s{&mbar[grp], 0u, true, 1u + grp};
    float loss = 0.0f;
    for (uint32_t tile = blockIdx.x + grp * gridDim.x; tile < tiles && s.ok; tile += kTiles * gridDim.x) {
        const uint32_t row = tile * 128 + t;
        const bool valid = row < n;
        float in[kInputs];
        for (int j = 0; j < kInputs; ++j) in[j] = valid ? p.inputs[(size_t)row * kInputs + j] : 0.0f;
        auto stage = [&](int f0, const float* g) {
            *(uint4*)(X + tc::kmajor_offset(t, f0 & (kHalf - 1), kHalf)) = half8(g);
        };
        encode<0>(sub, in, stage);
        gemm_round(s, tmem, X, W, kHalf, kFeatures, kHidden, false, false);
        if (!s.ok) break;
        encode<1>(sub, in, stage);
        float v[kCols];
        uint32_t live[kLayers - 1];   // (training) [H(l) > 0], a bit per column
#pragma unroll
        for (int l = 0; l < kLayers; ++l) {
            const uint32_t N = rc_layer_out(l);
            if (l == 0)   // the second half's columns of W1
                gemm_round(s, tmem, X, W + (kHalf / 8u) * 128u, kHalf, kFeatures, N, false, true);
            else gemm_round(s, tmem, X, W + rc_layer_offset(l) * 2, kHidden, kHidden, N, false, false);
            if (!s.ok) break;
            if (l < kLayers - 1) {
                read_row<kCols>(tmem + col, v);
                if (TRAIN) live[l] = 0u;
#pragma unroll
                for (uint32_t c0 = 0; c0 < kCols; c0 += 8) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        // (2^-25 and below round to an FP16 zero)
                        if (TRAIN && v[c0 + j] > 0x1p-25f) live[l] |= 1u << (c0 + j);
                        v[c0 + j] = fmaxf(v[c0 + j], 0.0f);
                    }
                    const uint4 q = half8(v + c0);
                    *(uint4*)(X + tc::kmajor_offset(t, col + c0, kHidden)) = q;
                    if (TRAIN && valid) *(uint4*)(p.h_out + ((size_t)l * n + row) * kHidden + col + c0) = q;
                }
                continue;
            }
            if (sub != 0) break;   // the output's columns are the first half's
            read_row<kOutPad>(tmem, v);
            if (!TRAIN) {
                if (valid && p.pixel) {
                    // atomic: several sample streams of a pixel may query in
                    // one frame (one add each, so one query gives the same bits
                    // as a plain read-modify-write)
                    const uint32_t px = p.pixel[row];
                    const float4 th = p.throughput[row];
                    float* a = reinterpret_cast<float*>(p.acc + px);
                    atomicAdd(a + 0, th.x * fminf(fmaxf(v[0], 0.0f), 1.0e4f));
                    atomicAdd(a + 1, th.y * fminf(fmaxf(v[1], 0.0f), 1.0e4f));
                    atomicAdd(a + 2, th.z * fminf(fmaxf(v[2], 0.0f), 1.0e4f));
                }
                if (valid && p.outputs)
                    for (int c = 0; c < kOutputs; ++c) p.outputs[(size_t)row * kOutputs + c] = v[c];
            } else {
                // relative L2: per channel (y - r)^2 / (sg(y)^2 + 0.01), whose
                // gradient is 2 (y - r) / (y^2 + 0.01)
                float g[8] = {};
                const bool has = valid && p.targets[(size_t)row * kOutputs] >= 0.0f;
                for (int c = 0; c < kOutputs && has; ++c) {
                    const float y = v[c], r = p.targets[(size_t)row * kOutputs + c];
                    const float den = y * y + 0.01f;
                    loss += (y - r) * (y - r) / den;
                    g[c] = fminf(fmaxf(2.0f * (y - r) / den, -kGradClamp), kGradClamp);
                }
                const uint4 g0 = bf8(g), g1 = make_uint4(0, 0, 0, 0);
                if (valid) {
                    if (p.outputs)
                        for (int c = 0; c < kOutputs; ++c) p.outputs[(size_t)row * kOutputs + c] = v[c];
                    uint4* dst = (uint4*)(p.dz6 + (size_t)row * kOutPad);
                    dst[0] = g0;
                    dst[1] = g1;
                }
                // dZ6 (128 x 16) is the backward pass's first A operand
                *(uint4*)(X + tc::kmajor_offset(t, 0, kOutPad)) = g0;
                *(uint4*)(X + tc::kmajor_offset(t, 8, kOutPad)) = g1;
            }
        }
        if constexpr (TRAIN) {
#pragma unroll
            for (int l = kLayers - 1; l >= 1 && s.ok; --l) {
                // dH(l-1) = dZ(l) · W(l); the B operand is W(l)ᵀ (rows = layer inputs)
                const uint32_t K = rc_layer_out(l);
                gemm_round(s, tmem, X, Wb + bwd_offset(l) * 2, K, K, kHidden, true, false);
                if (!s.ok) break;
                read_row<kCols>(tmem + col, v);
#pragma unroll
                for (uint32_t c0 = 0; c0 < kCols; c0 += 8) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[c0 + j] = (live[l - 1] >> (c0 + j)) & 1u ? v[c0 + j] : 0.0f;
                    const uint4 q = bf8(v + c0);
                    if (l > 1) *(uint4*)(X + tc::kmajor_offset(t, col + c0, kHidden)) = q;
                    if (valid) *(uint4*)(p.dz + ((size_t)(l - 1) * n + row) * kHidden + col + c0) = q;
                }
            }
        }
    }
    if (TRAIN && p.loss) {
        for (int o = 16; o > 0; o >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, o);
        if ((threadIdx.x & 31) == 0) atomicAdd(p.loss, loss);
    }
    cta_teardown(s, tmem_base, kFwdCols, p.status);
}

// ---- weight gradients -------------------------------------------------------------
// One job = (layer l, a block of up to 128 of its inputs).  For every tile of
// 128 samples the CTA stages A = H(l-1)ᵀ (inputs x samples) and B = dZ(l)ᵀ
// (outputs x samples), both MN-major with K = samples — thread t stores
// sample t's inputs and output gradients 8 at a time as 16-byte chunks,
// which keeps the stores free of bank conflicts (a K-major copy would be
// a transpose, 2 bytes per store) — and accumulates D[in x out] in TMEM
// across its tiles; D is then added to the FP32 gradient (gradient of
// W(l)[out][in] = D[in][out]).  One buffer per operand, so that four CTAs fit
// an SM and overlap one another's staging and MMAs, and as many splits as are
// resident: 16,384 samples took 25 us with two buffers, 32 splits and both
// layer-1 jobs encoding all 256 features, 16 us so, and 14 us with two threads
// per sample.
constexpr uint32_t kWgA = 128 * 128 * 2;
constexpr uint32_t kWgB = 64 * 128 * 2;
constexpr uint32_t kWgradSmem = kWgA + kWgB;

__global__ void __launch_bounds__(kGroup, kWgradPerSm)
rc_wgrad(RcWgrad p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    const uint32_t job = blockIdx.x % kWgradJobs, split = blockIdx.x / kWgradJobs;
    const int l = job < 2 ? 0 : (int)job - 1;
    const uint32_t in_base = job < 2 ? job * 128u : 0u;
    const uint32_t in_n = rc_layer_in(l) - in_base < 128u ? rc_layer_in(l) - in_base : 128u;
    const uint32_t out_n = rc_layer_out(l);
    const uint32_t tiles = (p.n + 127) / 128;
    if (split >= tiles) return;
    const uint32_t t = threadIdx.x & 127u, sub = threadIdx.x >> 7;
    unsigned char* A = smem;
    unsigned char* B = smem + kWgA;
    // rows in_n..127 of A (inputs a layer does not have) stay zero
    for (uint32_t c0 = in_n + 8 * sub; c0 < 128; c0 += 16)
        *(uint4*)(A + tc::mnmajor_offset(c0, t, 128)) = make_uint4(0, 0, 0, 0);
    // Stages tile `tile`.  (A sample past the end has zero output gradients;
    // layer 1's features of it are those of zero inputs.)
    auto stage = [&](uint32_t tile) {
        const uint32_t row = tile * 128 + t;
        const bool valid = row < p.n;
        if (l == 0) {
            float in[kInputs];
            for (int j = 0; j < kInputs; ++j) in[j] = valid ? p.inputs[(size_t)row * kInputs + j] : 0.0f;
            auto put = [&](int f0, const float* g) {
                *(uint4*)(A + tc::mnmajor_offset((uint32_t)f0 - in_base, t, 128)) = bf8(g);
            };
            if (in_base == 0) encode<0>(sub, in, put);
            else encode<1>(sub, in, put);
        } else {
            const uint16_t* h = p.h + ((size_t)(l - 1) * p.n + (valid ? row : 0)) * kHidden;
#pragma unroll
            for (uint32_t i = 0; i < (uint32_t)kHidden / 2; i += 8) {
                const uint32_t c0 = sub * (kHidden / 2) + i;
                const uint4 hv = valid ? *(const uint4*)(h + c0) : make_uint4(0, 0, 0, 0);
                *(uint4*)(A + tc::mnmajor_offset(c0, t, 128)) =
                    make_uint4(half_to_bf(hv.x), half_to_bf(hv.y), half_to_bf(hv.z), half_to_bf(hv.w));
            }
        }
        const uint16_t* dz = l == kLayers - 1 ? p.dz6 + (size_t)(valid ? row : 0) * kOutPad
                                              : p.dz + ((size_t)l * p.n + (valid ? row : 0)) * kHidden;
#pragma unroll
        for (uint32_t i = 0; i < (uint32_t)kHidden; i += 16) {
            if (i >= out_n) break;
            const uint32_t c0 = i + 8 * sub;
            const uint4 dv = valid ? *(const uint4*)(dz + c0) : make_uint4(0, 0, 0, 0);
            *(uint4*)(B + tc::mnmajor_offset(c0, t, 128)) = dv;
        }
    };
    const uint32_t tmem = cta_setup(&tmem_slot, &mbar, 1, kTmemCols);
    Sync s{&mbar, 0u, true, 1u};
    bool first = true;
    for (uint32_t tile = split; tile < tiles && s.ok; tile += p.splits) {
        stage(tile);   // (the previous tile's MMAs have completed)
        gemm_issue(s, tmem, A, B, 128, 128, out_n, true, !first, true);
        gemm_wait(s);
        first = false;
    }
    if (s.ok && !first) {
        float* g = p.grads + rc_layer_offset(l) + in_base + t;
        for (uint32_t o = 16 * sub; o < out_n; o += 32) {
            float v[16];
            read_row<16>(tmem + o, v);
            if (t < in_n)
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j) atomicAdd(g + (size_t)(o + j) * rc_layer_in(l), v[j]);
        }
    }
    cta_teardown(s, tmem, kTmemCols, p.status);
}

// ---- Adam and the operand copies ------------------------------------------------------
// One thread per weight w = (layer l, output o, input i): Adam on the FP32
// master copy (padded output rows 3..15 stay zero), then the FP16 forward
// operand (row o, column i of W(l)) and, for layers 2..6, the BF16 backward
// operand (row i, column o).  Clears the gradient for the next step.
__global__ void rc_adam(RcAdam p) {
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= kWeightCount) return;
    int l = 0;
    while (l < kLayers - 1 && w >= rc_layer_offset(l + 1)) ++l;
    const uint32_t local = w - rc_layer_offset(l);
    const uint32_t in_n = rc_layer_in(l), out_n = rc_layer_out(l);
    const uint32_t o = local / in_n, i = local % in_n;
    const bool real = o < (l == kLayers - 1 ? (uint32_t)kOutputs : out_n);
    float val = real ? p.params[w] : 0.0f;
    if (p.step > 0 && real) {
        const float g = p.grads[w] * p.grad_scale;
        const float m = p.beta1 * p.m[w] + (1.0f - p.beta1) * g;
        const float v = p.beta2 * p.v[w] + (1.0f - p.beta2) * g * g;
        p.m[w] = m;
        p.v[w] = v;
        const float mh = m / (1.0f - p.beta1_pow), vh = v / (1.0f - p.beta2_pow);
        val -= p.lr * mh / (sqrtf(vh) + p.eps);
        p.params[w] = val;
    }
    p.grads[w] = 0.0f;
    *(uint16_t*)((unsigned char*)p.weights_f16 + rc_layer_offset(l) * 2 + tc::kmajor_offset(o, i, in_n)) = f2h(val);
    if (l >= 1)
        *(uint16_t*)((unsigned char*)p.weights_bf16 + bwd_offset(l) * 2 + tc::kmajor_offset(i, o, out_n)) = f2b(val);
}

}  // namespace rc

// ---- launchers ---------------------------------------------------------------------------
namespace {
template <class K>
cudaError_t allow_smem(K kernel, uint32_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}
}  // namespace

cudaError_t rc_launch_forward(const RcForward& p, bool train, int grid, cudaStream_t s) {
    auto* kernel = train ? rc::rc_forward<true> : rc::rc_forward<false>;
    const uint32_t smem = rc::forward_smem(train);
    const cudaError_t e = allow_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<grid, rc::kGroup * rc::kTiles, smem, s>>>(p);
    return cudaGetLastError();
}

cudaError_t rc_launch_wgrad(const RcWgrad& p, cudaStream_t s) {
    cudaError_t e = allow_smem(rc::rc_wgrad, rc::kWgradSmem);
    if (e != cudaSuccess) return e;
    rc::rc_wgrad<<<kWgradJobs * p.splits, rc::kGroup, rc::kWgradSmem, s>>>(p);
    return cudaGetLastError();
}

cudaError_t rc_launch_adam(const RcAdam& p, cudaStream_t s) {
    rc::rc_adam<<<(kWeightCount + 255) / 256, 256, 0, s>>>(p);
    return cudaGetLastError();
}

}  // namespace orn
