// Quantise and pack in one kernel: fp16 weight [N, K] -> tile-ordered int4 `weight` + `zeros_scales`.
//
// Replaces, for the offline quantise-and-pack flow of the reference (quant_lmdeploy,
// test/nvidia/utils/quant_dequant_nvidia.py:5-32), the chain
//     quantize_tensor  (:124-148: seven fp16 torch elementwise / reduce kernels)
//  -> write_4bit_tensor (:79-88)
//  -> transpose_merge_zeros_scales (kernel/gemm_s4_f16/format.cu:206-239)
//  -> convert_ours_to_awq          (format.cu:151-201)
//  -> convert_awq_to_lmdeploy      (format.cu:135-149, 24-71: one nibble per thread iteration through atomicCAS)
// with ONE pass over the weight: a CTA takes a block of 32 out-features x 128 in-features, computes min/max, scale,
// zero point and the 4-bit codes of every quantisation group in it with the reference's fp16 operation order, and
// writes the packed 32x32 tiles directly in their final order (the AWQ intermediate never exists).
//
// Arithmetic, bit for bit what the torch fp16 ops of the reference produce (each step rounds to fp16 once,
// round-to-nearest-even; torch's half kernels compute in fp32 with IEEE division, see the kernel for what stands for it):
//     d      = fp16(max - min);  d = max(d, fp16(1e-5))              (.clamp(min=1e-5))
//     scale  = fp16(d / 15)
//     zero   = clamp(-rint(fp16(min / scale)), 0, 15)                (torch.round = half to even)
//     q      = clamp(fp16(rint(fp16(w / scale)) + zero), 0, 15)
//     w_fp16 = fp16((q - zero) * scale)                              (no flush-to-zero: this is the quantizer's own
//                                                                    dequantised copy, not the kernel's)
// Outputs: weight int32 [K, N/8] in tile order, zeros_scales fp16 [K/g, 2N] = (zero + 64, scale), and optionally
// w_fp16 [N, K], zeros / scales fp16 [N, K/g] and the reference's intermediate "ours" bytes uint8 [N, K/2].
#include "w4a16_common.cuh"

namespace w4a16 {
namespace {

constexpr int kBlockK = 128;      // in-features per CTA: one to four quantisation groups
constexpr int kRows   = 32;       // out-features per CTA: one packed tile column
constexpr int kThreads = 128;     // four 16-byte vectors of the block per thread, all requested before the first is used
constexpr int kRowWords = kBlockK / 2 + 4;      // code pairs per row in shared memory; 68 = 4 mod 32: the packing reads below
                                                // (8 rows x 4 consecutive words) fall in 32 distinct banks

struct QuantParams {
    const __half* w;        // [N, K]
    uint32_t* qweight;      // [K/32][N/32][32 lanes][4 words]
    __half2* zs;            // [K/g][N]
    __half* w_fp16;         // [N, K] or null
    __half* zeros;          // [N, K/g] or null
    __half* scales;         // [N, K/g] or null
    uint8_t* ours;          // [N, K/2] or null
    int N, K, g;
};

__device__ __forceinline__ float h2f(__half h) { return __half2float(h); }
__device__ __forceinline__ __half f2h(float f) { return __float2half_rn(f); }
__device__ __forceinline__ uint32_t bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }

// What bounds this kernel is HBM: 4 bytes a weight in and out plus 0.53 packed.  With one IEEE division a weight and
// scalar fp32 arithmetic it was bound by instructions (172 us on 16384 x 4096, 1.77 TB/s; now 74 us, 4.1 TB/s), hence:
//   * no division in the loop: w * rn(1 / scale) instead of w / scale.  rint(fp16(.)) of the two is the same for EVERY
//     pair of finite fp16 values (with W, S the 11-bit significands and M the 12-bit one of a rounding midpoint,
//     |w / s - m| >= m / (M S) > m 2^-23 (1 + 2^-12), more than the two fp32 roundings move the product by; below the
//     normal range of fp16, where midpoints can be hit, both round to integer 0; checked over all pairs).  Likewise
//     fp16(d / 15) == fp16(d * rn(1 / 15)) for every fp16 d;
//   * everything behind the scaled value in half2, two weights an instruction: h + 1536 rounds to the integer (half to
//     even, |h| < 512; beyond that the clamp decides), minus (1536 - zero) is exact; q - zero is exact and the product with
//     scale rounds once, as in fp32 followed by a rounding to fp16;
//   * q + 1024 has the code in its low nibble: pairs of codes are parked in shared memory in that form and the packed
//     words are four such pairs shifted over each other.
//
// kVec16 = false: some pointer is aligned for 8-byte vectors only (slices of larger buffers); same code in halves.
template <bool kVec16>
__global__ void __launch_bounds__(kThreads) quantize_pack_kernel(const QuantParams p)
{
    __shared__ uint32_t qs[kRows][kRowWords];           // (q + 1024, q' + 1024) of in-features 2i, 2i + 1
    __shared__ __half2 zs_s[kBlockK / 32][kRows];
    const int n0 = blockIdx.x * kRows, k0 = blockIdx.y * kBlockK;
    const int kw = min(kBlockK, p.K - k0);              // in-features of this block (a multiple of g and of 32)
    const int lanes_per_group = p.g / 8;                // a lane holds 8 consecutive in-features of a row
    const int groups_total = p.K / p.g;
    const int vec = threadIdx.x & 15, row0 = threadIdx.x >> 4;        // rows row0, row0 + 8, ...
    const bool live = 8 * vec < kw;
    const __half* src = p.w + (size_t)(n0 + row0) * p.K + k0 + 8 * vec;

    uint4 raw[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        raw[i] = make_uint4(0, 0, 0, 0);
        if (live) {
            const __half* s = src + (size_t)(8 * i) * p.K;
            if constexpr (kVec16) {
                raw[i] = ldg_nc_v4(s);
            } else {
                const uint2 a = reinterpret_cast<const uint2*>(s)[0], b = reinterpret_cast<const uint2*>(s)[1];
                raw[i] = make_uint4(a.x, a.y, b.x, b.y);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = row0 + 8 * i, n = n0 + row, k = k0 + 8 * vec;
        const __half2* v = reinterpret_cast<const __half2*>(&raw[i]);
        __half2 mx2 = __hmax2(__hmax2(v[0], v[1]), __hmax2(v[2], v[3])), mn2 = __hmin2(__hmin2(v[0], v[1]), __hmin2(v[2], v[3]));
        for (int off = 1; off < lanes_per_group; off <<= 1) {         // reduce inside the lanes of one group
            mx2 = __hmax2(mx2, __shfl_xor_sync(0xffffffffu, mx2, off));
            mn2 = __hmin2(mn2, __shfl_xor_sync(0xffffffffu, mn2, off));
        }
        const float mx = h2f(__hmax(__low2half(mx2), __high2half(mx2))), mn = h2f(__hmin(__low2half(mn2), __high2half(mn2)));
        // max, min are exact fp16 values; every step below rounds to fp16 like the reference's torch ops
        float d = h2f(f2h(mx - mn));
        d = fmaxf(d, h2f(f2h(1e-5f)));
        const __half scale_h = f2h(d * (1.f / 15.f));
        const float inv = __frcp_rn(h2f(scale_h));
        const float t = h2f(f2h(mn * inv));
        const float zero = fminf(fmaxf(-rintf(t), 0.f), 15.f);        // -rint(+-inf) clamps as torch does; min == 0 gives 0
        const __half2 scale2 = __half2half2(scale_h), zero2 = __half2half2(f2h(zero));
        const __half2 back2 = __half2half2(f2h(1536.f - zero)), k1536 = __half2half2(f2h(1536.f)), k1024 = __half2half2(f2h(1024.f));
        const __half2 zero_h2 = __half2half2(__half()), k15 = __half2half2(f2h(15.f));
        uint32_t code[4];
        __half2 deq[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 f = __half22float2(v[j]);
            const __half2 h = __floats2half2_rn(f.x * inv, f.y * inv);
            const __half2 q = __hmin2(__hmax2(__hsub2(__hadd2(h, k1536), back2), zero_h2), k15);
            code[j] = bits(__hadd2(q, k1024));
            deq[j] = __hmul2(__hsub2(q, zero2), scale2);
        }
        if (live) {
            *reinterpret_cast<uint4*>(&qs[row][4 * vec]) = make_uint4(code[0], code[1], code[2], code[3]);
            if (p.w_fp16) {
                __half* dst = p.w_fp16 + (size_t)n * p.K + k;
                if constexpr (kVec16) {
                    *reinterpret_cast<uint4*>(dst) = make_uint4(bits(deq[0]), bits(deq[1]), bits(deq[2]), bits(deq[3]));
                } else {
                    reinterpret_cast<uint2*>(dst)[0] = make_uint2(bits(deq[0]), bits(deq[1]));
                    reinterpret_cast<uint2*>(dst)[1] = make_uint2(bits(deq[2]), bits(deq[3]));
                }
            }
            if (p.ours) {
                uint32_t b = 0;                                        // high nibble = even k
#pragma unroll
                for (int j = 0; j < 4; ++j) b |= (((code[j] & 15u) << 4) | ((code[j] >> 16) & 15u)) << (8 * j);
                uint16_t* dst = reinterpret_cast<uint16_t*>(p.ours + (size_t)n * (p.K / 2) + k / 2);
                dst[0] = (uint16_t)b;
                dst[1] = (uint16_t)(b >> 16);
            }
            if ((vec & (lanes_per_group - 1)) == 0) {
                zs_s[vec / lanes_per_group][row] = __halves2half2(f2h(zero + 64.f), scale_h);       // zero + 64 is exact in fp16
                const int kg = k / p.g;
                if (p.zeros) p.zeros[(size_t)n * groups_total + kg] = f2h(zero);
                if (p.scales) p.scales[(size_t)n * groups_total + kg] = scale_h;
            }
        }
    }
    __syncthreads();

    // The block's kw / 32 packed tiles: warp t makes tile t, a lane its four words.  For element (n, k) of a tile:
    // lane = (n % 8) * 4 + (k % 8) / 2, word = ((k / 16) % 2) * 2 + (n / 16) % 2,
    // nibble = (k % 2) * 4 + ((k / 8) % 2) * 2 + (n / 8) % 2.
    const int t = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (t < kw / kTileK) {
        const int r = lane >> 2, c = t * (kTileK / 2) + (lane & 3);
        uint32_t w[4];
#pragma unroll
        for (int wd = 0; wd < 4; ++wd) {
            w[wd] = 0;
#pragma unroll
            for (int nib = 0; nib < 4; ++nib)
                w[wd] |= (qs[r + 8 * (nib & 1) + 16 * (wd & 1)][c + 4 * (nib >> 1) + 8 * (wd >> 1)] & 0x000f000fu) << (4 * nib);
        }
        uint32_t* dst = p.qweight + (((size_t)(k0 / kTileK + t) * (p.N / kTileN) + blockIdx.x) * 32 + lane) * 4;
        if constexpr (kVec16) {
            *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        } else {
#pragma unroll
            for (int wd = 0; wd < 4; ++wd) dst[wd] = w[wd];
        }
    }
    const int groups = kw / p.g;
    if ((int)threadIdx.x < groups * kRows)
        p.zs[(size_t)(k0 / p.g + (threadIdx.x >> 5)) * p.N + n0 + lane] = zs_s[threadIdx.x >> 5][lane];
}

}  // namespace
}  // namespace w4a16

using namespace w4a16;

extern "C" int w4a16_quantize_pack(const void* weight, void* qweight, void* zeros_scales, void* w_fp16, void* zeros,
                                   void* scales, void* qweight_ours, int in_features, int out_features, int group_size,
                                   void* stream)
{
    const int K = in_features, N = out_features, g = group_size;
    if (g != 32 && g != 64 && g != 128) return W4A16_ERR_GROUP_SIZE;
    if (N <= 0 || K <= 0 || (N % 32) || (K % g)) return W4A16_ERR_BAD_SHAPE;
    if ((long long)N * K >= (1ll << 40) || (K + kBlockK - 1) / kBlockK > 65535) return W4A16_ERR_BAD_SHAPE;
    if (!weight || !qweight || !zeros_scales) return W4A16_ERR_NULL_POINTER;
    if (((uintptr_t)weight & 7) || ((uintptr_t)qweight & 3) || ((uintptr_t)zeros_scales & 3) || ((uintptr_t)w_fp16 & 7) ||
        ((uintptr_t)zeros & 1) || ((uintptr_t)scales & 1) || ((uintptr_t)qweight_ours & 1))
        return W4A16_ERR_MISALIGNED;
    QuantParams p;
    p.w = (const __half*)weight; p.qweight = (uint32_t*)qweight; p.zs = (__half2*)zeros_scales;
    p.w_fp16 = (__half*)w_fp16; p.zeros = (__half*)zeros; p.scales = (__half*)scales; p.ours = (uint8_t*)qweight_ours;
    p.N = N; p.K = K; p.g = g;
    dim3 grid(N / kRows, (K + kBlockK - 1) / kBlockK);
    if (((uintptr_t)weight | (uintptr_t)qweight | (uintptr_t)w_fp16) & 15) quantize_pack_kernel<false><<<grid, kThreads, 0, (cudaStream_t)stream>>>(p);
    else quantize_pack_kernel<true><<<grid, kThreads, 0, (cudaStream_t)stream>>>(p);
    count_launch();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? W4A16_OK : record_cuda_error(e);
}
