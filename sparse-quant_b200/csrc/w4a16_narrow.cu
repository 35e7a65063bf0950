// Batched-decode kernel: W4A16 GEMM for a few dozen tokens on the 5th-generation tensor cores.
//
//   out[t, n] = fp16( sum_g s[n, g] * sum_{k in g} (q[n, k] - z[n, g]) * x[t, k] ) (+ bias[n])
//
// Replaces the 16-wide and 32-wide instantiations of gemm_s4_f16_nn (gemm_template.h:358-464, gemm_s4_f16.cu:66-87 of the
// reference).  Bound: the packed weights' way from HBM.  With mma.sync the batch is paid for in issue slots (8.2 cycles
// per m16n8k16 and scheduler, four of them per 16 x 16 weights at 32 tokens); here the cost of a weight does not depend
// on the batch: it is unpacked once, written to tensor memory and multiplied by tcgen05.mma.
//
// The arithmetic keeps the decode kernels' precision: what goes into the MMA is the integer q - z (exact in fp16), a
// quantisation group accumulates in fp32 in tensor memory, and the scale is applied in fp32 when the group's sums are
// added up in registers - the weight is never rounded to fp16 (a denormal scale is flushed, as mul.ftz does).
//
// One CTA per SM, warp specialised; a unit of work (stage) is 128 out-features x 128 k:
//   warps 0, 3  weights: one tensor copy of the four k-tile rows of four packed tiles, one of the (zero, scale) rows; a ring
//               as deep as shared memory allows (about 100 KB in flight); under programmatic launch they start before the
//               previous grid has ended
//   warp 1      activations: one tensor copy of two swizzled 64-k sub-tiles of T tokens.  One copy a stage and producer: with
//               two in one warp the producers' loops took 700 cycles a stage and set the pace
//   warp 2      tcgen05.mma, eight per stage, one commit
//   warps 4-19  dequantisers: a warp takes a 32-feature quarter of a stage, four sets of four take stages in turn (a barrier
//               round trip costs as much as unpacking a tile: a task of four tiles, not two)
//   warps 20..  scale and accumulate: tcgen05.ld of a group's sums, acc += s * sum, 16 tokens a warp (32 of the 64-token tile)
// Two barriers per stage tie the three together: `ready` (dequantised weights written, activations arrived, group sums
// of the slot's last user read: one probe for the MMA warp, whose loop sets the pace - with a barrier for each it issued a
// stage every 600 cycles, and eight MMAs take 360) and `done` (the stage's MMAs have completed).  Ring indexes run on
// across the CTA's out-feature blocks.  Edges need no code: copies past N, K or the tokens arrive as zeros, and a missing
// group's scale is zero.
//
// Split of the work: a cluster of S CTAs takes b out-feature blocks and splits K; the partial sums meet in shared memory
// and are added over the cluster in rank order (deterministic, no scratch in global memory, capturable).  Every mbarrier
// wait is bounded; a timeout raises the device error word.
#include <cooperative_groups.h>
#include <cuda.h>

#include "w4a16_common.cuh"
#include "w4a16_sm100.cuh"

namespace cg = cooperative_groups;

namespace w4a16 {

using namespace sm100;

namespace {

constexpr int kBlockN = 128, kBlockK = 128;
constexpr uint64_t kWaitBudgetNs = 400ull * 1000 * 1000;
constexpr int kMaxStages = 16;
constexpr int kFirstDequantWarp = 4, kFirstEpilogueWarp = 20;
constexpr int kDequantSets = (kFirstEpilogueWarp - kFirstDequantWarp) / 4;      // sets of four warps that take stages in turn
constexpr int kNarrowSmem = 227 * 1024;

template <int T, int G>
struct NarrowCfg {
    static constexpr int kGroups = kBlockK / G;                          // quantisation groups per stage
    static constexpr int kRing = T == 64 ? 4 : 6;                        // A ring, in stages
    static constexpr int kDRing = T == 32 && G == 64 ? 2 : (T == 64 && G == 64 ? 2 : 4);     // group sums, in stages
    static constexpr int kDCol = 64 * kRing;                             // first tensor memory column of the sums
    static constexpr int kXSub = T * 128, kXStage = 2 * kXSub;           // bytes
    static constexpr int kWStage = 16 * 512 + kGroups * 512;
    static constexpr int kEpiCols = T < 64 ? 16 : 32;                    // tokens per epilogue warp
    static constexpr int kEpiWarps = 4 * (T / kEpiCols);
    static constexpr int kThreads = 32 * (kFirstEpilogueWarp + kEpiWarps);
    static constexpr int kBarriers = 4 * kMaxStages;
    static constexpr int kBarBytes = 1024;
    static constexpr int kRedBytes = T * kBlockN * 4;                    // fp32 sums of one out-feature block
    static_assert(kDCol + T * kGroups * kDRing <= 512, "tensor memory");
    static_assert(8 * kBarriers + 8 <= kBarBytes, "barrier area");
    static bool guard(int stages) { return stages < kRing + kDequantSets; }
    static int stages(int blocks)                                        // depth of the weight and activation rings
    {
        const int room = (kNarrowSmem - 1024 - kBarBytes - blocks * kRedBytes) / (kXStage + kWStage);
        return room < kMaxStages ? room : kMaxStages;
    }
};

struct NarrowParams {
    const uint32_t* zs;
    const __half*   bias;
    const __half*   residual;
    __half*         out;
    int*            error;
    int tokens, N, K;
    int n_blocks;        // out-feature blocks of the matrix
    int blocks;          // out-feature blocks per cluster
    int splits;          // CTAs per cluster: parts of K
    int stages;          // Q: depth of the rings in shared memory and of the barriers
    int relu, silu_mul, pdl;
};

__device__ __forceinline__ float ld_cluster_f32(uint32_t local_addr, uint32_t rank)
{
    uint32_t remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}

// (64 + q) - (64 + z) of two lanes: exact, both are fp16 numbers of the same few binades
__device__ __forceinline__ uint32_t sub_h2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("sub.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// GUARD: the rings are so shallow that the dequantisers need the extra wait explained there (the 64-token tile's always are)
template <int T, int G, bool GUARD>
__global__ void __launch_bounds__(NarrowCfg<T, G>::kThreads, 1) narrow_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map,
                                                                           const __grid_constant__ CUtensorMap zs_map, const NarrowParams p)
{
    using Cfg = NarrowCfg<T, G>;
    constexpr int R = Cfg::kRing, DR = Cfg::kDRing, GPS = Cfg::kGroups;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char* smem = smem_raw + (smem_base - smem_u32(smem_raw));
    const int Q = p.stages;
    const uint32_t w_off = Q * Cfg::kXStage, red_off = w_off + Q * Cfg::kWStage, bar_off = red_off + p.blocks * Cfg::kRedBytes;
    const uint32_t bar_base = smem_base + bar_off;
    auto ready_bar  = [&](int s) { return bar_base + 8u * s; };
    auto done_bar   = [&](int s) { return bar_base + 8u * (kMaxStages + s); };
    auto wfull_bar  = [&](int s) { return bar_base + 8u * (2 * kMaxStages + s); };
    auto wempty_bar = [&](int s) { return bar_base + 8u * (3 * kMaxStages + s); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + bar_off + 8 * Cfg::kBarriers);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t red_base = smem_base + red_off;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (p.pdl) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int k_steps = (p.K + kBlockK - 1) / kBlockK;
    const int S = p.splits, rank = blockIdx.y;
    const int ks0 = k_steps * rank / S, ks1 = k_steps * (rank + 1) / S;
    const int nb0 = blockIdx.x * p.blocks, nblk = min(p.blocks, p.n_blocks - nb0);
    const int total = nblk * (ks1 - ks0);                            // stages of this CTA
    auto load_weights = [&](int sw, int nb, int ks) {                // one elected lane
        const uint32_t dst = smem_base + w_off + sw * Cfg::kWStage, bar = wfull_bar(sw);
        mbar_arrive_expect_tx(bar, 8192);
        tma_load_2d(dst, &w_map, nb * 256, ks * 4, bar);
    };
    // Under programmatic launch the previous grid may still run for as long as it likes (a fused exchange waits seconds for a
    // peer): whoever waits, directly or through others, for something the activations set off does so only behind this, or the
    // bounded waits would count the previous grid's time as their own and give up.
    auto after_previous = [&]() { if (p.pdl) asm volatile("griddepcontrol.wait;" ::: "memory"); };
    // Giving up.  A bounded wait may end differently for two lanes of a warp (they probe, read the timer and the flag one by
    // one), and behind the waits stand warp-wide instructions: no lane may leave a loop on its own.  The producers vote and
    // leave after the budget, which costs nothing.  In the other roles a vote, or a test in front of each arrival, costs 1 to 3 %
    // of a call.  They have twice the budget: by then every producer has left or is done and no copy has been issued for as
    // long, so an arrival too many cannot meet a barrier that only waits for bytes, and they just run their loops out.
    auto wait_all = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, kWaitBudgetNs)) != 0; };
    auto wait_on = [&](uint32_t bar, uint32_t parity) {
        constexpr uint32_t kProbeNs = 50000;
        constexpr int kRunOut = 2;
        if (mbar_try_wait(bar, parity, kProbeNs)) return;
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(bar, parity, kProbeNs)) {
            if (*abort_flag == kRunOut) return;
            if (globaltimer_ns() - t0 > 2 * kWaitBudgetNs) { *abort_flag = kRunOut; return; }
        }
    };
    constexpr int kEarly = 2;                                        // stages requested before the rest of the CTA is set up
    if (warp == 0) {
        if (lane < Q) {
            mbar_init(ready_bar(lane), 4 + Cfg::kEpiWarps + 1); mbar_init(done_bar(lane), 1);
            mbar_init(wfull_bar(lane), 2); mbar_init(wempty_bar(lane), 4);
        }
        mbar_fence_init();
        __syncwarp();
    }
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < kEarly && i < ks1 - ks0; ++i) load_weights(i, nb0, ks0 + i);
    }
    if (warp == 3) {
        tmem_alloc(smem_u32((const void*)tmem_slot), 512);
        tmem_relinquish();
    }
    if (warp == 1 && lane == 0) prefetch_tmap(&x_map);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---- packed weights ----
        int st = 0, nb = nb0, ks = ks0; uint32_t phase = 0;
        for (int it = 0; it < total; ++it) {
            if (it == Q) after_previous();
            if (it >= Q && !wait_all(wempty_bar(st), phase ^ 1u)) break;
            if ((it >= kEarly || it >= ks1 - ks0) && elect_one()) load_weights(st, nb, ks);
            __syncwarp();
            if (++ks == ks1) { ks = ks0; ++nb; }
            if (++st == Q) { st = 0; phase ^= 1u; }
        }
    } else if (warp == 1) {
        // ---- activations ----
        after_previous();
        int st = 0, ks = ks0; uint32_t phase = 0;
        for (int it = 0; it < total; ++it) {
            if (it >= Q && !wait_all(done_bar(st), phase ^ 1u)) break;
            if (elect_one()) {
                mbar_arrive_expect_tx(ready_bar(st), Cfg::kXStage);
                tma_load_3d(smem_base + st * Cfg::kXStage, &x_map, 0, 0, 2 * ks, ready_bar(st));
            }
            __syncwarp();
            if (++ks == ks1) ks = ks0;
            if (++st == Q) { st = 0; phase ^= 1u; }
        }
    } else if (warp == 3) {
        // ---- (zero, scale) rows ----
        int st = 0, nb = nb0, ks = ks0; uint32_t phase = 0;
        for (int it = 0; it < total; ++it) {
            if (it == Q) after_previous();
            if (it >= Q && !wait_all(wempty_bar(st), phase ^ 1u)) break;
            if (elect_one()) {
                mbar_arrive_expect_tx(wfull_bar(st), GPS * 512);
                tma_load_2d(smem_base + w_off + st * Cfg::kWStage + 8192, &zs_map, nb * kBlockN, ks * GPS, wfull_bar(st));
            }
            __syncwarp();
            if (++ks == ks1) { ks = ks0; ++nb; }
            if (++st == Q) { st = 0; phase ^= 1u; }
        }
    } else if (warp == 2) {
        // ---- MMA: the whole warp walks the loop, an elected lane issues (see elect_one) ----
        constexpr uint32_t idesc = idesc_f16_m128(T);
        const uint64_t bdesc0 = smem_desc_sw128(smem_base);
        // A probe of a barrier answers after some 200 cycles: each is asked two stages ahead, so that none is waited for.
        int st = 0, ahead = 0, slot = 0, d = 0; uint32_t phase = 0, ahead_phase = 0;
        bool ready0 = false, ready1 = false;
        auto probe = [&]() {
            const bool r = mbar_test_wait(ready_bar(ahead), ahead_phase);
            if (++ahead == Q) { ahead = 0; ahead_phase ^= 1u; }
            return r;
        };
        after_previous();
        ready0 = probe();
        ready1 = probe();
        for (int it = 0; it < total; ++it) {
            if (!ready0) wait_on(ready_bar(st), phase);
            __syncwarp();
            tc_fence_after_sync();
            const bool ready2 = probe();
            const uint64_t bdesc = bdesc0 + (uint64_t)((uint32_t)(st * Cfg::kXStage) >> 4);
            const uint32_t a_tmem = tmem_base + 64 * slot, d_tmem = tmem_base + Cfg::kDCol + d * (GPS * T);
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                    mma_f16_ts(d_tmem + (GPS == 2 && kk >= 4 ? T : 0), a_tmem + 8 * kk,
                               bdesc + (uint64_t)((kk >= 4 ? (Cfg::kXSub >> 4) : 0) + 2 * (kk & 3)), idesc, (GPS == 2 ? kk & 3 : kk) != 0);
                tc_commit(done_bar(st));
            }
            __syncwarp();
            if (++st == Q) { st = 0; phase ^= 1u; }
            if (++slot == R) slot = 0;
            if (++d == DR) d = 0;
            ready0 = ready1;
            ready1 = ready2;
        }
    } else if (warp >= kFirstDequantWarp && warp < kFirstEpilogueWarp) {
        // ---- dequantisers: tensor memory lane quarter = packed tile column = warp % 4 ----
        const int quarter = warp & 3, set = (warp - kFirstDequantWarp) >> 2;
        const uint32_t lane_field = (uint32_t)(quarter * 32) << 16;
        auto step = [](int& i, int by, int n) { i += by; const bool wrap = i >= n; if (wrap) i -= n; return wrap; };
        static_assert(kDequantSets <= R, "the first A slots are free");
        int st = set, slot = set, freed = set + Q - R; uint32_t phase = 0, freed_phase = 1;    // freed: the stage R back, whose A slot is taken
        // A wait names a round of a ring by its parity, which is only right where the round before is known to be complete.
        // What a set knows of the weights of stage it - Q, which another set unpacked, comes from its own last stage: all
        // MMAs up to it - 4 - R have run, so the weights up to there had landed.  With fewer than R + 4 stages that does not
        // reach it - Q: a set that overtook one still waiting for its weights would take those for its own, read them half
        // landed and hand their slot to the next copy.  There (GUARD) it waits for the MMAs of stage it - Q first.
        for (int it = set; it < total; it += kDequantSets) {
            {
                const bool turned = !(GUARD && it >= Q) || mbar_test_wait(done_bar(st), phase ^ 1u);
                bool loaded = mbar_test_wait(wfull_bar(st), phase);                  // the probes are in flight together
                const bool slot_free = it < R || mbar_test_wait(done_bar(freed), freed_phase);
                const bool first = it >= R && it < R + kDequantSets;                 // this set's first wait for an MMA
                if (!turned) {
                    if (first) after_previous();
                    wait_on(done_bar(st), phase ^ 1u);
                    loaded = false;                                                  // asked before that round was known to be over
                }
                if (!loaded) wait_on(wfull_bar(st), phase);
                const unsigned char* wst = smem + w_off + st * Cfg::kWStage;
                const uint4* wq = reinterpret_cast<const uint4*>(wst) + quarter * 32 + lane;
                const uint32_t* zsp = reinterpret_cast<const uint32_t*>(wst + 8192) + quarter * 32 + (lane >> 2);
                uint4 q[4];
                uint32_t zz[GPS][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) q[i] = wq[128 * i];
#pragma unroll
                for (int gi = 0; gi < GPS; ++gi)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t z = zsp[128 * gi + 8 * i];
                        zz[gi][i] = __byte_perm(z, z, 0x1010);
                    }
                __syncwarp();
                if (lane == 0) mbar_arrive(wempty_bar(st));
                if (first) after_previous();
                if (!slot_free) wait_on(done_bar(freed), freed_phase);
                __syncwarp();
                tc_fence_after_sync();
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int gi = GPS == 2 ? half : 0;
                    const uint32_t words[2][4] = {{q[2 * half].x, q[2 * half].y, q[2 * half].z, q[2 * half].w},
                                                  {q[2 * half + 1].x, q[2 * half + 1].y, q[2 * half + 1].z, q[2 * half + 1].w}};
#pragma unroll
                    for (int nh = 0; nh < 2; ++nh) {
                        uint32_t a[16];
#pragma unroll
                        for (int i = 0; i < 2; ++i)
#pragma unroll
                            for (int kh = 0; kh < 2; ++kh) {
                                uint32_t h[4];
                                unpack_s4x8(words[i][kh * 2 + nh], h);
                                uint32_t* o = a + i * 8 + kh * 4;
                                o[0] = sub_h2(h[0], zz[gi][nh * 2]);
                                o[1] = sub_h2(h[1], zz[gi][nh * 2 + 1]);
                                o[2] = sub_h2(h[2], zz[gi][nh * 2]);
                                o[3] = sub_h2(h[3], zz[gi][nh * 2 + 1]);
                            }
                        tmem_st_16x128b_x8(tmem_base + lane_field + ((uint32_t)(nh * 16) << 16) + 64 * slot + 32 * half, a);
                    }
                }
                tmem_wait_st();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(ready_bar(st));
            }
            if (step(st, kDequantSets, Q)) phase ^= 1u;
            step(slot, kDequantSets % R, R);
            if (step(freed, kDequantSets, Q)) freed_phase ^= 1u;
        }
    } else if (warp >= kFirstEpilogueWarp) {
        // ---- scale and accumulate: thread = out-feature (tensor memory lane), registers = tokens ----
        constexpr int EC = Cfg::kEpiCols;
        const int quarter = warp & 3, col0 = ((warp - kFirstEpilogueWarp) >> 2) * EC;
        const uint32_t lane_field = (uint32_t)(quarter * 32) << 16;
        if (lane == 0)
            for (int i = 0; i < DR && i < total; ++i) mbar_arrive(ready_bar(i));          // the first sums find their slots free
        // The scales come straight from global memory, four stages ahead of their use (the dequantisers' copy has just
        // brought the line into L2): no barrier, and the weight ring is not held up.
        constexpr int kAhead = 4;
        const int groups = p.K / G;
        uint32_t zs[kAhead][GPS];
        int fnb = nb0, fks = ks0;                                 // the stage of the next fetch
        auto fetch = [&](uint32_t (&w)[GPS]) {
            const int n = min(fnb * kBlockN + quarter * 32 + lane, p.N - 1);
#pragma unroll
            for (int gi = 0; gi < GPS; ++gi) {
                const int g = fks * GPS + gi;
                w[gi] = g < groups ? ldg_nc_u32(p.zs + (size_t)g * p.N + n) : 0u;
            }
            if (++fks == ks1) { fks = ks0; ++fnb; }
        };
#pragma unroll
        for (int i = 0; i < kAhead; ++i) if (i < total) fetch(zs[i]);
        int st = 0, d = 0, free_st = DR % Q, left = ks1 - ks0; uint32_t phase = 0;     // free_st: the stage that gets this sum's slot next
        float acc[EC];
#pragma unroll
        for (int i = 0; i < EC; ++i) acc[i] = 0.f;
        after_previous();
        float* red = reinterpret_cast<float*>(smem + red_off) + col0 * kBlockN + quarter * 32 + lane;
        for (int base = 0; base < total; base += kAhead) {
            // unrolled over the scales in flight: handing them down a register queue would wait for the newest load
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const int it = base + u;
                if (it >= total) break;
                wait_on(done_bar(st), phase);
                __syncwarp();
                tc_fence_after_sync();
                float s0[GPS];
#pragma unroll
                for (int gi = 0; gi < GPS; ++gi) {
                    uint32_t v = zs[u][gi];
                    asm("mul.ftz.f16x2 %0, %1, %2;" : "=r"(v) : "r"(v), "r"(0x3c003c00u));   // a denormal scale becomes 0, as under mul.ftz
                    s0[gi] = __half2float(__ushort_as_half((unsigned short)(v >> 16)));
                }
                const uint32_t src = tmem_base + lane_field + Cfg::kDCol + d * (GPS * T) + col0;
#pragma unroll
                for (int gi = 0; gi < GPS; ++gi)
#pragma unroll
                    for (int c = 0; c < EC; c += 16) {
                        uint32_t v[16];
                        tmem_ld_32x32b_x16(src + gi * T + c, v);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; ++i) acc[c + i] = fmaf(s0[gi], __uint_as_float(v[i]), acc[c + i]);
                    }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0 && it + DR < total) mbar_arrive(ready_bar(free_st));
                if (it + kAhead < total) fetch(zs[u]);
                if (++free_st == Q) free_st = 0;
                if (++st == Q) { st = 0; phase ^= 1u; }
                if (++d == DR) d = 0;
                if (--left == 0) {                                   // the block is complete
#pragma unroll
                    for (int i = 0; i < EC; ++i) { red[i * kBlockN] = acc[i]; acc[i] = 0.f; }
                    red += Cfg::kRedBytes / 4;
                    left = ks1 - ks0;
                }
            }
        }
    }

    // ---- the partial sums of the cluster meet: each rank finishes a slice of the outputs ----
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {                                               // let copies and MMAs in flight end before their memory goes
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000) { }
        if (threadIdx.x == 0) atomicExch(p.error, 1);
        __syncwarp();
    }
    if (warp == 3) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
    cg::cluster_group cluster = cg::this_cluster();
    if (S > 1) cluster.sync();
    after_previous();                                                // outputs and residual belong to earlier work until then
    auto total_of = [&](int blk, int tok, int f) {
        const uint32_t at = red_base + (uint32_t)(blk * Cfg::kRedBytes + (tok * kBlockN + f) * 4);
        float v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = q < S ? ld_cluster_f32(at, (uint32_t)q) : 0.f;
        float s = v[0];
#pragma unroll
        for (int q = 1; q < 8; ++q) s += v[q];
        return s;
    };
    auto finish = [&](float s, int n) {
        __half h = __float2half_rn(s);
        if (p.bias) h = __hadd(h, p.bias[n]);
        if (p.relu) h = __hmax(h, __half());
        return h;
    };
    const unsigned rows = (unsigned)p.tokens;
    if (p.silu_mul) {
        // gate and up tiles alternate: features f and f + 32 are a pair, one thread owns both (the roundings of the
        // separate activation and product kernels)
        const unsigned total = (unsigned)nblk * rows * (kBlockN / 2);
        const unsigned lo = total * rank / S, hi = total * (rank + 1) / S;
        for (unsigned e = lo + threadIdx.x; e < hi; e += Cfg::kThreads) {
            const int pl = e & 63, f = ((pl >> 5) << 6) + (pl & 31);
            const unsigned bt = e >> 6, blk = bt / rows, tok = bt - blk * rows;
            const int n = (nb0 + (int)blk) * kBlockN + f;
            if (n + 32 < p.N) {
                const float gate = __half2float(finish(total_of(blk, tok, f), n));
                const __half up = finish(total_of(blk, tok, f + 32), n + 32);
                p.out[(size_t)tok * (p.N >> 1) + (nb0 + (int)blk) * (kBlockN / 2) + pl] = __hmul(__float2half_rn(gate / (1.f + __expf(-gate))), up);
            }
        }
    } else {
        const unsigned total = (unsigned)nblk * rows * kBlockN;
        const unsigned lo = total * rank / S, hi = total * (rank + 1) / S;
#pragma unroll 2
        for (unsigned e = lo + threadIdx.x; e < hi; e += Cfg::kThreads) {
            const int f = e & (kBlockN - 1);
            const unsigned bt = e >> 7, blk = bt / rows, tok = bt - blk * rows;
            const int n = (nb0 + (int)blk) * kBlockN + f;
            if (n < p.N) {
                __half h = finish(total_of(blk, tok, f), n);
                const size_t at = (size_t)tok * p.N + n;
                if (p.residual) h = __hadd(h, p.residual[at]);
                p.out[at] = h;
            }
        }
    }
    if (S > 1) cluster.sync();                                       // peers may still be reading this CTA's sums
}

int g_force_blocks = 0, g_force_splits = 0;

struct NarrowPlan { int blocks, splits, stages; };

template <int T, int G, bool GUARD>
int prepare_instance(int* max_smem_set)
{
    static int configured[64] = {0};       // benign race: the attribute call is idempotent
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return record_cuda_error(e);
    if (dev >= 64 || !configured[dev]) {
        e = cudaFuncSetAttribute(narrow_kernel<T, G, GUARD>, cudaFuncAttributeMaxDynamicSharedMemorySize, kNarrowSmem);
        if (e != cudaSuccess) return record_cuda_error(e);
        if (dev < 64) configured[dev] = 1;
    }
    *max_smem_set = dev;
    return W4A16_OK;
}

// clusters of `sp` CTAs the device runs at once (a CTA takes an SM: a property of how the SMs are grouped); cached
template <int T, int G>
int max_clusters(int sp)
{
    static int cache[64][9] = {};          // benign race: the query is idempotent
    int dev = 0;
    if (sp <= 1) return device_sm_count();
    if (prepare_instance<T, G, true>(&dev) != W4A16_OK || dev >= 64) return 0;
    if (cache[dev][sp]) return cache[dev][sp] > 0 ? cache[dev][sp] : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, sp, 1);
    cfg.blockDim = dim3(NarrowCfg<T, G>::kThreads);
    cfg.dynamicSmemBytes = kNarrowSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = sp;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, narrow_kernel<T, G, true>, &cfg) != cudaSuccess) { n = 0; (void)cudaGetLastError(); }
    cache[dev][sp] = n > 0 ? n : -1;
    return n;
}

// Blocks per cluster and cluster size: the fewest stages in the busiest CTA among the shapes that run as one wave; a
// reduction over a cluster counts as two stages, a shallow weight ring as proportionally slower stages.
template <int T, int G>
NarrowPlan plan_narrow(int N, int K)
{
    const int n_blocks = (N + kBlockN - 1) / kBlockN, k_steps = (K + kBlockK - 1) / kBlockK;
    NarrowPlan best = {0, 0, 0};
    double best_cost = 0;
    for (int sp = 1; sp <= 8 && sp <= k_steps; ++sp) {
        if (g_force_splits && sp != g_force_splits) continue;
        const int room = max_clusters<T, G>(sp);
        if (room <= 0) continue;
        int b = (n_blocks + room - 1) / room;
        if (g_force_blocks) b = g_force_blocks < n_blocks ? g_force_blocks : n_blocks;
        const int q = NarrowCfg<T, G>::stages(b);
        if (q < NarrowCfg<T, G>::kRing) continue;
        const double cost = (double)b * ((k_steps + sp - 1) / sp) * (q >= 10 ? 1.0 : 10.0 / q) + (sp > 1 ? 2.0 : 0.0);
        if (best.blocks == 0 || cost < best_cost) { best_cost = cost; best = {b, sp, q}; }
    }
    return best;
}

template <int T, int G>
int launch_instance(const GemmArgs& a, cudaStream_t st)
{
    using Cfg = NarrowCfg<T, G>;
    const NarrowPlan pl = plan_narrow<T, G>(a.N, a.K);
    if (pl.blocks == 0) return W4A16_ERR_BAD_ALGO;
    // (with one k-step, and in other corners, the rings need no second round and no guard; the instance is chosen by depth alone)
    const bool guard = T == 64 || Cfg::guard(pl.stages);
    int dev = 0;
    int s = guard ? prepare_instance<T, G, true>(&dev) : prepare_instance<T, G, T == 64>(&dev);
    if (s != W4A16_OK) return s;
    CUtensorMap x_map, w_map, zs_map;
    {
        // as [K/64][tokens][64]: a box of two is a stage's two swizzled sub-tiles, one copy
        const uint64_t dims[3] = {64, (uint64_t)a.tokens, (uint64_t)(a.K / 64)}, strides[2] = {(uint64_t)a.K * sizeof(__half), 128};
        const uint32_t box[3] = {64, (uint32_t)T, 2};
        s = encode_tensor_map(&x_map, a.x, 2, 3, dims, strides, box, /*swizzle128*/ true);
        if (s != W4A16_OK) return s;
    }
    {
        // the packed matrix as 64-bit words, one row per k-tile row: a box of four rows of four packed tiles is one copy
        const uint64_t row_bytes = (uint64_t)(a.N / kTileN) * 512, dims[2] = {row_bytes / 8, (uint64_t)(a.K / kTileK)};
        const uint32_t box[2] = {256, 4};
        s = encode_tensor_map_2d(&w_map, a.qw, 8, dims, row_bytes, box, /*swizzle128*/ false);
        if (s != W4A16_OK) return s;
    }
    {
        const uint64_t dims[2] = {(uint64_t)a.N, (uint64_t)(a.K / G)};
        const uint32_t box[2] = {(uint32_t)kBlockN, (uint32_t)Cfg::kGroups};
        s = encode_tensor_map_2d(&zs_map, a.zs, 4, dims, (uint64_t)a.N * 4, box, /*swizzle128*/ false);
        if (s != W4A16_OK) return s;
    }
    NarrowParams p;
    p.zs = a.zs; p.bias = a.bias; p.residual = a.residual; p.out = a.out;
    p.error = device_error_word();
    if (!p.error) return W4A16_ERR_CUDA;
    p.tokens = a.tokens; p.N = a.N; p.K = a.K;
    p.n_blocks = (a.N + kBlockN - 1) / kBlockN; p.blocks = pl.blocks; p.splits = pl.splits; p.stages = pl.stages;
    p.relu = a.relu ? 1 : 0; p.silu_mul = a.silu_mul ? 1 : 0;
    p.pdl = a.static_weights && a.tokens <= 32 ? 1 : 0;              // beyond 32 tokens plain stream order, like the prefill kernel that shares the range
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.n_blocks + pl.blocks - 1) / pl.blocks, pl.splits, 1);
    cfg.blockDim = dim3(Cfg::kThreads);
    cfg.dynamicSmemBytes = 1024 + pl.stages * (Cfg::kXStage + Cfg::kWStage) + pl.blocks * Cfg::kRedBytes + Cfg::kBarBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = pl.splits;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.pdl ? 2 : 1;
    const cudaError_t e = guard ? cudaLaunchKernelEx(&cfg, narrow_kernel<T, G, true>, x_map, w_map, zs_map, p)
                                : cudaLaunchKernelEx(&cfg, narrow_kernel<T, G, T == 64>, x_map, w_map, zs_map, p);
    count_launch();
    return e == cudaSuccess ? W4A16_OK : record_cuda_error(e);
}

template <int T>
int launch_t(const GemmArgs& a, cudaStream_t st)
{
    return a.g == 64 ? launch_instance<T, 64>(a, st) : launch_instance<T, 128>(a, st);
}

}  // namespace

void narrow_force_config(int blocks, int splits) { g_force_blocks = blocks; g_force_splits = splits; }

bool narrow_supported(int tokens, int N, int K, int g)
{
    return tokens > 0 && tokens <= 64 && (g == 64 || g == 128) && (K % 64) == 0 && (N % kTileN) == 0;
}

// Time of a call of 33 to 64 tokens in ns, fitted to graphs of calls on weights from HBM (138 shapes, 768 <= K <= 16384,
// 768 <= N <= 22016, both group sizes, 33, 48 and 64 tokens: within 18 %).
template <int G>
static double narrow_time_ns(int tokens, int N, int K)
{
    const NarrowPlan pl = plan_narrow<64, G>(N, K);
    if (pl.blocks == 0) return 1e30;
    const int k_steps = (K + kBlockK - 1) / kBlockK, stages = pl.blocks * ((k_steps + pl.splits - 1) / pl.splits);
    return 5400.0 + stages * (G == 64 ? 680.0 : 460.0) + 1800.0 * pl.blocks - (pl.splits > 1 ? 1400.0 : 0.0) + 38.0 * (tokens - 32);
}

bool narrow_preferred(int tokens, int N, int K, int g)
{
    // Measured in graphs of calls on weights from HBM, us, mma.sync kernels / this one: at 32 tokens 12.8 / 8.5 (4096 -> 4096),
    // 23.9 / 15.8 (12288), 26.3 / 17.6 (16384), 32.3 / 17.8 (16384 -> 4096), 35.4 / 28.4 (4096 -> 22016, g = 64): from 17 on.
    // At 9 to 16 tokens they are level with groups of 128 (7.4 / 7.8, 14.9 / 14.1, 15.4 / 15.6, 16.6 / 16.6), this one
    // ahead with groups of 64, twice the scale work for them (29.6 / 23.3, 15.8 / 13.5; of 138 shapes the mma.sync kernels
    // were ahead by more than 3 % on six, all with K <= 2048 and 4096 <= N <= 9600, at most 5.6 / 6.3).
    // At 33 to 64 the prefill kernel's 64-token tile takes one CTA per out-feature block and leaves SMs idle on narrow
    // matrices, where this one splits K; on wide ones this one takes several blocks per cluster, on shallow rings, and its
    // share per stage is larger, with groups of 64 above all.  Prefill kernel / this one at 48 tokens: 17.0 / 10.2
    // (4096 -> 4096), 17.4 / 14.9 (9472), 17.6 / 18.2 (11008), 17.8 / 22.1 (12288); with g = 64 16.9 / 12.0, 17.5 / 18.1,
    // 17.6 / 22.8, 17.7 / 29.4; short K 7.5 / 8.0 (768 -> 4096, g = 64), 8.3 / 11.8 (11008).  So their times are compared;
    // over the 414 measured points the choice loses 0.3 % to the better one on average, 3 to 10 % on fourteen.
    if (!narrow_supported(tokens, N, K, g)) return false;
    if (tokens > 32) return (g == 64 ? narrow_time_ns<64>(tokens, N, K) : narrow_time_ns<128>(tokens, N, K)) < tc_small_time_ns(tokens, N, K);
    return tokens > (g == 64 ? 8 : 16);
}

int launch_narrow(const GemmArgs& a, cudaStream_t st)
{
    if (!narrow_supported(a.tokens, a.N, a.K, a.g)) return W4A16_ERR_BAD_ALGO;
    if (a.silu_mul && ((a.N % 64) || a.residual)) return W4A16_ERR_BAD_SHAPE;
    return a.tokens <= 16 ? launch_t<16>(a, st) : a.tokens <= 32 ? launch_t<32>(a, st) : launch_t<64>(a, st);
}

}  // namespace w4a16
