// Q8_0 weight times several activation rows on the 5th-generation tensor cores (tcgen05), sm_100a: the projections and
// FFN matrices of a prompt (or of any call with more than one new token).
//
// Replaces the reference's gemm_q8_f32_kernel (src/shainet/native/cuda_kernels.cu:581-629) for several rows in the library's own
// entries (the symbol gemm_q8_f32 has no scratch and keeps the row tiles) and, through the small kernels around it, the host loops between the projections (rms_norm.cr:18-37, swiglu_ff.cr:76-91,
// llama_block.cr:189-196), with the single-row kernels' precision:
//
//  * the int8 weights are exact in bfloat16;
//  * an fp32 activation is exactly the sum of three bfloat16 values (8 + 8 + 8 significand bits: truncate, subtract,
//    truncate, subtract; below 2^-109 what is lost is less than 2^-133), so three products per weight reproduce the fp32
//    product with nothing rounded away, whatever else stands in the row;
//  * the products of one 32-input scale block accumulate in fp32 in tensor memory; a block is then multiplied by its
//    fp32 scale and added to fp32 accumulators in registers, sixteen blocks at a time by themselves (a single chain over
//    8192 inputs loses twice as much).
// Against f64 the error (2-norm) is 0.9e-7 at 2048 inputs and 1.0e-7 at 8192, that of the row kernels 1.04e-7 and 1.21e-7.
//
// A pair of CTAs (cta_group::2) computes 256 weight rows x NT tokens.  The weights are the A operand: raw int8 tiles
// arrive by TMA, four convert warps (one thread per weight row) turn 32 of them at a time into pairs of bfloat16 and put
// them into tensor memory; the activations are the B operand, three bfloat16 planes prepared by a kernel ahead, each CTA
// loading its half of the tokens.  Lanes of tensor memory are weight rows, so a thread of the accumulating warps needs
// one scale per block and stores its outputs coalesced over the lanes.
//
// Bounds.  The tensor core multiplies 4096 pairs per cycle and SM, but an MMA of 16 inputs takes at least about 64
// cycles, however few its columns (the 128 rows of A have to pass).  At 128 tokens the three planes are three passes: 384
// cycles per 32-input block; a block takes 760 (at 1.64 GHz, which six MMAs a block leave of the clock: 0.43 us).  72 % of the issue
// slots go to the converting and accumulating warps and their waits over the three accumulators that tensor memory has room for.  At 64 tokens there is room for six.  With up to 32 tokens the planes lie
// side by side as 3 NT columns of one pass, and the accumulating warps add the three columns of a token; the launch is then
// bound by the convert warps and the contraction is split over the pairs (split-K) until they are all busy.
// Measured, planes and split sums included: 4096 x 2048 -> 16384 in 777 us (row tiles of four on the CUDA cores 20.7 ms),
// 64 x 2048 -> 8192 in 22 us (186 us).
#include <cuda_bf16.h>
#include <math.h>
#include <algorithm>
#include <atomic>
#include "kernels.h"
#include "q8_gemm_tc.h"
#include "tcgen05.cuh"

namespace shainet {

namespace {

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 qt_pack(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f32x2 qt_pack_bits(uint32_t lo, uint32_t hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ f32x2 qt_add(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 qt_fma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Instruction descriptor: fp32 accumulate, bfloat16 A and B (both K-major), dense.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// NT tokens per tile (128, 64, 32 or 16).
template <int NT_>
struct QT {
    static constexpr int NT = NT_;
    static constexpr int ROWS = 128;                     // weight rows per CTA, 256 per pair
    static constexpr bool STACK = NT <= 32;              // the planes are columns of one pass, not three passes
    static constexpr int D_COLS = STACK ? 3 * NT : NT;   // columns of one block accumulator
    static constexpr int ND = NT == 16 ? 8 : NT == 32 ? 4 : NT == 64 ? 6 : 3;   // block accumulators (and A slots) in tensor memory
    static constexpr int A_COLS = 16;                    // 32 bfloat16 per lane
    static constexpr int TMEM_A = ND * D_COLS;
    static constexpr int TMEM_COLS = 512;
    static constexpr int NB = 6;                         // B stages of 64 inputs
    static constexpr int PLANE_BYTES = (NT / 2) * 128;   // this CTA's half of the tokens, 64 bfloat16 each
    static constexpr int B_BYTES = 3 * PLANE_BYTES;
    static constexpr int NW = NT == 128 ? 3 : 6;         // raw weight stages of 128 inputs
    static constexpr int W_BYTES = ROWS * 128;
    static constexpr int NS = 8;                         // scale stages of 4 blocks
    static constexpr int S_BYTES = ROWS * 16;
    static constexpr int ACC_WARPS = NT == 128 ? 16 : 8;
    static constexpr int CW = NT == 16 ? 8 : NT == 32 ? 16 : 32;   // tokens of one accumulating warp
    static constexpr int GROUP = 16;                     // blocks summed by themselves before they join the total: short chains of fp32 adds
    static constexpr int HC = CW < 16 ? 8 : 16;          // tokens read from tensor memory at once
    // 768 threads have 80 registers each; the accumulating warpgroups take 96, the two others 48 (256 x 48 + 512 x 96 =
    // 768 x 80)
    static constexpr bool REG_SPLIT = ACC_WARPS == 16;
    static constexpr int THREADS = (8 + ACC_WARPS) * 32;
    static constexpr int BAR_BYTES = 640;
    static constexpr size_t SMEM_BYTES = (size_t)NB * B_BYTES + (size_t)NW * W_BYTES + (size_t)NS * S_BYTES + BAR_BYTES;
    static_assert(TMEM_A + ND * A_COLS <= TMEM_COLS, "tensor memory columns");
    static_assert((2 * (NB + NW + NS + ND) + ND) * 8 + 4 <= BAR_BYTES, "barrier area");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
};

// Position in a ring of N barriers and the parity of its current round.
template <int N>
struct RingPos {
    int slot = 0;
    uint32_t parity = 0;
    __device__ __forceinline__ void next() {
        if (++slot == N) {
            slot = 0;
            parity ^= 1;
        }
    }
};

template <int N>
__device__ __forceinline__ void setmaxnreg_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void setmaxnreg_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

template <int CW>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&v)[CW]) {
    if constexpr (CW == 16) tmem_ld16(taddr, v);
    else tmem_ld8(taddr, v);
}

// The output segment of column `col` (selects, not indexing: the arrays stay in the parameter space).
struct OutColumn {
    float* ptr;
    int pitch;
    int col;   // inside the segment
};
__device__ __forceinline__ OutColumn out_column(const Q8GemmOut& o, int col) {
    OutColumn r{o.ptr[0], o.pitch[0], col};
    if (o.segments > 1 && col >= o.begin[1]) r = OutColumn{o.ptr[1], o.pitch[1], col - o.begin[1]};
    if (o.segments > 2 && col >= o.begin[2]) r = OutColumn{o.ptr[2], o.pitch[2], col - o.begin[2]};
    return r;
}

struct QtArgs {
    int M, K;
    int n[2];           // rows of the two weights (the second may be absent: 0)
    int n_tiles0;       // 256-row tiles of the first weight
    int n_tiles;        // of both
    int t_tiles;
    int splits;
    Q8GemmOut out;
    AttnStatus* status;
};

// Where the planes share an accumulator the last MMA of a block cuts its fp32 result towards zero: on average by
// 2^-24 / (2 ln 2) of it, the mean of half an ulp over the value (measured 4.3e-8).  That is put back as a gain in the
// last sum, before it is rounded; what stays has zero mean.  Side by side the planes' sums are not cut: the first one's products
// have 15 bits, and the fp32 adds of the others round.
constexpr float TRUNCATED = 0.7213f * 5.9604645e-8f;

template <int NT>
__global__ void __launch_bounds__(QT<NT>::THREADS, 1)
q8_gemm_tc_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w0,
                  const __grid_constant__ CUtensorMap tm_s0, const __grid_constant__ CUtensorMap tm_w1,
                  const __grid_constant__ CUtensorMap tm_s1, const __grid_constant__ QtArgs a) {
    using C = QT<NT>;
    constexpr int ND = C::ND, NB = C::NB, NW = C::NW, NS = C::NS, CW = C::CW;
    extern __shared__ __align__(1024) unsigned char qt_smem[];
    unsigned char* b_s = qt_smem;                        // [NB][3 planes][NT/2 tokens][128 bytes], 128-byte swizzle
    unsigned char* w_s = b_s + NB * C::B_BYTES;          // [NW][128 rows][128 bytes], 128-byte swizzle
    unsigned char* s_s = w_s + NW * C::W_BYTES;          // [NS][128 rows][4 scales]
    uint64_t* bars = reinterpret_cast<uint64_t*>(s_s + NS * C::S_BYTES);
    uint64_t* b_full = bars;              // NB, the leader's: both CTAs' activation bytes
    uint64_t* b_free = b_full + NB;       // NB, in both CTAs: the MMAs of the stage are done
    uint64_t* w_full = b_free + NB;       // NW, own
    uint64_t* w_free = w_full + NW;       // NW, own: 4 convert warps
    uint64_t* s_full = w_free + NW;       // NS, own
    uint64_t* s_free = s_full + NS;       // NS, own: 8 accumulating warps
    uint64_t* a_full = s_free + NS;       // ND, the leader's: 8 convert warps of both CTAs
    uint64_t* d_full = a_full + ND;       // ND, in both CTAs: block accumulated (and its A slot free again)
    uint64_t* d_free = d_full + ND;       // ND, the leader's: 16 accumulating warps of both CTAs
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(d_free + ND);

    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NB; ++i) {
            mbar_init(&b_full[i], 1);
            mbar_init(&b_free[i], 1);
        }
        for (int i = 0; i < NW; ++i) {
            mbar_init(&w_full[i], 1);
            mbar_init(&w_free[i], 4);
        }
        for (int i = 0; i < NS; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&s_free[i], C::ACC_WARPS);
        }
        for (int i = 0; i < ND; ++i) {
            mbar_init(&a_full[i], 8);
            mbar_init(&d_full[i], 1);
            mbar_init(&d_free[i], 2 * C::ACC_WARPS);
        }
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(C::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // both CTAs' barriers exist before either signals the other's
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // Work items (weight tile fastest, then token tile, then split of the contraction) are dealt round-robin to the
    // pairs; the rings and their phases run on from one item to the next.
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int items = a.n_tiles * a.t_tiles * a.splits;
    const int groups = a.K / 128;
    struct Item {
        int nt, t0, z, g0, g1;
    };
    auto item_of = [&](int w) {
        Item it;
        it.nt = w % a.n_tiles;
        const int r = w / a.n_tiles;
        it.t0 = (r % a.t_tiles) * NT;
        it.z = r / a.t_tiles;
        it.g0 = (int)((long long)groups * it.z / a.splits);
        it.g1 = (int)((long long)groups * (it.z + 1) / a.splits);
        return it;
    };

    if (warp >= 8) {
        if constexpr (C::REG_SPLIT) setmaxnreg_inc<96>();
        // ---------------- accumulate: one weight row and CW tokens per thread ----------------
        const int quad = warp & 3, cq = (warp - 8) >> 2;
        const int r = quad * 32 + lane;
        const uint32_t d_addr = tmem + ((uint32_t)(quad * 32) << 16) + cq * (C::STACK ? 3 * CW : CW);
        const uint32_t d_leader = map_to_cta(smem_u32(&d_free[0]), 0u);
        pdl_wait();   // the residual comes from the kernels ahead
        RingPos<NS> rs;
        RingPos<ND> rd;
        bool ok = true;
        for (int w = pair; ok && w < items; w += pairs) {
            const Item it = item_of(w);
            f32x2 acc[CW / 2], grp[CW / 2];
#pragma unroll
            for (int c = 0; c < CW / 2; ++c) acc[c] = grp[c] = 0ull;
            for (int g = it.g0; ok && g < it.g1; ++g) {
                if (!(ok = mbar_wait(&s_full[rs.slot], rs.parity, a.status, 79))) break;
                const float4 sc4 = *reinterpret_cast<const float4*>(s_s + rs.slot * C::S_BYTES + r * 16);
                __syncwarp();
                if (lane == 0) mbar_arrive(&s_free[rs.slot]);
                rs.next();
                const float sc[4] = {sc4.x, sc4.y, sc4.z, sc4.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (!(ok = mbar_wait(&d_full[rd.slot], rd.parity, a.status, 80))) break;
                    tc_fence_after();
                    const uint32_t da = d_addr + rd.slot * C::D_COLS;
                    const f32x2 s2 = qt_pack(sc[q], sc[q]);
                    auto handed_back = [&] {   // the accumulator's columns are in registers
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(d_leader + 8u * (uint32_t)rd.slot);
                    };
#pragma unroll
                    for (int h = 0; h < CW; h += C::HC) {
                        uint32_t v[C::HC];
                        tmem_ld<C::HC>(da + h, v);
                        if constexpr (C::STACK) {
                            uint32_t v1[C::HC], v2[C::HC];
                            tmem_ld<C::HC>(da + CW + h, v1);
                            tmem_ld<C::HC>(da + 2 * CW + h, v2);
                            tmem_wait_ld();
                            if (h + C::HC == CW) handed_back();
#pragma unroll
                            for (int c = 0; c < C::HC; c += 2) {
                                const f32x2 low = qt_add(qt_pack_bits(v2[c], v2[c + 1]), qt_pack_bits(v1[c], v1[c + 1]));
                                grp[(h + c) / 2] = qt_fma(qt_add(low, qt_pack_bits(v[c], v[c + 1])), s2, grp[(h + c) / 2]);
                            }
                        } else {
                            tmem_wait_ld();
                            if (h + C::HC == CW) handed_back();
#pragma unroll
                            for (int c = 0; c < C::HC; c += 2)
                                grp[(h + c) / 2] = qt_fma(qt_pack_bits(v[c], v[c + 1]), s2, grp[(h + c) / 2]);
                        }
                    }
                    rd.next();
                }
                if ((g + 1 - it.g0) % (C::GROUP / 4) == 0 || g + 1 == it.g1) {
#pragma unroll
                    for (int c = 0; c < CW / 2; ++c) {
                        if (!C::STACK && g + 1 == it.g1) grp[c] = qt_fma(qt_add(acc[c], grp[c]), qt_pack(TRUNCATED, TRUNCATED), grp[c]);
                        acc[c] = qt_add(acc[c], grp[c]);
                        grp[c] = 0ull;
                    }
                }
            }
            if (!ok) break;
            // this thread's weight row of the NT/2 tokens: lanes are consecutive columns of the output
            const bool second = it.nt >= a.n_tiles0;
            const int n = (it.nt - (second ? a.n_tiles0 : 0)) * 256 + (int)rank * C::ROWS + r;
            if (n < (second ? a.n[1] : a.n[0])) {
                const int col = (second ? a.n[0] : 0) + n;
                const OutColumn oc = out_column(a.out, col);
                const int pitch = oc.pitch;
                float* dst = oc.ptr + (size_t)it.z * a.out.split_stride + oc.col;
                const int t0 = it.t0 + cq * CW;
#pragma unroll
                for (int c0 = 0; c0 < CW; c0 += 4) {   // the loads of four tokens together, then their stores
                    float res[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int t = t0 + c0 + c;
                        res[c] = (a.out.residual != nullptr && t < a.M) ? __ldcg(a.out.residual + (size_t)t * pitch + col) : 0.0f;
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        float lo, hi;
                        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[(c0 + c) / 2]));
                        float v = (c & 1) ? hi : lo;
                        if (a.out.residual != nullptr) v = __fadd_rn(res[c], v);
                        if (t0 + c0 + c < a.M) dst[(size_t)(t0 + c0 + c) * pitch] = v;
                    }
                }
            }
        }
    } else {
        if constexpr (C::REG_SPLIT) setmaxnreg_dec<48>();
        if (warp == 0) {
            // ---------------- activation producer: this CTA's half of the tokens, reported to the leader ----------------
            if (lane == 0) {
                pdl_wait();               // the planes are the work of the kernels ahead
                pdl_launch_dependents();
                uint32_t s = 0;           // running stage number
                bool ok = true;
                for (int w = pair; ok && w < items; w += pairs) {
                    const Item it = item_of(w);
                    for (int g = 2 * it.g0; g < 2 * it.g1; ++g, ++s) {
                        const int st = s % NB;
                        if (s >= NB && !(ok = mbar_wait(&b_free[st], ((s / NB) - 1) & 1, a.status, 71))) break;
                        if (leader) mbar_arrive_expect_tx(&b_full[st], 2 * C::B_BYTES);
                        const uint32_t bar = map_to_cta(smem_u32(&b_full[st]), 0u);
#pragma unroll
                        for (int p = 0; p < 3; ++p)
                            tma_load_2d_pair(b_s + st * C::B_BYTES + p * C::PLANE_BYTES, &tm_x, g * 64,
                                             p * a.M + it.t0 + (int)rank * (NT / 2), bar);
                    }
                }
            }
        } else if (warp == 2) {
            // ---------------- weight and scale producer: constants, nothing to wait for but free slots ----------------
            if (lane == 0) {
                uint32_t s = 0;
                bool ok = true;
                for (int w = pair; ok && w < items; w += pairs) {
                    const Item it = item_of(w);
                    const bool second = it.nt >= a.n_tiles0;
                    const CUtensorMap* mw = second ? &tm_w1 : &tm_w0;
                    const CUtensorMap* ms = second ? &tm_s1 : &tm_s0;
                    const int row = (it.nt - (second ? a.n_tiles0 : 0)) * 256 + (int)rank * C::ROWS;
                    for (int g = it.g0; g < it.g1; ++g, ++s) {
                        const int ws = s % NW, ss = s % NS;
                        if (s >= NW && !(ok = mbar_wait(&w_free[ws], ((s / NW) - 1) & 1, a.status, 72))) break;
                        mbar_arrive_expect_tx(&w_full[ws], C::W_BYTES);
                        tma_load_2d(w_s + ws * C::W_BYTES, mw, g * 128, row, &w_full[ws]);
                        if (s >= NS && !(ok = mbar_wait(&s_free[ss], ((s / NS) - 1) & 1, a.status, 73))) break;
                        mbar_arrive_expect_tx(&s_full[ss], C::S_BYTES);
                        tma_load_2d(s_s + ss * C::S_BYTES, ms, g * 4, row, &s_full[ss]);
                    }
                }
            }
        } else if (warp == 1) {
            // ---------------- MMA issuer: one warp of the leader, for both CTAs ----------------
            if (leader) {
                constexpr uint32_t idesc = idesc_bf16(2 * C::ROWS, C::D_COLS);
                uint32_t stages = 0;      // of all this pair's items: the last ones are not handed back (nobody waits for them)
                for (int w = pair; w < items; w += pairs) {
                    const Item it = item_of(w);
                    stages += 2 * (it.g1 - it.g0);
                }
                const uint64_t desc0 = smem_desc_sw128(smem_u32(b_s), 16, 1024);
                RingPos<NB> rb;
                RingPos<ND> rd;
                bool ok = true, first_round = true;   // the first ND blocks find their accumulators free
                for (uint32_t s = 0; ok && s < stages; ++s) {
                    if (!(ok = mbar_wait(&b_full[rb.slot], rb.parity, a.status, 74))) break;
                    const uint64_t bd = desc0 + (uint64_t)((rb.slot * C::B_BYTES) >> 4);
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        if (!first_round && !(ok = mbar_wait(&d_free[rd.slot], rd.parity ^ 1u, a.status, 76))) break;
                        if (!(ok = mbar_wait(&a_full[rd.slot], rd.parity, a.status, 75))) break;
                        tc_fence_after();
                        const uint32_t d = tmem + rd.slot * C::D_COLS;
                        const uint32_t aw = tmem + C::TMEM_A + rd.slot * C::A_COLS;
                        if (elect_one()) {
                            constexpr int PASSES = C::STACK ? 1 : 3;
#pragma unroll
                            for (int p = PASSES - 1; p >= 0; --p)   // smallest plane first
#pragma unroll
                                for (int kk = 0; kk < 2; ++kk)
                                    mma_ts_bf16_pair(d, aw + kk * 8, bd + (uint64_t)((p * C::PLANE_BYTES + half * 64 + kk * 32) >> 4),
                                                     idesc, (p < PASSES - 1 || kk > 0) ? 1u : 0u);
                            if (half == 1 && s + NB < stages) tc_commit_both(&b_free[rb.slot]);
                            tc_commit_both(&d_full[rd.slot]);
                        }
                        __syncwarp();
                        rd.next();
                        if (rd.slot == 0) first_round = false;
                    }
                    rb.next();
                }
            }
        } else if (warp >= 4 && warp < 8) {
            // ---------------- convert: int8 -> pairs of bfloat16 in tensor memory, one weight row per thread ----------------
            const int quad = warp & 3;
            const int r = quad * 32 + lane;
            const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
            const uint32_t a_leader = map_to_cta(smem_u32(&a_full[0]), 0u);
            RingPos<NW> rw;
            RingPos<ND> rd;
            bool ok = true, first_round = true;
            for (int w = pair; ok && w < items; w += pairs) {
                const Item it = item_of(w);
                for (int g = it.g0; ok && g < it.g1; ++g) {
                    if (!(ok = mbar_wait(&w_full[rw.slot], rw.parity, a.status, 77))) break;
                    const unsigned char* row = w_s + rw.slot * C::W_BYTES + r * 128;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint4 c0 = *reinterpret_cast<const uint4*>(row + (((2 * q) ^ (r & 7)) << 4));
                        const uint4 c1 = *reinterpret_cast<const uint4*>(row + (((2 * q + 1) ^ (r & 7)) << 4));
                        if (q == 3) {
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&w_free[rw.slot]);
                        }
                        const uint32_t words[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
                        uint32_t out[16];
                        // the low seven bits in the significand of a bfloat16 of 128 .. 255, minus 128 or, with the sign bit, 256: exact
#pragma unroll
                        for (int k = 0; k < 16; ++k) {
                            const uint32_t u = __byte_perm(words[k >> 1], 0x43434343u, (k & 1) ? 0x4342 : 0x4140);
                            asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(out[k]) : "r"(u & 0xff7fff7fu), "r"(u & 0xff80ff80u));
                        }
                        if (!first_round && !(ok = mbar_wait(&d_full[rd.slot], rd.parity ^ 1u, a.status, 78))) break;
                        tc_fence_after();
                        tmem_st16(tmem + lane_addr + C::TMEM_A + rd.slot * C::A_COLS, out);
                        tmem_wait_st();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(a_leader + 8u * (uint32_t)rd.slot);
                        rd.next();
                        if (rd.slot == 0) first_round = false;
                    }
                    rw.next();
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // neither CTA leaves while its shared and tensor memory may still be operands of the pair's MMAs
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TMEM_COLS) : "memory");
    }
}

// x as three bfloat16 whose sum is x exactly (Inf and NaN stay in the first).
__device__ __forceinline__ void split3(float x, unsigned short (&p)[3]) {
    uint32_t b = __float_as_uint(x);
    if ((b & 0x7f800000u) == 0x7f800000u) {
        p[0] = (unsigned short)((b & 0x007fffffu) ? 0x7fc0u : (b >> 16));
        p[1] = p[2] = 0;
        return;
    }
    const float hi = __uint_as_float(b & 0xffff0000u);
    const float r1 = __fsub_rn(x, hi);
    const uint32_t b1 = __float_as_uint(r1);
    const float r2 = __fsub_rn(r1, __uint_as_float(b1 & 0xffff0000u));
    p[0] = (unsigned short)(b >> 16);
    p[1] = (unsigned short)(b1 >> 16);
    p[2] = (unsigned short)(__float_as_uint(r2) >> 16);
}

__device__ __forceinline__ void store_planes(__nv_bfloat16* planes, size_t plane_elems, size_t at, const float4& v) {
    unsigned short p[4][3];
    split3(v.x, p[0]);
    split3(v.y, p[1]);
    split3(v.z, p[2]);
    split3(v.w, p[3]);
#pragma unroll
    for (int k = 0; k < 3; ++k)
        *reinterpret_cast<uint2*>(planes + k * plane_elems + at) =
            make_uint2((uint32_t)p[0][k] | (uint32_t)p[1][k] << 16, (uint32_t)p[2][k] | (uint32_t)p[3][k] << 16);
}

constexpr int ROW_THREADS = 256;

// One CTA per token row: [sum of the splits of the projection ahead + residual -> h], RMSNorm, bfloat16 planes.
// Memory-bound (4 bytes read, 6 written per element beside the partials).
__global__ void __launch_bounds__(ROW_THREADS) q8_rows_kernel(Q8RowsArgs a) {
    extern __shared__ __align__(16) float4 row_s[];   // the row, when it is needed twice (norm)
    __shared__ double red[ROW_THREADS / 32];
    const int m = blockIdx.x, n4 = a.K >> 2;
    const size_t base = (size_t)m * a.K;
    const float4* gam = reinterpret_cast<const float4*>(a.gamma);
    pdl_wait();
    pdl_launch_dependents();
    double sq = 0.0;
    for (int d = threadIdx.x; d < n4; d += ROW_THREADS) {
        float4 v = __ldcg(reinterpret_cast<const float4*>(a.x + base) + d);
        if (a.splits > 0) {
            for (int z = 1; z < a.splits; ++z) {
                const float4 p = __ldcg(reinterpret_cast<const float4*>(a.x + z * a.split_stride + base) + d);
                v = make_float4(v.x + p.x, v.y + p.y, v.z + p.z, v.w + p.w);
            }
            if (a.residual != nullptr) {
                const float4 p = __ldcg(reinterpret_cast<const float4*>(a.residual + base) + d);
                v = make_float4(__fadd_rn(p.x, v.x), __fadd_rn(p.y, v.y), __fadd_rn(p.z, v.z), __fadd_rn(p.w, v.w));
            }
            if (a.h != nullptr) reinterpret_cast<float4*>(a.h + base)[d] = v;
        }
        if (a.gamma == nullptr) {
            store_planes(a.planes, (size_t)a.M * a.K, base + 4 * d, v);
        } else {
            row_s[d] = v;
            sq += (double)v.x * (double)v.x + (double)v.y * (double)v.y + (double)v.z * (double)v.z + (double)v.w * (double)v.w;
        }
    }
    if (a.gamma == nullptr) return;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
    __syncthreads();
    double tot = 0.0;
#pragma unroll
    for (int w = 0; w < ROW_THREADS / 32; ++w) tot += red[w];
    // rms_norm.cr:29-32, as the single-row kernels do it: f64 sum, scaling and weight, one rounding to fp32
    const double inv_rms = rsqrt(tot / (double)a.K + a.eps);
    for (int d = threadIdx.x; d < n4; d += ROW_THREADS) {
        float4 v = row_s[d];
        const float4 g = __ldg(gam + d);
        v.x = (float)(((double)v.x * inv_rms) * (double)g.x);
        v.y = (float)(((double)v.y * inv_rms) * (double)g.y);
        v.z = (float)(((double)v.z * inv_rms) * (double)g.z);
        v.w = (float)(((double)v.w * inv_rms) * (double)g.w);
        store_planes(a.planes, (size_t)a.M * a.K, base + 4 * d, v);
    }
}

// hidden = silu(gate) * up in f64 (swiglu_ff.cr:83-88), rounded to fp32 once, as planes.  `gu`: [splits][M][2 ffn].  `parts` CTAs
// per token row, so that a few rows still use many SMs.  Bound by the f64 exponentials.
__global__ void __launch_bounds__(ROW_THREADS) q8_swiglu_kernel(const float* gu, int splits, size_t split_stride, int M, int ffn, int parts,
                                                                __nv_bfloat16* planes) {
    const int m = blockIdx.x / parts, part = blockIdx.x - m * parts;
    const int n4 = ffn >> 2, per = (n4 + parts - 1) / parts;
    const int d0 = min(n4, part * per), d1 = min(n4, d0 + per);
    pdl_wait();
    pdl_launch_dependents();
    auto act = [](float gf, float uf) {
        const double gd = (double)gf;
        return (float)((gd / (1.0 + exp(-gd))) * (double)uf);
    };
    for (int d = d0 + threadIdx.x; d < d1; d += ROW_THREADS) {
        const float* g = gu + (size_t)m * 2 * ffn + 4 * d;
        float4 gv = __ldcg(reinterpret_cast<const float4*>(g)), uv = __ldcg(reinterpret_cast<const float4*>(g + ffn));
        for (int z = 1; z < splits; ++z) {
            const float4 p = __ldcg(reinterpret_cast<const float4*>(g + z * split_stride));
            const float4 q = __ldcg(reinterpret_cast<const float4*>(g + z * split_stride + ffn));
            gv = make_float4(gv.x + p.x, gv.y + p.y, gv.z + p.z, gv.w + p.w);
            uv = make_float4(uv.x + q.x, uv.y + q.y, uv.z + q.z, uv.w + q.w);
        }
        store_planes(planes, (size_t)M * ffn, (size_t)m * ffn + 4 * d,
                     make_float4(act(gv.x, uv.x), act(gv.y, uv.y), act(gv.z, uv.z), act(gv.w, uv.w)));
    }
}

// Sum of the splits into the (up to three) outputs of a launch without a norm behind it.
__global__ void __launch_bounds__(256) q8_reduce_kernel(const float* part, int splits, size_t split_stride, int M, int N, Q8GemmOut out) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t total = (size_t)M * N;
    for (size_t e = (size_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (size_t)gridDim.x * 256) {
        const size_t m = e / N;
        const int col = (int)(e - m * N);
        float v = __ldcg(part + e);
        for (int z = 1; z < splits; ++z) v += __ldcg(part + z * split_stride + e);
        const OutColumn oc = out_column(out, col);
        const size_t at = m * oc.pitch + oc.col;
        if (out.residual != nullptr) v = __fadd_rn(__ldcg(out.residual + at), v);
        oc.ptr[at] = v;
    }
}

template <class... P, class... A>
cudaError_t launch_chain(void (*kernel)(P...), dim3 grid, int threads, size_t smem, int cluster, cudaStream_t s, const A&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <class K>
cudaError_t allow_smem(K kernel, size_t bytes, std::atomic<unsigned long long>& configured) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 64 || !(configured.load(std::memory_order_acquire) >> dev & 1ull)) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return e;
        if (dev < 64) configured.fetch_or(1ull << dev, std::memory_order_release);
    }
    return cudaSuccess;
}

template <int NT>
cudaError_t launch_nt(const Q8GemmArgs& g, const QtArgs& a, const CUtensorMap& tx, int grid, cudaStream_t s) {
    static std::atomic<unsigned long long> configured{0};
    cudaError_t e = allow_smem(q8_gemm_tc_kernel<NT>, QT<NT>::SMEM_BYTES, configured);
    if (e != cudaSuccess) return e;
    const Q8Maps& w1 = g.w[1] ? *g.w[1] : *g.w[0];
    return launch_chain(q8_gemm_tc_kernel<NT>, dim3(grid), QT<NT>::THREADS, QT<NT>::SMEM_BYTES, 2, s, tx, g.w[0]->w, g.w[0]->s, w1.w,
                        w1.s, a);
}

int token_tile(int M, int cap) {
    int nt = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
    return nt < cap ? nt : cap;
}

// What one 32-input block of a pair's tile takes, us: at every width the issue slots of the convert and accumulating
// warps first (fitted, with the constants of the plan, to 660 timed products of 512 to 9216 inputs, 2048 to 16384 outputs
// and 8 to 4096 tokens, tiles and splits varied; the plan is on average 0.4 % slower than the best of them).
double block_us(int nt) { return nt >= 128 ? 0.43 : nt >= 64 ? 0.32 : nt >= 32 ? 0.29 : 0.27; }

}  // namespace

bool q8_gemm_maps(Q8Maps* m, const signed char* q, const float* scales, int N, int K) {
    m->ok = false;
    if (K <= 0 || K % 128 != 0 || N <= 0 || ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(scales)) & 15u) != 0) return false;
    m->ok = make_map_2d(&m->w, CU_TENSOR_MAP_DATA_TYPE_UINT8, q, K, N, K, 128, 128, CU_TENSOR_MAP_SWIZZLE_128B) &&
            make_map_2d(&m->s, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, scales, K / 32, N, (uint64_t)K / 8, 4, 128, CU_TENSOR_MAP_SWIZZLE_NONE);
    m->N = N;
    m->K = K;
    return m->ok;
}

Q8GemmPlan q8_gemm_plan(int M, int K, int n0, int n1, int sm_count) {
    Q8GemmPlan best{};
    double best_t = 1e300;
    const int pairs = std::max(1, sm_count / 2), groups = K / 128;
    const int n_tiles = (n0 + 255) / 256 + (n1 + 255) / 256;
    for (int nt : {token_tile(M, 128), token_tile(M, 64)}) {
        const int t_tiles = (M + nt - 1) / nt;
        const long long tiles = (long long)n_tiles * t_tiles;
        for (int z = 1; z <= std::min(groups, 16); ++z) {
            const double waves = (double)((tiles * z + pairs - 1) / pairs);
            // an item's blocks, its start-up and its stores; then the splits written and read back
            const double t = waves * (std::ceil((double)groups / z) * 4 * block_us(nt) + 0.9) +
                             (z > 1 ? 2.5 + 0.63e-6 * z * (double)M * (n0 + n1) * 4 : 0.0);
            if (t < best_t) {
                best_t = t;
                best = Q8GemmPlan{nt, z};
            }
        }
    }
    return best;
}

cudaError_t launch_q8_gemm_tc(const Q8GemmArgs& g, const Q8GemmPlan& plan, int sm_count, cudaStream_t s) {
    if (g.M <= 0) return cudaSuccess;
    if (!g.w[0] || !g.w[0]->ok || g.w[0]->K != g.K || (g.w[1] && (!g.w[1]->ok || g.w[1]->K != g.K))) return cudaErrorInvalidValue;
    QtArgs a{};
    a.M = g.M;
    a.K = g.K;
    a.n[0] = g.w[0]->N;
    a.n[1] = g.w[1] ? g.w[1]->N : 0;
    a.n_tiles0 = (a.n[0] + 255) / 256;
    a.n_tiles = a.n_tiles0 + (a.n[1] + 255) / 256;
    a.t_tiles = (g.M + plan.nt - 1) / plan.nt;
    a.splits = plan.splits;
    a.out = g.out;
    a.status = g.status;
    CUtensorMap tx;
    if (!make_map_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, g.planes, g.K, 3ull * g.M, 2ull * g.K, 64, plan.nt / 2, CU_TENSOR_MAP_SWIZZLE_128B))
        return cudaErrorInvalidValue;
    const long long items = (long long)a.n_tiles * a.t_tiles * a.splits;
    if (items > 0x7fffffff) return cudaErrorInvalidValue;
    const int grid = 2 * (int)std::min<long long>(items, std::max(1, sm_count / 2));
    switch (plan.nt) {
        case 128: return launch_nt<128>(g, a, tx, grid, s);
        case 64: return launch_nt<64>(g, a, tx, grid, s);
        case 32: return launch_nt<32>(g, a, tx, grid, s);
        case 16: return launch_nt<16>(g, a, tx, grid, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_q8_rows(const Q8RowsArgs& a, cudaStream_t s) {
    if (a.M <= 0) return cudaSuccess;
    if (a.K % 4 != 0) return cudaErrorInvalidValue;
    const size_t smem = a.gamma ? (size_t)a.K * 4 : 0;   // the row is needed twice
    if (smem > 200 * 1024) return cudaErrorInvalidValue;
    if (smem > 40 * 1024) {
        static std::atomic<unsigned long long> configured{0};
        cudaError_t e = allow_smem(q8_rows_kernel, 200 * 1024, configured);
        if (e != cudaSuccess) return e;
    }
    return launch_chain(q8_rows_kernel, dim3(a.M), ROW_THREADS, smem, 1, s, a);
}

cudaError_t launch_q8_swiglu(const float* gu, int splits, size_t split_stride, int M, int ffn, __nv_bfloat16* planes, int sm_count, cudaStream_t s) {
    if (M <= 0) return cudaSuccess;
    if (ffn % 4 != 0) return cudaErrorInvalidValue;
    int parts = 1;   // as many as it takes to give every SM two CTAs
    while (parts < 8 && (long long)M * parts < 2ll * sm_count) parts *= 2;
    return launch_chain(q8_swiglu_kernel, dim3((unsigned)(M * parts)), ROW_THREADS, 0, 1, s, gu, splits, split_stride, M, ffn, parts, planes);
}

cudaError_t launch_q8_reduce(const float* part, int splits, size_t split_stride, int M, int N, const Q8GemmOut& out, cudaStream_t s) {
    if (M <= 0) return cudaSuccess;
    const size_t blocks = std::min<size_t>(((size_t)M * N + 255) / 256, 148 * 8);
    return launch_chain(q8_reduce_kernel, dim3((unsigned)blocks), 256, 0, 1, s, part, splits, split_stride, M, N, out);
}

}  // namespace shainet
