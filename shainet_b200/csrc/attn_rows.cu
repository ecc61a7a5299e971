// fp32 attention of a few query rows over the KV cache, CUDA cores, sm_100a: 2 to 63 new tokens of a sequence (a drafted
// continuation to verify, a short prompt), and single tokens whose query heads per kv head the decode kernel does not
// serve well.
//
// Same contract as the reference's attention_kv_kernel (src/shainet/native/cuda_kernels.cu:734-806) and the same fp32
// arithmetic as the decode kernel (no tensor core: its TF32 operands would lose bits these calls have).  All T x G query
// rows that share a kv head - G = query heads per kv head, row = t * G + g - are one tile, so a cache row is fetched once
// for all of them; a CTA takes BM = 64, 32 or 16 such rows and one slice of the positions (split-K), in tiles of 64
// positions fetched by bulk copies (TMA engine; K row by row into padded rows, V as one block).
//
// Bound: the fp32 pipe (2 * 64 * BM * head_dim multiply-adds per tile, packed as fma.rn.f32x2).  S = Q K^T is a register
// tile of 4 rows x 4 positions per thread (2 or 1 positions where the CTA has 32 or 16 rows: its eight warps then also
// divide the positions, each with its own running softmax, merged at the end); 16 lanes share a row, so maxima are four
// shuffles, and the probabilities go to P V through a strip of shared memory that only their own warp touches.
// Measured, 40 tokens over 1900 positions of the LLaMA-3.2-1B shape: 37 us per layer with norm/RoPE/append and merge, one
// CTA per (head, token) streaming the cache 490 us; 5 tokens over 4096 of the Qwen3-8B shape: 29 us, one decode CTA
// set per token 41 us.
#include <cuda_bf16.h>
#include <math.h>
#include <algorithm>
#include <atomic>
#include <type_traits>
#include "kernels.h"

namespace shainet {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr float LOG2E = 1.4426950408889634f;

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 ar_pack(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void ar_unpack(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 ar_fma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 ar_mul(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Four consecutive cache elements as two packed pairs (a bfloat16 is the upper half of the fp32 of the same value).
template <int ES>
__device__ __forceinline__ ulonglong2 four(const unsigned char* p) {
    if constexpr (ES == 4) {
        return *reinterpret_cast<const ulonglong2*>(p);
    } else {
        const uint2 w = *reinterpret_cast<const uint2*>(p);
        ulonglong2 r;
        asm("mov.b64 %0, {%1, %2};" : "=l"(r.x) : "r"(w.x << 16), "r"(w.x & 0xffff0000u));
        asm("mov.b64 %0, {%1, %2};" : "=l"(r.y) : "r"(w.y << 16), "r"(w.y & 0xffff0000u));
        return r;
    }
}

template <int HD_, int BM_, int ES_>
struct AR {
    static constexpr int HD = HD_, BM = BM_, ES = ES_;
    static constexpr int BN = 64;                     // positions per tile
    static constexpr int WARPS = 8;
    static constexpr int WR = BM / 8;                 // warps along the rows (8 rows each)
    static constexpr int WK = WARPS / WR;             // warps along the positions
    static constexpr int KW = BN / WK;                // positions of a warp
    static constexpr int KT = KW / 16;                // positions of a thread
    static constexpr int CT = HD / 64;                // 16-byte column chunks of a thread's output
    static constexpr int THREADS = (WARPS + 1) * 32;
    static constexpr int Q_STRIDE = HD + 4;           // floats
    static constexpr int K_STRIDE = HD * ES + 16;     // bytes: lanes on consecutive rows hit different banks
    static constexpr int K_BYTES = BN * K_STRIDE;
    static constexpr int V_BYTES = BN * HD * ES;
    static constexpr int STAGE = K_BYTES + V_BYTES;
    static constexpr int P_STRIDE = KW + 4;           // floats
    static constexpr int FIXED = BM * Q_STRIDE * 4 + WARPS * 8 * P_STRIDE * 4 + 128;
    static constexpr int NS = 2;
    static constexpr size_t SMEM = (size_t)FIXED + (size_t)NS * STAGE;
    static constexpr int CTAS = SMEM <= 110 * 1024 ? 2 : 1;
    static_assert((size_t)WARPS * (8 * HD + 16) * 4 <= (size_t)NS * STAGE, "merge area");
};

struct RowArgs {
    AttnArgs a;
    int groups;      // query heads per kv head
    int row_blocks;  // BM-row tiles per (sequence, kv head)
};

template <int HD, int BM, int ES>
__global__ void __launch_bounds__(AR<HD, BM, ES>::THREADS, AR<HD, BM, ES>::CTAS) attn_rows_kernel(RowArgs ra) {
    using C = AR<HD, BM, ES>;
    const AttnArgs& a = ra.a;
    extern __shared__ __align__(128) unsigned char ar_smem[];
    unsigned char* stages = ar_smem;                                            // [NS][K padded | V]
    float* qs = reinterpret_cast<float*>(ar_smem + (size_t)C::NS * C::STAGE);   // [BM][Q_STRIDE]
    float* ps = qs + BM * C::Q_STRIDE;                                          // [WARPS][8][P_STRIDE]
    uint64_t* full = reinterpret_cast<uint64_t*>(ps + C::WARPS * 8 * C::P_STRIDE);
    uint64_t* empty = full + C::NS;

    const int split = blockIdx.x, kv_h = blockIdx.y;
    const int b = blockIdx.z / ra.row_blocks, rb = blockIdx.z - b * ra.row_blocks;
    const int G = ra.groups, R = a.T * G, H = a.hs.num_heads;
    const SeqDesc sd = a.seqs.many ? a.seqs.many[b] : a.seqs.one;
    const int r0 = rb * BM, rn = min(BM, R - r0);          // this tile's rows
    const int visible = sd.start + (r0 + rn - 1) / G + 1;  // of its last token
    const int nsplit = (sd.start + a.T + a.chunk_rows - 1) / a.chunk_rows;
    if (split >= nsplit) return;
    const int k0 = split * a.chunk_rows, k1 = min(k0 + a.chunk_rows, visible);
    const int ntiles = k1 > k0 ? (k1 - k0 + C::BN - 1) / C::BN : 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::NS; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], C::WARPS);
        }
        fence_mbar_init();
    }
    __syncthreads();

    const int wr = warp % C::WR, wk = warp / C::WR;
    const int ty = lane >> 4, tx = lane & 15;
    const int row = wr * 8 + ty * 4;                       // this thread's four rows
    f32x2 o[4][C::CT * 2];
    float m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.0f;
#pragma unroll
        for (int c = 0; c < C::CT * 2; ++c) o[i][c] = 0ull;
    }
    if (warp == C::WARPS) {
        // ---------------- producer ----------------
        const size_t base = ((size_t)kv_h * sd.capacity + k0) * HD * ES;
        const unsigned char* kb = reinterpret_cast<const unsigned char*>(sd.k) + base;
        const unsigned char* vb = reinterpret_cast<const unsigned char*>(sd.v) + base;
        bool waited = false;
        for (int t = 0; t < ntiles; ++t) {
            const int s = t % C::NS;
            if (t >= C::NS && !mbar_wait(&empty[s], ((t / C::NS) - 1) & 1, a.status, 91)) break;
            const int n = min(C::BN, k1 - k0 - t * C::BN);
            // the kernel ahead in the stream writes the rows from `start` on; older ones may be fetched while it runs
            if (!waited && k0 + t * C::BN + n > sd.start) {
                asm volatile("griddepcontrol.wait;" ::: "memory");
                waited = true;
            }
            unsigned char* st = stages + (size_t)s * C::STAGE;
            if (lane == 0) mbar_arrive_expect_tx(&full[s], (uint32_t)(2 * n * HD * ES));
            __syncwarp();
            for (int i = lane; i < n; i += 32)
                bulk_g2s(st + i * C::K_STRIDE, kb + (size_t)(t * C::BN + i) * HD * ES, HD * ES, &full[s]);
            if (lane == 0) bulk_g2s(st + C::K_BYTES, vb + (size_t)t * C::BN * HD * ES, (uint32_t)(n * HD * ES), &full[s]);
        }
        if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    } else {
        // ---------------- consumers ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");   // the rotated q rows are the work of the kernel ahead
        for (int i = threadIdx.x; i < BM * (HD / 4); i += C::WARPS * 32) {
            const int rr = i / (HD / 4), c = i - rr * (HD / 4);
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (rr < rn) {
                const int t = (r0 + rr) / G, g = (r0 + rr) - t * G;
                v = __ldcg(reinterpret_cast<const float4*>(a.q_rot + (((size_t)b * a.T + t) * H + (size_t)kv_h * G + g) * HD) + c);
            }
            *reinterpret_cast<float4*>(qs + rr * C::Q_STRIDE + c * 4) = v;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(C::WARPS * 32) : "memory");
        int last[4];   // last position each of the four rows sees
#pragma unroll
        for (int i = 0; i < 4; ++i) last[i] = sd.start + (r0 + min(row + i, rn - 1)) / G;
        float* pw = ps + warp * 8 * C::P_STRIDE;
        for (int t = 0; t < ntiles; ++t) {
            const int s = t % C::NS;
            if (!mbar_wait(&full[s], (t / C::NS) & 1, a.status, 92)) break;
            const unsigned char* ks = stages + (size_t)s * C::STAGE + (wk * C::KW + tx) * C::K_STRIDE;
            const unsigned char* vs = stages + (size_t)s * C::STAGE + C::K_BYTES + (size_t)wk * C::KW * HD * ES;
            f32x2 acc[4][C::KT];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < C::KT; ++j) acc[i][j] = 0ull;
#pragma unroll 4
            for (int d = 0; d < HD; d += 4) {
                ulonglong2 qv[4], kv[C::KT];
#pragma unroll
                for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const ulonglong2*>(qs + (row + i) * C::Q_STRIDE + d);
#pragma unroll
                for (int j = 0; j < C::KT; ++j) kv[j] = four<ES>(ks + j * 16 * C::K_STRIDE + d * ES);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < C::KT; ++j) {
                        acc[i][j] = ar_fma(qv[i].x, kv[j].x, acc[i][j]);
                        acc[i][j] = ar_fma(qv[i].y, kv[j].y, acc[i][j]);
                    }
            }
            // running softmax: 16 lanes share a row
            const int key0 = k0 + t * C::BN + wk * C::KW + tx;
            const bool edge = k0 + (t + 1) * C::BN > sd.start + 1 || (t + 1) * C::BN > k1 - k0;   // some row does not see the whole tile
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float sc[C::KT], mx = -INFINITY;
#pragma unroll
                for (int j = 0; j < C::KT; ++j) {
                    float lo, hi;
                    ar_unpack(acc[i][j], lo, hi);
                    sc[j] = (lo + hi) * a.scale;
                    if (edge && (key0 + 16 * j > last[i] || key0 + 16 * j >= k1)) sc[j] = -INFINITY;
                    mx = fmaxf(mx, sc[j]);
                }
#pragma unroll
                for (int off = 8; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(FULL, mx, off));
                const float m_new = fmaxf(m[i], mx);
                const float m_use = m_new == -INFINITY ? 0.0f : m_new;   // nothing visible yet: every term is 0
                const float alpha = exp2f((m[i] - m_use) * LOG2E);
                m[i] = m_new;
                l[i] *= alpha;
                const f32x2 al = ar_pack(alpha, alpha);
#pragma unroll
                for (int c = 0; c < C::CT * 2; ++c) o[i][c] = ar_mul(o[i][c], al);
#pragma unroll
                for (int j = 0; j < C::KT; ++j) {
                    const float p = exp2f((sc[j] - m_use) * LOG2E);
                    l[i] += p;
                    pw[(ty * 4 + i) * C::P_STRIDE + tx + 16 * j] = p;
                }
            }
            __syncwarp();
            // O += P V, four positions at a time.  In an edge tile a row stops at the last position it sees: what lies behind is the V
            // row of a later token, or of an earlier tile where this one is short, and zero times an infinity would be NaN.
            // Only the few positions that some of the warp's eight rows see and others do not are checked row by row.
            int kfull = C::KW, kend = C::KW, seen[4];   // positions of this warp's strip that all its rows, that any of them, that a row sees
            if (edge) {
#pragma unroll
                for (int i = 0; i < 4; ++i) seen[i] = min(C::KW, min(last[i] + 1, k1) - (k0 + t * C::BN + wk * C::KW));
                kfull = max(0, __shfl_sync(FULL, seen[0], 0)) & ~3;
                kend = __shfl_sync(FULL, seen[3], 31);
            }
            auto pv = [&](int k, auto checked) {
                float4 p4[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) p4[i] = *reinterpret_cast<const float4*>(pw + (ty * 4 + i) * C::P_STRIDE + k);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    ulonglong2 vv[C::CT];
#pragma unroll
                    for (int c = 0; c < C::CT; ++c) vv[c] = four<ES>(vs + ((size_t)(k + kk) * HD + c * 64 + tx * 4) * ES);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (decltype(checked)::value && k + kk >= seen[i]) continue;
                        const float p = kk == 0 ? p4[i].x : kk == 1 ? p4[i].y : kk == 2 ? p4[i].z : p4[i].w;
                        const f32x2 pp = ar_pack(p, p);
#pragma unroll
                        for (int c = 0; c < C::CT; ++c) {
                            o[i][2 * c] = ar_fma(pp, vv[c].x, o[i][2 * c]);
                            o[i][2 * c + 1] = ar_fma(pp, vv[c].y, o[i][2 * c + 1]);
                        }
                    }
                }
            };
            if (!edge) {
#pragma unroll 2
                for (int k = 0; k < C::KW; k += 4) pv(k, std::false_type{});
            } else {
#pragma unroll 2
                for (int k = 0; k < kfull; k += 4) pv(k, std::false_type{});
#pragma unroll 1
                for (int k = kfull; k < kend; k += 4) pv(k, std::true_type{});
            }
            __syncwarp();   // the strip is rewritten in the next tile
            if (lane == 0) mbar_arrive(&empty[s]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) l[i] += __shfl_xor_sync(FULL, l[i], off);
    }
    __syncthreads();   // every copy has landed and been used: the stages are free
    // Merge of the WK warps of a row through shared memory: [warp][8 rows][HD] and [warp][8] maxima and sums.
    float* mo = reinterpret_cast<float*>(stages);
    float* mm = mo + C::WARPS * 8 * HD;
    if (warp < C::WARPS) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int rr = warp * 8 + ty * 4 + i;
#pragma unroll
            for (int c = 0; c < C::CT; ++c)
                *reinterpret_cast<ulonglong2*>(mo + (size_t)rr * HD + c * 64 + tx * 4) = make_ulonglong2(o[i][2 * c], o[i][2 * c + 1]);
            if (tx == 0) {
                mm[rr * 2] = m[i];
                mm[rr * 2 + 1] = l[i];
            }
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < rn * (HD / 4); e += C::THREADS) {
        const int rr = e / (HD / 4), c = e - rr * (HD / 4);
        float M = -INFINITY, L = 0.0f;
#pragma unroll
        for (int k = 0; k < C::WK; ++k) M = fmaxf(M, mm[((k * C::WR + (rr >> 3)) * 8 + (rr & 7)) * 2]);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < C::WK; ++k) {
            const int at = (k * C::WR + (rr >> 3)) * 8 + (rr & 7);
            const float w = mm[at * 2] == -INFINITY ? 0.0f : exp2f((mm[at * 2] - M) * LOG2E);
            const float4 v = *reinterpret_cast<const float4*>(mo + (size_t)at * HD + c * 4);
            L = fmaf(w, mm[at * 2 + 1], L);
            acc = make_float4(fmaf(w, v.x, acc.x), fmaf(w, v.y, acc.y), fmaf(w, v.z, acc.z), fmaf(w, v.w, acc.w));
        }
        const int t = (r0 + rr) / G, g = (r0 + rr) - t * G;
        const size_t hrow = ((size_t)b * a.T + t) * H + (size_t)kv_h * G + g;
        if (nsplit == 1) {
            *reinterpret_cast<float4*>(a.out + hrow * HD + c * 4) = make_float4(acc.x / L, acc.y / L, acc.z / L, acc.w / L);
        } else {
            const size_t pidx = hrow * a.max_splits + split;
            *reinterpret_cast<float4*>(a.part_o + pidx * HD + c * 4) = acc;
            if (c == 0) *reinterpret_cast<float2*>(a.part_ml + pidx * 2) = make_float2(M, L);
        }
    }
}

// out = sum_s w_s o_s / sum_s w_s l_s over the splits, one warp per (row, query head): the weights are formed by the
// lanes side by side, HD/4 lanes walk the partials with eight to sixteen loads in flight.
constexpr int CB_WARPS = 4;
template <int HD>
__global__ void __launch_bounds__(CB_WARPS * 32) attn_rows_combine_kernel(AttnArgs a) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t hrow = (size_t)blockIdx.x * CB_WARPS + warp;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (hrow >= (size_t)a.batch * a.T * a.hs.num_heads) return;
    const int b = (int)(hrow / ((size_t)a.T * a.hs.num_heads));
    const SeqDesc sd = a.seqs.many ? a.seqs.many[b] : a.seqs.one;
    const int ns = (sd.start + a.T + a.chunk_rows - 1) / a.chunk_rows;
    if (ns <= 1) return;   // the split kernel wrote the row
    const float2* ml = reinterpret_cast<const float2*>(a.part_ml) + hrow * a.max_splits;
    const float* po = a.part_o + hrow * a.max_splits * HD;
    const bool on = lane < HD / 4;
    auto partial = [&](int sp) {
        return (on && sp < ns) ? __ldcg(reinterpret_cast<const float4*>(po + (size_t)sp * HD) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    // the first partials are requested together with the maxima that weigh them
    float4 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = partial(k);
    const float2 first = lane < ns ? __ldcg(ml + lane) : make_float2(-INFINITY, 0.0f);
    float M = first.x;
    for (int s = 32 + lane; s < ns; s += 32) M = fmaxf(M, __ldcg(ml + s).x);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(FULL, M, off));
    float L = 0.0f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s0 = 0; s0 < ns; s0 += 32) {
        float w = 0.0f;
        if (s0 + lane < ns) {
            const float2 p = s0 == 0 ? first : __ldcg(ml + s0 + lane);
            w = p.x == -INFINITY ? 0.0f : exp2f((p.x - M) * LOG2E);
            L = fmaf(w, p.y, L);
        }
        const int n = min(32, ns - s0);
        for (int s1 = 0; s1 < n; s1 += 8) {
            float4 nxt[8];   // the next eight, while these are added
#pragma unroll
            for (int k = 0; k < 8; ++k) nxt[k] = partial(s0 + s1 + 8 + k);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float wk = __shfl_sync(FULL, w, s1 + k);   // zero past the last split
                acc = make_float4(fmaf(wk, v[k].x, acc.x), fmaf(wk, v[k].y, acc.y), fmaf(wk, v[k].z, acc.z), fmaf(wk, v[k].w, acc.w));
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = nxt[k];
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) L += __shfl_xor_sync(FULL, L, off);
    if (on)
        *(reinterpret_cast<float4*>(a.out + hrow * HD) + lane) = make_float4(acc.x / L, acc.y / L, acc.z / L, acc.w / L);
}

template <class K, class... A>
cudaError_t launch_pdl_any(K kernel, dim3 grid, int threads, size_t smem, cudaStream_t s, const A&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <int HD, int BM, int ES>
cudaError_t launch_rows(const AttnArgs& a, cudaStream_t s) {
    using C = AR<HD, BM, ES>;
    static std::atomic<unsigned long long> configured{0};   // bit per device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 64 || !(configured.load(std::memory_order_acquire) >> dev & 1ull)) {
        e = cudaFuncSetAttribute(attn_rows_kernel<HD, BM, ES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
        if (e != cudaSuccess) return e;
        if (dev < 64) configured.fetch_or(1ull << dev, std::memory_order_release);
    }
    RowArgs ra{};
    ra.a = a;
    ra.groups = a.hs.num_heads / a.hs.num_kv_heads;
    ra.row_blocks = (a.T * ra.groups + BM - 1) / BM;
    e = launch_pdl_any(attn_rows_kernel<HD, BM, ES>, dim3(a.max_splits, a.hs.num_kv_heads, a.batch * ra.row_blocks), C::THREADS, C::SMEM, s, ra);
    if (e != cudaSuccess || a.max_splits <= 1) return e;
    const long long hrows = (long long)a.batch * a.T * a.hs.num_heads;
    return launch_pdl_any(attn_rows_combine_kernel<HD>, dim3((unsigned)((hrows + CB_WARPS - 1) / CB_WARPS)), CB_WARPS * 32, 0, s, a);
}

template <int HD, int ES>
cudaError_t launch_rows_bm(const AttnArgs& a, int bm, cudaStream_t s) {
    switch (bm) {
        case 64: return launch_rows<HD, 64, ES>(a, s);
        case 32: return launch_rows<HD, 32, ES>(a, s);
        case 16: return launch_rows<HD, 16, ES>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

template <int HD, int ES>
int rows_ctas(int bm) {
    return bm == 64 ? AR<HD, 64, ES>::CTAS : bm == 32 ? AR<HD, 32, ES>::CTAS : AR<HD, 16, ES>::CTAS;
}

}  // namespace

bool attn_rows_supported(const HeadShape& hs) { return hs.head_dim == 64 || hs.head_dim == 128; }

namespace {
// Rows per CTA: the tile that costs least, a 32- or 16-row tile paying for its shared-memory reads (fewer multiply-adds per operand load)
int tile_rows(int R) {
    auto cost = [&](int bm) { return (double)((R + bm - 1) / bm) * bm * (bm == 64 ? 1.0 : bm == 32 ? 1.2 : 1.7); };
    int best = 64;
    for (int bm : {32, 16})
        if (cost(bm) < cost(best)) best = bm;
    return best;
}
}  // namespace

int attn_rows_tiles(const HeadShape& hs, int T) {
    const int R = T * (hs.num_heads / hs.num_kv_heads), bm = tile_rows(R);
    return (R + bm - 1) / bm;
}

AttnRowsPlan attn_rows_plan(const HeadShape& hs, int batch, int T, long long total_visible, int max_visible, int kv_elem_bytes, int sm_count) {
    const int R = T * (hs.num_heads / hs.num_kv_heads);
    AttnRowsPlan p{tile_rows(R), 64, 1};
    const int ctas_sm = hs.head_dim == 64 ? (kv_elem_bytes == 2 ? rows_ctas<64, 2>(p.bm) : rows_ctas<64, 4>(p.bm))
                                          : (kv_elem_bytes == 2 ? rows_ctas<128, 2>(p.bm) : rows_ctas<128, 4>(p.bm));
    // as many slices as fill the SMs once, each a whole number of 64-position tiles
    const long long slots = std::max<long long>(1, (long long)sm_count * ctas_sm);
    const long long tiles = (long long)((R + p.bm - 1) / p.bm) * hs.num_kv_heads;
    const long long avg = total_visible / std::max(1, T);   // positions of all sequences together
    long long chunk = (avg * tiles + slots - 1) / slots;
    chunk = std::max<long long>(64, (chunk + 63) / 64 * 64);
    p.chunk_rows = (int)std::min<long long>(chunk, 1 << 30);
    p.max_splits = (max_visible + p.chunk_rows - 1) / p.chunk_rows;
    (void)batch;
    return p;
}

cudaError_t launch_attn_rows(const AttnArgs& a, int bm, int kv_elem_bytes, cudaStream_t s) {
    if (a.batch * a.T == 0) return cudaSuccess;
    if (a.hs.head_dim == 64) return kv_elem_bytes == 2 ? launch_rows_bm<64, 2>(a, bm, s) : launch_rows_bm<64, 4>(a, bm, s);
    if (a.hs.head_dim == 128) return kv_elem_bytes == 2 ? launch_rows_bm<128, 2>(a, bm, s) : launch_rows_bm<128, 4>(a, bm, s);
    return cudaErrorInvalidValue;
}

}  // namespace shainet
