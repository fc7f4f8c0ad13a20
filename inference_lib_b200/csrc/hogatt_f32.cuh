// fp32 fragment attention for head sizes 64 and 128 (E == Ev): the CUDA-core path with the copies taken off its back.
//
// Same decomposition, workspace format and merge step as the other attention kernels (hogatt_plan.h).  What bounds it is
// HBM up to 16 query rows per kv head: a key costs 8 * HD bytes and 2 * R * HD fused multiply-adds, at HD = 128 43 cycles of
// an SM's share of the bandwidth against 16 (R = 8) or 32 (R = 16) cycles of its FMA pipes -- if the operands come out of
// shared memory cheaply enough, which is what the layout is about:
//   * one warp streams K and V tiles of 64 keys into a ring with bulk copies (the kernel before had every thread load,
//     convert and store each tile between two CTA barriers: 121 us per call at 8 rows over 8 kv heads and 7,402 keys).
//   * Q K^T: a lane is a key, a warp 32 keys x R/2 rows.  A key's 16-byte chunk is read once for R/2 rows, the queries'
//     chunks are broadcasts.  K lies in 8 groups of 8 consecutive keys, group pitch + 16 bytes, and the eight lanes of a
//     quarter warp take the same key of the eight groups: no bank conflicts although bulk copies land rows unpadded.
//   * P V: a lane is four columns, probabilities are broadcasts.  Products go two at a time (fma.rn.f32x2, each rounded
//     as the scalar instruction rounds it).
// Warps keep their own running maximum, sum and O; the four warps that share rows are folded where the CTA's share of a unit
// ends.  Row counts above 16 run as several blocks; the repeats of the keys are served by L2.
#pragma once
#include "hogatt_device.cuh"

namespace hogatt {

template <int HD, int R>
struct F32Cfg {
    // Eight warps: w & 1 the half of a tile's keys, (w >> 1) & 1 the half of the rows, w >> 2 which tiles (every other one).
    // One team of four had each scheduler wait out the latencies of its only warp.
    static constexpr int TILE = 64, TEAMS = 2, WARPS = 4 * TEAMS, THREADS = (WARPS + 1) * 32;
    static constexpr int RW = R / 2;                        // rows per warp
    static constexpr int GROUP_STRIDE = 8 * HD * 4 + 16;
    static constexpr int BUF_BYTES = 8 * GROUP_STRIDE;      // one K or V tile
    static constexpr int NBUF = HD == 128 ? 4 : 8;          // K and V tiles in turn; a multiple of 4, so that a buffer always serves the same team (parities)
    static constexpr int QPITCH = HD + 4;                   // floats
    static constexpr int CPL = HD / 32;                     // columns of O per lane and key: lanes cover 128 columns, or 64 twice
    static constexpr int OFF_Q = NBUF * BUF_BYTES;
    static constexpr int OFF_P = OFF_Q + R * QPITCH * 4;                   // [WARPS][32 keys][RW]
    static constexpr int OFF_FOLD = OFF_P + WARPS * 32 * RW * 4;           // [WARPS][RW][HD] O, [WARPS][RW] max, [WARPS][RW] sum
    static constexpr int OFF_LIM = OFF_FOLD + WARPS * RW * (HD + 2) * 4;
    static constexpr int OFF_BAR = (OFF_LIM + R * 4 + 15) / 16 * 16;
    static constexpr int OFF_PLAN = OFF_BAR + 2 * NBUF * 8 + 16;           // abort flag in between
};
template <int HD, int R>
__host__ __device__ constexpr size_t f32_smem_bytes(int F) {
    return 128 + F32Cfg<HD, R>::OFF_PLAN + ((size_t)2 * F + 1) * 4;
}

__device__ __forceinline__ float warp_max(float x) {
    float y;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float pair_sum(uint64_t v) {
    float lo, hi;
    unpair_f32(v, lo, hi);
    return lo + hi;
}

template <int HD, int R>
__global__ void __launch_bounds__(F32Cfg<HD, R>::THREADS, 1) f32_attention_kernel(const __grid_constant__ KernelArgs a) {
    using C = F32Cfg<HD, R>;
    constexpr int RW = C::RW;
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 127) & ~(uintptr_t)127);
    float* const qs = reinterpret_cast<float*>(base + C::OFF_Q);
    int* const lim_s = reinterpret_cast<int*>(base + C::OFF_LIM);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(base + C::OFF_BAR + 2 * C::NBUF * 8);
    int* vis = reinterpret_cast<int*>(base + C::OFF_PLAN);
    int* pre = vis + a.F;
    const uint32_t bufs = smem_u32(base), full = smem_u32(base + C::OFF_BAR), empty = full + 8 * C::NBUF;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int i = 0; i < C::NBUF; ++i) {
            mbar_init(full + 8 * i, 1);
            mbar_init(empty + 8 * i, 4);             // the warps of one team
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async_smem();
    }
    pdl_wait();
    pdl_trigger();
    build_tile_prefix(a, C::TILE, vis, pre);         // ends with __syncthreads(): the barriers are visible too
    const int TH = pre[a.F], units = a.row_blocks * a.Hkv;
    const int64_t N = (int64_t)units * TH;
    const int ctas = effective_ctas(N, gridDim.x);
    if (blockIdx.x == 0 && tid == 0) {
        a.header[0] = TH;
        a.header[1] = ctas;
    }
    const bool working = (int)blockIdx.x < ctas;
    const int64_t t0 = working ? cta_first_tile(blockIdx.x, N, ctas) : 0, t1 = working ? cta_first_tile(blockIdx.x + 1, N, ctas) : 0;
    int64_t u = working ? t0 / TH : 0;
    int j = (int)(t0 - u * TH), f = 0;

    if (warp == C::WARPS) {
        // ============================== K and V copies ==============================
        uint32_t n = 0;
        bool ok = true;
        for (int64_t t = t0; t < t1 && ok; ++t) {
            while (j >= pre[f + 1]) ++f;
            const int tok0 = (j - pre[f]) * C::TILE, ntok = min(C::TILE, vis[f] - tok0);
            const size_t row = (size_t)(u % a.Hkv) * a.ft.e[f].rows + tok0;
#pragma unroll
            for (int kv = 0; kv < 2; ++kv, ++n) {
                const uint32_t i = n % C::NBUF;
                ok = mbar_wait_bounded(empty + 8 * i, ((n / C::NBUF) & 1u) ^ 1u, abort_flag, a.status, STATUS_WAIT_EMPTY_TIMEOUT);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                if (lane == 0) mbar_arrive_expect_tx(full + 8 * i, (uint32_t)ntok * HD * 4);
                __syncwarp();
                const float* src = static_cast<const float*>(kv ? a.ft.e[f].v : a.ft.e[f].k) + row * HD;
                if (kv) {
                    if (lane == 0) bulk_load(bufs + i * C::BUF_BYTES, src, (uint32_t)ntok * HD * 4, full + 8 * i);
                } else if (lane < 8 && ntok > lane * 8) {
                    bulk_load(bufs + i * C::BUF_BYTES + lane * C::GROUP_STRIDE, src + lane * 8 * HD, (uint32_t)min(8, ntok - lane * 8) * HD * 4,
                              full + 8 * i);
                }
            }
            if (++j == TH) {
                j = 0;
                ++u;
                f = 0;
            }
        }
        // (do not leave while copies may still be landing in this CTA's shared memory)
        if (lane == 0)
            for (uint32_t k = n > C::NBUF ? n - C::NBUF : 0; k < n; ++k)
                drain_stage(full + 8 * (k % C::NBUF), (k / C::NBUF) & 1u, a.status);
        return;
    }

    // ============================== scores, softmax, values ==============================
    const int kh = warp & 1, rw0 = ((warp >> 1) & 1) * RW, team = warp >> 2;        // half of the keys, first row, which tiles
    const float* const q = static_cast<const float*>(a.q);
    float* const p_s = reinterpret_cast<float*>(base + C::OFF_P) + warp * 32 * RW;
    float* const fold = reinterpret_cast<float*>(base + C::OFF_FOLD);
    float* const fold_m = fold + C::WARPS * RW * HD;
    float* const fold_l = fold_m + C::WARPS * RW;
    const int my_key = (lane & 7) * 8 + kh * 4 + (lane >> 3);              // of the tile
    const int col = (lane * 4) % HD, vhalf = HD == 64 ? lane >> 4 : 0;     // HD 64: the half warps take every other key
    float m[RW], l[RW];
    uint64_t o[RW][2];
    uint32_t n = 0;
    int cur_u = -1, cur_f = -1;
    int lim[RW];
    bool wrote_rq = a.rq == nullptr || a.cos == nullptr;
    if (!working && !wrote_rq)
        write_rotated_queries<float>(a.q, a.rq, a.cos, a.sin, a.F, a.W, a.Hq, a.S, a.E, a.R, blockIdx.x * (C::WARPS * 32) + tid,
                                     gridDim.x * (C::WARPS * 32));
    for (int64_t t = t0; t < t1; ++t) {
        if ((int)u != cur_u) {
            cur_u = (int)u;
            cur_f = -1;
            f = 0;
#pragma unroll
            for (int r = 0; r < RW; ++r) {
                m[r] = -INFINITY;
                l[r] = 0.f;
                o[r][0] = o[r][1] = 0ull;
            }
        }
        while (j >= pre[f + 1]) ++f;
        if (f != cur_f) {
            cur_f = f;
            const int rb = cur_u / a.Hkv, hkv = cur_u % a.Hkv;
            named_barrier_sync(1, C::WARPS * 32);            // everyone has left the old queries
#pragma unroll 4
            for (int i = tid; i < R * HD; i += C::WARPS * 32) {
                const int r = i / HD, e = i - r * HD, gr = rb * 16 + r;
                float x = 0.f;
                if (gr < a.rows_total) {
                    const RowId id = decode_row(gr, a.G, a.S);
                    const int hq = hkv * a.G + id.g;
                    if (a.cos != nullptr) {
                        const size_t tab = ((size_t)(f * a.W + id.w) * a.S + id.s) * a.R;
                        x = rope_channel<float>(q + ((size_t)(id.w * a.Hq + hq) * a.S + id.s) * HD, a.cos + tab, a.sin + tab, e, a.R);
                    } else {
                        x = q[((size_t)((f * a.W + id.w) * a.Hq + hq) * a.S + id.s) * HD + e];
                    }
                }
                qs[r * C::QPITCH + e] = x;
            }
            if (tid < R) {
                const int gr = rb * 16 + tid;
                int visible = 0;
                if (gr < a.rows_total) {
                    const RowId id = decode_row(gr, a.G, a.S);
                    visible = min(a.loc[(f * a.W + id.w) * a.S + id.s], vis[f] - 1) + 1;
                }
                lim_s[tid] = visible;
            }
            if (!wrote_rq) {                                  // (while the first tiles are in flight)
                wrote_rq = true;
                write_rotated_queries<float>(a.q, a.rq, a.cos, a.sin, a.F, a.W, a.Hq, a.S, a.E, a.R, blockIdx.x * (C::WARPS * 32) + tid,
                                             gridDim.x * (C::WARPS * 32));
            }
            named_barrier_sync(1, C::WARPS * 32);
#pragma unroll
            for (int r = 0; r < RW; ++r) lim[r] = lim_s[rw0 + r];
        }
        const int tok0 = (j - pre[f]) * C::TILE, ntok = min(C::TILE, vis[f] - tok0);

        // ---- S = Q K^T: this lane's key against the warp's rows.  (A wait that runs out raises the CTA's abort flag: the
        // waits after it return at once, the results are void, and every warp still reaches every barrier.) ----
        if (((n >> 1) & 1u) == (uint32_t)team) {
            uint32_t i = n % C::NBUF;
            mbar_wait_bounded(full + 8 * i, (n / C::NBUF) & 1u, abort_flag, a.status, STATUS_WAIT_FULL_TIMEOUT);
            __syncwarp();
            uint64_t s2[RW];
#pragma unroll
            for (int r = 0; r < RW; ++r) s2[r] = 0ull;
            {
                const ulonglong2* k = reinterpret_cast<const ulonglong2*>(base + i * C::BUF_BYTES + (lane & 7) * C::GROUP_STRIDE + (my_key & 7) * HD * 4);
                const float* qr = qs + rw0 * C::QPITCH;
#pragma unroll 4
                for (int c = 0; c < HD / 4; ++c) {
                    const ulonglong2 kv = k[c];
#pragma unroll
                    for (int r = 0; r < RW; ++r) {
                        const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(qr + r * C::QPITCH + c * 4);
                        s2[r] = fma2(kv.x, qv.x, s2[r]);
                        s2[r] = fma2(kv.y, qv.y, s2[r]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + 8 * i);
            i = (n + 1) % C::NBUF;

            // ---- online softmax, base 2 ----
            const int key = tok0 + my_key;
            float s[RW];
            bool grew = false;
            float top[RW];
#pragma unroll
            for (int r = 0; r < RW; ++r) {
                s[r] = my_key < ntok && key < lim[r] ? pair_sum(s2[r]) * a.l2scale : -INFINITY;
                top[r] = fmaxf(m[r], warp_max(s[r]));
                grew |= top[r] != m[r];
            }
            if (grew) {                                           // (the same in every lane)
#pragma unroll
                for (int r = 0; r < RW; ++r) {
                    const float alpha = m[r] == -INFINITY ? 0.f : exp2f(m[r] - top[r]);
                    const uint64_t al2 = pair_f32(alpha, alpha);
                    l[r] *= alpha;
                    o[r][0] = fma2(o[r][0], al2, 0ull);
                    o[r][1] = fma2(o[r][1], al2, 0ull);
                    m[r] = top[r];
                }
            }
#pragma unroll
            for (int r = 0; r < RW; ++r) {
                s[r] = exp2f(s[r] - (m[r] == -INFINITY ? 0.f : m[r]));      // (hidden: 0; not a number stays one)
                l[r] += s[r];
            }
#pragma unroll
            for (int r = 0; r < RW; r += 4) *reinterpret_cast<float4*>(p_s + lane * RW + r) = make_float4(s[r], s[r + 1], s[r + 2], s[r + 3]);
            __syncwarp();

            // ---- O += P V: this lane's four columns ----
            mbar_wait_bounded(full + 8 * i, ((n + 1) / C::NBUF) & 1u, abort_flag, a.status, STATUS_WAIT_FULL_TIMEOUT);
            __syncwarp();
            {
                const float* v = reinterpret_cast<const float*>(base + i * C::BUF_BYTES) + col;
                constexpr int STEP = HD == 64 ? 2 : 1;
                auto values = [&](auto whole) {
#pragma unroll 8
                    for (int kk = 0; kk < 32; kk += STEP) {
                        const int x = kk + vhalf;                 // key of the warp's 32: lane x's
                        const int tk = (x & 7) * 8 + kh * 4 + (x >> 3);
                        ulonglong2 vv = make_ulonglong2(0ull, 0ull);
                        if (decltype(whole)::value || tk < ntok) vv = *reinterpret_cast<const ulonglong2*>(v + tk * HD);
#pragma unroll
                        for (int r = 0; r < RW; r += 4) {
                            const float4 p = *reinterpret_cast<const float4*>(p_s + x * RW + r);
                            const float pr[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const uint64_t pp = pair_f32(pr[e], pr[e]);
                                o[r + e][0] = fma2(vv.x, pp, o[r + e][0]);
                                o[r + e][1] = fma2(vv.y, pp, o[r + e][1]);
                            }
                        }
                    }
                };
                if (ntok == C::TILE) values(std::true_type());
                else values(std::false_type());
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + 8 * i);
        }
        n += 2;

        // ---- leave a partial result where this CTA's share of the unit ends: fold the two key halves of every row ----
        if (j == TH - 1 || t == t1 - 1) {
            int first, count;
            unit_ctas(u, TH, N, ctas, &first, &count);
            const size_t row0 = ((size_t)u * a.parts_per_unit + (blockIdx.x - first)) * 16;
#pragma unroll
            for (int r = 0; r < RW; ++r) {
                float sum = l[r];
#pragma unroll
                for (int x = 16; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
                float x[4];
                unpair_f32(o[r][0], x[0], x[1]);
                unpair_f32(o[r][1], x[2], x[3]);
                if constexpr (HD == 64) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) x[e] += __shfl_xor_sync(0xffffffffu, x[e], 16);
                }
                if (lane * 4 < HD) *reinterpret_cast<float4*>(fold + (warp * RW + r) * HD + lane * 4) = make_float4(x[0], x[1], x[2], x[3]);
                if (lane == 0) {
                    fold_m[warp * RW + r] = m[r];
                    fold_l[warp * RW + r] = sum;
                }
            }
            named_barrier_sync(1, C::WARPS * 32);
            for (int idx = tid; idx < R * HD / 4; idx += C::WARPS * 32) {
                const int r = idx / (HD / 4), c = (idx - r * (HD / 4)) * 4;
                // the row's warps: both key halves of both teams
                float M = -INFINITY, sum = 0.f;
#pragma unroll
                for (int x = 0; x < 2 * C::TEAMS; ++x) M = fmaxf(M, fold_m[((x >> 1) * 4 + (r / RW) * 2 + (x & 1)) * RW + r % RW]);
                const float mu = M == -INFINITY ? 0.f : M;
                float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int x = 0; x < 2 * C::TEAMS; ++x) {
                    const int slot = ((x >> 1) * 4 + (r / RW) * 2 + (x & 1)) * RW + r % RW;
                    const float w = exp2f(fold_m[slot] - mu);
                    const float4 y = *reinterpret_cast<const float4*>(fold + slot * HD + c);
                    acc.x = fmaf(y.x, w, acc.x);
                    acc.y = fmaf(y.y, w, acc.y);
                    acc.z = fmaf(y.z, w, acc.z);
                    acc.w = fmaf(y.w, w, acc.w);
                    sum = fmaf(fold_l[slot], w, sum);
                }
                *reinterpret_cast<float4*>(a.ws_o + (row0 + r) * HD + c) = acc;
                if (c == 0) {
                    a.ws_m[row0 + r] = M;
                    a.ws_l[row0 + r] = sum;
                }
            }
            named_barrier_sync(1, C::WARPS * 32);            // (read before the next share's fold)
        }
        if (++j == TH) {
            j = 0;
            ++u;
        }
    }
}

}  // namespace hogatt
