// fp32 fragment attention for head sizes 64 and 128 (E == Ev): the CUDA-core path with the copies taken off its back.
//
// Same decomposition, workspace format and merge step as the other attention kernels (hogatt_plan.h).  What bounds it is
// HBM up to 16 query rows per kv head, as long as shared memory keeps up: a tile of 64 keys is 64 KiB, 2,800 cycles of an
// SM's share of the bandwidth at HD = 128.  A 16-byte shared-memory load returns 512 bytes to a warp's registers and takes four
// cycles whether its lanes read different addresses or one, so what counts is how many products a loaded value goes into.  A lane
// that was one key against R / 2 rows (a load per 0.8 products of 16 bytes) and four columns against R / 2 rows took 4,100 cycles a
// tile at R = 8, 57 % of the kernel's life; now 2,200
// (8 rows over 8 kv heads and 7,402 keys: 29.7 -> 24.5 us per call; error against 64 bits 3.3e-7 -> 2.4e-7):
//   * one warp streams K and V tiles of 64 keys into a ring with bulk copies.
//   * Q K^T: a lane is four keys against four rows at a time (two products per load), a warp the whole tile over a quarter of the
//     channels; the four warps' sums meet in shared memory.  K lies in 8 groups of 8 consecutive keys, group pitch + 16 bytes,
//     and the eight lanes of a quarter warp take the same key of the eight groups: no bank conflicts although bulk copies
//     land rows unpadded.
//   * softmax: a warp is a quarter of the rows, a lane two keys.
//   * P V: a lane is eight columns against eight rows, a warp a quarter of the keys (R = 16: half of them, and half of the rows).
//     Products go two at a time (fma.rn.f32x2, each rounded as the scalar instruction rounds it).
// Two teams of four warps take alternate tiles, each with its own running maximum, sum and O; they are folded where the CTA's
// share of a unit ends.  Row counts above 16 run as several blocks; the repeats of the keys are served by L2.
#pragma once
#include "hogatt_device.cuh"

namespace hogatt {

template <int HD, int R>
struct F32Cfg {
    // Eight warps in two teams on alternate tiles.  (One team of four had each scheduler wait out the latencies of its only warp.)
    static constexpr int TILE = 64, TEAMS = 2, WARPS = 4 * TEAMS, THREADS = (WARPS + 1) * 32;
    static constexpr int RQ = R / 2;                        // rows of a lane in Q K^T
    static constexpr int RS = R / 4;                        // rows of a warp in the softmax
    static constexpr int RG = R / 8, KW = 16 * RG;          // P V: groups of eight rows; keys of a warp
    static constexpr int LC = HD / 8, KS = 32 / LC;         // ... lanes across the columns; keys at a time
    static constexpr int GROUP_STRIDE = 8 * HD * 4 + 16;
    static constexpr int BUF_BYTES = 8 * GROUP_STRIDE;      // one K or V tile
    static constexpr int NBUF = HD == 128 ? 4 : 8;          // K and V tiles in turn; a multiple of 4, so that a buffer always serves the same team (parities)
    static constexpr int QPITCH = HD + 4;                   // floats
    static constexpr int PPITCH = R + 4;
    static constexpr int OFF_Q = NBUF * BUF_BYTES;
    static constexpr int OFF_P = OFF_Q + R * QPITCH * 4;                   // [TEAMS][64 keys][PPITCH] probabilities
    static constexpr int OFF_S = OFF_P + TEAMS * TILE * PPITCH * 4;        // [TEAMS][4 warps][R][64 keys] sums over a quarter of the channels
    static constexpr int OFF_ALPHA = OFF_S + TEAMS * 4 * R * TILE * 4;     // [TEAMS][R] what O is multiplied with first
    static constexpr int OFF_FOLD = OFF_ALPHA + TEAMS * R * 4;             // [WARPS][8][HD] O, [TEAMS][R] max, [TEAMS][R] sum
    static constexpr int OFF_LIM = OFF_FOLD + (WARPS * 8 * HD + 2 * TEAMS * R) * 4;
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
    // The rotated queries are a side output that every CTA writes a share of: the copy warp when its copies are out, if that is a
    // few elements a lane (decode), the others in front of their first tile otherwise.
    const bool want_rq = a.rq != nullptr && a.cos != nullptr;
    const bool rq_by_copies = (int64_t)a.F * a.W * a.Hq * a.S * a.E <= (int64_t)8 * gridDim.x * 32;

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
        if (want_rq && rq_by_copies)
            write_rotated_queries<float>(a.q, a.rq, a.cos, a.sin, a.F, a.W, a.Hq, a.S, a.E, a.R, blockIdx.x * 32 + lane, gridDim.x * 32);
        // (do not leave while copies may still be landing in this CTA's shared memory)
        if (lane == 0)
            for (uint32_t k = n > C::NBUF ? n - C::NBUF : 0; k < n; ++k)
                drain_stage(full + 8 * (k % C::NBUF), (k / C::NBUF) & 1u, a.status);
        return;
    }

    // ============================== scores, softmax, values ==============================
    const int team = warp >> 2, wt = warp & 3;
    const float* const q = static_cast<const float*>(a.q);
    float* const p_s = reinterpret_cast<float*>(base + C::OFF_P) + team * C::TILE * C::PPITCH;
    float* const sums = reinterpret_cast<float*>(base + C::OFF_S) + team * 4 * R * C::TILE;
    float* const alpha_s = reinterpret_cast<float*>(base + C::OFF_ALPHA) + team * R;
    float* const fold = reinterpret_cast<float*>(base + C::OFF_FOLD);
    float* const fold_m = fold + C::WARPS * 8 * HD;
    float* const fold_l = fold_m + C::TEAMS * R;
    // place x of a tile's keys in the exchanges (a lane's four keys are four places in a row) and the key it stands for
    auto key_at = [](int x) { return ((x >> 2) & 7) * 8 + (x >> 5) + 2 * (x & 3); };
    const int rows_q = (lane >> 4) * C::RQ;                                // Q K^T: first row of this lane
    const int rg = wt % C::RG, kp = wt / C::RG;                            // P V: group of rows, part of the keys
    const int col = (lane % C::LC) * 4, sub = lane / C::LC;                // ... columns col .. col + 3 and HD / 2 further
    float m[C::RS], l[C::RS];                                              // softmax rows wt * RS ...; l: this lane's keys
    uint64_t o[8][4];
    uint32_t n = 0;
    int cur_u = -1, cur_f = -1;
    bool wrote_rq = !want_rq || rq_by_copies;
    if (!working && !wrote_rq)
        write_rotated_queries<float>(a.q, a.rq, a.cos, a.sin, a.F, a.W, a.Hq, a.S, a.E, a.R, blockIdx.x * (C::WARPS * 32) + tid,
                                     gridDim.x * (C::WARPS * 32));
    const int half = a.R >> 1;                               // tables in whole 16-byte pieces, partners of a piece in one
    const bool quads = a.R % 8 == 0 && (((uintptr_t)a.cos | (uintptr_t)a.sin) & 15u) == 0;
    for (int64_t t = t0; t < t1; ++t) {
        if ((int)u != cur_u) {
            cur_u = (int)u;
            cur_f = -1;
            f = 0;
#pragma unroll
            for (int r = 0; r < C::RS; ++r) {
                m[r] = -INFINITY;
                l[r] = 0.f;
            }
#pragma unroll
            for (int r = 0; r < 8; ++r) o[r][0] = o[r][1] = o[r][2] = o[r][3] = 0ull;
        }
        while (j >= pre[f + 1]) ++f;
        if (f != cur_f) {
            cur_f = f;
            const int rb = cur_u / a.Hkv, hkv = cur_u % a.Hkv;
            named_barrier_sync(1, C::WARPS * 32);            // everyone has left the old queries
            // Four channels of a row per thread: nothing of the unit moves before its queries are there, and an element per
            // thread and pass, each with its row's divisions in front of its loads, took 6,200 cycles (4,300 now, most of
            // them behind the first tiles' copies).
            int visible = 0;
            if (tid < R && rb * 16 + tid < a.rows_total) {
                const RowId id = decode_row(rb * 16 + tid, a.G, a.S);
                visible = min(a.loc[(f * a.W + id.w) * a.S + id.s], vis[f] - 1) + 1;
            }
            for (int i = tid; i < R * HD / 4; i += C::WARPS * 32) {
                const int r = i / (HD / 4), e = (i - r * (HD / 4)) * 4, gr = rb * 16 + r;
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                if (gr < a.rows_total) {
                    const RowId id = decode_row(gr, a.G, a.S);
                    const int hq = hkv * a.G + id.g;
                    const float* const row = q + ((size_t)((a.cos != nullptr ? id.w : f * a.W + id.w) * a.Hq + hq) * a.S + id.s) * HD;
                    const size_t tab = ((size_t)(f * a.W + id.w) * a.S + id.s) * a.R;
                    if (a.cos == nullptr || quads) {
                        x = *reinterpret_cast<const float4*>(row + e);
                        if (a.cos != nullptr && e < a.R) {                 // (rope_channel's arithmetic)
                            const bool lo = e < half;
                            const float4 y = *reinterpret_cast<const float4*>(row + (lo ? e + half : e - half));
                            const float4 c = *reinterpret_cast<const float4*>(a.cos + tab + e), s = *reinterpret_cast<const float4*>(a.sin + tab + e);
                            auto turn = [lo](float x, float y, float c, float s) {
                                const float u = __fmul_rn(x, c), v = __fmul_rn(y, s);
                                return lo ? __fsub_rn(u, v) : __fadd_rn(u, v);
                            };
                            x = make_float4(turn(x.x, y.x, c.x, s.x), turn(x.y, y.y, c.y, s.y), turn(x.z, y.z, c.z, s.z), turn(x.w, y.w, c.w, s.w));
                        }
                    } else {
                        float t[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) t[k] = rope_channel<float>(row, a.cos + tab, a.sin + tab, e + k, a.R);
                        x = make_float4(t[0], t[1], t[2], t[3]);
                    }
                }
                *reinterpret_cast<float4*>(qs + r * C::QPITCH + e) = x;
            }
            if (tid < R) lim_s[tid] = visible;
            if (!wrote_rq) {                                  // (while the first tiles are in flight)
                wrote_rq = true;
                write_rotated_queries<float>(a.q, a.rq, a.cos, a.sin, a.F, a.W, a.Hq, a.S, a.E, a.R, blockIdx.x * (C::WARPS * 32) + tid,
                                             gridDim.x * (C::WARPS * 32));
            }
            named_barrier_sync(1, C::WARPS * 32);
        }
        const int tok0 = (j - pre[f]) * C::TILE, ntok = min(C::TILE, vis[f] - tok0);

        // (A wait that runs out raises the CTA's abort flag: the waits after it return at once, the results are void, and every
        // warp still reaches every barrier.)
        if (((n >> 1) & 1u) == (uint32_t)team) {
            // ---- S = Q K^T over this warp's channels: this lane's four keys against its rows ----
            uint32_t i = n % C::NBUF;
            mbar_wait_bounded(full + 8 * i, (n / C::NBUF) & 1u, abort_flag, a.status, STATUS_WAIT_FULL_TIMEOUT);
            __syncwarp();
#pragma unroll 1
            for (int pass = 0; pass < C::RQ; pass += 4) {    // (four rows at a time: the sums of eight beside O do not fit the registers)
                constexpr int CH = HD / 16;                  // 16-byte pieces of a quarter of the channels
                uint64_t s2[4][4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int r = 0; r < 4; ++r) s2[k][r] = 0ull;
                const unsigned char* const kb = base + i * C::BUF_BYTES + (lane & 7) * C::GROUP_STRIDE + ((lane >> 3) & 1) * HD * 4 + wt * CH * 16;
                const float* const qr = qs + (rows_q + pass) * C::QPITCH + wt * CH * 4;
#pragma unroll 1
                for (int c = 0; c < CH; ++c) {
                    ulonglong2 kv[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) kv[k] = *reinterpret_cast<const ulonglong2*>(kb + k * 2 * HD * 4 + c * 16);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(qr + r * C::QPITCH + c * 4);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            s2[k][r] = fma2(kv[k].x, qv.x, s2[k][r]);
                            s2[k][r] = fma2(kv[k].y, qv.y, s2[k][r]);
                        }
                    }
                }
                float* const to = sums + (wt * R + rows_q + pass) * C::TILE + (lane & 15) * 4;
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    *reinterpret_cast<float4*>(to + r * C::TILE) = make_float4(pair_sum(s2[0][r]), pair_sum(s2[1][r]), pair_sum(s2[2][r]), pair_sum(s2[3][r]));
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + 8 * i);
            named_barrier_sync(2 + team, 128);               // the four warps' sums are there
            i = (n + 1) % C::NBUF;

            // ---- online softmax, base 2: rows wt * RS ..., this lane's places lane and lane + 32 ----
#pragma unroll
            for (int r = 0; r < C::RS; ++r) {
                const int lim = lim_s[wt * C::RS + r];
                float s[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float* const from = sums + (wt * C::RS + r) * C::TILE + h * 32 + lane;
                    float x = 0.f;
#pragma unroll
                    for (int w = 0; w < 4; ++w) x += from[w * R * C::TILE];
                    const int k = key_at(h * 32 + lane);
                    s[h] = k < ntok && tok0 + k < lim ? x * a.l2scale : -INFINITY;
                }
                const float top = fmaxf(m[r], warp_max(fmaxf(s[0], s[1])));
                const float alpha = top == m[r] ? 1.f : m[r] == -INFINITY ? 0.f : exp2f(m[r] - top);
                m[r] = top;
                const float mu = top == -INFINITY ? 0.f : top;
                s[0] = exp2f(s[0] - mu);                     // (hidden: 0; not a number stays one)
                s[1] = exp2f(s[1] - mu);
                l[r] = fmaf(l[r], alpha, s[0] + s[1]);
#pragma unroll
                for (int h = 0; h < 2; ++h) p_s[(h * 32 + lane) * C::PPITCH + wt * C::RS + r] = s[h];
                if (lane == 0) alpha_s[wt * C::RS + r] = alpha;
            }
            named_barrier_sync(2 + team, 128);               // the probabilities are there

            // ---- O += P V: this lane's eight columns against eight rows ----
            {
                float al[8];
                *reinterpret_cast<float4*>(al) = *reinterpret_cast<const float4*>(alpha_s + rg * 8);
                *reinterpret_cast<float4*>(al + 4) = *reinterpret_cast<const float4*>(alpha_s + rg * 8 + 4);
                bool grew = false;
#pragma unroll
                for (int r = 0; r < 8; ++r) grew |= al[r] != 1.f;
                if (grew) {                                  // (the same in every lane)
#pragma unroll
                    for (int r = 0; r < 8; ++r) {
                        const uint64_t al2 = pair_f32(al[r], al[r]);
#pragma unroll
                        for (int e = 0; e < 4; ++e) o[r][e] = fma2(o[r][e], al2, 0ull);
                    }
                }
            }
            mbar_wait_bounded(full + 8 * i, ((n + 1) / C::NBUF) & 1u, abort_flag, a.status, STATUS_WAIT_FULL_TIMEOUT);
            __syncwarp();
            {
                const float* const v = reinterpret_cast<const float*>(base + i * C::BUF_BYTES) + col;
                auto values = [&](auto whole) {
#pragma unroll 2
                    for (int kk = 0; kk < C::KW; kk += C::KS) {
                        const int x = kp * C::KW + kk + sub, tk = key_at(x);
                        ulonglong2 v0 = make_ulonglong2(0ull, 0ull), v1 = v0;
                        if (decltype(whole)::value || tk < ntok) {          // (what was not copied may hold anything)
                            v0 = *reinterpret_cast<const ulonglong2*>(v + tk * HD);
                            v1 = *reinterpret_cast<const ulonglong2*>(v + tk * HD + HD / 2);
                        }
                        float p[8];
                        *reinterpret_cast<float4*>(p) = *reinterpret_cast<const float4*>(p_s + x * C::PPITCH + rg * 8);
                        *reinterpret_cast<float4*>(p + 4) = *reinterpret_cast<const float4*>(p_s + x * C::PPITCH + rg * 8 + 4);
#pragma unroll
                        for (int r = 0; r < 8; ++r) {
                            const uint64_t pp = pair_f32(p[r], p[r]);
                            o[r][0] = fma2(v0.x, pp, o[r][0]);
                            o[r][1] = fma2(v0.y, pp, o[r][1]);
                            o[r][2] = fma2(v1.x, pp, o[r][2]);
                            o[r][3] = fma2(v1.y, pp, o[r][3]);
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

        // ---- leave a partial result where this CTA's share of the unit ends: fold the warps that share rows ----
        if (j == TH - 1 || t == t1 - 1) {
            int first, count;
            unit_ctas(u, TH, N, ctas, &first, &count);
            const size_t row0 = ((size_t)u * a.parts_per_unit + (blockIdx.x - first)) * 16;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                float x[8];
#pragma unroll
                for (int e = 0; e < 4; ++e) unpair_f32(o[r][e], x[2 * e], x[2 * e + 1]);
#pragma unroll
                for (int d = C::LC; d < 32; d *= 2)                        // lanes that took other keys of the same columns
#pragma unroll
                    for (int e = 0; e < 8; ++e) x[e] += __shfl_xor_sync(0xffffffffu, x[e], d);
                if (sub == 0) {
                    float* const to = fold + (warp * 8 + r) * HD + col;
                    *reinterpret_cast<float4*>(to) = make_float4(x[0], x[1], x[2], x[3]);
                    *reinterpret_cast<float4*>(to + HD / 2) = make_float4(x[4], x[5], x[6], x[7]);
                }
            }
#pragma unroll
            for (int r = 0; r < C::RS; ++r) {
                float sum = l[r];
#pragma unroll
                for (int x = 16; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
                if (lane == 0) {
                    fold_m[team * R + wt * C::RS + r] = m[r];
                    fold_l[team * R + wt * C::RS + r] = sum;
                }
            }
            named_barrier_sync(1, C::WARPS * 32);
            for (int idx = tid; idx < R * HD / 4; idx += C::WARPS * 32) {
                const int r = idx / (HD / 4), c = (idx - r * (HD / 4)) * 4;
                const float M = fmaxf(fold_m[r], fold_m[R + r]), mu = M == -INFINITY ? 0.f : M;
                float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                float sum = 0.f;
#pragma unroll
                for (int x = 0; x < C::TEAMS; ++x) {
                    const float w = exp2f(fold_m[x * R + r] - mu);
#pragma unroll
                    for (int k = 0; k < 4 / C::RG; ++k) {
                        const float4 y = *reinterpret_cast<const float4*>(fold + ((x * 4 + k * C::RG + r / 8) * 8 + r % 8) * HD + c);
                        acc.x = fmaf(y.x, w, acc.x);
                        acc.y = fmaf(y.y, w, acc.y);
                        acc.z = fmaf(y.z, w, acc.z);
                        acc.w = fmaf(y.w, w, acc.w);
                    }
                    sum = fmaf(fold_l[x * R + r], w, sum);
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
