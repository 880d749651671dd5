// Incremental decoding: one new token per sequence against a key/value cache.
// Not part of the reference (it has full-sequence kernels only); the operators are the same as
// in the full forward - matmul + bias (+ tanh-GELU) as in kernels/matmul/1_matmul_tiling.cuh:25-54
// and 9_matmul_async_cg_tf32_gelu.cuh:5-11, causal attention with scale 1/sqrt(HS) as in
// kernels/attention/1_attention_cublas.cuh:50-61 - evaluated for M = B rows (B <= 16).
// With so few rows every weight is used B times only: the step is bound by reading the weights
// and the cache out of HBM once, not by arithmetic, so these kernels run on the fp32 FMA pipe
// (exact fp32 products, no TF32 rounding) and are organised around coalesced streaming:
//   skinny_gemm_kernel      out[b,n] = act(sum_k x[b,k] W[n,k] + bias[n]); every CTA streams an equal
//                           share of W's rows against x staged in shared memory
//   kv_append_kernel        K and V columns of freshly computed qkv rows -> cache (prefill)
//   decode_attention_kernel a cluster per (sequence, head): stores the new position's K and V,
//                           its CTAs walk shares of the cached positions with an online softmax
//                           and the states are merged through (distributed) shared memory
//   decode_encoder_kernel   wte[token] + wpe[pos]
// The position is read from device memory, so one captured CUDA graph serves every step.
#include <cstdlib>
#include "kernels.h"
#include "decoder_math.cuh"
#include "../prim/sm100.cuh"

namespace b200 {

namespace {

constexpr int kSkinnyWarps = 8, kSkinnyThreads = 2 * 32 * kSkinnyWarps;  // warps along K; two such teams per CTA

// Optional prologue (ln_w != nullptr): the input rows are first formed as
//   r = resid_in + branch (branch may be null),  x = layernorm(r) * ln_w + ln_b
// by every CTA for itself (B rows of C = K floats: a few KB), and CTA 0 also stores r to
// resid_out - a different buffer than resid_in, which other CTAs are still reading.  That is the
// forward's fused residual + layernorm (two-pass variance, eps 1e-5) without a kernel of its own.
struct SkinnyArgs {
    float* out;
    const float* x;         // [B,K] input rows, or resid_in when the prologue is on
    const float* W;
    const float* bias;
    const float* branch;    // prologue: added to x before the layernorm (nullable)
    const float* ln_w;      // prologue switch
    const float* ln_b;
    float* resid_out;       // prologue: r is stored here by CTA 0
    int B, N, K, gelu;
    int k_splits;       // > 1: K is cut into slices computed by different CTAs; slice s writes its partial sums to out + s*B*N
    int kslice;         // floats of K per slice (K when k_splits == 1)
    int branch_parts;   // prologue: branch holds this many partial results [parts][B][K], summed in order
    const uint8_t* next;  // bytes that the step reads next (its next product's weights): asked for into L2; nullable
    size_t next_bytes;
};

// Bound by the weights' bytes where there are many, and by the chain wait - input rows - layernorm - sum - store where there are
// few, so: every CTA has the same number of rows (a share of N, not of whole tiles: with 16-row tiles 4800 rows would be 300
// tiles for 148 SMs, three rounds for two and a bit), each of its two teams of eight warps one half of them and each warp of a team an eighth of
// the columns; and everything that does not depend on the previous kernel - the first U steps of the weights, bias, layernorm
// parameters - is requested before waiting for it.  Eight lanes of a warp stand side by side in K and four in rows: a request is four rows'
// whole 128-byte lines, the input is read from shared memory once per R rows, and the sum over lanes takes three exchanges
// once per tile of 4 R rows.  Sixteen warps per SM and registers without spills are what hides the steps' latency (8 rows, GPT-2 XL, QKV:
// 27 us with eight warps of spilling threads, 22 without spills, 16 so); with one or two input rows 64 registers are enough for two
// CTAs on an SM, and the next kernel's requests are on their way while this one ends.  While it waits a kernel asks for the next
// one's weights into L2.  A decode step, against two rows per warp in whole rounds of 16-row tiles and K slices for narrow
// outputs: GPT-2 124M, 1 row behind 897 positions 540 -> 290 us; 8 rows, 543 positions 548 -> 404; XL, 8 rows, 300 positions 4810 -> 3271.
// NB: input rows, padded.  NV = float4 per lane that hold half a row in the layernorm prologue (0: no prologue compiled in).
template <int NB, int R> __host__ __device__ constexpr int skinny_steps() { return NB == 16 ? 3 : (R == 1 ? 4 : (R == 2 ? 3 : 2)); }
template <int NB, int R, int NV>
__global__ void __launch_bounds__(kSkinnyThreads, NB == 2 && NV < 7 && R < 4 ? 2 : 1)
skinny_gemm_kernel(const SkinnyArgs a) {
    constexpr int U = skinny_steps<NB, R>();  // steps of 32 columns on the way per warp
    constexpr int CNT = R * NB, HELD = CNT > 8 ? CNT / 8 : 1, TILE = 4 * R;
    extern __shared__ float4 xs4[];  // [NB][columns / 4]: the input rows; with the prologue the layernorm's weight and bias behind them
    __shared__ float red[2][2][kSkinnyWarps][4 * CNT];
    __shared__ float sums[2][2][8];
    float* xs = reinterpret_cast<float*>(xs4);
    const int B = a.B, N = a.N, K = a.K, K4 = a.K >> 2;
    const int tid = threadIdx.x, team = tid >> 8, warp = (tid >> 5) & 7, lane = tid & 31, c = lane & 7, g = lane >> 3;
    const int ks = blockIdx.x % a.k_splits, part = blockIdx.x / a.k_splits, parts = gridDim.x / a.k_splits;
    const int kbeg = ks * a.kslice, cols = min(K - kbeg, a.kslice), stride = NV > 0 ? K : a.kslice;
    const int n0 = (int)((long)N * part / parts), n2 = (int)((long)N * (part + 1) / parts), n1 = (n0 + n2 + 1) >> 1;
    const int n_begin = team ? n1 : n0, rows = (team ? n2 : n1) - n_begin;  // this team's rows (may be none)
    // this warp's steps of 32 columns, the last one perhaps narrower
    const int steps = (cols + 31) >> 5, s0 = steps * warp / kSkinnyWarps, ns = steps * (warp + 1) / kSkinnyWarps - s0;
    const int nsb = (ns + U - 1) / U, tiles = (rows + TILE - 1) / TILE;
    const int k0 = s0 * 32 + c * 4;  // this lane's first column in the slice
    const float* wbase = a.W + (size_t)n_begin * K + kbeg;
    int row_at[R];  // where the rows of the tile being requested begin (beyond the last row: that one again, and not stored)
    auto rows_of = [&](int tile) {
#pragma unroll
        for (int r = 0; r < R; ++r) row_at[r] = min(tile * TILE + r * 4 + g, rows - 1) * K;
    };
    float4 w[U][R];
    auto request = [&](int u, int s) {
        if (s < ns) {
            const int k = min(k0 + s * 32, cols - 4);
#pragma unroll
            for (int r = 0; r < R; ++r) w[u][r] = __ldg(reinterpret_cast<const float4*>(wbase + row_at[r] + k));
        }
    };
    if (tiles > 0) {
        rows_of(0);
#pragma unroll
        for (int u = 0; u < U; ++u) request(u, u);
    }
    float* lnw = xs + NB * K;
    float* lnb = lnw + K;
    if (NV > 0) {
        for (int i = tid; i < K4; i += kSkinnyThreads) {
            cp_async16(lnw + i * 4, a.ln_w + i * 4);
            cp_async16(lnb + i * 4, a.ln_b + i * 4);
        }
        cp_async_commit();
    }
    if (a.next && tid == 0) {
        const size_t share = ((a.next_bytes / gridDim.x) + 127) & ~(size_t)127, at = share * blockIdx.x;
        if (at < a.next_bytes) l2_prefetch_bulk(a.next + at, (uint32_t)(a.next_bytes - at < share ? a.next_bytes - at : share));
    }
    griddep_launch_dependents();
    griddep_wait();
    if (NV > 0) {
        // two warps per row; a lane holds every 64th float4 of the row
        constexpr int NVV = NV > 0 ? NV : 1;
        for (int b0 = 0; b0 < B; b0 += kSkinnyWarps) {
            const int b = b0 + warp;
            float4 v[NVV];
            float sum = 0.f, q = 0.f;
#pragma unroll
            for (int i = 0; i < NVV; ++i) {
                const int e = team * 32 + lane + i * 64;
                v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (b < B && e < K4 && a.branch) v[i] = *(reinterpret_cast<const float4*>(a.branch + (size_t)b * K) + e);
            }
            for (int p = 1; a.branch && p < a.branch_parts; ++p) {  // the producer's K slices, in order
#pragma unroll
                for (int i = 0; i < NVV; ++i) {
                    const int e = team * 32 + lane + i * 64;
                    if (b < B && e < K4) {
                        const float4 u = *(reinterpret_cast<const float4*>(a.branch + ((size_t)p * B + b) * K) + e);
                        v[i].x += u.x; v[i].y += u.y; v[i].z += u.z; v[i].w += u.w;
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < NVV; ++i) {
                const int e = team * 32 + lane + i * 64;
                if (b < B && e < K4) {
                    const float4 u = *(reinterpret_cast<const float4*>(a.x + (size_t)b * K) + e);
                    v[i].x += u.x; v[i].y += u.y; v[i].z += u.z; v[i].w += u.w;
                    if (blockIdx.x == 0) *(reinterpret_cast<float4*>(a.resid_out + (size_t)b * K) + e) = v[i];
                }
                sum += (v[i].x + v[i].y) + (v[i].z + v[i].w);
            }
            sum = warp_sum(sum);
            if (lane == 0) sums[0][team][warp] = sum;
            cp_async_wait<0>();
            __syncthreads();
            const float mean = (sums[0][0][warp] + sums[0][1][warp]) / (float)K;
#pragma unroll
            for (int i = 0; i < NVV; ++i) {
                if (team * 32 + lane + i * 64 < K4) {
                    const float dx = v[i].x - mean, dy = v[i].y - mean, dz = v[i].z - mean, dw = v[i].w - mean;
                    q += (dx * dx + dy * dy) + (dz * dz + dw * dw);
                }
            }
            q = warp_sum(q);
            if (lane == 0) sums[1][team][warp] = q;
            __syncthreads();
            const float rstd = rsqrtf((sums[1][0][warp] + sums[1][1][warp]) / (float)K + 1e-5f);
#pragma unroll
            for (int i = 0; i < NVV; ++i) {
                const int e = team * 32 + lane + i * 64;
                if (b < B && e < K4) {
                    const float4 lw = *reinterpret_cast<const float4*>(lnw + e * 4), lb = *reinterpret_cast<const float4*>(lnb + e * 4);
                    *reinterpret_cast<float4*>(xs + (size_t)b * K + e * 4) =
                        make_float4((v[i].x - mean) * rstd * lw.x + lb.x, (v[i].y - mean) * rstd * lw.y + lb.y,
                                    (v[i].z - mean) * rstd * lw.z + lb.z, (v[i].w - mean) * rstd * lw.w + lb.w);
                }
            }
        }
    } else {  // the columns of the warp and of its partner in the other team, every other row each
        const int cols4 = min(ns * 8, (cols >> 2) - s0 * 8);
        for (int b = team; b < B; b += 2)
            for (int i = lane; i < cols4; i += 32)
                cp_async16(xs + (size_t)b * stride + s0 * 32 + i * 4, a.x + (size_t)b * K + kbeg + s0 * 32 + i * 4);
        cp_async_commit();
        cp_async_wait<0>();
    }
    __syncthreads();
    float* __restrict__ out = a.out + (size_t)ks * B * N;
    const int first = scatter_first<CNT, 8>(lane);
    // the output that this thread stores: column of the tile, input row
    const int on = (tid & 255) % TILE, ob = (tid & 255) / TILE;
    const float* xl = xs + k0;
    for (int tile = 0; tile < tiles; ++tile) {
        const bool mine = ob < B && ob < NB && tile * TILE + on < rows;
        const int n = n_begin + tile * TILE + on;
        const float bias = mine && a.bias && ks == 0 ? __ldg(a.bias + n) : 0.f;
        float acc[CNT];
#pragma unroll
        for (int i = 0; i < CNT; ++i) acc[i] = 0.f;
        for (int sb = 0; sb < nsb; ++sb) {
            const bool last = sb + 1 == nsb;
            if (last && tile + 1 < tiles) rows_of(tile + 1);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int s = sb * U + u;
                if (s < ns) {
                    if (k0 + s * 32 < cols) {
#pragma unroll
                        for (int b = 0; b < NB; ++b) {
                            const float4 x = *reinterpret_cast<const float4*>(xl + b * stride + s * 32);
#pragma unroll
                            for (int r = 0; r < R; ++r) {
                                float t = acc[r * NB + b];
                                t = fmaf(w[u][r].x, x.x, t);
                                t = fmaf(w[u][r].y, x.y, t);
                                t = fmaf(w[u][r].z, x.z, t);
                                t = fmaf(w[u][r].w, x.w, t);
                                acc[r * NB + b] = t;
                            }
                        }
                    }
                }
                // (the registers are free again)
                if (!last) request(u, s + U);
                else if (tile + 1 < tiles) request(u, u);
            }
        }
        reduce_scatter<CNT, 8>(acc, lane);
        float (&rd)[kSkinnyWarps][4 * CNT] = red[team][tile & 1];
        if (scatter_owner<CNT, 8>(lane)) {
#pragma unroll
            for (int i = 0; i < HELD; ++i) rd[warp][g * CNT + first + i] = acc[i];
        }
        asm volatile("bar.sync %0, 256;" ::"r"(team + 1) : "memory");
        if (mine) {
            float v = bias;
            const int e = (on & 3) * CNT + (on >> 2) * NB + ob;
#pragma unroll
            for (int i = 0; i < kSkinnyWarps; ++i) v += rd[i][e];
            if (a.gelu) v = gelu_tanh(v);
            out[(size_t)ob * N + n] = v;
        }
    }
}

// qkv rows [rows = B*T, 3C] (q | k | v): the k and v parts go to cache[b][pos0 + t][C]
__global__ void kv_append_kernel(float4* __restrict__ kcache, float4* __restrict__ vcache,
                                 const float4* __restrict__ qkv, int B, int T, int C4, int pos0, int cache_T) {
    griddep_wait();
    griddep_launch_dependents();
    const size_t total = (size_t)B * T * C4;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % C4);
        const size_t row = i / C4;
        const int t = (int)(row % T), b = (int)(row / T);
        const size_t dst = ((size_t)b * cache_T + pos0 + t) * C4 + c;
        kcache[dst] = qkv[row * 3 * C4 + C4 + c];
        vcache[dst] = qkv[row * 3 * C4 + 2 * C4 + c];
    }
}

constexpr int kDecAttThreads = 256, kDecAttWarps = kDecAttThreads / 32;

// q: row b of qkv [B, 3C] (first C columns); caches [B][cache_T][C]; positions 0..pos take part.
// grid (splits, NH, B), a cluster of `splits` CTAs per (sequence, head): each walks its share of the positions.  Four lanes
// share a position (16 of the 64 dimensions each), so a score costs two exchanges and the weighted values none until the end; two
// positions per group of lanes are on their way at a time.  The softmax states of the groups, the warps and the CTAs are merged
// in a fixed order: exchanges, shared memory, the other CTAs' shared memory.
__global__ void __launch_bounds__(kDecAttThreads, 2)
decode_attention_kernel(float* __restrict__ out, const float* __restrict__ qkv, float* __restrict__ kcache, float* __restrict__ vcache, int C,
                        const int* __restrict__ pos_ptr, int cache_T) {
    constexpr int U = 2, GROUPS = 8, PER = kDecAttWarps * GROUPS * U;  // positions of a CTA on their way
    __shared__ float wm[kDecAttWarps], wl[kDecAttWarps], wo[kDecAttWarps][64];
    __shared__ float state[66];  // this CTA's weighted values, sum of weights, maximum
    griddep_launch_dependents();
    griddep_wait();
    const int splits = gridDim.x, z = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, j = lane & 3, grp = lane >> 2;
    // the query is requested together with the position (two independent round trips, not one after the other)
    const float* qrow = qkv + (size_t)b * 3 * C + h * 64 + j * 4;
    float4 q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const float4*>(qrow + 16 * i);
    const int pos = *pos_ptr;
    const int per = (pos + splits) / splits, t_begin = z * per, t_end = min(pos + 1, t_begin + per);
    float* kbase = kcache + (size_t)b * cache_T * C + h * 64 + j * 4;
    float* vbase = vcache + (size_t)b * cache_T * C + h * 64 + j * 4;
    // this head's slice of the new position goes into the cache; the one CTA that reads it takes it from the row itself
    if (warp == 0 && grp < 2 && pos >= t_begin && pos < t_end) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            *reinterpret_cast<float4*>((grp ? vbase : kbase) + (size_t)pos * C + 16 * i) = *reinterpret_cast<const float4*>(qrow + (1 + grp) * C + 16 * i);
    }
    const float scale = 0.125f;  // 1 / sqrt(64)
#pragma unroll
    for (int i = 0; i < 4; ++i) { q[i].x *= scale; q[i].y *= scale; q[i].z *= scale; q[i].w *= scale; }
    float m = -INFINITY, l = 0.f, o[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) o[i] = 0.f;
    for (int t0 = t_begin; t0 < t_end; t0 += PER) {
        float4 k[U][4], v[U][4];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int t = t0 + (u * kDecAttWarps + warp) * GROUPS + grp;
            const float* kp = t == pos ? qrow + C : kbase + (size_t)t * C;
            const float* vp = t == pos ? qrow + 2 * C : vbase + (size_t)t * C;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                k[u][i] = v[u][i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (t < t_end) {
                    k[u][i] = *reinterpret_cast<const float4*>(kp + 16 * i);
                    v[u][i] = *reinterpret_cast<const float4*>(vp + 16 * i);
                }
            }
        }
        float s[U], mn = m;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float d = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) d += (q[i].x * k[u][i].x + q[i].y * k[u][i].y) + (q[i].z * k[u][i].z + q[i].w * k[u][i].w);
            d += __shfl_xor_sync(0xffffffffu, d, 1);
            d += __shfl_xor_sync(0xffffffffu, d, 2);
            s[u] = t0 + (u * kDecAttWarps + warp) * GROUPS + grp < t_end ? d : -INFINITY;
            mn = fmaxf(mn, s[u]);
        }
        if (mn > -INFINITY) {
            const float corr = expf(m - mn);  // 0 on the first positions
            l *= corr;
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] *= corr;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float p = expf(s[u] - mn);
                l += p;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    o[4 * i] = fmaf(p, v[u][i].x, o[4 * i]); o[4 * i + 1] = fmaf(p, v[u][i].y, o[4 * i + 1]);
                    o[4 * i + 2] = fmaf(p, v[u][i].z, o[4 * i + 2]); o[4 * i + 3] = fmaf(p, v[u][i].w, o[4 * i + 3]);
                }
            }
            m = mn;
        }
    }
    // the warp's eight groups: element e of o is dimension 16 (e / 4) + 4 j + e % 4
    float cm = m;
#pragma unroll
    for (int s = 4; s < 32; s <<= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, s));
    const float f = m == -INFINITY ? 0.f : expf(m - cm);  // a group may have seen nothing
    l *= f;
#pragma unroll
    for (int i = 0; i < 16; ++i) o[i] *= f;
    int at = 0;
#pragma unroll
    for (int s = 4, held = 16; s < 32; s <<= 1, held >>= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, s);
        const bool up = (lane & s) != 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i < held / 2) {
                const float send = up ? o[i] : o[i + held / 2], keep = up ? o[i + held / 2] : o[i];
                o[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
            }
        if (up) at += held / 2;
    }
    *reinterpret_cast<float2*>(&wo[warp][16 * (at >> 2) + 4 * j + (at & 3)]) = make_float2(o[0], o[1]);
    if (lane == 0) { wm[warp] = cm; wl[warp] = l; }
    __syncthreads();
    if (tid < 66) {  // thread d < 64 owns dimension d; 64 and 65 the sum of weights and the maximum
        float mm = -INFINITY, acc = 0.f;
#pragma unroll
        for (int i = 0; i < kDecAttWarps; ++i) mm = fmaxf(mm, wm[i]);
#pragma unroll
        for (int i = 0; i < kDecAttWarps; ++i) acc += (tid < 64 ? wo[i][tid & 63] : wl[i]) * (wm[i] == -INFINITY ? 0.f : expf(wm[i] - mm));
        state[tid] = tid == 65 ? mm : acc;
    }
    cluster_sync_all();
    if (z == 0 && tid < 64) {
        const uint32_t mine = smem_u32(state);
        float ms[8], ls[8], os[8], mm = -INFINITY;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            ms[s] = -INFINITY; ls[s] = os[s] = 0.f;
            if (s < splits) {
                const uint32_t p = map_to_cta(mine, s);
                ms[s] = ld_cluster_f32(p + 65 * 4);
                ls[s] = ld_cluster_f32(p + 64 * 4);
                os[s] = ld_cluster_f32(p + tid * 4);
            }
            mm = fmaxf(mm, ms[s]);
        }
        float L = 0.f, O = 0.f;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const float w = ms[s] == -INFINITY ? 0.f : expf(ms[s] - mm);  // an empty share
            L += ls[s] * w;
            O += os[s] * w;
        }
        out[(size_t)b * C + h * 64 + tid] = O / L;
    }
    cluster_sync_all();  // the states have been read
}

// out[b,:] = wte[tok[b],:] + wpe[pos,:]  (one fp32 add, as the full-sequence encoder)
__global__ void decode_encoder_kernel(float4* __restrict__ out, const int* __restrict__ tok, const float4* __restrict__ wte,
                                      const float4* __restrict__ wpe, const int* __restrict__ pos_ptr, int B, int C4,
                                      int vocab_rows, int* status) {
    griddep_wait();
    griddep_launch_dependents();
    const int pos = *pos_ptr;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < B * C4; i += gridDim.x * blockDim.x) {
        const int b = i / C4, c = i % C4;
        int id = tok[b];
        if (id < 0 || id >= vocab_rows) {  // reported like the full-sequence encoder does
            atomicCAS(status, 0, 201);
            id = 0;
        }
        const float4 e = __ldg(wte + (size_t)id * C4 + c), p = __ldg(wpe + (size_t)pos * C4 + c);
        out[i] = make_float4(e.x + p.x, e.y + p.y, e.z + p.z, e.w + p.w);
    }
}

__global__ void set_int_kernel(int* dst, int value) { *dst = value; }

}  // namespace

int launch_set_int(b200_ctx* ctx, int* dst, int value) {
    set_int_kernel<<<1, 1, 0, ctx->stream>>>(dst, value);
    ctx->launches++;
    B200_CUDA(ctx, cudaGetLastError());
    return B200_OK;
}

// input rows that the kernels are built for
static int skinny_rows(int B) { return B <= 2 ? 2 : (B <= 8 ? 8 : 16); }

int launch_decode_encoder(b200_ctx* ctx, float* out, const int* tok, const float* wte, const float* wpe,
                          const int* pos_ptr, int B, int C, int vocab_rows) {
    const int n = B * (C / 4);
    cudaError_t le = launch_pdl(ctx, decode_encoder_kernel, dim3((n + 255) / 256), dim3(256), 0, reinterpret_cast<float4*>(out), tok,
                                reinterpret_cast<const float4*>(wte), reinterpret_cast<const float4*>(wpe), pos_ptr, B, C / 4,
                                vocab_rows, ctx->d_status);
    ctx->launches++;
    B200_CUDA(ctx, le);
    return B200_OK;
}

// K slices of a plain product whose input rows would take more shared memory than leaves room for a second CTA: each SM then
// stages a slice only.  The caller hands the same number to the consumer as branch_parts.
constexpr size_t kSkinnyTwoCtas = (size_t)104 * 1024, kSkinnyMost = (size_t)200 * 1024;
int skinny_gemm_k_splits(int B, int K) {
    for (int ks = 1; ks <= 4; ks <<= 1)
        if (K % (32 * ks) == 0 && (size_t)skinny_rows(B) * (K / ks) * 4 <= kSkinnyTwoCtas) return ks;
    return 1;
}

int launch_skinny_gemm(b200_ctx* ctx, float* out, const float* x, const float* W, const float* bias, int B,
                       int K, int N, int gelu, const float* branch, const float* ln_w, const float* ln_b,
                       float* resid_out, int k_splits, int branch_parts, const void* next, size_t next_bytes) {
    if (B < 1 || B > 16 || K % 4 || N < 1) return B200_ERR_SHAPE;
    if (ln_w && (K > 1664 || !ln_b || !resid_out || resid_out == x)) return B200_ERR_SHAPE;
    if (k_splits < 1 || branch_parts < 1) return B200_ERR_SHAPE;
    if (k_splits > 1 && (ln_w || gelu || K % (32 * k_splits))) return B200_ERR_SHAPE;
    const int nb = skinny_rows(B), sms = ctx->num_sms;
    const int kslice = K / k_splits;
    // (more than 8 rows of a wide product with a wide output are refused)
    if ((size_t)(B <= 8 ? 8 : 16) * K * 4 > kSkinnyMost && (k_splits == 1 || (N + 15) / 16 * 2 > sms)) return B200_ERR_LIMIT;
    const size_t smem = (size_t)nb * kslice * 4 + (ln_w ? (size_t)2 * K * 4 : 0);
    if (smem > kSkinnyMost) return B200_ERR_LIMIT;
    SkinnyArgs a;
    a.out = out; a.x = x; a.W = W; a.bias = bias; a.branch = branch; a.ln_w = ln_w; a.ln_b = ln_b; a.resid_out = resid_out;
    a.B = B; a.N = N; a.K = K; a.gelu = gelu;
    a.k_splits = k_splits; a.kslice = kslice; a.branch_parts = branch_parts;
    a.next = static_cast<const uint8_t*>(next); a.next_bytes = next_bytes & ~(size_t)15;
    // shares of the rows, one per SM (two where even half a share is long), at least four rows each; rows per lane: the
    // fewest steps for a team's half of a share, a tile's own cost being about half of a row's
    int parts = sms / k_splits;
    if (N >= 2 * sms * 64 && smem <= kSkinnyTwoCtas) parts *= 2;
    if (parts > (N + 3) / 4) parts = (N + 3) / 4;
    if (parts < 1) parts = 1;
    const int half = ((N + parts - 1) / parts + 1) / 2;
    int rows = 1, best = 0;
    for (int r = 1; r <= (nb == 16 ? 1 : (nb == 8 ? 3 : 4)); ++r) {
        if (nb == 2 && r == 3) continue;
        const int cost = (half + 4 * r - 1) / (4 * r) * (2 * r + 1);
        if (!best || cost <= best) { best = cost; rows = r; }
    }
    const dim3 grid(parts * k_splits);
    const int nv = !ln_w ? 0 : (K <= 768 ? 3 : 7);
    cudaError_t le = cudaSuccess;
#define B200_SKINNY(NB, R, NV)                                                                                      \
    do {                                                                                                            \
        static bool attr_set[64] = {};                                                                              \
        if (!attr_set[ctx->device & 63]) {                                                                          \
            B200_CUDA(ctx, cudaFuncSetAttribute(skinny_gemm_kernel<NB, R, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSkinnyMost)); \
            attr_set[ctx->device & 63] = true;                                                                      \
        }                                                                                                           \
        le = launch_pdl(ctx, skinny_gemm_kernel<NB, R, NV>, grid, dim3(kSkinnyThreads), smem, a);                   \
    } while (0)
#define B200_SKINNY_NV(NB, R) do { if (nv == 0) B200_SKINNY(NB, R, 0); else if (nv == 3) B200_SKINNY(NB, R, 3); else B200_SKINNY(NB, R, 7); } while (0)
    if (nb == 2) { if (rows == 1) B200_SKINNY_NV(2, 1); else if (rows == 2) B200_SKINNY_NV(2, 2); else B200_SKINNY_NV(2, 4); }
    else if (nb == 8) { if (rows == 1) B200_SKINNY_NV(8, 1); else if (rows == 2) B200_SKINNY_NV(8, 2); else B200_SKINNY_NV(8, 3); }
    else B200_SKINNY_NV(16, 1);
#undef B200_SKINNY_NV
#undef B200_SKINNY
    ctx->launches++;
    B200_CUDA(ctx, le);
    return B200_OK;
}

int launch_kv_append(b200_ctx* ctx, float* kcache, float* vcache, const float* qkv, int B, int T, int C, int pos0,
                     int cache_T) {
    const size_t total = (size_t)B * T * (C / 4);
    const int grid = (int)((total + 255) / 256 < (size_t)8 * ctx->num_sms ? (total + 255) / 256 : (size_t)8 * ctx->num_sms);
    cudaError_t le = launch_pdl(ctx, kv_append_kernel, dim3(grid), dim3(256), 0, reinterpret_cast<float4*>(kcache),
                                reinterpret_cast<float4*>(vcache), reinterpret_cast<const float4*>(qkv), B, T, C / 4,
                                pos0, cache_T);
    ctx->launches++;
    B200_CUDA(ctx, le);
    return B200_OK;
}

// CTAs per (sequence, head): eight while all of them are resident at once (two per SM), at least two
int launch_decode_attention(b200_ctx* ctx, float* out, const float* qkv, float* kcache, float* vcache, int B, int C,
                            int NH, const int* pos_ptr, int cache_T) {
    int splits = 8;
    while (splits > 2 && B * NH * splits > 2 * ctx->num_sms) splits >>= 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits, NH, B);
    cfg.blockDim = dim3(kDecAttThreads);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->pdl ? 2 : 1;
    cudaError_t le = cudaLaunchKernelEx(&cfg, decode_attention_kernel, out, qkv, kcache, vcache, C, pos_ptr, cache_T);
    ctx->launches++;
    B200_CUDA(ctx, le);
    return B200_OK;
}

}  // namespace b200
