// Gated delta rule: per head a state matrix S [D, V] in 32-bit, carried between steps.  For each token
//
//   S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
//
// (the read-out sees the token's own write), with q and k unit vectors per head (q also times D^-1/2),
// beta = sigmoid(b), g = exp(-exp(A_log) softplus(a + dt_bias)): one decay per head, or (`channel`) one per head and
// key channel, g [H, D], which then scales the rows of S one by one (a and dt_bias are [H D] wide, A_log stays per
// head).  The output gate is silu or (`gate_act` 1) a sigmoid.  A step of single tokens is one kernel (a block per
// request and head does all of it); spans of rows go one of two ways, which differ by rounding only:
//   * the walk (any sizes, both modes; shorter spans).  `prepare`: unit norms, beta and g for every row, all 32-bit.  The
//     recurrence: the columns of S are independent, so a block owns some columns of one head of one request and walks the
//     request's rows in order; P lanes of a warp share a column, each with DP of its D rows in registers; the operands of the
//     next sixteen tokens come into shared memory by asynchronous copies while the current sixteen are computed.
//   * chunks of 64 rows (bfloat16, longer spans, keys of up to 64): further below.
// The output norm is a kernel of its own: o / rms(o) * weight * silu(gate) per head, rounded to the model's dtype.
#include <cstdlib>
#include "mma_helpers.cuh"

__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(expf(v)); }

// qk_out [N, 2, G, D]: q then k, unit length (+ eps inside the root), q times D^-1/2;  bg_out [N, 2, H]: beta, g
// gch_out (channel decays only) [N, H, D]: g per head and key channel; bg_out then holds beta alone
template <typename T>
__global__ void delta_prepare_kernel(float* __restrict__ qk_out, float* __restrict__ bg_out, float* __restrict__ gch_out,
                                     const T* __restrict__ qkv, int qkv_stride, const T* __restrict__ b_in, int b_stride,
                                     const T* __restrict__ a_in, int a_stride, const float* __restrict__ a_log,
                                     const float* __restrict__ dt_bias, int H, int G, int D, float unit_eps,
                                     const int* __restrict__ cu_q, const int* __restrict__ seq_idx, int max_rows) {
    pdl_trigger();
    pdl_wait();
    if (seq_idx) {                                     // (rows of longer spans are another kernel's)
        const int s = seq_idx[blockIdx.x];
        if (cu_q[s + 1] - cu_q[s] > max_rows) return;
    }
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    const float q_scale = rsqrtf((float)D);
    for (int item = warp; item < 2 * G; item += nwarp) {
        const T* src = qkv + (size_t)t * qkv_stride + (size_t)item * D;       // q heads, then k heads
        float ss = 0.f;
        for (int d = lane; d < D; d += 32) {
            const float v = to_float(src[d]);
            ss += v * v;
        }
        ss = warp_sum(ss);
        const float inv = rsqrtf(ss + unit_eps) * (item < G ? q_scale : 1.f);
        float* dst = qk_out + ((size_t)t * 2 * G + item) * D;
        for (int d = lane; d < D; d += 32) dst[d] = to_float(src[d]) * inv;
    }
    for (int h = threadIdx.x; h < H; h += blockDim.x) {
        const float b = to_float(b_in[(size_t)t * b_stride + h]);
        bg_out[(size_t)t * 2 * H + h] = 1.f / (1.f + expf(-b));
        if (!gch_out) {
            const float a = to_float(a_in[(size_t)t * a_stride + h]);
            bg_out[(size_t)t * 2 * H + H + h] = expf(-expf(a_log[h]) * softplus_f(a + dt_bias[h]));
        }
    }
    if (gch_out) {
        for (int i = threadIdx.x; i < H * D; i += blockDim.x) {
            const float a = to_float(a_in[(size_t)t * a_stride + i]);
            gch_out[(size_t)t * H * D + i] = expf(-expf(a_log[i / D]) * softplus_f(a + dt_bias[i]));
        }
    }
}

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The operands of TB tokens (a stage of the ring; fewer where a head is large, so that two stages fit) in shared memory: per token k and q of the head (each P groups of DP values,
// a group padded to DP + 4 so that the P groups read by one warp lie in different banks, 16-byte aligned), beta, g,
// and the block's columns of v as 32-bit values.
// With channel decays a token also brings its head's D decays (a third group laid out like k and q), and a stage holds
// fewer tokens where a head is large.
template <int DP, int P, bool CH>
struct DeltaStage {
    static constexpr int GROUP = DP + 4, KQ = P * GROUP, VB = 128 / P, NG = CH ? 3 : 2, PER_TOKEN = NG * KQ + 4 + VB;
    static constexpr int TB = CH ? (DP * P > 128 ? 4 : (DP * P > 64 ? 8 : 16)) : (DP * P > 128 ? 8 : 16);
};

template <typename T, int DP, int P, bool CH>
__global__ void __launch_bounds__(128) gated_delta_kernel(
    float* __restrict__ o_out, const float* __restrict__ qk, const float* __restrict__ bg, const float* __restrict__ gch,
    const T* __restrict__ v_in,
    int v_stride, float* __restrict__ state, const int* __restrict__ cu_q, const int* __restrict__ slot_ids, int H, int G,
    int D, int V, int write_state, int num_slots, int* __restrict__ status, int max_rows) {
    using St = DeltaStage<DP, P, CH>;
    constexpr int VB = St::VB, TB = St::TB, NG = St::NG;
    __shared__ __align__(16) float ring[2][TB][St::PER_TOKEN];
    pdl_trigger();
    pdl_wait();
    const int seq = blockIdx.x, h = blockIdx.y, p = threadIdx.x % P, jl = threadIdx.x / P;
    const int j0 = blockIdx.z * VB;
    int j = j0 + jl;
    const bool live = j < V;
    if (!live) j = V - 1;                              // (stays for the shuffles, stores nothing)
    const int start = cu_q[seq], end = cu_q[seq + 1];
    if (end <= start || end - start > max_rows) return;
    const int slot = zai_checked_slot(slot_ids[seq], num_slots, status);
    const int kvh = h / (H / G), d0 = p * DP;
    float* st = state + (((size_t)slot * H + h) * D) * V + j;
    float S[DP];
#pragma unroll
    for (int i = 0; i < DP; ++i) S[i] = d0 + i < D ? st[(size_t)(d0 + i) * V] : 0.f;
    for (int i = threadIdx.x; i < 2 * TB * St::PER_TOKEN; i += 128) (&ring[0][0][0])[i] = 0.f;   // rows of k, q beyond D stay zero
    __syncthreads();

    // a stage's k, q, beta, g by asynchronous copies; its v columns through registers (converted to 32-bit)
    constexpr int V_PER_THREAD = (TB * VB + 127) / 128;
    float v_regs[V_PER_THREAD];
    auto issue = [&](int t0, int buf) {
        const int n = min(TB, end - t0);
        for (int r = threadIdx.x; r < NG * D; r += 128) {                                 // an element of k | q (| g), for every token
            const int which = r / D, d = r - which * D;                                   // which: 0 k, 1 q, 2 the channel decays
            const float* src = which == 2 ? gch + ((size_t)t0 * H + h) * D + d : qk + ((size_t)t0 * 2 * G + (which ? 0 : G) + kvh) * D + d;
            const size_t step = which == 2 ? (size_t)H * D : (size_t)2 * G * D;
            float* dst = &ring[buf][0][which * St::KQ + (d / DP) * St::GROUP + d % DP];
            for (int tok = 0; tok < n; ++tok) cp_async4(dst + tok * St::PER_TOKEN, src + tok * step);
        }
        for (int i = threadIdx.x; i < n * 2; i += 128) {
            const int tok = i / 2, which = i % 2;                                        // 0 beta, 1 g
            cp_async4(&ring[buf][tok][NG * St::KQ + which], bg + (size_t)(t0 + tok) * 2 * H + which * H + h);
        }
#pragma unroll
        for (int e = 0; e < V_PER_THREAD; ++e) {
            const int i = threadIdx.x + e * 128, tok = i / VB, col = i % VB;
            v_regs[e] = (tok < n && j0 + col < V) ? to_float(v_in[(size_t)(t0 + tok) * v_stride + (size_t)h * V + j0 + col]) : 0.f;
        }
    };
    auto land = [&](int buf) {
        cp_async_wait_all();
#pragma unroll
        for (int e = 0; e < V_PER_THREAD; ++e) {
            const int i = threadIdx.x + e * 128, tok = i / VB, col = i % VB;
            if (tok < TB) ring[buf][tok][NG * St::KQ + 4 + col] = v_regs[e];
        }
        __syncthreads();
    };
    issue(start, 0);
    land(0);
    int buf = 0, pend_t = -1;
    float pend_out = 0.f;
    for (int t0 = start; t0 < end; t0 += TB, buf ^= 1) {
        const bool more = t0 + TB < end;
        if (more) issue(t0 + TB, buf ^ 1);
        const int n = min(TB, end - t0);
        for (int tok = 0; tok < n; ++tok) {
            const float* row = ring[buf][tok];
            float kc[DP], qc[DP], gc[CH ? DP : 1];
#pragma unroll
            for (int i = 0; i < DP; i += 4) {
                const float4 a = *reinterpret_cast<const float4*>(row + p * St::GROUP + i);
                const float4 b = *reinterpret_cast<const float4*>(row + St::KQ + p * St::GROUP + i);
                kc[i] = a.x; kc[i + 1] = a.y; kc[i + 2] = a.z; kc[i + 3] = a.w;
                qc[i] = b.x; qc[i + 1] = b.y; qc[i + 2] = b.z; qc[i + 3] = b.w;
                if (CH) {
                    const float4 c = *reinterpret_cast<const float4*>(row + 2 * St::KQ + p * St::GROUP + i);
                    gc[i] = c.x; gc[i + 1] = c.y; gc[i + 2] = c.z; gc[i + 3] = c.w;
                }
            }
            const float beta = row[NG * St::KQ], g = row[NG * St::KQ + 1], vv = row[NG * St::KQ + 4 + jl];
            // a warp issues in order: four short chains of multiply-adds instead of one long one, and the last
            // token's read-out is summed over the lanes beside this token's S^T k (two exchanges in flight at once)
            float d4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < DP; ++i) {
                S[i] *= CH ? gc[i] : g;
                d4[i & 3] += S[i] * kc[i];
            }
            float dot = (d4[0] + d4[1]) + (d4[2] + d4[3]);
            float po = pend_out;
#pragma unroll
            for (int o = P / 2; o > 0; o >>= 1) {
                dot += __shfl_xor_sync(0xffffffffu, dot, o);
                po += __shfl_xor_sync(0xffffffffu, po, o);
            }
            if (pend_t >= 0 && p == 0 && live) o_out[(size_t)pend_t * H * V + (size_t)h * V + j] = po;
            const float u = beta * (vv - dot);
            float o4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < DP; ++i) {
                S[i] += kc[i] * u;
                o4[i & 3] += S[i] * qc[i];
            }
            pend_out = (o4[0] + o4[1]) + (o4[2] + o4[3]);
            pend_t = t0 + tok;
        }
        if (more) land(buf ^ 1);
    }
    {
        float po = pend_out;                           // the last token's read-out
#pragma unroll
        for (int o = P / 2; o > 0; o >>= 1) po += __shfl_xor_sync(0xffffffffu, po, o);
        if (pend_t >= 0 && p == 0 && live) o_out[(size_t)pend_t * H * V + (size_t)h * V + j] = po;
    }
    if (write_state && live) {
#pragma unroll
        for (int i = 0; i < DP; ++i)
            if (d0 + i < D) st[(size_t)(d0 + i) * V] = S[i];
    }
}

__device__ __forceinline__ float delta_gate(float gv, int gate_act) {       // 0: silu, 1: sigmoid
    const float s = 1.f / (1.f + expf(-gv));
    return gate_act ? s : gv * s;
}

// out[t, h, :] = o[t, h, :] * rsqrt(mean(o^2) + eps) * w * act(gate[t, h, :]); one warp per (row, head)
template <typename T>
__global__ void gated_rmsnorm_kernel(T* __restrict__ out, const float* __restrict__ o, const float* __restrict__ w,
                                     const T* __restrict__ gate, int gate_stride, float eps, int items, int H, int V,
                                     int gate_act) {
    pdl_trigger();
    pdl_wait();
    const int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (item >= items) return;
    const int t = item / H, h = item % H;
    const float* src = o + (size_t)item * V;
    float ss = 0.f;
    for (int d = lane; d < V; d += 32) ss += src[d] * src[d];
    ss = warp_sum(ss);
    const float inv = rsqrtf(ss / (float)V + eps);
    const T* grow = gate + (size_t)t * gate_stride + (size_t)h * V;
    for (int d = lane; d < V; d += 32) {
        const float gv = to_float(grow[d]);
        out[(size_t)item * V + d] = from_float<T>(src[d] * inv * (w ? w[d] : 1.f) * delta_gate(gv, gate_act));
    }
}

// The same for head sizes 4 L R: L lanes an item, four neighbouring columns a lane and load (R times), all of them asked for before the
// sum.  What bounds it is memory (8 bytes a column in bfloat16); with one column a lane and load the warps waited for loads one after
// another: 2048 rows of 32 heads of 128 25.5 -> 19.3 us, of 64 22.2 -> 10.8; of a delta layer of 2048 rows 226 -> 224.
template <typename T>
__device__ __forceinline__ void delta_four(const T* p, float (&v)[4]) {
    if (sizeof(T) == 4) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    } else {
        const uint2 x = *reinterpret_cast<const uint2*>(p);
        v[0] = __uint_as_float(x.x << 16), v[1] = __uint_as_float(x.x & 0xffff0000u);
        v[2] = __uint_as_float(x.y << 16), v[3] = __uint_as_float(x.y & 0xffff0000u);
    }
}
template <typename T, int L, int R>
__global__ void gated_rmsnorm_wide_kernel(T* __restrict__ out, const float* __restrict__ o, const float* __restrict__ w,
                                          const T* __restrict__ gate, int gate_stride, float eps, int items, int H, int gate_act) {
    constexpr int V = 4 * L * R;
    const int lane = threadIdx.x % L, mine = blockIdx.x * (blockDim.x / L) + threadIdx.x / L;
    const int item = min(mine, items - 1);                            // (the last block's spare lanes take part in the sums)
    const int t = item / H, h = item % H;
    pdl_trigger();
    float scale[R][4], x[R][4], g[R][4];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (w) delta_four(w + 4 * (lane + r * L), scale[r]);
        else scale[r][0] = scale[r][1] = scale[r][2] = scale[r][3] = 1.f;
    }
    pdl_wait();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        delta_four(o + (size_t)item * V + 4 * (lane + r * L), x[r]);
        delta_four(gate + (size_t)t * gate_stride + (size_t)h * V + 4 * (lane + r * L), g[r]);
    }
    float ss = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) ss += x[r][e] * x[r][e];
#pragma unroll
    for (int d = L / 2; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
    const float inv = rsqrtf(ss / (float)V + eps);
    if (mine >= items) return;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        T* dst = out + (size_t)item * V + 4 * (lane + r * L);
        __align__(16) T y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = from_float<T>(x[r][e] * inv * scale[r][e] * delta_gate(g[r][e], gate_act));
        if (sizeof(T) == 4) *reinterpret_cast<float4*>(dst) = *reinterpret_cast<const float4*>(y);
        else *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(y);
    }
}

// ---- a step of single tokens in one kernel: unit norms, beta and g, the state's update and read-out and the output
// norm for one head of one request per block (all V columns: P lanes a column, so P * V threads, at most 1024)
template <typename T, int DP, int P>
__global__ void __launch_bounds__(1024) gated_delta_single_kernel(
    T* __restrict__ out, const T* __restrict__ qkv, int qkv_stride, const T* __restrict__ b_in, int b_stride,
    const T* __restrict__ a_in, int a_stride, const T* __restrict__ gate, int gate_stride, const float* __restrict__ a_log,
    const float* __restrict__ dt_bias, const float* __restrict__ norm_w, float eps, float unit_eps, float* __restrict__ state,
    const int* __restrict__ slot_ids, int H, int G, int D, int V, int write_state, int num_slots, int* __restrict__ status,
    int channel, int gate_act) {
    extern __shared__ float sm[];                      // q [D], k [D], the decays [D], 33 for the block's sum
    float* qs = sm;
    float* ks = sm + D;
    float* gs = sm + 2 * D;
    float* red = sm + 3 * D;
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x, h = blockIdx.y, kvh = h / (H / G);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    const T* row = qkv + (size_t)t * qkv_stride;
    for (int item = warp; item < 2; item += nwarp) {                  // 0: q, 1: k of this head's q/k head
        const T* src = row + (size_t)(item * G + kvh) * D;
        float ss = 0.f;
        for (int d = lane; d < D; d += 32) {
            const float v = to_float(src[d]);
            ss += v * v;
        }
        ss = warp_sum(ss);
        const float inv = rsqrtf(ss + unit_eps) * (item == 0 ? rsqrtf((float)D) : 1.f);
        float* dst = item == 0 ? qs : ks;
        for (int d = lane; d < D; d += 32) dst[d] = to_float(src[d]) * inv;
    }
    {
        const float rate = expf(a_log[h]);
        for (int d = threadIdx.x; d < D; d += blockDim.x) {
            const int i = channel ? h * D + d : h;
            gs[d] = expf(-rate * softplus_f(to_float(a_in[(size_t)t * a_stride + i]) + dt_bias[i]));
        }
    }
    __syncthreads();
    const float beta = 1.f / (1.f + expf(-to_float(b_in[(size_t)t * b_stride + h])));
    const int p = threadIdx.x % P, d0 = p * DP;
    int j = threadIdx.x / P;
    const bool live = j < V;
    if (!live) j = V - 1;
    const int slot = zai_checked_slot(slot_ids[t], num_slots, status);
    float* st = state + (((size_t)slot * H + h) * D) * V + j;
    float S[DP];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < DP; ++i) {
        S[i] = d0 + i < D ? st[(size_t)(d0 + i) * V] * gs[d0 + i] : 0.f;
        dot += d0 + i < D ? S[i] * ks[d0 + i] : 0.f;
    }
#pragma unroll
    for (int o = P / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    const float u = beta * (to_float(row[(size_t)2 * G * D + (size_t)h * V + j]) - dot);
    float o_j = 0.f;
#pragma unroll
    for (int i = 0; i < DP; ++i) {
        if (d0 + i < D) {
            S[i] += ks[d0 + i] * u;
            o_j += S[i] * qs[d0 + i];
            if (write_state && live) st[(size_t)(d0 + i) * V] = S[i];
        }
    }
#pragma unroll
    for (int o = P / 2; o > 0; o >>= 1) o_j += __shfl_xor_sync(0xffffffffu, o_j, o);
    const float ss = block_sum((p == 0 && live) ? o_j * o_j : 0.f, red);
    const float inv = rsqrtf(ss / (float)V + eps);
    if (p == 0 && live) {
        const float gv = to_float(gate[(size_t)t * gate_stride + (size_t)h * V + j]);
        out[((size_t)t * H + h) * V + j] = from_float<T>(o_j * inv * (norm_w ? norm_w[j] : 1.f) * delta_gate(gv, gate_act));
    }
}

template <typename T, int DP, int P>
static int launch_delta_single(void* out, const void* qkv, int qkv_stride, const void* b_in, int b_stride, const void* a_in,
                               int a_stride, const void* gate, int gate_stride, const float* a_log, const float* dt_bias,
                               const float* norm_w, float eps, float unit_eps, float* state, const int* slot_ids, int B, int H, int G,
                               int D, int V, int write_state, int num_slots, int* status, int channel, int gate_act,
                               cudaStream_t stream) {
    const int threads = ((P * V + 31) / 32) * 32;
    if (threads > 1024) return ZAI_BAD_SIZE;
    return launch_pdl(gated_delta_single_kernel<T, DP, P>, dim3(B, H), dim3(threads), (size_t)(3 * D + 33) * sizeof(float), stream,
                      (T*)out, (const T*)qkv, qkv_stride, (const T*)b_in, b_stride, (const T*)a_in, a_stride, (const T*)gate,
                      gate_stride, a_log, dt_bias, norm_w, eps, unit_eps, state, slot_ids, H, G, D, V, write_state, num_slots, status,
                      channel, gate_act);
}

// 1 if a step of single tokens with these sizes can run as the one kernel above
ZAI_API int zai_gated_delta_single_supports(int D, int V) {
    const int P = D <= 128 ? 4 : 8;
    return D >= 1 && D <= 256 && V >= 1 && ((P * V + 31) / 32) * 32 <= 1024;
}

// out [B, H*V] in the model's dtype; qkv [B, qkv_stride] (q heads, k heads, v heads, after their convolutions);
// b_in [B, b_stride] (H values a row); a_in [B, a_stride] (H values a row, or H D with `channel`); gate [B, gate_stride];
// state [slots, H, D, V]; row i belongs to slot_ids[i]
ZAI_API int zai_gated_delta_single(void* out, const void* qkv, int qkv_stride, const void* b_in, int b_stride, const void* a_in,
                                   int a_stride, const void* gate, int gate_stride, int dtype, const float* a_log,
                                   const float* dt_bias, const float* norm_w, float eps, float unit_eps, float* state,
                                   const int* slot_ids, int B, int H, int G, int D, int V, int write_state, int num_slots, int* status,
                                   int channel, int gate_act, cudaStream_t stream) {
    if (B <= 0) return ZAI_OK;
    if (!zai_gated_delta_single_supports(D, V) || G < 1 || H % G != 0 || H > 65535) return ZAI_BAD_SIZE;
#define ZAI_DELTA1(DPV, PV) ZAI_DISPATCH(dtype, return launch_delta_single<T, DPV, PV>(out, qkv, qkv_stride, b_in, b_stride, a_in, a_stride, \
        gate, gate_stride, a_log, dt_bias, norm_w, eps, unit_eps, state, slot_ids, B, H, G, D, V, write_state, num_slots, status, channel, \
        gate_act, stream))
    if (D <= 16) ZAI_DELTA1(4, 4);
    if (D <= 32) ZAI_DELTA1(8, 4);
    if (D <= 64) ZAI_DELTA1(16, 4);
    if (D <= 128) ZAI_DELTA1(32, 4);
    ZAI_DELTA1(32, 8);
#undef ZAI_DELTA1
}

// gch_out null: one decay per head (into bg_out); else the decays per head and key channel [N, H, D].  With seq_idx [N] (the
// rows' requests) only rows of spans of at most max_rows rows are made.
ZAI_API int zai_delta_prepare(float* qk_out, float* bg_out, float* gch_out, const void* qkv, int qkv_stride, const void* b_in,
                              int b_stride, const void* a_in, int a_stride, int dtype, const float* a_log, const float* dt_bias,
                              int N, int H, int G, int D, float unit_eps, const int* cu_q, const int* seq_idx, int max_rows,
                              cudaStream_t stream) {
    if (N <= 0) return ZAI_OK;
    ZAI_DISPATCH(dtype, return launch_pdl(delta_prepare_kernel<T>, dim3(N), dim3(128), 0, stream, qk_out, bg_out, gch_out,
        (const T*)qkv, qkv_stride, (const T*)b_in, b_stride, (const T*)a_in, a_stride, a_log, dt_bias, H, G, D, unit_eps, cu_q,
        seq_idx, max_rows));
}

// Dynamic shared memory that keeps more than `per_sm` blocks of `kernel` off one SM.  The recurrence is a chain of
// dependent instructions per warp, so a block runs fastest with an SM's schedulers to itself; but a grid that is
// launched while the kernel before it still drains (as dependent launches are) is placed on the first SMs that have
// room, several blocks to an SM with other SMs left empty (measured: 64 blocks after a large kernel, 1130 us instead
// of 640).  Unused shared memory makes the placement even whatever runs before.
template <typename K>
static size_t delta_spread_smem(K kernel, long long blocks) {
    static int sms = 0, sm_smem = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaDeviceGetAttribute(&sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
        if (sms < 1) sms = 1;
    }
    const long long per_sm = (blocks + sms - 1) / sms;
    if (per_sm >= 4) return 0;
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) return 0;
    // every block takes its static and dynamic bytes and 1 KB of the system's: per_sm blocks fit, per_sm + 1 do not
    const long long each = sm_smem / per_sm - 1024 - (long long)fa.sharedSizeBytes - 1024;
    const long long next = sm_smem / (per_sm + 1) - 1024 - (long long)fa.sharedSizeBytes;
    if (each <= 0 || each <= next) return 0;
    const long long dyn = each > 160 * 1024 ? 160 * 1024 : each;
    if (dyn <= next || dyn <= 0) return 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn) != cudaSuccess) { cudaGetLastError(); return 0; }
    return (size_t)dyn;
}

template <typename T, int DP, int P>
static int launch_delta(float* o_out, const float* qk, const float* bg, const float* gch, const void* v_in, int v_stride,
                        float* state, const int* cu_q, const int* slot_ids, int n_seqs, int H, int G, int D, int V, int write_state,
                        int num_slots, int* status, int max_rows, cudaStream_t stream) {
    const int vb = 128 / P;
    const dim3 grid(n_seqs, H, (V + vb - 1) / vb);
    const long long blocks = (long long)grid.x * grid.y * grid.z;
    if (gch)
        return launch_pdl(gated_delta_kernel<T, DP, P, true>, grid, dim3(128), delta_spread_smem(gated_delta_kernel<T, DP, P, true>, blocks),
                          stream, o_out, qk, bg, gch, (const T*)v_in, v_stride, state, cu_q, slot_ids, H, G, D, V, write_state, num_slots,
                          status, max_rows);
    return launch_pdl(gated_delta_kernel<T, DP, P, false>, grid, dim3(128), delta_spread_smem(gated_delta_kernel<T, DP, P, false>, blocks),
                      stream, o_out, qk, bg, gch, (const T*)v_in, v_stride, state, cu_q, slot_ids, H, G, D, V, write_state, num_slots,
                      status, max_rows);
}

// o_out [N, H*V] 32-bit; qk, bg (and gch, or null) from zai_delta_prepare; v_in [N, v_stride] (heads of V values);
// state [slots, H, D, V]; only spans of at most max_rows rows are run
ZAI_API int zai_gated_delta(float* o_out, const float* qk, const float* bg, const float* gch, const void* v_in, int v_stride,
                            int dtype, float* state, const int* cu_q, const int* slot_ids, int N, int n_seqs, int H, int G, int D,
                            int V, int write_state, int num_slots, int* status, int max_rows, cudaStream_t stream) {
    if (N <= 0 || n_seqs <= 0) return ZAI_OK;
    if (D < 1 || D > 256 || V < 1 || G < 1 || H % G != 0 || H > 65535 || V > 65535 * 16) return ZAI_BAD_SIZE;
#define ZAI_DELTA(DPV, PV) ZAI_DISPATCH(dtype, return launch_delta<T, DPV, PV>(o_out, qk, bg, gch, v_in, v_stride, state, cu_q, \
        slot_ids, n_seqs, H, G, D, V, write_state, num_slots, status, max_rows, stream))
    // four lanes a column (eight for the largest heads): measured against two and one (fewer exchanges, longer
    // chains of multiply-adds a lane), four was the fastest or level at 64-wide heads
    if (D <= 16) ZAI_DELTA(4, 4);
    if (D <= 32) ZAI_DELTA(8, 4);
    if (D <= 64) ZAI_DELTA(16, 4);
    if (D <= 128) ZAI_DELTA(32, 4);
    ZAI_DELTA(32, 8);
#undef ZAI_DELTA
}

ZAI_API int zai_gated_rmsnorm(void* out, const float* o, const float* w, const void* gate, int gate_stride, int dtype, float eps,
                              int N, int H, int V, int gate_act, cudaStream_t stream) {
    const long long items = (long long)N * H;
    if (items <= 0) return ZAI_OK;
    const long long blocks = (items + 3) / 4;
    if (blocks > 0x7fffffffLL) return ZAI_BAD_SIZE;
    // four columns a load: the head sizes that designs have, where every row starts on such a load's boundary
    const uintptr_t ends = reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(gate);
    if ((ends & 15) == 0 && gate_stride % 4 == 0 && (V == 32 || V == 64 || V == 128 || V == 256)) {
#define ZAI_GATED(L, R)                                                                                                              \
    ZAI_DISPATCH(dtype, return launch_pdl(gated_rmsnorm_wide_kernel<T, L, R>, dim3((unsigned)((items + 128 / L - 1) / (128 / L))), \
        dim3(128), 0, stream, (T*)out, o, w, (const T*)gate, gate_stride, eps, (int)items, H, gate_act))
        if (V == 32) ZAI_GATED(8, 1);
        else if (V == 64) ZAI_GATED(16, 1);
        else if (V == 128) ZAI_GATED(32, 1);
        else ZAI_GATED(32, 2);
#undef ZAI_GATED
    }
    ZAI_DISPATCH(dtype, return launch_pdl(gated_rmsnorm_kernel<T>, dim3((unsigned)blocks), dim3(128), 0, stream, (T*)out, o, w,
        (const T*)gate, gate_stride, eps, (int)items, H, V, gate_act));
}

// ------------------------------------------------------------------------------------------------ chunks
// The walk is a chain of one request's rows (0.28 us a row on a fraction of the SMs).  A portion of a prompt is cut into chunks
// of DC rows instead.  With c_t the running sum of the log decays from the chunk's first row (one number a head, or one a key
// channel) and S_0 the state before the chunk, the rule unrolls to
//
//   u_t = beta_t (v_t - S_0^T (e^(c_t) k_t) - sum_{s<t} A_ts u_s),    A_ts = sum_d k_t k_s e^(c_t - c_s)
//   o_t = S_0^T (e^(c_t) q_t) + sum_{s<=t} P_ts u_s,                  P_ts = sum_d q_t k_s e^(c_t - c_s)
//   S   = e^(c_last) S_0 + sum_s (e^(c_last - c_s) k_s) u_s^T
//
// The first line is a triangular system with the same matrix for every column: its solution for the right sides beta_t v_t (U0)
// and beta_t e^(c_t) k_t (W) needs no state, and u = U0 - W S_0.  Two kernels:
//   * `delta_chunk_kernel`, every chunk and head at once: unit norms, decays, A, P, and the system solved in four steps of 16 rows,
//     16 right sides a warp: 32-bit substitution among the 16, their part in later rows on the tensor cores.  A and P are products
//     of bfloat16 rows, or, with a decay per channel, of rows in three parts scaled by e^(c_t - c_first) and e^(c_first - c_s) around the
//     first of 16 rows; inside 16 rows that decay by more than 2^-100 the pairs of rows are taken one by one instead.  Running
//     sums are made in 64-bit and kept in two parts, so that a difference of two is good to the last bits.
//   * `delta_carry_kernel`, a block a head and DN columns of S: carries S across a request's chunks on the tensor cores (four
//     warps: u, then the new S) and makes the chunks' read-outs beside that (four more warps).  S, u, W, P and the scaled k and q
//     are 32-bit and go into bfloat16 products as sums of three parts (24 bits; the six products that reach 2^-24 of the
//     result), with 32-bit sums by size.  What comes from the first kernel is laid out as a lane's operands of one m16n8k16
//     product lie, three parts beforehand: 16 bytes a load, nothing to convert.
// 2048 rows of 16 heads of 64 x 128 (norms, recurrence and output norm): 136 us where the walk takes 480, with a decay per channel
// 172 (601); of 32 heads 233 (581) and 292 (660), before the first kernel's system went to the tensor cores.  The first kernel (16 heads
// of 2048 rows, a decay per channel: 91 us with a right side a thread, 65 now; 32 heads of 1300 rows, one per head: 77 and 62) is bound by
// the instructions that a block issues (some 60 000, at half of what two blocks an SM could), the second (58) by a chunk's two
// dependent products, 1.8 us a chunk at 43 % of the tensor pipe.
#define DC 64                       // rows of a chunk
#define DCD 64                      // key size the chunk kernels are made for (smaller heads are filled up with zeros)
#define DC_LD 68                    // 32-bit row stride in shared memory

// A 64 x 64 operand of the carry in three parts: [part][tile of 16 rows][tile of 16 columns][lane], a lane's four registers
struct DeltaOperand { uint4 v[3][4][4][32]; };
struct DeltaChunk {                 // what the first kernel leaves for a chunk and head (U0 lies behind all of them)
    DeltaOperand w, k, q, p;        // W [t, d]; e^(c_last - c_s) k_s [d, s]; e^(c_t) q_t [t, d]; P [t, s]
    float keep[DCD];                // e^(c_last)
};

struct DeltaArgs {
    const bf16* qkv;                // [N, qkv_stride]: q heads, k heads, v heads
    const bf16 *b, *a;              // [N, b_stride] (H a row), [N, a_stride] (H, or H D with a decay per channel)
    int qkv_stride, b_stride, a_stride;
    const float *a_log, *dt_bias;
    float unit_eps;
    float* state;                   // [num_slots, H, D, V]
    const int *cu_q, *slot_ids;
    int* status;
    int num_slots, n_seqs, H, G, D, V, write_state, min_rows;
    DeltaChunk* chunks;             // [chunks, H]
    float* u0;                      // [chunks, H, DC, VP]
    int VP;                         // V rounded up to 32
    float* o;                       // [N, H V]
};

// Chunk b among all chunks of the step: the spans of min_rows rows or more in order, each cut into chunks of DC rows.
__device__ __forceinline__ bool delta_find_chunk(const DeltaArgs& a, int b, int& t0, int& t1) {
    for (int s = 0; s < a.n_seqs; ++s) {
        const int lo = a.cu_q[s], hi = a.cu_q[s + 1];
        if (hi - lo < a.min_rows) continue;
        const int n = (hi - lo + DC - 1) / DC;
        if (b < n) {
            t0 = lo + b * DC;
            t1 = min(t0 + DC, hi);
            return true;
        }
        b -= n;
    }
    return false;
}

__device__ __forceinline__ float delta_minus(float2 a, float2 b) { return (a.x - b.x) + (a.y - b.y); }
// log decay in units of ln 2.  Below 2^-1000 a decay is zero in 32-bit however it is split up: the sums stay finite.
__device__ __forceinline__ double delta_log_decay(float rate, float a) {
    const double l = -1.4426950408889634 * (double)(rate * softplus_f(a));
    return l < -1000.0 ? -1000.0 : l;
}
// 2^(x + y) for a small y
__device__ __forceinline__ float delta_exp2(float x, float y) {
    const float e = fast_exp2(x);
    return fmaf(e, 0.69314718f * y, e);
}

// an 8 x 8 matrix of 16-bit values, a row four lanes: its rows become its columns
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t v) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
// 16 sums over 16 neighbouring lanes at once: lane i of the 16 ends with the sum of v[i] in v[0]
__device__ __forceinline__ void sum16(float (&v)[16], int lane) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
}

// Writes an operand: get(row, column) gives two neighbouring columns (the first even); all 256 threads
template <typename F>
__device__ __forceinline__ void delta_put(DeltaOperand* out, F get) {
#pragma unroll 1
    for (int i = threadIdx.x; i < 4 * 4 * 32; i += 256) {
        const int lane = i & 31, kt = (i >> 5) & 3, mt = i >> 7, g = lane >> 2, tq = lane & 3;
        uint32_t part[4][3];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int row = mt * 16 + g + 8 * (r & 1), col = kt * 16 + 2 * tq + 8 * (r >> 1);
            const float2 x = get(row, col);
            split3_pair(x.x, x.y, part[r]);
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) out->v[p][mt][kt][lane] = make_uint4(part[0][p], part[1][p], part[2][p], part[3][p]);
    }
}

#define DR_LD (DCD + 8)             // bfloat16 row stride of rows in shared memory
#define DELTA_V_MAX 256             // value sizes up to which a chunk's rows of v are put into shared memory
#define DELTA_FAST 100.f            // log2 decays over 16 rows up to which e^(-c) is kept as a number of its own

struct DeltaShared {
    bf16 qk[2][DC][DR_LD];                                   // the rows of q and k as they came
    float inv[2][DC];                                        // what makes them unit rows (q: times D^-1/2)
    union {
        struct {
            bf16 left[2][3][16][DR_LD];                      // 16 rows of q and k times e^(c_t - c at their first), in three parts
            bf16 right[3][DC][DR_LD];                        // the rows of k up to them times e^(c at their first - c_s), likewise
        };
        bf16 a[DC][DR_LD];                                   // before that: what the decays per channel are made of
        bf16 v[DC * (DELTA_V_MAX + 8)];                      // then: the rows of v, V + 8 values apart
    };
    float m[DC][DC_LD];                                      // beta_t A_ts below the diagonal
    struct {
        float hi[DC][DCD];                                   // running log decays inside the 16 rows (one column: the chunk's), in
        bf16 lo[DC][DCD];                                    // two parts (32 bits of their sums)
    } c;
    float sum[4][DCD], sum_lo[4][DCD];                       // log decay of every 16 rows, in two parts
    float before[5][DCD], after[4][DCD];                     // ... of all 16s before (4: of the chunk), and after
    float beta[DC];
    double carry;
    // (which: 0 q, 1 k) a unit row's value; two neighbouring ones (d even)
    __device__ __forceinline__ float unit(int which, int t, int d) const { return to_float(qk[which][t][d]) * inv[which][t]; }
    __device__ __forceinline__ float2 unit_two(int which, int t, int d) const {
        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&qk[which][t][d]));
        const float i = inv[which][t];
        return make_float2(x.x * i, x.y * i);
    }
    __device__ __forceinline__ float2 at(int t, int d) const { return make_float2(c.hi[t][d], to_float(c.lo[t][d])); }
    // four neighbouring sums: their leading parts and what is left
    __device__ __forceinline__ void at_four(int t, int d, float (&x)[4], float (&y)[4]) const {
        const float4 hi = *reinterpret_cast<const float4*>(&c.hi[t][d]);
        const uint2 lo = *reinterpret_cast<const uint2*>(&c.lo[t][d]);
        x[0] = hi.x, x[1] = hi.y, x[2] = hi.z, x[3] = hi.w;
        y[0] = __uint_as_float(lo.x << 16), y[1] = __uint_as_float(lo.x & 0xffff0000u);
        y[2] = __uint_as_float(lo.y << 16), y[3] = __uint_as_float(lo.y & 0xffff0000u);
    }
    __device__ __forceinline__ void keep(int t, int d, double v) {
        c.hi[t][d] = (float)v;
        c.lo[t][d] = __float2bfloat16_rn((float)(v - (double)(float)v));
    }
};

// CH: a decay per key channel
template <bool CH>
__global__ void __launch_bounds__(256, 2) delta_chunk_kernel(const DeltaArgs a) {
    extern __shared__ __align__(16) unsigned char delta_raw[];
    DeltaShared& sm = *reinterpret_cast<DeltaShared*>(delta_raw);
    pdl_trigger();
    pdl_wait();
    int t0, t1;
    if (!delta_find_chunk(a, blockIdx.x, t0, t1)) return;
    const int h = blockIdx.y, kvh = h / (a.H / a.G), n = t1 - t0;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int D = a.D, V = a.V;
    const int part = CH ? 0 : blockIdx.z, parts = CH ? 1 : gridDim.z;      // (few chunks: two blocks make A each and share what comes of it)

    // the rows of q and k (zeros beyond the chunk and beyond D)
    if (((D | a.qkv_stride) & 7) == 0 && (reinterpret_cast<uintptr_t>(a.qkv) & 15) == 0) {
        for (int i = tid; i < 2 * DC * 8; i += 256) {
            const int which = i >> 9, t = (i >> 3) & 63, d = (i & 7) * 8;
            const bool ok = t < n && d < D;
            cp_async16(&sm.qk[which][t][d], a.qkv + (ok ? (size_t)(t0 + t) * a.qkv_stride + (size_t)(which * a.G + kvh) * D + d : 0), ok);
        }
    } else {
        for (int i = tid; i < 2 * DC * DCD; i += 256) {
            const int which = i >> 12, t = (i >> 6) & 63, d = i & 63;
            sm.qk[which][t][d] = (t < n && d < D) ? a.qkv[(size_t)(t0 + t) * a.qkv_stride + (size_t)(which * a.G + kvh) * D + d] : __float2bfloat16_rn(0.f);
        }
    }
    if constexpr (CH) {
        const bf16* from = a.a + (size_t)t0 * a.a_stride + h * D;
        if (((D | a.a_stride) & 7) == 0 && (reinterpret_cast<uintptr_t>(a.a) & 15) == 0) {
            for (int i = tid; i < DC * 8; i += 256) {
                const int t = i >> 3, d = (i & 7) * 8;
                const bool ok = t < n && d < D;
                cp_async16(&sm.a[t][d], from + (ok ? (size_t)t * a.a_stride + d : 0), ok);
            }
        } else {
            for (int i = tid; i < DC * DCD; i += 256) {
                const int t = i >> 6, d = i & 63;
                sm.a[t][d] = (t < n && d < D) ? from[(size_t)t * a.a_stride + d] : __float2bfloat16_rn(0.f);
            }
        }
    }
    cp_async_commit();
    // decays and beta
    if (tid < DC) sm.beta[tid] = tid < n ? 1.f / (1.f + expf(-to_float(a.b[(size_t)(t0 + tid) * a.b_stride + h]))) : 0.f;
    const float rate = expf(a.a_log[h]);
    if constexpr (CH) {
        const int d = tid & 63, seg = tid >> 6;              // 16 rows of a channel a thread
        const float bias = d < D ? a.dt_bias[h * D + d] : 0.f;
        cp_async_wait<0>();
        __syncthreads();
        double acc = 0.0;
#pragma unroll 2
        for (int t = seg * 16; t < seg * 16 + 16; ++t) {
            if (t < n && d < D) acc += delta_log_decay(rate, to_float(sm.a[t][d]) + bias);
            sm.keep(t, d, acc);
        }
        sm.sum[seg][d] = (float)acc;
        sm.sum_lo[seg][d] = (float)(acc - (double)(float)acc);
    } else {
        double l = 0.0;
        if (tid < DC) {
            if (tid < n) l = delta_log_decay(rate, to_float(a.a[(size_t)(t0 + tid) * a.a_stride + h]) + a.dt_bias[h]);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double up = __shfl_up_sync(0xffffffffu, l, o);
                if (lane >= o) l += up;
            }
            if (tid == 31) sm.carry = l;
        }
        __syncthreads();
        if (tid < DC) sm.keep(tid, 0, tid >= 32 ? l + sm.carry : l);
    }
    cp_async_wait<0>();
    __syncthreads();
    // what makes the rows unit rows: two threads a row
    {
        const int which = tid >> 7, t = (tid >> 1) & 63, part = tid & 1;
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < DCD / 2; i += 2) {
            const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&sm.qk[which][t][part * (DCD / 2) + i]));
            ss = fmaf(x.x, x.x, fmaf(x.y, x.y, ss));
        }
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        // (rows beyond the chunk stay zeros, whatever the norm's epsilon)
        if (part == 0) sm.inv[which][t] = t < n ? rsqrtf(ss + a.unit_eps) * (which ? 1.f : rsqrtf((float)D)) : 0.f;
    }
    if constexpr (CH) {
        if (tid < DCD) {                                     // (sums of numbers of one sign: their rounding is as small as their terms')
            float acc = 0.f;
            sm.before[0][tid] = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc += sm.sum[j][tid];
                sm.before[j + 1][tid] = acc;
            }
            acc = 0.f;
#pragma unroll
            for (int j = 3; j >= 0; --j) {
                sm.after[j][tid] = acc;
                acc += sm.sum[j][tid];
            }
        }
    }
    __syncthreads();

    // A and P on the tensor cores, 16 rows (I) at a time; a warp takes eight columns of one of the two
    const int mi = lane >> 3, r8 = lane & 7, g = lane >> 2, tq = lane & 3;
    DeltaChunk* out = a.chunks + (size_t)blockIdx.x * a.H + h;
    for (int I = 0; I < 4; ++I) {
        bool fast = true;
        if constexpr (CH) {
            // the largest decay of these 16 rows says whether e^(-c) inside them can be a factor by itself
            fast = !__syncthreads_or(tid < DCD && !(sm.sum[I][tid & 63] > -DELTA_FAST));
            const int rows = 16 * I + (fast ? 16 : 0);
            // (four channels a thread and turn)
#pragma unroll 1
            for (int i = tid; i < (rows + 32) * (DCD / 4); i += 256) {
                const int row = i / (DCD / 4), d = (i % (DCD / 4)) * 4;
                float e[4], hi[4], lo[4];
                bf16* dst;
                int part = DC * DR_LD, which = 1, t = row;
                if (row < rows) {                            // right: k_s e^(c at the first of the 16 - c_s)
                    const int J = row >> 4;
                    sm.at_four(row, d, hi, lo);
                    dst = &sm.right[0][row][d];
                    if (J == I) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) e[j] = delta_exp2(-hi[j], -lo[j]);
                    } else {
                        const float4 a0 = *reinterpret_cast<const float4*>(&sm.sum[J][d]), a1 = *reinterpret_cast<const float4*>(&sm.sum_lo[J][d]);
                        float f[4] = {(a0.x - hi[0]) + (a1.x - lo[0]), (a0.y - hi[1]) + (a1.y - lo[1]), (a0.z - hi[2]) + (a1.z - lo[2]),
                                      (a0.w - hi[3]) + (a1.w - lo[3])};
                        for (int K = J + 1; K < I; ++K) {
                            const float4 more = *reinterpret_cast<const float4*>(&sm.sum[K][d]);
                            f[0] += more.x;
                            f[1] += more.y;
                            f[2] += more.z;
                            f[3] += more.w;
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) e[j] = fast_exp2(f[j]);
                    }
                } else {                                     // left: q_t, k_t times e^(c_t - c at the first)
                    which = (row - rows) >> 4;
                    t = 16 * I + ((row - rows) & 15);
                    sm.at_four(t, d, hi, lo);
                    dst = &sm.left[which][0][t & 15][d];
                    part = 16 * DR_LD;
#pragma unroll
                    for (int j = 0; j < 4; ++j) e[j] = delta_exp2(hi[j], lo[j]);
                }
                const uint2 raw = *reinterpret_cast<const uint2*>(&sm.qk[which][t][d]);
                const float inv = sm.inv[which][t];
                const float2 x0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), x1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
                uint32_t p0[3], p1[3];
                split3_pair(x0.x * inv * e[0], x0.y * inv * e[1], p0);
                split3_pair(x1.x * inv * e[2], x1.y * inv * e[3], p1);
#pragma unroll
                for (int k = 0; k < 3; ++k) *reinterpret_cast<uint2*>(dst + k * part) = make_uint2(p0[k], p1[k]);
            }
            __syncthreads();
        }
        for (int unit = warp; unit < (I + (fast ? 1 : 0)) * 4; unit += 8) {
            const int which = unit & 1, nt = unit >> 1;      // which: 0 P (rows of q), 1 A (rows of k); columns 8 nt ..
            float acc[3][4] = {};
#pragma unroll
            for (int kt = 0; kt < 4; ++kt) {
                if constexpr (CH) {
                    uint32_t fa[3][4], fb[3][2];
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        ldmatrix_x4(fa[k], &sm.left[which][k][(mi & 1) * 8 + r8][kt * 16 + (mi >> 1) * 8]);
                        fb[k][0] = *reinterpret_cast<const uint32_t*>(&sm.right[k][nt * 8 + g][kt * 16 + 2 * tq]);
                        fb[k][1] = *reinterpret_cast<const uint32_t*>(&sm.right[k][nt * 8 + g][kt * 16 + 2 * tq + 8]);
                    }
#pragma unroll
                    for (int pa = 0; pa < 3; ++pa)
#pragma unroll
                        for (int pb = 0; pa + pb < 3; ++pb) mma_bf16(acc[pa + pb], fa[pa], fb[pb][0], fb[pb][1]);
                } else {                                     // (rows as they came are bfloat16: one product)
                    uint32_t fa[4];
                    ldmatrix_x4(fa, &sm.qk[which][16 * I + (mi & 1) * 8 + r8][kt * 16 + (mi >> 1) * 8]);
                    mma_bf16(acc[0], fa, *reinterpret_cast<const uint32_t*>(&sm.qk[1][nt * 8 + g][kt * 16 + 2 * tq]),
                             *reinterpret_cast<const uint32_t*>(&sm.qk[1][nt * 8 + g][kt * 16 + 2 * tq + 8]));
                }
            }
            float w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = 16 * I + g + 8 * (e >> 1), s = nt * 8 + 2 * tq + (e & 1);
                w[e] = acc[0][e] + (acc[1][e] + acc[2][e]);
                if constexpr (!CH) w[e] = acc[0][e] * sm.inv[which][t] * sm.inv[1][s] * fast_exp2(delta_minus(sm.at(t, 0), sm.at(s, 0)));
                if (s > t) w[e] = 0.f;                       // (what lies there is no part of the sums)
                if (which == 1 && s < t) sm.m[t][s] = sm.beta[t] * w[e];
            }
            if (which == 0 && part == 0) {                   // P goes out as it lies: half of a tile of 16 columns
                uint32_t lo[3], hi[3];
                split3_pair(w[0], w[1], lo);
                split3_pair(w[2], w[3], hi);
#pragma unroll
                for (int k = 0; k < 3; ++k) reinterpret_cast<uint2*>(&out->p.v[k][I][nt >> 1][lane])[nt & 1] = make_uint2(lo[k], hi[k]);
            }
        }
        if (CH && !fast) {
            // strong decays inside the 16 rows: every pair of rows by itself.  Thread (row r, four channels); the 16 threads of a
            // row add up its columns
            const int r = tid >> 4, dq = tid & 15, d0 = dq * 4, t = 16 * I + r;
            float2 ct[4];
            float kk[4], qq[4], va[16], vp[16];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                ct[j] = sm.at(t, d0 + j);
                kk[j] = sm.unit(1, t, d0 + j);
                qq[j] = sm.unit(0, t, d0 + j);
            }
#pragma unroll
            for (int s = 0; s < 16; ++s) {
                float x = 0.f, y = 0.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float w = sm.unit(1, 16 * I + s, d0 + j) * fast_exp2(delta_minus(ct[j], sm.at(16 * I + s, d0 + j)));
                    x = fmaf(kk[j], w, x);
                    y = fmaf(qq[j], w, y);
                }
                va[s] = s <= r ? x : 0.f;                    // (later rows have exponents above zero)
                vp[s] = s <= r ? y : 0.f;
            }
            sum16(va, lane);
            sum16(vp, lane);
            if (dq < r) sm.m[t][16 * I + dq] = sm.beta[t] * va[0];
            float third[3];
            split3(dq <= r ? vp[0] : 0.f, third[0], third[1], third[2]);
#pragma unroll
            for (int k = 0; k < 3; ++k)
                reinterpret_cast<bf16*>(&out->p.v[k][I][I][(r & 7) * 4 + ((dq & 7) >> 1)])[((r >> 3) + 2 * (dq >> 3)) * 2 + (dq & 1)] = __float2bfloat16_rn(third[k]);
        }
        if (CH) __syncthreads();                             // (the next 16 rows' operands take the place of these)
    }
    __syncthreads();

    // the rows of v come while the operands are put down
    const bool v_here = V <= DELTA_V_MAX;
    const bf16* v = a.qkv + (size_t)t0 * a.qkv_stride + (size_t)2 * a.G * D + (size_t)h * V;
    const bool v_vec = v_here && ((V | a.qkv_stride | (2 * a.G * D)) & 7) == 0 && (reinterpret_cast<uintptr_t>(a.qkv) & 15) == 0;
    if (v_vec) {
        const int per = V >> 3;
        for (int i = tid; i < DC * per; i += 256) {
            const int t = i / per, c = (i - t * per) * 8;
            cp_async16(&sm.v[t * (V + 8) + c], v + (size_t)(t < n ? t : 0) * a.qkv_stride + c, t < n);
        }
    } else if (v_here) {
        for (int i = tid; i < DC * V; i += 256) {
            const int t = i / V, c = i - t * V;
            sm.v[t * (V + 8) + c] = t < n ? v[(size_t)t * a.qkv_stride + c] : __float2bfloat16_rn(0.f);
        }
    }
    cp_async_commit();
    if (part == 0) delta_put(&out->q, [&](int t, int d) {
        const float2 x = sm.unit_two(0, t, d);
        if (!CH) {
            const float e = fast_exp2(sm.c.hi[t][0]);
            return make_float2(x.x * e, x.y * e);
        }
        const float2 hi = *reinterpret_cast<const float2*>(&sm.c.hi[t][d]), b = *reinterpret_cast<const float2*>(&sm.before[t >> 4][d]);
        return make_float2(x.x * fast_exp2(b.x + hi.x), x.y * fast_exp2(b.y + hi.y));
    });
    if (part == parts - 1) delta_put(&out->k, [&](int d, int s) {
        float e[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (CH) e[i] = sm.after[s >> 4][d] + delta_minus(make_float2(sm.sum[s >> 4][d], sm.sum_lo[s >> 4][d]), sm.at(s + i, d));
            else e[i] = delta_minus(sm.at(DC - 1, 0), sm.at(s + i, 0));
        }
        return make_float2(sm.unit(1, s, d) * fast_exp2(e[0]), sm.unit(1, s + 1, d) * fast_exp2(e[1]));
    });
    if (part == 0 && tid < DCD) out->keep[tid] = fast_exp2(CH ? sm.before[4][tid] : sm.c.hi[DC - 1][0]);

    cp_async_wait<0>();
    __syncthreads();
    // The triangular system, 16 right sides a warp at a time: the columns of e^(c_t) k_t, then those of v.  A lane has its share of
    // their rows (columns g, g + 8; rows 2 tq, + 1, + 8, + 9 of every 16).  Rows go in four steps of 16: the 16 among themselves are
    // substituted in 32-bit, and what they take off the later ones is a product on the tensor cores (columns are its rows, so the
    // solved 16 are its operand as they lie).  The steps are one loop's turns on purpose: every instruction runs once a turn, so
    // what the loop costs first is fetching its code (unrolled, 64 rows a thread: 106 KB of code, 28 of a block's 55 us).
    float* u0 = a.u0 + ((size_t)blockIdx.x * a.H + h) * DC * a.VP;
#pragma unroll 1
    for (int tile = warp * parts + part; tile < DCD / 16 + (V + 15) / 16; tile += 8 * parts) {
        const int c0 = tile * 16 - DCD;                      // its first column of v
        float x[4][2][4] = {};                               // [16 rows from this turn's on][tile of 8 rows][...]
#pragma unroll 1
        for (int I = 0; I < 4; ++I) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int t = 16 * I + (i >> 2) * 8 + 2 * tq + (i & 1), col = c0 + g + 8 * (i >> 1 & 1);
                float r = 0.f;
                if (c0 < 0) r = sm.unit(1, t, DCD + col) * fast_exp2(CH ? sm.before[I][DCD + col] + sm.c.hi[t][DCD + col] : sm.c.hi[t][0]);
                else if (col < V && v_here) r = to_float(sm.v[t * (V + 8) + col]);
                else if (col < V && t < n) r = to_float(v[(size_t)t * a.qkv_stride + col]);
                x[0][i >> 2][i & 3] = fmaf(sm.beta[t], r, x[0][i >> 2][i & 3]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {                    // rows 4 q .. of the 16 leave what they weigh in the later ones
                float4 m4[2][2];
#pragma unroll
                for (int i = q >> 1; i < 2; ++i)
#pragma unroll
                    for (int b = 0; b < 2; ++b) m4[i][b] = *reinterpret_cast<const float4*>(&sm.m[16 * I + i * 8 + 2 * tq + b][16 * I + 4 * q]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int s = 4 * q + j, from = (lane & ~3) | ((s & 7) >> 1);
                    const float u_lo = __shfl_sync(0xffffffffu, x[0][s >> 3][s & 1], from), u_hi = __shfl_sync(0xffffffffu, x[0][s >> 3][2 + (s & 1)], from);
#pragma unroll
                    for (int i = q >> 1; i < 2; ++i)
#pragma unroll
                        for (int b = 0; b < 2; ++b) {
                            const float m = j == 0 ? m4[i][b].x : j == 1 ? m4[i][b].y : j == 2 ? m4[i][b].z : m4[i][b].w;
                            const int behind = s - 8 * i - b;        // row 8 i + 2 tq + b lies behind s: 2 tq > this
                            if (behind < 0 || (behind < 6 && tq > behind / 2)) {
                                x[0][i][b] = fmaf(-m, u_lo, x[0][i][b]);
                                x[0][i][2 + b] = fmaf(-m, u_hi, x[0][i][2 + b]);
                            }
                        }
                }
            }
            uint32_t up[4][3];                               // the solved rows in three parts: a product's first operand
#pragma unroll
            for (int i = 0; i < 4; ++i) split3_pair(x[0][i >> 1][2 * (i & 1)], x[0][i >> 1][2 * (i & 1) + 1], up[i]);
            if (c0 < 0) {                                    // W, its rows and columns changed over
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    out->w.v[k][I][tile][lane] = make_uint4(movmatrix_trans(up[0][k]), movmatrix_trans(up[2][k]), movmatrix_trans(up[1][k]), movmatrix_trans(up[3][k]));
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int t = 16 * I + (i >> 2) * 8 + 2 * tq + (i & 1), col = c0 + g + 8 * (i >> 1 & 1);
                    if (col < V) u0[(size_t)t * a.VP + col] = x[0][i >> 2][i & 3];
                }
            }
#pragma unroll
            for (int j = 1; j < 4; ++j) {
                if (I + j > 3) break;
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    uint32_t fb[2][3];
                    float acc[3][4] = {};
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const float2 m2 = *reinterpret_cast<const float2*>(&sm.m[16 * (I + j) + nt * 8 + g][16 * I + 2 * tq + 8 * k]);
                        split3_pair(-m2.x, -m2.y, fb[k]);
                    }
#pragma unroll
                    for (int pa = 0; pa < 3; ++pa) {
                        const uint32_t f[4] = {up[0][pa], up[1][pa], up[2][pa], up[3][pa]};
#pragma unroll
                        for (int pb = 0; pa + pb < 3; ++pb) mma_bf16(acc[pa + pb], f, fb[0][pb], fb[1][pb]);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) x[j][nt][e] += acc[0][e] + (acc[1][e] + acc[2][e]);
                }
            }
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int e = 0; e < 8; ++e) x[j][e >> 2][e & 3] = x[j + 1][e >> 2][e & 3];
        }
    }
}

__device__ __forceinline__ void stmatrix_x4_trans(void* p, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};\n" ::"r"(smem_u32(p)), "r"(r0), "r"(r1),
                 "r"(r2), "r"(r3) : "memory");
}

#define DB_LD (DC + 8)              // bfloat16 row stride of the columns in shared memory

// Columns of a 64-row matrix in three parts as the second operand: [part][column][row]
template <int DN> struct DeltaColumns { bf16 v[3][DN][DB_LD]; };

// 16 rows (tile mt) x DN columns of a product's layout (rows g, g + 8; columns 2 tq, + 1 of every 8) into the columns' parts
template <int DN>
__device__ __forceinline__ void delta_put_columns(DeltaColumns<DN>& c, const float (&x)[DN / 8][4], int mt, int lane) {
#pragma unroll
    for (int nt = 0; nt < DN / 8; nt += 2) {
        uint32_t lo[2][3], hi[2][3];                         // rows g and g + 8 of the two tiles of eight columns
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            split3_pair(x[nt + j][0], x[nt + j][1], lo[j]);
            split3_pair(x[nt + j][2], x[nt + j][3], hi[j]);
        }
        const int mi = lane >> 3, r8 = lane & 7;
#pragma unroll
        for (int p = 0; p < 3; ++p)
            stmatrix_x4_trans(&c.v[p][(nt + (mi >> 1)) * 8 + r8][mt * 16 + (mi & 1) * 8], lo[0][p], hi[0][p], lo[1][p], hi[1][p]);
    }
}

// The part of a product's second operand that CAUSAL rows see only some of (16 rows, two tiles of eight columns; a lane has rows
// 2 tq, + 1, + 8, + 9 of columns g): a row's weight for what lies behind it is zero, and zero times infinity or NaN is NaN.  Such
// values leave the operand; rows from a column's first one on become NaN there.
template <int NT>
__device__ __forceinline__ void delta_take_odd(float (&acc)[NT][4], uint32_t (&fb)[3][4], int nt, int lane) {
    const int tq = lane & 3;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        int from = 16;
#pragma unroll
        for (int r = 1; r >= 0; --r) {
            const uint32_t odd = not_finite_pair(fb[0][2 * j + r]);
            if (odd >> 31) from = 2 * tq + 8 * r + 1;
            if (odd >> 15 & 1) from = 2 * tq + 8 * r;
            const uint32_t keep = (odd >> 31 ? 0u : 0xffff0000u) | (odd >> 15 & 1 ? 0u : 0x0000ffffu);
#pragma unroll
            for (int p = 0; p < 3; ++p) fb[p][2 * j + r] &= keep;
        }
        from = min(from, __shfl_xor_sync(0xffffffffu, from, 1));
        from = min(from, __shfl_xor_sync(0xffffffffu, from, 2));
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int first = __shfl_sync(0xffffffffu, from, (2 * tq + (e & 1)) * 4);
            if ((lane >> 2) + 8 * (e >> 1) >= first) acc[nt + j][e] = __int_as_float(0x7fc00000);
        }
    }
}

// acc[s] += (operand tile row: fa[part][kt]) x columns, sorted by size: s = 0 the leading parts, 2 the smallest products.  CAUSAL:
// in the last of the kts tiles of 16 rows a row sees those up to its own
template <int DN, bool CAUSAL = false>
__device__ __forceinline__ void delta_product(float (&acc)[3][DN / 8][4], const uint4 (&fa)[3][4], const DeltaColumns<DN>& c, int kts, int lane) {
    const int mi = lane >> 3, r8 = lane & 7;
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
        if (kt >= kts) continue;
#pragma unroll
        for (int nt = 0; nt < DN / 8; nt += 2) {
            uint32_t fb[3][4];
#pragma unroll
            for (int p = 0; p < 3; ++p) ldmatrix_x4(fb[p], &c.v[p][(nt + (mi >> 1)) * 8 + r8][kt * 16 + (mi & 1) * 8]);
            if (CAUSAL && kt == kts - 1
                && __any_sync(0xffffffffu, (not_finite_pair(fb[0][0]) | not_finite_pair(fb[0][1]) | not_finite_pair(fb[0][2]) | not_finite_pair(fb[0][3])) != 0))
                delta_take_odd(acc[0], fb, nt, lane);
#pragma unroll
            for (int pa = 0; pa < 3; ++pa) {
                const uint32_t f[4] = {fa[pa][kt].x, fa[pa][kt].y, fa[pa][kt].z, fa[pa][kt].w};
#pragma unroll
                for (int pb = 0; pa + pb < 3; ++pb) {
                    mma_bf16(acc[pa + pb][nt], f, fb[pb][0], fb[pb][1]);
                    mma_bf16(acc[pa + pb][nt + 1], f, fb[pb][2], fb[pb][3]);
                }
            }
        }
    }
}
__device__ __forceinline__ void delta_fetch(uint4 (&f)[3][4], const DeltaOperand& x, int mt, int lane, int kts) {
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int kt = 0; kt < 4; ++kt)
            if (kt < kts) f[p][kt] = x.v[p][mt][kt][lane];
}

// named barriers: of the carry's four warps (128 threads), and between them and the read-outs' four (256: one side arrives and
// goes on, the other waits)
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
#define DB_CARRY 1
#define DB_STATE 2                  // + turn: S before a chunk is there
#define DB_U 4                      // + turn: u of a chunk is there
#define DB_FREE 6                   // + turn: a chunk's read-outs are made, its buffers may be filled again

template <int DN>
__global__ void __launch_bounds__(256) delta_carry_kernel(const DeltaArgs a) {
    constexpr int NT = DN / 8;
    extern __shared__ __align__(16) unsigned char delta_raw[];
    DeltaColumns<DN>* ss = reinterpret_cast<DeltaColumns<DN>*>(delta_raw);    // [2] S before the chunk, by turns
    DeltaColumns<DN>* su = ss + 2;                                            // [2] u
    pdl_trigger();
    pdl_wait();
    // (one dimension, which holds any number of requests: blocks of columns fastest, then heads, then requests)
    const int per = (a.V + DN - 1) / DN, h = blockIdx.x / per % a.H, seq = blockIdx.x / per / a.H, v0 = blockIdx.x % per * DN;
    const int r0 = a.cu_q[seq], rows = a.cu_q[seq + 1] - r0;
    if (rows < a.min_rows) return;
    int first = 0;
    for (int s = 0; s < seq; ++s) {
        const int n = a.cu_q[s + 1] - a.cu_q[s];
        if (n >= a.min_rows) first += (n + DC - 1) / DC;
    }
    const int nc = (rows + DC - 1) / DC;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, mt = warp & 3, g = lane >> 2, tq = lane & 3;
    const DeltaChunk* ch = a.chunks + (size_t)first * a.H + h;
    const int D = a.D, V = a.V;

    if (warp >= 4) {                                         // ---- the read-outs
        uint4 fq[3][4], fp[3][4];
        delta_fetch(fq, ch->q, mt, lane, 4);
        delta_fetch(fp, ch->p, mt, lane, mt + 1);
        for (int c = 0; c < nc; ++c) {
            float acc[3][NT][4] = {};
            bar_sync(DB_STATE + (c & 1), 256);
            delta_product<DN>(acc, fq, ss[c & 1], 4, lane);
            ch += a.H;
            if (c + 1 < nc) delta_fetch(fq, ch->q, mt, lane, 4);
            bar_sync(DB_U + (c & 1), 256);
            delta_product<DN, true>(acc, fp, su[c & 1], mt + 1, lane);
            if (c + 2 < nc) bar_arrive(DB_FREE + (c & 1), 256);
            if (c + 1 < nc) delta_fetch(fp, ch->p, mt, lane, mt + 1);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = c * DC + mt * 16 + g + 8 * half;
                if (t >= rows) continue;
                float* o = a.o + ((size_t)(r0 + t) * a.H + h) * V;
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const int col = v0 + nt * 8 + 2 * tq;
                    const float y0 = acc[0][nt][2 * half] + (acc[1][nt][2 * half] + acc[2][nt][2 * half]);
                    const float y1 = acc[0][nt][2 * half + 1] + (acc[1][nt][2 * half + 1] + acc[2][nt][2 * half + 1]);
                    if ((V & 1) == 0 && col < V) *reinterpret_cast<float2*>(o + col) = make_float2(y0, y1);
                    else {
                        if (col < V) o[col] = y0;
                        if (col + 1 < V) o[col + 1] = y1;
                    }
                }
            }
        }
        return;
    }

    // ---- u and the state: warp mt has rows 16 mt .. of both
    const int slot = zai_checked_slot(a.slot_ids[seq], a.num_slots, a.status);
    float* st = a.state + ((size_t)slot * a.H + h) * D * V;
    float S[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int d = mt * 16 + g + 8 * (e >> 1), col = v0 + nt * 8 + 2 * tq + (e & 1);
            S[nt][e] = (d < D && col < V) ? st[(size_t)d * V + col] : 0.f;
        }
    const size_t u_step = (size_t)a.H * DC * a.VP;
    const float* u0 = a.u0 + ((size_t)first * a.H + h) * DC * a.VP + (size_t)(mt * 16 + g) * a.VP + v0 + 2 * tq;
    uint4 fw[3][4], fk[3][4];
    float2 ua[NT], ub[NT];
    float keep_a, keep_b;
    auto fetch_u = [&]() {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            ua[nt] = *reinterpret_cast<const float2*>(u0 + nt * 8);
            ub[nt] = *reinterpret_cast<const float2*>(u0 + (size_t)8 * a.VP + nt * 8);
        }
    };
    delta_fetch(fw, ch->w, mt, lane, 4);
    delta_fetch(fk, ch->k, mt, lane, 4);
    fetch_u();
    keep_a = ch->keep[mt * 16 + g];
    keep_b = ch->keep[mt * 16 + g + 8];
    delta_put_columns<DN>(ss[0], S, mt, lane);
    bar_arrive(DB_STATE, 256);
    for (int c = 0; c < nc; ++c) {
        const bool more = c + 1 < nc;
        bar_sync(DB_CARRY, 128);                             // S before chunk c is there
        float x[NT][4];
        {
            float acc[3][NT][4] = {};
            delta_product<DN>(acc, fw, ss[c & 1], 4, lane);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                x[nt][0] = ua[nt].x - (acc[0][nt][0] + (acc[1][nt][0] + acc[2][nt][0]));
                x[nt][1] = ua[nt].y - (acc[0][nt][1] + (acc[1][nt][1] + acc[2][nt][1]));
                x[nt][2] = ub[nt].x - (acc[0][nt][2] + (acc[1][nt][2] + acc[2][nt][2]));
                x[nt][3] = ub[nt].y - (acc[0][nt][3] + (acc[1][nt][3] + acc[2][nt][3]));
            }
        }
        delta_put_columns<DN>(su[c & 1], x, mt, lane);
        bar_arrive(DB_U + (c & 1), 256);
        ch += a.H;
        u0 += u_step;
        if (more) {
            delta_fetch(fw, ch->w, mt, lane, 4);
            fetch_u();
        }
        bar_sync(DB_CARRY, 128);                             // u of chunk c is there
        {
            float acc[3][NT][4] = {};
            delta_product<DN>(acc, fk, su[c & 1], 4, lane);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    S[nt][e] = fmaf(e < 2 ? keep_a : keep_b, S[nt][e], acc[0][nt][e] + (acc[1][nt][e] + acc[2][nt][e]));
        }
        if (more) {
            if (c > 0) bar_sync(DB_FREE + ((c + 1) & 1), 256);       // (chunk c - 1's, whose turn chunk c + 1 has)
            delta_put_columns<DN>(ss[(c + 1) & 1], S, mt, lane);
            bar_arrive(DB_STATE + ((c + 1) & 1), 256);
            delta_fetch(fk, ch->k, mt, lane, 4);
            keep_a = ch->keep[mt * 16 + g];
            keep_b = ch->keep[mt * 16 + g + 8];
        }
    }
    if (a.write_state) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int d = mt * 16 + g + 8 * (e >> 1), col = v0 + nt * 8 + 2 * tq + (e & 1);
                if (d < D && col < V) st[(size_t)d * V + col] = S[nt][e];
            }
    }
}

template <int DN>
static int delta_carry(const DeltaArgs& a, cudaStream_t stream) {
    constexpr size_t smem = 4 * sizeof(DeltaColumns<DN>);
    static unsigned long long done = 0;
    if (zai_first_on_device(&done)) {
        const cudaError_t e = cudaFuncSetAttribute(delta_carry_kernel<DN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    const long long blocks = (long long)a.n_seqs * a.H * ((a.V + DN - 1) / DN);
    if (blocks > 0x7fffffffLL) return ZAI_BAD_SIZE;
    return launch_pdl(delta_carry_kernel<DN>, dim3((unsigned)blocks), dim3(256), smem, stream, a);
}

ZAI_API int zai_gated_delta_chunk_rows() { return DC; }
ZAI_API int zai_gated_delta_chunked_supports(int D, int V) { return D >= 1 && D <= DCD && V >= 1 && V <= 65535 * 16; }
// bytes of scratch a chunk and head takes
ZAI_API int zai_gated_delta_chunk_bytes(int V) { return (int)(sizeof(DeltaChunk) + (size_t)DC * ((V + 31) & ~31) * sizeof(float)); }

// o_out [N, H V] 32-bit and the state of every span of min_rows rows or more, bfloat16, in chunks.  scratch: max_chunks x H x
// zai_gated_delta_chunk_bytes(V) bytes, on a boundary of 16; rows / DC + n_seqs chunks are always enough.  `channel`: a decay per
// head and key channel (a and dt_bias H D wide).  n_spans: how many such spans there are (or the most there may be).
ZAI_API int zai_gated_delta_chunked(float* o_out, const void* qkv, int qkv_stride, const void* b_in, int b_stride, const void* a_in,
                                    int a_stride, const float* a_log, const float* dt_bias, float unit_eps, float* state, const int* cu_q,
                                    const int* slot_ids, int num_slots, int* status, int n_seqs, int H, int G, int D, int V, int channel,
                                    int write_state, int min_rows, int n_spans, void* scratch, int max_chunks, cudaStream_t stream) {
    if (n_seqs <= 0 || max_chunks <= 0) return ZAI_OK;
    if (H < 1 || H > 65535 || G < 1 || H % G || !zai_gated_delta_chunked_supports(D, V)) return ZAI_BAD_SIZE;
    DeltaChunk* chunks = (DeltaChunk*)scratch;
    const DeltaArgs a = {(const bf16*)qkv, (const bf16*)b_in, (const bf16*)a_in, qkv_stride, b_stride, a_stride, a_log, dt_bias, unit_eps,
                         state, cu_q, slot_ids, status, num_slots, n_seqs, H, G, D, V, write_state, min_rows < 1 ? 1 : min_rows,
                         chunks, (float*)(chunks + (size_t)max_chunks * H), (V + 31) & ~31, o_out};
    static unsigned long long done = 0;
    if (zai_first_on_device(&done)) {
        cudaError_t e = cudaFuncSetAttribute(delta_chunk_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DeltaShared));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chunk_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DeltaShared));
        if (e != cudaSuccess) return (int)e;
    }
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) sms = 148;
    }
    // Few chunks and more tiles of right sides than a block has warps: two blocks a chunk, or the last round of tiles is a few warps'
    // work while most SMs have none.  One decay a head, us with one and two: 4 heads of 64 x 128, 64 rows 23.8 and 18.5, 256 rows 28.7
    // and 23.4; 16 heads, 64 rows 24.5 and 23.3, 512 rows (144 blocks) 44.8 and 39.3, 1024 (256; two an SM) 71.7 and 81.6.  With a decay
    // per channel, where A and P are more of a block's time, it goes up as often as down (16 heads, 64 rows 35.7 and 37.9, 100 rows 46.7
    // and 39.6).
    const int parts = !channel && V > 64 && (long long)max_chunks * H <= sms ? 2 : 1;
    const int rc = channel ? launch_pdl(delta_chunk_kernel<true>, dim3(max_chunks, H), dim3(256), sizeof(DeltaShared), stream, a)
                           : launch_pdl(delta_chunk_kernel<false>, dim3(max_chunks, H, parts), dim3(256), sizeof(DeltaShared), stream, a);
    if (rc) return rc;
    // 16 columns a block while that leaves no SM with two, else 32 (half the operand loads a column; the same sums a column)
    if ((long long)((V + 15) / 16) * H * n_spans <= sms) return delta_carry<16>(a, stream);
    return delta_carry<32>(a, stream);
}
