// Selective scan (the Mamba recurrence) over the rows of a step, with the per-request state carried
// in 32-bit between steps:
//
//   dt[t, c]  = softplus( sum_r Wdt[c, r] * p[t, r] + bdt[c] )                 p = [dt_in: R | B: S | C: S] per token
//   h[c, n]  <- exp(dt[t, c] * A[c, n]) * h[c, n] + dt[t, c] * x[t, c] * B[t, n]        A = -exp(A_log)
//   y[t, c]   = ( sum_n h[c, n] * C[t, n] + D[c] * x[t, c] ) * silu(z[t, c])
//
// Everything but the stored activations (x, p, z, y in the model's dtype) is 32-bit: the step size, the
// decay, the state and the sums.  The products dt_in . Wdt^T of all rows are one matrix product made beforehand
// (on the tensor cores where the model is bfloat16).  Two kernels:
//   * steps of single tokens: a lane holds K consecutive states of a channel (a whole channel where S <= 16, else G lanes
//     of a warp share it), loads its row's values and sums its step size itself;
//   * steps with portions: a block walks one request's rows in order, two states a lane (four and eight beyond 64 and 128), fed by warps
//     of its own; long spans of few channels are cut into chunks that are walked at once (below).
#include <cfloat>
#include "mma_helpers.cuh"

// Exponentials and the softplus: exact library functions where the model is 32-bit; where activations are
// bfloat16 the hardware approximations (relative error about 2^-21, far below the 2^-9 of a stored activation).
template <typename T> __device__ __forceinline__ float exp_for(float v) { return expf(v); }
template <> __device__ __forceinline__ float exp_for<bf16>(float v) { return __expf(v); }
template <typename T> __device__ __forceinline__ float softplus_for(float v) { return v > 20.f ? v : log1pf(expf(v)); }
template <> __device__ __forceinline__ float softplus_for<bf16>(float v) {
    const float s = __logf(1.f + __expf(v));           // (made for every value: a choice, not a branch)
    return v > 20.f ? v : s;
}
template <typename T> __device__ __forceinline__ float silu_for(float v) { return v / (1.f + expf(-v)); }
template <> __device__ __forceinline__ float silu_for<bf16>(float v) { return __fdividef(v, 1.f + __expf(-v)); }

// K consecutive values as 32-bit; `vec`: the address is a multiple of 8 bytes and K of four (16-bit values, 8 bytes a load)
template <int K>
__device__ __forceinline__ void load_run(const float* p, float (&d)[K], int n_valid, bool vec) {
#pragma unroll
    for (int k = 0; k < K; ++k) d[k] = k < n_valid ? p[k] : 0.f;
}
template <int K>
__device__ __forceinline__ void load_run(const bf16* p, float (&d)[K], int n_valid, bool vec) {
    if (K % 4 == 0 && vec && n_valid == K) {
#pragma unroll
        for (int k = 0; k < K; k += 4) {
            const uint2 v = *reinterpret_cast<const uint2*>(p + k);
            const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
            const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
            d[k] = a.x; d[k + 1] = a.y; d[k + 2] = b.x; d[k + 3] = b.y;
        }
    } else {
#pragma unroll
        for (int k = 0; k < K; ++k) d[k] = k < n_valid ? __bfloat162float(p[k]) : 0.f;
    }
}

// dt_in . wrow over R terms, split over the G lanes of the channel (16 bytes a load where rows are aligned)
template <typename T, int G>
__device__ __forceinline__ float step_size_product(const T* __restrict__ wrow, const T* __restrict__ prow, int R, int g, bool vec) {
    float s = 0.f;
    if (sizeof(T) == 2 && vec) {
        for (int r = g * 8; r < R; r += G * 8) {
            const uint4 wv = *reinterpret_cast<const uint4*>(wrow + r), pv = *reinterpret_cast<const uint4*>(prow + r);
            const __nv_bfloat162* wp = reinterpret_cast<const __nv_bfloat162*>(&wv);
            const __nv_bfloat162* pp = reinterpret_cast<const __nv_bfloat162*>(&pv);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 a = __bfloat1622float2(wp[e]), b = __bfloat1622float2(pp[e]);
                s += a.x * b.x + a.y * b.y;
            }
        }
    } else {
        for (int r = g; r < R; r += G) s += to_float(wrow[r]) * to_float(prow[r]);
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// a lane's K states from / to memory (16 bytes a time where the run is aligned)
template <int K>
__device__ __forceinline__ void state_io(float* st, float (&h)[K], int n_valid, bool store) {
    if (K % 4 == 0 && n_valid == K && (reinterpret_cast<uintptr_t>(st) & 15) == 0) {
#pragma unroll
        for (int k = 0; k < K; k += 4) {
            float4* p = reinterpret_cast<float4*>(st + k);
            if (store) *p = make_float4(h[k], h[k + 1], h[k + 2], h[k + 3]);
            else { const float4 v = *p; h[k] = v.x; h[k + 1] = v.y; h[k + 2] = v.z; h[k + 3] = v.w; }
        }
    } else {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (k < n_valid) { if (store) st[k] = h[k]; else h[k] = st[k]; }
            else if (!store) h[k] = 0.f;
        }
    }
}

// ---- one row of a request, by 128 threads of a block: the step's only row of that request
template <typename T, int K, int G>
__device__ __forceinline__ void scan_one_row(T* __restrict__ y, const T* __restrict__ x, const T* __restrict__ proj, int proj_stride,
                                             const T* __restrict__ z, int z_stride, const float* __restrict__ dt_raw, const T* __restrict__ w_dt,
                                             const float* __restrict__ b_dt, const float* __restrict__ a_log, const float* __restrict__ d_skip,
                                             float* __restrict__ state, int t, int slot, int I, int S, int R, int write_state) {
    const int g = threadIdx.x % G;
    int c = blockIdx.y * (128 / G) + threadIdx.x / G;
    const bool live = c < I;
    if (!live) c = I - 1;                              // (keeps the lane in the shuffles; it stores nothing)
    const int n_mine = max(min(S - g * K, K), 0);
    float* st = state + ((size_t)slot * I + c) * S + g * K;
    float h[K], a[K], bv[K], cv[K];
    state_io<K>(st, h, n_mine, false);
#pragma unroll
    for (int k = 0; k < K; ++k) a[k] = k < n_mine ? -expf(a_log[(size_t)c * S + g * K + k]) : 0.f;
    const T* prow = proj + (size_t)t * proj_stride;
    const bool vec = sizeof(T) == 2 && ((proj_stride | R | S) & 3) == 0 && (reinterpret_cast<uintptr_t>(proj) & 7) == 0;
    load_run<K>(prow + R + g * K, bv, n_mine, vec);
    load_run<K>(prow + R + S + g * K, cv, n_mine, vec);
    const float xv = to_float(x[(size_t)t * I + c]), zv = to_float(z[(size_t)t * z_stride + c]);
    float dt;
    if (dt_raw) {
        dt = dt_raw[(size_t)t * I + c];
    } else {                                           // (the product is summed here, no launch for it)
        const T* wrow = w_dt + (size_t)c * R;
        const bool vec8 = ((proj_stride | R) & 7) == 0 && ((reinterpret_cast<uintptr_t>(proj) | reinterpret_cast<uintptr_t>(wrow)) & 15) == 0;
        dt = step_size_product<T, G>(wrow, prow, R, g, vec8);
    }
    dt = softplus_for<T>(dt + b_dt[c]);
    const float dx = dt * xv;
    float out = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        h[k] = exp_for<T>(dt * a[k]) * h[k] + dx * bv[k];
        out += h[k] * cv[k];
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) out += __shfl_xor_sync(0xffffffffu, out, o);
    if (g == 0 && live) y[(size_t)t * I + c] = from_float<T>((out + d_skip[c] * xv) * silu_for<T>(zv));
    if (write_state && live) state_io<K>(st, h, n_mine, true);
}

// ---- a step of single tokens, row i of request i
template <typename T, int K, int G>
__global__ void __launch_bounds__(128) selective_scan_single_kernel(
    T* __restrict__ y, const T* __restrict__ x, const T* __restrict__ proj, int proj_stride, const T* __restrict__ z,
    int z_stride, const float* __restrict__ dt_raw, const T* __restrict__ w_dt, const float* __restrict__ b_dt,
    const float* __restrict__ a_log, const float* __restrict__ d_skip, float* __restrict__ state, const int* __restrict__ cu_q,
    const int* __restrict__ slot_ids, int I, int S, int R, int write_state, int num_slots, int* __restrict__ status) {
    pdl_trigger();
    pdl_wait();
    const int t = cu_q[blockIdx.x];
    if (cu_q[blockIdx.x + 1] <= t) return;
    scan_one_row<T, K, G>(y, x, proj, proj_stride, z, z_stride, dt_raw, w_dt, b_dt, a_log, d_skip, state, t,
                          zai_checked_slot(slot_ids[blockIdx.x], num_slots, status), I, S, R, write_state);
}

// ---- steps with portions.  A block walks one request's rows for 128 / G channels, in tiles of 64 rows (32 with more than
// 64 states).  Four warps walk: a lane holds K states of a channel, and what a row gives it comes out of shared memory as 32-bit
// numbers, four rows ahead of their use.  Four more warps put the next tile there meanwhile (step sizes, their products with x, the
// gates; a tile's loads are issued while the tile before it is walked) and take the read-outs of the tile before to y.  One barrier
// a tile.
//
// What bounds it: S exponentials a row and channel, which the special-function units make at 16 a cycle and SM, and, where the
// channels are few, a row's chain of dependent instructions (38 ns with two states a lane, 53 with four).  A walk makes the exponentials
// once; with two states a lane 2048 channels of 16 states give every scheduler of the chip a warp.  One span of 2048 rows, 16 states
// (us, without the step sizes' product): 119 for 4096 channels (three passes over chunks of 16 to 64 rows: 296), 82 for 2048 (160);
// 512 rows of 4096 channels 31 (94).  States a lane, by S: up to 16 states 2 on 8 lanes (8 states, 4096 channels: 118, 2 on 4 lanes
// 150, whose feeding warps are too slow), 64 states 4 on 16 lanes (1024 channels: 109; 2 on 32 lanes 130), 128 states 4 on 32 lanes
// (512 channels: 212; 8 on 16 lanes 281), 256 states 8 on 32 lanes (200 states, 512 channels: 447; 16 on 16 lanes, which spills, 1018).
// (a rate beyond the largest number counts as that: a row with a step of zero leaves the state alone, zero times infinity would not)
__device__ __forceinline__ float decay_bound(float a) { return a < -FLT_MAX ? -FLT_MAX : a; }
template <typename T> __device__ __forceinline__ float decay_scale(float a) { return decay_bound(a); }
template <> __device__ __forceinline__ float decay_scale<bf16>(float a) { return decay_bound(a * 1.4426950408889634f); }
template <typename T> __device__ __forceinline__ float decay_of(float v) { return expf(v); }
template <> __device__ __forceinline__ float decay_of<bf16>(float v) { return fast_exp2(v); }

// two 32-bit numbers in one register pair: one instruction multiplies (and adds) both, each rounded as by itself
__device__ __forceinline__ uint64_t mul_pair(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t make_pair(float x, float y) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
    return d;
}
__device__ __forceinline__ float2 pair_of(uint64_t v) {
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
    return d;
}

// four neighbouring values as they lie in memory
template <typename T> struct Four;
template <> struct Four<float> {
    float4 v;
    __device__ __forceinline__ void load(const float* p) { v = *reinterpret_cast<const float4*>(p); }
    __device__ __forceinline__ void zero() { v = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ void load_some(const float* p, int n) {
        v = make_float4(n > 0 ? p[0] : 0.f, n > 1 ? p[1] : 0.f, n > 2 ? p[2] : 0.f, n > 3 ? p[3] : 0.f);
    }
    __device__ __forceinline__ float4 get() const { return v; }
    static __device__ __forceinline__ void store(float* p, const float (&o)[4]) { *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]); }
};
template <> struct Four<bf16> {
    uint2 v;
    __device__ __forceinline__ void load(const bf16* p) { v = *reinterpret_cast<const uint2*>(p); }
    __device__ __forceinline__ void zero() { v = make_uint2(0u, 0u); }
    __device__ __forceinline__ void load_some(const bf16* p, int n) {
        v.x = pack_bf16(n > 0 ? to_float(p[0]) : 0.f, n > 1 ? to_float(p[1]) : 0.f);
        v.y = pack_bf16(n > 2 ? to_float(p[2]) : 0.f, n > 3 ? to_float(p[3]) : 0.f);
    }
    __device__ __forceinline__ float4 get() const {
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
        const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
    static __device__ __forceinline__ void store(bf16* p, const float (&o)[4]) {
        *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]));
    }
};

template <int K, int G>
struct ScanTile {                                            // a tile in shared memory
    static constexpr int CB = 128 / G, SP = K * G;           // channels and states (with padding) of a block
    static constexpr int TT = SP > 64 ? 32 : 64;             // rows
    static constexpr int LDS = CB + 8;                       // read-outs: four rows of a warp's channels lie in different banks
    float4 step[TT][CB + 1];                                 // step size twice, its product with x twice (rows a bank group apart)
    float2 last[TT][CB + 2];                                 // D x, silu(z)
    float bc[TT][2 * SP];                                    // B | C
    float sum[TT][LDS];                                      // the walk's read-outs
};

// the rows' way in and out, by 128 threads.  VEC: channels, states and every row of x, z, proj, dt_raw and y lie in fours on
// boundaries of four.  ENDS: nothing goes out
template <typename T, int K, int G, bool VEC, bool ENDS>
__device__ __forceinline__ void scan_feed(ScanTile<K, G>* tiles, int tid, int c0, int start, int end, T* __restrict__ y,
                                          const T* __restrict__ x, const T* __restrict__ proj, int proj_stride, const T* __restrict__ z,
                                          int z_stride, const float* __restrict__ dt_raw, const float* __restrict__ b_dt,
                                          const float* __restrict__ d_skip, int I, int S, int R) {
    using Tile = ScanTile<K, G>;
    constexpr int CB = Tile::CB, SP = Tile::SP, TT = Tile::TT, QC = CB / 4, ROWS = 128 / QC, PER = TT > ROWS ? TT / ROWS : 1;
    constexpr int FOURS = TT * 2 * SP / 4, BC = FOURS / 128;          // fours of B and C: of a tile, of a thread
    static_assert(BC >= 1 && FOURS % 128 == 0, "a tile is shared evenly");
    const int cq = (tid % QC) * 4, r0 = tid / QC;            // this thread's four channels, and its rows r0 + i ROWS
    const int n_c = min(I - c0 - cq, 4), n_tiles = (end - start + TT - 1) / TT;
    float bias[4], skip[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        bias[k] = k < n_c ? b_dt[c0 + cq + k] : 0.f;
        skip[k] = k < n_c ? d_skip[c0 + cq + k] : 0.f;
    }
    struct Raw { Four<float> dt[PER]; Four<T> xv[PER], zv[PER], bc[BC]; };
    auto fetch = [&](int n, Raw& in) {
        const int t0 = start + n * TT;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int t = t0 + r0 + i * ROWS;
            const int nc = (t < end && r0 + i * ROWS < TT) ? n_c : 0;
            if (VEC) {
                if (nc > 0) {
                    in.dt[i].load(dt_raw + (size_t)t * I + c0 + cq);
                    in.xv[i].load(x + (size_t)t * I + c0 + cq);
                    if (!ENDS) in.zv[i].load(z + (size_t)t * z_stride + c0 + cq);
                } else {
                    in.dt[i].zero(); in.xv[i].zero(); in.zv[i].zero();
                }
            } else {
                in.dt[i].load_some(dt_raw + (size_t)t * I + c0 + cq, nc);
                in.xv[i].load_some(x + (size_t)t * I + c0 + cq, nc);
                if (!ENDS) in.zv[i].load_some(z + (size_t)t * z_stride + c0 + cq, nc);
            }
        }
#pragma unroll
        for (int i = 0; i < BC; ++i) {
            const int e = tid + i * 128, r = e / (2 * SP / 4), q = e % (2 * SP / 4) * 4, which = q >= SP, s = q - which * SP;
            const int ns = t0 + r < end ? S - s : 0;
            const T* p = proj + (size_t)(t0 + r) * proj_stride + R + which * S + s;
            if (VEC) { if (ns > 0) in.bc[i].load(p); else in.bc[i].zero(); }
            else in.bc[i].load_some(p, ns);
        }
    };
    auto leave = [&](int n) {                                // the read-outs of tile n go to y
        const Tile& tile = tiles[n & 1];
        const int t0 = start + n * TT;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int r = r0 + i * ROWS;
            if (r >= TT || t0 + r >= end) continue;
            float v[4];
            const float4 m = *reinterpret_cast<const float4*>(&tile.sum[r][cq]);
            const float4 l = *reinterpret_cast<const float4*>(&tile.last[r][cq]), k = *reinterpret_cast<const float4*>(&tile.last[r][cq + 2]);
            v[0] = (m.x + l.x) * l.y;
            v[1] = (m.y + l.z) * l.w;
            v[2] = (m.z + k.x) * k.y;
            v[3] = (m.w + k.z) * k.w;
            T* p = y + (size_t)(t0 + r) * I + c0 + cq;
            if (VEC) { if (n_c > 0) Four<T>::store(p, v); }
            else {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (k < n_c) p[k] = from_float<T>(v[k]);
            }
        }
    };
    Raw in;
    fetch(0, in);
    for (int n = 0; n <= n_tiles; ++n) {
        const int t0 = start + n * TT;
        if (!ENDS && n >= 2) leave(n - 2);                   // (its buffer is the one that tile n is put into)
        if (n < n_tiles) {
            Tile& tile = tiles[n & 1];
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int r = r0 + i * ROWS;
                if (r >= TT || t0 + r >= end + 3) continue;  // (rows in fours)
                const bool on = t0 + r < end;
                const float4 df = in.dt[i].get(), xf = in.xv[i].get(), zf = ENDS ? make_float4(0.f, 0.f, 0.f, 0.f) : in.zv[i].get();
                const float d4[4] = {df.x, df.y, df.z, df.w}, x4[4] = {xf.x, xf.y, xf.z, xf.w}, z4[4] = {zf.x, zf.y, zf.z, zf.w};
                float2 l[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float d = on ? softplus_for<T>(d4[k] + bias[k]) : 0.f;          // (a row beyond the span changes no state)
                    const float dx = d * x4[k];
                    tile.step[r][cq + k] = make_float4(d, d, dx, dx);
                    if (!ENDS) l[k] = make_float2(skip[k] * x4[k], silu_for<T>(z4[k]));
                }
                if (!ENDS) {
#pragma unroll
                    for (int k = 0; k < 4; k += 2) *reinterpret_cast<float4*>(&tile.last[r][cq + k]) = make_float4(l[k].x, l[k].y, l[k + 1].x, l[k + 1].y);
                }
            }
#pragma unroll
            for (int i = 0; i < BC; ++i) *reinterpret_cast<float4*>(&tile.bc[0][0] + (tid + i * 128) * 4) = in.bc[i].get();
            if (n + 1 < n_tiles) fetch(n + 1, in);
        }
        __syncthreads();                                     // tile n is there, tile n - 1 has been walked
    }
    if (!ENDS) leave(n_tiles - 1);
}

// A walk is one chain of rows: where a layer's channels are few blocks and a span is long, most of the chip waits for it.  Spans of
// min_rows rows or more are cut into chunks of SCAN_CHUNK rows there, which run as
//   ENDS      every chunk walked from a state of zero: its end state E and, state by state, the product P of its decays
//   carry     across a request's chunks, in order: E <- the state before the chunk, which becomes P state + E
//   the walk  of every chunk from its own first state
// The recurrence is linear in its state: the same sums in another order.  One span of 16 states, walked and in chunks (us): 2048 rows
// of 256 channels 82 and 37, of 1024 80 and 51, of 2048 (128 blocks) 82 and 84; 8192 rows of 512 channels 313 and 100.
#define SCAN_CHUNK 512
struct ScanChunks {
    float *ends, *decays;                                    // [chunks, I, S]; null: spans are walked whole
    int n_seqs, min_rows, max_rows;                          // (whole: spans of up to max_rows)
};
// the rows of chunk b among all chunks of the step: those of the spans of min_rows rows or more, in order
__device__ __forceinline__ bool scan_find_chunk(const int* __restrict__ cu_q, const ScanChunks& ch, int b, int& start, int& end) {
    for (int s = 0; s < ch.n_seqs; ++s) {
        const int lo = cu_q[s], hi = cu_q[s + 1];
        if (hi - lo < ch.min_rows) continue;
        const int n = (hi - lo + SCAN_CHUNK - 1) / SCAN_CHUNK;
        if (b < n) {
            start = lo + b * SCAN_CHUNK;
            end = min(start + SCAN_CHUNK, hi);
            return true;
        }
        b -= n;
    }
    return false;
}

template <typename T, int K, int G, bool ENDS>
__global__ void __launch_bounds__(256) selective_scan_kernel(
    T* __restrict__ y, const T* __restrict__ x, const T* __restrict__ proj, int proj_stride, const T* __restrict__ z,
    int z_stride, const float* __restrict__ dt_raw, const float* __restrict__ b_dt,
    const float* __restrict__ a_log, const float* __restrict__ d_skip, float* __restrict__ state, const int* __restrict__ cu_q,
    const int* __restrict__ slot_ids, int I, int S, int R, int write_state, int num_slots, int* __restrict__ status, int vec, const ScanChunks ch) {
    using Tile = ScanTile<K, G>;
    constexpr int CB = Tile::CB, SP = Tile::SP, TT = Tile::TT;
    extern __shared__ __align__(16) unsigned char scan_raw[];
    Tile* tiles = reinterpret_cast<Tile*>(scan_raw);         // [2]
    pdl_trigger();
    pdl_wait();
    const int seq = blockIdx.x, c0 = blockIdx.y * CB;
    int start, end;
    if (ch.ends) {
        if (!scan_find_chunk(cu_q, ch, blockIdx.x, start, end)) return;
    } else {
        start = cu_q[seq], end = cu_q[seq + 1];
        if (end <= start || end - start > ch.max_rows) return;
    }
    if (!ENDS && !ch.ends && end - start == 1) {             // (a decoding request beside the portions: no tile for one row)
        if (threadIdx.x < 128)
            scan_one_row<T, K, G>(y, x, proj, proj_stride, z, z_stride, dt_raw, nullptr, b_dt, a_log, d_skip, state, start,
                                  zai_checked_slot(slot_ids[seq], num_slots, status), I, S, R, write_state);
        return;
    }
    const int n_tiles = (end - start + TT - 1) / TT;
    if (threadIdx.x >= 128) {
        if (vec) scan_feed<T, K, G, true, ENDS>(tiles, threadIdx.x - 128, c0, start, end, y, x, proj, proj_stride, z, z_stride, dt_raw, b_dt, d_skip, I, S, R);
        else scan_feed<T, K, G, false, ENDS>(tiles, threadIdx.x - 128, c0, start, end, y, x, proj, proj_stride, z, z_stride, dt_raw, b_dt, d_skip, I, S, R);
        return;
    }

    // ---- the walk
    const int lane = threadIdx.x & 31, g = threadIdx.x % G, cl = threadIdx.x / G;
    int c = c0 + cl;
    const bool live = c < I;
    if (!live) c = I - 1;
    const int n_mine = max(min(S - g * K, K), 0);
    float* st = ch.ends ? ch.ends + ((size_t)blockIdx.x * I + c) * S + g * K
                        : state + ((size_t)zai_checked_slot(slot_ids[seq], num_slots, status) * I + c) * S + g * K;
    float h1[K] = {};
    uint64_t h[K / 2], a[K / 2], product[K / 2];             // states in pairs
    if (!ENDS) state_io<K>(st, h1, n_mine, false);
#pragma unroll
    for (int k = 0; k < K; k += 2) {
        const float* al = a_log + (size_t)c * S + g * K + k;
        h[k / 2] = make_pair(h1[k], h1[k + 1]);
        product[k / 2] = make_pair(1.f, 1.f);
        a[k / 2] = make_pair(k < n_mine ? decay_scale<T>(-expf(al[0])) : 0.f, k + 1 < n_mine ? decay_scale<T>(-expf(al[1])) : 0.f);
    }
    struct Rows { ulonglong2 d[4]; uint64_t b[4][K / 2], c[4][K / 2]; };    // four rows' operands
    auto take = [&](const Tile& tile, int r, Rows& o) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            o.d[u] = *reinterpret_cast<const ulonglong2*>(&tile.step[r + u][cl]);
            const uint64_t* p = reinterpret_cast<const uint64_t*>(&tile.bc[r + u][g * K]);
#pragma unroll
            for (int k = 0; k < K / 2; ++k) {
                o.b[u][k] = p[k];
                if (!ENDS) o.c[u][k] = p[SP / 2 + k];
            }
        }
    };
    // the G lanes' sums of four rows at once, in steps that run beside the next rows' sums: each exchange halves the rows a lane
    // goes on with
    const bool b0 = lane & 1, b1 = lane & 2;
    auto settle = [&](Tile& tile, int r, int at, float (&v)[4]) {
        if (at == 0) {
            v[0] = (b0 ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, b0 ? v[0] : v[1], 1);
            v[2] = (b0 ? v[3] : v[2]) + __shfl_xor_sync(0xffffffffu, b0 ? v[2] : v[3], 1);
        } else if (at == 1) {
            v[0] = (b1 ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, b1 ? v[0] : v[2], 2);
        } else if (at == 2) {
#pragma unroll
            for (int o = 4; o < G; o <<= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        } else if (G == 4 || g < 4) {
            tile.sum[r + (lane & 3)][cl] = v[0];
        }
    };
    __syncthreads();                                         // tile 0 is there
    for (int n = 0; n < n_tiles; ++n) {
        Tile& tile = tiles[n & 1];
        const int rows = min(TT, end - start - n * TT);      // (up to three rows behind them change no state)
        Rows now;
        take(tile, 0, now);
        float before[4] = {0.f, 0.f, 0.f, 0.f};
        int r = 0;
#pragma unroll 2
        for (; r < rows; r += 4) {
            Rows next;
            take(tile, r + 4 < TT ? r + 4 : r, next);
            float out[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                uint64_t sum = 0;
#pragma unroll
                for (int k = 0; k < K / 2; ++k) {
                    const float2 v = pair_of(mul_pair(now.d[u].x, a[k]));
                    const uint64_t decay = make_pair(decay_of<T>(v.x), decay_of<T>(v.y));
                    h[k] = fma_pair(decay, h[k], mul_pair(now.d[u].y, now.b[u][k]));
                    if (ENDS) product[k] = mul_pair(product[k], decay);
                    else sum = k ? fma_pair(h[k], now.c[u][k], sum) : mul_pair(h[k], now.c[u][k]);
                }
                const float2 both = pair_of(sum);
                out[u] = both.x + both.y;
                if (!ENDS && r > 0) settle(tile, r - 4, u, before);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) before[u] = out[u];
            now = next;
        }
        if (!ENDS) {
#pragma unroll
            for (int u = 0; u < 4; ++u) settle(tile, r - 4, u, before);
        }
        __syncthreads();                                     // this tile has been walked, the next one is there
    }
    if (live && (ENDS || (write_state && !ch.ends))) {
#pragma unroll
        for (int k = 0; k < K; k += 2) {
            const float2 v = pair_of(h[k / 2]);
            h1[k] = v.x;
            h1[k + 1] = v.y;
        }
        state_io<K>(st, h1, n_mine, true);
        if (ENDS) {
#pragma unroll
            for (int k = 0; k < K; k += 2) {
                const float2 v = pair_of(product[k / 2]);
                h1[k] = v.x;
                h1[k + 1] = v.y;
            }
            state_io<K>(ch.decays + ((size_t)blockIdx.x * I + c) * S + g * K, h1, n_mine, true);
        }
    }
}

// a thread carries one state of a request (blockIdx.x) across its chunks
__global__ void __launch_bounds__(128) selective_scan_carry_kernel(float* __restrict__ state, const int* __restrict__ cu_q, const int* __restrict__ slot_ids,
                                                                   int IS, int write_state, int num_slots, int* __restrict__ status, const ScanChunks ch) {
    pdl_trigger();
    pdl_wait();
    const int seq = blockIdx.x, rows = cu_q[seq + 1] - cu_q[seq], idx = blockIdx.y * blockDim.x + threadIdx.x;
    if (rows < ch.min_rows || idx >= IS) return;
    int first = 0;
    for (int s = 0; s < seq; ++s) {
        const int n = cu_q[s + 1] - cu_q[s];
        if (n >= ch.min_rows) first += (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
    }
    const int nc = (rows + SCAN_CHUNK - 1) / SCAN_CHUNK;
    float* st = state + (size_t)zai_checked_slot(slot_ids[seq], num_slots, status) * IS + idx;
    float h = *st;
    for (int c = 0; c < nc; ++c) {
        float* e = ch.ends + (size_t)(first + c) * IS + idx;
        const float end = *e, decay = ch.decays[(size_t)(first + c) * IS + idx];
        *e = h;
        h = fmaf(decay, h, end);
    }
    if (write_state) *st = h;
}

template <typename T, int K, int G>
static int launch_scan_single(void* y, const void* x, const void* proj, int proj_stride, const void* z, int z_stride, const float* dt_raw,
                              const void* w_dt, const float* b_dt, const float* a_log, const float* d_skip, float* state, const int* cu_q,
                              const int* slot_ids, int n_seqs, int I, int S, int R, int write_state, int num_slots, int* status,
                              cudaStream_t stream) {
    const unsigned cb = (unsigned)((I + 128 / G - 1) / (128 / G));
    if (cb > 65535) return ZAI_BAD_SIZE;
    return launch_pdl(selective_scan_single_kernel<T, K, G>, dim3(n_seqs, cb), dim3(128), 0, stream, (T*)y, (const T*)x,
                      (const T*)proj, proj_stride, (const T*)z, z_stride, dt_raw, (const T*)w_dt, b_dt, a_log, d_skip, state,
                      cu_q, slot_ids, I, S, R, write_state, num_slots, status);
}

template <typename T, int K, int G>
static int launch_scan(void* y, const void* x, const void* proj, int proj_stride, const void* z, int z_stride, const float* dt_raw,
                       const float* b_dt, const float* a_log, const float* d_skip, float* state, const int* cu_q,
                       const int* slot_ids, int n_seqs, int I, int S, int R, int write_state, int num_slots, int* status,
                       const ScanChunks& chunks, int max_chunks, cudaStream_t stream) {
    const unsigned cb = (unsigned)((I + 128 / G - 1) / (128 / G));
    if (cb > 65535) return ZAI_BAD_SIZE;
    constexpr size_t smem = 2 * sizeof(ScanTile<K, G>);
    static_assert(smem <= 227 * 1024, "two tiles fit");
    static unsigned long long done = 0;
    if (zai_first_on_device(&done)) {
        cudaError_t e = cudaFuncSetAttribute(selective_scan_kernel<T, K, G, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(selective_scan_kernel<T, K, G, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    const uintptr_t four = 4 * sizeof(T) - 1;
    const int vec = ((I | S | R | proj_stride | z_stride) & 3) == 0 && (reinterpret_cast<uintptr_t>(dt_raw) & 15) == 0
                    && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(z) | reinterpret_cast<uintptr_t>(proj)) & four) == 0;
    auto walk = [&](void (*kernel)(T*, const T*, const T*, int, const T*, int, const float*, const float*, const float*, const float*, float*,
                                   const int*, const int*, int, int, int, int, int, int*, int, const ScanChunks), int blocks, const ScanChunks& ch) {
        return launch_pdl(kernel, dim3(blocks, cb), dim3(256), smem, stream, (T*)y, (const T*)x, (const T*)proj, proj_stride, (const T*)z,
                          z_stride, dt_raw, b_dt, a_log, d_skip, state, cu_q, slot_ids, I, S, R, write_state, num_slots, status, vec, ch);
    };
    if (max_chunks > 0) {
        if ((long long)I * S > 65535LL * 128) return ZAI_BAD_SIZE;
        int rc = walk(selective_scan_kernel<T, K, G, true>, max_chunks, chunks);
        if (rc) return rc;
        rc = launch_pdl(selective_scan_carry_kernel, dim3(n_seqs, (I * S + 127) / 128), dim3(128), 0, stream, state, cu_q, slot_ids, I * S, write_state,
                        num_slots, status, chunks);
        if (rc) return rc;
        rc = walk(selective_scan_kernel<T, K, G, false>, max_chunks, chunks);
        if (rc || chunks.max_rows < 1) return rc;
    }
    return walk(selective_scan_kernel<T, K, G, false>, n_seqs, ScanChunks{nullptr, nullptr, n_seqs, 0, chunks.max_rows});
}

// channels of a block of the kernel that walks portions, by the number of states
ZAI_API int zai_selective_scan_channels(int S) { return S <= 16 ? 16 : S <= 64 ? 8 : 4; }
ZAI_API int zai_selective_scan_chunk_rows() { return SCAN_CHUNK; }

// y [N, I]; x [N, I]; proj [N, proj_stride] (dt_in | B | C, of which B and C are read here); z [N, z_stride];
// dt_raw [N, I]: the products dt_in . w_dt^T in 32-bit (a matrix product made beforehand), or null in a step of single
// tokens, which then sums them from w_dt [I, R] itself; state [slots, I, S].
// single_tokens: every request brings one row (a leaner kernel).
// With max_chunks > 0 spans of min_rows rows or more run in chunks of SCAN_CHUNK rows: ends and decays [max_chunks, I, S] 32-bit scratch,
// max_chunks at least the number of their chunks; `others`: there may be shorter spans too.
ZAI_API int zai_selective_scan(void* y, const void* x, const void* proj, int proj_stride, const void* z, int z_stride, int dtype,
                               const float* dt_raw, const void* w_dt, const float* b_dt, const float* a_log, const float* d_skip,
                               float* state, const int* cu_q, const int* slot_ids, int N, int n_seqs, int I, int S, int R, int write_state,
                               int num_slots, int* status, int single_tokens, float* ends, float* decays, int max_chunks, int min_rows, int others,
                               cudaStream_t stream) {
    if (N <= 0 || n_seqs <= 0) return ZAI_OK;
    if (I < 1 || S < 1 || S > 256 || R < 1 || (!dt_raw && !w_dt)) return ZAI_BAD_SIZE;
    if (single_tokens && N == n_seqs) {
#define ZAI_SCAN(KK, GG) ZAI_DISPATCH(dtype, return launch_scan_single<T, KK, GG>(y, x, proj, proj_stride, z, z_stride, dt_raw, w_dt, b_dt, \
        a_log, d_skip, state, cu_q, slot_ids, n_seqs, I, S, R, write_state, num_slots, status, stream))
        if (S <= 4) ZAI_SCAN(4, 1);
        if (S <= 8) ZAI_SCAN(8, 1);
        if (S <= 16) ZAI_SCAN(16, 1);
        if (S <= 32) ZAI_SCAN(16, 2);
        if (S <= 64) ZAI_SCAN(16, 4);
        if (S <= 128) ZAI_SCAN(16, 8);
        ZAI_SCAN(16, 16);
#undef ZAI_SCAN
    }
    if (!dt_raw || (max_chunks > 0 && (!ends || !decays || min_rows < 1))) return ZAI_BAD_SIZE;
    const ScanChunks chunks = {ends, decays, n_seqs, min_rows, max_chunks <= 0 ? 0x7fffffff : others ? min_rows - 1 : 0};
#define ZAI_SCAN(KK, GG) ZAI_DISPATCH(dtype, return launch_scan<T, KK, GG>(y, x, proj, proj_stride, z, z_stride, dt_raw, b_dt, a_log, \
        d_skip, state, cu_q, slot_ids, n_seqs, I, S, R, write_state, num_slots, status, chunks, max_chunks, stream))
    if (S <= 16) ZAI_SCAN(2, 8);
    if (S <= 32) ZAI_SCAN(2, 16);
    if (S <= 64) ZAI_SCAN(4, 16);
    if (S <= 128) ZAI_SCAN(4, 32);
    ZAI_SCAN(8, 32);
#undef ZAI_SCAN
}
