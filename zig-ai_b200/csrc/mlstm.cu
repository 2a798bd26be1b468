// A matrix memory with exponential gates kept in logarithms (the mLSTM cell of the xLSTM family), per request and head:
//
//   i_t = cap tanh((x_i + b_i) / cap),   f_t = logsigmoid(cap tanh((x_f + b_f) / cap))          log gates, one pair a head
//   m_t = max(f_t + m_(t-1), i_t)                                                                   running maximum, m_(-1) = 0
//   S_t = exp(f_t + m_(t-1) - m_t) S_(t-1) + exp(i_t - m_t) k_t v_t^T,   n_t likewise with k_t alone
//   o_t = S_t^T q_t / (max(|n_t . q_t|, exp(-m_t)) + 1e-6),   q_t = x_q D^(-1/2)
//   out = o / rms(o) per head * weight * sigmoid(gate)
//
// The normaliser n is one more column of S (the column of a value that is always 1), and every column carries its own
// copy of m in a row behind its D rows: the kept state is [heads, D + 1, Dv + 1], 32-bit, and a column's walk needs
// nothing from another column.  Gates, decays, the state and the sums are 32-bit in both modes.  Two ways through a step's rows,
// which differ by rounding only; which one a span takes depends on its own length alone:
//   * the walk (any sizes, both modes; short spans and single tokens): in `mlstm_scan_kernel` a warp owns 32 columns of one head
//     of one request and walks the request's rows of the step in order, its column of S in registers, the rows' q, k and gates
//     staged in shared memory a tile of rows at a time by a second warp (the next tile comes in while a tile is walked); it
//     leaves S^T q per column, n . q and m per row.  `mlstm_output_kernel` divides, norms per head and gates.
//   * chunks of 64 rows on the tensor cores (bfloat16, longer spans, heads of up to 128), further below.
#include "mma_helpers.cuh"

// Rows staged at a time: as many as make the staged q and k 2 x 1024 values, at most 32 (a lane computes one row's gates).
template <int DMAX> struct MlstmTile { static constexpr int TT = 1024 / DMAX < 32 ? 1024 / DMAX : 32; };

__device__ __forceinline__ float mlstm_logsigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

// Two warps a block: warp 1 brings the rows of the next tile from memory into one of two shared buffers (q scaled, k, the
// lanes' values, the two log gates, all as 32-bit numbers; zeros beyond D and beyond the span) while warp 0, which owns the 32
// columns, walks the tile before; they meet at one barrier a tile.
template <typename T, int DMAX>
__global__ void __launch_bounds__(64) mlstm_scan_kernel(
    float* __restrict__ part, const T* __restrict__ y, int y_stride, int q_at, int k_at, int v_at, int i_at, int f_at,
    const float* __restrict__ bias_i, const float* __restrict__ bias_f, float cap, float* __restrict__ state,
    const int* __restrict__ cu_q, const int* __restrict__ slot_ids, int num_slots, int* __restrict__ status, int H, int D, int Dv,
    int write_state, int max_rows) {
    constexpr int TT = MlstmTile<DMAX>::TT, PER = TT * DMAX / 32;      // staged values of q (and of k) a lane brings
    __shared__ __align__(16) float sq[2][TT * DMAX], sk[2][TT * DMAX], sv[2][TT * 32], sg[2][TT * 2];
    pdl_trigger();
    pdl_wait();
    const int s = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.z * 32 + lane;         // this lane's column; column Dv is the normaliser
    const bool live = c <= Dv;
    const int r0 = cu_q[s], r1 = cu_q[s + 1];
    if (r1 <= r0 || r1 - r0 > max_rows) return;   // (a longer span is another kernel's)
    const int n_tiles = (r1 - r0 + TT - 1) / TT;

    if (warp == 1) {                              // ---- the rows' way into shared memory
        const float qscale = rsqrtf((float)D);
        const float bi = bias_i[h], bf = bias_f[h];
        for (int n = 0; n < n_tiles; ++n) {
            const int t0 = r0 + n * TT, nt = min(TT, r1 - t0), buf = n & 1;
            // all of the tile's loads are issued before any of them is used: one trip to memory a tile, not one a batch
            T fq[PER], fk[PER], fv[TT];
            float gate_i = 0.f, gate_f = 0.f;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int e = lane + 32 * i, tt = e / DMAX, d = e % DMAX;
                const bool ok = tt < nt && d < D;
                const T* row = y + (size_t)(t0 + (ok ? tt : 0)) * y_stride + h * D + (ok ? d : 0);
                fq[i] = ok ? row[q_at] : from_float<T>(0.f);
                fk[i] = ok ? row[k_at] : from_float<T>(0.f);
            }
#pragma unroll
            for (int tt = 0; tt < TT; ++tt)
                fv[tt] = (tt < nt && c < Dv) ? y[(size_t)(t0 + tt) * y_stride + v_at + h * Dv + c] : from_float<T>(1.f);
            if (lane < nt) {
                const T* row = y + (size_t)(t0 + lane) * y_stride;
                gate_i = to_float(row[i_at + h]);
                gate_f = to_float(row[f_at + h]);
            }
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                sq[buf][lane + 32 * i] = to_float(fq[i]) * qscale;
                sk[buf][lane + 32 * i] = to_float(fk[i]);
            }
#pragma unroll
            for (int tt = 0; tt < TT; ++tt) sv[buf][tt * 32 + lane] = to_float(fv[tt]);
            if (lane < nt) {
                sg[buf][2 * lane] = cap * tanhf((gate_i + bi) / cap);
                sg[buf][2 * lane + 1] = mlstm_logsigmoid(cap * tanhf((gate_f + bf) / cap));
            }
            __syncthreads();                      // tile n is there; tile n - 1 has been walked (its buffer is filled next)
        }
        __syncthreads();
        return;
    }

    // ---- the walk
    const int slot = zai_checked_slot(slot_ids[s], num_slots, status);
    float* st = state + (((size_t)slot * H + h) * (D + 1)) * (Dv + 1);
    float col[DMAX];
#pragma unroll
    for (int d = 0; d < DMAX; ++d) col[d] = (live && d < D) ? st[(size_t)d * (Dv + 1) + c] : 0.f;
    float m = live ? st[(size_t)D * (Dv + 1) + c] : 0.f;
    __syncthreads();                              // tile 0 is there
    for (int n = 0; n < n_tiles; ++n) {
        const int t0 = r0 + n * TT, nt = min(TT, r1 - t0), buf = n & 1;
        for (int tt = 0; tt < nt; ++tt) {
            const float gi = sg[buf][2 * tt], gf = sg[buf][2 * tt + 1];
            const float m_new = fmaxf(gf + m, gi);
            const float keep = expf(gf + m - m_new), take = expf(gi - m_new) * sv[buf][tt * 32 + lane];
            const float* qr = sq[buf] + tt * DMAX;
            const float* kr = sk[buf] + tt * DMAX;
            float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
            // (beyond D the staged q and k are zeros and the column stays zero: no bound is checked)
#pragma unroll
            for (int d = 0; d < DMAX; d += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(kr + d), q4 = *reinterpret_cast<const float4*>(qr + d);
                col[d] = fmaf(keep, col[d], take * k4.x);
                col[d + 1] = fmaf(keep, col[d + 1], take * k4.y);
                col[d + 2] = fmaf(keep, col[d + 2], take * k4.z);
                col[d + 3] = fmaf(keep, col[d + 3], take * k4.w);
                a0 = fmaf(col[d], q4.x, a0);
                a1 = fmaf(col[d + 1], q4.y, a1);
                a2 = fmaf(col[d + 2], q4.z, a2);
                a3 = fmaf(col[d + 3], q4.w, a3);
            }
            m = m_new;
            if (live) {
                float* o = part + ((size_t)(t0 + tt) * H + h) * (Dv + 2);
                o[c] = (a0 + a1) + (a2 + a3);
                if (c == Dv) o[Dv + 1] = m_new;
            }
        }
        __syncthreads();                          // this tile's buffer may be filled again; the next tile is there
    }
    if (write_state && live) {
#pragma unroll
        for (int d = 0; d < DMAX; ++d)
            if (d < D) st[(size_t)d * (Dv + 1) + c] = col[d];
        st[(size_t)D * (Dv + 1) + c] = m;
    }
}

// part [N, H, Dv + 2]: S^T q per column, then n . q, then m.  One block a row, a warp a head at a time.  Rows of spans longer
// than max_rows are left alone.
template <typename T>
__global__ void __launch_bounds__(128) mlstm_output_kernel(T* __restrict__ out, const float* __restrict__ part, const T* __restrict__ gate,
                                                           int gate_stride, const float* __restrict__ weight, float eps, int H, int Dv,
                                                           const int* __restrict__ cu_q, const int* __restrict__ seq_idx, int max_rows) {
    pdl_trigger();
    pdl_wait();
    if (seq_idx) {
        const int s = seq_idx[blockIdx.x];
        if (cu_q[s + 1] - cu_q[s] > max_rows) return;
    }
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    for (int h = warp; h < H; h += nwarp) {
        const float* p = part + ((size_t)t * H + h) * (Dv + 2);
        const float den = fmaxf(fabsf(p[Dv]), expf(-p[Dv + 1])) + 1e-6f;
        float ss = 0.f;
        for (int c = lane; c < Dv; c += 32) {
            const float o = p[c] / den;
            ss += o * o;
        }
        const float inv = rsqrtf(warp_sum(ss) / (float)Dv + eps);
        for (int c = lane; c < Dv; c += 32) {
            const float g = to_float(gate[(size_t)t * gate_stride + h * Dv + c]);
            out[((size_t)t * H + h) * Dv + c] = from_float<T>(p[c] / den * inv * weight[h * Dv + c] / (1.f + expf(-g)));
        }
    }
}

// ------------------------------------------------------------------------------------------------ chunks
// The walk is a chain of one request's rows (0.25 us a row on two warps, most of the chip idle); a portion of a prompt is cut
// into chunks of MLSTM_Q rows instead, whose sums are products on the tensor cores: 2048 rows of 8 heads of 64 x 128 take 46 us
// (launches included) where the walk took 520, of 8 heads of 128 x 128 69 us (1300).  Chunks of 64 rows make 256 blocks of such a
// portion, all of them on the chip at once; what is left is the latency of three kernels that read 20 MB from L2.  With F_t the sum of the log forget gates
// from the chunk's first row to row t, u_s = i_s - F_s and M_t = max(m_in, max_{s <= t} u_s), the recurrence unrolls to
//
//   m_t = F_t + M_t,   S_t = exp(m_in - M_t) S_in + sum_{s <= t} exp(u_s - M_t) k_s v_s^T       (n_t: the same with v = 1)
//
//   pass 1   E = sum_s exp(u_s - a) k_s v_s^T with a = max_s u_s, for every chunk at once (no weight is above 1)
//   pass 2   m_out = F_last + max(m_in, a);  S <- exp(F_last + m_in - m_out) S + exp(F_last + a - m_out) E across a request's
//            chunks, E replaced by the state before its chunk
//   pass 3   the read-outs of a chunk's 64 rows of one head, their division, norm and gate, for every chunk at once
//
// q, k and v are bfloat16 and go into the products as they are; the weighted v, the weighted scores and the state are 32-bit
// and go in as three bfloat16 parts (24 bits) with 32-bit sums.  F and u are summed in 64-bit and kept as two 32-bit numbers,
// so that a difference of two is good to the last bits whatever the rows before it summed up to.
#define MLSTM_Q 64                  // rows of a chunk
#define MLSTM_PAD 8                 // bfloat16 values behind every row in shared memory (no bank conflicts for ldmatrix)

struct MlstmArgs {
    const bf16* y;
    int y_stride, q_at, k_at, v_at, g_at, i_at, f_at;
    const float *bias_i, *bias_f;
    float cap;
    float* state;                   // [num_slots, H, D + 1, Dv + 1]
    const int *cu_q, *slot_ids;
    int* status;
    int num_slots, n_seqs, H, D, Dv, write_state, min_rows;
    float* ends;                    // [chunks, H, D, VP]: E with the normaliser as column Dv, then the state before the chunk
    double* gates;                  // [chunks, H, 2]: F_last and a
    float* m_in;                    // [chunks, H]: the running maximum before the chunk
    int VP;                         // Dv + 1 rounded up to a multiple of four
};

// Chunk b among all chunks of the step: the spans of min_rows rows or more in order, each cut into chunks of MLSTM_Q rows.
// `first`: the request whose first chunk of the step it is, else -1.
__device__ __forceinline__ bool mlstm_find_chunk(const MlstmArgs& a, int b, int& t0, int& t1, int& first) {
    for (int s = 0; s < a.n_seqs; ++s) {
        const int lo = a.cu_q[s], hi = a.cu_q[s + 1];
        if (hi - lo < a.min_rows) continue;
        const int n = (hi - lo + MLSTM_Q - 1) / MLSTM_Q;
        if (b < n) {
            t0 = lo + b * MLSTM_Q;
            t1 = min(t0 + MLSTM_Q, hi);
            first = b == 0 ? s : -1;
            return true;
        }
        b -= n;
    }
    return false;
}

// a double as two 32-bit numbers, and the difference of two such pairs
__device__ __forceinline__ float2 mlstm_pair(double v) {
    const float hi = (float)v;
    return make_float2(hi, (float)(v - (double)hi));
}
__device__ __forceinline__ float mlstm_minus(float2 a, float2 b) { return (a.x - b.x) + (a.y - b.y); }

#define MLSTM_LOG2E 1.4426950408889634

// The gates of the chunk's rows, by the first 64 threads (everyone calls it): s_u[j] = u_j and, with `s_top`, s_top[j] = the
// largest u up to row j, both in units of ln 2 as pairs; s_f[j] = F_j (natural).  Rows beyond the chunk repeat its last sums
// with u = -inf.  s_carry holds two values.
__device__ __forceinline__ void mlstm_gates(const MlstmArgs& a, int h, int t0, int t1, float2* s_u, double* s_top, double* s_f, double* s_carry) {
    const int j = threadIdx.x, lane = threadIdx.x & 31;
    double F = 0.0, u = -INFINITY, gi = 0.0;
    const bool live = j < MLSTM_Q && t0 + j < t1;
    if (j < MLSTM_Q) {
        if (live) {
            const bf16* row = a.y + (size_t)(t0 + j) * a.y_stride;
            gi = (double)(a.cap * tanhf((to_float(row[a.i_at + h]) + a.bias_i[h]) / a.cap));
            F = (double)mlstm_logsigmoid(a.cap * tanhf((to_float(row[a.f_at + h]) + a.bias_f[h]) / a.cap));
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, F, o);
            if (lane >= o) F += up;
        }
        if (j == 31) s_carry[0] = F;
    }
    __syncthreads();
    if (j < MLSTM_Q) {
        if (j >= 32) F += s_carry[0];
        if (live) u = gi - F;
        double top = u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, top, o);
            if (lane >= o) top = fmax(top, up);
        }
        if (j == 31) s_carry[1] = top;
        s_u[j] = live ? mlstm_pair(u * MLSTM_LOG2E) : make_float2(-INFINITY, 0.f);
        s_top[j] = top;
        s_f[j] = F;
    }
    __syncthreads();
    if (j >= 32 && j < MLSTM_Q) s_top[j] = fmax(s_top[j], s_carry[1]);
    __syncthreads();
}

// rows t0.. of a column slice of y into shared memory [MLSTM_Q][ld] (zeros beyond the chunk and beyond `cols` up to `cols_p`)
__device__ __forceinline__ void mlstm_load_rows(bf16* dst, int ld, const MlstmArgs& a, int at, int cols, int cols_p, int t0, int t1) {
    const bool vec = ((cols | at | a.y_stride) & 7) == 0 && (reinterpret_cast<uintptr_t>(a.y) & 15) == 0;
    if (vec) {
        const int per = cols_p >> 3;
        for (int i = threadIdx.x; i < MLSTM_Q * per; i += blockDim.x) {
            const int r = i / per, c = (i % per) * 8;
            const bool ok = t0 + r < t1 && c < cols;
            cp_async16(dst + r * ld + c, a.y + (ok ? (size_t)(t0 + r) * a.y_stride + at + c : 0), ok);
        }
    } else {
        for (int i = threadIdx.x; i < MLSTM_Q * cols_p; i += blockDim.x) {
            const int r = i / cols_p, c = i % cols_p;
            dst[r * ld + c] = (t0 + r < t1 && c < cols) ? a.y[(size_t)(t0 + r) * a.y_stride + at + c] : __float2bfloat16_rn(0.f);
        }
    }
}

// pass 1: a block makes 64 columns of a chunk's E of one head (eight warps, each in turn 16 rows of S x 32 columns); the block
// of the first columns also the normaliser.
__global__ void __launch_bounds__(256) mlstm_chunk_state_kernel(const MlstmArgs a) {
    extern __shared__ __align__(16) unsigned char ml_raw[];
    __shared__ float2 s_u[MLSTM_Q];
    __shared__ double s_top[MLSTM_Q], s_f[MLSTM_Q], s_carry[2];
    __shared__ float s_w[MLSTM_Q];
    constexpr int VT = 64, LDX = VT + MLSTM_PAD;
    const int dp = (a.D + 15) & ~15, ldk = dp + MLSTM_PAD;
    bf16* sk = reinterpret_cast<bf16*>(ml_raw);              // [Q][ldk]
    bf16* sx = sk + MLSTM_Q * ldk;                           // [3][Q][LDX]
    pdl_trigger();
    pdl_wait();
    int t0, t1, first;
    if (!mlstm_find_chunk(a, blockIdx.x, t0, t1, first)) return;
    const int h = blockIdx.y, v0 = blockIdx.z * VT, nv = min(VT, a.Dv - v0);
    mlstm_load_rows(sx, LDX, a, a.v_at + h * a.Dv + v0, nv, VT, t0, t1);
    cp_async_commit();
    mlstm_load_rows(sk, ldk, a, a.k_at + h * a.D, a.D, dp, t0, t1);
    cp_async_commit();
    mlstm_gates(a, h, t0, t1, s_u, s_top, s_f, s_carry);
    const double top = s_top[MLSTM_Q - 1];
    if (threadIdx.x < MLSTM_Q) s_w[threadIdx.x] = exp2f(mlstm_minus(s_u[threadIdx.x], mlstm_pair(top * MLSTM_LOG2E)));
    if (threadIdx.x == 0 && v0 == 0) {
        double* g = a.gates + ((size_t)blockIdx.x * a.H + h) * 2;
        g[0] = s_f[MLSTM_Q - 1];
        g[1] = top;
        if (first >= 0) {                                    // the request's maximum before the step (pass 2 replaces it)
            const int slot = zai_checked_slot(a.slot_ids[first], a.num_slots, a.status);
            a.m_in[(size_t)blockIdx.x * a.H + h] = a.state[(((size_t)slot * a.H + h) * (a.D + 1) + a.D) * (a.Dv + 1) + a.Dv];
        }
    }
    cp_async_wait<1>();
    __syncthreads();
#pragma unroll
    for (int i = threadIdx.x; i < MLSTM_Q * VT / 2; i += 256) {
        const int j = i / (VT / 2), c = (i % (VT / 2)) * 2;
        uint32_t* p = reinterpret_cast<uint32_t*>(sx + j * LDX + c);
        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
        const float w = s_w[j];
        uint32_t q[3];
        split3_pair(x.x * w, x.y * w, q);
        p[0] = q[0];
        p[MLSTM_Q * LDX / 2] = q[1];
        p[MLSTM_Q * LDX] = q[2];
    }
    cp_async_wait<0>();
    __syncthreads();
    float* e = a.ends + ((size_t)blockIdx.x * a.H + h) * a.D * a.VP;
    if (v0 == 0)
        for (int d = threadIdx.x; d < a.D; d += 256) {
            float n0 = 0.f, n1 = 0.f;
            for (int j = 0; j < MLSTM_Q; j += 2) {
                n0 = fmaf(s_w[j], __bfloat162float(sk[j * ldk + d]), n0);
                n1 = fmaf(s_w[j + 1], __bfloat162float(sk[(j + 1) * ldk + d]), n1);
            }
            e[(size_t)d * a.VP + a.Dv] = n0 + n1;
        }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, mi = lane >> 3, r8 = lane & 7, tq = lane & 3;
    for (int item = warp; item < dp / 16 * 2; item += 8) {
        const int mt = item >> 1, vb = (item & 1) * 32;
        if (vb >= nv) continue;
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < MLSTM_Q / 16; ++ks) {
            uint32_t fa[4];
            ldmatrix_x4_trans(fa, sk + (ks * 16 + (mi >> 1) * 8 + r8) * ldk + mt * 16 + (mi & 1) * 8);
#pragma unroll
            for (int p = 2; p >= 0; --p) {                   // the small parts first
#pragma unroll
                for (int vp = 0; vp < 2; ++vp) {
                    uint32_t fb[4];
                    ldmatrix_x4_trans(fb, sx + (p * MLSTM_Q + ks * 16 + (mi & 1) * 8 + r8) * LDX + vb + vp * 16 + (mi >> 1) * 8);
                    mma_bf16(acc[2 * vp], fa, fb[0], fb[1]);
                    mma_bf16(acc[2 * vp + 1], fa, fb[2], fb[3]);
                }
            }
        }
        const int d = mt * 16 + (lane >> 2);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c = vb + i * 8 + 2 * tq;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int dd = d + 8 * half;
                if (dd >= a.D || c >= nv) continue;
                float* p = e + (size_t)dd * a.VP + v0 + c;   // (VP is even: a pair of columns is one 8-byte store)
                if (c + 1 < nv) *reinterpret_cast<float2*>(p) = make_float2(acc[i][2 * half], acc[i][2 * half + 1]);
                else p[0] = acc[i][2 * half];
            }
        }
    }
}

// pass 2: a thread carries four neighbouring columns of one row of S across every chunk of a request; the maximum's
// way is the same sum in every thread.
__global__ void __launch_bounds__(128) mlstm_state_pass_kernel(const MlstmArgs a) {
    constexpr int AHEAD = 8;                                 // chunks whose loads are in flight
    pdl_trigger();
    pdl_wait();
    // (one dimension, which holds any number of requests: blocks of a head's state fastest, then heads, then requests)
    const int blocks = (a.D * (a.VP / 4) + 127) / 128, h = blockIdx.x / blocks % a.H, s = blockIdx.x / blocks / a.H;
    const int rows = a.cu_q[s + 1] - a.cu_q[s];
    if (rows < a.min_rows) return;
    int c0 = 0;
    for (int q = 0; q < s; ++q) {
        const int n = a.cu_q[q + 1] - a.cu_q[q];
        if (n >= a.min_rows) c0 += (n + MLSTM_Q - 1) / MLSTM_Q;
    }
    const int nc = (rows + MLSTM_Q - 1) / MLSTM_Q, per = a.VP / 4;
    const int idx = blockIdx.x % blocks * blockDim.x + threadIdx.x;
    if (idx >= a.D * per) return;
    const int d = idx / per, col = (idx % per) * 4, cols = a.Dv + 1;
    const int slot = zai_checked_slot(a.slot_ids[s], a.num_slots, a.status);
    float* st = a.state + ((size_t)slot * a.H + h) * (a.D + 1) * cols;
    float S[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) S[k] = col + k < cols ? st[(size_t)d * cols + col + k] : 0.f;
    float m = a.m_in[(size_t)c0 * a.H + h];
    const size_t step = (size_t)a.H * a.D * a.VP;
    float* e0 = a.ends + ((size_t)c0 * a.H + h) * a.D * a.VP + (size_t)d * a.VP + col;
    const double* g0 = a.gates + ((size_t)c0 * a.H + h) * 2;
    for (int c = 0; c < nc; c += AHEAD) {
        float4 e[AHEAD];
        double2 g[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            if (c + i >= nc) continue;
            e[i] = *reinterpret_cast<const float4*>(e0 + (size_t)(c + i) * step);
            g[i] = *reinterpret_cast<const double2*>(g0 + (size_t)(c + i) * a.H * 2);
        }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            if (c + i >= nc) continue;
            *reinterpret_cast<float4*>(e0 + (size_t)(c + i) * step) = make_float4(S[0], S[1], S[2], S[3]);
            if (idx == 0 && c + i > 0) a.m_in[(size_t)(c0 + c + i) * a.H + h] = m;
            const double from = g[i].x + (double)m, own = g[i].x + g[i].y;
            const float m_out = (float)fmax(from, own);
            const float keep = expf((float)(from - (double)m_out)), take = expf((float)(own - (double)m_out));
            S[0] = fmaf(keep, S[0], take * e[i].x);
            S[1] = fmaf(keep, S[1], take * e[i].y);
            S[2] = fmaf(keep, S[2], take * e[i].z);
            S[3] = fmaf(keep, S[3], take * e[i].w);
            m = m_out;
        }
    }
    if (a.write_state) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (col + k < cols) {
                st[(size_t)d * cols + col + k] = S[k];
                if (d == 0) st[(size_t)a.D * cols + col + k] = m;
            }
    }
}

// pass 3: a block makes the 64 output rows of a chunk of one head.  Eight warps: 16 rows x half of the columns each; the scores
// are made by both halves.  VT: columns, Dv rounded up.
template <int VT>
__global__ void __launch_bounds__(256) mlstm_chunk_out_kernel(const MlstmArgs a, bf16* __restrict__ out, const float* __restrict__ weight, float eps) {
    extern __shared__ __align__(16) unsigned char ml_raw[];
    __shared__ float2 s_u[MLSTM_Q];
    __shared__ double s_top[MLSTM_Q], s_f[MLSTM_Q], s_carry[2];
    __shared__ float s_nq[MLSTM_Q], s_ss[2][MLSTM_Q];
    __shared__ int s_odd, s_from[VT];                        // a value of v that is infinite or NaN: whether, and a column's first row with one
    constexpr int LDX = VT + MLSTM_PAD, VW = VT / 2;
    const int dp = (a.D + 15) & ~15, ldk = dp + MLSTM_PAD;
    bf16* sq = reinterpret_cast<bf16*>(ml_raw);              // [Q][ldk]
    bf16* sk = sq + MLSTM_Q * ldk;                           // [Q][ldk]
    bf16* sv = sk + MLSTM_Q * ldk;                           // [Q][LDX]
    bf16* sg = sv + MLSTM_Q * LDX;                           // [Q][LDX]: the output gate
    bf16* ss = sg + MLSTM_Q * LDX;                           // [3][dp][LDX]: the state before the chunk
    float* sn = reinterpret_cast<float*>(ss + 3 * dp * LDX); // [dp]: its normaliser
    pdl_trigger();
    pdl_wait();
    int t0, t1, first;
    if (!mlstm_find_chunk(a, blockIdx.x, t0, t1, first)) return;
    if (threadIdx.x < VT) s_from[threadIdx.x] = MLSTM_Q;
    if (threadIdx.x == 0) s_odd = 0;
    const int h = blockIdx.y;
    mlstm_load_rows(sq, ldk, a, a.q_at + h * a.D, a.D, dp, t0, t1);
    mlstm_load_rows(sk, ldk, a, a.k_at + h * a.D, a.D, dp, t0, t1);
    mlstm_load_rows(sv, LDX, a, a.v_at + h * a.Dv, a.Dv, VT, t0, t1);
    mlstm_load_rows(sg, LDX, a, a.g_at + h * a.Dv, a.Dv, VT, t0, t1);
    cp_async_commit();
    const float* S = a.ends + ((size_t)blockIdx.x * a.H + h) * a.D * a.VP;
    const float m_in = a.m_in[(size_t)blockIdx.x * a.H + h];
    {
        constexpr int PER = VT / 4, U = 4;                   // four loads in flight a thread
        for (int i0 = threadIdx.x; i0 < dp * PER; i0 += 256 * U) {
            float4 v[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const int i = i0 + 256 * k, d = i / PER, c = (i % PER) * 4;
                v[k] = (d < a.D && c < a.Dv) ? *reinterpret_cast<const float4*>(S + (size_t)d * a.VP + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                if (c + 1 >= a.Dv) v[k].y = 0.f;             // (columns from Dv on hold the normaliser and padding)
                if (c + 2 >= a.Dv) v[k].z = 0.f;
                if (c + 3 >= a.Dv) v[k].w = 0.f;
            }
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const int i = i0 + 256 * k, d = i / PER, c = (i % PER) * 4;
                if (d >= dp) continue;
                uint32_t p[3], q[3];
                split3_pair(v[k].x, v[k].y, p);
                split3_pair(v[k].z, v[k].w, q);
#pragma unroll
                for (int m = 0; m < 3; ++m) *reinterpret_cast<uint2*>(ss + (m * dp + d) * LDX + c) = make_uint2(p[m], q[m]);
            }
        }
    }
    for (int d = threadIdx.x; d < dp; d += 256) sn[d] = d < a.D ? S[(size_t)d * a.VP + a.Dv] : 0.f;
    mlstm_gates(a, h, t0, t1, s_u, s_top, s_f, s_carry);
    cp_async_wait<0>();
    __syncthreads();
    {   // n . q of every row, four threads a row
        const int r = threadIdx.x >> 2, part = threadIdx.x & 3;
        float n = 0.f;
        for (int d = part * 2; d < dp; d += 8) {
            const float2 q = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sq + r * ldk + d));
            n = fmaf(q.x, sn[d], fmaf(q.y, sn[d + 1], n));
        }
        n += __shfl_xor_sync(0xffffffffu, n, 1);
        n += __shfl_xor_sync(0xffffffffu, n, 2);
        if (part == 0) s_nq[r] = n;
    }
    // (a later row's weight is zero, and zero times such a value is NaN: it leaves the product, and its column ends as NaN from its row on)
    for (int i = threadIdx.x; i < MLSTM_Q * (VT / 8); i += 256) {
        const int r = i / (VT / 8), c = (i % (VT / 8)) * 8;
        uint32_t* p = reinterpret_cast<uint32_t*>(sv + r * LDX + c);
        const uint4 x = *reinterpret_cast<const uint4*>(p);
        if ((not_finite_pair(x.x) | not_finite_pair(x.y) | not_finite_pair(x.z) | not_finite_pair(x.w)) == 0) continue;
        for (int k = 0; k < 8; ++k)
            if (not_finite_pair(p[k >> 1]) >> (k & 1 ? 31 : 15) & 1) {
                sv[r * LDX + c + k] = __float2bfloat16_rn(0.f);
                atomicMin(&s_from[c + k], r);
            }
        s_odd = 1;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, mi = lane >> 3, r8 = lane & 7, tq = lane & 3;
    const int wr = warp & 3, side = warp >> 2, vb = side * VW;
    const int i0 = wr * 16, ra = i0 + (lane >> 2), rb = ra + 8;
    const double Ma = fmax((double)m_in, s_top[ra]), Mb = fmax((double)m_in, s_top[rb]);
    const float2 la = mlstm_pair(Ma * MLSTM_LOG2E), lb = mlstm_pair(Mb * MLSTM_LOG2E);

    // scores q . k of this warp's rows with the rows up to its own last one, and the read-out of the state before the chunk
    float sco[MLSTM_Q / 8][4], acc[VW / 8][4];
#pragma unroll
    for (int i = 0; i < MLSTM_Q / 8; ++i) sco[i][0] = sco[i][1] = sco[i][2] = sco[i][3] = 0.f;
#pragma unroll
    for (int i = 0; i < VW / 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll 2
    for (int ks = 0; ks < dp / 16; ++ks) {
        uint32_t fa[4];
        ldmatrix_x4(fa, sq + (i0 + (mi & 1) * 8 + r8) * ldk + ks * 16 + (mi >> 1) * 8);
#pragma unroll
        for (int jp = 0; jp < MLSTM_Q / 16; ++jp) {
            if (jp > wr) continue;
            uint32_t fb[4];
            ldmatrix_x4(fb, sk + (jp * 16 + (mi >> 1) * 8 + r8) * ldk + ks * 16 + (mi & 1) * 8);
            mma_bf16(sco[2 * jp], fa, fb[0], fb[1]);
            mma_bf16(sco[2 * jp + 1], fa, fb[2], fb[3]);
        }
#pragma unroll
        for (int p = 2; p >= 0; --p) {
#pragma unroll
            for (int vp = 0; vp < VW / 16; ++vp) {
                uint32_t fb[4];
                ldmatrix_x4_trans(fb, ss + (p * dp + ks * 16 + (mi & 1) * 8 + r8) * LDX + vb + vp * 16 + (mi >> 1) * 8);
                mma_bf16(acc[2 * vp], fa, fb[0], fb[1]);
                mma_bf16(acc[2 * vp + 1], fa, fb[2], fb[3]);
            }
        }
    }
    const float qs = rsqrtf((float)a.D);
    const float ea = expf((float)((double)m_in - Ma)) * qs, eb = expf((float)((double)m_in - Mb)) * qs;
#pragma unroll
    for (int i = 0; i < VW / 8; ++i) {
        acc[i][0] *= ea; acc[i][1] *= ea; acc[i][2] *= eb; acc[i][3] *= eb;
    }
    if (s_odd) {
#pragma unroll
        for (int i = 0; i < VW / 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if ((e < 2 ? ra : rb) >= s_from[vb + i * 8 + 2 * tq + (e & 1)]) acc[i][e] = __int_as_float(0x7fc00000);
    }
    // the chunk's own rows
    float na = 0.f, nb = 0.f;
#pragma unroll
    for (int ks = 0; ks < MLSTM_Q / 16; ++ks) {
        if (ks > wr) continue;
        uint32_t f[3][4];
#pragma unroll
        for (int half = 0; half < 2; ++half) {               // columns ks * 16 + 8 half + 2 tq, + 1
            const int j = ks * 16 + 8 * half + 2 * tq;
            const float2 u0 = s_u[j], u1 = s_u[j + 1];
            const float* g4 = sco[2 * ks + half];
            const float a0 = j <= ra ? g4[0] * (exp2f(mlstm_minus(u0, la)) * qs) : 0.f;
            const float a1 = j + 1 <= ra ? g4[1] * (exp2f(mlstm_minus(u1, la)) * qs) : 0.f;
            const float b0 = j <= rb ? g4[2] * (exp2f(mlstm_minus(u0, lb)) * qs) : 0.f;
            const float b1 = j + 1 <= rb ? g4[3] * (exp2f(mlstm_minus(u1, lb)) * qs) : 0.f;
            na += a0 + a1;
            nb += b0 + b1;
            uint32_t p[3], q[3];
            split3_pair(a0, a1, p);
            split3_pair(b0, b1, q);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                f[k][2 * half] = p[k];
                f[k][2 * half + 1] = q[k];
            }
        }
#pragma unroll
        for (int vp = 0; vp < VW / 16; ++vp) {
            uint32_t fb[4];
            ldmatrix_x4_trans(fb, sv + (ks * 16 + (mi & 1) * 8 + r8) * LDX + vb + vp * 16 + (mi >> 1) * 8);
#pragma unroll
            for (int p = 2; p >= 0; --p) {
                mma_bf16(acc[2 * vp], f[p], fb[0], fb[1]);
                mma_bf16(acc[2 * vp + 1], f[p], fb[2], fb[3]);
            }
        }
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        na += __shfl_xor_sync(0xffffffffu, na, o);
        nb += __shfl_xor_sync(0xffffffffu, nb, o);
    }
    const float da = fmaxf(fabsf(fmaf(ea, s_nq[ra], na)), expf(-(float)(s_f[ra] + Ma))) + 1e-6f;
    const float db = fmaxf(fabsf(fmaf(eb, s_nq[rb], nb)), expf(-(float)(s_f[rb] + Mb))) + 1e-6f;
    float qa = 0.f, qb = 0.f;                                // (columns beyond Dv are zeros)
#pragma unroll
    for (int i = 0; i < VW / 8; ++i) {
        acc[i][0] /= da; acc[i][1] /= da; acc[i][2] /= db; acc[i][3] /= db;
        qa += acc[i][0] * acc[i][0] + acc[i][1] * acc[i][1];
        qb += acc[i][2] * acc[i][2] + acc[i][3] * acc[i][3];
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        qa += __shfl_xor_sync(0xffffffffu, qa, o);
        qb += __shfl_xor_sync(0xffffffffu, qb, o);
    }
    if (tq == 0) {
        s_ss[side][ra] = qa;
        s_ss[side][rb] = qb;
    }
    __syncthreads();
    const float ia = rsqrtf((s_ss[0][ra] + s_ss[1][ra]) / (float)a.Dv + eps), ib = rsqrtf((s_ss[0][rb] + s_ss[1][rb]) / (float)a.Dv + eps);
    const bool even = (a.Dv & 1) == 0;
#pragma unroll
    for (int i = 0; i < VW / 8; ++i) {
        const int c = vb + i * 8 + 2 * tq;
        if (c >= a.Dv) continue;
        const bool two = c + 1 < a.Dv;
        const float w0 = weight[h * a.Dv + c], w1 = two ? weight[h * a.Dv + c + 1] : 0.f;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = half ? rb : ra;
            if (t0 + r >= t1) continue;
            const float inv = half ? ib : ia;
            const float y0 = acc[i][2 * half] * inv * w0 / (1.f + expf(-__bfloat162float(sg[r * LDX + c])));
            const float y1 = acc[i][2 * half + 1] * inv * w1 / (1.f + expf(-__bfloat162float(sg[r * LDX + c + 1])));
            bf16* o = out + ((size_t)(t0 + r) * a.H + h) * a.Dv + c;
            if (even) *reinterpret_cast<uint32_t*>(o) = pack_bf16(y0, y1);
            else { o[0] = __float2bfloat16_rn(y0); if (two) o[1] = __float2bfloat16_rn(y1); }
        }
    }
}

static size_t mlstm_state_smem(int D) {
    const size_t dp = (D + 15) & ~15;
    return (MLSTM_Q * (dp + MLSTM_PAD) + 3 * MLSTM_Q * (64 + MLSTM_PAD)) * sizeof(bf16);
}
static size_t mlstm_out_smem(int D, int VT) {
    const size_t dp = (D + 15) & ~15, ldx = VT + MLSTM_PAD;
    return (2 * MLSTM_Q * (dp + MLSTM_PAD) + 2 * MLSTM_Q * ldx + 3 * dp * ldx) * sizeof(bf16) + dp * sizeof(float);
}

ZAI_API int zai_mlstm_chunk_rows() { return MLSTM_Q; }
// 1 if spans of these head sizes can run in chunks (the state of a head and a chunk's rows in one block's shared memory)
ZAI_API int zai_mlstm_chunked_supports(int D, int Dv) { return D >= 1 && D <= 128 && Dv >= 1 && Dv <= 128; }

template <int VT>
static int mlstm_chunk_out(const MlstmArgs& a, bf16* out, const float* weight, float eps, int max_chunks, cudaStream_t stream) {
    static unsigned long long done = 0;
    if (zai_first_on_device(&done)) {
        const cudaError_t e = cudaFuncSetAttribute(mlstm_chunk_out_kernel<VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlstm_out_smem(128, VT));
        if (e != cudaSuccess) return (int)e;
    }
    return launch_pdl(mlstm_chunk_out_kernel<VT>, dim3(max_chunks, a.H), dim3(256), mlstm_out_smem(a.D, VT), stream, a, out, weight, eps);
}

// The same as zai_mlstm (out and state) over every span of min_rows rows or more, bfloat16, in chunks on the tensor cores.  ends
// [max_chunks, H, D, Dv + 1 rounded up to 4] and m_in [max_chunks, H] 32-bit, gates [max_chunks, H, 2] 64-bit: scratch;
// rows / MLSTM_Q + n_seqs chunks are always enough.
ZAI_API int zai_mlstm_chunked(void* out, const void* y, int y_stride, int q_at, int k_at, int v_at, int g_at, int i_at, int f_at,
                              const float* bias_i, const float* bias_f, float cap, const float* weight, float eps, float* state,
                              const int* cu_q, const int* slot_ids, int num_slots, int* status, int n_seqs, int H, int D, int Dv,
                              int write_state, int min_rows, float* ends, double* gates, float* m_in, int max_chunks, cudaStream_t stream) {
    if (n_seqs <= 0 || max_chunks <= 0) return ZAI_OK;
    if (H < 1 || H > 65535 || cap <= 0.f || !zai_mlstm_chunked_supports(D, Dv)) return ZAI_BAD_SIZE;
    const MlstmArgs a = {(const bf16*)y, y_stride, q_at, k_at, v_at, g_at, i_at, f_at, bias_i, bias_f, cap, state, cu_q, slot_ids, status,
                         num_slots, n_seqs, H, D, Dv, write_state, min_rows < 1 ? 1 : min_rows, ends, gates, m_in, (Dv + 4) & ~3};
    static unsigned long long done = 0;
    if (zai_first_on_device(&done)) {
        const cudaError_t e = cudaFuncSetAttribute(mlstm_chunk_state_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlstm_state_smem(128));
        if (e != cudaSuccess) return (int)e;
    }
    int rc = launch_pdl(mlstm_chunk_state_kernel, dim3(max_chunks, H, (Dv + 63) / 64), dim3(256), mlstm_state_smem(D), stream, a);
    if (rc) return rc;
    const long long blocks = (long long)n_seqs * H * ((D * (a.VP / 4) + 127) / 128);
    if (blocks > 0x7fffffffLL) return ZAI_BAD_SIZE;
    rc = launch_pdl(mlstm_state_pass_kernel, dim3((unsigned)blocks), dim3(128), 0, stream, a);
    if (rc) return rc;
    return Dv <= 64 ? mlstm_chunk_out<64>(a, (bf16*)out, weight, eps, max_chunks, stream)
                    : mlstm_chunk_out<128>(a, (bf16*)out, weight, eps, max_chunks, stream);
}

// y [N, y_stride]: the stacked projections, with q (H D), k (H D), v (H Dv), the gate (H Dv) and the two log gates' inputs (H
// each) starting at the given columns.  state [num_slots, H, D + 1, Dv + 1] 32-bit; part [N, H, Dv + 2] 32-bit scratch;
// out [N, H Dv].  With seq_idx [N] (the rows' requests) only spans of at most max_rows rows are run.
ZAI_API int zai_mlstm(void* out, float* part, const void* y, int y_stride, int dtype, int q_at, int k_at, int v_at, int g_at, int i_at,
                      int f_at, const float* bias_i, const float* bias_f, float cap, const float* weight, float eps, float* state,
                      const int* cu_q, const int* slot_ids, int num_slots, int* status, int N, int S, int H, int D, int Dv,
                      int write_state, const int* seq_idx, int max_rows, cudaStream_t stream) {
    if (N <= 0 || S <= 0) return ZAI_OK;
    if (H < 1 || H > 65535 || D < 1 || D > 256 || Dv < 1 || cap <= 0.f) return ZAI_BAD_SIZE;
    if (!seq_idx) max_rows = 0x7fffffff;
    const dim3 grid(S, H, (Dv + 1 + 31) / 32);
    int rc;
#define MLSTM_GO(DM) ZAI_DISPATCH(dtype, rc = launch_pdl(mlstm_scan_kernel<T, DM>, grid, dim3(64), 0, stream, part, (const T*)y, \
        y_stride, q_at, k_at, v_at, i_at, f_at, bias_i, bias_f, cap, state, cu_q, slot_ids, num_slots, status, H, D, Dv, write_state, max_rows))
    if (D <= 16) MLSTM_GO(16);
    else if (D <= 32) MLSTM_GO(32);
    else if (D <= 64) MLSTM_GO(64);
    else if (D <= 128) MLSTM_GO(128);
    else MLSTM_GO(256);
#undef MLSTM_GO
    if (rc != 0) return rc;
    ZAI_DISPATCH(dtype, return launch_pdl(mlstm_output_kernel<T>, dim3(N), dim3(128), 0, stream, (T*)out, part, (const T*)y + g_at,
                                          y_stride, weight, eps, H, Dv, cu_q, seq_idx, max_rows));
}
