// Causal grouped-query attention over the paged cache, general kernels (any element type, head size, page size, window): one
// warp per (row, query head), and for steps with spans of rows tiles of 32 (row, query head) pairs (further below).
//
//   s_j = q . k_j * scale  for cached positions j <= pos (and j > pos - window, or j in the chunk of pos), same request
//   o   = sum_j softmax(s)_j v_j
//
// Scale 1/sqrt(D) by default (src/transformer/hybrid_attn.zig:571), causal bound on the token's
// absolute position (:587; src/cuda/paged_attention.cu:245-248), max-subtracted softmax in 32-bit
// (:578-600), query head h reads kv head h / (Hq/Hkv) (src/cuda/paged_attention.cu:142).  Like the
// reference's kernels (paged_attention.cu:121-225, 230-337) a warp walks the keys with an online
// softmax; unlike them the lanes take 32 keys at a time for the scores and share each value row
// for the weighted sum.  Keys are always visited from the first visible position in steps of 32,
// so a row's result does not depend on how the request was cut into steps or on its batch.
// Pages: [num_pages, 2, Hkv, page_size, D].
//
// `zai_paged_attention_scored` is the same kernel with the options of designs that shape their scores (`ZaiScoreOptions`
// in common.cuh: a cap, a bias by distance, a sink, kept first positions under a window; here with the exact `tanhf`).
// The kept positions are a second range of keys, walked before the window's, again in steps of 32 from position 0.
#include <type_traits>

#include "common.cuh"


template <typename T, int MAXR, bool EXT>
__global__ void paged_attention_warp_kernel(T* __restrict__ out, const T* __restrict__ q, const T* __restrict__ pages,
                                            const int* __restrict__ block_table, int table_width,
                                            const int* __restrict__ positions, const int* __restrict__ seq_idx,
                                            int page_size, int Hq, int Hkv, int D, float scale, int window,
                                            int num_pages, int* __restrict__ status, const ZaiScoreOptions opt) {
    extern __shared__ float qs[];                 // [D]
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x, h = blockIdx.y, lane = threadIdx.x;
    const int kvh = h / (Hq / Hkv);
    const int pos = positions[t];
    const ZaiTableRow table{block_table + (size_t)seq_idx[t] * table_width, table_width, num_pages, status};
    const T* qrow = q + ((size_t)t * Hq + h) * D;
    for (int d = lane; d < D; d += 32) qs[d] = to_float(qrow[d]) * scale;
    __syncwarp();
    const int kend = pos + 1;
    const int kstart = zai_first_visible(pos, window);
    // kept first positions: the walk starts with them (in steps of 32 from position 0) and goes on at the window's start
    const int kept = EXT && window > 0 ? min(opt.keep_first, kstart) : 0;
    const size_t page_stride = (size_t)2 * Hkv * page_size * D;
    const size_t v_off = (size_t)Hkv * page_size * D;
    float m = -INFINITY, l = 0.f;
    float acc[MAXR];
#pragma unroll
    for (int r = 0; r < MAXR; ++r) acc[r] = 0.f;
    for (int part = kept > 0 ? 0 : 1; part < 2; ++part) {
    const int stop = part == 0 ? kept : kend;
    for (int base = part == 0 ? 0 : kstart; base < stop; base += 32) {
        const int j = base + lane;
        const bool valid = j < stop;
        float s = -INFINITY;
        size_t krow = 0;
        if (valid) {
            const int page = table.page(j / page_size);
            krow = (size_t)page * page_stride + ((size_t)kvh * page_size + (j % page_size)) * D;
            const T* kp = pages + krow;
            float dot = 0.f;
            for (int d = 0; d < D; ++d) dot += qs[d] * to_float(kp[d]);
            s = dot;
            if (EXT) {
                if (opt.softcap > 0.f) s = opt.softcap * tanhf(s / opt.softcap);
                if (opt.bias) s += opt.bias[(size_t)min(pos - j, opt.bias_rows - 1) * Hq + h];
            }
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float p = valid ? expf(s - m_new) : 0.f;
        const float corr = expf(m - m_new);                 // m = -inf at first: 0
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int r = 0; r < MAXR; ++r) acc[r] *= corr;
        const int n = min(32, stop - base);
        for (int jj = 0; jj < n; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const unsigned long long rj = __shfl_sync(0xffffffffu, (unsigned long long)krow, jj);
            const T* vp = pages + rj + v_off;
#pragma unroll
            for (int r = 0; r < MAXR; ++r) {
                const int d = lane + 32 * r;
                if (d < D) acc[r] += pj * to_float(vp[d]);
            }
        }
        m = m_new;
    }
    }
    if (EXT && opt.sink) {                                  // the sink: a term of the denominator alone
        const float sk = opt.sink[h], m_new = fmaxf(m, sk);
        const float corr = expf(m - m_new);
        l = l * corr + expf(sk - m_new);
#pragma unroll
        for (int r = 0; r < MAXR; ++r) acc[r] *= corr;
    }
    const float inv = 1.f / l;
    T* orow = out + ((size_t)t * Hq + h) * D;
#pragma unroll
    for (int r = 0; r < MAXR; ++r) {
        const int d = lane + 32 * r;
        if (d < D) orow[d] = from_float<T>(acc[r] * inv);
    }
}

// ---- spans of rows: a block owns AT_M (row, query head) pairs of one key/value head and one request (neighbouring rows, the heads
// that share the keys) and walks the keys in tiles of AT_N, 32-bit multiply-adds throughout.  A thread makes 4 pairs x 4 keys of the
// scores (rows ty 4 .., keys tx + 16 j) and 4 pairs x DM / 16 columns of the output; the 16 threads of a row are neighbouring lanes,
// so its maximum, sum and weights need no block barrier.  Key tiles start at multiples of AT_N whatever the span: a row's result is
// the same in any portion and batch (steps of single tokens run the kernel above, whose sums have another order).
//
// What bounds it: 32-bit multiply-adds; eight 16-byte loads from shared memory feed 64 of them, and four blocks an SM (two at 128)
// cover each other's loads and barriers.  A warp a row read every key and value from L2 once per row and head, keys by 32 lanes on
// 32 rows at a time.  32-bit, 16 heads
// of 64 over 8: 384 rows behind 128 positions 585 -> 64 us, 2048 rows 8585 -> 394 us (22 TFLOP/s of the about 70 of the units),
// 2 rows behind 2000 positions 403 -> 150; 32 rows alone 18 -> 22 (the call's host time).
#define AT_M 32
#define AT_N 64

template <int DM>
struct AtTile {
    static constexpr int LD = DM + 4;                        // (rows four banks apart)
    float q[AT_M][LD], k[AT_N][LD], v[AT_N][LD], p[AT_M][AT_N + 4];
    long long row[2][AT_N];                                  // where a tile's keys lie in the pages
};

// four neighbouring values of a row of D as 32-bit numbers, zeros beyond D; `vec`: D and the address are multiples of four
__device__ __forceinline__ float4 at_four(const float* p, int d, int D, bool vec) {
    if (vec && d < D) return *reinterpret_cast<const float4*>(p + d);
    return make_float4(d < D ? p[d] : 0.f, d + 1 < D ? p[d + 1] : 0.f, d + 2 < D ? p[d + 2] : 0.f, d + 3 < D ? p[d + 3] : 0.f);
}
__device__ __forceinline__ float4 at_four(const bf16* p, int d, int D, bool vec) {
    if (vec && d < D) {
        const uint2 v = *reinterpret_cast<const uint2*>(p + d);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
        const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
    return make_float4(d < D ? to_float(p[d]) : 0.f, d + 1 < D ? to_float(p[d + 1]) : 0.f, d + 2 < D ? to_float(p[d + 2]) : 0.f,
                       d + 3 < D ? to_float(p[d + 3]) : 0.f);
}

// AHEAD: a tile's keys and values are asked for while the tile before is used, and wait in registers
template <typename T, int DM, bool EXT, bool AHEAD>
__global__ void __launch_bounds__(128) paged_attention_tile_kernel(
    T* __restrict__ out, const T* __restrict__ q, const T* __restrict__ pages, const int* __restrict__ block_table, int table_width,
    const int* __restrict__ positions, const int* __restrict__ cu_q, int n_seqs, int page_size, int Hq, int Hkv, int D, float scale,
    int window, int num_pages, int* __restrict__ status, const ZaiScoreOptions opt) {
    using Tile = AtTile<DM>;
    constexpr int NC = DM / 16;                              // output columns of a thread: fours (twos) 64 (32) apart
    extern __shared__ __align__(16) unsigned char at_raw[];
    Tile& sm = *reinterpret_cast<Tile*>(at_raw);
    pdl_trigger();
    pdl_wait();
    const int kvh = blockIdx.y, group = Hq / Hkv, rows_of = AT_M / group;
    int seq = 0, r0 = 0, n_rows = 0, b = blockIdx.x;
    for (; seq < n_seqs; ++seq) {
        const int lo = cu_q[seq], len = cu_q[seq + 1] - lo, nt = (len + rows_of - 1) / rows_of;
        if (b < nt) {
            r0 = lo + b * rows_of;
            n_rows = min(rows_of, lo + len - r0);
            break;
        }
        b -= nt;
    }
    if (n_rows <= 0) return;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, n_pairs = n_rows * group;
    const ZaiTableRow table{block_table + (size_t)seq * table_width, table_width, num_pages, status};
    const size_t page_stride = (size_t)2 * Hkv * page_size * D, v_off = (size_t)Hkv * page_size * D;
    const bool vec = (D & 3) == 0 && ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(pages)) & (4 * sizeof(T) - 1)) == 0;
    const int first_pos = positions[r0], last_pos = positions[r0 + n_rows - 1];
    // a pair's query (scaled); pairs that do not exist are zeros
    for (int i = tid; i < AT_M * (DM / 4); i += 128) {
        const int p = i / (DM / 4), d = (i % (DM / 4)) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p < n_pairs) v = at_four(q + ((size_t)(r0 + p / group) * Hq + kvh * group + p % group) * D, d, D, vec);
        *reinterpret_cast<float4*>(&sm.q[p][d]) = make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale);
    }
    int pos[4], from[4], kept[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int p = ty * 4 + i;
        pos[i] = p < n_pairs ? first_pos + p / group : -1;   // (-1: sees no key)
        from[i] = zai_first_visible(pos[i], window);
        kept[i] = EXT && window > 0 ? min(opt.keep_first, from[i]) : 0;
    }
    // the tiles: those of the kept first positions, then from the first row's first visible one on
    const int seen_from = zai_first_visible(first_pos, window), start = seen_from / AT_N * AT_N;
    const int keep_end = EXT && window > 0 ? min(opt.keep_first, zai_first_visible(last_pos, window)) : 0;
    const int n_kept = min((keep_end + AT_N - 1) / AT_N, start / AT_N), n_tiles = n_kept + (last_pos - start) / AT_N + 1;
    auto base_of = [&](int n) { return n < n_kept ? n * AT_N : start + (n - n_kept) * AT_N; };
    auto find_rows = [&](int n) {
        if (tid < AT_N && n < n_tiles) {
            const int j = base_of(n) + tid;
            long long at = -1;                               // (no row sees it: zeros)
            if (j <= last_pos && (j >= seen_from || j < keep_end)) at = (long long)((size_t)table.page(j / page_size) * page_stride + ((size_t)kvh * page_size + j % page_size) * D);
            sm.row[n & 1][tid] = at;
        }
    };
    float m[4], l[4], o[4][NC];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < NC; ++c) o[i][c] = 0.f;
    }
    constexpr int PER = AT_N * (DM / 4) / 128;               // fours of keys (and of values) a thread brings of a tile
    float4 next_k[AHEAD ? PER : 1], next_v[AHEAD ? PER : 1];
    auto fetch = [&](int n, int r, float4& kv, float4& vv) { // the r-th of them
        const int i = tid + r * 128, j = i / (DM / 4), d = (i % (DM / 4)) * 4;
        const long long at = sm.row[n & 1][j];
        kv = vv = make_float4(0.f, 0.f, 0.f, 0.f);
        if (at >= 0) {
            kv = at_four(pages + at, d, D, vec);
            vv = at_four(pages + at + v_off, d, D, vec);
        }
    };
    find_rows(0);
    if (AHEAD) {
        __syncthreads();
#pragma unroll
        for (int r = 0; r < PER; ++r) fetch(0, r, next_k[r], next_v[r]);
    }
    for (int n = 0; n < n_tiles; ++n) {
        bool odd = false;                                    // one of the thread's values is infinite or NaN
        __syncthreads();                                     // the tile before has been used; this one's rows are known
        auto put = [&](int r, const float4& kv, const float4& vv) {
            const int i = tid + r * 128, j = i / (DM / 4), d = (i % (DM / 4)) * 4;
            *reinterpret_cast<float4*>(&sm.k[j][d]) = kv;
            *reinterpret_cast<float4*>(&sm.v[j][d]) = vv;
            odd |= !(fmaf(vv.x, 0.f, fmaf(vv.y, 0.f, fmaf(vv.z, 0.f, vv.w * 0.f))) == 0.f);       // (NaN for either)
        };
        if (AHEAD) {
#pragma unroll
            for (int r = 0; r < PER; ++r) put(r, next_k[r], next_v[r]);
        } else {
#pragma unroll 4
            for (int r = 0; r < PER; ++r) {
                float4 kv, vv;
                fetch(n, r, kv, vv);
                put(r, kv, vv);
            }
        }
        find_rows(n + 1);
        odd = __syncthreads_or(odd);
        if (AHEAD && n + 1 < n_tiles) {
#pragma unroll
            for (int r = 0; r < PER; ++r) fetch(n + 1, r, next_k[r], next_v[r]);
        }
        float s[4][4] = {};
#pragma unroll 4
        for (int d = 0; d < DM; d += 4) {
            float4 a[4], k4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(&sm.q[ty * 4 + i][d]);
#pragma unroll
            for (int j = 0; j < 4; ++j) k4[j] = *reinterpret_cast<const float4*>(&sm.k[tx + 16 * j][d]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = fmaf(a[i].w, k4[j].w, fmaf(a[i].z, k4[j].z, fmaf(a[i].y, k4[j].y, fmaf(a[i].x, k4[j].x, s[i][j]))));
        }
        const int base = base_of(n);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float top = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = base + tx + 16 * j;
                const bool seen = key <= pos[i] && (key >= from[i] || key < kept[i]);
                if (EXT && seen) {
                    if (opt.softcap > 0.f) s[i][j] = opt.softcap * tanhf(s[i][j] / opt.softcap);
                    if (opt.bias) s[i][j] += opt.bias[(size_t)min(pos[i] - key, opt.bias_rows - 1) * Hq + kvh * group + (ty * 4 + i) % group];
                }
                if (!seen) s[i][j] = -INFINITY;
                top = fmaxf(top, s[i][j]);
            }
#pragma unroll
            for (int w = 8; w > 0; w >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, w));
            const float m_new = fmaxf(m[i], top);
            const float ref = m_new == -INFINITY ? 0.f : m_new;               // (no key of the row so far: weights of zero)
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float w = expf(s[i][j] - ref);
                sm.p[ty * 4 + i][tx + 16 * j] = w;
                sum += w;
            }
#pragma unroll
            for (int w = 8; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
            const float corr = expf(m[i] - ref);                              // m = -inf at first: 0
            l[i] = l[i] * corr + sum;
            m[i] = m_new;
#pragma unroll
            for (int c = 0; c < NC; ++c) o[i][c] *= corr;
        }
        __syncwarp();                                        // (a row's weights come from its own 16 lanes)
        if (odd) {
            // a hidden key's weight is zero, and zero times such a value is NaN: each pair takes the keys that it sees, one by one
            for (int j = 0; j < AT_N; ++j) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int key = base + j;
                    if (!(key <= pos[i] && (key >= from[i] || key < kept[i]))) continue;
#pragma unroll
                    for (int c = 0; c < NC; ++c)
                        o[i][c] = fmaf(sm.p[ty * 4 + i][j], sm.v[j][NC == 2 ? tx * 2 + c : (c / 4) * 64 + tx * 4 + c % 4], o[i][c]);
                }
            }
            continue;
        }
#pragma unroll 2
        for (int j = 0; j < AT_N; j += 4) {
            float4 w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(&sm.p[ty * 4 + i][j]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float v[NC];
                if constexpr (NC == 2) {
                    const float2 x = *reinterpret_cast<const float2*>(&sm.v[j + e][tx * 2]);
                    v[0] = x.x; v[1] = x.y;
                } else {
#pragma unroll
                    for (int c = 0; c < NC; c += 4) {
                        const float4 x = *reinterpret_cast<const float4*>(&sm.v[j + e][c * 16 + tx * 4]);
                        v[c] = x.x; v[c + 1] = x.y; v[c + 2] = x.z; v[c + 3] = x.w;
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float p = e == 0 ? w[i].x : e == 1 ? w[i].y : e == 2 ? w[i].z : w[i].w;
#pragma unroll
                    for (int c = 0; c < NC; ++c) o[i][c] = fmaf(p, v[c], o[i][c]);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int p = ty * 4 + i;
        if (p >= n_pairs) continue;
        const int h = kvh * group + p % group;
        if (EXT && opt.sink) {                               // the sink: a term of the denominator alone
            const float sk = opt.sink[h], m_new = fmaxf(m[i], sk), corr = expf(m[i] - m_new);
            l[i] = l[i] * corr + expf(sk - m_new);
#pragma unroll
            for (int c = 0; c < NC; ++c) o[i][c] *= corr;
        }
        const float inv = 1.f / l[i];
        T* orow = out + ((size_t)(r0 + p / group) * Hq + h) * D;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int d = NC == 2 ? tx * 2 + c : (c / 4) * 64 + tx * 4 + c % 4;
            if (d < D) orow[d] = from_float<T>(o[i][c] * inv);
        }
    }
}

ZAI_API int zai_paged_attention_tiles_supports(int D, int Hq, int Hkv) { return D >= 1 && D <= 128 && Hkv >= 1 && Hq % Hkv == 0 && Hq / Hkv <= AT_M && Hkv <= 65535; }
// rows of a tile: n_tiles of the launcher is the sum over the spans of their rows divided by this, rounded up (or more)
ZAI_API int zai_paged_attention_tile_rows(int Hq, int Hkv) { return AT_M / (Hq / Hkv); }

template <typename T, int DM, bool EXT, bool AHEAD>
static int launch_tiles_of(void* out, const void* q, const void* pages, const int* block_table, int table_width, const int* positions,
                        const int* cu_q, int n_seqs, int n_tiles, int page_size, int Hq, int Hkv, int D, float scale, int window,
                        int num_pages, int* status, const ZaiScoreOptions& opt, cudaStream_t stream) {
    static unsigned long long done = 0;
    if (zai_first_on_device(&done)) {
        const cudaError_t e = cudaFuncSetAttribute(paged_attention_tile_kernel<T, DM, EXT, AHEAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(AtTile<DM>));
        if (e != cudaSuccess) return (int)e;
    }
    return launch_pdl(paged_attention_tile_kernel<T, DM, EXT, AHEAD>, dim3(n_tiles, Hkv), dim3(128), sizeof(AtTile<DM>), stream, (T*)out,
                      (const T*)q, (const T*)pages, block_table, table_width, positions, cu_q, n_seqs, page_size, Hq, Hkv, D, scale,
                      window, num_pages, status, opt);
}
// Whether a tile of keys is brought while the one before is used.  A tile's trip to memory is not hidden by other blocks in grids of up
// to about 7/4 blocks an SM; fuller ones do without the 40 registers a thread.  For 32-bit heads of 32 and 64 values whose rows are all
// 16-byte loads, and requests of more than two tiles of keys (known by the width of the table).  us without and with, 8 heads of 64: 20
// rows alone 8.8, 9.5, behind 60 positions 13.5, 13.7, behind 200 23.2, 21.9; 400 behind 400 (104 blocks) 66.9, 59.4; 800 rows (200)
// 83.3, 72.5; 1000 (256) 110, 107; 1184 behind 1000 (296) 239, 245; 3000 (752) 455, 477.  Of 32: 20 alone 7.0, 7.5, 400 behind 400
// 42.3, 39.0, 880 rows (224 blocks) 60, 57, 2048 rows of 4 heads (256) 129, 132.  Of 40 (bounds in every load) 590 rows 56.7, 59.0; heads
// of 128 would wait in 128 registers more.  bfloat16 of 40, whose values would wait as 32-bit numbers: 400 behind 400 72, 107.
template <typename T, int DM, bool EXT>
static int launch_tiles(void* out, const void* q, const void* pages, const int* block_table, int table_width, const int* positions,
                        const int* cu_q, int n_seqs, int n_tiles, int page_size, int Hq, int Hkv, int D, float scale, int window,
                        int num_pages, int* status, const ZaiScoreOptions& opt, cudaStream_t stream) {
    if constexpr (std::is_same<T, float>::value && DM <= 64) {
        static int sms = 0;
        if (!sms) {
            int dev = 0;
            if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) sms = 148;
        }
        if (D == DM && ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(pages)) & 15) == 0
            && (long long)table_width * page_size > 2 * AT_N && (long long)n_tiles * Hkv * 8 <= (DM == 64 ? 14LL : 13LL) * sms)
            return launch_tiles_of<T, DM, EXT, true>(out, q, pages, block_table, table_width, positions, cu_q, n_seqs, n_tiles, page_size, Hq, Hkv, D,
                                                     scale, window, num_pages, status, opt, stream);
    }
    return launch_tiles_of<T, DM, EXT, false>(out, q, pages, block_table, table_width, positions, cu_q, n_seqs, n_tiles, page_size, Hq, Hkv, D,
                                              scale, window, num_pages, status, opt, stream);
}

// A step's spans in tiles of rows (positions of a span's rows follow one another); the score options as below, all off by zeros
// and null pointers.
ZAI_API int zai_paged_attention_tiles(void* out, const void* q, const void* pages, int dtype, const int* block_table, int table_width,
                                      const int* positions, const int* cu_q, int n_seqs, int n_tiles, int page_size, int Hq, int Hkv,
                                      int D, float scale, int window, int num_pages, int* status, float softcap, const float* bias,
                                      int bias_rows, const float* sink, int keep_first, cudaStream_t stream) {
    if (softcap < 0.f || (bias && bias_rows < 1) || keep_first < 0 || (keep_first && window <= 0)) return ZAI_BAD_SIZE;
    if (n_tiles <= 0 || n_seqs <= 0) return ZAI_OK;
    if (!zai_paged_attention_tiles_supports(D, Hq, Hkv)) return ZAI_BAD_SIZE;
    const ZaiScoreOptions opt = {softcap, bias, bias_rows, sink, keep_first, scale};
    const bool ext = softcap > 0.f || bias || sink || keep_first;
#define ZAI_TILES(DM, EXT) ZAI_DISPATCH(dtype, return launch_tiles<T, DM, EXT>(out, q, pages, block_table, table_width, positions, cu_q, n_seqs, \
        n_tiles, page_size, Hq, Hkv, D, scale, window, num_pages, status, opt, stream))
    if (ext) {
        if (D <= 32) ZAI_TILES(32, true);
        if (D <= 64) ZAI_TILES(64, true);
        ZAI_TILES(128, true);
    }
    if (D <= 32) ZAI_TILES(32, false);
    if (D <= 64) ZAI_TILES(64, false);
    ZAI_TILES(128, false);
#undef ZAI_TILES
}

ZAI_API int zai_paged_attention_general(void* out, const void* q, const void* pages, int dtype, const int* block_table,
                                        int table_width, const int* positions, const int* seq_idx, int page_size,
                                        int N, int Hq, int Hkv, int D, float scale, int window, int num_pages, int* status,
                                        cudaStream_t stream) {
    const ZaiScoreOptions opt = {0.f, nullptr, 0, nullptr, 0, 1.f};
    if (N <= 0) return ZAI_OK;
    if (D < 1 || D > 512 || Hkv < 1 || Hq % Hkv != 0 || Hq > 65535) return ZAI_BAD_SIZE;
    const dim3 grid(N, Hq);
    const size_t smem = (size_t)D * sizeof(float);
    if (D <= 64) {
        ZAI_DISPATCH(dtype, return launch_pdl(paged_attention_warp_kernel<T, 2, false>, grid, dim3(32), smem, stream,
            (T*)out, (const T*)q, (const T*)pages, block_table, table_width, positions, seq_idx, page_size, Hq, Hkv,
            D, scale, window, num_pages, status, opt));
    } else if (D <= 256) {
        ZAI_DISPATCH(dtype, return launch_pdl(paged_attention_warp_kernel<T, 8, false>, grid, dim3(32), smem, stream,
            (T*)out, (const T*)q, (const T*)pages, block_table, table_width, positions, seq_idx, page_size, Hq, Hkv,
            D, scale, window, num_pages, status, opt));
    } else {
        ZAI_DISPATCH(dtype, return launch_pdl(paged_attention_warp_kernel<T, 16, false>, grid, dim3(32), smem, stream,
            (T*)out, (const T*)q, (const T*)pages, block_table, table_width, positions, seq_idx, page_size, Hq, Hkv,
            D, scale, window, num_pages, status, opt));
    }
    return launch_status();
}

// The same with the score options above.
ZAI_API int zai_paged_attention_scored(void* out, const void* q, const void* pages, int dtype, const int* block_table,
                                        int table_width, const int* positions, const int* seq_idx, int page_size,
                                        int N, int Hq, int Hkv, int D, float scale, int window, int num_pages, int* status,
                                        float softcap, const float* bias, int bias_rows, const float* sink, int keep_first,
                                        cudaStream_t stream) {
    if (softcap < 0.f || (bias && bias_rows < 1) || keep_first < 0 || (keep_first && window <= 0)) return ZAI_BAD_SIZE;
    const ZaiScoreOptions opt = {softcap, bias, bias_rows, sink, keep_first, scale};
    if (N <= 0) return ZAI_OK;
    if (D < 1 || D > 512 || Hkv < 1 || Hq % Hkv != 0 || Hq > 65535) return ZAI_BAD_SIZE;
    const dim3 grid(N, Hq);
    const size_t smem = (size_t)D * sizeof(float);
    if (D <= 64) {
        ZAI_DISPATCH(dtype, return launch_pdl(paged_attention_warp_kernel<T, 2, true>, grid, dim3(32), smem, stream,
            (T*)out, (const T*)q, (const T*)pages, block_table, table_width, positions, seq_idx, page_size, Hq, Hkv,
            D, scale, window, num_pages, status, opt));
    } else if (D <= 256) {
        ZAI_DISPATCH(dtype, return launch_pdl(paged_attention_warp_kernel<T, 8, true>, grid, dim3(32), smem, stream,
            (T*)out, (const T*)q, (const T*)pages, block_table, table_width, positions, seq_idx, page_size, Hq, Hkv,
            D, scale, window, num_pages, status, opt));
    } else {
        ZAI_DISPATCH(dtype, return launch_pdl(paged_attention_warp_kernel<T, 16, true>, grid, dim3(32), smem, stream,
            (T*)out, (const T*)q, (const T*)pages, block_table, table_width, positions, seq_idx, page_size, Hq, Hkv,
            D, scale, window, num_pages, status, opt));
    }
    return launch_status();
}
