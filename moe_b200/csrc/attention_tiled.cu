// Attention of this step's queries over the cache and the step's own keys, tiled through shared
// memory: 64 queries of one (sequence, head) against key tiles of 64, on the CUDA cores in 32-bit.
//
// Same formulas and the same sources of keys as attention_generic.cu (reference:
// src/model.rs:794-827): keys before the step come from the paged cache, those of the step from
// k_new / v_new (use_local), or all from the cache (a layer that reads another layer's cache).
// Scores, the running maximum and sum and the weighted sum are float32 whatever the storage type.
//
// This is the kernel of the true 32-bit path for prompts, and in both dtypes of every step that
// the tensor-core kernels do not take: a prompt that goes on from the cache (chunks of a long
// prompt, steps that mix continued and fresh sequences) and head sizes other than theirs.  Where
// attention_generic.cu fetches every key from global memory once per QUERY, a block here fetches it
// once per 64 queries: a 24,000-token prompt reads 64 times less.
//
// A block of 256 threads: thread (ty, tx), ty = tid / 16, tx = tid % 16, owns the scores of query
// rows 4 ty .. 4 ty + 3 against key columns 4 tx .. 4 tx + 3, and of the output the same rows and
// the head-dimension columns 4 tx + 64 i.  Q and K sit in shared memory transposed ([d][row]), so
// that both operands of the score product are read as float4; P goes through shared memory to
// every thread of its rows (in the keys' place, which keeps a block of heads of 128 at 103 KB: two
// to an SM).  Key tiles start at multiples of 64 = the page size, so a tile of
// cached keys is one contiguous [64][head_dim] block of one page.
#include "common.cuh"

namespace {

constexpr int BQ = 64, BK = 64, PAD = 4, THREADS = 256;

template <typename T>
__device__ __forceinline__ void load_chunk(const T* p, float* out);
template <>
__device__ __forceinline__ void load_chunk<float>(const float* p, float* out) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    out[0] = v.x, out[1] = v.y, out[2] = v.z, out[3] = v.w;
}
template <>
__device__ __forceinline__ void load_chunk<__nv_bfloat16>(const __nv_bfloat16* p, float* out) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    out[0] = __uint_as_float(v.x << 16), out[1] = __uint_as_float(v.x & 0xffff0000u);
    out[2] = __uint_as_float(v.y << 16), out[3] = __uint_as_float(v.y & 0xffff0000u);
}

template <typename T>
__global__ void __launch_bounds__(THREADS)
attn_tiled_kernel(const T* __restrict__ q, const T* __restrict__ k_new, const T* __restrict__ v_new,
                  const T* __restrict__ k_cache, const T* __restrict__ v_cache, T* __restrict__ out,
                  const int* __restrict__ cu_seqlens, const int* __restrict__ seq_start, const int* __restrict__ slots,
                  const int* __restrict__ tables, int table_stride, int ring, int num_pages, int num_seqs, int nh,
                  int nkv, int hd, int window, float scale, int use_local, int* status, const AttnVariant var) {
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_seq, s_tile;
    float* Qt = sm;                               // [hd][BQ + PAD]
    float* Kt = Qt + (size_t)hd * (BQ + PAD);     // [hd][BK + PAD]
    float* V = Kt + (size_t)hd * (BK + PAD);      // [BK][hd + PAD]
    float* P = Kt;                                // [BQ][BK + PAD]: in the keys' place, once the scores are formed
                                                  // (hd >= 64; smaller heads get room of their own behind V)
    if (hd < BQ) P = V + (size_t)BK * (hd + PAD);
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int h = blockIdx.y, kvh = h / (nh / nkv);

    // which (sequence, tile of 64 of its new tokens): tiles are numbered sequence by sequence
    if (tid == 0) {
        int tile = blockIdx.x, seq = -1;
        for (int s = 0; s < num_seqs; s++) {
            const int tiles = (cu_seqlens[s + 1] - cu_seqlens[s] + BQ - 1) / BQ;
            if (tile < tiles) {
                seq = s;
                break;
            }
            tile -= tiles;
        }
        s_seq = seq, s_tile = tile;
    }
    __syncthreads();
    const int seq = s_seq;
    if (seq < 0) return;
    const int tok0 = cu_seqlens[seq], cnt = cu_seqlens[seq + 1] - tok0, start = seq_start[seq];
    const int r0 = s_tile * BQ;                                    // first new token of the tile (within the step)
    const int rows = min(BQ, cnt - r0);
    const int p_first = start + r0, p_last = p_first + rows - 1;   // positions of the tile's queries
    const int local_from = use_local ? start : p_last + 1;         // positions from here on come from k_new / v_new
    const int lo_min = attn_lo(p_first, window, var.chunk);   // (the first query's: lo never decreases with p)
    const int* table = tables + (size_t)slots[seq] * table_stride;
    const int QS = BQ + PAD, KS = BK + PAD, VS = hd + PAD, PS = BK + PAD;

    // ---- the queries, transposed --------------------------------------------------------------
    for (int idx = tid; idx < BQ * (hd / 4); idx += THREADS) {
        const int r = idx / (hd / 4), d = (idx % (hd / 4)) * 4;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (r < rows) load_chunk<T>(q + ((size_t)(tok0 + r0 + r) * nh + h) * hd + d, v);
#pragma unroll
        for (int e = 0; e < 4; e++) Qt[(size_t)(d + e) * QS + r] = v[e];
    }

    float m[4], l[4], o[4][16];          // running maximum and sum of this thread's rows; its part of the output
#pragma unroll
    for (int r = 0; r < 4; r++) {
        m[r] = -INFINITY, l[r] = 0.f;
#pragma unroll
        for (int i = 0; i < 16; i++) o[r][i] = 0.f;
    }
    const int ncol = hd / 64 + (hd % 64 ? 1 : 0);      // float4 column groups of the output per thread: d = 4 tx + 64 i

    // (kept first positions: their tiles come first, then those of the window)
    const int tile_lo = lo_min / BK, kept_tiles = min((var.keep + BK - 1) / BK, tile_lo), pinned = attn_pinned(var);
    for (int tile = 0; attn_seen(tile, kept_tiles, tile_lo) * BK <= p_last; tile++) {
        const int j0 = attn_seen(tile, kept_tiles, tile_lo) * BK;
        __syncthreads();                 // the previous tile's K, V and P are no longer read
        // ---- a tile of keys (transposed) and values -------------------------------------------
        for (int idx = tid; idx < BK * (hd / 4); idx += THREADS) {
            const int c = idx / (hd / 4), d = (idx % (hd / 4)) * 4;
            const int j = j0 + c;
            float kv[4] = {0.f, 0.f, 0.f, 0.f}, vv[4] = {0.f, 0.f, 0.f, 0.f};
            if (j <= p_last && (j >= lo_min || j < var.keep)) {
                if (j >= local_from) {
                    const size_t at = ((size_t)(tok0 + (j - start)) * nkv + kvh) * hd + d;
                    load_chunk<T>(k_new + at, kv);
                    load_chunk<T>(v_new + at, vv);
                } else {
                    const CachePos cp = cache_pos(j, ring, table, BK, num_pages, status, pinned);
                    const size_t at = cache_index(cp, kvh, nkv, BK, hd) + d;
                    load_chunk<T>(k_cache + at, kv);
                    load_chunk<T>(v_cache + at, vv);
                }
            }
#pragma unroll
            for (int e = 0; e < 4; e++) Kt[(size_t)(d + e) * KS + c] = kv[e];
            *reinterpret_cast<float4*>(V + (size_t)c * VS + d) = make_float4(vv[0], vv[1], vv[2], vv[3]);
        }
        __syncthreads();
        // ---- scores of 4 rows x 4 columns -----------------------------------------------------
        float s[4][4];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) s[r][c] = 0.f;
#pragma unroll 4
        for (int d = 0; d < hd; d++) {
            const float4 a = *reinterpret_cast<const float4*>(Qt + (size_t)d * QS + ty * 4);
            const float4 b = *reinterpret_cast<const float4*>(Kt + (size_t)d * KS + tx * 4);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) s[r][c] = fmaf(av[r], bv[c], s[r][c]);
        }
        // ---- mask, running maximum and sum, P --------------------------------------------------
        __syncthreads();                 // every thread has read the keys: P may take their place
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int row = ty * 4 + r, p = p_first + row;
            const int lo = attn_lo(p, window, var.chunk);
            float mx = -INFINITY;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int j = j0 + tx * 4 + c;
                const bool seen = row < rows && j <= p && (j >= lo || j < var.keep);
                s[r][c] = seen ? attn_logit(var, h, s[r][c], scale) : -INFINITY;
                mx = fmaxf(mx, s[r][c]);
            }
#pragma unroll
            for (int off = 8; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
            const float m_new = fmaxf(m[r], mx);
            float alpha = 1.f, sum = 0.f, pr[4] = {0.f, 0.f, 0.f, 0.f};
            if (m_new != -INFINITY) {                    // (the same for the 16 threads of the row)
                alpha = m[r] == -INFINITY ? 0.f : expf(m[r] - m_new);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    pr[c] = s[r][c] == -INFINITY ? 0.f : expf(s[r][c] - m_new);
                    sum += pr[c];
                }
            }
#pragma unroll
            for (int off = 8; off >= 1; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            l[r] = l[r] * alpha + sum;
            m[r] = m_new;
#pragma unroll
            for (int i = 0; i < 16; i++) o[r][i] *= alpha;
            *reinterpret_cast<float4*>(P + (size_t)row * PS + tx * 4) = make_float4(pr[0], pr[1], pr[2], pr[3]);
        }
        __syncthreads();
        // ---- output rows += P V -----------------------------------------------------------------
        for (int c0 = 0; c0 < BK; c0 += 4) {
            float pv[4][4];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float4 t4 = *reinterpret_cast<const float4*>(P + (size_t)(ty * 4 + r) * PS + c0);
                pv[r][0] = t4.x, pv[r][1] = t4.y, pv[r][2] = t4.z, pv[r][3] = t4.w;
            }
#pragma unroll
            for (int c = 0; c < 4; c++) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (i >= ncol) break;
                    const int d = tx * 4 + 64 * i;
                    if (d >= hd) break;
                    const float4 v4 = *reinterpret_cast<const float4*>(V + (size_t)(c0 + c) * VS + d);
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        o[r][4 * i] = fmaf(pv[r][c], v4.x, o[r][4 * i]);
                        o[r][4 * i + 1] = fmaf(pv[r][c], v4.y, o[r][4 * i + 1]);
                        o[r][4 * i + 2] = fmaf(pv[r][c], v4.z, o[r][4 * i + 2]);
                        o[r][4 * i + 3] = fmaf(pv[r][c], v4.w, o[r][4 * i + 3]);
                    }
                }
            }
        }
    }
    // ---- normalise and store --------------------------------------------------------------------
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int row = ty * 4 + r;
        if (row >= rows) continue;
        const float inv = l[r] > 0.f ? 1.0f / attn_denominator(m[r], l[r], var.sink, attn_sink_value(var, h)) : 0.f;
        T* dst = out + ((size_t)(tok0 + r0 + row) * nh + h) * hd;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int d = tx * 4 + 64 * i;
            if (i >= ncol || d >= hd) break;
#pragma unroll
            for (int e = 0; e < 4; e++) st_f(dst + d + e, o[r][4 * i + e] * inv);
        }
    }
}

// ---- the 32-bit path's form for heads of 64 and 128 and steps of many tokens a sequence -------------------------------
// 128 queries of one (sequence, head) against key tiles of 128 (two pages): an 8 x 8 part of the scores and 8 x HD / 16
// of the output a thread, so that sixteen 16-byte reads of shared memory feed 256 multiply-adds (the form above: eight
// feed 64, and the reads, not the multiply-adds, are what bounds it: 13 of 74 TFLOP/s).  Nothing is transposed: queries,
// keys and values lie in shared memory as they lie in global memory (cp.async), a thread's rows (ty + 16 i) and columns
// (tx + 16 j) are interleaved so that neighbouring threads read neighbouring rows (a pitch of HD + 4: different banks),
// and both products walk four of their inner index at a time, in order.  The values arrive under the score product.
// The heads are the fast index of the grid and a sequence's last queries, which see most keys, come first: one head after
// another left SMs with long blocks while others had none left (a third of the multiply-add rate on average, 57 % on the
// fullest SM).
constexpr int FQ = 128, FK = 128;
template <int HD>
__host__ __device__ constexpr int f32_floats() {
    return FQ * (HD + 4) + FK * (HD + 4) + (HD < FK ? FQ * (FK + 4) : 0) + FK * (HD + 4);
}
__device__ __forceinline__ void cp16z(float* dst, const float* src, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 16 : 0)
                 : "memory");
}

// PLAIN: neither a cap on the scores nor sigmoid weights; compiled apart because sixty-four inlined copies of those leave no
// room in the instruction cache for the loops (two thirds of the time was spent waiting for instructions).
template <int HD, bool PLAIN>
__global__ void __launch_bounds__(THREADS, 1)
attn_f32_kernel(const float* __restrict__ q, const float* __restrict__ k_new, const float* __restrict__ v_new,
                const float* __restrict__ k_cache, const float* __restrict__ v_cache, float* __restrict__ out,
                const int* __restrict__ cu_seqlens, const int* __restrict__ seq_start, const int* __restrict__ slots,
                const int* __restrict__ tables, int table_stride, int ring, int num_pages, int num_seqs, int nh, int nkv,
                int window, float scale, int use_local, int* status, const AttnVariant var) {
    constexpr int HP = HD + 4, PP = FK + 4, OC = HD / 16;       // OC: output columns a thread (4 tx + 64 j + 0..3)
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_seq, s_tile;
    float* Q = sm;                                  // [FQ][HP]
    float* K = Q + FQ * HP;                         // [FK][HP]
    float* P = HD < FK ? K + FK * HP : K;           // [FQ][PP]: in the keys' place where it fits there
    float* V = HD < FK ? P + FQ * PP : K + FK * HP; // [FK][HP]
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int h = blockIdx.x, kvh = h / (nh / nkv);
    if (tid == 0) {
        int tile = blockIdx.y, seq = -1;
        for (int s = 0; s < num_seqs; s++) {
            const int tiles = (cu_seqlens[s + 1] - cu_seqlens[s] + FQ - 1) / FQ;
            if (tile < tiles) {
                seq = s, tile = tiles - 1 - tile;
                break;
            }
            tile -= tiles;
        }
        s_seq = seq, s_tile = tile;
    }
    __syncthreads();
    const int seq = s_seq;
    if (seq < 0) return;
    const int tok0 = cu_seqlens[seq], cnt = cu_seqlens[seq + 1] - tok0, start = seq_start[seq];
    const int r0 = s_tile * FQ, rows = min(FQ, cnt - r0);
    const int p_first = start + r0, p_last = p_first + rows - 1;
    const int local_from = use_local ? start : p_last + 1;
    const int lo_min = attn_lo(p_first, window, var.chunk), pinned = attn_pinned(var);
    const int* table = tables + (size_t)slots[seq] * table_stride;
    for (int idx = tid; idx < FQ * (HD / 4); idx += THREADS) {
        const int r = idx / (HD / 4), d = (idx % (HD / 4)) * 4;
        cp16z(Q + r * HP + d, q + ((size_t)(tok0 + r0 + (r < rows ? r : 0)) * nh + h) * HD + d, r < rows);
    }
    float m[8], l[8], o[8][OC];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        m[i] = -INFINITY, l[i] = 0.f;
#pragma unroll
        for (int j = 0; j < OC; j++) o[i][j] = 0.f;
    }
    // The first 64 queries take no value behind the last of them and the others none in front of their window, not even with a
    // weight of 0: an infinite or NaN value reaches as many queries that do not see it as in the form above, and no more.
    const int low_to = p_first + FQ / 2 - 1, high_from = attn_lo(p_first + FQ / 2, window, var.chunk);
    const int tile_lo = lo_min / FK, kept_tiles = min((var.keep + FK - 1) / FK, tile_lo);
    for (int tile = 0; attn_seen(tile, kept_tiles, tile_lo) * FK <= p_last; tile++) {
        const int j0 = attn_seen(tile, kept_tiles, tile_lo) * FK;
        // a thread copies one 16-byte column of every (THREADS * 4 / HD)-th key, then of the values
        constexpr int STEP = THREADS / (HD / 4);
        const int d = (tid % (HD / 4)) * 4, c_first = tid / (HD / 4);
        __syncthreads();                            // K, V and P of the tile before are no longer read
        const float* vsrc[FK / STEP];
#pragma unroll
        for (int i = 0; i < FK / STEP; i++) {
            const int c = c_first + i * STEP, j = j0 + c;
            const float* ks = nullptr;
            vsrc[i] = nullptr;
            if (j <= p_last && (j >= lo_min || j < var.keep)) {
                if (j >= local_from) {
                    const size_t at = ((size_t)(tok0 + (j - start)) * nkv + kvh) * HD + d;
                    ks = k_new + at, vsrc[i] = v_new + at;
                } else {
                    const CachePos cp = cache_pos(j, ring, table, BK, num_pages, status, pinned);
                    const size_t at = cache_index(cp, kvh, nkv, BK, HD) + d;
                    ks = k_cache + at, vsrc[i] = v_cache + at;
                }
            }
            cp16z(K + c * HP + d, ks ? ks : q, ks != nullptr);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
        for (int i = 0; i < FK / STEP; i++) cp16z(V + (c_first + i * STEP) * HP + d, vsrc[i] ? vsrc[i] : q, vsrc[i] != nullptr);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        float s[8][8];
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) s[i][j] = 0.f;
#pragma unroll 2
        for (int e = 0; e < HD; e += 4) {
            float4 a[8];
#pragma unroll
            for (int i = 0; i < 8; i++) a[i] = *reinterpret_cast<const float4*>(Q + (ty + 16 * i) * HP + e);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float4 b = *reinterpret_cast<const float4*>(K + (tx + 16 * j) * HP + e);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    s[i][j] = fmaf(a[i].x, b.x, s[i][j]), s[i][j] = fmaf(a[i].y, b.y, s[i][j]);
                    s[i][j] = fmaf(a[i].z, b.z, s[i][j]), s[i][j] = fmaf(a[i].w, b.w, s[i][j]);
                }
            }
        }
        if (P == K) __syncthreads();                // every thread has read the keys: P may take their place
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int row = ty + 16 * i, p = p_first + row, lo = attn_lo(p, window, var.chunk);
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int key = j0 + tx + 16 * j;
                const bool seen = row < rows && key <= p && (key >= lo || key < var.keep);
                s[i][j] = seen ? (PLAIN ? s[i][j] * scale : attn_logit(var, h, s[i][j], scale)) : -INFINITY;
                mx = fmaxf(mx, s[i][j]);
            }
#pragma unroll
            for (int off = 8; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
            const float m_new = fmaxf(m[i], mx);
            float alpha = 1.f, sum = 0.f;
            if (m_new != -INFINITY) {               // (the same for the 16 threads of the row)
                alpha = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    s[i][j] = s[i][j] == -INFINITY ? 0.f : expf(s[i][j] - m_new);
                    sum += s[i][j];
                }
            } else {
#pragma unroll
                for (int j = 0; j < 8; j++) s[i][j] = 0.f;
            }
#pragma unroll
            for (int off = 8; off >= 1; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            l[i] = l[i] * alpha + sum;
            m[i] = m_new;
#pragma unroll
            for (int j = 0; j < OC; j++) o[i][j] *= alpha;
#pragma unroll
            for (int j = 0; j < 8; j++) P[row * PP + tx + 16 * j] = s[i][j];
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        // keys [c_lo, c_hi) are for both halves of the queries; a key outside for the half that may take it
        const int c_lo = high_from > j0 && j0 + FK > var.keep ? min(FK, (high_from - j0 + 3) & ~3) : 0;
        const int c_hi = max(c_lo, min(FK, (low_to - j0 + 1) & ~3));
        auto for_one_half = [&](int from, int to) {
#pragma unroll 1
            for (int c = from; c < to; c++) {
                const int key = j0 + c;
                const bool low = key <= low_to, high = key >= high_from || key < var.keep;
                float4 v4[OC / 4];
#pragma unroll
                for (int j = 0; j < OC; j += 4) v4[j / 4] = *reinterpret_cast<const float4*>(V + c * HP + 4 * tx + 16 * j);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    if (!(i < 4 ? low : high)) continue;
                    const float pv = P[(ty + 16 * i) * PP + c];
#pragma unroll
                    for (int j = 0; j < OC; j += 4) {
                        o[i][j] = fmaf(pv, v4[j / 4].x, o[i][j]), o[i][j + 1] = fmaf(pv, v4[j / 4].y, o[i][j + 1]);
                        o[i][j + 2] = fmaf(pv, v4[j / 4].z, o[i][j + 2]), o[i][j + 3] = fmaf(pv, v4[j / 4].w, o[i][j + 3]);
                    }
                }
            }
        };
        for_one_half(0, c_lo);
#pragma unroll 1
        for (int c = c_lo; c < c_hi; c += 4) {
            float4 a[8];
#pragma unroll
            for (int i = 0; i < 8; i++) a[i] = *reinterpret_cast<const float4*>(P + (ty + 16 * i) * PP + c);
#pragma unroll
            for (int e = 0; e < 4; e++)
#pragma unroll
                for (int j = 0; j < OC; j += 4) {
                    const float4 v4 = *reinterpret_cast<const float4*>(V + (c + e) * HP + 4 * tx + 16 * j);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const float pv = e == 0 ? a[i].x : e == 1 ? a[i].y : e == 2 ? a[i].z : a[i].w;
                        o[i][j] = fmaf(pv, v4.x, o[i][j]), o[i][j + 1] = fmaf(pv, v4.y, o[i][j + 1]);
                        o[i][j + 2] = fmaf(pv, v4.z, o[i][j + 2]), o[i][j + 3] = fmaf(pv, v4.w, o[i][j + 3]);
                    }
                }
        }
        for_one_half(c_hi, min(FK, p_last - j0 + 1));
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int row = ty + 16 * i;
        if (row >= rows) continue;
        const float inv = l[i] > 0.f ? 1.0f / attn_denominator(m[i], l[i], var.sink, attn_sink_value(var, h)) : 0.f;
        float* dst = out + ((size_t)(tok0 + r0 + row) * nh + h) * HD;
#pragma unroll
        for (int j = 0; j < OC; j += 4)
            *reinterpret_cast<float4*>(dst + 4 * tx + 16 * j) = make_float4(o[i][j] * inv, o[i][j + 1] * inv, o[i][j + 2] * inv, o[i][j + 3] * inv);
    }
}

size_t tiled_smem(int hd) {
    // Q, K (P takes K's place when the head is at least as long as a tile is wide), V
    return ((size_t)hd * (BQ + PAD) + (size_t)hd * (BK + PAD) + (size_t)BK * (hd + PAD) +
            (hd < BQ ? (size_t)BQ * (BK + PAD) : 0)) * sizeof(float);
}

}  // namespace

// Same arguments as moe_attention_generic, without the per-token arrays (a block finds its rows from
// cu_seqlens).  The page size must be 64.  Rows of no sequence (a padded step) are not written.
// Returns -1 (nothing launched) for sizes this kernel does not take: the caller uses the plain kernel.
MOE_API int moe_attention_tiled(const void* q, const void* k_new, const void* v_new, const void* k_cache,
                                const void* v_cache, void* out, int dt, const int* cu_seqlens, const int* seq_start,
                                const int* slots, const int* tables, int table_stride, int ring, int page_size,
                                int num_pages, int num_seqs, int num_tokens, int nh, int nkv, int hd, int window,
                                float scale, int use_local, int* status, int chunk, float softcap, int sink,
                                const float* sink_vals, int keep, cudaStream_t stream) {
    if (num_tokens <= 0 || num_seqs <= 0) return 0;
    const AttnVariant av{chunk, softcap, sink, sink_vals, keep};
    if (hd > 256) return -1;
    if (hd % 16 != 0 || hd <= 0 || nkv <= 0 || nh % nkv != 0 || nh > 65535) return (int)cudaErrorInvalidValue;
    if (page_size != BK || (ring % BK) != 0) return -1;
    const size_t align = dt == DT_F32 ? 16 : 8;          // rows are read four elements at a time
    if (((uintptr_t)q | (uintptr_t)k_new | (uintptr_t)v_new | (uintptr_t)k_cache | (uintptr_t)v_cache) % align) return -1;
    // many new tokens a sequence: 128 of them to a block.  (With fewer than that most of its rows would be padding, and
    // the form of 64 has twice the blocks.)
    if (dt == DT_F32 && (hd == 64 || hd == 128) && num_tokens >= FQ * num_seqs &&
        (num_tokens + FQ - 1) / FQ + num_seqs <= 65535 && !((uintptr_t)out % 16)) {
        const dim3 grid(nh, (unsigned)((num_tokens + FQ - 1) / FQ + num_seqs));
#define GO(HD, PLAIN)                                                                                                 \
    do {                                                                                                              \
        const int bytes = f32_floats<HD>() * 4;                                                                       \
        cudaError_t e = cudaFuncSetAttribute(attn_f32_kernel<HD, PLAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); \
        if (e != cudaSuccess) return (int)e;                                                                          \
        attn_f32_kernel<HD, PLAIN><<<grid, THREADS, bytes, stream>>>(                                                        \
            (const float*)q, (const float*)k_new, (const float*)v_new, (const float*)k_cache, (const float*)v_cache,  \
            (float*)out, cu_seqlens, seq_start, slots, tables, table_stride, ring, num_pages, num_seqs, nh, nkv, window, \
            scale, use_local, status, av);                                                                            \
        return launch_status();                                                                                       \
    } while (0)
        const bool simple = !(softcap > 0.f) && sink != ATTN_SIGMOID;
        if (hd == 64) {
            if (simple) GO(64, true);
            GO(64, false);
        }
        if (simple) GO(128, true);
        GO(128, false);
#undef GO
    }
    const size_t smem = tiled_smem(hd);
    const long long tiles = (long long)(num_tokens + BQ - 1) / BQ + num_seqs;
    if (tiles > 0x7fffffffLL) return -1;
    dim3 grid((unsigned)tiles, nh);
#define GO(TT)                                                                                                        \
    do {                                                                                                              \
        static size_t configured = 0;                                                                                 \
        if (smem > 48 * 1024 && smem > configured) {                                                                  \
            cudaError_t e = cudaFuncSetAttribute(attn_tiled_kernel<TT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
            if (e != cudaSuccess) return (int)e;                                                                      \
            configured = smem;                                                                                        \
        }                                                                                                             \
        attn_tiled_kernel<TT><<<grid, THREADS, smem, stream>>>(                                                       \
            (const TT*)q, (const TT*)k_new, (const TT*)v_new, (const TT*)k_cache, (const TT*)v_cache, (TT*)out,       \
            cu_seqlens, seq_start, slots, tables, table_stride, ring, num_pages, num_seqs, nh, nkv, hd, window, scale, \
            use_local, status, av);                                                                                   \
    } while (0)
    if (dt == DT_F32)
        GO(float);
    else
        GO(__nv_bfloat16);
#undef GO
    return launch_status();
}
