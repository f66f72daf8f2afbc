// The plain matrix product of the library: C[m, n] = sum_k A[row(m), k] * W[g][n, k] (+ bias[n]).
//
// Every projection of the model is stored [out_features, in_features] row-major
// and applied as y = W x (reference: src/quant.rs:476-506).  These kernels are the
// true 32-bit path (FFMA on CUDA cores, no reduced-precision matrix
// mode) and the fallback of the bfloat16 path for shapes and dtypes the
// tensor-core kernels refuse.  They take any M, N, K.
//
// Every kernel here forms an output in ONE order: the products of 256 neighbouring k (a chunk) are added by
// one accumulator, k ascending, and the chunks' sums are added in order to a total that starts at zero.  So a
// token's projection is the same to the bit whichever kernel forms it, alone (a decode step) or among
// thousands (a prompt); and the chunks of a few rows' products can be formed side by side by several warps.
//
//   * rows of A may be gathered through `a_rows` (expert dispatch);
//   * rows may be partitioned into groups by `group_offsets[G+1]`, group g using
//     the weight slab W + g * w_group_stride (routed experts).
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, THREADS = 256;
constexpr int CHUNK = 256;       // k whose products one accumulator adds up (see above)

template <typename T>
__device__ __forceinline__ void load4(const T* p, bool vec_ok, int valid, float* out);

template <>
__device__ __forceinline__ void load4<float>(const float* p, bool vec_ok, int valid, float* out) {
    if (vec_ok && valid == 4) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        out[0] = v.x, out[1] = v.y, out[2] = v.z, out[3] = v.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) out[i] = i < valid ? p[i] : 0.f;
    }
}
template <>
__device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, bool vec_ok, int valid, float* out) {
    if (vec_ok && valid == 4) {
        const uint2 v = *reinterpret_cast<const uint2*>(p);
        out[0] = __uint_as_float(v.x << 16), out[1] = __uint_as_float(v.x & 0xffff0000u);
        out[2] = __uint_as_float(v.y << 16), out[3] = __uint_as_float(v.y & 0xffff0000u);
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) out[i] = i < valid ? __bfloat162float(p[i]) : 0.f;
    }
}

// Which group and which tile of `rows` rows of it block tile `tile` is: (group, first row, end of the group's rows),
// group -1 for none.  By the block's first warp, 32 groups at a time; the caller synchronises.
__device__ __forceinline__ void find_tile(const int* __restrict__ group_offsets, int num_groups, int tile, int rows, int M,
                                          int* s_group, int* s_row0, int* s_row1) {
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    int g = -1, r0 = 0, r1 = M;
    if (!group_offsets) {
        r0 = tile * rows;
        g = r0 < M ? 0 : -1;
    } else {
        for (int base = 0; base < num_groups; base += 32) {
            const int i = base + lane;
            const int b = i < num_groups ? group_offsets[i] : 0, e = i < num_groups ? group_offsets[i + 1] : 0;
            const int mine = (e - b + rows - 1) / rows;
            int upto = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            const unsigned hit = __ballot_sync(0xffffffffu, upto > tile);
            if (hit) {
                const int l = __ffs(hit) - 1;
                g = base + l;
                r0 = __shfl_sync(0xffffffffu, b + (tile - (upto - mine)) * rows, l), r1 = __shfl_sync(0xffffffffu, e, l);
                break;
            }
            tile -= __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    if (lane == 0) *s_group = g, *s_row0 = r0, *s_row1 = r1;
}

// The plain tile kernel: any dtype, any alignment.
template <typename AT, typename WT, typename OT>
__global__ void __launch_bounds__(THREADS)
gemm_generic_kernel(const AT* __restrict__ A, int lda, const int* __restrict__ a_rows, int a_src_rows,
                    const WT* __restrict__ W, long long w_group_stride, OT* __restrict__ C, int ldc,
                    const float* __restrict__ bias, const int* __restrict__ group_offsets, int num_groups, int M,
                    int N, int K, int a_vec_ok, int w_vec_ok, int* status) {
    __shared__ __align__(16) float As[BK][BM + 4];
    __shared__ __align__(16) float Ws[BK][BN + 4];
    __shared__ int s_group, s_row0, s_row1;

    find_tile(group_offsets, num_groups, blockIdx.y, BM, M, &s_group, &s_row0, &s_row1);
    __syncthreads();
    const int g = s_group;
    if (g < 0) return;
    const int row0 = s_row0, row_end = s_row1;
    const int n0 = blockIdx.x * BN;
    const WT* Wg = W + (size_t)g * (size_t)w_group_stride;

    const int tid = threadIdx.x;
    const int lr = tid >> 2;         // 0..63: row of the tile this thread loads
    const int lk = (tid & 3) * 4;    // 0,4,8,12: first k it loads
    const int ty = tid >> 4, tx = tid & 15;

    // source row of A for the row this thread loads
    const int arow = row0 + lr;
    long long a_src = -1;
    if (arow < row_end) {
        a_src = a_rows ? a_rows[arow] : arow;
        if (a_src < 0 || a_src >= a_src_rows) {
            atomicOr(status, ST_BAD_ROW);
            a_src = -1;
        }
    }
    const int wrow = n0 + lr;

    float acc[4][4], tot[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = tot[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        float av[4], wv[4];
        const int k = k0 + lk;
        int valid = K - k;
        valid = valid < 0 ? 0 : (valid > 4 ? 4 : valid);
        if (a_src >= 0 && valid > 0)
            load4<AT>(A + (size_t)a_src * lda + k, a_vec_ok, valid, av);
        else
            av[0] = av[1] = av[2] = av[3] = 0.f;
        if (wrow < N && valid > 0)
            load4<WT>(Wg + (size_t)wrow * K + k, w_vec_ok, valid, wv);
        else
            wv[0] = wv[1] = wv[2] = wv[3] = 0.f;
        __syncthreads();   // previous tile fully consumed
#pragma unroll
        for (int i = 0; i < 4; i++) {
            As[lk + i][lr] = av[i];
            Ws[lk + i][lr] = wv[i];
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            const float4 a = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
            const float4 b = *reinterpret_cast<const float4*>(&Ws[kk][tx * 4]);
            const float ar[4] = {a.x, a.y, a.z, a.w};
            const float br[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(ar[i], br[j], acc[i][j]);
        }
        if ((k0 + BK) % CHUNK == 0 || k0 + BK >= K) {
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) tot[i][j] += acc[i][j], acc[i][j] = 0.f;
        }
    }

#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = row0 + ty * 4 + i;
        if (r >= row_end) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int c = n0 + tx * 4 + j;
            if (c >= N) continue;
            float v = tot[i][j];
            if (bias) v += bias[c];
            st_f(C + (size_t)r * ldc + c, v);
        }
    }
}

// The same product for FEW rows (a step of one token per sequence), any dtype and alignment.
// A block takes 64 output features and up to RT rows of A; piece by piece of KC k it brings the
// weights [64][KC] (coalesced, 16 bytes a thread) and the rows [RT][KC] into shared memory, and
// thread (feature f, row pair) walks the piece.  Groups and gathered rows as above, in tiles of RT rows.
constexpr int RT = 8, RF = 64, KC = 128, WS = KC + 4, RTHREADS = 256;

template <typename AT, typename WT, typename OT>
__global__ void __launch_bounds__(RTHREADS)
gemm_rows_kernel(const AT* __restrict__ A, int lda, const int* __restrict__ a_rows, int a_src_rows,
                 const WT* __restrict__ W, long long w_group_stride, OT* __restrict__ C, int ldc,
                 const float* __restrict__ bias, const int* __restrict__ group_offsets, int num_groups, int M, int N,
                 int K, int a_vec_ok, int w_vec_ok, int* status) {
    __shared__ __align__(16) float Ws[RF][WS];
    __shared__ __align__(16) float As[RT][KC];
    __shared__ int s_group, s_row0, s_row1;
    __shared__ long long s_src[RT];
    find_tile(group_offsets, num_groups, blockIdx.y, RT, M, &s_group, &s_row0, &s_row1);
    __syncthreads();
    const int g = s_group;
    if (g < 0) return;
    const int row0 = s_row0, rows = min(RT, s_row1 - row0);
    if (threadIdx.x < RT) {
        long long src = -1;
        if ((int)threadIdx.x < rows) {
            src = a_rows ? a_rows[row0 + threadIdx.x] : row0 + threadIdx.x;
            if (src < 0 || src >= a_src_rows) {
                atomicOr(status, ST_BAD_ROW);
                src = -1;
            }
        }
        s_src[threadIdx.x] = src;
    }
    const int tid = threadIdx.x, f = tid % RF, rg = tid / RF;      // this thread's feature and pair of rows
    const int n0 = blockIdx.x * RF;
    const WT* Wg = W + (size_t)g * (size_t)w_group_stride;
    float acc0 = 0.f, acc1 = 0.f, tot0 = 0.f, tot1 = 0.f;

    // A chunk's loads are issued one chunk ahead, into registers, and so are in flight while the
    // chunk before it is multiplied.
    constexpr int WPT = RF * (KC / 4) / RTHREADS;      // 16-byte pieces of the weight chunk per thread
    float wr[WPT][4], ar[4];
    __syncthreads();                                   // s_src is written
    auto fetch = [&](int c0) {
        const int kc = min(KC, K - c0);
#pragma unroll
        for (int i = 0; i < WPT; i++) {
            const int idx = tid + i * RTHREADS, fl = idx / (KC / 4), k = (idx % (KC / 4)) * 4;
            const int valid = min(4, kc - k);
            wr[i][0] = wr[i][1] = wr[i][2] = wr[i][3] = 0.f;
            if (n0 + fl < N && valid > 0) load4<WT>(Wg + (size_t)(n0 + fl) * K + c0 + k, w_vec_ok, valid, wr[i]);
        }
        const int r = tid / (KC / 4), k = (tid % (KC / 4)) * 4;           // RT * KC / 4 == RTHREADS
        const long long src = s_src[r];
        const int valid = min(4, kc - k);
        ar[0] = ar[1] = ar[2] = ar[3] = 0.f;
        if (src >= 0 && valid > 0) load4<AT>(A + (size_t)src * lda + c0 + k, a_vec_ok, valid, ar);
    };
    if (K > 0) fetch(0);
    for (int c0 = 0; c0 < K; c0 += KC) {
        const int kc = min(KC, K - c0);
        __syncthreads();              // the previous chunk is no longer read
#pragma unroll
        for (int i = 0; i < WPT; i++) {
            const int idx = tid + i * RTHREADS, fl = idx / (KC / 4), k = (idx % (KC / 4)) * 4;
            *reinterpret_cast<float4*>(&Ws[fl][k]) = make_float4(wr[i][0], wr[i][1], wr[i][2], wr[i][3]);
        }
        *reinterpret_cast<float4*>(&As[tid / (KC / 4)][(tid % (KC / 4)) * 4]) = make_float4(ar[0], ar[1], ar[2], ar[3]);
        __syncthreads();
        if (c0 + KC < K) fetch(c0 + KC);
#pragma unroll 8
        for (int k = 0; k < KC; k += 4) {
            if (k >= kc) break;       // (a chunk's tail is zero anyway; this only saves the work)
            const float4 w = *reinterpret_cast<const float4*>(&Ws[f][k]);
            const float4 a = *reinterpret_cast<const float4*>(&As[2 * rg][k]);
            const float4 b = *reinterpret_cast<const float4*>(&As[2 * rg + 1][k]);
            acc0 = fmaf(a.x, w.x, acc0), acc0 = fmaf(a.y, w.y, acc0), acc0 = fmaf(a.z, w.z, acc0), acc0 = fmaf(a.w, w.w, acc0);
            acc1 = fmaf(b.x, w.x, acc1), acc1 = fmaf(b.y, w.y, acc1), acc1 = fmaf(b.z, w.z, acc1), acc1 = fmaf(b.w, w.w, acc1);
        }
        if ((c0 + KC) % CHUNK == 0 || c0 + KC >= K) tot0 += acc0, tot1 += acc1, acc0 = acc1 = 0.f;
    }
    const int n = n0 + f;
    if (n < N) {
        const float bv = bias ? bias[n] : 0.f;
        if (2 * rg < rows) st_f(C + (size_t)(row0 + 2 * rg) * ldc + n, bias ? tot0 + bv : tot0);
        if (2 * rg + 1 < rows) st_f(C + (size_t)(row0 + 2 * rg + 1) * ldc + n, bias ? tot1 + bv : tot1);
    }
}
static_assert(RT * (KC / 4) == RTHREADS && RT == 2 * (RTHREADS / RF) && CHUNK % KC == 0 && CHUNK % BK == 0,
              "the thread layout and the pieces of gemm_rows_kernel");

// ---- 32-bit operands in whole 16-byte units: the forms that the float32 path runs -------------------------------
__device__ __forceinline__ void cp16(void* smem, const void* global, int bytes) {      // bytes < 16: the rest is zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(global),
                 "r"(bytes));
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// two independent 32-bit multiply-adds in one instruction, each rounded as fmaf rounds
__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

// Many rows: TM x 128 outputs a block, 16 k a stage, two stages.  Bound by the multiply-add units (148 SMs x 128 lanes: 70
// TFLOP/s measured with nothing else in the loop), so what counts is how little else an SM does beside them.
// fma.rn.f32x2 forms two outputs (neighbouring features) an instruction, which leaves issue slots for the loads; a thread's
// RM x RN outputs decide how many bytes of shared memory a multiply-add needs.  Measured at 4,736 x 6,144 x 2,048:
// 4 x 4 a thread (the plain kernel above) 34 TFLOP/s; 8 x 8 with single multiply-adds 47; 8 x 8 as here 50, 8 x 16 with two blocks of
// 128 threads an SM 54, one of 256 threads 50, 16 x 8 52.  The chunks' totals wait in shared memory: in registers they cost
// the second block.
constexpr int TN = 128, TK = 16;
template <int RM, int RN, int WM, int WN, int BLOCKS>
struct TileForm {
    static constexpr int M = RM, N = RN, WARPS_M = WM, WARPS_N = WN, MIN_BLOCKS = BLOCKS;
    static constexpr int TM = WM * 4 * RM, NT = WM * WN * 32;
    static constexpr int PA = TM + 4, PW = TN + 4;            // floats a row of k (padded: the stores are transposing)
    static constexpr int STAGE = TK * (PA + PW);
    static constexpr int SPLIT_BYTES = 2 * STAGE * 4, BYTES = SPLIT_BYTES + TM * TN * 4;
    static_assert(WN * 8 * RN == TN && (TM * TK / 4) % NT == 0, "the threads cover the tile");
};
typedef TileForm<8, 16, 4, 1, 2> Tile128;
typedef TileForm<8, 8, 2, 2, 3> Tile64;
typedef TileForm<8, 8, 1, 2, 6> Tile32;

// SPLIT (few blocks for the SMs): blockIdx.z takes `per_split` of the chunks and leaves every chunk's sums in `part`
// [chunk][M][N]; sum_chunks_kernel adds them in order, so the result is that of the other form to the bit.
template <typename F, typename OT, bool SPLIT>
__global__ void __launch_bounds__(F::NT, F::MIN_BLOCKS)
sgemm_tile_kernel(const float* __restrict__ A, int lda, const int* __restrict__ a_rows, int a_src_rows,
                  const float* __restrict__ W, long long w_group_stride, OT* __restrict__ C, int ldc,
                  const float* __restrict__ bias, const int* __restrict__ group_offsets, int num_groups, int M, int N, int K,
                  int* status, int per_split, float* __restrict__ part) {
    constexpr int NT = F::NT, PA = F::PA, PW = F::PW, STAGE = F::STAGE, RM = F::M, RN = F::N;
    constexpr int AP = F::TM * (TK / 4) / NT, WP = TN * (TK / 4) / NT;      // 16-byte pieces of a stage a thread
    extern __shared__ __align__(16) float sg_smem[];
    __shared__ int s_group, s_row0, s_row1;
    find_tile(group_offsets, num_groups, blockIdx.y, F::TM, M, &s_group, &s_row0, &s_row1);
    __syncthreads();
    const int g = s_group;
    if (g < 0) return;
    const int row0 = s_row0, row_end = s_row1, n0 = blockIdx.x * TN;
    const float* Wg = W + (size_t)g * (size_t)w_group_stride;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* tots = sg_smem + 2 * STAGE + tid;                  // this thread's totals, NT floats apart
    const int kp = (tid & 3) * 4, lr = tid >> 2;              // this thread loads k kp..kp+3 of rows lr, lr + NT / 4, ...
    const float* ap[AP];
#pragma unroll
    for (int i = 0; i < AP; i++) {
        const int r = row0 + lr + i * (NT / 4);
        long long src = -1;
        if (r < row_end) {
            src = a_rows ? a_rows[r] : r;
            if (src < 0 || src >= a_src_rows) {
                atomicOr(status, ST_BAD_ROW);
                src = -1;
            }
        }
        ap[i] = src >= 0 ? A + (size_t)src * lda : nullptr;
    }
    float4 ra[AP], rw[WP];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch = [&](int k0) {
        const bool in = k0 + kp < K;                          // (K is a multiple of 4)
#pragma unroll
        for (int i = 0; i < AP; i++) ra[i] = ap[i] && in ? *reinterpret_cast<const float4*>(ap[i] + k0 + kp) : zero;
#pragma unroll
        for (int i = 0; i < WP; i++) {
            const int n = n0 + lr + i * (NT / 4);
            rw[i] = n < N && in ? __ldg(reinterpret_cast<const float4*>(Wg + (size_t)n * K + k0 + kp)) : zero;
        }
    };
    auto stage = [&](float* s) {
#pragma unroll
        for (int i = 0; i < AP; i++) {
            const float v[4] = {ra[i].x, ra[i].y, ra[i].z, ra[i].w};
#pragma unroll
            for (int j = 0; j < 4; j++) s[(kp + j) * PA + lr + i * (NT / 4)] = v[j];
        }
        float* w = s + TK * PA;
#pragma unroll
        for (int i = 0; i < WP; i++) {
            const float v[4] = {rw[i].x, rw[i].y, rw[i].z, rw[i].w};
#pragma unroll
            for (int j = 0; j < 4; j++) w[(kp + j) * PW + lr + i * (NT / 4)] = v[j];
        }
    };
    // a warp's outputs: 4 RM rows x 8 RN features; a thread's rows m0 + {0..3} + 16 i, its features nn + {0..3} + 32 j
    const int m0 = (warp / F::WARPS_N) * 4 * RM + (lane >> 3) * 4, nn = (warp % F::WARPS_N) * 8 * RN + (lane & 7) * 4;
    unsigned long long acc[RM][RN / 2];
#pragma unroll
    for (int i = 0; i < RM; i++)
#pragma unroll
        for (int j = 0; j < RN / 2; j++) acc[i][j] = 0ull;
    const int k_begin = SPLIT ? blockIdx.z * per_split * CHUNK : 0, k_end = SPLIT ? min(K, k_begin + per_split * CHUNK) : K;
    fetch(k_begin);
    stage(sg_smem);
    __syncthreads();
    int buf = 0;
    for (int k0 = k_begin; k0 < k_end; k0 += TK) {
        const bool more = k0 + TK < k_end;
        if (more) fetch(k0 + TK);
        const float* sa = sg_smem + buf * STAGE + m0;
        const float* sw = sg_smem + buf * STAGE + TK * PA + nn;
#pragma unroll
        for (int kk = 0; kk < TK; kk++) {
            float a[RM];
            unsigned long long w[RN / 2];
#pragma unroll
            for (int i = 0; i < RM / 4; i++) {
                const float4 v = *reinterpret_cast<const float4*>(sa + kk * PA + 16 * i);
                a[4 * i] = v.x, a[4 * i + 1] = v.y, a[4 * i + 2] = v.z, a[4 * i + 3] = v.w;
            }
#pragma unroll
            for (int j = 0; j < RN / 4; j++) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(sw + kk * PW + 32 * j);
                w[2 * j] = v.x, w[2 * j + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < RM; i++) {
                const unsigned long long both = pack2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < RN / 2; j++) fma2(acc[i][j], both, w[j]);
            }
        }
        if (SPLIT && (!more || (k0 + TK) % CHUNK == 0)) {
            float* dst = part + (size_t)(k0 / CHUNK) * M * N;
#pragma unroll
            for (int i = 0; i < RM; i++) {
                const int r = row0 + m0 + (i & 3) + 16 * (i >> 2);
#pragma unroll
                for (int j = 0; j < RN / 2; j++) {
                    const int c = n0 + nn + 32 * (j >> 1) + 2 * (j & 1);
                    float v[2];
                    unpack2(acc[i][j], v[0], v[1]);
                    acc[i][j] = 0ull;
#pragma unroll
                    for (int q = 0; q < 2; q++)
                        if (r < row_end && c + q < N) dst[(size_t)r * N + c + q] = v[q];
                }
            }
        }
        if (!SPLIT && (!more || (k0 + TK) % CHUNK == 0)) {
            const bool first = k0 < CHUNK;
#pragma unroll
            for (int i = 0; i < RM; i++)
#pragma unroll
                for (int j = 0; j < RN / 2; j++) {
                    float lo, hi;
                    unpack2(acc[i][j], lo, hi);
                    float* t = tots + (i * RN + 2 * j) * NT;
                    t[0] = (first ? 0.f : t[0]) + lo, t[NT] = (first ? 0.f : t[NT]) + hi;
                    acc[i][j] = 0ull;
                }
        }
        if (more) stage(sg_smem + (buf ^ 1) * STAGE);         // (read last before the barrier that ended the stage before)
        __syncthreads();
        buf ^= 1;
    }
    if (SPLIT) return;
    const bool whole = sizeof(OT) == 4 && ldc % 4 == 0 && ((uintptr_t)C & 15) == 0;
#pragma unroll
    for (int i = 0; i < RM; i++) {
        const int r = row0 + m0 + (i & 3) + 16 * (i >> 2);
        if (r >= row_end) continue;
        OT* dst = C + (size_t)r * ldc;
#pragma unroll
        for (int j = 0; j < RN; j += 4) {
            const int c = n0 + nn + 8 * j;
            float v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                v[q] = tots[(i * RN + j + q) * NT];
                if (bias && c + q < N) v[q] += bias[c + q];
            }
            if (whole && c + 4 <= N) {
                *reinterpret_cast<float4*>(dst + c) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (c + q < N) st_f(dst + c + q, v[q]);
            }
        }
    }
}
static_assert(CHUNK % TK == 0, "a chunk is whole stages");

// C[r, n] = the chunks' sums of (r, n) in order (+ bias[n]); with groups, rows of none (before the first, past the last) are left alone
template <typename OT>
__global__ void __launch_bounds__(256)
sum_chunks_kernel(const float* __restrict__ part, int chunks, OT* __restrict__ C, int ldc, const float* __restrict__ bias,
                  const int* __restrict__ group_offsets, int num_groups, int M, int N) {
    const size_t n = (size_t)M * N, i = (size_t)blockIdx.x * 256 + threadIdx.x;
    const size_t from = group_offsets ? (size_t)max(0, group_offsets[0]) * N : 0;
    const size_t live = group_offsets ? (size_t)min(M, group_offsets[num_groups]) * N : n;
    if (i < from || i >= live) return;
    float t = 0.f;
#pragma unroll 4
    for (int c = 0; c < chunks; c++) t += part[(size_t)c * n + i];
    const int r = (int)(i / N), col = (int)(i % N);
    st_f(C + (size_t)r * ldc + col, bias ? t + bias[col] : t);
}

// Few rows: the time is the weight stream, so what counts is the bytes in flight on every SM, also for the narrow
// products (2,048 features).  A block takes 16 FL features and up to R rows; its eight warps take the chunks of k in turn, each
// with cp.async stages of its own (SK k of the weight rows and of the R rows), so nobody waits for a block-wide barrier
// while it streams; after each round of eight chunks their sums are added in order.  A lane holds FL features and half of the
// rows: every 16-byte read of shared memory costs an SM four cycles whatever it reads, so the rows a tile does not have
// are not read (a decode step's experts have one or two), and two features a lane halve the reads of the rows.  Measured
// with 8 tokens, us (the kernel above / one feature a lane and all rows read / as here): 2,048 x 151,936 weights 393 / 337 /
// 235 (5.3 TB/s); 60 experts of 2,048 x 2,816, four a token, 195 / 178 / 97 (5.9 TB/s); 5,632 x 2,048 89 / 21 / 20.
constexpr int SWARPS = 8;
template <int R, int FL>
struct RowsForm {
    static constexpr int SK = FL == 1 ? 64 : 32, SP = SK + 4, SF = 16 * FL;
    static constexpr int STAGE = (SF + R) * SP;               // floats a warp and stage
    static constexpr int PART = SWARPS * SF * R;              // chunk sums of a round
    static constexpr int BYTES = (2 * SWARPS * STAGE + 2 * PART) * 4;
    static_assert(CHUNK % SK == 0, "a chunk is whole pieces");
};
template <int R, int FL, typename OT>
__global__ void __launch_bounds__(SWARPS * 32)
sgemm_rows_kernel(const float* __restrict__ A, int lda, const int* __restrict__ a_rows, int a_src_rows,
                  const float* __restrict__ W, long long w_group_stride, OT* __restrict__ C, int ldc,
                  const float* __restrict__ bias, const int* __restrict__ group_offsets, int num_groups, int M, int N, int K,
                  int* status) {
    using F = RowsForm<R, FL>;
    constexpr int STAGE = F::STAGE, PART = F::PART, SK = F::SK, SP = F::SP, SF = F::SF, PIECES = CHUNK / SK;
    constexpr int UNITS = SK / 4, LROWS = 32 / UNITS;         // 16-byte units a staged row; rows a warp copies at once
    extern __shared__ __align__(16) float sg_smem[];
    __shared__ int s_group, s_row0, s_row1;
    find_tile(group_offsets, num_groups, blockIdx.y, R, M, &s_group, &s_row0, &s_row1);
    __syncthreads();
    const int g = s_group;
    if (g < 0) return;
    const int row0 = s_row0, rows = min(R, s_row1 - row0), n0 = blockIdx.x * SF;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // this lane copies 16-byte unit kq of weight rows rq, rq + LROWS, ... and of rows rq, rq + LROWS, ...
    const int kq = (lane % UNITS) * 4, rq = lane / UNITS;
    const float* Wg = W + (size_t)g * (size_t)w_group_stride + (size_t)n0 * K;
    constexpr int AL = (R + LROWS - 1) / LROWS;
    const float* ap[AL];
#pragma unroll
    for (int i = 0; i < AL; i++) {
        const int r = rq + LROWS * i;
        long long src = -1;
        if (r < rows) {
            src = a_rows ? a_rows[row0 + r] : row0 + r;
            if (src < 0 || src >= a_src_rows) {
                atomicOr(status, ST_BAD_ROW);
                src = -1;
            }
        }
        ap[i] = src >= 0 ? A + (size_t)src * lda : nullptr;
    }
    float* mine = sg_smem + warp * 2 * STAGE;
    float* part = sg_smem + SWARPS * 2 * STAGE;
    const int chunks = (K + CHUNK - 1) / CHUNK, rounds = (chunks + SWARPS - 1) / SWARPS;
    // step s of this warp: piece s % PIECES of chunk (s / PIECES) * SWARPS + warp
    auto issue = [&](int s) {
        const int k = ((s / PIECES) * SWARPS + warp) * CHUNK + (s % PIECES) * SK + kq;
        float* d = mine + (s & 1) * STAGE + kq;
#pragma unroll
        for (int i = 0; i < SF / LROWS; i++) {
            const int f = rq + LROWS * i;
            const bool ok = k < K && n0 + f < N;
            cp16(d + f * SP, ok ? Wg + (size_t)f * K + k : W, ok ? 16 : 0);
        }
#pragma unroll
        for (int i = 0; i < AL; i++) {
            if (LROWS * i >= rows) break;
            const bool ok = k < K && ap[i];
            if (rq + LROWS * i < R) cp16(d + (SF + rq + LROWS * i) * SP, ok ? ap[i] + k : A, ok ? 16 : 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int f = lane & 15, h = lane >> 4;
    const int steps = rounds * PIECES;
    issue(0);
    issue(1);
    constexpr int OUTS = (SF * R + SWARPS * 32 - 1) / (SWARPS * 32);
    float total[OUTS];                                        // of outputs tid + 256 i: (feature % SF, row / SF)
#pragma unroll
    for (int i = 0; i < OUTS; i++) total[i] = 0.f;
    // RL: rows a lane (of the two halves) really holds
    auto walk = [&](auto rl) {
        constexpr int RL = decltype(rl)::value;
        for (int r = 0; r < rounds; r++) {
            float acc[FL][RL];
#pragma unroll
            for (int e = 0; e < FL; e++)
#pragma unroll
                for (int i = 0; i < RL; i++) acc[e][i] = 0.f;
#pragma unroll 1
            for (int p = 0; p < PIECES; p++) {
                const int s = r * PIECES + p;
                if (s + 1 < steps)
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                else
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                __syncwarp();
                const float* w = mine + (s & 1) * STAGE + f * SP;
                const float* a = mine + (s & 1) * STAGE + (SF + h * RL) * SP;
                // (pieces beyond K are zeros: they add 0 * 0; a chunk that does not exist is not added up below)
#pragma unroll
                for (int k = 0; k < SK; k += 4) {
                    float4 wv[FL];
#pragma unroll
                    for (int e = 0; e < FL; e++) wv[e] = *reinterpret_cast<const float4*>(w + e * 16 * SP + k);
#pragma unroll
                    for (int i = 0; i < RL; i++) {
                        const float4 av = *reinterpret_cast<const float4*>(a + i * SP + k);
#pragma unroll
                        for (int e = 0; e < FL; e++) {
                            acc[e][i] = fmaf(av.x, wv[e].x, acc[e][i]), acc[e][i] = fmaf(av.y, wv[e].y, acc[e][i]);
                            acc[e][i] = fmaf(av.z, wv[e].z, acc[e][i]), acc[e][i] = fmaf(av.w, wv[e].w, acc[e][i]);
                        }
                    }
                }
                __syncwarp();
                if (s + 2 < steps) issue(s + 2);
            }
            float* pr = part + (r & 1) * PART;
#pragma unroll
            for (int i = 0; i < RL; i++)
#pragma unroll
                for (int e = 0; e < FL; e++) pr[(warp * R + h * RL + i) * SF + f + 16 * e] = acc[e][i];
            __syncthreads();
            const int have = min(SWARPS, chunks - r * SWARPS);
#pragma unroll
            for (int i = 0; i < OUTS; i++) {
                const int at = tid + i * SWARPS * 32;
                if (at < SF * 2 * RL)
                    for (int c = 0; c < have; c++) total[i] += pr[c * R * SF + at];
            }
        }
    };
    if (rows <= 2) walk(std::integral_constant<int, 1>());
    else if (rows <= 4) walk(std::integral_constant<int, 2>());
    else if (R <= 8 || rows <= 8) walk(std::integral_constant<int, 4>());
    else walk(std::integral_constant<int, R / 2>());
#pragma unroll
    for (int i = 0; i < OUTS; i++) {
        const int at = tid + i * SWARPS * 32, n = n0 + at % SF, row = at / SF;
        if (row < rows && n < N) st_f(C + (size_t)(row0 + row) * ldc + n, bias ? total[i] + bias[n] : total[i]);
    }
}

// Which form a product of 32-bit operands takes.
constexpr long long SCRATCH_FLOATS = 1ll << 25;      // chunk sums a launch may leave (128 MB)
struct Plan {
    int rows;            // > 0: sgemm_rows_kernel with so many rows a tile; else sgemm_tile_kernel
    int tile;            // 128, 64 or 32 rows a tile
    int splits, per;     // K splits and chunks a split
    int pass;            // rows a launch (all, or with splits as many as SCRATCH_FLOATS has room for)
};
long long plan_floats(const Plan& p, int N, int K) {
    return p.splits > 1 ? (long long)((K + CHUNK - 1) / CHUNK) * p.pass * N : 0;
}
Plan plan_f32(int M, int N, int K, bool grouped, int num_groups) {
    Plan p = {0, 0, 1, 0, M};
    const int groups = grouped ? num_groups : 1, each = M / groups, chunks = (K + CHUNK - 1) / CHUNK;
    // Few rows a group: the weight stream is the time.  (Measured, us: 60 groups of 2,048 x 2,816 with 7 rows each 297
    // against 814 in tiles of 32; beyond 16 rows a tile of it would have to read the weights twice.)
    if (grouped ? each <= 16 : M <= 16) {
        p.rows = grouped ? (M <= 64 || each <= 6 ? 8 : 16) : (M <= 8 ? 8 : 16);
        return p;
    }
    // The tile whose waves take least: blocks over the blocks the SMs hold, times a wave's rows, by the rate the
    // form reaches with all SMs full (TFLOP/s, measured).  A group's last tile is half empty on average.  Less than half a wave:
    // the chunks of k side by side (2,048 x 6,144 weights at 24 / 64 / 100 rows: 53 / 56 / 97 us, 243 / 201 / 185 without); every chunk's
    // sums go through memory, so a product without groups whose sums find no room goes over its rows in passes.
    const int cols = (N + TN - 1) / TN, tms[3] = {128, 64, 32};
    // blocks an SM holds: with the totals in shared memory (no splits) the form of 32 rows is at five.  (Room for a sixth, the few bytes that
    // say which tile it is in the padding, leaves L1 too little: 60 groups of 17 rows, 2,816 x 2,048, 592 -> 683 us.)
    auto slots = [](int f, bool split) { return f == 0 ? 2 : f == 1 ? 3 : split ? 6 : 5; };
    auto rate = [](int f, bool split) { return f == 0 ? 54.f : f == 1 ? 50.f : split ? 43.6f : 36.3f; };
    float best = 0.f;
    for (int f = 0; f < 3; f++) {
        // the plan for `pass` rows a launch, with K splits if asked for and two blocks or more find room
        auto consider = [&](int pass, bool split) {
            const long long blocks = cols * (long long)(grouped ? M / tms[f] + (num_groups + 1) / 2 : (pass + tms[f] - 1) / tms[f]);
            const int here = slots(f, split);
            const long long room = (long long)here * scan_sms();
            int splits = split ? (int)(room / blocks < chunks ? room / blocks : chunks) : 1;
            if (split && splits < 2) return;
            const int per = (chunks + splits - 1) / splits;
            splits = (chunks + per - 1) / per;
            const float waves = (float)((blocks * splits + room - 1) / room) * per / chunks;
            // us: a wave's multiply-adds at the form's rate; the chunks' sums written and read at some 8 TB/s, and a launch more
            float cost = waves * here * tms[f] / rate(f, split) * scan_sms() * TN * 2e-6f * K;
            if (splits > 1) cost += 8.f * chunks * pass * N / 8e6f + 3.f;
            const int passes = (M + pass - 1) / pass;
            if (passes > 1) cost *= 1.25f * passes;          // (as measured: the weights come from memory again, the last one is not whole)
            if (!p.tile || cost < best) p.tile = tms[f], p.splits = splits, p.per = per, p.pass = pass, best = cost;
        };
        consider(M, false);
        const long long fit = SCRATCH_FLOATS / ((long long)chunks * N);      // rows whose sums find room
        if (fit >= M)
            consider(M, true);
        else if (!grouped && fit >= tms[f]) {
            const int most = (int)(fit / tms[f]) * tms[f], passes = (M + most - 1) / most;
            consider(((M + passes - 1) / passes + tms[f] - 1) / tms[f] * tms[f], true);
        }
    }
    return p;
}

// The forms above, for 32-bit operands whose rows are whole 16-byte units; -1 where they do not apply.
template <typename OT>
int launch_f32(const float* A, int lda, const int* a_rows, int a_src_rows, const float* W, long long w_group_stride, OT* C,
               int ldc, const float* bias, const int* group_offsets, int num_groups, int M, int N, int K, int* status,
               float* scratch, long long scratch_floats, cudaStream_t stream) {
    Plan p = plan_f32(M, N, K, group_offsets != nullptr, num_groups);
    if (plan_floats(p, N, K) > scratch_floats) p.splits = 1, p.pass = M;
#define RUN(kernel, bytes, grid, threads, ...)                                                                              \
    {                                                                                                                      \
        const dim3 gr = grid;                                                                                              \
        if (gr.y > 65535) return -1;                                                                                       \
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);                  \
        if (e != cudaSuccess) return (int)e;                                                                               \
        kernel<<<gr, threads, bytes, stream>>>(a_rows ? A : A + (size_t)r0 * lda, lda, a_rows ? a_rows + r0 : nullptr,      \
                                               a_rows ? a_src_rows : a_src_rows - r0, W, w_group_stride, C + (size_t)r0 * ldc, ldc, \
                                               bias, group_offsets, num_groups, m, N, K, status __VA_OPT__(, ) __VA_ARGS__); \
    }
    int r0 = 0, m = M;              // the rows of a pass
    if (p.rows) {
        const int tiles = group_offsets ? (M < num_groups ? M : num_groups) + M / p.rows : (M + p.rows - 1) / p.rows;
#define ROWS(R, FL) RUN((sgemm_rows_kernel<R, FL, OT>), (RowsForm<R, FL>::BYTES), dim3((N + 16 * FL - 1) / (16 * FL), tiles), SWARPS * 32)
        // two features a lane where that still leaves every SM a block
        const bool wide = (long long)((N + 31) / 32) * tiles >= scan_sms();
        if (p.rows == 8) {
            if (wide) ROWS(8, 2) else ROWS(8, 1)
        } else {
            if (wide) ROWS(16, 2) else ROWS(16, 1)
        }
#undef ROWS
        return launch_status();
    }
    const int cols = (N + TN - 1) / TN;
    for (; r0 < M; r0 += p.pass) {
        m = M - r0 < p.pass ? M - r0 : p.pass;
        const int tiles = (m + p.tile - 1) / p.tile + (group_offsets ? (m < num_groups ? m : num_groups) : 0);
#define TILE(F)                                                                                                            \
    {                                                                                                                      \
        if (p.splits > 1) RUN((sgemm_tile_kernel<F, OT, true>), F::SPLIT_BYTES, dim3(cols, tiles, p.splits), F::NT, p.per, scratch) \
        else RUN((sgemm_tile_kernel<F, OT, false>), F::BYTES, dim3(cols, tiles), F::NT, 0, nullptr)                        \
    }
        if (p.tile == 128) TILE(Tile128)
        else if (p.tile == 64) TILE(Tile64)
        else TILE(Tile32)
#undef TILE
#undef RUN
        if (p.splits > 1) {
            const long long n = (long long)m * N;
            sum_chunks_kernel<OT><<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(scratch, (K + CHUNK - 1) / CHUNK, C + (size_t)r0 * ldc, ldc,
                                                                                  bias, group_offsets, num_groups, m, N);
        }
        const int rc = launch_status();
        if (rc) return rc;
    }
    return 0;
}

template <typename AT, typename WT, typename OT>
int launch(const void* A, int lda, const int* a_rows, int a_src_rows, const void* W, long long w_group_stride, void* C,
           int ldc, const float* bias, const int* group_offsets, int num_groups, int M, int N, int K, int* status,
           float* scratch, long long scratch_floats, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || (group_offsets && num_groups <= 0)) return 0;      // (rows of no group are left alone)
    const int a_vec = (K % 4 == 0) && (lda % 4 == 0) && ((uintptr_t)A % 16 == 0);
    const int w_vec = (K % 4 == 0) && ((uintptr_t)W % 16 == 0) && ((w_group_stride * (long long)sizeof(WT)) % 16 == 0);
    if constexpr (sizeof(AT) == 4 && sizeof(WT) == 4) {
        if (a_vec && w_vec && K > 0) {
            const int rc = launch_f32<OT>((const float*)A, lda, a_rows, a_src_rows, (const float*)W, w_group_stride, (OT*)C, ldc, bias,
                                          group_offsets, num_groups, M, N, K, status, scratch, scratch_floats, stream);
            if (rc != -1) return rc;
        }
    }
    if (M <= (group_offsets ? 8 * RT : 2 * RT)) {
        // few rows: the weight stream is what takes the time
        const int r_tiles = group_offsets ? (M < num_groups ? M : num_groups) + M / RT : (M + RT - 1) / RT;
        dim3 rgrid((N + RF - 1) / RF, r_tiles);
        gemm_rows_kernel<AT, WT, OT><<<rgrid, RTHREADS, 0, stream>>>(
            (const AT*)A, lda, a_rows, a_src_rows, (const WT*)W, w_group_stride, (OT*)C, ldc, bias, group_offsets,
            num_groups, M, N, K, a_vec, w_vec, status);
        return launch_status();
    }
    const int m_tiles = (M + BM - 1) / BM + (group_offsets ? num_groups : 0);
    dim3 grid((N + BN - 1) / BN, m_tiles);
    if (grid.y > 65535) return (int)cudaErrorInvalidValue;
    gemm_generic_kernel<AT, WT, OT><<<grid, THREADS, 0, stream>>>(
        (const AT*)A, lda, a_rows, a_src_rows, (const WT*)W, w_group_stride, (OT*)C, ldc, bias, group_offsets,
        num_groups, M, N, K, a_vec, w_vec, status);
    return launch_status();
}

}  // namespace

// Floats of scratch that moe_gemm_generic can use for such a product of 32-bit operands, 2^25 at most (without them it takes
// the form that needs none: the same result, fewer blocks).
MOE_API long long moe_gemm_scratch_floats(int M, int N, int K, int num_groups) {
    if (M <= 0 || N <= 0 || K <= 0 || K % 4) return 0;
    return plan_floats(plan_f32(M, N, K, num_groups > 0, num_groups), N, K);
}
// Blocks of the tile form of `tile` rows that an SM holds (split: with K splits).
MOE_API int moe_gemm_tile_room(int tile, int split) {
    int n = -1;
#define ROOM(F)                                                                                                            \
    {                                                                                                                      \
        auto kernel = split ? sgemm_tile_kernel<F, float, true> : sgemm_tile_kernel<F, float, false>;                      \
        const int bytes = split ? F::SPLIT_BYTES : F::BYTES;                                                               \
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess ||             \
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, F::NT, bytes) != cudaSuccess)                        \
            return -1;                                                                                                     \
    }
    if (tile == 128) ROOM(Tile128)
    else if (tile == 64) ROOM(Tile64)
    else if (tile == 32) ROOM(Tile32)
#undef ROOM
    return n;
}
// The form such a product takes: rows a tile of the form for few rows (or 0), rows a tile, K splits, chunks a split, rows a pass.
MOE_API void moe_gemm_plan(int M, int N, int K, int num_groups, int* out) {
    const Plan p = plan_f32(M, N, K, num_groups > 0, num_groups);
    out[0] = p.rows, out[1] = p.rows ? 0 : p.tile, out[2] = p.splits, out[3] = p.per, out[4] = p.pass;
}

// A: [*, lda] of a_dt; W: [G][N, K] of w_dt; C: [M, ldc] of c_dt.  `a_rows` (may be
// null) maps output row -> row of A; `a_src_rows` bounds it.  `group_offsets`
// (may be null) has num_groups + 1 entries on the device.
MOE_API int moe_gemm_generic(const void* A, int a_dt, int lda, const int* a_rows, int a_src_rows, const void* W,
                             int w_dt, long long w_group_stride, void* C, int c_dt, int ldc, const float* bias,
                             const int* group_offsets, int num_groups, int M, int N, int K, int* status,
                             float* scratch, long long scratch_floats, cudaStream_t stream) {
#define GO(AT, WT, OT)                                                                                              \
    return launch<AT, WT, OT>(A, lda, a_rows, a_src_rows, W, w_group_stride, C, ldc, bias, group_offsets, num_groups, \
                              M, N, K, status, scratch, scratch_floats, stream)
    typedef __nv_bfloat16 bf;
    if (a_dt == DT_F32 && w_dt == DT_F32 && c_dt == DT_F32) GO(float, float, float);
    if (a_dt == DT_F32 && w_dt == DT_F32 && c_dt == DT_BF16) GO(float, float, bf);
    if (a_dt == DT_F32 && w_dt == DT_BF16 && c_dt == DT_F32) GO(float, bf, float);
    if (a_dt == DT_F32 && w_dt == DT_BF16 && c_dt == DT_BF16) GO(float, bf, bf);
    if (a_dt == DT_BF16 && w_dt == DT_F32 && c_dt == DT_F32) GO(bf, float, float);
    if (a_dt == DT_BF16 && w_dt == DT_F32 && c_dt == DT_BF16) GO(bf, float, bf);
    if (a_dt == DT_BF16 && w_dt == DT_BF16 && c_dt == DT_F32) GO(bf, bf, float);
    if (a_dt == DT_BF16 && w_dt == DT_BF16 && c_dt == DT_BF16) GO(bf, bf, bf);
#undef GO
    return (int)cudaErrorInvalidValue;
}
