// Matrix product on the CUDA cores: C[M,N] (+)= A[M,K] * W[N,K]^T.
//
// Float32 multiply-adds, no tensor cores, no reduced-precision mode: the part of the 32-bit path that gemm_split.cu does not
// take (float32 weights, and bfloat16 weights of less than 65,536 elements or off a 16-byte boundary), and the fallback for
// operand types or sizes that the tensor-core kernels refuse.  Operands may be float32 or bfloat16 in any combination
// (widening bfloat16 is exact).
//
// One order of summation for every element, whatever kernel computes it: K is cut into segments
// of SEG terms, a segment is accumulated in float32 with one fused multiply-add per term, k
// ascending, from zero, and the segments' sums are added in ascending order to a total that
// starts at zero.  So an output element's value does not depend on M, on the tile it falls in or
// on its neighbours, and a product of few rows can give its segments to different lanes.
#include "common.cuh"
#include "tape.cuh"

namespace {

constexpr int SEG = 256;

// ---- many rows: tiles in shared memory -----------------------------------------------------
// A block computes BM x BN.  GROUPS groups of four warps take its segments in turn, each with
// tiles of its own, and the block adds a round's sums in ascending order: the groups cover one
// another's load latency, and a narrow output (64 x 64 tiles of 466 x 1,024 are 128 blocks)
// still keeps sixteen warps on an SM.  A thread multiplies TM x TN, as pairs of rows with the
// packed multiply-add (two float32 lanes, each rounded like fmaf).  Tiles lie in shared memory
// with k as the row, a row's columns exchanged in groups of eight by the k group they belong to:
// the stores of one warp (8 rows x 4 k groups) then hit 32 banks, and a thread's TM or TN
// neighbouring values stay neighbours.  Bound by the multiply-add pipe (57 % busy at 466 x 6,144 x
// 1,024, the rest waits on loads and barriers): the packed form does what two plain multiply-adds
// do in as many pipe cycles but halves the instructions (466 x 6,144 x 1,024: 183 us, plain 211;
// a 64 x 128 tile of 8 x 8 a thread 212).  Against one group with a tile ahead in registers, 64 x
// 64 and 4 x 4 a thread: 466 x 6,144 x 1,024 303 -> 183 us, 466 x 1,024 x 3,072 242 -> 94, 100 x
// 4,096 x 1,024 87 -> 34 (bfloat16 weights; 31 to 38 TFLOP/s).
constexpr int BM = 64, BN = 64, TM = 8, TN = 4, GROUP = BM / TM * BN / TN;
constexpr int BK = 16;

__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& x, float& y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// 16 / sizeof(T) neighbouring elements of a row from column kk on, zeros behind the row's end.
template <typename T, bool VEC>
__device__ __forceinline__ void load_piece(const T* row, bool live, int kk, int k, float (&v)[16 / sizeof(T)]) {
    constexpr int P = 16 / sizeof(T);
    if (VEC && live && kk + P <= k) {
        const uint4 raw = *reinterpret_cast<const uint4*>(row + kk);
        const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int i = 0; i < P; ++i) v[i] = to_f32(e[i]);
    } else {
#pragma unroll
        for (int i = 0; i < P; ++i) v[i] = live && kk + i < k ? to_f32(row[kk + i]) : 0.0f;
    }
}

// A tile's BK columns of ROWS rows: registers first (ahead of the multiply-adds), shared memory later.
template <typename T, int ROWS, bool VEC>
struct TileLoader {
    static constexpr int P = 16 / sizeof(T), PER_ROW = BK / P, N = ROWS * PER_ROW / GROUP;
    static_assert(ROWS * PER_ROW % GROUP == 0, "every thread loads the same number of pieces");
    float v[N][P];
    __device__ __forceinline__ void load(const T* base, int ld, int row0, int rows, int k0, int k, int tid) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int id = tid + i * GROUP, r = row0 + id / PER_ROW;
            load_piece<T, VEC>(base + (size_t)r * ld, r < rows, k0 + id % PER_ROW * P, k, v[i]);
        }
    }
    __device__ __forceinline__ void store(float (*tile)[ROWS], int tid) const {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int id = tid + i * GROUP, r = id / PER_ROW, kk = id % PER_ROW * P;
#pragma unroll
            for (int j = 0; j < P; ++j) tile[kk + j][r ^ (((kk + j) >> 2 & 3) * 8)] = v[i][j];
        }
    }
};

template <typename TA, typename TW, int GROUPS, bool VEC>
__global__ void __launch_bounds__(GROUP * GROUPS)
gemm_tiled_kernel(const TA* a, const TW* __restrict__ w, float* c, int m, int n, int k, int lda, int ldw, int ldc,
                  int accumulate) {
    extern __shared__ __align__(16) float tiles[];               // a group's 2 x BK x (BM + BN), its sums afterwards
    static_assert(2 * BK * (BM + BN) == BM * BN, "a group's sums take the place of its tiles");
    constexpr int MINE = BM * BN / 4 / (GROUP * GROUPS);         // float4 of the total per thread
    const int group = threadIdx.x / GROUP, tid = threadIdx.x % GROUP;
    const int lane = tid & 31, warp = tid >> 5;
    const int ty = (warp % 2 * 4 + lane / 8) * TM, tx = (warp / 2 * 8 + lane % 8) * TN;       // a warp: 4 x 8 threads
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float(*as)[BK][BM] = reinterpret_cast<float(*)[BK][BM]>(tiles + group * BM * BN);
    float(*ws)[BK][BN] = reinterpret_cast<float(*)[BK][BN]>(tiles + group * BM * BN + 2 * BK * BM);
    auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(GROUP) : "memory"); };

    float4 tot[MINE];
#pragma unroll
    for (int i = 0; i < MINE; ++i) tot[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    TileLoader<TA, BM, VEC> la;
    TileLoader<TW, BN, VEC> lw;
    const int segs = (k + SEG - 1) / SEG;
    pdl_launch();
    for (int seg0 = 0; seg0 < segs; seg0 += GROUPS) {
        const int seg = seg0 + group;
        if (seg < segs) {
            const int first = seg * SEG, blocks = (min(SEG, k - first) + BK - 1) / BK;
            unsigned long long acc[TM / 2][TN];
#pragma unroll
            for (int i = 0; i < TM / 2; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
            lw.load(w, ldw, n0, n, first, k, tid);
            if (seg0 == 0) pdl_wait();
            la.load(a, lda, m0, m, first, k, tid);
            la.store(as[0], tid);
            lw.store(ws[0], tid);
            group_sync();
            for (int kb = 0; kb < blocks; ++kb) {
                const int buf = kb & 1;
                if (kb + 1 < blocks) {
                    la.load(a, lda, m0, m, first + (kb + 1) * BK, k, tid);
                    lw.load(w, ldw, n0, n, first + (kb + 1) * BK, k, tid);
                }
#pragma unroll
                for (int kk = 0; kk < BK; ++kk) {
                    const int x = (kk >> 2 & 3) * 8;
                    unsigned long long av[TM / 2], wv[TN];
#pragma unroll
                    for (int i = 0; i < TM / 2; i += 2) {
                        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(&as[buf][kk][(ty ^ x) + 2 * i]);
                        av[i] = t.x;
                        av[i + 1] = t.y;
                    }
                    const float4 t = *reinterpret_cast<const float4*>(&ws[buf][kk][tx ^ x]);
                    wv[0] = pack2(t.x, t.x);
                    wv[1] = pack2(t.y, t.y);
                    wv[2] = pack2(t.z, t.z);
                    wv[3] = pack2(t.w, t.w);
#pragma unroll
                    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) acc[i][j] = fma2(av[i], wv[j], acc[i][j]);
                }
                if (kb + 1 < blocks) {
                    la.store(as[buf ^ 1], tid);
                    lw.store(ws[buf ^ 1], tid);
                }
                group_sync();
            }
            float* sums = tiles + group * BM * BN;
#pragma unroll
            for (int i = 0; i < TM / 2; ++i) {
                float v[2][TN];
#pragma unroll
                for (int j = 0; j < TN; ++j) unpack2(acc[i][j], v[0][j], v[1][j]);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    *reinterpret_cast<float4*>(&sums[(ty + 2 * i + h) * BN + tx]) =
                        make_float4(v[h][0], v[h][1], v[h][2], v[h][3]);
            }
        } else if (seg0 == 0) {
            pdl_wait();
        }
        __syncthreads();
        const int here = min(GROUPS, segs - seg0);
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
            for (int g = 0; g < here; ++g) {
                const float4 v = *reinterpret_cast<const float4*>(&tiles[g * BM * BN + (threadIdx.x + i * GROUP * GROUPS) * 4]);
                tot[i].x += v.x;
                tot[i].y += v.y;
                tot[i].z += v.z;
                tot[i].w += v.w;
            }
        }
        if (seg0 + GROUPS < segs) __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
        const int at = (threadIdx.x + i * GROUP * GROUPS) * 4, row = m0 + at / BN, col = n0 + at % BN;
        if (row >= m) continue;
        const float v[4] = {tot[i].x, tot[i].y, tot[i].z, tot[i].w};
        float* p = c + (size_t)row * ldc + col;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (col + j < n) p[j] = accumulate ? p[j] + v[j] : v[j];
    }
}

// ---- few rows: weights streamed, a lane per (column, segment) -------------------------------
// A warp takes 8 columns and a span of 4 segments; a lane walks its segment for MT rows at once.
// The warp's weights (8 x 4 pieces of SEG elements, each contiguous in memory) travel by cp.async
// into rows of their own in shared memory, all of them requested before the wait on the kernel
// before; rows there are 16 bytes longer than a piece, so that eight lanes reading 16 bytes each
// of eight rows hit all banks.  The rows of A follow, a segment's piece likewise.  A block has
// `ws` warps side by side along K and as many column groups as its other warps; longer K goes
// on in rounds.  One row is bound by the stream of the weights (151,936 x 1,024 in bfloat16: 61 us,
// 5.1 TB/s; the tiles took 693), several rows by the reads of A from shared memory (three rows 121
// us, 17 rows 454); narrow products by one chain of latencies (3 x 1,024 x 3,072 under 10 us, the
// tiles 251).
constexpr int SPAN = 4 * SEG, COLS = 8, MAX_ROWS = 32;

__device__ __forceinline__ void cp16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

template <typename TW>
constexpr int piece_pitch() { return SEG * (int)sizeof(TW) + 16; }

template <typename TW>
size_t rows_smem(int ws, int wc, int mt) {
    return (size_t)ws * wc * 32 * piece_pitch<TW>() + (size_t)mt * ws * 4 * piece_pitch<float>() +
           (size_t)(ws * 4 * mt + MAX_ROWS) * wc * COLS * 4;
}

template <typename TW, int MT>
__global__ void __launch_bounds__(128)
gemm_rows_kernel(const float* a, const TW* __restrict__ w, float* c, int m, int n, int k, int lda, int ldw, int ldc,
                 int accumulate, int ws, int wc) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int WP = piece_pitch<TW>(), AP = piece_pitch<float>(), PER = 16 / sizeof(TW);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wk = warp % ws, wn = warp / ws, cols = wc * COLS;
    unsigned char* wbuf = smem + (size_t)warp * 32 * WP;
    unsigned char* abuf = smem + (size_t)ws * wc * 32 * WP;
    float* part = reinterpret_cast<float*>(abuf + (size_t)MT * ws * 4 * AP);     // [segment][column][row]
    float* total = part + (size_t)ws * 4 * cols * MT;                            // [row][column]
    const int col0 = blockIdx.x * cols;
    const int segs = (k + SEG - 1) / SEG;
    const int rounds = (segs + 4 * ws - 1) / (4 * ws);
    const int my_col = lane & 7, my_seg = lane >> 3;
    for (int i = threadIdx.x; i < MAX_ROWS * cols; i += blockDim.x) total[i] = 0.0f;

    for (int round = 0; round < rounds; ++round) {
        const int seg0 = (round * ws + wk) * 4;                  // first segment of this warp
#pragma unroll
        for (int r = 0; r < 32; ++r) {                           // piece r: column r & 7, segment r >> 3
            const int seg = seg0 + (r >> 3), col = min(n - 1, col0 + wn * COLS + (r & 7));
            const int left = k - seg * SEG;
            for (int at = lane * PER; at < min(SEG, left); at += 32 * PER)
                cp16(wbuf + r * WP + at * sizeof(TW), w + (size_t)col * ldw + (size_t)seg * SEG + at);
        }
        if (round == 0) {
            pdl_launch();
            pdl_wait();
        }
        for (int m0 = 0; m0 < m; m0 += MT) {
            const int k0 = round * ws * SPAN;                    // the round's first column of A
            const int len = min(ws * SPAN, k - k0);
            for (int id = threadIdx.x; id < MT * ws * SPAN / 4; id += blockDim.x) {
                const int row = id / (ws * SPAN / 4), at = id % (ws * SPAN / 4) * 4;
                if (at < len)
                    cp16(abuf + (row * ws * 4 + at / SEG) * AP + at % SEG * 4,
                         a + (size_t)min(m - 1, m0 + row) * lda + k0 + at);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            float acc[MT];
#pragma unroll
            for (int r = 0; r < MT; ++r) acc[r] = 0.0f;
            const int mine = min(SEG, k - (seg0 + my_seg) * SEG);            // may be negative
            const unsigned char* wp = wbuf + lane * WP;
            const unsigned char* ap = abuf + (wk * 4 + my_seg) * AP;
#pragma unroll 2
            for (int kk = 0; kk < mine; kk += PER) {
                const uint4 raw = *reinterpret_cast<const uint4*>(wp + kk * sizeof(TW));
                const TW* e = reinterpret_cast<const TW*>(&raw);
#pragma unroll
                for (int q = 0; q < PER; q += 4) {
#pragma unroll
                    for (int r = 0; r < MT; ++r) {
                        const float4 x = *reinterpret_cast<const float4*>(ap + r * ws * 4 * AP + (kk + q) * 4);
                        acc[r] = fmaf(x.x, to_f32(e[q]), acc[r]);
                        acc[r] = fmaf(x.y, to_f32(e[q + 1]), acc[r]);
                        acc[r] = fmaf(x.z, to_f32(e[q + 2]), acc[r]);
                        acc[r] = fmaf(x.w, to_f32(e[q + 3]), acc[r]);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < MT; ++r) part[((wk * 4 + my_seg) * cols + wn * COLS + my_col) * MT + r] = acc[r];
            __syncthreads();
            for (int id = threadIdx.x; id < cols * MT; id += blockDim.x) {
                const int row = m0 + id / cols, col = id % cols;
                if (row >= m) continue;
                float t = total[row * cols + col];
                const int here = min(ws * 4, segs - round * ws * 4);
                for (int s = 0; s < here; ++s) t += part[(s * cols + col) * MT + id / cols];
                total[row * cols + col] = t;
                if (round + 1 == rounds && col0 + col < n) {
                    float* p = c + (size_t)row * ldc + col0 + col;
                    *p = accumulate ? *p + t : t;
                }
            }
            if (m0 + MT < m || round + 1 < rounds) __syncthreads();
        }
    }
}

template <typename TW, int MT>
int launch_rows(const float* a, const TW* w, float* c, int m, int n, int k, int lda, int ldw, int ldc, int accumulate,
                int ws, int wc, size_t smem, cudaStream_t s) {
    static TiPerDevice seen;
    if (seen.first_use()) {
        if (cudaFuncSetAttribute(gemm_rows_kernel<TW, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) !=
            cudaSuccess)
            return ti_check_launch("gemm_simple (shared memory)");
        seen.mark();
    }
    ti_launch_pdl(gemm_rows_kernel<TW, MT>, dim3((n + wc * COLS - 1) / (wc * COLS)), dim3(32 * ws * wc), smem, s, a, w, c,
                  m, n, k, lda, ldw, ldc, accumulate, ws, wc);
    return ti_check_launch("gemm_simple");
}

template <typename T>
bool aligned16(const void* p, int ld) {
    return (uintptr_t)p % 16 == 0 && (size_t)ld * sizeof(T) % 16 == 0;
}

template <typename TA, typename TW, int GROUPS, bool VEC>
int launch_tiles(const TA* a, const TW* w, float* c, int m, int n, int k, int lda, int ldw, int ldc, int accumulate,
                 cudaStream_t s) {
    constexpr int SMEM = GROUPS * BM * BN * 4;
    static TiPerDevice seen;
    if (SMEM > 48 * 1024 && seen.first_use()) {
        if (cudaFuncSetAttribute(gemm_tiled_kernel<TA, TW, GROUPS, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) !=
            cudaSuccess)
            return ti_check_launch("gemm_simple (shared memory)");
        seen.mark();
    }
    ti_launch_pdl(gemm_tiled_kernel<TA, TW, GROUPS, VEC>, dim3((n + BN - 1) / BN, (m + BM - 1) / BM), dim3(GROUP * GROUPS),
                  SMEM, s, a, w, c, m, n, k, lda, ldw, ldc, accumulate);
    return ti_check_launch("gemm_simple");
}

int device_sms() {
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return sms;
}

// Whether the streaming kernel takes a product of up to 32 rows (both kernels give the same bits): by a model of the two
// times in ns, fitted to 2,926 products (8 to 32,768 columns, K of 8 to 12,288, 1 to 32 rows, both types of weights).  The
// streaming kernel passes a round's weights once for every MT rows and holds few blocks on an SM; a tile of 64 rows costs
// the same whatever it holds, and groups of warps beside one another slow each other down.  The choice lies 0.5 % above
// the faster one on average.  us, streaming / tiles: float32 weights, 32 rows of 8 x 8 23 / 2.3, 17 of 128 x 64 21.5 / 4.3,
// 32 of 4,096 x 12,288 1,410 / 342, 8 of 1,024 x 1,024 16 / 29; bfloat16 weights, 17 rows of 12,288 x 1,024 60 / 63, 4 of
// 1,024 x 3,072 9.5 / 91.
bool rows_pay(int m, int n, int k, int w_size, int mt, int ws, int wc, size_t smem) {
    const int sms = device_sms();
    const double kk = k < SEG ? k : SEG, segs = (k + SEG - 1) / SEG;
    const int blocks = (n + wc * COLS - 1) / (wc * COLS), rounds = ((int)segs + 4 * ws - 1) / (4 * ws);
    const int per_sm = (int)(227 * 1024 / (smem + 1024)) < 16 ? (int)(227 * 1024 / (smem + 1024)) : 16;
    const int waves = (blocks + sms * per_sm - 1) / (sms * per_sm), passes = (m + mt - 1) / mt;
    const double rows = 480 + (double)waves * rounds * (640 + passes * (730 + 370 * mt + kk * (6.8 + 3.2 * mt)));
    const double beside = segs < 4 ? segs : 4, alone = (int)(segs + 3) / 4;
    const double shared = segs * ((n + BN - 1) / BN) * 0.43 / sms;
    const double tiles = 1500 + (int)(kk + BK - 1) / BK * 880 * (1 + 0.32 * (beside - 1)) * (alone > shared ? alone : shared);
    return rows < tiles;
}

template <typename TA, typename TW>
int launch(const TA* a, const TW* w, float* c, int m, int n, int k, int lda, int ldw, int ldc, int accumulate,
           cudaStream_t s) {
    // Operands that cannot be read 16 bytes at a time take the tiles, whose loader falls back to single elements.
    const bool aligned = aligned16<TA>(a, lda) && aligned16<TW>(w, ldw);
    if constexpr (sizeof(TA) == 4) {
        if (m <= MAX_ROWS && aligned && k % (16 / (int)sizeof(TW)) == 0 && k % 4 == 0) {
            const int mt = m <= 2 ? m : m <= 4 ? 4 : 8, spans = (k + SPAN - 1) / SPAN;
            const int most = sizeof(TW) == 2 ? 4 : 2;            // shared memory: 33 KB of float32 weights a warp
            const int ws = spans < most ? spans : most;
            // one span: four column groups share the rows of A where there are columns enough for all SMs
            const int wc = ws == 1 && n > 2048 ? 4 : 1;
            const size_t smem = rows_smem<TW>(ws, wc, mt);
            if (rows_pay(m, n, k, sizeof(TW), mt, ws, wc, smem)) {
                if (mt == 1) return launch_rows<TW, 1>(a, w, c, m, n, k, lda, ldw, ldc, accumulate, ws, wc, smem, s);
                if (mt == 2) return launch_rows<TW, 2>(a, w, c, m, n, k, lda, ldw, ldc, accumulate, ws, wc, smem, s);
                if (mt == 4) return launch_rows<TW, 4>(a, w, c, m, n, k, lda, ldw, ldc, accumulate, ws, wc, smem, s);
                return launch_rows<TW, 8>(a, w, c, m, n, k, lda, ldw, ldc, accumulate, ws, wc, smem, s);
            }
        }
    }
    // Groups of warps by segments and tiles; a group without a segment still helps to store a tile, and leaves room for
    // fewer tiles on an SM.  us at one, two and four groups (float32): 2,048 x 32,768 x 256 759 / 896 / 1,323, 100 x 4,096 x
    // 64 5.6 / 5.9 / 5.0, 466 x 1,000 x 1,001 (rows not aligned) 66 / 65 / 37.
    const long long tiles = (long long)((n + BN - 1) / BN) * ((m + BM - 1) / BM);
    const int sms = device_sms();
    const int groups = tiles <= sms || k > 2 * SEG ? 4 : tiles <= 2 * sms || k > SEG ? 2 : 1;
#define TILES(G)                                                                                          \
    (aligned ? launch_tiles<TA, TW, G, true>(a, w, c, m, n, k, lda, ldw, ldc, accumulate, s)               \
             : launch_tiles<TA, TW, G, false>(a, w, c, m, n, k, lda, ldw, ldc, accumulate, s))
    return groups == 4 ? TILES(4) : groups == 2 ? TILES(2) : TILES(1);
#undef TILES
}

}  // namespace

extern "C" int ti_gemm_simple(const void* a, int a_dtype, const void* w, int w_dtype, float* c,
                              int m, int n, int k, int lda, int ldw, int ldc, int accumulate,
                              void* stream) {
    if (m == 0 || n == 0) return 0;
    TI_REQUIRE(k > 0, "gemm: inner size %d", k);
    TI_REQUIRE((m + BM - 1) / BM <= 65535, "gemm: %d rows exceed the grid limit", m);
    cudaStream_t s = (cudaStream_t)stream;
    if (a_dtype == TI_F32 && w_dtype == TI_F32)
        return launch((const float*)a, (const float*)w, c, m, n, k, lda, ldw, ldc, accumulate, s);
    if (a_dtype == TI_F32 && w_dtype == TI_BF16)
        return launch((const float*)a, (const bf16*)w, c, m, n, k, lda, ldw, ldc, accumulate, s);
    if (a_dtype == TI_BF16 && w_dtype == TI_F32)
        return launch((const bf16*)a, (const float*)w, c, m, n, k, lda, ldw, ldc, accumulate, s);
    if (a_dtype == TI_BF16 && w_dtype == TI_BF16)
        return launch((const bf16*)a, (const bf16*)w, c, m, n, k, lda, ldw, ldc, accumulate, s);
    return ti_fail("gemm: dtype codes %d x %d are not float32/bfloat16", a_dtype, w_dtype);
}

TI_TAPED(ti_gemm_simple)
