// Product of float32 rows with bfloat16 weights on the 5th-generation tensor cores, without rounding the rows:
// C[M,N] (+)= A[M,K] * W[N,K]^T.
//
// A float32 number is the sum of three bfloat16 numbers (its 24 significant bits in runs of eight; bfloat16 ends at 2^-133, so
// an element below 2^-109 may be cut short, by less than 2^-133), and a product of two bfloat16 numbers is exact in float32,
// so W times the three parts of A is W times A.  What a tensor core does not do is round its sums to nearest (they are cut
// off, which over a thousand terms adds up to 1e-6 of the result), so sums are made there over 64 terms only and then added,
// rounded to nearest, in registers.  Against 64 bits an element is off by 0.9e-7 of the norm (K = 1,024, normal terms; one
// fused multiply-add per term in runs of 256: 2.9e-7).
//
// One order of summation for every number of rows: a run of 64 terms gives first part + (second + third part); chunk sum =
// its eight runs, ascending, from zero; total = chunk sums, ascending, from zero; C = total or C + total.  A block may have
// all of a tile, some of its chunks or, for few rows, some of its runs (every chunk's or run's sum goes to scratch and the
// tile's last block adds them in that order).
//
// Roles of a block of 512 threads: warp 0 brings W by TMA (128 rows x 64 columns a stage), warp 1 issues the products, W as
// the M side and the three parts of NT tokens beside one another as the N side (a product of 16 columns takes the tensor
// core as long as one of 48: it reads W), warps 4 to 7 read a stage's sums out of tensor memory while the next ones multiply,
// warps 8 to 15 read A, cut it into its parts and write them to shared memory in the swizzle that the products read.  An
// infinite or NaN element of A stays itself; an infinite weight gives NaN where a part is zero, so an element that is NaN is
// made again by multiply-adds.
//
// What bounds it: few rows by the stream of W and, for small W, by the launch, a run's chain (450 to 900 cycles) and the adding
// of the sums that blocks have left (gemm_split_few_kernel); many by the cutting of A and the handing on of stages (466 x 6,144 x
// 1,024: the tensor pipe is busy 16 % of the time, issue slots 40 %, memory 3 %).  us against the multiply-adds of
// gemm_simple.cu: 466 x 6,144 x 1,024 182 -> 50, 466 x 1,024 x 3,072 93 -> 34, 64 x 4,096 x 4,096 120 -> 31, six rows of 6,144 x
// 1,024 12.3 -> 8.8, three rows of 151,936 x 1,024 125 -> 51, of 4,096 x 4,096 34 -> 11.4, of 1,024 x 3,072 9.0 -> 8.9; one and two
// rows of a small matrix still pay for the longer chain (4,096 x 1,024 4.4 and 4.8 -> 6.2 and 6.4, 1,024 x 2,048 4.4 and 5.4 -> 5.5
// and 5.7, 6,144 x 1,024 5.0 and 5.4 -> 6.7 and 6.9, 1,024 x 3,072 4.7 and 5.8 -> 6.4 and 7.0).  With three products of NT columns
// in place of one of 3 NT 466 x 6,144 x 1,024 took 63.
#include "sm100.cuh"
#include "tape.cuh"

namespace {

using namespace sm100;

constexpr int BW = 128, BK = 64, CHUNK = 8;              // CHUNK: runs of BK terms in a chunk
constexpr int THREADS = 512, PRODUCERS = 256;
enum { TI_ERR_TIMEOUT = 2 };

template <int NT> struct Split {
    static constexpr int STAGE_W = BW * BK * 2, STAGE_A = NT * BK * 2, STAGE = STAGE_W + 3 * STAGE_A;
    static constexpr int STAGES = 4;
    static constexpr int TOTAL = STAGES * STAGE, BARS = TOTAL + NT * BW * 4;
    static constexpr int SMEM = BARS + 256 + 1024;
    static constexpr int SUMS = NT == 16 ? 4 : 2;        // stages whose sums lie in tensor memory
    static constexpr unsigned TMEM_COLS = NT == 16 ? 256 : 512;
    static constexpr int BLOCKS = NT == 16 ? 2 : 1;
    static constexpr int TEAMS = NT == 16 ? 2 : 1, AHEAD = NT == 16 ? 4 : 3;
};
static_assert(Split<64>::SMEM <= 227 * 1024 && 2 * (Split<16>::SMEM + 1024) <= 228 * 1024, "shared memory");

__device__ __forceinline__ void drain_sync() { asm volatile("bar.sync 1, 128;\n" ::: "memory"); }

// Eight numbers as three rows of bfloat16: the leading eight bits of what is left, three times.  Infinite and NaN numbers
// (their remainder is NaN) go into the first row alone.
__device__ __forceinline__ void three_parts(const float (&x)[8], uint4 (&parts)[3]) {
    unsigned q[3][4];
    float seen = 0.0f;
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
        const unsigned a = __float_as_uint(x[e]), b = __float_as_uint(x[e + 1]);
        const float ra = x[e] - __uint_as_float(a & 0xffff0000u), rb = x[e + 1] - __uint_as_float(b & 0xffff0000u);
        const unsigned ua = __float_as_uint(ra), ub = __float_as_uint(rb);
        const float sa = ra - __uint_as_float(ua & 0xffff0000u), sb = rb - __uint_as_float(ub & 0xffff0000u);
        q[0][e >> 1] = __byte_perm(a, b, 0x7632);
        q[1][e >> 1] = __byte_perm(ua, ub, 0x7632);
        q[2][e >> 1] = __byte_perm(__float_as_uint(sa), __float_as_uint(sb), 0x7632);
        seen += ra + rb;
    }
    if (seen != seen) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const unsigned b = __float_as_uint(x[e]), keep = e & 1 ? 0x0000ffffu : 0xffff0000u, at = (e & 1) * 16;
            if ((b & 0x7f800000u) != 0x7f800000u) continue;
            q[0][e >> 1] = (q[0][e >> 1] & keep) | ((b << 1) > 0xff000000u ? 0x7fffu : b >> 16) << at;
            q[1][e >> 1] &= keep;
            q[2][e >> 1] &= keep;
        }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) parts[r] = make_uint4(q[r][0], q[r][1], q[r][2], q[r][3]);
}
// Elements of one row of W by multiply-adds: of the tokens t, t + step, ... whose bits are set
__device__ __noinline__ void plain_sums(unsigned tokens, int t, int step, const float* a, int lda, const bf16* w, int k, float* c,
                                        int ldc, int accumulate) {
    for (; tokens; t += step, tokens >>= 1) {
        if (!(tokens & 1)) continue;
        const float* row = a + (size_t)t * lda;
        float sum = 0.0f;
        for (int i = 0; i < k && sum == sum; ++i) sum = fmaf(row[i], __bfloat162float(w[i]), sum);
        float* p = c + (size_t)t * ldc;
        *p = accumulate ? *p + sum : sum;
    }
}

// 16 columns of each of the three parts of a stage's sums (`apart` columns from one another), all on their way at once
__device__ __forceinline__ void tmem_load16(unsigned taddr, float (&v)[16]) {
    unsigned r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        asm volatile("" : "+r"(r[j]));                   // not used before the wait
        v[j] = __uint_as_float(r[j]);
    }
}
__device__ __forceinline__ void tmem_load_cols(unsigned taddr, float (&v)[16]) { tmem_load16(taddr, v); }
__device__ __forceinline__ void tmem_load_cols(unsigned taddr, float (&v)[32]) { tmem_load32(taddr, v); }
__device__ __forceinline__ void load_sums(unsigned taddr, unsigned apart, float (&v)[3][16]) {
    unsigned r[3][16];
#pragma unroll
    for (int i = 0; i < 3; ++i)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
            : "=r"(r[i][0]), "=r"(r[i][1]), "=r"(r[i][2]), "=r"(r[i][3]), "=r"(r[i][4]), "=r"(r[i][5]), "=r"(r[i][6]),
              "=r"(r[i][7]), "=r"(r[i][8]), "=r"(r[i][9]), "=r"(r[i][10]), "=r"(r[i][11]), "=r"(r[i][12]), "=r"(r[i][13]),
              "=r"(r[i][14]), "=r"(r[i][15])
            : "r"(taddr + i * apart));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            asm volatile("" : "+r"(r[i][j]));            // not used before the wait
            v[i][j] = __uint_as_float(r[i][j]);
        }
}

// C of one row of W from the sums that a tile's blocks have left: every STEP-th token from t0 on, TS of them and PS sums asked
// for at a time; chunks in ascending order or, RUNS, the runs of a chunk first.
template <int TS, int PS, bool RUNS, int STEP, typename Out>
__device__ __forceinline__ void add_parts(const float* part, int nt, int parts, int tokens, int t0, Out out) {
    static_assert(!RUNS || PS % CHUNK == 0, "whole chunks of runs");
    for (; t0 < tokens; t0 += STEP * TS) {
        float all[TS];
#pragma unroll
        for (int i = 0; i < TS; ++i) all[i] = 0.0f;
        for (int p0 = 0; p0 < parts; p0 += PS) {
            float got[PS][TS], chunk[TS];
#pragma unroll
            for (int p = 0; p < PS; ++p)
#pragma unroll
                for (int i = 0; i < TS; ++i)
                    got[p][i] = p0 + p < parts && t0 + STEP * i < tokens ? __ldcg(part + ((size_t)(p0 + p) * nt + t0 + STEP * i) * BW) : 0.0f;
#pragma unroll
            for (int p = 0; p < PS; ++p) {
                if (p0 + p >= parts) continue;
                const bool first = !RUNS || p % CHUNK == 0, last = !RUNS || p % CHUNK == CHUNK - 1 || p0 + p + 1 == parts;
#pragma unroll
                for (int i = 0; i < TS; ++i) {
                    chunk[i] = (first ? 0.0f : chunk[i]) + got[p][i];
                    if (last) all[i] += chunk[i];
                }
            }
        }
#pragma unroll
        for (int i = 0; i < TS; ++i)
            if (t0 + STEP * i < tokens) out(t0 + STEP * i, all[i]);
    }
}

template <int NT>
__global__ void __launch_bounds__(THREADS, Split<NT>::BLOCKS)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const float* a, const bf16* __restrict__ w, float* c, float* ws,
                  int* __restrict__ tickets, int m, int n, int k, int lda, int ldw, int ldc, int accumulate, int vec,
                  int* __restrict__ status) {
    using T = Split<NT>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float* total = reinterpret_cast<float*>(smem + T::TOTAL);                // [token][row of W]
    unsigned long long* bars = (unsigned long long*)(smem + T::BARS);
    unsigned long long* full = bars;                     // [STAGES] W and the parts of A are there
    unsigned long long* empty = bars + T::STAGES;        // [STAGES] the products have read them
    unsigned long long* sum_full = bars + 2 * T::STAGES;         // [SUMS] a stage's sums are in tensor memory
    unsigned long long* sum_empty = sum_full + T::SUMS;          // [SUMS] and have been read
    unsigned* tmem_slot = (unsigned*)(sum_empty + T::SUMS);
    int* ticket_slot = (int*)(tmem_slot + 1);            // whether this block finishes the tile
    int* failed_slot = ticket_slot + 1;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * NT, n0 = blockIdx.y * BW;
    // the block's stages: whole chunks of them
    const int stages_all = (k + BK - 1) / BK, splits = gridDim.z;
    const int parts = (stages_all + CHUNK - 1) / CHUNK;  // sums that a tile's blocks leave, if there are several
    const int kb_lo = (int)((long long)parts * blockIdx.z / splits) * CHUNK;
    const int kb_hi = min(stages_all, (int)((long long)parts * (blockIdx.z + 1) / splits) * CHUNK);
    auto stage_w = [&](int s) { return smem + s * T::STAGE; };
    auto stage_a = [&](int s, int part) { return smem + s * T::STAGE + T::STAGE_W + part * T::STAGE_A; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < T::STAGES; ++s) { mbar_init(&full[s], 1 + PRODUCERS / 32 / T::TEAMS); mbar_init(&empty[s], 1); }
        for (int b = 0; b < T::SUMS; ++b) { mbar_init(&sum_full[b], 1); mbar_init(&sum_empty[b], 4); }
        *ticket_slot = splits == 1;
        *failed_slot = 0;
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, T::TMEM_COLS);
    pdl_launch();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = *tmem_slot;

    const int tile = blockIdx.y * gridDim.x + blockIdx.x, tokens = min(NT, m - m0);
    bool ok = true;
    if (warp == 0) {
        if (lane == 0) {                                 // the weights do not depend on the kernel before this one
            for (int kb = kb_lo, it = 0; kb < kb_hi && ok; ++kb, ++it) {
                const int s = it % T::STAGES;
                ok = mbar_wait(&empty[s], ((it / T::STAGES) & 1) ^ 1);
                if (!ok) break;
                mbar_expect_tx(&full[s], T::STAGE_W);
                tma_load_2d(stage_w(s), &map_w, &full[s], kb * BK, n0);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const unsigned idesc = umma_idesc(BW, 3 * NT);
            const unsigned long long dw0 = umma_desc(stage_w(0)), da0 = umma_desc(stage_a(0, 0));
            for (int kb = kb_lo, it = 0; kb < kb_hi && ok; ++kb, ++it) {
                const int s = it % T::STAGES, buf = it % T::SUMS;
                ok = mbar_wait(&sum_empty[buf], ((it / T::SUMS) & 1) ^ 1);
                if (ok) ok = mbar_wait(&full[s], (it / T::STAGES) & 1);
                if (!ok) break;
                tc_fence_after();
                const unsigned long long dw = dw0 + (unsigned long long)(s * (T::STAGE >> 4));
                const unsigned long long da = da0 + (unsigned long long)(s * (T::STAGE >> 4));
#pragma unroll
                for (int kk = 0; kk < BK / 16; ++kk)
                    umma_bf16(tmem_base + buf * 3 * NT, dw + (unsigned long long)(kk * 2), da + (unsigned long long)(kk * 2),
                              idesc, kk != 0);
                umma_commit(&empty[s]);
                umma_commit(&sum_full[buf]);
            }
        }
    } else if (warp >= 8) {
        // A piece: eight neighbouring columns of a token, 16 bytes of each part.  TEAMS groups of warps take the stages in
        // turn, and every thread has its pieces of the next AHEAD stages of its own on their way: a load from L2 takes
        // longer than a stage's products.
        constexpr int TEAM = PRODUCERS / T::TEAMS, PER = NT * 8 / TEAM;
        static_assert(NT * 8 % TEAM == 0, "a stage's pieces over a team");
        const int team = (threadIdx.x - (THREADS - PRODUCERS)) / TEAM, p0 = (threadIdx.x - (THREADS - PRODUCERS)) % TEAM;
        const int stages = kb_hi - kb_lo;
        float v[T::AHEAD][PER][8];
        auto fetch = [&](int it, float (&v)[PER][8]) {
            if (it >= stages) return;
            const int kb = kb_lo + it;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int p = p0 + i * TEAM, row = m0 + p / 8, col = kb * BK + p % 8 * 8;
                const float* src = a + (size_t)row * lda + col;
                if (row < m && vec && col + 8 <= k) {
                    const float4 x = *reinterpret_cast<const float4*>(src), y = *reinterpret_cast<const float4*>(src + 4);
                    v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w;
                    v[i][4] = y.x; v[i][5] = y.y; v[i][6] = y.z; v[i][7] = y.w;
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[i][e] = row < m && col + e < k ? src[e] : 0.0f;
                }
            }
        };
        pdl_wait();
#pragma unroll
        for (int d = 0; d < T::AHEAD; ++d) fetch(team + d * T::TEAMS, v[d]);
        for (int first = team; first < stages && ok; first += T::AHEAD * T::TEAMS) {
#pragma unroll
            for (int d = 0; d < T::AHEAD; ++d) {
                const int it = first + d * T::TEAMS, s = it % T::STAGES;
                if (it >= stages || !ok) break;
                ok = __all_sync(0xffffffffu, mbar_wait(&empty[s], ((it / T::STAGES) & 1) ^ 1));
                if (!ok) break;
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int p = p0 + i * TEAM, row = p / 8, at = row * 128 + ((p % 8) ^ (row & 7)) * 16;
                    uint4 parts[3];
                    three_parts(v[d][i], parts);
#pragma unroll
                    for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(stage_a(s, q) + at) = parts[q];
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
                fetch(it + T::AHEAD * T::TEAMS, v[d]);
            }
        }
    } else if (warp >= 4) {
        const int row = (warp & 3) * 32 + lane;
        const unsigned lane_addr = (unsigned)((warp & 3) * 32) << 16;
        pdl_wait();                                      // the scratch and the tickets belong to the chain
        float acc[NT];
        for (int kb = kb_lo, it = 0; kb < kb_hi; ++kb, ++it) {
            const int buf = it % T::SUMS;
            const bool first = kb % CHUNK == 0, last = kb % CHUNK == CHUNK - 1 || kb + 1 == stages_all;
            ok = __all_sync(0xffffffffu, mbar_wait(&sum_full[buf], (it / T::SUMS) & 1));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int t0 = 0; t0 < NT; t0 += 16) {
                float v[3][16];
                load_sums(tmem_base + lane_addr + buf * 3 * NT + t0, NT, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[t0 + i] = (first ? 0.0f : acc[t0 + i]) + (v[0][i] + (v[1][i] + v[2][i]));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sum_empty[buf]);
            if (!last) continue;
            if (splits > 1) {
                float* part = ws + ((size_t)tile * parts + kb / CHUNK) * NT * BW + row;
#pragma unroll
                for (int t = 0; t < NT; ++t)
                    if (t < tokens) part[t * BW] = acc[t];
            } else {
                const bool one = kb < CHUNK;             // the first chunk
#pragma unroll
                for (int t = 0; t < NT; ++t) total[t * BW + row] = (one ? 0.0f : total[t * BW + row]) + acc[t];
            }
        }
        if (splits > 1) {
            // the tile is complete when all its blocks have stored their sums; the last one adds them
            __threadfence();
            drain_sync();
            if (threadIdx.x == 128) {
                const bool finish = atomicAdd(&tickets[tile], 1) == splits - 1;
                if (finish) tickets[tile] = 0;
                *ticket_slot = finish;
                __threadfence();
            }
        }
    }
    if (!ok) *failed_slot = 1;
    __syncthreads();
    if (*ticket_slot && !*failed_slot) {                 // four threads a row of W
        pdl_wait();                                      // C belongs to the chain
        const int row = threadIdx.x & (BW - 1), t0 = threadIdx.x / BW, n_row = n0 + row;
        unsigned again = 0;                              // tokens t0, t0 + 4, ... whose sum is NaN
        auto out = [&](int t, float v) {
            float* p = c + (size_t)(m0 + t) * ldc + n_row;
            if (v != v) again |= 1u << (t >> 2);
            if (!accumulate) *p = v;
            else if (v == v) *p += v;
        };
        const float* part = ws + (size_t)tile * parts * NT * BW + row;
        if (n_row >= n) {
        } else if (splits == 1) {
            for (int t = t0; t < tokens; t += 4) out(t, total[t * BW + row]);
        } else if (tokens <= 4) {
            add_parts<1, 16, false, 4>(part, NT, parts, tokens, t0, out);
        } else {
            add_parts<4, 4, false, 4>(part, NT, parts, tokens, t0, out);
        }
        if (again)
            plain_sums(again, t0, 4, a + (size_t)m0 * lda, lda, w + (size_t)n_row * ldw, k, c + (size_t)m0 * ldc + n_row, ldc,
                       accumulate);
    }
    if (!ok) atomicCAS(status, 0, TI_ERR_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, T::TMEM_COLS);
    }
}

// Up to eight rows.  The three parts of four or eight tokens lie beside one another in the columns of one product, a warp cuts a
// stage's rows, and a block of 256 threads is small enough that the next launch's blocks find a place beside it and have their
// weights on the way while this one ends.  us at 1, 4 and 8 rows, the kernel above / this: 4,096 x 1,024 7.1 / 6.2, 7.8 / 6.7 and
// 10.9 / 8.0, 1,024 x 2,048 8.8 / 5.5, 9.2 / 7.1 and 10.3 / 8.8, 6,144 x 1,024 7.8 / 6.8, 8.6 / 7.3 and 10.8 / 8.9, 1,024 x 3,072
// 9.2 / 6.3, 9.7 / 9.0 and 11.8 / 11.3, 151,936 x 1,024 at 1, 4 and 6 rows 63.6 / 50.2, 64.5 / 51.1 and 65.7 / 55.8.  A cluster's
// blocks that exchange their sums through shared memory start later: 4,096 x 1,024 7.8, 1,024 x 2,048 6.8 at one row.
constexpr int FEW = 8, FEW_THREADS = 256;
template <int NT> struct Few {                           // NT: tokens, 4 or 8
    static constexpr int COLS = NT == 4 ? 16 : 32;       // their parts, and columns without a token
    static constexpr int STAGE = BW * BK * 2 + COLS * BK * 2, STAGES = NT == 4 ? 4 : 3, SUMS = 4, CUTTERS = 2;
    static constexpr int PIECES = NT / 4, AHEAD = 4 / PIECES;
    static constexpr int BARS = STAGES * STAGE, SMEM = BARS + 256 + 1024;
    static constexpr unsigned TMEM_COLS = SUMS * COLS;
};
static_assert(3 * (Few<4>::SMEM + 1024) <= 228 * 1024 && 3 * (Few<8>::SMEM + 1024) <= 228 * 1024, "shared memory");

template <int NT>
__global__ void __launch_bounds__(FEW_THREADS, 3)
gemm_split_few_kernel(const __grid_constant__ CUtensorMap map_w, const float* a, const bf16* __restrict__ w, float* c, float* ws,
                      int* __restrict__ tickets, int m, int n, int k, int lda, int ldw, int ldc, int accumulate, int vec, int fine,
                      int* __restrict__ status) {
    using T = Few<NT>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned long long* bars = (unsigned long long*)(smem + T::BARS);
    unsigned long long *full = bars, *empty = bars + T::STAGES, *sum_full = bars + 2 * T::STAGES, *sum_empty = sum_full + T::SUMS;
    unsigned* tmem_slot = (unsigned*)(sum_empty + T::SUMS);
    int* ticket_slot = (int*)(tmem_slot + 1);
    int* failed_slot = ticket_slot + 1;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n0 = blockIdx.x * BW;
    const int stages_all = (k + BK - 1) / BK, splits = gridDim.y, per = fine ? 1 : CHUNK;
    const int parts = (stages_all + per - 1) / per;
    const int kb_lo = (int)((long long)parts * blockIdx.y / splits) * per;
    const int kb_hi = min(stages_all, (int)((long long)parts * (blockIdx.y + 1) / splits) * per);
    auto stage_w = [&](int s) { return smem + s * T::STAGE; };
    auto stage_a = [&](int s) { return smem + s * T::STAGE + BW * BK * 2; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < T::STAGES; ++s) { mbar_init(&full[s], 2); mbar_init(&empty[s], 1); }
        for (int b = 0; b < T::SUMS; ++b) { mbar_init(&sum_full[b], 1); mbar_init(&sum_empty[b], 4); }
        *failed_slot = 0;
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, T::TMEM_COLS);
    for (int i = threadIdx.x; i < T::STAGES * T::COLS * 8; i += FEW_THREADS)         // rows without a token stay zeros
        *reinterpret_cast<uint4*>(stage_a(i / (T::COLS * 8)) + i % (T::COLS * 8) * 16) = make_uint4(0u, 0u, 0u, 0u);
    fence_async_smem();
    pdl_launch();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = *tmem_slot;
    const int stages = kb_hi - kb_lo;

    bool ok = true;
    float all[NT] = {};                                 // one block a tile: the total
    if (warp == 0) {
        if (lane == 0) {                                 // the weights do not depend on the kernel before this one
            for (int it = 0; it < stages && ok; ++it) {
                const int s = it % T::STAGES;
                ok = mbar_wait(&empty[s], ((it / T::STAGES) & 1) ^ 1);
                if (!ok) break;
                mbar_expect_tx(&full[s], BW * BK * 2);
                tma_load_2d(stage_w(s), &map_w, &full[s], (kb_lo + it) * BK, n0);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const unsigned idesc = umma_idesc(BW, T::COLS);
            const unsigned long long dw0 = umma_desc(stage_w(0)), da0 = umma_desc(stage_a(0));
            for (int it = 0; it < stages && ok; ++it) {
                const int s = it % T::STAGES, buf = it % T::SUMS;
                ok = mbar_wait(&sum_empty[buf], ((it / T::SUMS) & 1) ^ 1);
                if (ok) ok = mbar_wait(&full[s], (it / T::STAGES) & 1);
                if (!ok) break;
                tc_fence_after();
                const unsigned long long step = (unsigned long long)(s * (T::STAGE >> 4));
#pragma unroll
                for (int kk = 0; kk < BK / 16; ++kk)
                    umma_bf16(tmem_base + buf * T::COLS, dw0 + step + (unsigned long long)(kk * 2), da0 + step + (unsigned long long)(kk * 2),
                              idesc, kk != 0);
                umma_commit(&empty[s]);
                umma_commit(&sum_full[buf]);
            }
        }
    } else if (warp < 4) {
        // a lane has eight neighbouring columns of a token, or of two; the two warps take the stages in turn
        const int piece = lane & 7, team = warp - 2;
        float v[T::AHEAD][T::PIECES][8];
        auto fetch = [&](int it, float (&v)[T::PIECES][8]) {
            const int col = (kb_lo + it) * BK + piece * 8;
#pragma unroll
            for (int i = 0; i < T::PIECES; ++i) {
                const int t = (lane >> 3) + 4 * i;
                if (it >= stages || t >= m) continue;
                const float* row = a + (size_t)t * lda;
                if (vec && col + 8 <= k) {
                    const float4 x = *reinterpret_cast<const float4*>(row + col), y = *reinterpret_cast<const float4*>(row + col + 4);
                    v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w;
                    v[i][4] = y.x; v[i][5] = y.y; v[i][6] = y.z; v[i][7] = y.w;
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[i][e] = col + e < k ? row[col + e] : 0.0f;
                }
            }
        };
        pdl_wait();
#pragma unroll
        for (int d = 0; d < T::AHEAD; ++d) fetch(team + d * T::CUTTERS, v[d]);
        for (int first = team; first < stages && ok; first += T::AHEAD * T::CUTTERS) {
#pragma unroll
            for (int d = 0; d < T::AHEAD; ++d) {
                const int it = first + d * T::CUTTERS, s = it % T::STAGES;
                if (it >= stages || !ok) break;
                ok = __all_sync(0xffffffffu, mbar_wait(&empty[s], ((it / T::STAGES) & 1) ^ 1));
                if (!ok) break;
#pragma unroll
                for (int i = 0; i < T::PIECES; ++i) {
                    const int t = (lane >> 3) + 4 * i;
                    if (t >= m) continue;
                    uint4 part[3];
                    three_parts(v[d][i], part);
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        const int at = q * NT + t;
                        *reinterpret_cast<uint4*>(stage_a(s) + at * 128 + (piece ^ (at & 7)) * 16) = part[q];
                    }
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
                fetch(it + T::AHEAD * T::CUTTERS, v[d]);
            }
        }
    } else {
        const int row = (warp & 3) * 32 + lane;
        const unsigned lane_addr = (unsigned)((warp & 3) * 32) << 16;
        pdl_wait();                                       // the scratch and the tickets belong to the chain
        float acc[NT];
        for (int kb = kb_lo, it = 0; kb < kb_hi; ++kb, ++it) {
            const int buf = it % T::SUMS;
            const bool first = kb % CHUNK == 0 || fine, last = kb % CHUNK == CHUNK - 1 || kb + 1 == stages_all || fine;
            ok = __all_sync(0xffffffffu, mbar_wait(&sum_full[buf], (it / T::SUMS) & 1));
            if (!ok) break;
            tc_fence_after();
            float v[T::COLS];
            tmem_load_cols(tmem_base + lane_addr + buf * T::COLS, v);
#pragma unroll
            for (int t = 0; t < NT; ++t)
                acc[t] = (first ? 0.0f : acc[t]) + (v[t] + (v[NT + t] + v[2 * NT + t]));
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sum_empty[buf]);
            if (!last) continue;
            float* part = ws + ((size_t)blockIdx.x * parts + kb / per) * NT * BW + row;
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                if (splits > 1) { if (t < m) part[t * BW] = acc[t]; }
                else all[t] += acc[t];
            }
        }
        if (splits > 1) {
            // the tile is complete when all its blocks have stored their sums; the last one adds them
            drain_sync();
            if (threadIdx.x == 128) {
                __threadfence();
                const bool finish = atomicAdd(&tickets[blockIdx.x], 1) == splits - 1;
                if (finish) tickets[blockIdx.x] = 0;
                *ticket_slot = finish;
                __threadfence();
            }
        }
    }
    if (!ok) *failed_slot = 1;
    __syncthreads();
    if (!*failed_slot && (splits == 1 ? warp >= 4 : *ticket_slot)) {
        pdl_wait();                                       // C belongs to the chain
        const int row = threadIdx.x & (BW - 1), t0 = splits == 1 ? 0 : threadIdx.x / BW;
        unsigned again = 0;                               // tokens whose sum is NaN
        auto store = [&](int t, float v) {
            float* p = c + (size_t)t * ldc + n0 + row;
            *p = accumulate ? *p + v : v;
        };
        auto out = [&](int t, float v) {
            if (v != v) again |= 1u << t;
            else store(t, v);
        };
        const float* part = ws + (size_t)blockIdx.x * parts * NT * BW + row;
        if (n0 + row >= n) {
        } else if (splits == 1) {
#pragma unroll
            for (int t = 0; t < NT; ++t)
                if (t < m) out(t, all[t]);
        } else if (fine && m <= 2) {
            add_parts<1, 32, true, 2>(part, NT, parts, m, t0, out);
        } else if (fine) {
            add_parts<NT / 2, 64 / NT, true, 2>(part, NT, parts, m, t0, out);
        } else {
            add_parts<NT / 2, 32 / NT, false, 2>(part, NT, parts, m, t0, out);
        }
        if (again) plain_sums(again, 0, 1, a, lda, w + (size_t)(n0 + row) * ldw, k, c + n0 + row, ldc, accumulate);
    }
    if (!ok) atomicCAS(status, 0, TI_ERR_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, T::TMEM_COLS);
    }
}

int few_tile(int m) { return m <= 4 ? 4 : 8; }
int token_tile(int m) { return m <= 16 ? 16 : 64; }

// How a tile's K is shared.  Up to eight rows: some two blocks an SM, a run or more each or, where a tile gets fewer blocks than
// twice its chunks, whole chunks, whose sums are fewer to add (us at 1 and 4 rows, runs / chunks: 1,024 x 3,072 6.4 / 7.9 and
// 8.7 / 8.7, 4,096 x 4,096 10.8 / 11.1 and 13.6 / 11.5); four runs are not shared (256 x 256 4.4 / 3.5).  More rows: as many
// blocks as fill the SMs once (twice where two fit on one), a chunk or more each.
struct Cut { int splits, fine; long long floats; int tickets; };
Cut choose_cut(int m, int n, int k) {
    int device = 0, sms = 148;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const bool few = m <= FEW;
    const int nt = few ? few_tile(m) : token_tile(m), stages = (k + BK - 1) / BK, chunks = (stages + CHUNK - 1) / CHUNK;
    const long long tiles = (long long)((m + nt - 1) / nt) * ((n + BW - 1) / BW), room = (long long)sms * (nt <= 16 ? 2 : 1);
    const long long s = room / tiles;
    Cut cut;
    cut.fine = few && s >= 2 * chunks && stages > 4;
    const int most = cut.fine ? stages : chunks;
    cut.splits = s < 1 ? 1 : s > most ? most : (int)s;
    cut.floats = cut.splits > 1 ? tiles * most * nt * BW : 0;
    cut.tickets = cut.splits > 1 ? (int)tiles : 0;
    return cut;
}

template <int NT>
int launch(const CUtensorMap& map_w, const float* a, const bf16* w, float* c, float* ws, int* tickets, int m, int n, int k, int lda,
           int ldw, int ldc, int accumulate, const Cut& cut, int* status, cudaStream_t s) {
    static TiPerDevice configured;
    if (configured.first_use()) {
        cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Split<NT>::SMEM);
        if (e != cudaSuccess) return ti_fail("gemm_split: %s", cudaGetErrorString(e));
        configured.mark();
    }
    const int vec = (uintptr_t)a % 16 == 0 && lda % 4 == 0;
    const dim3 grid((m + NT - 1) / NT, (n + BW - 1) / BW, cut.splits);
    TI_REQUIRE(grid.y <= 65535, "gemm_split: %d rows of weights exceed the grid limit", n);
    ti_launch_pdl(gemm_split_kernel<NT>, grid, dim3(THREADS), Split<NT>::SMEM, s, map_w, a, w, c, ws, tickets, m, n, k, lda,
                  ldw, ldc, accumulate, vec, status);
    return ti_check_launch("gemm_split");
}

template <int NT>
int launch_few(const CUtensorMap& map_w, const float* a, const bf16* w, float* c, float* ws, int* tickets, int m, int n, int k,
               int lda, int ldw, int ldc, int accumulate, const Cut& cut, int* status, cudaStream_t s) {
    static TiPerDevice configured;
    if (configured.first_use()) {
        cudaError_t e = cudaFuncSetAttribute(gemm_split_few_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Few<NT>::SMEM);
        if (e != cudaSuccess) return ti_fail("gemm_split: %s", cudaGetErrorString(e));
        configured.mark();
    }
    const int vec = (uintptr_t)a % 16 == 0 && lda % 4 == 0;
    ti_launch_pdl(gemm_split_few_kernel<NT>, dim3((n + BW - 1) / BW, cut.splits), dim3(FEW_THREADS), Few<NT>::SMEM, s, map_w, a, w, c,
                  ws, tickets, m, n, k, lda, ldw, ldc, accumulate, vec, cut.fine, status);
    return ti_check_launch("gemm_split");
}

}  // namespace

// Float32 values of scratch and tickets (zero before a launch and after it) that ti_gemm_split wants.
extern "C" int ti_gemm_split_scratch(int m, int n, int k, long long* floats, int* tickets) {
    const Cut cut = choose_cut(m, n, k);
    *floats = cut.floats;
    *tickets = cut.tickets;
    return 0;
}

// a: float32 [m, k] (rows lda apart), w: bfloat16 [n, k] (16-byte aligned, ldw a multiple of 8), c: float32 [m, n]
extern "C" int ti_gemm_split(const float* a, const void* w, float* c, int m, int n, int k, int lda, int ldw, int ldc,
                             int accumulate, float* ws, int* tickets, int* status, void* stream) {
    if (m == 0 || n == 0) return 0;
    TI_REQUIRE(k > 0, "gemm_split: inner size %d", k);
    TI_REQUIRE((uintptr_t)w % 16 == 0 && ldw % 8 == 0, "gemm_split: weights must be 16-byte aligned with rows a multiple of "
               "8 elements apart");
    const Cut cut = choose_cut(m, n, k);
    TI_REQUIRE(cut.splits == 1 || (ws != nullptr && tickets != nullptr), "gemm_split: %d blocks a tile need scratch", cut.splits);
    CUtensorMap map_w;
    if (int rc = make_map_bf16(&map_w, w, n, k, ldw, BW, "gemm_split")) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    auto run = m <= 4 ? launch_few<4> : m <= FEW ? launch_few<8> : token_tile(m) == 16 ? launch<16> : launch<64>;
    return run(map_w, a, (const bf16*)w, c, ws, tickets, m, n, k, lda, ldw, ldc, accumulate, cut, status, s);
}

TI_TAPED(ti_gemm_split)
