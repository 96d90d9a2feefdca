// The three four-step passes of a column map on the tensor cores, in one
// persistent launch over column chunks.
//
// A map NTT_S(f(i) * INTT_S(column)) with S = N1 * N2 and f(k1 + N1 k2) = u(k1) v(k2)
// (the extension's twist g^i / S, a coset's, the decoder's h^(+-i) / S) is, with input
// index i = N2 i1 + i2 and output index m = m1 + N2 m2,
//   A  y[k1][i2] = w_S^(-i2 k1) * sum_i1 w_N1^(-i1 k1) x[N2 i1 + i2]
//   M  z[k1][m1] = u(k1) w_S^(k1 m1) * sum_i2 C[m1 - i2] y[k1][i2]
//   B  out[m1 + N2 m2] = sum_k1 w_N1^(k1 m2) z[k1][m1]
// with the fixed circulant C[d] = sum_k2 v(k2) w_N2^(k2 d): the INTT's second half,
// the factor and the NTT's first half are one N2 x N2 matrix. Each pass is a matrix
// of 32 or 64 points times the columns of a tile, then one factor per output: an
// integer product on the tensor cores over the values' bytes (tcgen05.cuh), whose
// four sums per output are reduced to one signed word (tp_fold) and multiplied by the
// factor (tp_mul): 9 integer instructions per output and pass where the butterflies of 64
// points take about 21, and 6 in pass B, which has no factor in an extension.
//
// Work: a tile is 8192 values of one column block (one i2, k1 or m1): 32 points x 256
// adjacent columns or 64 points x 128, so a tile's factors are the same for all its
// columns and its rows are segments of 512 or 1024 bytes. The passes run chunk by chunk
// of CW columns; the intermediate matrix of a chunk lives in a ring of chunk slots that
// stays in L2. Work items are (chunk, pass, tile); round r holds pass A of chunk r, M of
// chunk r - depth and B of chunk r - 2 depth, dealt in that order by a global counter. M
// waits for all A tiles of its chunk, B for all M tiles, A for the B tiles that read the
// slot it overwrites: only items dealt earlier, to CTAs that are running them, so the
// launch cannot deadlock whatever the number of resident CTAs. Every wait is bounded.
//
// A CTA (one per SM) is a pipeline of roles:
//   dealer    draws items, waits for what they depend on
//   loader    one thread: TMA of a tile's two halves (32 rows x 128 columns each), its factor row
//   copier    one thread: the even rows leave by TMA straight from there
//   4 warps   move a tile into tensor memory (lane = column; a value's 4 bytes are one
//             32-bit column: no transposition)
//   product   one thread: operand in tensor memory times the matrix in shared memory, as
//             two sets of 32 outputs x 128 columns
//   2 x 8 warps  read a set's sums back, reduce, store (lane = column: 128-byte stores)
//   signal    one thread: publishes finished tiles
//
// What bounds it: the card's power limit. In a burst (1.9 GHz) a 4096 square takes 9.1 ms
// and the instruction issue of the read-back is nearest its limit; under the 1000 W cap
// the SM clock settles near 1.5 GHz and it takes 9.6 .. 9.9 ms, 2.65 TB/s of the 12 bytes a
// value that must move (the butterfly passes: 12.6 ms, the single pass 20.7). 2048: 2.26 ..
// 2.30 ms against 3.29. A tile's products take 1024 of its about 3000 cycles (64 points), its
// HBM traffic is the 12 bytes a value plus 27% for ring lines that leave L2.
#pragma once
#include "dft.cuh"
#include "tcgen05.cuh"

namespace zb {

struct TensorArgs {
    uint64_t in_pitch, copy_pitch;  // u32 between rows (host side)
    const uint32_t* in;    // pass A input: row r (< in_rows, others are zeros) at in + r * in_pitch
    uint32_t* copy;        // copy of input row r (zeros past in_rows) for r < copy_rows, or nullptr
    uint32_t in_rows, copy_rows;
    const uint2* pre;      // PRE: factor of input row N2 i1 + i2 (Shoup pair) at [i2][i1]
    // output m (< out_rows) at out + (m >> out_shift) * out_pitch; out_shift 1: only even m
    uint32_t* out;
    uint64_t out_pitch;
    uint32_t out_rows, out_shift;  // out_shift: the kernel's OSH (host side)
    uint32_t cols;         // columns of the matrix
    // tables: byte operands of the three matrices (B shares A's: w^-1 with its
    // rows mirrored) and the factors (w, s) as [column block][output]
    const uint4* mat_a;
    const uint4* mat_m;
    const int2* fac_a;
    const int2* fac_m;
    const int2* fac_b;  // outputs in matrix row order, or nullptr: no factors
    uint32_t* ring;        // slots of S x CW u32
    uint32_t slots;
    uint32_t nchunks, depth;
    uint32_t* counters;  // [0] items drawn; then tiles done per chunk: A, M, B
    uint32_t wait_extra;  // fault injection: added to every count waited for
    int* err;
};
// Tensor maps as [i1][i2][column], boxes of 32 x 1 x 128. Rows r = N2 i1 + i2 below a
// limit are no box of that shape: column blocks i2 < limit % N2 have one row i1 more, so
// each matrix has two maps, [1] for those.
struct TensorMaps {
    CUtensorMap in[2], copy[2];
    CUtensorMap ring_m, ring_b;  // the ring as [slot, k1][i2][column]: boxes 1 x 32 x 128 and 32 x 1 x 128
};

constexpr int TP_BOX = 128;   // columns of a half tile's box
constexpr int TP_EPI = 16;    // read-back warps, a group of 8 for each set of a tile
constexpr int TP_W_CONV = TP_EPI, TP_W_DEAL = TP_W_CONV + 4, TP_W_LOAD = TP_W_DEAL + 1, TP_W_MMA = TP_W_LOAD + 1,
              TP_W_SIG = TP_W_MMA + 1, TP_W_COPY = TP_W_SIG + 1;
constexpr int TP_THREADS = (TP_W_COPY + 1) * 32;
#ifndef ZB_TP_RUN
#define ZB_TP_RUN 2
#endif
#ifndef ZB_TP_NR
#define ZB_TP_NR 8
#endif
constexpr int TP_RUN = ZB_TP_RUN;  // items drawn together, one lane each
constexpr int TP_QN = TP_RUN;      // dealt tiles waiting for the loader
constexpr int TP_RF = 8;           // tiles between the loader and the signal
constexpr uint32_t TP_RAW = 32 * TP_BOX * 4;  // bytes of a half tile

template <int L1, int L2>
struct TPassGeom {
    static constexpr int N1 = 1 << L1, N2 = 1 << L2, NMAX = N1 > N2 ? N1 : N2;
    static constexpr int TC1 = 8192 / N1, TC2 = 8192 / N2;     // columns of a tile of A and B, of M
    static constexpr int CW = TC1 > TC2 ? TC1 : TC2;           // columns of a chunk
    static constexpr uint32_t MAT_A = 16u * N1 * N1, MAT_M = 16u * N2 * N2;  // bytes
    // tensor memory: three sets of sums (32 outputs x 4 planes), two operands (64 columns)
    static constexpr int NB = 3, NA = 2;
    static constexpr uint32_t DCOLS = 128, ACOL = NB * DCOLS;
    static constexpr uint32_t OFF_M = MAT_A;
    static constexpr uint32_t OFF_F = OFF_M + MAT_M;
    static constexpr uint32_t OFF_P = OFF_F + TP_RF * NMAX * 8;  // PRE: the input factors of a tile of A
    static constexpr uint32_t OFF_T = OFF_P + TP_RF * N1 * 8;
    static constexpr uint32_t OFF_BAR = OFF_T + (TP_RF + TP_QN) * 32;
    static constexpr uint32_t OFF_R = (OFF_BAR + 512 + 127) / 128 * 128;
    static constexpr int NR_FIT = (int)((232448 - OFF_R) / TP_RAW);
    static constexpr int NR = NR_FIT < ZB_TP_NR ? NR_FIT : ZB_TP_NR;  // half tiles the loads land in
    static constexpr uint32_t SMEM = OFF_R + NR * TP_RAW;
    static_assert(NR >= 3 && NR <= TP_RF && SMEM <= 232448, "shared memory per CTA");
    static_assert(NMAX <= 64 && N1 >= 32 && N2 >= 32, "points of a pass");
    static_assert((2 * NR + 2 * NA + 2 * NB + 2 * TP_RF + 2 * TP_QN + 1) * 8 + 16 <= 512, "barriers");
    // tiles of a chunk's passes
    static constexpr uint32_t TA = N2 * (CW / TC1), TM = N1 * (CW / TC2);
    // ring: u32 of a slot, of a row, rows as k1 N2 + i2
    static constexpr uint32_t SLOT = (uint32_t)N1 * N2 * CW;
};

struct TTile {  // a tile: pass (or an end mark), column block, its first column in the matrix, ring slot
    uint32_t ph, j, x, slot;
    uint32_t* dst;    // where output 0 of its first column goes (pass B: output index S, see there)
    const int2* fac;  // its factor row, or nullptr
};
constexpr uint32_t TP_END = 8;

// The reduction of an output's sums, and the product with its factor (w, s), s the rounded w
// 2^32 / p of the centered w. (Both in one step, with a second factor 2^16 w, takes two
// instructions less but 16 bytes of factor an output, and the factors' loads cost more.)
//   y = (Y0 + 2^16 Y1) mod p, centered, Y0 = a0 + 2^8 a1, Y1 = a2 + 2^8 a3: y = Y0 + 2^16 Y1 -
//       q p with q the rounded Y1 2^16 / p, off by less than 1/2 + |Y1| / 2^33, so |y| < p / 2 +
//       |Y1| / 4 + |Y0| <= p for |Y0|, |Y1| <= TP_SUM_MAX. The host checks that of its matrices
//       for any input bytes (tensorpass.cu).
//   r = y w - q p in (0, 3/2 p), q = floor(y s / 2^32 - 1/4), off by less than |y| / 2^33 <= 1/4:
//       a valid 32-bit input of the next pass
constexpr int64_t TP_SUM_MAX = 2 * (int64_t)P / 5 - 1;
static_assert((int64_t)P / 2 + TP_SUM_MAX / 4 + TP_SUM_MAX < (int64_t)P, "|y| < p");
__device__ __forceinline__ int32_t tp_fold(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
    constexpr int32_t s1 = (int32_t)(((1ull << 48) + P / 2) / P);
    const int32_t y0 = (int32_t)(a0 + (a1 << 8)), y1 = (int32_t)(a2 + (a3 << 8));
    const int64_t t = (int64_t)y1 * s1 + 0x80000000ll;
    return (int32_t)((uint32_t)y0 + ((uint32_t)y1 << 16) - (uint32_t)(t >> 32) * P);
}
__device__ __forceinline__ uint32_t tp_mul(int32_t y, int32_t w, int32_t s) {
    const int64_t t = (int64_t)y * s - 0x40000000ll;
    return (uint32_t)y * (uint32_t)w - (uint32_t)(t >> 32) * P;
}
// y in (-p, p) -> [0, p)
__device__ __forceinline__ uint32_t tp_canonical(int32_t y) { return min((uint32_t)y, (uint32_t)y + P); }

__device__ __forceinline__ bool tp_wait_count(const uint32_t* p, uint32_t need) {
    for (uint32_t i = 0; i < (1u << 20); i++) {
        uint32_t v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        if (v >= need) return true;
        __nanosleep(64);
    }
    return false;
}
// eight values to p, p + STEP bytes, ..
template <int STEP, int U = 0>
__device__ __forceinline__ void tp_store8(uint32_t* p, const uint32_t (&r)[8]) {
    if constexpr (U < 8) {
        asm volatile("st.global.b32 [%0 + %1], %2;" ::"l"(p), "n"(U * STEP), "r"(r[U]) : "memory");
        tp_store8<STEP, U + 1>(p, r);
    }
}
// mbar_wait_bounded as four instructions a poll: 25 waiting warps' polls are a fifth of
// all instructions the launch issues (side 4096: 2% faster than the C loop, 5% under the
// power cap)
__device__ __forceinline__ bool tp_wait1(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p, q;\n .reg .u32 n;\n mov.u32 n, 262144;\n"
        "W_%=:\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n @p bra D_%=;\n"
        " sub.u32 n, n, 1;\n setp.ne.u32 q, n, 0;\n @q bra W_%=;\nD_%=:\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// the same for a whole warp
__device__ __forceinline__ bool tp_wait(uint64_t* bar, uint32_t parity) {
    return __all_sync(0xFFFFFFFFu, tp_wait1(bar, parity));
}

// The products of set h of a tile of N points: 32 points: the operand's column half h
// against the whole matrix; 64 points: all of it against the matrix's outputs 32 h ...
// Unrolled, with the descriptors one addition apart: the issuing thread has to keep up
// with a product every 64 cycles.
template <int N>
__device__ __forceinline__ void set_products(uint32_t d, uint32_t x, uint64_t desc, int h) {
    if (N == 32) x += 32 * h;
    else desc += h * (2048 >> 4);
#pragma unroll
    for (int k = 0; k < N / 8; k++)
        tc_mma_i8_ta(d, x + 8 * k, desc + k * ((128 * N) >> 4), tc_idesc_u8s8(128, 128), k != 0);
}

template <int L1, int L2, bool PRE, int OSH>
__global__ void __launch_bounds__(TP_THREADS, 1)
    k_tensor_passes(const __grid_constant__ TensorArgs a, const __grid_constant__ TensorMaps maps) {
    using G = TPassGeom<L1, L2>;
    constexpr int N1 = G::N1, N2 = G::N2, S = N1 * N2, CW = G::CW;
    constexpr uint32_t TB = G::TA >> OSH;
    constexpr uint32_t PER_ROUND = G::TA + G::TM + TB;
    extern __shared__ __align__(1024) unsigned char smem[];
    int2* fac = reinterpret_cast<int2*>(smem + G::OFF_F);
    TTile* tiles = reinterpret_cast<TTile*>(smem + G::OFF_T);  // tile i at i % TP_RF
    TTile* queue = tiles + TP_RF;                              // dealt
    unsigned char* raw = smem + G::OFF_R;
    uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem + G::OFF_BAR);  // a half tile landed
    uint64_t* raw_empty = raw_full + G::NR;  // moved on (4 warps) and copied out
    uint64_t* op_full = raw_empty + G::NR;   // a tile's operand is in tensor memory
    uint64_t* op_empty = op_full + G::NA;    // its products are done
    uint64_t* sums = op_empty + G::NA;       // a set's sums complete
    uint64_t* taken = sums + G::NB;          // and read back
    uint64_t* stored = taken + G::NB;        // a tile's stores issued
    uint64_t* tfree = stored + TP_RF;        // its descriptor and factors are no longer needed
    uint64_t* qfull = tfree + TP_RF;
    uint64_t* qempty = qfull + TP_QN;
    uint64_t* mats = qempty + TP_QN;         // the matrices have landed
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(mats + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < G::NR; i++) {
            mbar_init(&raw_full[i], 1);
            mbar_init(&raw_empty[i], 5);
        }
        for (int i = 0; i < G::NA; i++) {
            mbar_init(&op_full[i], 4);
            mbar_init(&op_empty[i], 1);
        }
        for (int i = 0; i < G::NB; i++) {
            mbar_init(&sums[i], 2);  // the products, and the thread that issued them
            mbar_init(&taken[i], TP_EPI / 2);
        }
        for (int i = 0; i < TP_RF; i++) {
            mbar_init(&stored[i], TP_EPI);
            mbar_init(&tfree[i], 1);
        }
        for (int i = 0; i < TP_QN; i++) {
            mbar_init(&qfull[i], 1);
            mbar_init(&qempty[i], 1);
        }
        mbar_init(mats, 1);
        fence_mbar_init();
        mbar_expect_tx(mats, G::MAT_A + G::MAT_M);
        bulk_load_1d(smem, a.mat_a, G::MAT_A, mats);
        bulk_load_1d(smem + G::OFF_M, a.mat_m, G::MAT_M, mats);
    }
    if (warp == TP_W_MMA) tc_alloc(s_tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;
    uint32_t* done_a = a.counters + 1;
    uint32_t* done_m = done_a + a.nchunks;
    uint32_t* done_b = done_m + a.nchunks;
    // Every wait is bounded; a role whose wait gives up flags the error and ends, the
    // others then run out of theirs, and all meet at the barrier at the end. Tiles
    // i = 0, 1, .. of the CTA, their half tiles 2 i + h and their sets 2 i + h each rotate
    // over their buffers; the parity of a wait is that of the buffer's use count.
    auto fail = [&](int code) {
        if (lane == 0) atomicOr(a.err, code);
    };

    if (warp < TP_EPI) {
        // ---- read-back: set h = warp / 8 of every tile; lane = column 32 (warp % 4) + lane
        // of the set, outputs 16 ((warp / 4) % 2) .. + 15. With 32 points a set is a column
        // half, with 64 points a half of the outputs.
        const int h = warp >> 3, half = (warp >> 2) & 1;
        const uint32_t col0 = 32u * (warp & 3) + lane;
        const bool cut = a.out_rows < (uint32_t)S;
        const uint64_t bstep = (uint64_t)(N2 >> OSH) * a.out_pitch;
        for (uint32_t i = 0;; i++) {
            const uint32_t d = 2 * i + h, b = d % G::NB, ts = i % TP_RF;
            if (!tp_wait(&sums[b], (d / G::NB) & 1)) {
                fail(1);
                break;
            }
            tc_fence_after();
            const TTile* tl = tiles + ts;
            const uint32_t ph = tl->ph;
            if (ph != TP_END) {
                const bool wide = (ph == 1 ? N2 : N1) == 32;
                const uint32_t col = col0 + (wide ? TP_BOX * h : 0);
                const uint32_t k0 = 16 * half + (wide ? 0 : 32 * h);  // the first output
                uint32_t* dst = tl->dst + col;
                const int4* f = reinterpret_cast<const int4*>(fac + ts * G::NMAX + k0);  // two outputs each
                const uint32_t t0 = tmem + b * G::DCOLS + 64 * half + ((uint32_t)(32 * (warp & 3)) << 16);
#pragma unroll 1  // the roles' code shares the instruction cache
                for (int g = 0; g < 2; g++) {
                    uint32_t v[32];
                    tc_ld(v, t0 + 32 * g);
                    if (g == 1) {  // the last read of these sums
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&taken[b]);
                    }
                    uint32_t r[8];
                    if (ph != 2 || a.fac_b) {
#pragma unroll
                        for (int u = 0; u < 8; u += 2) {
                            const int4 w = f[4 * g + u / 2];
                            r[u] = tp_mul(tp_fold(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]), w.x, w.y);
                            r[u + 1] = tp_mul(tp_fold(v[4 * u + 4], v[4 * u + 5], v[4 * u + 6], v[4 * u + 7]), w.z, w.w);
                        }
                        if (ph == 2) {
#pragma unroll
                            for (int u = 0; u < 8; u++) r[u] = reduce_2p(r[u]);
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < 8; u++)
                            r[u] = tp_canonical(tp_fold(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]));
                    }
                    const uint32_t k = k0 + 8 * g;
                    if (ph == 0) {  // output k1 = k of column block i2 at row k1 N2 + i2 of the slot
                        tp_store8<N2 * CW * 4>(dst + k * (N2 * CW), r);
                    } else if (ph == 1) {  // output m1 = k of block k1 at row k1 N2 + m1
                        tp_store8<CW * 4>(dst + k * CW, r);
                    } else if (tl->x + col < a.cols) {
                        // row k of w^-1 is output m2 = -k mod N1 of the forward transform: dst is
                        // output m1 + S, k rows of N2 up from there; k = 0 wraps to m1
                        uint32_t* q = dst - k * bstep;
                        uint32_t* q0 = k == 0 ? q - N1 * bstep : q;
                        if (!cut) {
#pragma unroll
                            for (int u = 0; u < 8; u++) {
                                __stcs(u == 0 ? q0 : q, r[u]);
                                q -= bstep;
                            }
                        } else {
                            const uint32_t m = (tl->j << OSH) + (uint32_t)S - k * N2;
#pragma unroll
                            for (int u = 0; u < 8; u++) {
                                if ((u == 0 && k == 0 ? m - (uint32_t)S : m - u * N2) < a.out_rows)
                                    __stcs(u == 0 ? q0 : q, r[u]);
                                q -= bstep;
                            }
                        }
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&stored[ts]);
            if (ph == TP_END) break;
        }
    } else if (warp < TP_W_CONV + 4) {
        // ---- operand: lane = column 32 (warp % 4) + lane of each half tile, its 32 values to
        // columns 32 h .. of the operand
        const int q = warp & 3;
        const uint32_t t0 = tmem + G::ACOL + ((uint32_t)(32 * q) << 16);
        bool ok = true, end = false;
        for (uint32_t i = 0; ok && !end; i++) {
            const uint32_t st = i % G::NA;
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                if (!ok || end) continue;
                const uint32_t s = 2 * i + h, sl = s % G::NR;
                ok = tp_wait(&raw_full[sl], (s / G::NR) & 1);
                if (!ok) continue;
                if (h == 0) {
                    end = tiles[i % TP_RF].ph == TP_END;
                    // the end mark arrives on op_full too: not before tile i - NA's phase is over,
                    // or it would stand in for a slower warp's operand
                    if (end && i >= G::NA) ok = tp_wait(&op_empty[st], ((i / G::NA) - 1) & 1);
                }
                if (!ok || end) continue;
                const uint32_t* src = reinterpret_cast<const uint32_t*>(raw + sl * TP_RAW) + 32 * q + lane;
                uint32_t v[32];
#pragma unroll
                for (int r = 0; r < 32; r++) v[r] = src[r * TP_BOX];
                if constexpr (PRE) {
                    // from shared memory, two a load (32 loads of L2 lines N2 entries apart bound
                    // these warps: a map of 2048 x 32768 took 338 us, 210 without factors; the
                    // recovery of 1024 x 65536 2343 -> 2211 us)
                    const uint32_t ts = i % TP_RF;
                    if (tiles[ts].ph == 0) {
                        const uint4* pre =
                            reinterpret_cast<const uint4*>(smem + G::OFF_P + ts * N1 * 8) + (N1 == 32 ? 0 : 16 * h);
#pragma unroll
                        for (int r = 0; r < 32; r += 2) {
                            const uint4 f = pre[r / 2];
                            v[r] = mul_tw(v[r], f.x, f.y);
                            v[r + 1] = mul_tw(v[r + 1], f.z, f.w);
                        }
                    }
                }
                if (h == 0) {
                    if (i >= G::NA) ok = tp_wait(&op_empty[st], ((i / G::NA) - 1) & 1);
                    if (!ok) continue;
                    tc_fence_after();
                }
                tc_st(t0 + st * 64 + 32 * h, v);
                __syncwarp();
                if (lane == 0) mbar_arrive(&raw_empty[sl]);
            }
            if (!ok) {
                fail(1);
                break;
            }
            if (!end) tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&op_full[st]);
        }
    } else if (warp == TP_W_DEAL) {
        // ---- dealer: draws runs of TP_RUN items, one lane each, so that their dependency
        // polls overlap; the next run is drawn while this one is waited for
        const uint32_t total = (a.nchunks + 2 * a.depth) * PER_ROUND;  // the host keeps this below 2^31
        const bool drawer = lane < TP_RUN;
        auto draw = [&]() {
            uint32_t v = 0;
            if (lane == 0) v = atomicAdd(a.counters, (uint32_t)TP_RUN);
            return v;
        };
        uint32_t i = 0;  // tiles pushed
        auto push = [&](uint32_t at, const TTile& t) {
            const uint32_t qs = at % TP_QN;
            if (at >= TP_QN && !tp_wait1(&qempty[qs], ((at / TP_QN) - 1) & 1)) return false;
            queue[qs] = t;
            mbar_arrive(&qfull[qs]);
            return true;
        };
        bool ok = true;
        uint32_t next = draw();
        for (;;) {
            const uint32_t item = __shfl_sync(0xFFFFFFFFu, next, 0) + lane;
            if (!__any_sync(0xFFFFFFFFu, drawer && item < total)) break;
            next = draw();
            const uint32_t r = item / PER_ROUND;
            uint32_t j = item - r * PER_ROUND, ph = 0;
            int32_t c = (int32_t)r;
            if (j >= G::TA) {
                j -= G::TA;
                ph = 1;
                c -= (int32_t)a.depth;
                if (j >= G::TM) {
                    j -= G::TM;
                    ph = 2;
                    c -= (int32_t)a.depth;
                }
            }
            const bool live = drawer && item < total && c >= 0 && c < (int32_t)a.nchunks;
            TTile t{ph, 0, 0, 0, nullptr, nullptr};
            if (live) {
                // column part of the chunk, then the column block
                const uint32_t parts = ph == 1 ? CW / G::TC2 : CW / G::TC1;
                const uint32_t xo = (j % parts) * (ph == 1 ? G::TC2 : G::TC1);
                t.j = j / parts;
                t.x = (uint32_t)c * CW + xo;
                t.slot = (uint32_t)c % a.slots;
                uint32_t* slot = a.ring + (uint64_t)t.slot * G::SLOT + xo;
                if (ph == 0) {
                    t.dst = slot + t.j * CW;
                    t.fac = a.fac_a + t.j * N1;
                } else if (ph == 1) {
                    t.dst = slot + t.j * (N2 * CW);
                    t.fac = a.fac_m + t.j * N2;
                } else {
                    t.dst = a.out + (uint64_t)(t.j + (S >> OSH)) * a.out_pitch + t.x;
                    t.fac = a.fac_b ? a.fac_b + t.j * N1 : nullptr;
                }
                if (ph == 1) ok = tp_wait_count(done_a + c, G::TA + a.wait_extra);
                else if (ph == 2) ok = tp_wait_count(done_m + c, G::TM + a.wait_extra);
                else if (c >= (int32_t)a.slots) ok = tp_wait_count(done_b + c - a.slots, TB + a.wait_extra);
                if (!ok) atomicOr(a.err, 4);
            }
            if (__any_sync(0xFFFFFFFFu, !ok)) break;
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, live);
            if (live && !push(i + __popc(m & ((1u << lane) - 1)), t)) {
                atomicOr(a.err, 2);
                ok = false;
            }
            if (__any_sync(0xFFFFFFFFu, !ok)) break;
            i += __popc(m);
        }
        if (lane == 0 && !push(i, TTile{TP_END, 0, 0, 0, nullptr, nullptr})) atomicOr(a.err, 2);
    } else if (warp == TP_W_LOAD) {
        if (lane == 0) {
            const uint64_t stream = l2_evict_first();
            const uint32_t in_more = a.in_rows % N2;
            bool end = false, ok = true;
            for (uint32_t i = 0; ok && !end; i++) {
                const uint32_t qs = i % TP_QN, ts = i % TP_RF;
                ok = tp_wait1(&qfull[qs], (i / TP_QN) & 1);
                if (ok && i >= TP_RF) ok = tp_wait1(&tfree[ts], ((i / TP_RF) - 1) & 1);
                if (!ok) break;
                const TTile tl = queue[qs];
                mbar_arrive(&qempty[qs]);
                end = tl.ph == TP_END;
                const bool wide = (tl.ph == 1 ? N2 : N1) == 32;
                const int xh = wide ? TP_BOX : 0, yh = wide ? 0 : 32;  // the second half's offset
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t s = 2 * i + h, sl = s % G::NR;
                    if (ok && s >= G::NR) ok = tp_wait1(&raw_empty[sl], ((s / G::NR) - 1) & 1);
                    if (!ok) continue;
                    // written only now: the copier, in half tile order, is past the tile TP_RF back
                    if (h == 0) tiles[ts] = tl;
                    if (end) {
                        if (h == 0) mbar_arrive(&raw_full[sl]);
                        continue;
                    }
                    unsigned char* dst = raw + sl * TP_RAW;
                    const uint32_t fbytes = tl.fac ? (tl.ph == 1 ? N2 : N1) * 8 : 0;
                    const uint32_t pbytes = PRE && tl.ph == 0 ? N1 * 8 : 0;
                    mbar_expect_tx(&raw_full[sl], h == 0 ? TP_RAW + fbytes + pbytes : TP_RAW);
                    if (h == 0 && pbytes)
                        bulk_load_1d(smem + G::OFF_P + ts * N1 * 8, a.pre + tl.j * N1, pbytes, &raw_full[sl]);
                    if (tl.ph == 0)
                        tma_load_3d_hint(dst, &maps.in[tl.j < in_more], (int)tl.x + xh * h, (int)tl.j, yh * h,
                                         &raw_full[sl], stream);
                    else if (tl.ph == 1)  // block k1 = j: consecutive rows of the slot
                        tma_load_3d(dst, &maps.ring_m, (int)(tl.x % CW) + xh * h, yh * h, (int)(tl.slot * N1 + tl.j),
                                    &raw_full[sl]);
                    else  // column block m1: rows N2 apart
                        tma_load_3d(dst, &maps.ring_b, (int)(tl.x % CW) + xh * h, (int)(tl.j << OSH),
                                    (int)(tl.slot * N1) + yh * h, &raw_full[sl]);
                    if (h == 0 && fbytes) bulk_load_1d(fac + ts * G::NMAX, tl.fac, fbytes, &raw_full[sl]);
                }
            }
            if (!ok) atomicOr(a.err, 2);
        }
    } else if (warp == TP_W_MMA) {
        // ---- products
        if (lane == 0) {
            const uint64_t desc_a = tc_smem_desc(smem_u32(smem), 64 * N1, 128, TC_SWZ_NONE);
            const uint64_t desc_m = tc_smem_desc(smem_u32(smem + G::OFF_M), 64 * N2, 128, TC_SWZ_NONE);
            bool ok = tp_wait1(mats, 0), end = false;
            for (uint32_t i = 0; ok && !end; i++) {
                const uint32_t st = i % G::NA;
                ok = tp_wait1(&op_full[st], (i / G::NA) & 1);
                if (!ok) break;
                const uint32_t ph = tiles[i % TP_RF].ph;
                end = ph == TP_END;
                const uint32_t x = tmem + G::ACOL + st * 64;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t d = 2 * i + h, b = d % G::NB;
                    if (ok && d >= G::NB) ok = tp_wait1(&taken[b], ((d / G::NB) - 1) & 1);
                    if (!ok) continue;
                    mbar_arrive(&sums[b]);
                    if (end) {
                        mbar_arrive(&sums[b]);
                        continue;
                    }
                    tc_fence_after();
                    const uint32_t dd = tmem + b * G::DCOLS;
                    if (ph == 1) set_products<N2>(dd, x, desc_m, h);
                    else set_products<N1>(dd, x, desc_a, h);
                    tc_commit(&sums[b]);
                }
                if (ok && !end) tc_commit(&op_empty[st]);
            }
            if (!ok) atomicOr(a.err, 1);
        }
    } else if (warp == TP_W_SIG) {
        // ---- signal: finished tiles' stores, ordered by the mbarrier, are fenced (the
        // fence is cumulative over them; their readers load them through the async proxy)
        // before the counts that others wait for; one fence covers all tiles that are ready
        if (lane == 0) {
            bool end = false;
            for (uint32_t i = 0; !end;) {
                if (!tp_wait1(&stored[i % TP_RF], (i / TP_RF) & 1)) {
                    atomicOr(a.err, 1);
                    break;
                }
                uint32_t* cnt[4];
                int n = 0;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (k == n && !end && (k == 0 || mbar_try_wait(&stored[i % TP_RF], (i / TP_RF) & 1))) {
                        const TTile* tl = tiles + i % TP_RF;
                        const uint32_t ph = tl->ph;
                        end = ph == TP_END;
                        if (!end) {
                            cnt[k] = (ph == 0 ? done_a : ph == 1 ? done_m : done_b) + tl->x / CW;
                            mbar_arrive(&tfree[i % TP_RF]);
                            n = k + 1;
                            i++;
                        }
                    }
                }
                __threadfence();
                asm volatile("fence.proxy.async;" ::: "memory");
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (k < n) atomicAdd(cnt[k], 1u);
            }
        }
    } else if (warp == TP_W_COPY) {
        // ---- copier: the even rows of pass A's half tiles; one is given back once its store
        // has been read, one store later
        if (lane == 0) {
            const uint64_t stream = l2_evict_first();
            const uint32_t more_rows = a.copy_rows % N2, full_rows = a.copy_rows / N2;
            uint32_t pending = 0;
            bool has = false, end = false, ok = true;
            for (uint32_t i = 0; ok && !end; i++) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    if (!ok || end) continue;
                    const uint32_t s = 2 * i + h, sl = s % G::NR;
                    ok = tp_wait1(&raw_full[sl], (s / G::NR) & 1);
                    if (!ok) continue;
                    const TTile* tl = tiles + i % TP_RF;
                    end = tl->ph == TP_END;
                    if (end) continue;
                    const bool st = tl->ph == 0 && a.copy;
                    if (st) {
                        const bool more = tl->j < more_rows;
                        const int x = (int)tl->x + (N1 == 32 ? TP_BOX * h : 0), z = N1 == 32 ? 0 : 32 * h;
                        if (x < (int)a.cols && z < (int)(full_rows + (more ? 1 : 0)))
                            tma_store_3d_hint(&maps.copy[more], x, (int)tl->j, z, raw + sl * TP_RAW, stream);
                        bulk_commit();
                    }
                    if (has) {
                        if (st) bulk_wait_read1();
                        else bulk_wait_read0();
                        mbar_arrive(&raw_empty[pending]);
                    }
                    has = st;
                    if (st) pending = sl;
                    else mbar_arrive(&raw_empty[sl]);
                }
            }
            if (!ok) atomicOr(a.err, 1);
            bulk_wait0();
        }
    }
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    if (warp == TP_W_MMA) tc_dealloc(tmem, 512);
}

}  // namespace zb
