// Launcher and tables of the tensor-core column passes (tensorpass.cuh).
#include "tensorpass.cuh"
#include "tensorsmall.cuh"
#include "tensorsq.cuh"

#include <algorithm>
#include <cstring>
#include <vector>

#include "internal.hpp"
#include "tma_host.hpp"

namespace zb {
namespace {

// Items a CTA holds between drawing one and publishing it: the pipeline depth is the
// rounds that as many items over the whole grid make up. Fewer and the dependency waits
// stall the CTAs, more and the ring no longer stays in L2. Measured (ms, sides 1024 /
// 2048 / 4096 over 2^27, 2^29 and 2^30 values): 9 0.56 / 2.08 / 4.7, 12 0.51 / 2.05 /
// 4.5, 18 0.54 / 2.17 / 4.9.
#ifndef ZB_TENSOR_HELD
#define ZB_TENSOR_HELD 12
#endif
constexpr uint64_t TENSOR_COUNTERS = 1 << 18;  // bytes: 3 counts a chunk

// Rounds between a chunk's passes, and the ring's slots: a slot is reused that many rounds
// after the last read of the chunk before it.
uint64_t pipe_depth(uint64_t grid, uint64_t per_round) {
    return std::max<uint64_t>(1, ((uint64_t)ZB_TENSOR_HELD * grid + per_round - 1) / per_round);
}
template <class G>
size_t ring_bytes(const zoda_ctx* ctx) {  // the widest launch: full grid, fewest items a round
    const uint64_t d = pipe_depth((uint64_t)ctx->sm_count, G::TA + G::TM + G::TA / 2);
    return (size_t)(3 * d + 1) * G::SLOT * 4;
}

struct Blob {  // one table's parts, as byte offsets
    size_t mat_a, mat_m, fac_a, fac_m;
    size_t bytes;
    explicit Blob(int L) {
        const size_t N1 = 1ull << (L / 2), N2 = 1ull << (L - L / 2), S = 1ull << L;
        mat_a = 0;
        mat_m = mat_a + 16 * N1 * N1;
        fac_a = mat_m + 16 * N2 * N2;
        fac_m = fac_a + 8 * S;
        bytes = fac_m + 8 * S;
    }
};

int32_t centered_host(uint32_t r) { return (int32_t)(r > (P - 1) / 2 ? r - P : r); }
// round(w * 2^32 / p) of the centered w
int32_t quot_host(int32_t w) {
    const int64_t n = (int64_t)w * (1ll << 32), h = P / 2;
    return (int32_t)(n >= 0 ? (n + h) / (int64_t)P : -((-n + h) / (int64_t)P));
}
void put_factor(int32_t* f, uint32_t w) {
    f[0] = centered_host(w);
    f[1] = quot_host(f[0]);
}
// entry (output k, input i) of an n-point matrix operand: digit planes n = 4 k + b,
// inner byte 4 i + y holds digit b of c * 2^(8 y)
void put_entry(uint8_t* mat, uint32_t n, uint32_t k, uint32_t i, uint32_t c) {
    for (uint32_t y = 0; y < 4; y++) {
        const uint32_t d = balanced_digits(c);
        const uint32_t kb = 4 * i + y;
        for (uint32_t b = 0; b < 4; b++) {
            const uint32_t row = 4 * k + b;
            mat[(kb / 16) * (64 * n) + (row / 8) * 128 + (row % 8) * 16 + kb % 16] = (uint8_t)(d >> (8 * b));
        }
        c = mulmod_c(c, 256u);
    }
}

// Whether |a_b + 2^8 a_{b+1}| of every output, b = 0 and 2, stays below `most` for any
// input bytes: the positive or the negative coefficients alone, times 255.
bool plane_sums_below(const uint8_t* mat, uint32_t n, int64_t most) {
    for (uint32_t row = 0; row < 4 * n; row += 2) {
        int64_t pos = 0, neg = 0;
        for (uint32_t kb = 0; kb < 4 * n; kb++) {
            auto d = [&](uint32_t r) { return (int8_t)mat[(kb / 16) * (64 * n) + (r / 8) * 128 + (r % 8) * 16 + kb % 16]; };
            const int64_t v = d(row) + 256 * (int64_t)d(row + 1);
            (v > 0 ? pos : neg) += v;
        }
        if (255 * pos > most || -255 * neg > most) return false;
    }
    return true;
}

template <int L1, int L2, bool PRE, int OSH>
zoda_status set_attr() {
    ZB_CUDA(cudaFuncSetAttribute(k_tensor_passes<L1, L2, PRE, OSH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)TPassGeom<L1, L2>::SMEM));
    return ZODA_OK;
}

// [i1][i2][cols] map of the rows N2 i1 + i2 of a matrix, i1 < n1, i2 < n2, boxes box1 x box2 x 128
zoda_status make_map3(CUtensorMap* m, const void* base, uint64_t cols, uint64_t n2, uint64_t n1, uint64_t pitch,
                      uint64_t block, uint32_t box2 = 1, uint32_t box1 = 32) {
    auto fn = encode_fn();
    if (!fn) {
        set_last_error_text("cuTensorMapEncodeTiled unavailable");
        return ZODA_ERR_CUDA;
    }
    const cuuint64_t dims[3] = {cols, n2, n1};
    const cuuint64_t strides[2] = {pitch * 4, block * pitch * 4};
    const cuuint32_t box[3] = {TP_BOX, box2, box1}, estr[3] = {1, 1, 1};
    const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_last_error_text("cuTensorMapEncodeTiled failed with CUresult " + std::to_string((int)r));
        return ZODA_ERR_CUDA;
    }
    return ZODA_OK;
}
// The two maps of the first `rows` rows (TensorMaps); rows >= N2.
template <class G>
zoda_status make_row_maps(CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, uint64_t pitch) {
    const uint64_t full = rows / G::N2, rem = rows % G::N2;
    zoda_status s = make_map3(&m[0], base, cols, G::N2, full, pitch, G::N2);
    if (s != ZODA_OK) return s;
    m[1] = m[0];
    return rem ? make_map3(&m[1], base, cols, rem, full + 1, pitch, G::N2) : ZODA_OK;
}
template <class G>
zoda_status make_maps(TensorMaps* m, const TensorArgs& a, uint64_t cols) {
    zoda_status s = make_row_maps<G>(m->in, a.in, cols, a.in_rows, a.in_pitch);
    if (s != ZODA_OK) return s;
    m->copy[0] = m->copy[1] = m->in[0];
    if (a.copy && (s = make_row_maps<G>(m->copy, a.copy, cols, a.copy_rows, a.copy_pitch)) != ZODA_OK) return s;
    const uint64_t n1 = (uint64_t)a.slots * G::N1;
    if ((s = make_map3(&m->ring_m, a.ring, G::CW, G::N2, n1, G::CW, G::N2, 32, 1)) != ZODA_OK) return s;
    return make_map3(&m->ring_b, a.ring, G::CW, G::N2, n1, G::CW, G::N2);
}

template <int L1, int L2, bool PRE, int OSH>
zoda_status launch_t(zoda_ctx* ctx, TensorArgs a, uint64_t cols, cudaStream_t st) {
    using G = TPassGeom<L1, L2>;
    const uint64_t nch = (cols + G::CW - 1) / G::CW;
    const uint64_t per_round = G::TA + G::TM + (G::TA >> OSH);
    const uint64_t grid = std::min<uint64_t>((uint64_t)ctx->sm_count, nch * per_round);
    const uint64_t depth = pipe_depth(grid, per_round);
    if (cols >= (1ull << 31) || (nch + 2 * depth) * per_round + 16 * grid >= (1ull << 31)) return ZODA_ERR_UNSUPPORTED;
    a.nchunks = (uint32_t)nch;
    a.depth = (uint32_t)depth;
    a.cols = (uint32_t)cols;
    a.slots = (uint32_t)std::min<uint64_t>(nch, 3 * depth + 1);
    const size_t cbytes = (size_t)(1 + 3 * nch) * sizeof(uint32_t);
    if (cbytes > TENSOR_COUNTERS || TENSOR_COUNTERS + (size_t)a.slots * G::SLOT * 4 > ctx->tensor_buf.bytes)
        return ZODA_ERR_UNSUPPORTED;
    a.counters = (uint32_t*)ctx->tensor_buf.p;
    a.ring = (uint32_t*)((unsigned char*)ctx->tensor_buf.p + TENSOR_COUNTERS);
    a.err = ctx->d_err;
    TensorMaps maps;
    zoda_status s = make_maps<G>(&maps, a, cols);
    if (s != ZODA_OK) return s;
    std::lock_guard<std::mutex> lock(ctx->tensor_mu);
    if (ctx->fault_site == ZODA_FAULT_PIPE_WAIT && ctx->fault_after-- == 0) {
        ctx->fault_site = 0;
        a.wait_extra = 1;  // a count no chunk reaches: every dependency wait runs out
    }
    // launches on other streams share the counters and the ring: each waits for the one before
    ZB_CUDA(cudaStreamWaitEvent(st, ctx->tensor_done, 0));
    ZB_CUDA(cudaMemsetAsync(a.counters, 0, cbytes, st));
    k_tensor_passes<L1, L2, PRE, OSH><<<(unsigned)grid, TP_THREADS, G::SMEM, st>>>(a, maps);
    ZB_CUDA(cudaGetLastError());
    ZB_CUDA(cudaEventRecord(ctx->tensor_done, st));
    return ZODA_OK;
}

}  // namespace

zoda_status tensor_init(zoda_ctx* ctx) {
    zoda_status s = set_attr<5, 6, false, 0>();
    ZB_CUDA(cudaFuncSetAttribute(k_tensor_square, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TSqGeom::SMEM));
    if (s == ZODA_OK) s = set_attr<6, 6, false, 0>();
    if (s == ZODA_OK) s = set_attr<5, 6, true, 0>();
    if (s == ZODA_OK) s = set_attr<6, 6, true, 0>();
    if (s == ZODA_OK) s = set_attr<5, 6, false, 1>();
    if (s == ZODA_OK) s = set_attr<6, 6, false, 1>();
    if (s != ZODA_OK) return s;
    for (int L = TENSOR_SMALL_MIN_LOG; L <= TENSOR_SMALL_MAX_LOG; L++) {
        const uint32_t S = 1u << L, g = root_of_unity(L + 1), w = root_of_unity(L), sinv = powmod_c(S, P - 2);
        std::vector<uint8_t> h(16 * (size_t)S * S);
        for (uint32_t d = 0; d < S; d++) {
            uint32_t c = 0, x = sinv;
            const uint32_t r = mulmod_c(g, powmod_c(w, d));
            for (uint32_t k = 0; k < S; k++, x = mulmod_c(x, r)) c = (uint32_t)(((uint64_t)c + x) % P);
            for (uint32_t j = 0; j < S; j++) put_entry(h.data(), S, (j + d) & (S - 1), j, c);
        }
        if (!plane_sums_below(h.data(), S, TP_SUM_MAX)) return ZODA_ERR_STATE;
        ZB_CUDA(cudaMalloc(&ctx->tables.tensor[L], h.size()));
        ZB_CUDA(cudaMemcpy(ctx->tables.tensor[L], h.data(), h.size(), cudaMemcpyHostToDevice));
    }
    ZB_CUDA(cudaFuncSetAttribute(k_tensor_small<5>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TSmallGeom<5>::SMEM));
    ZB_CUDA(cudaFuncSetAttribute(k_tensor_small<6>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TSmallGeom<6>::SMEM));
    const size_t ring = std::max(ring_bytes<TPassGeom<5, 6>>(ctx), ring_bytes<TPassGeom<6, 6>>(ctx));
    // without room for the ring (74 MiB) the context runs the single-pass kernels (tensor_fits)
    if (ctx->tensor_buf.ensure(TENSOR_COUNTERS + ring) != ZODA_OK) cudaGetLastError();
    ZB_CUDA(cudaEventCreateWithFlags(&ctx->tensor_done, cudaEventDisableTiming));
    for (int L = TENSOR_MIN_LOG; L <= TENSOR_MAX_LOG; L++) {
        std::vector<uint8_t> h;
        if (!tensor_tables_host(L, root_of_unity(L + 1), false, &h)) return ZODA_ERR_STATE;
        ZB_CUDA(cudaMalloc(&ctx->tables.tensor[L], h.size()));
        ZB_CUDA(cudaMemcpy(ctx->tables.tensor[L], h.data(), h.size(), cudaMemcpyHostToDevice));
    }
    return ZODA_OK;
}

void tensor_release(zoda_ctx* ctx) {
    ctx->tensor_buf.release();
    if (ctx->tensor_done) cudaEventDestroy(ctx->tensor_done);
    for (auto* t : ctx->tables.tensor)
        if (t) cudaFree(t);
}

bool tensor_fits(const zoda_ctx* ctx, int L, uint64_t cols, cudaStream_t st) {
    if (L == 10) return true;  // nothing shared (tensorsq.cuh)
    if (L < TENSOR_MIN_LOG || L > TENSOR_MAX_LOG) return false;
    const uint64_t cw = L == 12 ? TPassGeom<6, 6>::CW : TPassGeom<5, 6>::CW;
    if ((1 + 3 * ((cols + cw - 1) / cw)) * sizeof(uint32_t) > TENSOR_COUNTERS) return false;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) {
        cudaGetLastError();  // another stream's capture forbids the query: as if capturing
        return false;
    }
    return ctx->tensor_buf.p && cap == cudaStreamCaptureStatusNone;
}

bool tensor_tables_host(int L, uint32_t base, bool lower_half, std::vector<uint8_t>* out) {
    const Blob bl(L);
    const int L1 = L / 2, L2 = L - L1;
    const uint32_t N1 = 1u << L1, N2 = 1u << L2, S = 1u << L;
    out->assign(bl.bytes, 0);
    uint8_t* o = out->data();
    const uint32_t w1 = root_pow(L1, 1, true), w2 = root_of_unity(L2), wS = root_of_unity(L), wSi = root_pow(L, 1, true);
    for (uint32_t k = 0; k < N1; k++)
        for (uint32_t i = 0, x = 1, st = powmod_c(w1, k); i < N1; i++, x = mulmod_c(x, st))
            put_entry(o + bl.mat_a, N1, k, i, x);
    // C[d] = S^-1 sum_k2 base^(N1 k2) w_N2^(k2 d), k2 < N2 / 2 only with lower_half
    const uint32_t sinv = powmod_c(S, P - 2), bn = powmod_c(base, N1);
    std::vector<uint32_t> C(N2);
    for (uint32_t d = 0; d < N2; d++) {
        uint32_t sum = 0, x = sinv;
        const uint32_t st = mulmod_c(bn, powmod_c(w2, d));
        for (uint32_t k2 = 0; k2 < (lower_half ? N2 / 2 : N2); k2++, x = mulmod_c(x, st))
            sum = (uint32_t)(((uint64_t)sum + x) % P);
        C[d] = sum;
    }
    for (uint32_t m = 0; m < N2; m++)
        for (uint32_t i = 0; i < N2; i++) put_entry(o + bl.mat_m, N2, m, i, C[(m - i) & (N2 - 1)]);
    // factors as [column block][output]; 1024 points (tensorsq.cuh): outputs 2 k and 2 k + 1 of
    // every column block as [k][column block]
    auto at = [&](uint32_t block, uint32_t k, uint32_t n) -> size_t {
        return L == 10 ? 16 * (32 * (k / 2) + block) + 8 * (k % 2) : 8 * ((size_t)block * n + k);
    };
    for (uint32_t i2 = 0; i2 < N2; i2++)
        for (uint32_t k1 = 0, x = 1, st = powmod_c(wSi, i2); k1 < N1; k1++, x = mulmod_c(x, st))
            put_factor(reinterpret_cast<int32_t*>(o + bl.fac_a + at(i2, k1, N1)), x);
    for (uint32_t k1 = 0, u = 1; k1 < N1; k1++, u = mulmod_c(u, base))
        for (uint32_t m1 = 0, x = u, st = powmod_c(wS, k1); m1 < N2; m1++, x = mulmod_c(x, st))
            put_factor(reinterpret_cast<int32_t*>(o + bl.fac_m + at(k1, m1, N2)), x);
    return plane_sums_below(o + bl.mat_a, N1, TP_SUM_MAX) && plane_sums_below(o + bl.mat_m, N2, TP_SUM_MAX);
}

namespace {
// One launch with the tables at `tab` (device); a holds the views and limits.
zoda_status launch_tensor(zoda_ctx* ctx, int L, const uint8_t* tab, TensorArgs a, uint64_t cols, cudaStream_t st) {
    if (cols == 0) return ZODA_OK;
    const Blob bl(L);
    a.mat_a = reinterpret_cast<const uint4*>(tab + bl.mat_a);
    a.mat_m = reinterpret_cast<const uint4*>(tab + bl.mat_m);
    a.fac_a = reinterpret_cast<const int2*>(tab + bl.fac_a);
    a.fac_m = reinterpret_cast<const int2*>(tab + bl.fac_m);
    switch (L) {
#define ZB_CASE(L, L1, L2)                                                          \
    case L:                                                                         \
        if (a.pre) return launch_t<L1, L2, true, 0>(ctx, a, cols, st);              \
        return a.out_shift ? launch_t<L1, L2, false, 1>(ctx, a, cols, st) : launch_t<L1, L2, false, 0>(ctx, a, cols, st);
        ZB_CASE(11, 5, 6) ZB_CASE(12, 6, 6)
#undef ZB_CASE
        default: return ZODA_ERR_UNSUPPORTED;
    }
}

__device__ __forceinline__ int32_t centered_dev(uint32_t r) { return (int32_t)(r > (P - 1) / 2 ? r - P : r); }
// round(w * 2^32 / p) of a centered w, as quot_host
__device__ __forceinline__ int32_t quot_dev(int32_t w) {
    const uint64_t n = (uint64_t)(w < 0 ? -(int64_t)w : (int64_t)w) << 32;
    const int64_t q = (int64_t)((n + P / 2) / P);
    return (int32_t)(w < 0 ? -q : q);
}
// The decoder's factors per row as the passes read them: pass B's [m1][k] from the output's,
// out[m1 + N2 ((N1 - k) mod N1)], pass A's [i2][i1] from the input's, in[N2 i1 + i2].
__global__ void k_row_factors(const uint2* __restrict__ row, const uint2* __restrict__ in, int l1, int l2,
                              int2* __restrict__ out, uint2* __restrict__ in_t) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 1u << (l1 + l2)) return;
    const uint32_t m1 = i >> l1, k = i & ((1u << l1) - 1);
    in_t[i] = in[(k << l2) + m1];
    const uint32_t w = row[m1 + ((((1u << l1) - k) & ((1u << l1) - 1)) << l2)].x;
    const int32_t a = centered_dev(w);
    out[i] = make_int2(a, quot_dev(a));
}

// The tables of one map, kept in the context under `key` (the caller holds ctx->mu).
zoda_status map_tables(zoda_ctx* ctx, int key, int L, uint32_t base, bool lower_half, const uint8_t** out) {
    DevBuf& b = ctx->coset_tabs[key];
    if (!b.p) {
        std::vector<uint8_t> h;
        if (!tensor_tables_host(L, base, lower_half, &h)) return ZODA_ERR_UNSUPPORTED;
        zoda_status s = b.ensure(h.size());
        if (s != ZODA_OK) return s;
        ZB_CUDA(cudaMemcpy(b.p, h.data(), h.size(), cudaMemcpyHostToDevice));
    }
    *out = (const uint8_t*)b.p;
    return ZODA_OK;
}
}  // namespace

// The decoder's two maps over N = 2^L points (general.cu): g~ / Z(h w) = izh(j) NTT(h^i / N
// INTT(zk y)) into the scratch [N][w], izh as pass B's factors; then the even outputs of
// NTT(h^-i / N [i < N/2] INTT(.)), which are the data rows.
zoda_status tensor_recover_tables(zoda_ctx* ctx, int L, const uint2* zk, const uint2* izh, void* fac, cudaStream_t st) {
    k_row_factors<<<(1u << L) / 128, 128, 0, st>>>(izh, zk, L / 2, L - L / 2, (int2*)fac, (uint2*)fac + (1u << L));
    ZB_CUDA(cudaGetLastError());
    return ZODA_OK;
}
zoda_status tensor_recover(zoda_ctx* ctx, int L, const uint32_t* code, uint64_t code_pitch, const void* fac,
                           uint32_t* scratch, uint32_t* data, uint64_t data_pitch, uint64_t w,
                           cudaStream_t st) {
    const uint8_t *ta = nullptr, *tb = nullptr;
    zoda_status s = map_tables(ctx, -(500000000 + 2 * L), L, GENERATOR, false, &ta);
    if (s == ZODA_OK) s = map_tables(ctx, -(500000001 + 2 * L), L, powmod_c(GENERATOR, P - 2), true, &tb);
    if (s != ZODA_OK) return s;
    TensorArgs a{};
    a.in = code;
    a.in_pitch = code_pitch;
    a.in_rows = 1u << L;
    a.pre = (const uint2*)fac + (1u << L);
    a.fac_b = (const int2*)fac;
    a.out = scratch;
    a.out_pitch = w;
    a.out_rows = 1u << L;
    if ((s = launch_tensor(ctx, L, ta, a, w, st)) != ZODA_OK) return s;
    TensorArgs b{};
    b.in = scratch;
    b.in_pitch = w;
    b.in_rows = 1u << L;
    b.out = data;
    b.out_pitch = data_pitch;
    b.out_rows = 1u << L;
    b.out_shift = 1;
    return launch_tensor(ctx, L, tb, b, w, st);
}

namespace {
template <int LOG_S>
zoda_status tensor_small_t(const zoda_ctx* ctx, const uint32_t* in, uint32_t* out, uint64_t cols, cudaStream_t st,
                           bool odd_only, uint32_t in_rows, uint32_t out_rows) {
    using G = TSmallGeom<LOG_S>;
    const uint64_t ntiles = (cols + G::COLS - 1) / G::COLS;
    if (ntiles == 0) return ZODA_OK;
    if (cols >= (1ull << 31)) return ZODA_ERR_UNSUPPORTED;
    TensorSmallArgs a{};
    a.out = odd_only ? out : out + cols;
    a.pitch = odd_only ? cols : 2 * cols;
    a.cols = (uint32_t)cols;
    a.ntiles = (uint32_t)ntiles;
    a.rows = out_rows / 2;
    a.copy_rows = odd_only ? 0 : (out_rows + 1) / 2;
    a.mat = (const uint4*)ctx->tables.tensor[LOG_S];
    a.err = ctx->d_err;
    CUtensorMap mi, mc;
    zoda_status s = make_map(&mi, in, cols, in_rows, cols * 4, G::COLS, G::S);
    if (s != ZODA_OK) return s;
    mc = mi;
    if (a.copy_rows && (s = make_map(&mc, out, cols, a.copy_rows, cols * 8, G::COLS, G::S)) != ZODA_OK) return s;
    const uint64_t grid = std::min<uint64_t>(ntiles, (uint64_t)ctx->sm_count * (G::S == 32 ? 2 : 1));
    k_tensor_small<LOG_S><<<(unsigned)grid, G::THREADS, G::SMEM, st>>>(a, mi, mc);
    ZB_CUDA(cudaGetLastError());
    return ZODA_OK;
}
}  // namespace

zoda_status tensor_small_extend(const zoda_ctx* ctx, int L, const uint32_t* in, uint32_t* out, uint64_t cols,
                                cudaStream_t st, bool odd_only, uint32_t in_rows, uint32_t out_rows) {
    if (L == 5) return tensor_small_t<5>(ctx, in, out, cols, st, odd_only, in_rows, out_rows);
    return tensor_small_t<6>(ctx, in, out, cols, st, odd_only, in_rows, out_rows);
}

// The map with the tables at `tab` over 1024 points in one CTA per 16 columns: input rows
// in_rows of [.][cols], copied to the first copy_rows rows at `copy` when given; output m
// (< out_rows) at out + m * out_pitch.
zoda_status tensor_square(const zoda_ctx* ctx, const uint8_t* tab, const uint32_t* in, uint32_t in_rows, uint64_t cols,
                          uint32_t* copy, uint64_t copy_pitch, uint32_t copy_rows, uint32_t* out, uint64_t out_pitch,
                          uint32_t out_rows, cudaStream_t st) {
    using G = TSqGeom;
    const Blob bl(10);
    const uint64_t ntiles = (cols + 2 * G::C - 1) / (2 * G::C);
    if (ntiles == 0 || out_rows == 0) return ZODA_OK;
    if (cols >= (1ull << 31)) return ZODA_ERR_UNSUPPORTED;
    TensorSqArgs a{};
    a.ntiles = (uint32_t)ntiles;
    a.out_rows = out_rows;
    a.copy_rows = copy ? copy_rows : 0;
    a.mat_a = (const uint4*)(tab + bl.mat_a);
    a.mat_m = (const uint4*)(tab + bl.mat_m);
    a.fac_a = (const int4*)(tab + bl.fac_a);
    a.fac_m = (const int4*)(tab + bl.fac_m);
    a.err = ctx->d_err;
    CUtensorMap mi, mc, mo;
    zoda_status s = make_map(&mi, in, cols, in_rows, cols * 4, 2 * G::C, 256);
    if (s != ZODA_OK) return s;
    if ((s = make_map(&mo, out, cols, out_rows, out_pitch * 4, 2 * G::C, 256)) != ZODA_OK) return s;
    mc = mi;
    if (copy && (s = make_map(&mc, copy, cols, copy_rows, copy_pitch * 4, 2 * G::C, 256)) != ZODA_OK) return s;
    const uint64_t grid = std::min<uint64_t>(ntiles, (uint64_t)ctx->sm_count);
    k_tensor_square<<<(unsigned)grid, G::THREADS, G::SMEM, st>>>(a, mi, mc, mo);
    ZB_CUDA(cudaGetLastError());
    return ZODA_OK;
}

zoda_status tensor_extend(zoda_ctx* ctx, int L, const uint32_t* in, uint32_t* out, uint64_t cols, cudaStream_t st,
                          bool odd_only, uint32_t in_rows, uint32_t out_rows) {
    if (L == 10)
        return tensor_square(ctx, ctx->tables.tensor[L], in, in_rows, cols, odd_only ? nullptr : out, 2 * cols,
                             (out_rows + 1) / 2, odd_only ? out : out + cols, odd_only ? cols : 2 * cols, out_rows / 2,
                             st);
    TensorArgs a{};
    a.in = in;
    a.in_pitch = cols;
    a.in_rows = in_rows;
    if (!odd_only) {
        a.copy = out;
        a.copy_pitch = 2 * cols;
        a.copy_rows = (out_rows + 1) / 2;
    }
    a.out = odd_only ? out : out + cols;
    a.out_pitch = odd_only ? cols : 2 * cols;
    a.out_rows = out_rows / 2;
    return launch_tensor(ctx, L, ctx->tables.tensor[L], a, cols, st);
}

// Coset c of the encode over 2^ln points with n_k = 2^L (general.cu): output row R m + c, R =
// 2^(ln - L), for m < mc; with `copy`, coset 0 (the zero-padded data, m < m0) as well.
zoda_status tensor_coset(zoda_ctx* ctx, int L, int ln, uint32_t c, const uint32_t* in, uint32_t k, uint64_t cols,
                         uint32_t* out, uint32_t mc, bool copy, uint32_t m0, cudaStream_t st) {
    const uint8_t* tab = nullptr;
    const uint32_t R = 1u << (ln - L);
    zoda_status s = map_tables(ctx, -(600000000 + ((L * 32 + ln) * TENSOR_MAX_COSETS + (int)c)), L,
                               root_pow(ln, c, false), false, &tab);
    if (s != ZODA_OK) return s;
    uint32_t* dst = out + c * cols;
    if (L == 10)
        return tensor_square(ctx, tab, in, k, cols, copy ? out : nullptr, R * cols, m0, dst, R * cols, mc, st);
    TensorArgs a{};
    a.in = in;
    a.in_pitch = cols;
    a.in_rows = k;
    if (copy) {
        a.copy = out;
        a.copy_pitch = R * cols;
        a.copy_rows = m0;
    }
    a.out = dst;
    a.out_pitch = R * cols;
    a.out_rows = mc;
    return launch_tensor(ctx, L, tab, a, cols, st);
}

}  // namespace zb
