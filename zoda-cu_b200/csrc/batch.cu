// Batched extension of many squares in one graph launch (the
// zoda_batch_* entry points of include/zoda_b200.h).
//
// Host side of k_extend_batch (extend_tma.cuh): one BatchSquare descriptor per
// square (two TMA maps, output pointer, shape, first global tile index),
// squares ordered by decreasing side, a device counter the CTAs draw tiles
// from, and a CUDA graph holding the counter reset and the launch. Wide squares of
// side 1024 are launches of k_tensor_square (tensorsq.cuh) in the same graph, those of
// side 2048 launches of k_tensor_passes before it.
#include <algorithm>
#include <new>
#include <vector>

#include "tma_host.hpp"

struct zoda_batch {
    zoda_ctx* ctx = nullptr;
    uint32_t nsq = 0;  // of the queue
    std::vector<zoda_square> wide;    // side 1024, in launches of their own in the graph
    std::vector<zoda_square> ringed;  // side 2048, launched before the graph: they share the context's ring
    uint64_t total_tiles = 0;
    uint64_t elements = 0;
    zb::DevBuf squares;  // BatchSquare[nsq]
    zb::DevBuf counter;  // unsigned long long
    zb::DevBuf tables;   // SideTables[26]: radix 16 at [log_s], radix 8 at [13 + log_s]
    int lept = 4;        // level radix 2^lept of this batch's launch
    cudaStream_t cap = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
};

namespace zb {
namespace {

template <int LOG_S>
zoda_status fill_square(BatchSquare* b, const zoda_square& q, int promo) {
    using TP = TPlan<LOG_S>;
    zoda_status s = make_tile_maps<TP>(&b->in_map, &b->even_map, q.d_in, q.d_out, q.cols, promo);
    if (s != ZODA_OK) return s;
    b->out = q.d_out;
    b->cols = q.cols;
    b->log_s = LOG_S;
    b->ntiles = (uint32_t)((q.cols + TP::C - 1) / TP::C);
    return ZODA_OK;
}

int log2_side(uint32_t k) {
    if (k == 0 || (k & (k - 1))) return -1;
    int l = 0;
    while ((1u << l) < k) l++;
    return l;
}

}  // namespace

zoda_status make_batch_square(const zoda_square& q, BatchSquare* b, int promo) {
    const int ls = log2_side(q.k);
    if (!q.d_in || !q.d_out || ls < 0 || q.cols % 4 || (((uintptr_t)q.d_in | (uintptr_t)q.d_out) & 15))
        return ZODA_ERR_ARG;
    if (ls < BATCH_MIN_LOG || ls > BATCH_MAX_LOG) {
        set_last_error_text("batched sides are 32 .. 2048");
        return ZODA_ERR_UNSUPPORTED;
    }
    memset(b, 0, sizeof *b);
    switch (ls) {
        case 5: return fill_square<5>(b, q, promo);
        case 6: return fill_square<6>(b, q, promo);
        case 7: return fill_square<7>(b, q, promo);
        case 8: return fill_square<8>(b, q, promo);
        case 9: return fill_square<9>(b, q, promo);
        case 10: return fill_square<10>(b, q, promo);
        default: return fill_square<11>(b, q, promo);
    }
}

// Squares of side 1024 and 2048 leave the queue for the tensor cores where a launch of their
// own pays. Side 1024 from 16384 columns (alone, tensor / TMA-staged: 8192 columns 39 / 43 us,
// 16384 65 / 90, 131072 498 / 576; batches, launches / queue: one square of 16384 columns 64 /
// 112, eight 481 / 578, one beside 16 of 256 x 4096 148 / 183, 48 squares of sides 32 .. 1024
// 4441 / 4922; another box 4613 / 4907). Side 2048 where the single call does (tensor_pays): 96
// squares of sides 32 .. 2048 37.1 / 48.8 ms, and requests of those sides, 2000 a second, 7368 /
// 5991 Gb/s with a median latency of 4.4 / 92 ms. A plan that was set for
// the side, or for the context, keeps deciding.
constexpr uint64_t WIDE_MIN_COLS = 16384;
bool leaves_queue(const zoda_ctx* ctx, const zoda_square& q) {
    const int L = log2_side(q.k);
    if (L != 10 && L != 11) return false;
    if (L == 10 ? q.cols < WIDE_MIN_COLS : !tensor_pays(ctx, L, q.cols, TensorUse::square)) return false;
    return q.cols < (1ull << 31) && ctx->impl == ZODA_IMPL_AUTO && (!ctx->planned[L] || is_tensor_plan(ctx->plan[L]));
}
zoda_status launch_alone(const zoda_ctx* ctx, const zoda_square& q, cudaStream_t st) {
    const int L = log2_side(q.k);
    return launch_plan(ctx, L, default_plan(L), q.d_in, q.d_out, q.cols, st, false, q.k, 2 * q.k);
}

zoda_status launch_batch_kernel(const zoda_ctx* ctx, const BatchSquare* d_sq, uint32_t nsq, uint64_t total_tiles,
                                unsigned long long* d_counter, const SideTables* d_tables, int lept, cudaStream_t st) {
    if (total_tiles == 0) return ZODA_OK;
    const uint64_t grid = total_tiles < (uint64_t)ctx->sm_count ? total_tiles : (uint64_t)ctx->sm_count;
    if (lept == 3)
        k_extend_batch<3><<<(unsigned)grid, BatchGeom<3>::THREADS, BatchGeom<3>::SMEM, st>>>(
            d_sq, nsq, total_tiles, d_counter, d_tables, ctx->d_err);
    else
        k_extend_batch<4><<<(unsigned)grid, BatchGeom<4>::THREADS, BatchGeom<4>::SMEM, st>>>(
            d_sq, nsq, total_tiles, d_counter, d_tables, ctx->d_err);
    ZB_CUDA(cudaGetLastError());
    return ZODA_OK;
}

zoda_status set_batch_kernel_attributes() {
    ZB_CUDA(cudaFuncSetAttribute(k_extend_batch<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)BatchGeom<4>::SMEM));
    ZB_CUDA(cudaFuncSetAttribute(k_extend_batch<3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)BatchGeom<3>::SMEM));
    return ZODA_OK;
}

int batch_lept(const zoda_ctx* ctx, int max_log) {
    if (max_log >= 0 && max_log <= 12 && ctx->planned[max_log] && ctx->plan[max_log].impl == ZODA_IMPL_TMA &&
        ctx->plan[max_log].radix == 8)
        return 3;
    return 4;
}

namespace {

// The graph: two chains, so that a launch's blocks take over the SMs as those of the one
// before it end. The squares' launches go to the chains in turn; the queue (counter = 0,
// then the persistent kernel, one CTA per SM) comes last, its tiles fill what is left.
zoda_status capture_batch(zoda_batch* bt) {
    zoda_ctx* ctx = bt->ctx;
    const bool fork = bt->wide.size() + (bt->total_tiles != 0) > 1;
    struct Side {
        cudaStream_t st = nullptr;
        cudaEvent_t begin = nullptr, end = nullptr;
        ~Side() {
            if (begin) cudaEventDestroy(begin);
            if (end) cudaEventDestroy(end);
            if (st) cudaStreamDestroy(st);
        }
    } side;
    if (fork) {
        ZB_CUDA(cudaStreamCreateWithFlags(&side.st, cudaStreamNonBlocking));
        ZB_CUDA(cudaEventCreateWithFlags(&side.begin, cudaEventDisableTiming));
        ZB_CUDA(cudaEventCreateWithFlags(&side.end, cudaEventDisableTiming));
    }
    ZB_CUDA(cudaStreamBeginCapture(bt->cap, cudaStreamCaptureModeThreadLocal));
    auto record = [&]() -> zoda_status {
        if (fork) {
            ZB_CUDA(cudaEventRecord(side.begin, bt->cap));
            ZB_CUDA(cudaStreamWaitEvent(side.st, side.begin, 0));
        }
        uint32_t n = 0;
        auto next = [&] { return fork && (n++ & 1) ? side.st : bt->cap; };
        zoda_status s = ZODA_OK;
        for (const zoda_square& q : bt->wide)
            if ((s = launch_alone(ctx, q, next())) != ZODA_OK) break;
        if (s == ZODA_OK && bt->total_tiles) {
            cudaStream_t st = next();
            ZB_CUDA(cudaMemsetAsync(bt->counter.p, 0, sizeof(unsigned long long), st));
            s = launch_batch_kernel(ctx, (const BatchSquare*)bt->squares.p, bt->nsq, bt->total_tiles,
                                    (unsigned long long*)bt->counter.p,
                                    (const SideTables*)bt->tables.p + (bt->lept == 3 ? 13 : 0), bt->lept, st);
        }
        if (fork) {
            ZB_CUDA(cudaEventRecord(side.end, side.st));
            ZB_CUDA(cudaStreamWaitEvent(bt->cap, side.end, 0));
        }
        return s;
    };
    const zoda_status s = record();
    const cudaError_t e = cudaStreamEndCapture(bt->cap, &bt->graph);
    if (s != ZODA_OK) return s;
    if (e != cudaSuccess) {
        set_last_error("cudaStreamEndCapture", e);
        return ZODA_ERR_CUDA;
    }
    return ZODA_OK;
}

}  // namespace
}  // namespace zb

using namespace zb;

extern "C" {

zoda_status zoda_batch_create(zoda_ctx* ctx, const zoda_square* squares, uint32_t n, zoda_batch** out) {
    if (!ctx || !out || (n && !squares)) return ZODA_ERR_ARG;
    *out = nullptr;
    std::vector<uint32_t> order(n);
    for (uint32_t i = 0; i < n; i++) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return squares[a].k > squares[b].k; });
    std::vector<BatchSquare> host;
    std::vector<zoda_square> wide, ringed;
    host.reserve(n);
    uint64_t first = 0, elements = 0;
    for (uint32_t j = 0; j < n; j++) {
        const zoda_square& q = squares[order[j]];
        BatchSquare b;
        const zoda_status s = make_batch_square(q, &b, side_l2_promo(ctx, log2_side(q.k)));
        if (s != ZODA_OK) return s;
        elements += (uint64_t)q.k * q.cols;
        if (leaves_queue(ctx, q)) {
            (q.k == 1024 ? wide : ringed).push_back(q);
            continue;
        }
        b.first = first;
        first += b.ntiles;
        host.push_back(b);
    }
    const uint32_t nq = (uint32_t)host.size();
    zoda_batch* bt = new (std::nothrow) zoda_batch();
    if (!bt) return ZODA_ERR_NOMEM;
    bt->ctx = ctx;
    bt->nsq = nq;
    bt->wide = std::move(wide);
    bt->ringed = std::move(ringed);
    bt->total_tiles = first;
    bt->elements = elements;
    auto fail = [&](zoda_status s) {
        zoda_batch_destroy(bt);
        return s;
    };
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) {
        set_last_error("cudaSetDevice", e);
        return fail(ZODA_ERR_CUDA);
    }
    zoda_status s;
    if ((s = bt->squares.ensure(std::max<size_t>(1, nq) * sizeof(BatchSquare))) != ZODA_OK) return fail(s);
    if ((s = bt->counter.ensure(sizeof(unsigned long long))) != ZODA_OK) return fail(s);
    if ((s = bt->tables.ensure(26 * sizeof(SideTables))) != ZODA_OK) return fail(s);
    std::vector<SideTables> tabs(26);
    for (int ls = BATCH_MIN_LOG; ls <= BATCH_MAX_LOG; ls++) {
        tabs[ls] = side_tables(ctx, ls, 4);
        tabs[13 + ls] = side_tables(ctx, ls, 3);
    }
    bt->lept = batch_lept(ctx, nq ? (int)host[0].log_s : 0);
    if (nq && (e = cudaMemcpy(bt->squares.p, host.data(), nq * sizeof(BatchSquare), cudaMemcpyHostToDevice)) !=
                 cudaSuccess) {
        set_last_error("cudaMemcpy(batch squares)", e);
        return fail(ZODA_ERR_CUDA);
    }
    if ((e = cudaMemcpy(bt->tables.p, tabs.data(), 26 * sizeof(SideTables), cudaMemcpyHostToDevice)) != cudaSuccess) {
        set_last_error("cudaMemcpy(batch tables)", e);
        return fail(ZODA_ERR_CUDA);
    }
    if ((s = set_batch_kernel_attributes()) != ZODA_OK) return fail(s);
    *out = bt;
    return ZODA_OK;
}

zoda_status zoda_batch_run(zoda_batch* bt, void* stream) {
    if (!bt) return ZODA_ERR_ARG;
    zoda_ctx* ctx = bt->ctx;
    ZB_CUDA(cudaSetDevice(ctx->device));
    for (const zoda_square& q : bt->ringed) {
        const zoda_status s = launch_alone(ctx, q, (cudaStream_t)stream);
        if (s != ZODA_OK) return s;
    }
    if (bt->total_tiles == 0 && bt->wide.empty()) return ZODA_OK;
    if (!bt->exec) {
        if (!bt->cap) ZB_CUDA(cudaStreamCreateWithFlags(&bt->cap, cudaStreamNonBlocking));
        const zoda_status s = capture_batch(bt);
        if (s != ZODA_OK) return s;
        ZB_CUDA(cudaGraphInstantiate(&bt->exec, bt->graph, 0));
    }
    ZB_CUDA(cudaGraphLaunch(bt->exec, (cudaStream_t)stream));
    return ZODA_OK;
}

uint64_t zoda_batch_elements(const zoda_batch* bt) { return bt ? bt->elements : 0; }

void zoda_batch_destroy(zoda_batch* bt) {
    if (!bt) return;
    if (bt->ctx) cudaSetDevice(bt->ctx->device);
    cudaDeviceSynchronize();  // a replay may still be running on the caller's stream
    if (bt->exec) cudaGraphExecDestroy(bt->exec);
    if (bt->graph) cudaGraphDestroy(bt->graph);
    if (bt->cap) cudaStreamDestroy(bt->cap);
    bt->squares.release();
    bt->counter.release();
    bt->tables.release();
    delete bt;
}

}  // extern "C"
