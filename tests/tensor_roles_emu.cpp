// Runs the role code of k_tensor_passes (csrc/tensorpass.cuh) on the CPU: every thread of
// one CTA is a fiber, mbarriers, tensor memory, TMA and the asynchronous products are
// modelled, and the order in which warps run is chosen by the caller. A warp can be made to
// lag: it runs only when no other one can. The kernel's text is compiled as it is;
// test_tensor_roles.py removes its inline-PTX helpers, which are restated here.
#include <ucontext.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <memory>
#include <random>
#include <vector>

#define __host__
#define __device__
#define __global__
#define __shared__
#define __constant__ static
#define __forceinline__ inline
#define __restrict__
#define __grid_constant__
#define __align__(n)
#define __launch_bounds__(...)

struct uint2 { uint32_t x, y; };
struct int2 { int32_t x, y; };
struct uint4 { uint32_t x, y, z, w; };
struct int4 { int32_t x, y, z, w; };
inline uint32_t min(uint32_t a, uint32_t b) { return a < b ? a : b; }
inline uint32_t __viaddmin_u32(uint32_t a, uint32_t b, uint32_t c) { return min(a + b, c); }
inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)((uint64_t)a * b >> 32); }
inline int __popc(uint32_t x) { return __builtin_popcount(x); }

struct CUtensorMap {
    unsigned char* base;
    uint64_t dim[3], stride[2];  // elements; bytes of the two outer dimensions
    uint32_t box[3];
};

// ---- fibers --------------------------------------------------------------------------
namespace emu {
[[noreturn]] void die(const char* what) {
    fprintf(stderr, "tensor_roles_emu: %s\n", what);
    fflush(stderr);
    _Exit(3);
}
constexpr size_t STACK = 64 << 10;
struct Fiber {
    ucontext_t uc;
    std::unique_ptr<char[]> stack;
    bool done = false;
    std::function<bool()> ready;  // empty: runnable
};
struct Group {  // threads that meet: a warp or the CTA
    int size = 0, count = 0;
    uint64_t gen = 0;
    std::vector<uint32_t> in, out;
};
struct Block {
    std::vector<Fiber> f;
    std::vector<Group> warp;
    Group all;
    ucontext_t sched;
    int cur = 0;
    std::mt19937 rng;
    std::vector<std::function<void()>> loads;  // TMA loads in flight, any order
    std::deque<std::function<void()>> tensor;  // products and commits, in order
    std::deque<std::vector<std::function<void()>>> stores;  // committed groups of the copier
    std::vector<std::function<void()>> open;
    std::vector<uint32_t> tmem = std::vector<uint32_t>(128 * 512, 0xDEADBEEFu);
} *B;

void switch_out() { swapcontext(&B->f[B->cur].uc, &B->sched); }
void wait_for(std::function<bool()> p) {
    if (p()) return;
    B->f[B->cur].ready = std::move(p);
    switch_out();
}
void yield() {
    B->f[B->cur].ready = [] { return true; };
    switch_out();
}
uint32_t lane() { return (uint32_t)B->cur & 31; }
std::vector<uint32_t>& meet(Group& g, int i, uint32_t v) {
    g.in[i] = v;
    if (++g.count == g.size) {
        g.out = g.in;
        g.count = 0;
        g.gen++;
    } else {
        const uint64_t gen = g.gen;
        wait_for([&g, gen] { return g.gen != gen; });
    }
    return g.out;
}
std::vector<uint32_t>& meet_warp(uint32_t v) { return meet(B->warp[B->cur / 32], B->cur % 32, v); }

std::function<void()> g_entry;
void trampoline() {
    g_entry();
    B->f[B->cur].done = true;
    switch_out();
}
}  // namespace emu
struct Idx3 { uint32_t x; };
static Idx3 threadIdx;

inline bool __all_sync(uint32_t, bool p) {
    for (uint32_t v : emu::meet_warp(p)) if (!v) return false;
    return true;
}
inline bool __any_sync(uint32_t, bool p) {
    for (uint32_t v : emu::meet_warp(p)) if (v) return true;
    return false;
}
inline uint32_t __ballot_sync(uint32_t, bool p) {
    uint32_t m = 0, i = 0;
    for (uint32_t v : emu::meet_warp(p)) m |= (v ? 1u : 0u) << i++;
    return m;
}
inline uint32_t __shfl_sync(uint32_t, uint32_t v, int src) { return emu::meet_warp(v)[src]; }
inline void __syncwarp() { emu::meet_warp(0); }
inline void __syncthreads() { emu::meet(emu::B->all, emu::B->cur, 0); }
inline void __threadfence() {}
inline uint32_t atomicAdd(uint32_t* p, uint32_t v) {
    const uint32_t o = *p;
    *p += v;
    return o;
}
inline void atomicOr(int* p, int v) { *p |= v; }
inline void __stcs(uint32_t* p, uint32_t v) { *p = v; }
inline void emu_fence() {}

#include "emu_field.inc"  // csrc/field.cuh

namespace zb {
alignas(1024) unsigned char smem[256 << 10];
inline uint32_t smem_u32(const void* p) { return (uint32_t)((const unsigned char*)p - smem); }

// ---- mbarriers -----------------------------------------------------------------------
struct MBar {
    uint8_t init, pend, phase, pad;
    int32_t tx;
};
inline MBar* mb(uint64_t* b) { return reinterpret_cast<MBar*>(b); }
inline void mb_check(MBar* m) {
    if (m->pend == 0 && m->tx == 0) {
        m->phase ^= 1;
        m->pend = m->init;
    }
}
inline void mb_arrive(MBar* m) {
    if (m->pend == 0) emu::die("more arrivals in a phase than the barrier expects");
    m->pend--;
    mb_check(m);
}
inline void mbar_init(uint64_t* b, uint32_t n) { *mb(b) = MBar{(uint8_t)n, (uint8_t)n, 0, 0, 0}; }
inline void fence_mbar_init() {}
inline void mbar_arrive(uint64_t* b) {
    mb_arrive(mb(b));
    emu::yield();
}
inline void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
    mb(b)->tx += (int32_t)bytes;
    mb_arrive(mb(b));
}
inline void mb_complete(uint64_t* b, uint32_t bytes) {
    mb(b)->tx -= (int32_t)bytes;
    mb_check(mb(b));
}
inline bool mbar_try_wait(uint64_t* b, uint32_t parity) { return mb(b)->phase != (parity & 1); }
inline bool tp_wait1(uint64_t* b, uint32_t parity) {
    emu::wait_for([=] { return mbar_try_wait(b, parity); });
    return true;
}
inline bool tp_wait_count(const uint32_t* p, uint32_t need) {
    emu::wait_for([=] { return *p >= need; });
    return true;
}
template <int STEP>
inline void tp_store8(uint32_t* p, const uint32_t (&r)[8]) {
    for (int u = 0; u < 8; u++) p[u * (STEP / 4)] = r[u];
}

// ---- copies --------------------------------------------------------------------------
inline void box_copy(const CUtensorMap& m, int x, int y, int z, unsigned char* s, bool load) {
    for (uint32_t c = 0; c < m.box[2]; c++)
        for (uint32_t b = 0; b < m.box[1]; b++)
            for (uint32_t a = 0; a < m.box[0]; a++, s += 4) {
                const uint64_t X = x + a, Y = y + b, Z = z + c;
                const bool in = X < m.dim[0] && Y < m.dim[1] && Z < m.dim[2];
                unsigned char* g = m.base + X * 4 + Y * m.stride[0] + Z * m.stride[1];
                if (load) {
                    if (in) memcpy(s, g, 4);
                    else memset(s, 0, 4);
                } else if (in) {
                    memcpy(g, s, 4);
                }
            }
}
inline void bulk_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    emu::B->loads.push_back([=] {
        memcpy(dst, src, bytes);
        mb_complete(bar, bytes);
    });
}
inline void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    if (x % 4) emu::die("TMA column not on a 16-byte boundary");
    const CUtensorMap m = *map;
    emu::B->loads.push_back([=] {
        box_copy(m, x, y, z, (unsigned char*)dst, true);
        mb_complete(bar, m.box[0] * m.box[1] * m.box[2] * 4);
    });
}
inline uint64_t l2_evict_first() { return 0; }
inline void tma_load_3d_hint(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar, uint64_t) {
    tma_load_3d(dst, map, x, y, z, bar);
}
// a store reads its shared memory as late as it may: when its group is waited for
inline void tma_store_3d_hint(const CUtensorMap* map, int x, int y, int z, const void* src, uint64_t) {
    const CUtensorMap m = *map;
    emu::B->open.push_back([=] { box_copy(m, x, y, z, (unsigned char*)src, false); });
}
inline void bulk_commit() {
    emu::B->stores.push_back(std::move(emu::B->open));
    emu::B->open.clear();
}
inline void bulk_wait_n(size_t left) {
    while (emu::B->stores.size() > left) {
        for (auto& f : emu::B->stores.front()) f();
        emu::B->stores.pop_front();
    }
}
inline void bulk_wait_read0() { bulk_wait_n(0); }
inline void bulk_wait_read1() { bulk_wait_n(1); }
inline void bulk_wait0() { bulk_wait_n(0); }

// ---- tensor memory and products --------------------------------------------------------
inline void tc_alloc(uint32_t* slot, uint32_t) { *slot = 0; }
inline void tc_dealloc(uint32_t, uint32_t) {}
inline void tc_fence_before() {}
inline void tc_fence_after() {}
inline uint32_t* tmem_row(uint32_t addr) {
    const uint32_t w = (uint32_t)emu::B->cur / 32;
    if (addr >> 16 != 32 * (w % 4)) emu::die("tensor-memory lanes of another warp");
    return emu::B->tmem.data() + ((addr >> 16) + emu::lane()) * 512 + (addr & 0xFFFF);
}
inline void tc_ld(uint32_t (&r)[32], uint32_t addr) { memcpy(r, tmem_row(addr), 128); }
inline void tc_st(uint32_t addr, const uint32_t (&r)[32]) { memcpy(tmem_row(addr), r, 128); }
inline void tc_wait_st() { emu::yield(); }
inline void tc_mma_i8_ta(uint32_t d, uint32_t a, uint64_t desc, uint32_t, bool accumulate) {
    emu::B->tensor.push_back([=] {
        const uint32_t base = (uint32_t)(desc & 0x3FFF) << 4, lbo = (uint32_t)(desc >> 16 & 0x3FFF) << 4,
                       sbo = (uint32_t)(desc >> 32 & 0x3FFF) << 4;
        static int32_t bt[32][128];
        for (int n = 0; n < 128; n++)
            for (int k = 0; k < 32; k++)
                bt[k][n] = (int8_t)smem[base + (k / 16) * lbo + (n / 8) * sbo + (n % 8) * 16 + k % 16];
        for (int m = 0; m < 128; m++) {
            uint32_t* row = emu::B->tmem.data() + m * 512;
            int32_t* dst = (int32_t*)row + (d & 0xFFFF);
            if (!accumulate) memset(dst, 0, 512);
            const uint8_t* src = (const uint8_t*)(row + (a & 0xFFFF));
            for (int k = 0; k < 32; k++) {
                const int32_t v = src[k];
                for (int n = 0; n < 128; n++) dst[n] += v * bt[k][n];
            }
        }
    });
}
inline void tc_commit(uint64_t* bar) {
    emu::B->tensor.push_back([=] { mb_arrive(mb(bar)); });
}
}  // namespace zb

#include "emu_kernel.inc"  // csrc/tcgen05.cuh (digits and descriptors), csrc/tensorpass.cuh, the host tables

namespace zb {
CUtensorMap map3(void* base, uint64_t cols, uint64_t n2, uint64_t n1, uint64_t pitch, uint64_t block, uint32_t box2,
                 uint32_t box1) {
    return CUtensorMap{(unsigned char*)base, {cols, n2, n1}, {pitch * 4, block * pitch * 4}, {TP_BOX, box2, box1}};
}

// The extension's map over [2^L][cols] -> out [2^(L+1)][cols], one CTA. `lag`: the warp that
// runs only when no other can, or -1. Returns 0; 1: a role flagged an error, 2: nothing can run.
template <int L1, int L2>
int run(uint32_t seed, int lag, uint32_t* in, uint32_t* out, uint32_t cols) {
    using G = TPassGeom<L1, L2>;
    constexpr int L = L1 + L2;
    constexpr uint32_t S = 1u << L;
    std::vector<uint8_t> tab;
    if (!tensor_tables_host(L, root_of_unity(L + 1), false, &tab)) return 3;
    const Blob bl(L);
    TensorArgs a{};
    a.nchunks = (cols + G::CW - 1) / G::CW;
    a.depth = 1;
    a.slots = a.nchunks < 4 ? a.nchunks : 4;
    std::vector<uint32_t> ring((size_t)a.slots * G::SLOT, 0x55555555u), counters(1 + 3 * a.nchunks, 0);
    int err = 0;
    a.in = in;
    a.in_pitch = cols;
    a.in_rows = S;
    a.copy = out;
    a.copy_pitch = 2 * cols;
    a.copy_rows = S;
    a.out = out + cols;
    a.out_pitch = 2 * cols;
    a.out_rows = S;
    a.cols = cols;
    a.mat_a = (const uint4*)(tab.data() + bl.mat_a);
    a.mat_m = (const uint4*)(tab.data() + bl.mat_m);
    a.fac_a = (const int2*)(tab.data() + bl.fac_a);
    a.fac_m = (const int2*)(tab.data() + bl.fac_m);
    a.ring = ring.data();
    a.counters = counters.data();
    a.err = &err;
    TensorMaps maps;
    maps.in[0] = maps.in[1] = map3(in, cols, G::N2, G::N1, cols, G::N2, 1, 32);
    maps.copy[0] = maps.copy[1] = map3(out, cols, G::N2, G::N1, 2 * cols, G::N2, 1, 32);
    maps.ring_m = map3(ring.data(), G::CW, G::N2, (uint64_t)a.slots * G::N1, G::CW, G::N2, 32, 1);
    maps.ring_b = map3(ring.data(), G::CW, G::N2, (uint64_t)a.slots * G::N1, G::CW, G::N2, 1, 32);

    using namespace emu;
    Block blk;
    B = &blk;
    blk.rng.seed(seed);
    constexpr int NW = TP_THREADS / 32;
    blk.warp.resize(NW);
    auto group = [](Group& g, int n) {
        g.size = n;
        g.in.assign(n, 0);
        g.out.assign(n, 0);
    };
    for (auto& w : blk.warp) group(w, 32);
    group(blk.all, TP_THREADS);
    blk.f.resize(TP_THREADS);
    g_entry = [&] { k_tensor_passes<L1, L2, false, 0>(a, maps); };
    for (auto& f : blk.f) {
        f.stack.reset(new char[STACK]);
        getcontext(&f.uc);
        f.uc.uc_stack.ss_sp = f.stack.get();
        f.uc.uc_stack.ss_size = STACK;
        f.uc.uc_link = nullptr;
        makecontext(&f.uc, trampoline, 0);
    }
    std::vector<int> order(NW);
    for (int i = 0; i < NW; i++) order[i] = i;
    auto run_warp = [&](int w) {
        bool any = false;
        for (int t = 32 * w; t < 32 * w + 32; t++) {
            Fiber& f = blk.f[t];
            if (f.done || (f.ready && !f.ready())) continue;
            f.ready = nullptr;
            blk.cur = t;
            threadIdx.x = (uint32_t)t;
            swapcontext(&blk.sched, &f.uc);
            any = true;
        }
        return any;
    };
    for (int left = 1; left;) {
        std::shuffle(order.begin(), order.end(), blk.rng);
        bool any = false;
        for (int w : order)
            if (w != lag) any |= run_warp(w);
        for (size_t n = blk.rng() % 4 + (any ? 0 : 1); n && !blk.loads.empty(); n--) {
            std::swap(blk.loads[blk.rng() % blk.loads.size()], blk.loads.back());
            auto f = std::move(blk.loads.back());
            blk.loads.pop_back();
            f();
            any = true;
        }
        for (size_t n = blk.rng() % 6 + (any ? 0 : 1); n && !blk.tensor.empty(); n--) {
            auto f = std::move(blk.tensor.front());
            blk.tensor.pop_front();
            f();
            any = true;
        }
        if (!any && lag >= 0) any = run_warp(lag);
        left = 0;
        for (auto& f : blk.f) left += !f.done;
        if (!any && left) return 2;
    }
    return err ? 1 : 0;
}
}  // namespace zb

extern "C" int tensor_roles_run(int log_s, uint32_t seed, int lag, uint32_t* in, uint32_t* out, uint32_t cols) {
    if (log_s == 11) return zb::run<5, 6>(seed, lag, in, out, cols);
    return log_s == 12 ? zb::run<6, 6>(seed, lag, in, out, cols) : 4;
}
extern "C" int tensor_roles_first_operand_warp() { return zb::TP_W_CONV; }
