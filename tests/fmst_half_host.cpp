// Test harness: the march by half a warp (jdsurfg_b200/csrc/
// swdk_fmst_march.cuh) on the host.  Each of the warp's 32 lanes is a context
// of its own that runs to the next warp function; the warp functions exchange
// values once every lane has come to the same one.  Built by
// tests/test_fmst_half_host.py with -ffp-contract=off.
#include <stdint.h>
#include <ucontext.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <vector>

namespace {

struct Warp {
    ucontext_t home, lane[32];
    std::vector<char> stack[32];
    bool done[32];
    int cur = 0, op = 0;       // running lane; warp functions completed
    int at[32];                // warp functions each lane has entered
    uint32_t val[2][32];       // what the lanes bring, two functions in turn
    std::function<void()> body;
} W;

// every lane has brought v to this warp function
const uint32_t* meet(uint32_t v) {
    const int k = W.at[W.cur]++;
    W.val[k & 1][W.cur] = v;
    const int me = W.cur;
    swapcontext(&W.lane[me], &W.home);
    return W.val[k & 1];
}

struct { unsigned x; } threadIdx;

inline int __ffs(unsigned x) { return __builtin_ffs((int)x); }
inline int __clz(int x) { return x ? __builtin_clz((unsigned)x) : 32; }
inline void __syncwarp() { meet(0); }
unsigned __ballot_sync(unsigned, bool p) {
    const uint32_t* v = meet(p);
    unsigned b = 0;
    for (int i = 0; i < 32; ++i) b |= (v[i] ? 1u : 0u) << i;
    return b;
}
bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
template <class T>
T pick(T x, int src) {
    uint32_t u;
    static_assert(sizeof(T) == 4, "");
    __builtin_memcpy(&u, &x, 4);
    const uint32_t r = meet(u)[src & 31];
    __builtin_memcpy(&x, &r, 4);
    return x;
}
template <class T>
T __shfl_sync(unsigned, T x, int src) { return pick(x, src); }
template <class T>
T __shfl_xor_sync(unsigned, T x, int m) { return pick(x, W.cur ^ m); }

void lane_main() {
    W.body();
    W.done[W.cur] = true;
}

// body on 32 lanes in lockstep; aborts when lanes meet at different functions
void run_warp(std::function<void()> body) {
    W.body = std::move(body);
    for (int i = 0; i < 32; ++i) {
        W.stack[i].resize(256 << 10);
        W.done[i] = false;
        W.at[i] = 0;
        getcontext(&W.lane[i]);
        W.lane[i].uc_stack.ss_sp = W.stack[i].data();
        W.lane[i].uc_stack.ss_size = W.stack[i].size();
        W.lane[i].uc_link = &W.home;
        makecontext(&W.lane[i], lane_main, 0);
    }
    for (;;) {
        int running = 0;
        for (int i = 0; i < 32; ++i) {
            if (W.done[i]) continue;
            W.cur = i;
            threadIdx.x = (unsigned)i;
            swapcontext(&W.home, &W.lane[i]);
            running += !W.done[i];
        }
        if (!running) return;
        if (running != 32) {
            fprintf(stderr, "lanes of a warp parted\n");
            abort();
        }
        W.op++;
    }
}

}  // namespace

#define FM_HOST_WARP 1
struct float4;
static inline float4 make_float4(float x, float y, float z, float w);
#include "swdk_fmst_march.cuh"
static inline float4 make_float4(float x, float y, float z, float w) { return float4{x, y, z, w}; }

using namespace swdk_fmst_march;

// Two heaps of n[0] and n[1] entries (keys, heap-ordered), one per half; ops
// values: a value that is not NaN joins the heap, NaN takes the root off.
// half 1 stops after nops1 operations.  The heap's keys and nodes after each
// half's operations by half a warp must be those of addtree / downtree;
// returns the number of entries or node positions that differ.
extern "C" int fm_half_heap(const int* n, const float* keys0, const float* keys1, const float* ops, int nops,
                            int nops1, int cap) {
    const int ld = 512;
    std::vector<FHeap> heap[2], ref[2];
    std::vector<FNode> nd[2], rnd[2];
    March M[2], R[2];
    int fresh[2];
    for (int h = 0; h < 2; ++h) {
        const float* keys = h ? keys1 : keys0;
        const int N = n[h] + nops + 1;
        const int nx = (N + ld - 1) / ld + 1;
        heap[h].assign((size_t)cap + 2, FHeap{0.0f, 0});
        nd[h].assign((size_t)nx * ld, FNode{0.0f, -1});
        for (int i = 1; i <= n[h]; ++i) {
            heap[h][i] = FHeap{keys[i - 1], ((i - 1) % ld) | ((i - 1) / ld) << 16};
            nd[h][i - 1] = FNode{keys[i - 1], i};
        }
        fresh[h] = n[h];
        ref[h] = heap[h];
        rnd[h] = nd[h];
        M[h] = March{};
        M[h].heap = heap[h].data();
        M[h].nd = nd[h].data();
        M[h].ld = ld;
        M[h].nnx = nx;
        M[h].nnz = ld;
        M[h].cap = cap;
        M[h].ntr = n[h];
        R[h] = M[h];
        R[h].heap = ref[h].data();
        R[h].nd = rnd[h].data();
    }
    March L[32];
    for (int i = 0; i < 32; ++i) L[i] = M[i >> 4];
    int first[2] = {fresh[0], fresh[1]};
    run_warp([&]() {
        const int lane = (int)threadIdx.x, half = lane >> 4, l = lane & 15, sh = lane & 16;
        March& m = L[lane];
        const int lv = l ? 31 - __clz(l) : 0;
        unsigned amask = 0, rmask = 0;
        for (int c = l; c > 1; c >>= 1) {
            amask |= 1u << (c >> 1);
            if (c & 1) rmask |= 1u << (c >> 1);
        }
        int next = first[half];
        for (int k = 0; k < nops; ++k) {
            const bool on = half == 0 || k < nops1;
            const float key = ops[k];
            if (key != key) {
                m.down_half(on && m.ntr > 0, l, sh, lv, amask, rmask);
            } else {
                const int pk = (next % ld) | (next / ld) << 16, node = next;
                const bool added = m.grow_half(on, node, key, l);
                if (cap >= 65536) m.sift_up_half<true>(added, m.ntr, pk, node, key, l, sh);
                else m.sift_up_half<false>(added, m.ntr, pk, node, key, l, sh);
                if (on) ++next;
            }
        }
    });
    int bad = 0;
    for (int h = 0; h < 2; ++h) {
        March& r = R[h];
        int next = fresh[h];
        for (int k = 0; k < (h ? nops1 : nops); ++k) {
            const float key = ops[k];
            if (key != key) {
                if (r.ntr > 0) r.downtree();
            } else {
                rnd[h][next].t = key;
                r.addtree((next % ld) | (next / ld) << 16, key);
                ++next;
            }
        }
        const March& m = L[16 * h];
        bad += m.ntr != r.ntr || m.overflow != r.overflow || m.ntr_max != r.ntr_max;
        for (int i = 1; i <= r.ntr; ++i) {
            bad += __float_as_int(heap[h][i].key) != __float_as_int(ref[h][i].key) ||
                   heap[h][i].node != ref[h][i].node;
            const int q = r.lin(ref[h][i].node);
            bad += nd[h][q].s != rnd[h][q].s;
        }
    }
    return bad;
}

// the same bits; any NaN is as good as another
static bool same(float a, float b) { return (a != a && b != b) || __float_as_int(a) == __float_as_int(b); }

// npairs sources on one map, marched two per warp (the last of an odd number
// alone) and one by one (mode 0): the number of propagation-grid nodes whose
// time or status differs, plus differing pair outcomes.  cap: heap entries of
// the propagation grid (0: the full heap); shared: the heaps where the device
// keeps them in shared memory (both grids then hold cap entries).  out:
// {overflowed pairs, largest band}.
extern "C" int fm_half_pairs(int nx, int ny, float goxd, float gozd, float dvxd, float dvzd, int npairs,
                             const float* srcx, const float* srcz, const double* map, int cap, int shared, int* out) {
    const Grid G = make_grid(nx, ny, goxd, gozd, dvxd, dvzd);
    std::vector<float> risti_c, risti_r;
    make_risti(G, risti_c, risti_r);
    const size_t N = (size_t)G.nnx * G.nnz, F = (size_t)RMAX * RMAX;
    if (cap <= 0) cap = (int)std::lround(0.5f * (float)(G.nnx * G.nnz));
    const bool deep = cap >= 65536;
    const int hs = (cap + 2) & ~1;
    std::vector<float> slwn(N);
    for (int stx = 1; stx <= G.nnx; ++stx)
        for (int stz = 1; stz <= G.nnz; ++stz)
            slwn[(stz - 1) + (size_t)(stx - 1) * G.nnz] = 1.0f / dice_node(map, G, stz, stx);
    std::vector<FNode> coarse[2];
    std::vector<PairGeo> geo[2];
    std::vector<int32_t> zero(npairs, 0);
    unsigned int cnt[2][2] = {{0, 0}, {0, 0}};
    for (int side = 0; side < 2; ++side) {
        coarse[side].assign(N * npairs, FNode{0.0f, -1});
        geo[side].resize(npairs);
        std::vector<FNode> fine(F * npairs);
        std::vector<FHeap> heap((size_t)hs * npairs), fheap((size_t)(RCAP + 1) * npairs), sheap(2 * (size_t)hs);
        std::vector<float> rvel(F * npairs), rslw(F * npairs);
        for (int p = 0; p < npairs; ++p) {
            PairGeo& g = geo[side][p];
            g = pair_geometry(G, srcx[p], srcz[p]);
            if (g.status) continue;
            for (int a = 1; a <= g.nrnx; ++a)
                for (int b = 1; b <= g.nrnz; ++b) {
                    const size_t i = F * p + (b - 1) + (size_t)(a - 1) * RMAX;
                    rvel[i] = refine_node(map, G, g, a, b);
                    rslw[i] = 1.0f / rvel[i];
                }
        }
        Scratch S;
        S.coarse = coarse[side].data();
        S.heap = heap.data();
        S.fine = fine.data();
        S.rvel = rvel.data();
        S.rslw = rslw.data();
        S.fheap = fheap.data();
        S.geo = geo[side].data();
        S.N = N;
        S.cap = cap;
        S.hstride = hs;
        if (side == 0) {
            for (int p = 0; p < npairs; ++p)
                march_pair(G, p, p, srcx, srcz, zero.data(), slwn.data(), risti_c.data(), risti_r.data(), S, cnt[0],
                           shared ? sheap.data() : nullptr, cap, 0, 0, 1u);
        } else {
            for (int p0 = 0; p0 < npairs; p0 += 2)
                run_warp([&]() {
                    const int half = (int)threadIdx.x >> 4;
                    const bool mine = p0 + half < npairs;
                    const int p = mine ? p0 + half : p0;
                    const unsigned mask = mine ? 0xffffu << (16 * half) : 0u;
                    if (shared)
                        march_pair<1>(G, p, p, srcx, srcz, zero.data(), slwn.data(), risti_c.data(), risti_r.data(),
                                      S, cnt[1], sheap.data() + (size_t)half * hs, cap, 2, threadIdx.x & 15, mask);
                    else if (deep)
                        march_pair<2>(G, p, p, srcx, srcz, zero.data(), slwn.data(), risti_c.data(), risti_r.data(),
                                      S, cnt[1], nullptr, 0, 2, threadIdx.x & 15, mask);
                    else
                        march_pair<0>(G, p, p, srcx, srcz, zero.data(), slwn.data(), risti_c.data(), risti_r.data(),
                                      S, cnt[1], nullptr, 0, 2, threadIdx.x & 15, mask);
                });
        }
    }
    int bad = 0;
    for (int p = 0; p < npairs; ++p) {
        bad += geo[0][p].status != geo[1][p].status;
        if (geo[0][p].status) continue;  // an overflowed band's grid is marched again
        for (size_t i = N * p; i < N * (p + 1); ++i)
            bad += !same(coarse[0][i].t, coarse[1][i].t) || coarse[0][i].s != coarse[1][i].s;
    }
    bad += cnt[0][0] != cnt[1][0] || cnt[0][1] != cnt[1][1];
    out[0] = (int)cnt[0][0];
    out[1] = (int)cnt[0][1];
    return bad;
}
