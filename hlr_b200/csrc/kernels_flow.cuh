// A one-vector FP64 product as one launch.
//
// Small products are chains of short dependent passes: with a launch per pass
// the host's launch rate (3 to 6 us each, plus the events of the near field's
// side stream) sets their time.  Measured at n = 8192 (1D log, 19 MB, L2
// resident): 28 us with a launch per pass, 14 us as one launch, of which 13 us
// on the device: four hand-overs of about 2 us (ticket, descriptor and data
// loads, completion count).  Here resident CTAs take work items (an output tile, an input tile, a few
// finish groups) from two queues: the passes of the chain in order, and the
// near field D x (op T / C: the tile T-form of D^T x), which depends on nothing
// but x.  An item of pass s waits
// until every item of the pass before it is done; it loads its descriptors
// and its first matrix columns before that wait.  Part of the CTAs start on
// the near field; the pass that adds to y after it (op T / C: its finish) drains
// that queue first and then waits for it.
//
// Progress.  A queue is a counter: tickets are taken in pass order, so the
// items an item waits for are held by CTAs that already run, whatever part of
// the grid is resident; no co-residency is needed.  Every wait is bounded
// (wait_ns): one that runs out sets bit 0 of the error word and a stop mark
// on which all CTAs leave.
//
// Counters.  Each counter holds the number of the product that uses it above
// FLOW_CNT_BITS bits of count.  A product's number is larger than those before
// it on the same counters, and every CTA first raises the counters to it
// (atomicMax), so whatever an earlier product left there, one that gave up or
// products that wrongly overlapped on one workspace, reads as zero.  A ticket
// of another number means such an overlap: the CTA reports it (bit 0) and
// leaves, as it does for a ticket out of range.
//
// Vectors written in the launch are read through L2 (__ldcg): L1 is not
// coherent with other SMs' writes.  The sums are those of the separate
// kernels (kernels_f64.cuh), in the same order.
#pragma once

#include <cuda_runtime.h>

#include "kernels_f64.cuh"
#include "layout.hpp"

namespace hlrc {

constexpr int FLOW_MAXST = 12;        // passes of a product
constexpr int FLOW_CTRS = 3 + FLOW_MAXST;   // tickets (main, side), stop mark; items done per pass
constexpr int FLOW_CNT_BITS = 20;     // count of a counter (5.6 years of products of 10 us for the number above it)
constexpr unsigned long long FLOW_CNT_MASK = (1ull << FLOW_CNT_BITS) - 1;
constexpr int FLOW_CTAS = 2;          // CTAs per SM: 128 registers (three: 80, spills, 33 us against 25 us at n = 8192)

enum : int32_t { FLOW_N = 0, FLOW_TT = 1, FLOW_FINISH = 2, FLOW_T = 3, FLOW_TFINISH = 4 };

struct FlowStage {
    const void* items;     // NSeg / TTSeg / TGroup / TUnit
    const void* data;      // NChunk / TTChunk / - / TSlab
    int32_t kind;
    int32_t n;             // segments, groups or units
    int32_t per;           // of them per item (finish, unit T-form: one per warp and round)
    int32_t nitems;
    int32_t first;         // first ticket of the pass in its queue
    int32_t dep;           // the pass that has to be done first (-1: none)
    int32_t join;          // the near-field pass to wait for as well (-1: none)
    int8_t in, vt, out, add;   // VecName of inputs and output (4, 5: partial sums; vt: those of T-forms and finishes);
                               // add: 0 set, 1 add alpha * s, 2 add s
};
static_assert(sizeof(FlowStage) == 48, "FlowStage is 48 bytes");

struct FlowArgs {
    FlowStage st[FLOW_MAXST];        // in the kernel's parameters: no loads, no copy at upload
    int nst, side;                   // passes; the near-field pass (-1: none)
    int main_items, side_items;
    int main_ctas;                   // CTAs that start on the chain
    const double* A;
    double* v[6];                    // by VecName; [4] the partial sums, [5] those of a side pass
    double alpha;
    unsigned long long* ctr;
    unsigned long long base;         // the product's number << FLOW_CNT_BITS
    int* err;
    uint64_t wait_ns;
    int skip;                        // test hook: the first item of the chain is never counted as done
};

// N-form of one output tile by a CTA of W warps, the sums of k_nform_f64 in the
// same order (the separate kernel keeps its own loop: with the first chunk
// loaded ahead it measured 6 % slower).  ready() is
// called once, by every thread, when the descriptors and the first matrix
// columns are under way and before any vector is touched; false: the tile is
// left.
template <int W, typename Ready>
__device__ __forceinline__ void flow_nform(const NSeg& sg, const NChunk* __restrict__ chunks,
                                           const double* __restrict__ A, const double* vx, const double* vt, double* out,
                                           double alpha, int add, double (&red)[W][TILE], Ready&& ready) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = 2 * lane;
    const bool active = r < sg.ld;
    double acc0 = 0.0, acc1 = 0.0;
    double2 m[NCHUNK];
    auto load = [&](const NChunk& ch) {
        const double* a = A + ch.a_off + r;
#pragma unroll
        for (int j = 0; j < NCHUNK; ++j)
            m[j] = active && j < ch.nc ? ld_stream(a + size_t(j) * sg.ld) : make_double2(0.0, 0.0);
    };
    auto add_chunk = [&](const NChunk& ch) {
        const double* v = (ch.v_off & VEC_T) ? vt + (ch.v_off & ~VEC_T) : vx + ch.v_off;
        double vv[NCHUNK];
#pragma unroll
        for (int j = 0; j < NCHUNK; ++j) vv[j] = j < ch.nc ? __ldcg(v + j) : 0.0;
#pragma unroll
        for (int j = 0; j < NCHUNK; ++j) {
            acc0 = fma(m[j].x, vv[j], acc0);
            acc1 = fma(m[j].y, vv[j], acc1);
        }
    };
    uint32_t c = sg.cb + warp;
    NChunk ch{0, 0, 0, 0};
    if (c < sg.ce) {
        ch = chunks[c];
        load(ch);
    }
    if (!ready()) return;
    vx = past(vx);
    vt = past(vt);
    if (c < sg.ce) {
        add_chunk(ch);
        for (c += W; c < sg.ce; c += W) {
            ch = chunks[c];
            load(ch);
            add_chunk(ch);
        }
    }
    red[warp][r] = acc0;
    red[warp][r + 1] = acc1;
    __syncthreads();
    if (threadIdx.x < sg.rows) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < W; ++w) s += red[w][threadIdx.x];
        double* o = out + sg.out + threadIdx.x;
        if (add) *o = ld_out(o) + alpha * s;
        else *o = s;
    }
}

// Tile T-form of one input tile by a CTA of W warps, as k_ttform_f64.  ready()
// as in flow_nform.
template <int W, typename Ready>
__device__ __forceinline__ void flow_ttform(const TTSeg& sg, const TTChunk* __restrict__ chunks,
                                            const double* __restrict__ A, const double* vin, double* out, double* part,
                                            double alpha, int add, Ready&& ready) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = 2 * lane;
    const bool active = r < sg.ld;
    // software pipeline: the loads of chunk c + W are issued before chunk c
    // is reduced and written; descriptors are fetched two iterations ahead
    uint32_t c = sg.cb + warp;
    TTChunk cur{0, 0, 0, 0}, nxt{0, 0, 0, 0};
    if (c < sg.ce) cur = chunks[c];
    if (c + W < sg.ce) nxt = chunks[c + W];
    double2 m[TCOLS];
    auto issue = [&](const TTChunk& q) {
        const double* a = A + q.a_off + r;
#pragma unroll
        for (int j = 0; j < TCOLS; ++j)
            m[j] = (active && j < q.nc) ? ld_stream(a + size_t(j) * sg.ld) : make_double2(0.0, 0.0);
    };
    issue(cur);
    if (!ready()) return;
    if (c >= sg.ce) return;
    vin = past(vin);
    const double v0 = (r < sg.rows) ? __ldcg(vin + sg.v_off + r) : 0.0;
    const double v1 = (r + 1 < sg.rows) ? __ldcg(vin + sg.v_off + r + 1) : 0.0;
    for (; c < sg.ce; c += W) {
        double p[TCOLS];
#pragma unroll
        for (int j = 0; j < TCOLS; ++j) p[j] = fma(m[j].y, v1, m[j].x * v0);
        const TTChunk ch = cur;
        if (c + W < sg.ce) {
            cur = nxt;
            issue(cur);
            if (c + 2 * W < sg.ce) nxt = chunks[c + 2 * W];
        }
        TransposeReduce<TCOLS, 16>::run(p, lane);
        constexpr int SH = 5 - Log2<TCOLS>::v;
        const int col = lane >> SH;
        if ((lane & ((1 << SH) - 1)) == 0 && col < ch.nc) {
            if (ch.flags & TT_DIRECT) {
                double* o = out + ch.out + col;
                if (add) *o = ld_out(o) + alpha * p[0];
                else *o = p[0];
            } else {
                part[ch.out + col] = p[0];
            }
        }
    }
}

__device__ __forceinline__ unsigned long long flow_load(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__global__ void __launch_bounds__(256, FLOW_CTAS)
k_flow_f64(const __grid_constant__ FlowArgs a) {
    constexpr int W = 8;
    __shared__ double red[W][TILE];
    __shared__ int s_item[2];
    __shared__ int s_ok[2];
    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_wait();
    unsigned long long* const stop = a.ctr + 2;
    unsigned long long* const done = a.ctr + 3;
    if (threadIdx.x < FLOW_CTRS && threadIdx.x != 2) atomicMax(a.ctr + threadIdx.x, a.base);
    __syncthreads();
    int flip = 0, flip_ok = 0;   // a slot is written again only two barriers later
    bool ok = true;          // no wait ran out (the same in every thread)
    uint32_t seen = 0;       // passes known to be done
    // the next ticket of queue q (0 chain, 1 near field); -1: not one of this product
    auto take = [&](int q) {
        flip ^= 1;
        if (threadIdx.x == 0) {
            const unsigned long long v = atomicAdd(a.ctr + q, 1ull), num = v & ~FLOW_CNT_MASK;
            if (num != a.base) {   // another product runs on these counters: its ticket is lost as well
                atomicOr(a.err, 1);
                atomicExch(stop, num);
            }
            s_item[flip] = num == a.base ? int(v & FLOW_CNT_MASK) : -1;
        }
        __syncthreads();
        return s_item[flip];
    };
    // waits for pass d (every thread of the CTA)
    auto wait_one = [&](int d) {
        if (d < 0 || (seen >> d & 1u) || !ok) return;
        flip_ok ^= 1;
        if (threadIdx.x == 0) {
            const unsigned long long want = a.base + unsigned(a.st[d].nitems);
            bool good = true;
            if (flow_load(done + d) < want) {
                const uint64_t t0 = tree_clock();
                for (uint32_t i = 1; flow_load(done + d) < want; ++i) {
                    if ((i & 15u) != 0u) continue;
                    if (flow_load(stop) == a.base) {
                        atomicOr(a.err, 1);   // marked by this product, or by another that took its ticket
                        good = false;
                        break;
                    }
                    if (tree_clock() - t0 > a.wait_ns) {
                        atomicOr(a.err, 1);
                        atomicExch(stop, a.base);
                        good = false;
                        break;
                    }
                }
            }
            s_ok[flip_ok] = good;
        }
        __syncthreads();
        ok = s_ok[flip_ok] != 0;
        seen |= 1u << d;
    };
    auto run = [&](int s, int item) {
        const FlowStage& p = a.st[s];
        auto ready = [&]() {
            wait_one(p.dep);
            wait_one(p.join);
            return ok;
        };
        const double* in = a.v[p.in];
        double* out = a.v[p.out];
        const double alpha = p.add == 2 ? 1.0 : a.alpha;
        if (p.kind == FLOW_N) {
            const NSeg sg = static_cast<const NSeg*>(p.items)[item];
            flow_nform<W>(sg, static_cast<const NChunk*>(p.data), a.A, in, a.v[p.vt], out, alpha, p.add != 0, red,
                          ready);
        } else if (p.kind == FLOW_TT) {
            const TTSeg sg = static_cast<const TTSeg*>(p.items)[item];
            flow_ttform<W>(sg, static_cast<const TTChunk*>(p.data), a.A, in, out, a.v[p.vt], alpha, p.add != 0, ready);
        } else {
            const int e = min(p.n, (item + 1) * p.per);
            int i = item * p.per + warp;
            TGroup g{};   // the first descriptor comes before the wait (units are as large)
            static_assert(sizeof(TGroup) == sizeof(TUnit), "one descriptor size");
            if (i < e) g = static_cast<const TGroup*>(p.items)[i];
            const bool go = ready();
            in = past(in);
            double* const part = past(a.v[p.vt]);
            while (go && i < e) {
                if (p.kind == FLOW_FINISH) {
                    ttfinish_group<true>(g, part, out, alpha, p.add != 0, lane);
                } else if (p.kind == FLOW_TFINISH) {
                    tfinish_group<true>(g, part, out, alpha, p.add != 0, lane);
                } else {
                    TUnit u;
                    memcpy(&u, &g, sizeof(u));
                    tform_unit<TCOLS, true>(u, static_cast<const TSlab*>(p.data), a.A, in, out, part, alpha, p.add != 0,
                                        lane);
                }
                i += W;
                if (i < e) g = static_cast<const TGroup*>(p.items)[i];
            }
        }
        __syncthreads();
        if (threadIdx.x == 0 && ok && !(a.skip && s != a.side && p.first + item == 0)) {
            asm volatile("red.release.gpu.global.add.u64 [%0], 1;\n" ::"l"(done + s) : "memory");
        }
    };
    // one item per round: from the near field's queue while `side` (at the
    // start of part of the CTAs, and before the pass that waits for it), else
    // from the chain's; `held` is a chain item taken before that queue was
    // drained
    bool side = int(blockIdx.x) >= a.main_ctas && a.side >= 0, drained = a.side < 0;
    int held = -1;
    while (ok) {
        int s = a.side, item;
        if (side) {
            item = take(1);
            if (item < 0) break;
            if (item >= a.side_items) {
                side = false;
                drained = true;
                continue;
            }
        } else {
            item = held >= 0 ? held : take(0);
            held = -1;
            if (item < 0) break;
            if (item >= a.main_items) {   // no chain left; nor a near field that no pass waits for
                if (drained) break;
                side = true;
                continue;
            }
            s = 0;
            while (s == a.side || item >= a.st[s].first + a.st[s].nitems) ++s;
            if (a.st[s].join >= 0 && !drained) {
                side = true;
                held = item;
                continue;
            }
            item -= a.st[s].first;
        }
        run(s, item);
    }
}

}  // namespace hlrc
