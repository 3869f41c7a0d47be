// FP64 products of 16, 24 or 32 vectors per pass of the matrix (FP64 tensor
// cores, mma.sync m8n8k4): NT tiles of 8 vectors, NT = 2, 3 or 4.
//
// The 8-vector kernels (kernels_mr.cuh) read the matrix once per 8 vectors
// and are bound by HBM; with 32 vectors the same matrix elements feed 32
// multiply-adds, 8 flop per byte, which is where HBM and the FP64 tensor pipe
// take about the same time.  Measured, one pass against blocks of 8 (B200):
// n = 50021 exponential, 16 vectors, adjoint 1.63 -> 0.95 ms; n = 20011, 32 vectors,
// op N 1.09 -> 0.52 ms; uniform-H sphere of 32768 triangles, 32 vectors
// 380 -> 179 us.  What bounds the passes: the FP64 tensor pipe and its operand
// latency at 24 and 32 vectors, HBM with the coefficient traffic at 16 (0.25
// bytes of coefficients more per matrix byte).
//
// Sums.  An MMA rounds its sum four times; a warp that keeps one sum per output
// over all its chunks rounds at the size of that sum for each of its matrix
// columns, and there are half as many warps to an output as in the 8-vector
// kernels.  So 8 columns (16 with NT = 4) or 8 rows are summed from zero and the
// result added to the output's sum.  Error of the product against long double,
// with one sum -> summed apart, and of the 8-vector kernels (1e-16, relative
// 2-norm): n = 20011 exponential, op N, 32 vectors 10.4 -> 3.3 (7.2), adjoint
// 5.2 -> 2.3 (3.5); 1D log n = 100003 4.7 -> 2.2 (3.1); uniform-H sphere of 32768
// triangles 5.4 -> 2.5 (4.0).  It costs 2 adds per 2 MMAs (4 with NT = 4): op N of
// n = 20011, 16 / 24 / 32 vectors 352 / 409 / 472 -> 355 / 452 / 524 us.
//
// Vector blocks are row-major with RB = 8 NT doubles per entry.  A 16-byte
// load of a vector row serves two tiles: tile 2p + b takes vector
// 16p + 2g + b as its fragment column g, so an accumulator of tile 2p + b
// holds vectors 16p + 4t + 2e + b.  An odd last tile (NT = 3) takes vector
// 16p + g.
#pragma once

#include <cuda_runtime.h>

#include "kernels_mr.cuh"
#include "layout.hpp"

namespace hlrc {

constexpr int DW_MAXNT = 4;    // most 8-vector tiles per pass
// the vector of accumulator e of tile n in a lane with quad index t
template <int NT> __device__ __forceinline__ int dw_vec(int n, int t, int e) {
    return n == NT - 1 && NT % 2 == 1 ? 8 * n + 2 * t + e : 16 * (n >> 1) + 4 * t + 2 * e + (n & 1);
}

// xr[i * RB + r] = X[i + (r0 + r) * ldx] for r < nr, 0 for nr <= r < RB: 32
// entries per CTA through shared memory, so that the reads run down the
// columns of X and the writes along the rows of xr
template <int NT>
__global__ void __launch_bounds__(256)
k_dw_rows(const double* X, int64_t ldx, int64_t n, int r0, int nr, double* __restrict__ xr) {
    constexpr int RB = 8 * NT;
    __shared__ double s[RB][33];
    pdl_trigger();
    pdl_wait(X);
    const int64_t i0 = int64_t(blockIdx.x) * 32;
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < RB; r += 8)
        s[r][lane] = r < nr && i0 + lane < n ? __ldca(X + i0 + lane + int64_t(r0 + r) * ldx) : 0.0;
    __syncthreads();
    for (int q = threadIdx.x; q < 32 * RB; q += 256)
        if (i0 + q / RB < n) xr[i0 * RB + q] = s[q % RB][q / RB];
}

// N-form.  A warp owns all 64 rows and all vectors of the output tile for
// every W-th chunk: 8 x NT accumulator tiles, so a chunk's operands are read
// once; the W sums are added in order through shared memory.  The operands
// go through shared memory in a ring of D chunks per warp (cp.async): a
// fragment's lanes read 4 columns at once, which are multiples of 128 bytes
// apart in the store, so direct 16-byte loads take four L1 wavefronts per
// 128 bytes (that kept the L1 at 65 % and the MMAs at 46 % of their rates on
// 64-row tiles).  The column strides 544 and 8 RB + pad (32 modulo 128) give
// one.  Rows past the tile height hold stale data: they only feed rows that
// are not written.
constexpr int DW_WARPS = 4;
constexpr int DW_AS = TILE * 8 + 32;                                          // matrix column stride, bytes
template <int NT> constexpr int dw_bs() { return 64 * NT + (NT % 2 ? (NT == 3 ? 96 : 32) : 32); }   // vector column
template <int NT> constexpr int dw_chunk() { return 8 * (DW_AS + dw_bs<NT>()); }
// Chunks whose products are summed apart before they are added to a tile's sums
// (a ring slot's), ring depth, CTAs per SM, and whether the vector operands are
// read again for every 16 rows instead of held in registers.  32 vectors: two
// chunks halve the adds; op N of n = 20011 exponential / 1D log n = 100003 / uniform-H
// sphere of 32768 triangles 565 / 290 / 190 us with one, 524 / 282 / 179 with two.
// 24 vectors: 448 / 208 / 145 us as here, 479 / 244 / 159 with two chunks (and
// two CTAs, for the registers).
template <int NT> constexpr int dw_fold() { return NT == 4 ? 2 : 1; }
template <int NT> constexpr int dw_stage() { return dw_fold<NT>() * dw_chunk<NT>(); }
template <int NT> constexpr int dw_depth() { return NT == 2 ? 3 : 2; }
template <int NT> constexpr int dw_ctas() { return NT == 4 ? 2 : 3; }
template <int NT> constexpr bool dw_vp() { return NT > 2; }
template <int NT> constexpr int dw_nsmem() {
    constexpr int ring = DW_WARPS * dw_depth<NT>() * dw_stage<NT>(), red = DW_WARPS * TILE * (8 * NT + 1) * 8;
    return ring > red ? ring : red;
}

__device__ __forceinline__ void dw_cp16(uint32_t dst, const void* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

template <int NT, bool SP>
__global__ void __launch_bounds__(DW_WARPS * 32, dw_ctas<NT>())
k_nform_dw(const NSeg* __restrict__ segs, const NChunk* __restrict__ chunks, const double* __restrict__ A,
           const double* vx, const double* vt, OutMap om, double alpha, int add) {
    constexpr int RB = 8 * NT, NP = NT / 2, W = DW_WARPS, RS = RB + 1, D = dw_depth<NT>(), BS = dw_bs<NT>();
    constexpr int F = dw_fold<NT>();
    constexpr bool VP = dw_vp<NT>();
    static_assert(D * F <= 4, "the ring's column counts fit 32 bits");
    constexpr bool ODD = NT % 2 == 1;
    constexpr int VU = RB / 2;   // 16-byte units of a vector row
    extern __shared__ __align__(16) double dw_sn[];
    pdl_trigger();
    const NSeg sg = SP ? seg_part(segs[blockIdx.x]) : segs[blockIdx.x];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int np = (sg.rows + 15) / 16;      // 16-row groups
    uint8_t* ring = reinterpret_cast<uint8_t*>(dw_sn) + warp * (D * dw_stage<NT>());
    const uint32_t ring_s = static_cast<uint32_t>(__cvta_generic_to_shared(ring));
    double acc[8][NT][2];   // row 16p + 2g + b at [2p + b], vector dw_vec(n, t, e)
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[i][n][0] = acc[i][n][1] = 0.0;
    const NChunk none{0, 0, 0, 0};
    auto desc = [&](uint32_t i) { return i < sg.ce ? chunks[i] : none; };   // nc == 0 past the end
    const bool unit = 2 * lane < sg.ld;      // this lane's 16 bytes of a matrix column exist
    // copies chunk q to `at`: its columns, then its vector rows; the columns up to
    // the next multiple of 4 are zero-filled
    auto issue = [&](const NChunk& q, uint32_t at) {
        const double* v = (q.v_off & VEC_T) ? vt + size_t(q.v_off & ~VEC_T) * RB : vx + size_t(q.v_off) * RB;
        const double* a = A + q.a_off + 2 * lane;
        const uint32_t sb = at + 8 * DW_AS;
        const int up = (q.nc + 3) & ~3;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (j < up && unit) dw_cp16(at + j * DW_AS + lane * 16, j < q.nc ? a + size_t(j) * sg.ld : A, j < q.nc);
#pragma unroll
        for (int k = 0; k < 8 * VU / 32; ++k) {
            const int u = 32 * k + lane, j = u / VU;
            if (j < up) dw_cp16(sb + j * BS + (u % VU) * 16, j < q.nc ? v + 2 * u : A, j < q.nc);
        }
    };
    // the F chunks of slot d, ncs: their columns, 8 bits each.  A k-step takes four
    // columns; FULL (one chunk a slot): it has two of them
    auto compute = [&](uint32_t ncs, int d) {
        const uint8_t* sa = ring + d * dw_stage<NT>() + t * DW_AS + g * 16;
        const uint8_t* sb = ring + d * dw_stage<NT>() + 8 * DW_AS + t * BS;
        auto step = [&](int k) { return (int(ncs >> (8 * (k >> 1))) & 0xff) > 4 * (k & 1); };   // is there a k-step k?
        auto body = [&](auto full) {
            constexpr bool FULL = decltype(full)::value;
            double v[VP ? 1 : 2 * F][NT];
            auto load = [&](int k, double (&o)[NT]) {   // the vector operand of k-step k
                const uint8_t* q = sb + (k >> 1) * dw_chunk<NT>() + 4 * (k & 1) * BS;
#pragma unroll
                for (int h = 0; h < NP; ++h) {
                    const double2 w = *reinterpret_cast<const double2*>(q + 128 * h + 16 * g);
                    o[2 * h] = w.x;
                    o[2 * h + 1] = w.y;
                }
                if constexpr (ODD) o[NT - 1] = *reinterpret_cast<const double*>(q + 128 * NP + 8 * g);
            };
            if constexpr (!VP) {
#pragma unroll
                for (int k = 0; k < 2 * F; ++k)
                    if (FULL || step(k)) load(k, v[k]);
            }
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                if (p >= np) break;
                double s[2][NT][2];
#pragma unroll
                for (int k = 0; k < 2 * F; ++k) {
                    if (k > 0 && !FULL && !step(k)) continue;
                    const double2 m = *reinterpret_cast<const double2*>(sa + (k >> 1) * dw_chunk<NT>() +
                                                                        4 * (k & 1) * DW_AS + 128 * p);
                    if constexpr (VP) load(k, v[0]);
#pragma unroll
                    for (int n = 0; n < NT; ++n)
#pragma unroll
                        for (int b = 0; b < 2; ++b) {
                            if (k == 0) dmma0(s[b][n], b ? m.y : m.x, v[0][n]);
                            else dmma(s[b][n], b ? m.y : m.x, v[VP ? 0 : k][n]);
                        }
                }
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int b = 0; b < 2; ++b)
                        acc[2 * p + b][n][0] += s[b][n][0], acc[2 * p + b][n][1] += s[b][n][1];
            }
        };
        if (F == 1 && step(1)) body(std::true_type{});
        else body(std::false_type{});
    };
    uint32_t c = sg.cb + warp;
    uint32_t ncs = 0;   // columns of the chunks in the ring, 8 bits per chunk
    NChunk q = desc(c);
    uint32_t ci = c;    // the chunk q describes, the next one to issue
    auto issue_next = [&](int d) {
#pragma unroll
        for (int f = 0; f < F; ++f) {
            const int at = 8 * (d * F + f);
            ncs = (ncs & ~(0xffu << at)) | (uint32_t(q.nc) << at);
            if (ci < sg.ce) {
                issue(q, ring_s + uint32_t(d * dw_stage<NT>() + f * dw_chunk<NT>()));
                ci += W;
                q = desc(ci);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    pdl_wait(vx, vt);
#pragma unroll
    for (int d = 0; d < D - 1; ++d) issue_next(d);
    for (int d = 0; c < sg.ce; c += F * W) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(D - 2) : "memory");
        __syncwarp();    // the slot's copies of all lanes landed, and every lane is done with the slot before it
        issue_next(d == 0 ? D - 1 : d - 1);
        compute(ncs >> (8 * F * d), d);
        d = d == D - 1 ? 0 : d + 1;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();     // the rings become the sums [warp][row][vector]
    double* red = dw_sn;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                red[(warp * TILE + 16 * (i >> 1) + 2 * g + (i & 1)) * RS + dw_vec<NT>(n, t, e)] = acc[i][n][e];
    __syncthreads();
    nform_update<RB, W * 32, SP>(
        int(sg.out), sg.rows, om, alpha, add,
        [&](int row, int kk) {
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < W; ++w) s += red[(w * TILE + row) * RS + kk];
            return s;
        },
        [&](int row, int kk) { return red + row * RS + kk; });
}

// Stores one column's results of a vector group (tiles 2 vg and, with TWO,
// 2 vg + 1): d[n][e] of chunk column g, to base[v * cs] for vectors v < nr.
template <bool TWO>
__device__ __forceinline__ void dw_store(const double (&d)[2][2], int vg, int t, double* base, int64_t cs, int nr,
                                         double alpha, int add) {
#pragma unroll
    for (int n = 0; n < (TWO ? 2 : 1); ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int k = 16 * vg + (TWO ? 4 * t + 2 * e + n : 2 * t + e);
            if (k >= nr) continue;
            if (add) base[int64_t(k) * cs] += alpha * d[n][e];
            else base[int64_t(k) * cs] = d[n][e];
        }
}

// Group T-form: a CTA per segment (GTSeg: chunks of up to GT_TILES input
// tiles).  The x rows of the tiles are staged in shared memory once per CTA;
// a warp takes every W-th chunk, contracts it over its tiles and writes one
// result per column: clusters of at most GT_TILES tiles need no partials.
// The row stride of the staged x (RB + 2 doubles) puts the 16-byte reads of a
// quarter warp (2 vector pairs x 4 row pairs) into different banks.  The
// matrix data of the next slab is loaded while one multiplies.
constexpr int DW_GWARPS = 8;
template <int NT> constexpr int dw_xs() { return 8 * NT + 2; }
template <int NT> constexpr int dw_gsmem() { return GT_TILES * TILE * dw_xs<NT>() * 8; }

template <int NT, bool FINE>
__global__ void __launch_bounds__(DW_GWARPS * 32, 2)
k_gtform_dw(const GTSeg* __restrict__ segs, const GTChunk* __restrict__ chunks, const GTTile* __restrict__ tiles,
            const double* __restrict__ A, const double* vin, OutMap om, double* __restrict__ part, double alpha,
            int add) {
    constexpr int RB = 8 * NT, NP = NT / 2, XS = dw_xs<NT>(), W = DW_GWARPS;
    constexpr bool ODD = NT % 2 == 1;
    constexpr int CH = NT <= 2 && !FINE ? 2 : 1;   // sets of sums, for alternate groups of 8 rows
    extern __shared__ __align__(16) double dw_sx[];   // [tile][row][XS]
    pdl_trigger();
    const GTSeg sg = segs[blockIdx.x];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    pdl_wait(vin);
    for (uint32_t s = 0; s < sg.ntiles; ++s) {
        const GTTile tl = tiles[sg.tile0 + s];
        const double2* src = reinterpret_cast<const double2*>(vin + size_t(tl.v_off) * RB);
#pragma unroll 4
        for (int i = threadIdx.x; i < TILE * (RB / 2); i += W * 32) {
            const int row = i / (RB / 2), u = i % (RB / 2);
            *reinterpret_cast<double2*>(dw_sx + (s * TILE + row) * XS + 2 * u) =
                row < tl.rows ? __ldca(src + i) : make_double2(0.0, 0.0);
        }
    }
    int ld[GT_TILES];
#pragma unroll
    for (int s = 0; s < GT_TILES; ++s) ld[s] = uint32_t(s) < sg.ntiles ? tiles[sg.tile0 + s].ld : 0;
    __syncthreads();
    uint32_t c = sg.cb + warp;
    if (c >= sg.ce) return;
    const double* base = A + sg.base;
    // slab s of chunk q: column g, rows 8j + 2t, +1
    auto issue = [&](const GTChunk& q, int s, double2 (&m)[8]) {
        uint32_t off = q.a[0];
        int l = ld[0];
#pragma unroll
        for (int k = 1; k < GT_TILES; ++k)
            if (s == k) off = q.a[k], l = ld[k];
        const double* a = base + 2 * size_t(off) + size_t(g) * l;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int row = 8 * (NT < 4 ? j ^ (g & 1) : j) + 2 * t;
            m[j] = g < q.nc && row < l ? ld_stream(a + row) : make_double2(0.0, 0.0);
        }
    };
    // odd columns load the row groups of each pair in the other order, so that
    // the two columns of a quarter warp read different halves of a 128-byte
    // line (one L1 wavefront instead of two); swapped back here (with 32
    // vectors the swap's registers spill, and the L1 is not the limit)
    auto unswap = [&](double2 (&m)[8]) {
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            const double2 a = m[j], b = m[j + 1];
            m[j] = g & 1 ? b : a;
            m[j + 1] = g & 1 ? a : b;
        }
    };
    auto next_slab = [&](const GTChunk& q, int s) {   // the first slab of q after s (GT_TILES: none)
        int r = GT_TILES;
#pragma unroll
        for (int k = GT_TILES - 1; k >= 0; --k)
            if (k > s && q.a[k] != GT_NONE) r = k;
        return r;
    };
    double d[CH][NT][2];
    auto zero = [&]() {
#pragma unroll
        for (int h = 0; h < CH; ++h)
#pragma unroll
            for (int n = 0; n < NT; ++n) d[h][n][0] = d[h][n][1] = 0.0;
    };
    auto multiply = [&](int s, const double2 (&m)[8]) {
        const double* x = dw_sx + (s * TILE + 2 * t) * XS;
        int l = ld[0];
#pragma unroll
        for (int k = 1; k < GT_TILES; ++k)
            if (s == k) l = ld[k];
        double f[NT][2];   // FINE: the sums of this slab
#pragma unroll
        for (int j = 0; j < 8; ++j) {   // rows past the tile: zero x and zero matrix entries
            if (8 * j >= l) break;
            const double *x0 = x + 8 * j * XS, *x1 = x0 + XS;
            double e[NT][2];
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const double2 v = *reinterpret_cast<const double2*>(x0 + 16 * p + 2 * g);
                dmma0(e[2 * p], m[j].x, v.x);
                dmma0(e[2 * p + 1], m[j].x, v.y);
            }
            if constexpr (ODD) dmma0(e[NT - 1], m[j].x, x0[16 * NP + g]);
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const double2 v = *reinterpret_cast<const double2*>(x1 + 16 * p + 2 * g);
                dmma(e[2 * p], m[j].y, v.x);
                dmma(e[2 * p + 1], m[j].y, v.y);
            }
            if constexpr (ODD) dmma(e[NT - 1], m[j].y, x1[16 * NP + g]);
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                if constexpr (!FINE) d[j % CH][n][0] += e[n][0], d[j % CH][n][1] += e[n][1];
                else if (j == 0) f[n][0] = e[n][0], f[n][1] = e[n][1];
                else f[n][0] += e[n][0], f[n][1] += e[n][1];
            }
        }
        if constexpr (FINE) {
#pragma unroll
            for (int n = 0; n < NT; ++n) d[0][n][0] += f[n][0], d[0][n][1] += f[n][1];
        }
    };
    auto store = [&](const GTChunk& q) {
        if (g >= q.nc) return;
        if constexpr (CH == 2) {
#pragma unroll
            for (int n = 0; n < NT; ++n) d[0][n][0] += d[CH - 1][n][0], d[0][n][1] += d[CH - 1][n][1];
        }
        const bool direct = (q.flags & TT_DIRECT) != 0;
        double* o = direct ? om.base + int64_t(q.out + g) * om.rs : part + size_t(q.out + g) * RB;
        const int64_t cs = direct ? om.cs : 1;
        const bool ad = direct && add;
        const int nr = direct ? om.nr : RB;
        if (cs == 1 && nr == RB && !ad) {   // a row of the partials or coefficients: 16-byte stores
#pragma unroll
            for (int p = 0; p < NP; ++p)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    *reinterpret_cast<double2*>(o + 16 * p + 4 * t + 2 * e) =
                        make_double2(d[0][2 * p][e], d[0][2 * p + 1][e]);
            if constexpr (ODD) *reinterpret_cast<double2*>(o + 16 * NP + 2 * t) = make_double2(d[0][NT - 1][0], d[0][NT - 1][1]);
            return;
        }
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int k = dw_vec<NT>(n, t, e);
                if (k >= nr) continue;
                if (ad) o[int64_t(k) * cs] += alpha * d[0][n][e];
                else o[int64_t(k) * cs] = d[0][n][e];
            }
    };
    const GTChunk none{{GT_NONE, GT_NONE, GT_NONE, GT_NONE}, 0, 0, 0};
    double2 mA[8], mB[8];
    GTChunk q = chunks[c], qn = c + W < sg.ce ? chunks[c + W] : none;
    int s = next_slab(q, -1);
    issue(q, s, mA);
    zero();
    // one slab: the following one is issued, this one multiplied, and the
    // chunk written after its last; false after the last chunk
    auto step = [&](double2 (&cur)[8], double2 (&nxt)[8]) {
        int s2 = next_slab(q, s);
        const bool last = s2 == GT_TILES;
        if (last) s2 = next_slab(qn, -1);
        if (s2 < GT_TILES) {
            if (last) issue(qn, s2, nxt);
            else issue(q, s2, nxt);
        }
        if constexpr (NT < 4) unswap(cur);
        multiply(s, cur);
        s = s2;
        if (!last) return true;
        store(q);
        zero();
        c += W;
        if (c >= sg.ce) return false;
        q = qn;
        qn = c + W < sg.ce ? chunks[c + W] : none;
        return true;
    };
    while (step(mA, mB) && step(mB, mA)) {
    }
}

// Unit T-form (the transposed couplings): a warp per unit (a run of slabs x
// at most 8 columns) and vector group.
template <int NT>
__global__ void __launch_bounds__(256)
k_tform_dw(const TUnit* __restrict__ units, int nunits, const TSlab* __restrict__ slabs, const double* __restrict__ A,
           const double* vin, OutMap om, double* __restrict__ part, double alpha, int add) {
    constexpr int RB = 8 * NT, NG = (NT + 1) / 2;
    pdl_trigger();
    const int wid = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (wid >= nunits * NG) return;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int vg = wid % NG;
    const TUnit u = units[wid / NG];
    pdl_wait(vin);
    auto body = [&](auto two) {
        constexpr bool TWO = decltype(two)::value;
        double d[2][2] = {}, f[2][2] = {};
        TSlab sl = u.sb < u.se ? slabs[u.sb] : TSlab{0, 0, 0, 0};
        for (uint32_t s = u.sb; s < u.se; ++s) {
            const TSlab cur = sl;
            if (s + 1 < u.se) sl = slabs[s + 1];
            const double* a = A + cur.a_off + size_t(u.c0 + g) * cur.ld;
            const double* x = vin + size_t(cur.v_off) * RB + 16 * vg + (TWO ? 2 * g : g);
#pragma unroll 4
            for (int j = 0; 8 * j < cur.ld; ++j) {
                const int row = 8 * j + 2 * t;
                const double2 m = g < u.nc && row < cur.ld ? __ldg(reinterpret_cast<const double2*>(a + row))
                                                           : make_double2(0.0, 0.0);
                double2 v[2];
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const bool ok = row + b < cur.rows;
                    if constexpr (TWO) v[b] = ok ? __ldca(reinterpret_cast<const double2*>(x + size_t(row + b) * RB))
                                                 : make_double2(0.0, 0.0);
                    else v[b] = make_double2(ok ? __ldca(x + size_t(row + b) * RB) : 0.0, 0.0);
                }
                dmma8(j & 1 ? f[0] : d[0], m.x, v[0].x, m.y, v[1].x);
                if constexpr (TWO) dmma8(j & 1 ? f[1] : d[1], m.x, v[0].y, m.y, v[1].y);
            }
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) d[n][0] += f[n][0], d[n][1] += f[n][1];
        if (g >= u.nc) return;
        if (u.flags & TU_DIRECT)
            dw_store<TWO>(d, vg, t, om.base + int64_t(u.out + g) * om.rs, om.cs, om.nr, alpha, add);
        else
            dw_store<TWO>(d, vg, t, part + (size_t(u.out) * 32 + g) * RB, 1, RB, 1.0, 0);
    };
    if (2 * vg + 1 < NT) body(std::true_type{});
    else body(std::false_type{});
}

// Sums the partial slots of multi-unit outputs in slot order: a thread per
// column and vector, 8 columns per group.
template <int NT>
__global__ void __launch_bounds__(256)
k_tfinish_dw(const TGroup* __restrict__ groups, int ngroups, const double* part, OutMap om, double alpha,
             int add) {
    constexpr int RB = 8 * NT;
    pdl_trigger();
    const int64_t idx = int64_t(blockIdx.x) * 256 + threadIdx.x;
    const int64_t gi = idx / (TCOLS * RB);
    if (gi >= ngroups) return;
    const TGroup g = groups[gi];
    const int c = int(idx / RB) % TCOLS, k = int(idx % RB);
    if (c >= int(g.nc) || k >= om.nr) return;
    pdl_wait(part);
    double s = 0.0;
    for (uint32_t i = 0; i < g.nslots; ++i) s += __ldca(part + (size_t(g.slot0 + i) * 32 + c) * RB + k);
    double* o = om.base + int64_t(g.out + c) * om.rs + int64_t(k) * om.cs;
    if (add) *o += alpha * s;
    else *o = s;
}

}  // namespace hlrc
