// precond_mma.cu -- layers and weight gradient of the learned preconditioner (precond.h), on the
// tensor cores and, for layers that would mostly pad their tiles, in FP32 arithmetic.
//
// Layer: out_o(x) = sum_k U_k(x) [ sum_i W[o][i][k] in_i(x + k) ], k = 0..8, with U_0 = 1.
// The spin mixing in brackets is one matrix product per path, the same weights for every
// column (site, colour, RHS): A (rows (o, s', re/im), K = (i, s, re/im)) times B (the raw
// neighbour spinors).  The link acts on the product's colours, in FP32.
//
// FP32 products on the 16-bit MMA (mma.sync m16n8k16, FP32 accumulation): operands are scaled
// by powers of two so that their largest entries sit at 2^14 and split into FP16 pieces.  On every
// path the weights have a scale per row (o, s') and per input channel, w_oi / (q_o p_i) against
// p_i x_i, and the field one per column of p_i x_i: neither the size of a channel, between which a
// linear network is free to shift factors, nor that of a right-hand side costs bits.
//   first pieces  w0, x0: the values rounded to multiples of 2^6, so 9 bits of the largest entry.
//                 Products of two of them are multiples of 2^12 up to 2^30, and 64 of them (the
//                 gradient's K; a layer's is 32) add up within 24 bits: exact.
//   the rest      w x = w0 x0 + w0 (x - x0) + (w - w0) x, with x - x0 = (x1 + x2) / 2^9,
//                 w - w0 = (w1 + w2) / 2^9 and x = h + l: w0 x1 + w0 x2 + w1 h + w1 l + w2 h, five
//                 more products.  The factor 2^9 keeps the pieces clear of FP16's subnormal
//                 numbers.  What is lost of an entry is below 2^-23 of itself, or 2^-48 of the
//                 largest entry under its scale: FP32's own precision.
// The exactness of the first product matters because the MMA truncates: it keeps 2 bits
// below FP32's last place of the largest addend and rounds the sum toward zero (measured: with
// 11-bit pieces a sum over K = 64 is short by 9e-8 of itself on average).  That bias is the same at
// every site, so it adds up in the weight gradient: 1.1e-6 of it, against 3.5e-8 with FP32
// arithmetic.  The five small products are truncated 2^-9 lower.  The sums of one step (a path, up
// to 4 input channels) are accumulated from zero and added to the FP32 result outside the MMA with
// one rounding, so an output is a chain of 2 N FMAs a link path and step, 16 N + 1 for up to 4
// input channels.
//
// Fragments (PTX ISA, mma.m16n8k16): lane 4 g + t holds A rows g, g + 8 at K 2t..2t+1 and
// 2t+8..2t+9, B column g at the same K, D rows g, g + 8 at columns 2t, 2t + 1.  K-step j holds
// channels 2j (K 0..7) and 2j + 1 (K 8..15), each as 4 spins (re, im): lane t loads spin t of
// column g.  Rows 0..7 of a tile are the real parts of two output channels x 4 spins, rows
// 8..15 the imaginary parts: a lane's D registers are whole complex numbers.
//
// No reference code; the CPU restatement oracle_ptc_forward is the checker.
#include <utility>

#include "precond.h"

namespace qcub {

int sm_count();

namespace {

constexpr int kPaths = 9;
constexpr int kMmaThreads = 256;
constexpr int kPieces = 3;                        // of a weight
constexpr int kStepVecs = kPieces * 32;           // uint4 of one (path, row tile, K step)
constexpr int kStepBytes = kStepVecs * 16;

__device__ __forceinline__ void mma16(float (&d)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// the same from a zero accumulator
__device__ __forceinline__ void mma16_zero(float (&d)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "f"(0.f));
}

__device__ __forceinline__ uint32_t half_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }

// two FP32 numbers in one register pair and their packed arithmetic (same rounding as the
// scalar instructions, half the issue slots)
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Splits of a scaled pair (below 2^15).
// v = h + l, both FP16
__device__ __forceinline__ void split_float(f32x2 v, uint32_t& h, uint32_t& l) {
    const __half2 b = __float22half2_rn(unpack2(v));
    const float2 e = __half22float2(b), d = unpack2(fma2(pack2(e.x, e.y), pack2(-1.f, -1.f), v));
    h = half_bits(b);
    l = half_bits(__float22half2_rn(d));
}
// v rounded to a multiple of 2^6 (adding 1.5 x 2^29 leaves no lower bits), and 2^9 times the rest in
// two pieces; kRest brings the rest's products back
constexpr float kRestUp = 512.f, kRest = 1.f / 512.f;
__device__ __forceinline__ void split_rest(f32x2 v, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    constexpr float c = 1.5f * (float)(1 << 29);
    const f32x2 f = add2(add2(v, pack2(c, c)), pack2(-c, -c));
    p0 = half_bits(__float22half2_rn(unpack2(f)));   // exact
    split_float(fma2(f, pack2(-kRestUp, -kRestUp), mul2(v, pack2(kRestUp, kRestUp))), p1, p2);
}
struct Pieces {
    uint32_t p0, p1, p2, h, l;
};
__device__ __forceinline__ Pieces split_field(f32x2 v) {
    Pieces r;
    split_rest(v, r.p0, r.p1, r.p2);
    split_float(v, r.h, r.l);
    return r;
}

// power of two that brings a maximum m into [2^14, 2^15), and its inverse
__device__ __forceinline__ float scale_to_half(float m, float* inv) {
    const int eb = (int)((__float_as_uint(m) >> 23) & 255u);
    const int f = min(max(268 - eb, 1), 253);
    *inv = __uint_as_float((uint32_t)(254 - f) << 23);
    return __uint_as_float((uint32_t)f << 23);
}

// ---- weights ----
// A fragments of one layer: [path][row tile][K step][piece][lane] uint4, then for
// every path the input channels' factors p_i and the rows' inverse scales.  adj: of the adjoint
// layer, W'[i][o][-k] = W[o][i][k]^dag.
struct FragShape {
    int mt, ks;        // row tiles (2 output channels each) and K steps (2 input channels), padded
    int tiles, steps;  // per block and per channel chunk
};

// Two channel pairs a step (four would put the pieces of 4 more channels into registers: 760 bytes
// spilled a thread, and an 8 -> 8 layer three times slower).  Row tiles up to the output channels, at most 4 (SU(2), SU(3)) or 2 (SU(4), whose
// 4 tiles of sums, link and pieces spill 460 bytes: 18.8 ms against 15.6 ms for 4 layers of 8 channels
// at 16^4, m = 8) and to the 227 KB of shared memory: more than that are further blocks, which load
// the field again.
FragShape frag_shape(int nc, int cin, int cout) {
    FragShape s;
    s.steps = cin <= 2 ? 1 : 2;
    s.ks = (cin + 2 * s.steps - 1) / (2 * s.steps) * s.steps;
    s.tiles = cout <= 2 ? 1 : (cout <= 4 || nc == 4 ? 2 : 4);
    if (s.tiles == 4 && (size_t)kPaths * 4 * s.ks * kStepBytes > 224 * 1024) s.tiles = 2;
    s.mt = (cout + 2 * s.tiles - 1) / (2 * s.tiles) * s.tiles;
    return s;
}

__host__ __device__ inline int frag_channels(int ks) { return 2 * ks; }
__host__ __device__ inline int frag_rows(int mt) { return 8 * mt; }

struct PrepLayer {
    const float2* w;
    uint4* frag;
    float *chan, *row;   // [path][2 ks] factors of the input channels, [path][8 mt] inverse row scales
    int cin, cout;       // of the layer that the fragments compute
    int mt, ks;
};
struct PrepArgs {
    PrepLayer l[16];
    int adj;
};

__device__ __forceinline__ int opposite_path(int k) { return k == 0 ? 0 : (((k - 1) & 1) ? k - 1 : k + 1); }

__device__ __forceinline__ float finite_abs(float v) { return fabsf(v) <= 3.4028235e38f ? fabsf(v) : 0.f; }

// power of two at or below m (of the smallest normal number for m below it), and its inverse
__device__ __forceinline__ float power_of(float m, float* inv) {
    const int e = min(max((int)(__float_as_uint(m) >> 23), 1), 253);
    *inv = __uint_as_float((uint32_t)(254 - e) << 23);
    return __uint_as_float((uint32_t)e << 23);
}

// One block per (layer, path).
__global__ void ptc_prepare_kernel(PrepArgs a) {
    const PrepLayer L = a.l[blockIdx.x];
    const int k = blockIdx.y;
    // maxima as bit patterns (ordered as the numbers): rows, channels of w / q, rows of w / (q p)
    __shared__ unsigned qmax[64], cmax[16], rmax[64];
    __shared__ int shift;
    // entry (o, s'), (i, s) of the path's matrix
    auto weight = [&](int o, int sp, int i, int t) {
        if (!a.adj) return L.w[((int64_t)(o * L.cin + i) * kPaths + k) * 16 + sp * 4 + t];
        // stored W[o' = i][i' = o][opposite k][s' = t][s = sp]
        const float2 v = L.w[((int64_t)(i * L.cout + o) * kPaths + opposite_path(k)) * 16 + t * 4 + sp];
        return make_float2(v.x, -v.y);
    };
    auto exponent = [](unsigned m) { return max((int)(m >> 23), 1) - 127; };
    const int n = L.cin * L.cout * 16;
    for (int e = threadIdx.x; e < 64; e += blockDim.x) {
        qmax[e] = rmax[e] = 0u;
        if (e < 16) cmax[e] = 0u;
    }
    __syncthreads();
#pragma unroll 1
    for (int pass = 0; pass < 3; ++pass) {
        for (int e = threadIdx.x; e < n; e += blockDim.x) {
            const int i = (e >> 4) % L.cin, o = (e >> 4) / L.cin, sp = (e >> 2) & 3, r = 4 * o + sp;
            const float2 v = weight(o, sp, i, e & 3);
            // an infinity decides over no other entry
            float mx = fmaxf(finite_abs(v.x), finite_abs(v.y));
            if (pass > 0) mx = scalbnf(mx, -exponent(qmax[r]) - (pass > 1 ? exponent(cmax[i]) : 0));
            atomicMax(pass == 0 ? &qmax[r] : (pass == 1 ? &cmax[i] : &rmax[r]), __float_as_uint(mx));
        }
        __syncthreads();
    }
    // the channels' factors lie between 2^-126 and 2 so far; their middle goes to 1, so that p_i x_i
    // leaves FP32's range on either side only where the channels' sizes differ by as much
    if (threadIdx.x == 0) {
        int lo = 0;
        for (int i = 0; i < L.cin; ++i)
            if (cmax[i] != 0u) lo = min(lo, exponent(cmax[i]));
        shift = -lo / 2;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < frag_channels(L.ks); i += blockDim.x)
        L.chan[k * frag_channels(L.ks) + i] = scalbnf(1.f, exponent(cmax[i]) + (cmax[i] != 0u ? shift : 0));
    for (int r = threadIdx.x; r < frag_rows(L.mt); r += blockDim.x) {
        float inv;
        scale_to_half(__uint_as_float(rmax[r]), &inv);
        L.row[k * frag_rows(L.mt) + r] = scalbnf(inv, exponent(qmax[r]) - shift);
    }
    for (int e = threadIdx.x; e < L.mt * L.ks * 32; e += blockDim.x) {
        const int lane = e & 31, j = (e >> 5) % L.ks, mt = (e >> 5) / L.ks;
        const int g = lane >> 2, t = lane & 3;
        const int o = 2 * mt + (g >> 2), sp = g & 3;
        float inv;
        const float sc = scale_to_half(__uint_as_float(rmax[4 * o + sp]), &inv);
        uint32_t w0[4], w1[4], w2[4];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int i = 2 * j + c;
            float2 v = make_float2(0.f, 0.f);
            if (o < L.cout && i < L.cin) {
                v = weight(o, sp, i, t);
                const int e2 = -exponent(qmax[4 * o + sp]) - exponent(cmax[i]);
                v.x = scalbnf(v.x, e2) * sc;
                v.y = scalbnf(v.y, e2) * sc;
            }
            split_rest(pack2(v.x, -v.y), w0[2 * c], w1[2 * c], w2[2 * c]);               // real row
            split_rest(pack2(v.y, v.x), w0[2 * c + 1], w1[2 * c + 1], w2[2 * c + 1]);   // imaginary row
        }
        uint4* f = L.frag + (int64_t)(((k * L.mt + mt) * L.ks + j)) * kStepVecs + lane;
        f[0] = make_uint4(w0[0], w0[1], w0[2], w0[3]);
        f[32] = make_uint4(w1[0], w1[1], w1[2], w1[3]);
        f[64] = make_uint4(w2[0], w2[1], w2[2], w2[3]);
    }
}

// ---- layer ----
struct LayerArgs {
    float2* out;
    const float2* in;
    const uint4* frag;
    const float *chan, *row;
    const float2* gauge;
    Geom g;
    int m, cin, cout, mt, ks;
    float t_sign;
    const int* done;
};

// full-lattice site (even half first) as coordinates
struct PtcSite {
    int p, xh, y, z, t;
    uint32_t idx;
};
__device__ __forceinline__ PtcSite ptc_site(const Geom& g, uint32_t site) {
    PtcSite s;
    s.p = site >= (uint32_t)g.vh;
    s.idx = site - (s.p ? (uint32_t)g.vh : 0u);
    const SiteXYZT c = site_coords(g, s.idx);
    s.xh = c.xh;
    s.y = c.y;
    s.z = c.z;
    s.t = c.t;
    return s;
}
// path k >= 1 of a site: source site (full lattice), link (index into [4][2][Vh]; backward links
// are conjugate-transposed) and whether it crosses the t boundary
__device__ __forceinline__ void ptc_step(const Geom& g, const PtcSite& s, int k, uint32_t& src, uint32_t& link, bool& wrap) {
    const uint32_t vh = (uint32_t)g.vh, lxh = (uint32_t)g.lxh, Ly = (uint32_t)g.L[1], Lz = (uint32_t)g.L[2],
                   Lt = (uint32_t)g.L[3];
    const uint32_t sy = lxh, sz = lxh * Ly, st = sz * Lz, xh = (uint32_t)s.xh;
    const int mu = (k - 1) >> 1;
    const bool f = ((k - 1) & 1) == 0;
    uint32_t nb;
    wrap = false;
    if (mu == 0) {
        const bool xodd = ((s.p ^ (s.y + s.z + s.t)) & 1) != 0;
        const uint32_t row = s.idx - xh;
        nb = row + (f ? (xodd ? (xh + 1 == lxh ? 0u : xh + 1) : xh) : (xodd ? xh : (xh == 0 ? lxh - 1 : xh - 1)));
    } else if (mu == 1) {
        nb = f ? s.idx + sy - ((uint32_t)s.y + 1 == Ly ? Ly * sy : 0u) : s.idx - sy + (s.y == 0 ? Ly * sy : 0u);
    } else if (mu == 2) {
        nb = f ? s.idx + sz - ((uint32_t)s.z + 1 == Lz ? Lz * sz : 0u) : s.idx - sz + (s.z == 0 ? Lz * sz : 0u);
    } else {
        wrap = f ? (uint32_t)s.t + 1 == Lt : s.t == 0;
        nb = f ? s.idx + st - (wrap ? Lt * st : 0u) : s.idx - st + (wrap ? Lt * st : 0u);
    }
    src = (s.p ? 0u : vh) + nb;
    link = (uint32_t)(2 * mu + (f ? s.p : 1 - s.p)) * vh + (f ? s.idx : nb);
}

__device__ __forceinline__ float2 cfma2(float2 a, float2 b, float2 c) {   // c + a b
    c.x = fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x));
    c.y = fmaf(a.x, b.y, fmaf(a.y, b.x, c.y));
    return c;
}

// One warp per tile of 8 consecutive columns (site, RHS) of the flattened full lattice, all
// colours, 2 MT output channels, input channels 2 KS at a time.  The block's weights (its MT row
// tiles) stay in shared memory (216 KB for 8 x 8 channels), so one block of 8 warps runs on an SM, at
// up to 255 registers: a step's spinors and link are requested under the products of the step
// before it.  16^4, SU(3), m = 8, one 8 -> 8 layer: 6.5 ms as FP32 arithmetic with a thread per (site,
// output channel, RHS); 1.86 ms with five products, two pieces of a field and one scale for many
// channels, which lost bits of all but the largest entries; 2.64 ms so.  6 MT KS NC MMAs a step (288 a
// path) bound it at 1.26 ms; the rest is the fixed latency of the MMA and FP32 chains at 8 warps.
template <int NC, int MT, int KS>
__global__ void __launch_bounds__(kMmaThreads, 1) ptc_mma_kernel(const LayerArgs a) {
    if (a.done != nullptr && *a.done) return;
    constexpr int CG = NC == 4 && KS > 1 ? 1 : NC;   // fewer spills than 2 or 4
    extern __shared__ uint4 sw[];
    const int mt0 = blockIdx.y * MT;
    const int per_path = MT * a.ks * kStepVecs;
    for (int e = threadIdx.x; e < kPaths * per_path; e += blockDim.x) {
        const int k = e / per_path, r = e - k * per_path;
        sw[e] = a.frag[(int64_t)(k * a.mt + mt0) * a.ks * kStepVecs + r];
    }
    const int nch = frag_channels(a.ks);
    float* const chan = reinterpret_cast<float*>(sw + kPaths * per_path);   // [path][2 ks]
    float* const row = chan + kPaths * nch;                                 // [path][8 MT]
    for (int e = threadIdx.x; e < kPaths * nch; e += blockDim.x) chan[e] = a.chan[e];
    for (int e = threadIdx.x; e < kPaths * frag_rows(MT); e += blockDim.x)
        row[e] = a.row[(e / frag_rows(MT)) * frag_rows(a.mt) + frag_rows(mt0) + e % frag_rows(MT)];
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int m = a.m;
    const uint32_t um = (uint32_t)m;
    const uint32_t cols = 2u * (uint32_t)a.g.vh * um;
    const int64_t slen = 4 * NC * (int64_t)m, field = 2 * a.g.vh * slen;
    const bool odd = (m & 1) != 0;   // the columns 2t, 2t + 1 may belong to two sites
    const uint32_t nw = gridDim.x * (kMmaThreads / 32);
    for (uint32_t tile = blockIdx.x * (kMmaThreads / 32) + (threadIdx.x >> 5); tile * 8 < cols; tile += nw) {
        const uint32_t col = min(tile * 8 + g, cols - 1);
        const uint32_t site = col / um, r = col - site * um;
        const PtcSite ps = ptc_site(a.g, site);
        const float2* const in = a.in + (int64_t)(t * NC) * m + r;
        // output of this lane's rows, columns (2t, 2t + 1) as pairs
        f32x2 re[MT][NC], im[MT][NC];
#pragma unroll
        for (int q = 0; q < MT; ++q)
#pragma unroll
            for (int c = 0; c < NC; ++c) re[q][c] = im[q][c] = 0ull;
        // a step: path k, channel chunk j0; its spinors (spin t, column g) are requested before the
        // products of the step before it
        float2 x[2 * KS][NC];
        uint32_t link = 0;
        bool wrap = false;
        float2 u0[NC][NC];   // link of column 2t, as stored (transposed for backward paths)
        auto step = [&](int k) {   // base of path k's spinors
            uint32_t src = site;
            if (k) ptc_step(a.g, ps, k, src, link, wrap);
            return in + (int64_t)src * slen;
        };
        auto load_link = [&](int k) {
            if (k == 0) return;
            const float2* U = a.gauge + (int64_t)__shfl_sync(0xffffffffu, link, 8 * t) * (NC * NC);
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int d = 0; d < NC; ++d) u0[c][d] = __ldg(U + ((k & 1) ? c * NC + d : d * NC + c));
        };
        // channels past the last meet zero weights: any finite number of the field will do
        auto load_colour = [&](const float2* v, int j0, int c) {
#pragma unroll
            for (int i = 0; i < 2 * KS; ++i) x[i][c] = __ldg(v + (int64_t)min(2 * j0 + i, a.cin - 1) * field + c * m);
        };
        {
            const float2* v = step(0);
#pragma unroll
            for (int c = 0; c < NC; ++c) load_colour(v, 0, c);
        }
#pragma unroll 1
        for (int k = 0, j0 = 0; k < kPaths;) {
            float mx = 0.f;
#pragma unroll
            for (int i = 0; i < 2 * KS; ++i) {
                const float pc = chan[k * nch + 2 * j0 + i];
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    x[i][c] = unpack2(mul2(pack2(x[i][c].x, x[i][c].y), pack2(pc, pc)));
                    mx = fmaxf(mx, fmaxf(fabsf(x[i][c].x), fabsf(x[i][c].y)));
                }
            }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            float inv;
            const float sc = scale_to_half(mx, &inv);
            // scale, link and boundary of this lane's D columns 2t and 2t + 1
            float dinv[2];
            f32x2 ur[NC][NC], ui[NC][NC];
#pragma unroll
            for (int b = 0; b < 2; ++b) dinv[b] = __shfl_sync(0xffffffffu, inv, 8 * t + 4 * b);
            if (k) {
                const bool fwd = (k & 1) != 0;
                const int w0 = __shfl_sync(0xffffffffu, (int)wrap, 8 * t), w1 = __shfl_sync(0xffffffffu, (int)wrap, 8 * t + 4);
                const uint32_t l1 = __shfl_sync(0xffffffffu, link, 8 * t + 4);
                const float s0 = w0 ? a.t_sign : 1.f, s1 = w1 ? a.t_sign : 1.f;
                const float2* U = a.gauge + (int64_t)l1 * (NC * NC);
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int d = 0; d < NC; ++d) {
                        float2 e = u0[c][d];
                        if (odd) e = __ldg(U + (fwd ? c * NC + d : d * NC + c));
                        ur[c][d] = pack2(u0[c][d].x * s0, e.x * s1);
                        ui[c][d] = pack2(u0[c][d].y * (fwd ? s0 : -s0), e.y * (fwd ? s1 : -s1));
                    }
            }
            const int k0 = k, j00 = j0;
            j0 += KS;
            if (j0 >= a.ks) {
                j0 = 0;
                ++k;
            }
            const bool more = k < kPaths;
            const float2* next = in;
            if (more) {
                next = step(k);
                if (j0 == 0) load_link(k);
            }
            // CG colours at a time: their pieces, then the next step's spinors into the registers that
            // the pieces leave, then the products
#pragma unroll
            for (int c0 = 0; c0 < NC; c0 += CG) {
                Pieces y[2 * KS][CG];
#pragma unroll
                for (int i = 0; i < 2 * KS; ++i)
#pragma unroll
                    for (int c = 0; c < CG; ++c)
                        y[i][c] = split_field(mul2(pack2(x[i][c0 + c].x, x[i][c0 + c].y), pack2(sc, sc)));
                if (more) {
#pragma unroll
                    for (int c = 0; c < CG; ++c) load_colour(next, j0, c0 + c);
                }
#pragma unroll
                for (int q = 0; q < MT; ++q) {
                    const uint4* A = sw + (size_t)((k0 * MT + q) * a.ks + j00) * kStepVecs + lane;
                    float d1[CG][4], d2[CG][4];
#pragma unroll
                    for (int j = 0; j < KS; ++j) {
                        const uint4 a0 = A[j * kStepVecs], a1 = A[j * kStepVecs + 32], a2 = A[j * kStepVecs + 64];
#pragma unroll
                        for (int c = 0; c < CG; ++c) {
                            const Pieces &u = y[2 * j][c], &v = y[2 * j + 1][c];
                            if (j == 0) {
                                mma16_zero(d2[c], a2, u.h, v.h);
                                mma16_zero(d1[c], a0, u.p0, v.p0);
                            } else {
                                mma16(d2[c], a2, u.h, v.h);
                                mma16(d1[c], a0, u.p0, v.p0);
                            }
                            mma16(d2[c], a0, u.p2, v.p2);
                            mma16(d2[c], a1, u.l, v.l);
                            mma16(d2[c], a0, u.p1, v.p1);
                            mma16(d2[c], a1, u.h, v.h);
                        }
                    }
                    const f32x2 kr = pack2(kRest, kRest);
                    const float rinv = row[k0 * frag_rows(MT) + 8 * q + g];
                    const f32x2 back = pack2(rinv * dinv[0], rinv * dinv[1]);
#pragma unroll
                    for (int c = 0; c < CG; ++c) {
                        const f32x2 dr = mul2(fma2(pack2(d2[c][0], d2[c][1]), kr, pack2(d1[c][0], d1[c][1])), back);
                        const f32x2 di = mul2(fma2(pack2(d2[c][2], d2[c][3]), kr, pack2(d1[c][2], d1[c][3])), back);
                        if (k0 == 0) {
                            re[q][c0 + c] = add2(re[q][c0 + c], dr);
                            im[q][c0 + c] = add2(im[q][c0 + c], di);
                        } else {
                            const f32x2 nd = mul2(di, pack2(-1.f, -1.f));
#pragma unroll
                            for (int r = 0; r < NC; ++r) {
                                re[q][r] = fma2(ur[r][c0 + c], dr, re[q][r]);
                                im[q][r] = fma2(ur[r][c0 + c], di, im[q][r]);
                                re[q][r] = fma2(ui[r][c0 + c], nd, re[q][r]);
                                im[q][r] = fma2(ui[r][c0 + c], dr, im[q][r]);
                            }
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const uint32_t oc = tile * 8 + 2 * t + b;
            if (oc >= cols || (b && !odd)) continue;
            const uint32_t os = oc / um, orr = oc - os * um;
#pragma unroll
            for (int q = 0; q < MT; ++q) {
                const int o = 2 * (mt0 + q) + (g >> 2);
                if (o >= a.cout) continue;
                float2* dst = a.out + (int64_t)o * field + (int64_t)os * slen + (int64_t)((g & 3) * NC) * m + orr;
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const float2 r2 = unpack2(re[q][c]), i2 = unpack2(im[q][c]);
                    if (!odd)   // both columns: adjacent RHS of one site
                        *reinterpret_cast<float4*>(dst + c * m) =
                            make_float4(r2.x, i2.x, r2.y, i2.y);
                    else
                        dst[c * m] = b ? make_float2(r2.y, i2.y) : make_float2(r2.x, i2.x);
                }
            }
        }
    }
}

template <int NC, int MT, int KS>
int layer_launch(const LayerArgs& a, cudaStream_t st) {
    auto k = ptc_mma_kernel<NC, MT, KS>;
    const size_t smem = (size_t)kPaths * (MT * a.ks * kStepBytes + (frag_channels(a.ks) + frag_rows(MT)) * sizeof(float));
    if (int rc = smem_optin(reinterpret_cast<const void*>(k), smem)) return rc;
    const int ny = a.mt / MT;
    const int64_t tiles = (2 * a.g.vh * a.m + 7) / 8, want = (tiles + kMmaThreads / 32 - 1) / (kMmaThreads / 32);
    const int64_t cap = sm_count() / ny > 0 ? sm_count() / ny : 1;
    k<<<dim3((unsigned)(want < cap ? want : cap), (unsigned)ny), kMmaThreads, smem, st>>>(a);
    QCUB_CHECK_LAUNCH();
    return QCU_SUCCESS;
}

template <int NC>
int layer_nc(const LayerArgs& a, const FragShape& f, cudaStream_t st) {
    if constexpr (NC < 4) {   // frag_shape
        if (f.tiles == 4) return f.steps == 1 ? layer_launch<NC, 4, 1>(a, st) : layer_launch<NC, 4, 2>(a, st);
    }
    switch (f.tiles * 2 + f.steps) {
        case 2 + 1: return layer_launch<NC, 1, 1>(a, st);
        case 2 + 2: return layer_launch<NC, 1, 2>(a, st);
        case 4 + 1: return layer_launch<NC, 2, 1>(a, st);
        default: return layer_launch<NC, 2, 2>(a, st);
    }
}

// ---- layer in FP32 arithmetic ----
// A thread per (site, output channel, RHS), which transports every input itself; the layer's
// weights in shared memory.  FP32 issue bounds it (62 % at 24 % of the warps).
struct SimtArgs {
    float2* out;
    const float2* in;
    const float2* w;
    const float2* gauge;
    Geom g;
    int m, cin, cout, adj;
    float t_sign;
    const int* done;
};
constexpr int kSimtThreads = 256;

// tv = U_k(x) f(x + k) for one RHS: f points at the channel's field + r
template <int NC>
__device__ __forceinline__ void ptc_transport(float2 (&tv)[4][NC], const float2* __restrict__ f,
                                              const float2* __restrict__ U, int k, float sg, int m) {
    if (k == 0) {
#pragma unroll
        for (int e = 0; e < 4 * NC; ++e) tv[e / NC][e % NC] = f[e * m];
        return;
    }
    const bool fwd = (k & 1) != 0;
    float2 u[NC][NC];
#pragma unroll
    for (int a = 0; a < NC; ++a)
#pragma unroll
        for (int b = 0; b < NC; ++b) {
            const float2 e = fwd ? U[a * NC + b] : U[b * NC + a];
            u[a][b] = make_float2(sg * e.x, fwd ? sg * e.y : -sg * e.y);
        }
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        float2 in[NC];
#pragma unroll
        for (int b = 0; b < NC; ++b) in[b] = f[(s * NC + b) * m];
#pragma unroll
        for (int a = 0; a < NC; ++a) {
            float2 acc = make_float2(0.f, 0.f);
#pragma unroll
            for (int b = 0; b < NC; ++b) acc = cfma2(u[a][b], in[b], acc);
            tv[s][a] = acc;
        }
    }
}

template <int NC>
__global__ void __launch_bounds__(kSimtThreads, 2) ptc_simt_kernel(const SimtArgs a) {
    if (a.done != nullptr && *a.done) return;
    extern __shared__ float2 sw2[];   // [cout][cin][path][4][4]
    const int cin = a.cin, cout = a.cout, m = a.m;
    for (int e = threadIdx.x; e < cout * cin * kPaths * 16; e += blockDim.x) {
        if (!a.adj) {
            sw2[e] = a.w[e];
        } else {   // W'[o][i][k][s'][s] = conj W[i][o][opposite k][s][s']
            const int s = e & 3, sp = (e >> 2) & 3, k = (e >> 4) % kPaths, oi = (e >> 4) / kPaths;
            const float2 v = a.w[(((int64_t)(oi % cin) * cout + oi / cin) * kPaths + opposite_path(k)) * 16 + s * 4 + sp];
            sw2[e] = make_float2(v.x, -v.y);
        }
    }
    __syncthreads();
    const int per = m * cout, spb = blockDim.x / per;
    if ((int)threadIdx.x >= spb * per) return;
    const int r = threadIdx.x % m, o = (threadIdx.x / m) % cout;
    const int64_t slen = 4 * NC * (int64_t)m, field = 2 * a.g.vh * slen;
    for (int64_t site = (int64_t)blockIdx.x * spb + threadIdx.x / per; site < 2 * a.g.vh; site += (int64_t)gridDim.x * spb) {
        const PtcSite ps = ptc_site(a.g, (uint32_t)site);
        float2 acc[4][NC];
#pragma unroll
        for (int e = 0; e < 4 * NC; ++e) acc[e / NC][e % NC] = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int k = 0; k < kPaths; ++k) {
            uint32_t src = (uint32_t)site, link = 0;
            bool wrap = false;
            if (k) ptc_step(a.g, ps, k, src, link, wrap);
#pragma unroll 1
            for (int i = 0; i < cin; ++i) {
                float2 tv[4][NC];
                ptc_transport<NC>(tv, a.in + i * field + (int64_t)src * slen + r, a.gauge + (int64_t)link * (NC * NC), k,
                                  wrap ? a.t_sign : 1.f, m);
                const float2* W = sw2 + ((o * cin + i) * kPaths + k) * 16;
#pragma unroll
                for (int sp = 0; sp < 4; ++sp)
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        const float2 wv = W[sp * 4 + s];
#pragma unroll
                        for (int c = 0; c < NC; ++c) acc[sp][c] = cfma2(wv, tv[s][c], acc[sp][c]);
                    }
            }
        }
        float2* dst = a.out + o * field + site * slen + r;
#pragma unroll
        for (int e = 0; e < 4 * NC; ++e) dst[e * m] = acc[e / NC][e % NC];
    }
}

template <int NC>
int simt_launch(const SimtArgs& a, cudaStream_t st) {
    const size_t smem = (size_t)a.cout * a.cin * kPaths * 16 * sizeof(float2);
    if (int rc = smem_optin(reinterpret_cast<const void*>(ptc_simt_kernel<NC>), smem)) return rc;
    const int per = a.m * a.cout, block = kSimtThreads / per * per, spb = block / per;
    const int64_t want = (2 * a.g.vh + spb - 1) / spb, cap = (int64_t)sm_count() * 8;
    ptc_simt_kernel<NC><<<(int)(want < cap ? want : cap), block, smem, st>>>(a);
    QCUB_CHECK_LAUNCH();
    return QCU_SUCCESS;
}

// Whether FP32 arithmetic is the faster one.
// One input channel: at every size (2^4 to 8^4, SU(3), m = 3, 1 -> 8: 15-37 us against 27-48), but for
// SU(4) with a short row on a small lattice (4^4, m = 1, 1 -> 1: 45 / 22 us; m cout = 4: 22 / 26).
// More: not for fewer columns than the MMA kernel takes in its one wave of tiles, where it takes the
// time of one tile whatever the size (8^4, m = 1, 8 -> 1: 68 / 36 us).  Above that the MMA's cost goes
// with the padded channels, and one output channel fills half a row tile.  16^4, SU(3), m = 8:
//   1 -> 8 and 8 -> 1 together 1645 / 2320     2 -> 2 376 / 536     3 -> 3 851 / 900
//   5 -> 5 (0.39 of the products of the padded tiles in use) 2330 / 2630, that of 6 -> 6 (0.56)
// SU(4), and SU(2) where the field is loaded again for further row tiles, need more of the products in
// use (SU(4), 6 -> 6, 0.56: 4520 / 5980 us; SU(2), 9 -> 9, 0.56: 4150 / 5460 us).  One or two right-hand
// sides leave the FP32 kernel's rows short: with SU(2) and SU(3) only the edges are faster there.  A last
// wave that is mostly empty counts as padding (8^4, SU(3), m = 3, 6 -> 6: 80 / 120 us).
bool simt_faster(int nc, const FragShape& f, int cin, int cout, int m, int64_t vh) {
    if (m * cout > kSimtThreads) return false;
    const int64_t cols = 2 * vh * m, tiles = (kMmaThreads / 32) * 8;   // of one block
    const bool large = cols > sm_count() * tiles;
    if (cin == 1) return nc < 4 || large || m * cout >= 4;
    if (!large) return false;
    if (cout == 1 || cin * cout <= 4) return true;
    const float need = nc == 4 ? 0.6f : (nc == 2 && f.mt > f.tiles ? 0.57f : 0.45f);
    const int64_t wave = max(sm_count() * f.tiles / f.mt, 1) * tiles;
    const float filled = (float)cols / (float)((cols + wave - 1) / wave * wave);
    return (m >= 3 || nc == 4) && (cin * cout <= 9 || cin * cout * filled < need * (4 * f.mt * f.ks));
}

// ---- weight gradient ----
// gw[o][i][k][s'][s] = sum_{x, c, r} g_o[s'][c][r](x) conj((T_k in_i)[s][c][r](x))
//                    = sum_{x, c, r} (U_k^dag g_o)[s'][c][r](x) conj(in_i[s][c][r](x + k))
//                    = conj sum_{x, c, r} (U_-k^dag in_i)[s][c][r](x) conj(g_o[s'][c][r](x - k)):
// one matrix product per path over all columns, of the first form or, for one output channel of
// several inputs (4 of 16 rows in the first form), of the last: the same sum with the two fields'
// parts exchanged, path -k for k.  In the first form's terms, A: rows (o, s'), K = (column, re/im) of the
// transported gradient; B: columns (i, s, re/im), the pair (v.re, v.im) for the real part and
// (-v.im, v.re) for the imaginary part, so a lane's D registers are whole complex numbers.
// A column is a (site, RHS) pair, and the operands' sizes run in opposite directions: the loss
// divides by ||b_j||^2, so g goes as 1 / ||b_j|| where in goes as ||b_j|| (the layers are linear).  The
// columns of right-hand side j are therefore taken as g p and in / p with the power of two p at
// ||b_j||: exact, and gone from the product.  After that A has one scale per row (o, s') and B one
// per input channel, each common to the 8 columns of a step: neither the size of a right-hand side
// nor that of a channel costs bits, and a channel that overflows does so alone.
// Both operands keep 24 bits as the layer's: the first pieces' products add up exactly (K <= 64), the
// other five go to a second accumulator.  A step's products (6 NC MMAs per tile, one rounding)
// are added to FP64 sums in shared memory; warps, blocks and chunks are summed in a fixed order.
// 8^3x16, SU(3), m = 8, 8 -> 8 and 8 -> 1: 1358 and 693 us as FP32 arithmetic with a block per (o, i, k),
// 449 and 295 us with four products, shared scales and FP32 sums of 8 steps, 625 and 221 us so (the
// second with the fields exchanged; 442 us without).  MMA and FP32 chain latency at 8 warps bound it.
constexpr int kGradWarps = 8;
constexpr int kGradChunks = 16;   // blocks per path: 9 x 16 blocks of 8 warps, one per SM

struct GradArgs {
    double* part;          // [chunk][path][gridDim.z][MT CI 128]
    const float2* gout;
    const float2* in;
    const float2* gauge;
    const double* bnorm;   // ||b_j||
    Geom g;
    int m, cin, cout;
    bool swapped;          // gout is the layer's input, in its output gradient
    float t_sign;
};

// maximum over the 4 lanes of a row (g)
__device__ __forceinline__ float row_max(float v) {
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
    return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}

// MT row tiles (4 output channels each), CI input channels per block
template <int NC, int MT, int CI>
__global__ void __launch_bounds__(kGradWarps * 32, 1) ptc_grad_kernel(const GradArgs a) {
    extern __shared__ double sacc[];   // [warp][MT CI 4][lane]
    __shared__ float2 sizes[kMaxRhs];  // the right-hand sides' powers of two and their inverses
    if (threadIdx.x < a.m) {
        float inv;
        const float p = power_of((float)a.bnorm[threadIdx.x], &inv);
        sizes[threadIdx.x] = a.swapped ? make_float2(inv, p) : make_float2(p, inv);
    }
    __syncthreads();
    constexpr int NA = MT * CI * 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int k = blockIdx.y, ni = (a.cin + CI - 1) / CI;
    const int i0 = (int)(blockIdx.z % ni) * CI, o0 = (int)(blockIdx.z / ni) * MT * 4;
    const uint32_t um = (uint32_t)a.m, cols = 2u * (uint32_t)a.g.vh * um;
    const int m = a.m;
    const int64_t slen = 4 * NC * (int64_t)m, field = 2 * a.g.vh * slen;
    const bool fwd = (k & 1) != 0;
    double* const own = sacc + (size_t)warp * NA * 32 + lane;
#pragma unroll
    for (int e = 0; e < NA; ++e) own[e * 32] = 0.0;
#pragma unroll 1
    for (uint32_t tile = blockIdx.x * kGradWarps + warp; tile * 8 < cols; tile += gridDim.x * kGradWarps) {
        // this lane's columns t and t + 4: transported gradient rows g and g + 8 of every tile
        uint32_t src[2], rr[2];
        float2 h[MT][4][NC];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const uint32_t cw = tile * 8 + 4 * b + t;
            const bool in_range = cw < cols;
            const uint32_t col = in_range ? cw : cols - 1;
            const uint32_t site = col / um;
            rr[b] = col - site * um;
            uint32_t link = 0;
            bool wrap = false;
            src[b] = site;
            if (k) ptc_step(a.g, ptc_site(a.g, site), k, src[b], link, wrap);
            float2 u[NC][NC];   // U_k^dag
            if (k) {
                const float2* U = a.gauge + (int64_t)link * (NC * NC);
                const float sg = wrap ? a.t_sign : 1.f;
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int d = 0; d < NC; ++d) {
                        const float2 e = __ldg(U + (fwd ? d * NC + c : c * NC + d));
                        u[c][d] = make_float2(sg * e.x, fwd ? -sg * e.y : sg * e.y);
                    }
            }
#pragma unroll
            for (int q = 0; q < MT; ++q)
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const int o = o0 + 4 * q + 2 * w + (g >> 2);
                    const float2* gp = a.gout + (int64_t)o * field + (int64_t)site * slen + (int64_t)((g & 3) * NC) * m + rr[b];
                    float2 v[NC];
#pragma unroll
                    for (int c = 0; c < NC; ++c)
                        v[c] = in_range && o < a.cout ? __ldg(gp + (int64_t)c * m) : make_float2(0.f, 0.f);
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        float2 x = make_float2(0.f, 0.f);
                        if (k) {
#pragma unroll
                            for (int d = 0; d < NC; ++d) x = cfma2(u[c][d], v[d], x);
                        } else {
                            x = v[c];
                        }
                        h[q][2 * b + w][c] = x;
                    }
                }
        }
        const float2* const v0 = a.in + (int64_t)src[0] * slen + (int64_t)((g >> 1) * NC) * m + rr[0];
        const float2* const v1 = a.in + (int64_t)src[1] * slen + (int64_t)((g >> 1) * NC) * m + rr[1];
        // all channels' spinors requested first (one exposed latency a step instead of CI); channels
        // past the last are computed and not used
        float2 xs[CI][NC][2];
#pragma unroll
        for (int i = 0; i < CI; ++i) {
            const int64_t fo = (int64_t)min(i0 + i, a.cin - 1) * field;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                xs[i][c][0] = __ldg(v0 + fo + c * m);
                xs[i][c][1] = __ldg(v1 + fo + c * m);
            }
        }
        const float2 size[2] = {sizes[rr[0]], sizes[rr[1]]};
        float ainv[MT][2];
        uint4 a0[MT][NC], a1[MT][NC], a2[MT][NC];
#pragma unroll
        for (int q = 0; q < MT; ++q) {
            float asc[2];
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                float mx = 0.f;
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        float2& v = h[q][2 * b + w][c];
                        v.x *= size[b].x;
                        v.y *= size[b].x;
                        mx = fmaxf(mx, fmaxf(fabsf(v.x), fabsf(v.y)));
                    }
                asc[w] = scale_to_half(row_max(mx), &ainv[q][w]);
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                uint32_t p0[4], p1[4], p2[4];
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    split_rest(mul2(pack2(h[q][e][c].x, h[q][e][c].y), pack2(asc[e & 1], asc[e & 1])), p0[e], p1[e], p2[e]);
                a0[q][c] = make_uint4(p0[0], p0[1], p0[2], p0[3]);
                a1[q][c] = make_uint4(p1[0], p1[1], p1[2], p1[3]);
                a2[q][c] = make_uint4(p2[0], p2[1], p2[2], p2[3]);
            }
        }
#pragma unroll
        for (int i = 0; i < CI; ++i) {
            float2 (&x)[NC][2] = xs[i];
            float bx = 0.f;
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    x[c][b].x *= size[b].y;
                    x[c][b].y *= size[b].y;
                    bx = fmaxf(bx, fmaxf(fabsf(x[c][b].x), fabsf(x[c][b].y)));
                }
            float binv;
            const float bsc = scale_to_half(warp_max(bx), &binv);
            Pieces y[NC][2];
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const float re = x[c][b].x * bsc, im = x[c][b].y * bsc;
                    y[c][b] = split_field((g & 1) ? pack2(-im, re) : pack2(re, im));
                }
#pragma unroll
            for (int q = 0; q < MT; ++q) {
                const float dinv[2] = {ainv[q][0] * binv, ainv[q][1] * binv};   // of rows g and g + 8
                float d1[4], d2[4];
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const Pieces &u = y[c][0], &v = y[c][1];
                    if (c == 0) {
                        mma16_zero(d2, a2[q][c], u.h, v.h);
                        mma16_zero(d1, a0[q][c], u.p0, v.p0);
                    } else {
                        mma16(d2, a2[q][c], u.h, v.h);
                        mma16(d1, a0[q][c], u.p0, v.p0);
                    }
                    mma16(d2, a0[q][c], u.p2, v.p2);
                    mma16(d2, a1[q][c], u.l, v.l);
                    mma16(d2, a0[q][c], u.p1, v.p1);
                    mma16(d2, a1[q][c], u.h, v.h);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    own[((q * CI + i) * 4 + e) * 32] += (double)(fmaf(d2[e], kRest, d1[e]) * dinv[e >> 1]);
            }
        }
    }
    __syncthreads();
    double* dst = a.part + (((size_t)blockIdx.x * kPaths + k) * gridDim.z + blockIdx.z) * (NA * 32);
    for (int e = threadIdx.x; e < NA * 32; e += blockDim.x) {
        double s = 0.0;
        for (int w = 0; w < kGradWarps; ++w) s += sacc[(size_t)w * NA * 32 + e];
        dst[e] = s;
    }
}

// sum of the chunks, into gw; swapped: of the exchanged form, element (o, i, k, s', s) to the conjugate
// at (i, o, -k, s, s')
__global__ void ptc_grad_sum_kernel(double2* __restrict__ gw, const double* __restrict__ part, int mt, int ci,
                                    int cin, int cout, int nz, bool swapped) {
    const int na = mt * ci * 128;   // doubles of one (chunk, path, z)
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= kPaths * nz * na / 2) return;
    const int lane = e & 31, w = (e >> 5) & 1;
    int q = e >> 6;                 // (path, z, tile, channel)
    const int i = q % ci; q /= ci;
    const int tile = q % mt; q /= mt;
    const int z = q % nz, k = q / nz;
    const int ni = (cin + ci - 1) / ci;
    const int ii = (z % ni) * ci + i, o = (z / ni) * mt * 4 + 4 * tile + 2 * w + (lane >> 4);
    if (ii >= cin || o >= cout) return;
    const double* src = part + ((size_t)k * nz + z) * na + ((tile * ci + i) * 4 + 2 * w) * 32 + lane;
    double2 s = make_double2(0.0, 0.0);
#pragma unroll
    for (int c = 0; c < kGradChunks; ++c) {
        s.x += src[(size_t)c * kPaths * nz * na];
        s.y += src[(size_t)c * kPaths * nz * na + 32];
    }
    const int sp = (lane >> 2) & 3, sc = lane & 3;
    if (swapped)
        gw[(((int64_t)ii * cout + o) * kPaths + opposite_path(k)) * 16 + sc * 4 + sp] = make_double2(s.x, -s.y);
    else
        gw[(((int64_t)o * cin + ii) * kPaths + k) * 16 + sp * 4 + sc] = s;
}

bool grad_swapped(int cin, int cout) { return cout == 1 && cin > 1; }

// Row tiles of 4 output channels and input channels of a block: all of up to 8 x 8.
struct GradShape {
    int mt, ci, nz;
};
GradShape grad_shape(int cin, int cout) {
    GradShape s;
    s.mt = cout <= 4 ? 1 : 2;
    s.ci = cin == 1 ? 1 : (cin <= 4 ? 4 : 8);
    s.nz = (cin + s.ci - 1) / s.ci * ((cout + 4 * s.mt - 1) / (4 * s.mt));
    return s;
}

template <int NC, int MT, int CI>
int grad_launch(const GradArgs& a, double2* gw, int nz, cudaStream_t st) {
    auto k = ptc_grad_kernel<NC, MT, CI>;
    const size_t smem = (size_t)kGradWarps * MT * CI * 128 * sizeof(double);
    if (int rc = smem_optin(reinterpret_cast<const void*>(k), smem)) return rc;
    k<<<dim3(kGradChunks, kPaths, (unsigned)nz), kGradWarps * 32, smem, st>>>(a);
    QCUB_CHECK_LAUNCH();
    const int n = kPaths * nz * MT * CI * 64;
    ptc_grad_sum_kernel<<<(n + 255) / 256, 256, 0, st>>>(gw, a.part, MT, CI, a.cin, a.cout, nz, a.swapped);
    QCUB_CHECK_LAUNCH();
    return QCU_SUCCESS;
}

template <int NC>
int grad_nc(const GradArgs& a, const GradShape& s, double2* gw, cudaStream_t st) {
    switch (s.mt * 16 + s.ci) {
        case 16 + 1: return grad_launch<NC, 1, 1>(a, gw, s.nz, st);
        case 16 + 4: return grad_launch<NC, 1, 4>(a, gw, s.nz, st);
        case 32 + 1: return grad_launch<NC, 2, 1>(a, gw, s.nz, st);
        default: return grad_launch<NC, 2, 8>(a, gw, s.nz, st);
    }
}

}  // namespace

size_t ptc_grad_bytes(int cin, int cout) {
    const GradShape s = grad_shape(grad_swapped(cin, cout) ? cout : cin, grad_swapped(cin, cout) ? cin : cout);
    return (size_t)kGradChunks * kPaths * s.nz * s.mt * s.ci * 128 * sizeof(double);
}

int ptc_grad(int nc, double2* gw, void* part, const float2* gout, const float2* in, const float2* gauge,
             const double* bnorm, const Geom& g, int m, int cin, int cout, float t_sign, cudaStream_t st) {
    GradArgs a{static_cast<double*>(part), gout, in, gauge, bnorm, g, m, cin, cout, grad_swapped(cin, cout), t_sign};
    if (a.swapped) {
        std::swap(a.gout, a.in);
        std::swap(a.cin, a.cout);
    }
    const GradShape s = grad_shape(a.cin, a.cout);
    switch (nc) {
        case 2: return grad_nc<2>(a, s, gw, st);
        case 3: return grad_nc<3>(a, s, gw, st);
        case 4: return grad_nc<4>(a, s, gw, st);
        default: return set_error(QCU_ERR_UNSUPPORTED, "preconditioner n_color=%d (2..4)", nc);
    }
}

size_t ptc_frag_bytes(int nc, int cin, int cout) {
    const FragShape f = frag_shape(nc, cin, cout);
    const size_t b = (size_t)kPaths * (f.mt * f.ks * kStepBytes + (frag_channels(f.ks) + frag_rows(f.mt)) * sizeof(float));
    return (b + 15) & ~(size_t)15;
}

namespace {
// the parts of a layer's fragments
struct FragParts {
    uint4* frag;
    float *chan, *row;
};
FragParts frag_parts(void* base, const FragShape& f) {
    FragParts p;
    p.frag = static_cast<uint4*>(base);
    p.chan = reinterpret_cast<float*>(p.frag + (size_t)kPaths * f.mt * f.ks * kStepVecs);
    p.row = p.chan + kPaths * frag_channels(f.ks);
    return p;
}
}  // namespace

int ptc_prepare(int nc, const float2* const* w, void* const* frag, const int* cin, const int* cout, int layers, bool adj,
                cudaStream_t st) {
    PrepArgs a{};
    a.adj = adj;
    for (int l = 0; l < layers; ++l) {
        const int ci = adj ? cout[l] : cin[l], co = adj ? cin[l] : cout[l];
        const FragShape f = frag_shape(nc, ci, co);
        const FragParts p = frag_parts(frag[l], f);
        a.l[l] = PrepLayer{w[l], p.frag, p.chan, p.row, ci, co, f.mt, f.ks};
    }
    ptc_prepare_kernel<<<dim3(layers, kPaths), 256, 0, st>>>(a);
    QCUB_CHECK_LAUNCH();
    return QCU_SUCCESS;
}

int ptc_layer(int nc, float2* out, const float2* in, const float2* w, bool adj, const void* frag, const float2* gauge,
              const Geom& g, int m, int cin, int cout, float t_sign, const int* done, cudaStream_t st) {
    const FragShape f = frag_shape(nc, cin, cout);
    if (simt_faster(nc, f, cin, cout, m, g.vh)) {
        const SimtArgs a{out, in, w, gauge, g, m, cin, cout, adj, t_sign, done};
        switch (nc) {
            case 2: return simt_launch<2>(a, st);
            case 3: return simt_launch<3>(a, st);
            case 4: return simt_launch<4>(a, st);
            default: return set_error(QCU_ERR_UNSUPPORTED, "preconditioner n_color=%d (2..4)", nc);
        }
    }
    const FragParts p = frag_parts(const_cast<void*>(frag), f);
    const LayerArgs a{out, in, p.frag, p.chan, p.row, gauge, g, m, cin, cout, f.mt, f.ks, t_sign, done};
    switch (nc) {
        case 2: return layer_nc<2>(a, f, st);
        case 3: return layer_nc<3>(a, f, st);
        case 4: return layer_nc<4>(a, f, st);
        default: return set_error(QCU_ERR_UNSUPPORTED, "preconditioner n_color=%d (2..4)", nc);
    }
}

}  // namespace qcub
