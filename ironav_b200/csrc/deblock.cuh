// deblock.cuh — K4: the in-loop deblocking filter of a reconstructed picture (h264/deblock.rs), frame
// pictures, 4:2:0, 8-bit (uint8_t) or 10-bit (uint16_t) samples.
//
// The reference filters macroblocks in raster order (deblock_picture, deblock.rs:410-429); filtering a
// macroblock changes up to 3 samples on either side of its left and top edges, so macroblock (x, y) must
// see the final samples of (x - 1, y) and of (x + 1, y - 1) — the dependency deblock_picture_par keeps with
// its row wavefront (deblock.rs:583-605). Here the picture's macroblock rows go by groups of 4, a
// CTA a group and plane kind handed out by ticket, one warp a row left to right. Inside a macroblock the lanes take lines: 16 luma lines, or 8 Cb
// and 8 Cr lines (rows for the vertical edges, in registers, then columns for the horizontal edges, in shared memory).
// The rows of a group hand over through rings in shared memory; between groups, samples move through L2 and are
// published with a release store of the row's progress.
#pragma once
#include "common.cuh"

namespace ironav {

constexpr int DBK_WARPS = 4;
constexpr unsigned DBK_ALL = 0xffffffffu;

// alpha' / beta' by indexA / indexB, tC0 by (indexA, bS 1..3) — Tables 8-16 and 8-17 of the standard as
// h264/tables.rs holds them — and the chroma QP for qPi >= 30 (h264/mb.rs:211).
static __device__ __constant__ uint8_t c_dbk_alpha[52] = {
    0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 4, 4, 5, 6, 7, 8, 9, 10, 12, 13,
    15, 17, 20, 22, 25, 28, 32, 36, 40, 45, 50, 56, 63, 71, 80, 90, 101, 113, 127, 144, 162, 182, 203, 226, 255, 255};
static __device__ __constant__ uint8_t c_dbk_beta[52] = {0, 0, 0, 0, 0, 0, 0, 0, 0,  0,  0,  0,  0,  0,  0,  0,  2,  2,
                                                        2, 3, 3, 3, 3, 4, 4, 4, 6,  6,  7,  7,  8,  8,  9,  9,  10, 10,
                                                        11, 11, 12, 12, 13, 13, 14, 14, 15, 15, 16, 16, 17, 17, 18, 18};
static __device__ __constant__ uint8_t c_dbk_tc0[52][3] = {
    {0, 0, 0},  {0, 0, 0},   {0, 0, 0},   {0, 0, 0},   {0, 0, 0},    {0, 0, 0},    {0, 0, 0},    {0, 0, 0},    {0, 0, 0},
    {0, 0, 0},  {0, 0, 0},   {0, 0, 0},   {0, 0, 0},   {0, 0, 0},    {0, 0, 0},    {0, 0, 0},    {0, 0, 0},    {0, 0, 1},
    {0, 0, 1},  {0, 0, 1},   {0, 0, 1},   {0, 1, 1},   {0, 1, 1},    {1, 1, 1},    {1, 1, 1},    {1, 1, 1},    {1, 1, 1},
    {1, 1, 2},  {1, 1, 2},   {1, 1, 2},   {1, 1, 2},   {1, 2, 3},    {1, 2, 3},    {2, 2, 3},    {2, 2, 4},    {2, 3, 4},
    {2, 3, 4},  {3, 3, 5},   {3, 4, 6},   {3, 4, 6},   {4, 5, 7},    {4, 5, 8},    {4, 6, 9},    {5, 7, 10},   {6, 8, 11},
    {6, 8, 13}, {7, 10, 14}, {8, 11, 16}, {9, 12, 18}, {10, 13, 20}, {11, 15, 23}, {13, 17, 25}};
static __device__ __constant__ uint8_t c_dbk_cqp[22] = {29, 30, 31, 32, 32, 33, 34, 34, 35, 35, 36,
                                                       36, 37, 37, 37, 38, 38, 38, 39, 39, 39, 39};

// One deblocking launch.
struct DbkParams {
    uint8_t* planes[3];               // Y, Cb, Cr (byte addresses; samples of the launch's type)
    int ys, cs;                       // row strides in samples
    const ironav_dbk_mb* mbs;
    const ironav_dbk_slice* slices;
    int nslices, mb_w, mb_h, bd;
    unsigned* progress;               // per macroblock row, luma then chroma: macroblocks done (zeroed before the launch)
    unsigned* ticket;                 // next row
    unsigned* err;                    // 1: a wait gave up; 4: a slice id beyond the table
    unsigned wait_limit;              // polls before a wait gives up
};


// chroma_qp, h264/mb.rs:214-221
__device__ __forceinline__ int dbk_chroma_qp(int qp, int off, int bd) {
    const int qpi = min(max(qp + off, -6 * (bd - 8)), 51);
    return qpi < 30 ? qpi : (int)c_dbk_cqp[qpi - 30];
}

// coded, deblock.rs:336-345
__device__ __forceinline__ bool dbk_coded(const ironav_dbk_mb& m, int bx, int by) {
    if (m.t8x8) {
        const int x0 = bx & 2, y0 = by & 2;
        return (m.nnz[y0 * 4 + x0] | m.nnz[y0 * 4 + x0 + 1] | m.nnz[(y0 + 1) * 4 + x0] | m.nnz[(y0 + 1) * 4 + x0 + 1]) != 0;
    }
    return m.nnz[by * 4 + bx] != 0;
}

// far, deblock.rs:347-350
__device__ __forceinline__ bool dbk_far(const int16_t* a, const int16_t* b) { return abs(a[0] - b[0]) >= 4 || abs(a[1] - b[1]) >= 4; }

// motion_differs, deblock.rs:352-383 (frame macroblocks: the vertical limit is 4 quarter samples)
static __device__ bool dbk_motion_differs(const ironav_dbk_mb& p, int pbx, int pby, const ironav_dbk_mb& q, int qbx, int qby) {
    const int pi = pby * 4 + pbx, qi = qby * 4 + qbx;
    const int p8 = (pby >> 1) * 2 + (pbx >> 1), q8 = (qby >> 1) * 2 + (qbx >> 1);
    const int pr0 = p.ref_id[0][p8], pr1 = p.ref_id[1][p8], qr0 = q.ref_id[0][q8], qr1 = q.ref_id[1][q8];
    const int16_t *pm0 = p.mv[0][pi], *pm1 = p.mv[1][pi], *qm0 = q.mv[0][qi], *qm1 = q.mv[1][qi];
    const int np = (pr0 >= 0) + (pr1 >= 0), nq = (qr0 >= 0) + (qr1 >= 0);
    if (np != nq) return true;
    if (np == 1) {
        const bool lp = pr0 < 0, lq = qr0 < 0;
        return (lp ? pr1 : pr0) != (lq ? qr1 : qr0) || dbk_far(lp ? pm1 : pm0, lq ? qm1 : qm0);
    }
    if (!((pr0 == qr0 && pr1 == qr1) || (pr0 == qr1 && pr1 == qr0))) return true;
    if (pr0 != pr1) {
        if (pr0 == qr0) return dbk_far(pm0, qm0) || dbk_far(pm1, qm1);
        return dbk_far(pm0, qm1) || dbk_far(pm1, qm0);
    }
    return (dbk_far(pm0, qm0) || dbk_far(pm1, qm1)) && (dbk_far(pm0, qm1) || dbk_far(pm1, qm0));
}

// An edge as a line's filter wants it: the thresholds at the picture's depth (alpha 0: not filtered, no sample differs
// by less), tC0 by the line's strength, and which sides are kept.
struct DbkEdge {
    int b, alpha, beta, tc0;
    bool keep_p, keep_q;
};
// From an edge word and the line's strength b on it.
__device__ __forceinline__ DbkEdge dbk_edge(uint32_t wv, int b, int bd) {
    DbkEdge e;
    e.b = b;
    e.alpha = b ? (int)(wv & 0xff) << (bd - 8) : 0;
    e.beta = (int)((wv >> 8) & 0x1f) << (bd - 8);
    e.tc0 = (int)((wv >> (8 + 5 * (b & 3))) & 0x1f) << (bd - 8);  // strength 4 has none
    e.keep_p = (wv >> 28) & 1;
    e.keep_q = (wv >> 29) & 1;
    return e;
}

// filter_line, deblock.rs:279-333, on a line in registers whose first sample past the edge is q[0]; the side of a
// keep macroblock (I_PCM / lossless) is left as it was (filter_edge, deblock.rs:251-272). OUTER: a macroblock's
// outer edge, the only kind whose strength can be 4 (all along the edge, so the warp takes one path). Everything a line's own samples decide
// is selected, not branched on: the filter is a serial chain of eight edges a macroblock on one warp, where a branch costs
// as much as ten instructions.
template <bool CHROMA, bool OUTER>
__device__ __forceinline__ void dbk_line(int* q, const DbkEdge& E, int maxv) {
    const int p0 = q[-1], q0 = q[0], p1 = q[-2], q1 = q[1];
    const bool f = abs(p0 - q0) < E.alpha && abs(p1 - p0) < E.beta && abs(q1 - q0) < E.beta;
    const bool fp = f && !E.keep_p, fq = f && !E.keep_q;
    const bool strong = OUTER && E.b == 4;
    if constexpr (CHROMA) {
        const int tc = E.tc0 + 1;
        const int delta = min(max((((q0 - p0) << 2) + (p1 - q1) + 4) >> 3, -tc), tc);
        const int np0 = strong ? (2 * p1 + p0 + q1 + 2) >> 2 : min(max(p0 + delta, 0), maxv);
        const int nq0 = strong ? (2 * q1 + q0 + p1 + 2) >> 2 : min(max(q0 - delta, 0), maxv);
        q[-1] = fp ? np0 : p0;
        q[0] = fq ? nq0 : q0;
        return;
    }
    const int p2 = q[-3], q2 = q[2];
    const bool ap = abs(p2 - p0) < E.beta, aq = abs(q2 - q0) < E.beta;
    if (!strong) {
        const int tc = E.tc0 + ap + aq, avg = (p0 + q0 + 1) >> 1;
        const int delta = min(max((((q0 - p0) << 2) + (p1 - q1) + 4) >> 3, -tc), tc);
        q[-1] = fp ? min(max(p0 + delta, 0), maxv) : p0;
        q[0] = fq ? min(max(q0 - delta, 0), maxv) : q0;
        q[-2] = fp && ap ? p1 + min(max((p2 + avg - (p1 << 1)) >> 1, -E.tc0), E.tc0) : p1;
        q[1] = fq && aq ? q1 + min(max((q2 + avg - (q1 << 1)) >> 1, -E.tc0), E.tc0) : q1;
    } else {
        const bool small = abs(p0 - q0) < (E.alpha >> 2) + 2;
        const bool sp = ap && small, sq = aq && small;
        const int p3 = q[-4], q3 = q[3], m = p0 + q0;
        q[-1] = fp ? (sp ? (p2 + 2 * p1 + 2 * m + q1 + 4) >> 3 : (2 * p1 + p0 + q1 + 2) >> 2) : p0;
        q[0] = fq ? (sq ? (q2 + 2 * q1 + 2 * m + p1 + 4) >> 3 : (2 * q1 + q0 + p1 + 2) >> 2) : q0;
        q[-2] = fp && sp ? (p2 + p1 + m + 2) >> 2 : p1;
        q[1] = fq && sq ? (q2 + q1 + m + 2) >> 2 : q1;
        q[-3] = fp && sp ? (2 * p3 + 3 * p2 + p1 + m + 4) >> 3 : p2;
        q[2] = fq && sq ? (2 * q3 + 3 * q2 + q1 + m + 4) >> 3 : q2;
    }
}

// The thresholds of one edge (deblock.rs:647-651, 680-683), packed alpha' | beta' << 8 | tC0(bS 1, 2, 3)
// << 13, 18, 23 (all before the bit-depth shift; beta' <= 18 and tC0 <= 25 fit 5 bits); 0 when alpha' or
// beta' is 0 (filter_edge leaves the edge alone, deblock.rs:233-235).
__device__ __forceinline__ uint32_t dbk_thresholds(int qpav, const ironav_dbk_slice& sp) {
    const int ia = min(max(qpav + sp.alpha_offset, 0), 51), ib = min(max(qpav + sp.beta_offset, 0), 51);
    const uint32_t a = c_dbk_alpha[ia], b = c_dbk_beta[ib];
    if (a == 0 || b == 0) return 0u;
    return a | b << 8 | (uint32_t)c_dbk_tc0[ia][0] << 13 | (uint32_t)c_dbk_tc0[ia][1] << 18 | (uint32_t)c_dbk_tc0[ia][2] << 23;
}

// What the filter of one macroblock needs besides its samples, worked out before the wavefront (it depends
// on the macroblock records only). An edge word is its thresholds (dbk_thresholds) | keep << 28 (bit 0:
// the p side is a keep macroblock, bit 1: the q side); 0 means the edge is not filtered at all.
struct DbkEdges {
    uint8_t bs[2][4][4];        // [dir][edge][segment]
    uint32_t luma[2][4];        // [dir][edge]
    uint32_t chroma[2][2][2];   // [comp][dir][edge / 2]
};
static_assert(sizeof(DbkEdges) == 96, "DbkEdges layout");

// Pass 1: the boundary strengths (strength, deblock.rs:391-408) and edge words of every macroblock
// (deblock_mb's decisions, deblock.rs:608-695), one warp per macroblock, all macroblocks independent.
// One macroblock's boundary strengths and edge words (pass 1): R holds 3 records of shared memory (the
// macroblock, its left and its top neighbour), Bs the strengths [dir][edge][segment].
__device__ __forceinline__ void dbk_edges_mb(const DbkParams& P, DbkEdges* __restrict__ out, int idx, ironav_dbk_mb* R,
                                             uint8_t (*Bs)[4][4]) {
    const int lane = threadIdx.x & 31;
    const int x = idx % P.mb_w, y = idx / P.mb_w;
    for (int k = lane; k < 3 * 48; k += 32) {
        const int which = k / 48, wd = k % 48;
        const int src = which == 0 ? idx : (which == 1 ? (x > 0 ? idx - 1 : idx) : (y > 0 ? idx - P.mb_w : idx));
        reinterpret_cast<uint32_t*>(&R[which])[wd] = __ldg(reinterpret_cast<const uint32_t*>(&P.mbs[src]) + wd);
    }
    __syncwarp();
    const ironav_dbk_mb& m = R[0];
    // the neighbours across the left and top edges; at the picture's edges the macroblock itself, whose
    // outer edges are then not filtered (deblock.rs:618-621)
    const ironav_dbk_mb& lm = R[1];
    const ironav_dbk_mb& tm = R[2];
    bool live = m.slice != 0;
    if (live && m.slice > P.nslices) {
        if (lane == 0) atomicOr(P.err, 4u);
        live = false;
    }
    ironav_dbk_slice sp = {};
    if (live) sp = P.slices[m.slice - 1];
    live = live && sp.disable_deblocking != 1;
    const bool left_ok = x > 0 && lm.slice != 0 && (sp.disable_deblocking == 0 || lm.slice == m.slice);
    const bool top_ok = y > 0 && tm.slice != 0 && (sp.disable_deblocking == 0 || tm.slice == m.slice);
    // inner edges of an inter macroblock moving as a whole with no coefficients are not filtered
    // (uniform_motion, deblock.rs:385-389, and deblock.rs:625)
    bool same = true;
    if (lane < 16) {
        same = m.nnz[lane] == 0 && m.mv[0][lane][0] == m.mv[0][0][0] && m.mv[0][lane][1] == m.mv[0][0][1] &&
               m.mv[1][lane][0] == m.mv[1][0][0] && m.mv[1][lane][1] == m.mv[1][0][1];
        if (lane < 4)
            same = same && m.ref_idx[0][lane] == m.ref_idx[0][0] && m.ref_idx[1][lane] == m.ref_idx[1][0] &&
                   m.ref_id[0][lane] == m.ref_id[0][0] && m.ref_id[1][lane] == m.ref_id[1][0];
    }
    const bool still = m.inter && __all_sync(DBK_ALL, same);
    // boundary strengths: lane = dir * 16 + edge * 4 + segment
    {
        const int dir = lane >> 4, e = (lane >> 2) & 3, i = lane & 3;
        const ironav_dbk_mb& o = e == 0 ? (dir == 0 ? lm : tm) : m;
        int b = 0;
        if (!(e > 0 && still)) {
            if (!m.inter || !o.inter) {
                b = e == 0 ? 4 : 3;
            } else {
                const int qx = dir == 0 ? e : i, qy = dir == 0 ? i : e;
                const int px = dir == 0 ? (e == 0 ? 3 : e - 1) : i, py = dir == 0 ? i : (e == 0 ? 3 : e - 1);
                b = (dbk_coded(m, qx, qy) || dbk_coded(o, px, py)) ? 2 : (dbk_motion_differs(o, px, py, m, qx, qy) ? 1 : 0);
            }
        }
        Bs[dir][e][i] = (uint8_t)b;
    }
    __syncwarp();
    DbkEdges& E = out[idx];
    if (lane < 8) reinterpret_cast<uint32_t*>(E.bs)[lane] = reinterpret_cast<const uint32_t*>(Bs)[lane];
    // edge words: lanes 0-7 luma (dir, edge), lanes 8-15 chroma (comp, dir, edge / 2)
    if (lane < 16) {
        const bool chroma = lane >= 8;
        const int dir = chroma ? ((lane - 8) >> 1) & 1 : lane >> 2;
        const int e = chroma ? ((lane - 8) & 1) * 2 : lane & 3;
        const int comp = (lane - 8) >> 2;
        const ironav_dbk_mb& o = e == 0 ? (dir == 0 ? lm : tm) : m;
        const bool any = *reinterpret_cast<const uint32_t*>(Bs[dir][e]) != 0;
        uint32_t wv = 0;
        if (live && any && !(e == 0 && !(dir == 0 ? left_ok : top_ok)) && !(!chroma && m.t8x8 && (e & 1))) {
            if (chroma) {
                const int off = sp.chroma_qp_offset[comp];
                wv = dbk_thresholds((dbk_chroma_qp(o.qp, off, P.bd) + dbk_chroma_qp(m.qp, off, P.bd) + 1) >> 1, sp);
            } else {
                wv = dbk_thresholds((o.qp + m.qp + 1) >> 1, sp);
            }
            if (wv) wv |= (uint32_t)((o.keep ? 1 : 0) | (m.keep ? 2 : 0)) << 28;
        }
        if (chroma) E.chroma[comp][dir][e >> 1] = wv;
        else E.luma[dir][e] = wv;
    }
    __syncwarp();
}

static __global__ void __launch_bounds__(DBK_WARPS * 32) deblock_edges_kernel(const __grid_constant__ DbkParams P, DbkEdges* __restrict__ out) {
    __shared__ ironav_dbk_mb rec[DBK_WARPS][3];
    __shared__ uint8_t bsm[DBK_WARPS][2][4][4];
    const int wid = threadIdx.x >> 5;
    const int nmb = P.mb_w * P.mb_h;
    for (int idx = blockIdx.x * DBK_WARPS + wid; idx < nmb; idx += gridDim.x * DBK_WARPS) dbk_edges_mb(P, out, idx, rec[wid], bsm[wid]);
}

// ---- pass 2: the samples, in the row wavefront ---------------------------------------------------------

// N samples of type T from ints to p (aligned to their size, at most 16 bytes), through L2.
template <class T, int N>
__device__ __forceinline__ void dbk_store(T* p, const int* v) {
    constexpr int NB = N * (int)sizeof(T);
    uint32_t w[NB >= 4 ? NB / 4 : 1] = {};
#pragma unroll
    for (int k = 0; k < N; k++) w[(k * (int)sizeof(T)) >> 2] |= (uint32_t)v[k] << ((k * 8 * (int)sizeof(T)) & 31);
    if constexpr (NB == 16) __stcg(reinterpret_cast<uint4*>(p), make_uint4(w[0], w[1], w[2], w[3]));
    else if constexpr (NB == 8) __stcg(reinterpret_cast<uint2*>(p), make_uint2(w[0], w[1]));
    else if constexpr (NB == 4) __stcg(reinterpret_cast<unsigned*>(p), w[0]);
    else __stcg(reinterpret_cast<unsigned short*>(p), (unsigned short)w[0]);
}
// The four (luma) or two (chroma) edges across one line of NS samples (luma: 20 = 4 before the macroblock + 16; chroma: 10
// = 2 + 8) in registers: luma edges at 4, 8, 12, 16; chroma edges at 2 and 6.
template <bool CHROMA, int NS>
__device__ __forceinline__ void dbk_outer(int (&v)[NS], const DbkEdge (&e)[CHROMA ? 2 : 4], int maxv) {
    dbk_line<CHROMA, true>(&v[CHROMA ? 2 : 4], e[0], maxv);
}
template <bool CHROMA, int NS>
__device__ __forceinline__ void dbk_inner(int (&v)[NS], const DbkEdge (&e)[CHROMA ? 2 : 4], int maxv) {
#pragma unroll
    for (int k = 1; k < (CHROMA ? 2 : 4); k++) dbk_line<CHROMA, false>(&v[CHROMA ? 2 + 4 * k : 4 + 4 * k], e[k], maxv);
}

__device__ __forceinline__ unsigned ld_relaxed(const unsigned* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// Acquire load and release store of a word in shared memory, ordered within the CTA.
__device__ __forceinline__ unsigned ld_acquire_cta(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
    return v;
}
__device__ __forceinline__ void st_shared(unsigned* p, unsigned v) {  // relaxed; a fence before it makes a release
    asm volatile("st.relaxed.cta.shared.u32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release_cta(unsigned* p, unsigned v) {
    asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}

// A CTA filters a group of DBK_ROWS macroblock rows of one plane kind, one warp a row, with the rows of a
// group handing over through shared memory. What bounds the filter is the chain of mb_w + 2 (mb_h - 1)
// dependent macroblocks, so a step may wait on nothing slower than shared memory:
//   - a macroblock's samples and edge words come from global memory DBK_AHEAD - 1 steps ahead (cp.async);
//   - a row leaves the bottom rows (4 luma, 2 chroma) of its macroblocks in a ring that the row below reads,
//     with a progress word and a consumed word in shared memory (release and acquire at CTA scope);
//   - the group's first row reads a ring that a fetch warp fills from global memory, several macroblocks at
//     a time, as the group above publishes its last row; the publishing, with its device-scope fence, is a
//     warp of its own too. A group boundary then costs its latency once a picture, not once a step;
//   - a macroblock waits for the row above only when its top edge is filtered, and a direction without a
//     filtered edge skips its pass (and its transposition through shared memory).
// Four rows a group: a row's step is one warp's chain of ~650 instructions, and more rows an SM slow each other down (1080p
// with every edge filtered: 460, 405, 370 and 353 us at 14, 10, 6 and 4 rows), while a group boundary adds ~3 us. A P
// picture's records at 1080p, 8 bits: 188 us; a warp a row on its own, handing over every step through L2 (a device-scope release and an
// acquire, ~3 us a step), took 822 us.
constexpr int DBK_ROWS = 4;
constexpr int DBK_AHEAD = 4;
constexpr int DBK_GROUP_THREADS = (DBK_ROWS + 2) * 32;
// Polls of a shared-memory word before a warp gives up: four to one of global memory, which sleeps between most of them.
__device__ __forceinline__ unsigned dbk_spins(const DbkParams& P) { return P.wait_limit < 1u << 30 ? P.wait_limit << 2 : ~0u; }

template <class T>
struct DbkGroup {
    static constexpr int RING = sizeof(T) == 1 ? 8 : 4;  // macroblocks a ring holds
    __align__(16) T ring[DBK_ROWS][RING][64];            // above row j: luma [4][16], chroma [comp][2][8]
    __align__(16) T own[DBK_ROWS][DBK_AHEAD][256];       // luma [16][16], chroma [comp][8][8]
    __align__(16) DbkEdges e[DBK_ROWS][DBK_AHEAD];
    unsigned prog[DBK_ROWS + 1];  // [j]: macroblocks whose bottom rows above row j are final
    unsigned cons[DBK_ROWS];      // [j]: macroblocks row j has done with
    unsigned stop, ticket;
};

template <int NB>
__device__ __forceinline__ void dbk_cp_async(void* dst, const void* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (NB == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// Waits until the shared word reaches `need`; false when it gave up or another warp of the group did.
template <class T>
__device__ __forceinline__ bool dbk_spin(const DbkParams& P, DbkGroup<T>& G, const unsigned* w, unsigned need) {
    for (unsigned i = 0;; i++) {
        if (ld_acquire_cta(w) >= need) return true;
        if ((i & 15) == 15) {
            if (ld_acquire_cta(&G.stop)) return false;
            if (i >= dbk_spins(P)) {
                atomicOr(P.err, 1u);
                st_release_cta(&G.stop, 1u);
                return false;
            }
            __nanosleep(20);
        }
    }
}

// NW 32-bit words between registers and memory (16-, 8- or 4-byte pieces; the address aligned to them).
template <int NW>
__device__ __forceinline__ void dbk_words_ld(const void* p, uint32_t* w) {
    if constexpr (NW % 4 == 0) {
#pragma unroll
        for (int k = 0; k < NW / 4; k++) {
            const uint4 q = reinterpret_cast<const uint4*>(p)[k];
            w[4 * k] = q.x, w[4 * k + 1] = q.y, w[4 * k + 2] = q.z, w[4 * k + 3] = q.w;
        }
    } else {
        const uint2 q = *reinterpret_cast<const uint2*>(p);
        w[0] = q.x, w[1] = q.y;
    }
}
template <int NW>
__device__ __forceinline__ void dbk_words_st(void* p, const uint32_t* w) {
    if constexpr (NW % 4 == 0) {
#pragma unroll
        for (int k = 0; k < NW / 4; k++) reinterpret_cast<uint4*>(p)[k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
    } else {
        *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
    }
}
// N samples of type T from ints to shared memory at p (aligned to their size).
template <class T, int N>
__device__ __forceinline__ void dbk_store_shared(T* p, const int* v) {
#pragma unroll
    for (int k = 0; k < N; k++) p[k] = (T)v[k];
}
template <class T>
__device__ __forceinline__ int dbk_sample(const uint32_t* w, int k) {
    return (int)((w[(k * (int)sizeof(T)) >> 2] >> ((k * 8 * (int)sizeof(T)) & 31)) & ((1u << (8 * sizeof(T))) - 1));
}

// Row j of the group (macroblock row y), left to right, by one warp. Luma: lanes 0-15 hold the macroblock's
// 16 rows; chroma: lanes 0-7 the Cb rows, 8-15 the Cr rows; lanes 16-31 work on the same lines and store nothing, so that
// the warp does not diverge. The vertical edges are filtered in those registers, with the LEFT samples kept from the
// previous macroblock; the outer one makes the previous macroblock final, so its last columns go out and its bottom rows are
// published. The horizontal edges are filtered on columns, the macroblock in its staging buffer and the rows above in
// the ring. below: this group has a row j + 1, which the ring above it is filled for.
template <class T, bool CHROMA>
__device__ __forceinline__ void dbk_group_row(const DbkParams& P, const DbkEdges* __restrict__ edges, DbkGroup<T>& G, int j, int y, bool below) {
    constexpr int W = CHROMA ? 8 : 16;    // samples of a macroblock row (and rows)
    constexpr int LEFT = CHROMA ? 2 : 4;  // samples kept to its left
    constexpr int H = CHROMA ? 2 : 4;     // rows above
    constexpr int NE = CHROMA ? 2 : 4;    // edges a direction
    constexpr int NW = W * (int)sizeof(T) / 4;
    constexpr int N = DbkGroup<T>::RING;
    constexpr int RB = W * (int)sizeof(T);  // bytes of a macroblock row
    const int lane = threadIdx.x & 31, ln = lane & 15;
    const bool active = lane < 16;
    const int comp = CHROMA ? ln >> 3 : 0, line = CHROMA ? ln & 7 : ln;
    T* const Pl = reinterpret_cast<T*>(P.planes[CHROMA ? 1 + comp : 0]);
    const int stride = CHROMA ? P.cs : P.ys, mb_w = P.mb_w, bd = P.bd;
    T* const grow = Pl + (size_t)(y * W + line) * stride;       // this lane's row
    T* const gtop = Pl + ((ptrdiff_t)y * W - H + line) * stride;  // lanes line < H: a row above
    const DbkEdges* const erow = edges + (size_t)y * mb_w;
    const int maxv = (1 << bd) - 1, sh = 8 * (CHROMA ? line >> 1 : line >> 2);
    const bool bottom = active && below && line >= W - H, above = active && y > 0 && line >= 1 && line < H;
    const int rrow = (CHROMA ? comp * 16 : 0) + (line - (W - H)) * W;  // a bottom row's place in a ring slot
    // macroblock x's samples and edge words into stage x % DBK_AHEAD
    auto issue = [&](int x) {
        if (x < mb_w) {
            const int s = x % DBK_AHEAD;
            if (active) {
                const uint8_t* g = reinterpret_cast<const uint8_t*>(grow + x * W);
                uint8_t* d = reinterpret_cast<uint8_t*>(G.own[j][s]) + ln * RB;
                dbk_cp_async<(RB < 16 ? 8 : 16)>(d, g);
                if constexpr (RB == 32) dbk_cp_async<16>(d + 16, g + 16);
            } else if (lane < 22) {
                dbk_cp_async<16>(reinterpret_cast<uint4*>(&G.e[j][s]) + (lane - 16), reinterpret_cast<const uint4*>(&erow[x]) + (lane - 16));
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int k = 0; k < DBK_AHEAD - 1; k++) issue(k);
    int left[LEFT];
#pragma unroll
    for (int k = 0; k < LEFT; k++) left[k] = 0;
    for (int x = 0; x < mb_w; x++) {
        issue(x + DBK_AHEAD - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(DBK_AHEAD - 1) : "memory");
        __syncwarp();
        const int s = x % DBK_AHEAD;
        T* const own = G.own[j][s];
        const DbkEdges& E = G.e[j][s];
        uint32_t rw[NW];
        dbk_words_ld<NW>(own + ln * W, rw);
        // the words of the two directions: luma's four edges; chroma's two, of this lane's component
        uint32_t vw[NE], hw[NE];
        bool vany, hany, v0, top;
        if constexpr (CHROMA) {
            const uint4 a = *reinterpret_cast<const uint4*>(E.chroma[0]), b = *reinterpret_cast<const uint4*>(E.chroma[1]);
            vany = (a.x | a.y | b.x | b.y) != 0, hany = (a.z | a.w | b.z | b.w) != 0;
            v0 = (a.x | b.x) != 0, top = y > 0 && (a.z | b.z) != 0;
            vw[0] = comp ? b.x : a.x, vw[1] = comp ? b.y : a.y, hw[0] = comp ? b.z : a.z, hw[1] = comp ? b.w : a.w;
        } else {
            dbk_words_ld<4>(E.luma[0], vw);
            dbk_words_ld<4>(E.luma[1], hw);
            vany = (vw[0] | vw[1] | vw[2] | vw[3]) != 0, hany = (hw[0] | hw[1] | hw[2] | hw[3]) != 0;
            v0 = vw[0] != 0, top = y > 0 && hw[0] != 0;
        }
        uint32_t bq[8];
        dbk_words_ld<8>(E.bs[0], bq);
        int lv[LEFT + W];
        DbkEdge ve[NE];
        if (vany) {
#pragma unroll
            for (int k = 0; k < NE; k++) ve[k] = dbk_edge(vw[k], (int)((bq[CHROMA ? 2 * k : k] >> sh) & 0xff), bd);
#pragma unroll
            for (int k = 0; k < LEFT; k++) lv[k] = left[k];
#pragma unroll
            for (int k = 0; k < W; k++) lv[LEFT + k] = dbk_sample<T>(rw, k);
            if (v0) {
                // (x > 0: an outer edge at the picture's left has no word) the previous macroblock's last columns are final now
                dbk_outer<CHROMA>(lv, ve, maxv);
                if (active) dbk_store<T, LEFT>(grow + x * W - LEFT, lv);
                if (bottom) dbk_store_shared<T, LEFT>(G.ring[j + 1][(x - 1) % N] + rrow + W - LEFT, lv);
            }
        }
        __syncwarp();
        // published as soon as the outer edge is done: the row below waits for no more than that
        if (lane == 0) {
            __threadfence_block();
            st_shared(&G.prog[j + 1], (unsigned)x);
            st_shared(&G.cons[j], (unsigned)x);
        }
        if (vany) {
            dbk_inner<CHROMA>(lv, ve, maxv);
#pragma unroll
            for (int k = 0; k < NW; k++) {
                constexpr int PER = 4 / (int)sizeof(T);
                uint32_t w = (uint32_t)lv[LEFT + PER * k];
#pragma unroll
                for (int i = 1; i < PER; i++) w |= (uint32_t)lv[LEFT + PER * k + i] << (8 * (int)sizeof(T) * i);
                rw[k] = w;
            }
        }
        if (hany) {
            if (vany) {
                if (active) dbk_words_st<NW>(own + ln * W, rw);
                __syncwarp();
            }
            T* const rg = G.ring[j][x % N] + (CHROMA ? comp * 16 : 0);
            T* const ow = own + (CHROMA ? comp * 64 : 0);
            DbkEdge he[NE];
#pragma unroll
            for (int k = 0; k < NE; k++) he[k] = dbk_edge(hw[k], (int)((bq[4 + (CHROMA ? 2 * k : k)] >> sh) & 0xff), bd);
            int cv[H + W];
#pragma unroll
            for (int k = 0; k < W; k++) cv[H + k] = (int)ow[k * W + line];
            if (top) {
                if (!__all_sync(DBK_ALL, dbk_spin(P, G, &G.prog[j], (unsigned)(x + 1)))) return;
#pragma unroll
                for (int k = 0; k < H; k++) cv[k] = (int)rg[k * W + line];
                dbk_outer<CHROMA>(cv, he, maxv);
                if (active) {
#pragma unroll
                    for (int k = 1; k < H; k++) rg[k * W + line] = (T)cv[k];
                }
            }
            dbk_inner<CHROMA>(cv, he, maxv);
            if (active) {
#pragma unroll
                for (int k = 0; k < W; k++) ow[k * W + line] = (T)cv[H + k];
            }
            __syncwarp();
            dbk_words_ld<NW>(own + ln * W, rw);
            if (top && above) {
                // the rows above, final in this macroblock's columns: the row above has applied the next one's left edge
                uint32_t tw[NW];
                dbk_words_ld<NW>(rg + line * W, tw);
                dbk_words_st<NW>(gtop + x * W, tw);
            }
        }
        if (active && (vany || hany)) dbk_words_st<NW>(grow + x * W, rw);
        if (below) {
            if (x >= N && !__all_sync(DBK_ALL, dbk_spin(P, G, &G.cons[j + 1], (unsigned)(x - N + 1)))) return;
            if (bottom) dbk_words_st<NW>(G.ring[j + 1][x % N] + rrow, rw);
        }
#pragma unroll
        for (int k = 0; k < LEFT; k++) left[k] = dbk_sample<T>(rw, W - LEFT + k);
    }
    __syncwarp();
    if (lane == 0) {
        __threadfence_block();
        st_shared(&G.prog[j + 1], (unsigned)mb_w);
        st_shared(&G.cons[j], (unsigned)mb_w);
    }
}

// The group's fetch warp: the bottom rows of macroblock row y - 1 (another CTA's, published in `above`) into ring 0,
// up to eight macroblocks at a time (a lane per macroblock and row), as far as they are published and the ring has room.
template <class T, bool CHROMA>
__device__ __forceinline__ void dbk_group_fetch(const DbkParams& P, DbkGroup<T>& G, int y, const unsigned* above) {
    constexpr int W = CHROMA ? 8 : 16, H = CHROMA ? 2 : 4, NW = W * (int)sizeof(T) / 4;
    constexpr unsigned N = DbkGroup<T>::RING;
    const int lane = threadIdx.x & 31, r = lane & 3;
    const T* const src = CHROMA ? reinterpret_cast<const T*>(P.planes[1 + (r >> 1)]) + (size_t)(y * W - H + (r & 1)) * P.cs
                                : reinterpret_cast<const T*>(P.planes[0]) + (size_t)(y * W - H + r) * P.ys;
    unsigned f = 0;
    const unsigned n = (unsigned)P.mb_w;
    for (unsigned i = 0; f < n; i++) {
        // macroblocks the first row has already passed (their top edges are not filtered) need no fetching
        const unsigned c = __shfl_sync(DBK_ALL, ld_acquire_cta(&G.cons[0]), 0);
        f = max(f, c);
        const unsigned p = __shfl_sync(DBK_ALL, ld_relaxed(above), 0);
        const unsigned lim = min(p, c + N);
        if (f < lim) {
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            const unsigned k = min(lim - f, 8u), m = f + (unsigned)(lane >> 2);
            if (m < f + k) {
                const uint4* g = reinterpret_cast<const uint4*>(src + (size_t)m * W);
                T* d = G.ring[0][m % N] + r * W;
                if constexpr (NW == 2) {
                    *reinterpret_cast<uint2*>(d) = __ldcg(reinterpret_cast<const uint2*>(g));
                } else {
#pragma unroll
                    for (int q = 0; q < NW / 4; q++) reinterpret_cast<uint4*>(d)[q] = __ldcg(g + q);
                }
            }
            __syncwarp();
            f += k;
            if (lane == 0) st_release_cta(&G.prog[0], f);
            i = 0;
            continue;
        }
        if ((i & 63) == 63) {
            const bool gone = (ld_acquire(P.err) & 1u) || ld_acquire_cta(&G.stop);
            if (__any_sync(DBK_ALL, gone) || i >= P.wait_limit) {
                if (lane == 0) {
                    atomicOr(P.err, 1u);
                    st_release_cta(&G.stop, 1u);
                }
                return;
            }
        }
        if (i >= 16) __nanosleep(64);
    }
}

// The group's publishing warp: the last row's progress (nr rows in the group) for the group below, each time it moves.
template <class T>
__device__ __forceinline__ void dbk_group_publish(const DbkParams& P, DbkGroup<T>& G, int nr, unsigned* mine) {
    const int lane = threadIdx.x & 31;
    unsigned last = 0;
    for (unsigned i = 0; last < (unsigned)P.mb_w; i++) {
        const unsigned p = __shfl_sync(DBK_ALL, ld_acquire_cta(&G.prog[nr]), 0);
        if (p > last) {
            // the row's stores, seen by this warp through the shared word, before the device-scope release
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            if (lane == 0) st_release(mine, p);
            last = p;
            i = 0;
            continue;
        }
        if ((i & 15) == 15) {
            if (__any_sync(DBK_ALL, ld_acquire_cta(&G.stop) != 0)) return;
            if (i >= dbk_spins(P)) {
                if (lane == 0) {
                    atomicOr(P.err, 1u);
                    st_release_cta(&G.stop, 1u);
                }
                return;
            }
        }
        __nanosleep(20);
    }
}

// One group of a picture by the whole CTA: local ticket lt = 2 * group + (1 for chroma).
template <class T>
__device__ __forceinline__ void dbk_group(const DbkParams& P, const DbkEdges* __restrict__ edges, DbkGroup<T>& G, unsigned lt) {
    const int tid = threadIdx.x, w = tid >> 5;
    const bool chroma = (lt & 1u) != 0;
    const int y0 = (int)(lt >> 1) * DBK_ROWS, nr = min(DBK_ROWS, P.mb_h - y0);
    if (tid <= DBK_ROWS) G.prog[tid] = 0;
    if (tid < DBK_ROWS) G.cons[tid] = 0;
    if (tid == 0) G.stop = 0;
    __syncthreads();
    unsigned* const words = P.progress + (chroma ? P.mb_h : 0);
    if (w < DBK_ROWS) {
        if (w < nr) {
            if (chroma) dbk_group_row<T, true>(P, edges, G, w, y0 + w, w + 1 < nr);
            else dbk_group_row<T, false>(P, edges, G, w, y0 + w, w + 1 < nr);
            asm volatile("cp.async.wait_all;" ::: "memory");  // none left in flight, also where a wait gave up
        }
    } else if (w == DBK_ROWS) {
        if (y0 > 0) {
            if (chroma) dbk_group_fetch<T, true>(P, G, y0, words + y0 - 1);
            else dbk_group_fetch<T, false>(P, G, y0, words + y0 - 1);
        }
    } else if (y0 + nr < P.mb_h) {
        dbk_group_publish<T>(P, G, nr, words + y0 + nr - 1);
    }
    __syncthreads();
}

__host__ __device__ constexpr int dbk_groups(int mb_h) { return (mb_h + DBK_ROWS - 1) / DBK_ROWS; }

// Pass 2: the groups of the two plane kinds handed out by ticket; a group waits only on the group above of
// its own kind, which holds a smaller ticket.
template <class T>
__global__ void __launch_bounds__(DBK_GROUP_THREADS, 2) deblock_rows_kernel(const __grid_constant__ DbkParams P,
                                                                            const DbkEdges* __restrict__ edges) {
    __shared__ DbkGroup<T> G;
    for (;;) {
        if (threadIdx.x == 0) G.ticket = atomicAdd(P.ticket, 1u);
        __syncthreads();
        const unsigned t = G.ticket;
        if (t >= 2u * (unsigned)dbk_groups(P.mb_h)) return;
        dbk_group<T>(P, edges, G, t);
        if (__syncthreads_or((int)(ld_acquire(P.err) & 1u))) return;
    }
}

// ---- many streams in one launch per pass (the batched form) ------------------------------------------

// One stream of a batched deblocking launch: its parameters (planes, records, slices, progress words, the
// batch's ticket and error words), its edge records, and its first macroblock in the launch's flat index.
struct DbkJob {
    DbkParams P;
    DbkEdges* edges;
    int mb0;
};

// Pass 1 for every stream: the flat macroblock index over the streams (stream by binary search on mb0).
static __global__ void __launch_bounds__(DBK_WARPS * 32) deblock_edges_batch_kernel(const DbkJob* __restrict__ jobs, int njobs, int total) {
    __shared__ ironav_dbk_mb rec[DBK_WARPS][3];
    __shared__ uint8_t bsm[DBK_WARPS][2][4][4];
    const int wid = threadIdx.x >> 5;
    for (int idx = blockIdx.x * DBK_WARPS + wid; idx < total; idx += gridDim.x * DBK_WARPS) {
        int lo = 0, hi = njobs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (jobs[mid].mb0 <= idx) lo = mid;
            else hi = mid - 1;
        }
        const DbkJob& J = jobs[lo];
        dbk_edges_mb(J.P, J.edges, idx - J.mb0, rec[wid], bsm[wid]);
    }
}

// Pass 2 for every stream: ticket t is order[t] = stream << 20 | the stream's own group ticket (dbk_group), the
// streams' groups interleaved by their own tickets, so a group waits only on its own stream's group above, which
// holds a smaller ticket.
template <class T>
__global__ void __launch_bounds__(DBK_GROUP_THREADS, 2) deblock_rows_batch_kernel(const DbkJob* __restrict__ jobs,
                                                                                  const uint32_t* __restrict__ order, unsigned ntickets,
                                                                                  unsigned* ticket, const unsigned* err) {
    __shared__ DbkGroup<T> G;
    __shared__ DbkParams P;
    __shared__ const DbkEdges* edges;
    for (;;) {
        if (threadIdx.x == 0) {
            G.ticket = atomicAdd(ticket, 1u);
            if (G.ticket < ntickets) {
                const DbkJob& J = jobs[order[G.ticket] >> 20];
                P = J.P;
                edges = J.edges;
            }
        }
        __syncthreads();
        if (G.ticket >= ntickets) return;
        dbk_group<T>(P, edges, G, order[G.ticket] & 0xFFFFFu);
        if (__syncthreads_or((int)(ld_acquire(err) & 1u))) return;
    }
}

}  // namespace ironav
