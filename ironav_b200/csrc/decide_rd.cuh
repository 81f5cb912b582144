// decide_rd.cuh — K9: code_mb with CABAC on the device (the reference encoder's default decision: decide_rd,
// enc/frame.rs:1462-1513, after code_mb's P_Skip tests, best_i16 and best_inter, 715-760), and the CABAC
// slice writer.
//
// Under CABAC a macroblock's rate-distortion cost counts its bins against the slice's contexts as the
// macroblocks before it left them, so a slice band is one chain in raster order: a CTA of five warps walks a band. For each
// macroblock every candidate the reference tries is coded (P_Skip, best_inter's partitioning with the 4x4 and, with
// transform8, the 8x8 transform, Intra16x16, Intra4x4, Intra8x8, each intra one with its chroma), into the picture or a scratch
// plane and then into shared memory (code and reconstruction), with its squared error, and its bins are priced on its own copy
// of the contexts (cab::price); the least SSD + lambda2 * bits in the reference's order (strict '<') is kept, and its code,
// reconstruction and advanced contexts are copied into place.
//
// The candidates reuse decide mode's warp-level coders (decide.cuh, residual.cuh); Intra8x8 (code_i8,
// enc/frame.rs:1307-1388) is coded here: block by block, its edges filtered (8.3.2.2.1), nine modes'
// SATD over 36 lane-units of (mode, 4x4 quadrant) from a table of the predictors (i8_entry), the chosen
// block's 8x8 transform on eight lanes.
#pragma once
#include <type_traits>

#include "cabac.cuh"
#include "decide.cuh"

namespace ironav {

constexpr int RD_CANDS = 6;  // P_Skip, inter with the 4x4 transform, inter with the 8x8, Intra16x16, Intra4x4, Intra8x8

struct RdParams {
    DecideParams D;         // decide mode's parameters: the analysis, the coder, the outputs (codes, states)
    uint32_t* nbs;          // per macroblock, what the contexts read of it as a neighbour (cab::Nb, NB_WORDS words)
    const int* band_rows;   // chain i walks the rows [band_rows[i], band_rows[i + 1])
    const uint32_t* step;   // the contexts' step table (cab::STEP_ENTRIES)
    double lam2;            // 1.6 * 2^((QP'Y - 12) / 3), computed on the host in f64 as the reference does
    int nbands;
    int t8;                 // transform_8x8_mode_flag
    // the scratch planes of warps 1 to 4 (luma, Cb, Cr of each), pw x ph and cw x ch samples, rows scr_ys
    // and scr_cs samples apart
    uint8_t* scr[12];
    int scr_ys, scr_cs;
};

template <class T, int W>
struct RdSmem {
    DecideSmem<T> s[W];              // each warp's working set
    ironav_mbcode cand[RD_CANDS];    // the candidates' codes
    __align__(16) T crec[RD_CANDS][384];  // and reconstructions (luma, Cb, Cr)
    __align__(16) uint8_t live[1024];           // the chain's contexts after the macroblocks before this one
    __align__(16) uint8_t cst[RD_CANDS][1024];  // each candidate's copy, advanced by its bins
    uint16_t list[W][cab::PRICE_CAP];           // each warp's list of bins
    uint32_t step[cab::STEP_ENTRIES];
    cab::Nb nb[2];                   // the left and top neighbours as the contexts see them
    cab::Nb done;                    // the macroblock just decided, the next one's left
    ironav_mbstate state[RD_CANDS];  // each candidate's MbState
    long long ssd[RD_CANDS];
    long long cssd[RD_CANDS];        // the chroma part of ssd
    unsigned bits[RD_CANDS];
    int valid[RD_CANDS];
    // of the macroblocks a group tests for P_Skip, the verdict, the skip vector and the top neighbour; the intra
    // chroma's coded block pattern bits; best_inter's decision for the 8x8-transform candidate, and whether that is tried
    int skip[W];
    int2 sv[W];
    cab::Nb top[W], nbs[W];          // (nbs: the P_Skip macroblocks' own)
    uint32_t ccbp;
    uint16_t idec[40];
    int try_t8;
    // the Intra8x8 trial
    int i8rec[256];       // its reconstruction
    int raw[25], e8[26];  // a block's edges, raw and filtered: [0] top-left, [1 + i] the 16 above, [17 + j] the 8 left,
                          // e8[25] the DC mode's value
    unsigned i8tab[9 * 64];  // i8_entry per mode and sample
    int sat[36];          // SATD per (mode, 4x4 quadrant)
    int pred8[64];
    int t8b[8][9];
    int co8b[64];
    int16_t lv8b[64];
    uint8_t i8modes[16];
    int i8meta[4];        // chosen mode, predicted mode, DC value, non-zero levels
};

// The 8x8 intra predictors as a table, as decide mode's 4x4 ones (i4_entry): every sample of every mode is
// (E[a] + 2 E[b] + E[c] + 2) >> 2 over the block's filtered edge array E (E[0] the top-left sample, E[1 + i]
// the 16 above, E[17 + j] the 8 to the left, E[25] the DC mode's value): a copy has a = b = c, a two-sample
// average (p + q + 1) >> 1 has a = c = p, b = q, and (p + 3q + 2) >> 2 has b = c = q. Entry: a | b << 5 | c << 10.
// The cases are predict_nxn's for n = 8 (h264/intra.rs:30-128; ITU-T H.264 8.3.2.2.2-8.3.2.2.10).
__device__ __forceinline__ unsigned i8_entry(int mode, int x, int y) {
    auto T = [](int i) { return i < 0 ? 0 : 1 + i; };
    auto L = [](int j) { return j < 0 ? 0 : 17 + j; };
    auto E3 = [](int a, int b, int c) { return (unsigned)(a | b << 5 | c << 10); };
    switch (mode) {
    case 0: return E3(T(x), T(x), T(x));
    case 1: return E3(L(y), L(y), L(y));
    case 2: return E3(25, 25, 25);
    case 3: return (x == 7 && y == 7) ? E3(T(14), T(15), T(15)) : E3(T(x + y), T(x + y + 1), T(x + y + 2));
    case 4:
        if (x > y) return E3(T(x - y - 2), T(x - y - 1), T(x - y));
        if (x < y) return E3(L(y - x - 2), L(y - x - 1), L(y - x));
        return E3(T(0), 0, L(0));
    case 5: {
        const int z = 2 * x - y, i = x - (y >> 1);
        if (z >= 0 && (z & 1) == 0) return E3(T(i - 1), T(i), T(i - 1));
        if (z >= 0) return E3(T(i - 2), T(i - 1), T(i));
        if (z == -1) return E3(L(0), 0, T(0));
        return E3(L(y - 2 * x - 1), L(y - 2 * x - 2), L(y - 2 * x - 3));
    }
    case 6: {
        const int z = 2 * y - x, j = y - (x >> 1);
        if (z >= 0 && (z & 1) == 0) return E3(L(j - 1), L(j), L(j - 1));
        if (z >= 0) return E3(L(j - 2), L(j - 1), L(j));
        if (z == -1) return E3(L(0), 0, T(0));
        return E3(T(x - 2 * y - 1), T(x - 2 * y - 2), T(x - 2 * y - 3));
    }
    case 7: {
        const int i = x + (y >> 1);
        return (y & 1) == 0 ? E3(T(i), T(i + 1), T(i)) : E3(T(i), T(i + 1), T(i + 2));
    }
    default: {
        const int z = x + 2 * y, j = y + (x >> 1);
        if (z > 13) return E3(L(7), L(7), L(7));
        if (z == 13) return E3(L(6), L(7), L(7));
        if ((z & 1) == 0) return E3(L(j), L(j + 1), L(j));
        return E3(L(j), L(j + 1), L(j + 2));
    }
    }
}

__device__ __forceinline__ int i8_pred(const int* E, unsigned e) { return (E[e & 31] + 2 * E[(e >> 5) & 31] + E[e >> 10] + 2) >> 2; }

// code_i8, enc/frame.rs:1307-1388: the luma of an Intra8x8 macroblock, block by block in S.i8rec (each
// block predicted from the filtered edges of the reconstruction so far, its mode the cheapest by SATD +
// lambda * (1 predicted, 4 otherwise), quantised with the intra rounding), its levels, modes and counts
// into out (zeroed by the caller with the Intra4x4 modes 2), and the reconstruction into wy.
// Returns the luma coded block pattern (every lane).
template <class T, int W>
__device__ uint32_t code_i8_d(const DecideParams& P, DecideSmem<T>& S, RdSmem<T, W>& R, int mbx, int mby, bool ta, bool la, bool tra,
                              ironav_mbcode* out, T* wy, int wys) {
    // P.C.rec: the picture the edges are read from; wy (rows wys samples apart): where the luma goes. The
    // predictor table of R.i8tab is filled once a chain (rdw_chain)
    const int lane = threadIdx.x & 31;
    const CodeParams& C = P.C;
    const int bd = C.bd, maxv = (1 << bd) - 1, lam = C.A.lambda;
    const int qp = C.qp + 6 * (bd - 8), m6 = qp % 6, qbits = 16 + qp / 6, f = (1 << qbits) / 3;
    const T* Y = reinterpret_cast<const T*>(C.rec[0]);
    const int x0 = mbx * 16, y0 = mby * 16;
    if (lane < 16) R.i8modes[lane] = 2;
    __syncwarp();
    uint32_t cbp = 0;
    for (int i8 = 0; i8 < 4; i8++) {
        const int bx = i8 & 1, by = i8 >> 1;
        const bool hl = bx > 0 || la, ht = by > 0 || ta;
        const bool htl = bx > 0 ? (by > 0 ? true : ta) : (by > 0 ? la : (la && ta));
        const bool htr = i8 == 0 ? ta : (i8 == 1 ? tra : i8 == 2);
        // the raw edges: the row above (the top-right half after the rest), the column to the left, the corner
        if (lane < 8) {
            const int x = bx * 8 + lane;
            R.raw[1 + lane] = !ht ? 0 : (by == 0 ? S.top[1 + x] : R.i8rec[7 * 16 + x]);
            R.raw[17 + lane] = !hl ? 0 : (bx == 0 ? S.left[by * 8 + lane] : R.i8rec[(by * 8 + lane) * 16 + 7]);
        } else if (lane == 8) {
            int v = 0;
            if (htl) v = by == 0 ? S.top[bx * 8] : (bx == 0 ? S.left[7] : R.i8rec[7 * 16 + 7]);
            R.raw[0] = v;
        }
        __syncwarp();
        if (lane < 8) {
            int v = 0;
            if (ht) {
                if (!htr) v = R.raw[8];  // the last sample above, repeated
                else if (by == 1) v = R.i8rec[7 * 16 + 8 + lane];
                else if (bx == 0) v = S.top[1 + 8 + lane];
                else v = (int)Y[(size_t)(y0 - 1) * C.ys + x0 + 16 + lane];  // the top-right macroblock's bottom row
            }
            R.raw[9 + lane] = v;
        }
        __syncwarp();
        // filter_8x8_edges, h264/intra.rs:131-158
        if (lane < 25) {
            const int* p = R.raw;
            int v = p[lane];
            if (lane == 0) {
                if (htl) {
                    if (ht && hl) v = (p[1] + 2 * p[0] + p[17] + 2) >> 2;
                    else if (ht) v = (3 * p[0] + p[1] + 2) >> 2;
                    else if (hl) v = (3 * p[0] + p[17] + 2) >> 2;
                }
            } else if (lane <= 16) {
                const int x = lane - 1;
                if (ht) {
                    if (x == 0) v = htl ? (p[0] + 2 * p[1] + p[2] + 2) >> 2 : (3 * p[1] + p[2] + 2) >> 2;
                    else if (x == 15) v = (p[15] + 3 * p[16] + 2) >> 2;
                    else v = (p[x] + 2 * p[x + 1] + p[x + 2] + 2) >> 2;
                }
            } else {
                const int y = lane - 17;
                if (hl) {
                    if (y == 0) v = htl ? (p[0] + 2 * p[17] + p[18] + 2) >> 2 : (3 * p[17] + p[18] + 2) >> 2;
                    else if (y == 7) v = (p[23] + 3 * p[24] + 2) >> 2;
                    else v = (p[16 + y] + 2 * p[17 + y] + p[18 + y] + 2) >> 2;
                }
            }
            R.e8[lane] = v;
        }
        __syncwarp();
        if (lane == 0) {
            const int* E = R.e8;
            int st = 0, sl = 0;
            for (int i = 0; i < 8; i++) st += E[1 + i], sl += E[17 + i];
            R.i8meta[2] = (ht && hl) ? (st + sl + 8) >> 4 : (hl ? (sl + 4) >> 3 : (ht ? (st + 4) >> 3 : 1 << (bd - 1)));
            R.e8[25] = R.i8meta[2];
            R.i8meta[1] = cab::pred_mode(S.nbm, R.i8modes, bx * 2, by * 2);
        }
        __syncwarp();
        // the nine modes' SATD, a lane per (mode, 4x4 quadrant)
        for (int u = lane; u < 36; u += 32) {
            const int mode = u >> 2, q = u & 3;
            const bool ok = (mode == 0 || mode == 3 || mode == 7) ? ht : (mode == 1 || mode == 8) ? hl : mode == 2 ? true : (ht && hl && htl);
            int s = 0;
            if (ok) {
                int d[16];
#pragma unroll
                for (int r = 0; r < 4; r++)
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int px = (q & 1) * 4 + k, py = (q >> 1) * 4 + r;
                        d[r * 4 + k] = src_at(S.a, bx * 8 + px, by * 8 + py) - i8_pred(R.e8, R.i8tab[mode * 64 + py * 8 + px]);
                    }
                s = satd4_d(d);
            }
            R.sat[u] = ok ? s : -1;
        }
        __syncwarp();
        if (lane == 0) {
            int bm = 2, bc = 0x7fffffff;
            for (int mode = 0; mode < 9; mode++) {
                if (R.sat[mode * 4] < 0) continue;
                const int c = R.sat[mode * 4] + R.sat[mode * 4 + 1] + R.sat[mode * 4 + 2] + R.sat[mode * 4 + 3] +
                              lam * (mode == R.i8meta[1] ? 1 : 4);
                if (c < bc) bm = mode, bc = c;
            }
            R.i8meta[0] = bm;
        }
        __syncwarp();
        const int bm = R.i8meta[0];
        for (int i = lane; i < 64; i += 32) R.pred8[i] = i8_pred(R.e8, R.i8tab[bm * 64 + i]);
        __syncwarp();
        // quant8 (intra rounding) and idct8_add, enc/frame.rs:56-72 and h264/idct.rs:33-74, eight lanes
        const int j = lane & 7;
        if (lane < 8) {
            int d[8], o[8];
#pragma unroll
            for (int k = 0; k < 8; k++) d[k] = src_at(S.a, bx * 8 + k, by * 8 + j) - R.pred8[j * 8 + k];
            q_fdct8_1d_d(d, o);
#pragma unroll
            for (int k = 0; k < 8; k++) R.t8b[j][k] = o[k];
        }
        __syncwarp();
        if (lane < 8) {
            int d[8], o[8];
#pragma unroll
            for (int k = 0; k < 8; k++) d[k] = R.t8b[k][j];
            q_fdct8_1d_d(d, o);
#pragma unroll
            for (int k = 0; k < 8; k++) R.co8b[k * 8 + j] = o[k];
        }
        __syncwarp();
        int dq[8];
        int nz = 0;
        if (lane < 8) {
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int sk = j * 8 + k, pz = c_zz8[sk];
                const int l = q_quant_d(R.co8b[pz], c_q_mf8[m6][q_class8_d(pz)], f, qbits);
                R.lv8b[sk] = (int16_t)l;
                nz += l != 0;
                int v = 0;
                if (l != 0) {
                    const int vv = l * 16 * c_q_dq8[m6][q_class8_d(pz)];
                    v = qp >= 36 ? vv << (qp / 6 - 6) : (vv + (1 << (5 - qp / 6))) >> (6 - qp / 6);
                }
                dq[k] = v;
            }
        }
        __syncwarp();
        if (lane < 8) {
#pragma unroll
            for (int k = 0; k < 8; k++) R.co8b[c_zz8[j * 8 + k]] = dq[k];
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) nz += __shfl_xor_sync(FULL, nz, off);
        __syncwarp();
        if (lane < 8 && nz > 0) {
            int d[8], o[8];
#pragma unroll
            for (int k = 0; k < 8; k++) d[k] = R.co8b[j * 8 + k];
            q_row8_d(d, o);
#pragma unroll
            for (int k = 0; k < 8; k++) R.t8b[j][k] = o[k];
        }
        __syncwarp();
        if (lane < 8) {
            int o[8];
            if (nz > 0) {
                int d[8];
#pragma unroll
                for (int k = 0; k < 8; k++) d[k] = R.t8b[k][j];
                q_row8_d(d, o);
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int pv = R.pred8[i * 8 + j];
                R.i8rec[(by * 8 + i) * 16 + bx * 8 + j] = nz > 0 ? min(max(pv + ((o[i] + 32) >> 6), 0), maxv) : pv;
            }
        }
        for (int k = lane; k < 64; k += 32) out->res.luma8[i8][k] = R.lv8b[k];
        if (lane < 4) {
            const int b = (by * 2 + (lane >> 1)) * 4 + bx * 2 + (lane & 1);
            R.i8modes[b] = (uint8_t)bm;
            out->res.nnz[b] = (uint8_t)nz;
        }
        if (nz > 0) cbp |= 1u << i8;
        __syncwarp();
    }
    for (int i = lane; i < 256; i += 32) wy[(size_t)(y0 + (i >> 4)) * wys + x0 + (i & 15)] = (T)R.i8rec[i];
    if (lane < 16) out->modes[lane] = R.i8modes[lane];
    if (lane == 0) {
        out->kind = KIND_I8;
        out->res.t8x8 = 1;
    }
    __syncwarp();
    return cbp;
}

// MbCode::new (enc/frame.rs:302-306): zero, the Intra4x4 modes 2 (words 371-374 of the code).
__device__ __forceinline__ void code_init(ironav_mbcode* o) {
    const int lane = threadIdx.x & 31;
    uint32_t* w = reinterpret_cast<uint32_t*>(o);
    for (int k = lane; k < (int)(sizeof(ironav_mbcode) / 4); k += 32) w[k] = (k >= 371 && k < 375) ? 0x02020202u : 0u;
    __syncwarp();
}

// A candidate coded into the planes C (the picture, or a warp's scratch planes): its squared error (ssd_mb,
// enc/frame.rs:1432-1449) and a copy of its reconstruction (save_mb, 1406-1417); chroma false: the luma
// only, the chroma added later from another candidate's. The candidate counts from here on.
template <class T, int W>
__device__ void rd_take(const CodeParams& C, RdSmem<T, W>& R, const DecideSmem<T>& S, int k, int mbx, int mby, bool chroma = true) {
    // a lane's half row of luma and four chroma samples, as words. The sums are 32 bits wide at 8 bits (384 squares of 255 fit), 64 at
    // 10, whose 16-bit samples are taken as they are given.
    const int lane = threadIdx.x & 31;
    constexpr int B = (int)sizeof(T);
    using Sum = std::conditional_t<B == 1, uint32_t, unsigned long long>;
    uint32_t* const dst = reinterpret_cast<uint32_t*>(R.crec[k]);
    __syncwarp();
    auto squares = [](uint32_t a, uint32_t b, Sum acc) {
        if constexpr (B == 1) {
            const uint32_t d = __vabsdiffu4(a, b);
            return __dp4a(d, d, acc);
        } else {
            const uint32_t lo = (uint32_t)abs((int)(a & 0xffffu) - (int)(b & 0xffffu)), hi = (uint32_t)abs((int)(a >> 16) - (int)(b >> 16));
            return acc + (Sum)lo * lo + (Sum)hi * hi;
        }
    };
    auto warp_sum = [](Sum v) {
        if constexpr (B == 1) {
            return __reduce_add_sync(FULL, v);
        } else {
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) v += __shfl_xor_sync(FULL, v, off);
            return v;
        }
    };
    Sum ssd = 0, cssd = 0;
    {
        const int row = lane >> 1, half = lane & 1;
        const uint32_t* rec = reinterpret_cast<const uint32_t*>(reinterpret_cast<const T*>(C.rec[0]) + (size_t)(mby * 16 + row) * C.ys + mbx * 16 + half * 8);
        const uint32_t* src = &S.a.src[(row * 4 + half * 2) * B];
        uint32_t v[2 * B], cv[B], cs[B];
#pragma unroll
        for (int i = 0; i < 2 * B; i++) v[i] = rec[i];
        if (chroma) {
            const int cc = lane >> 4, j = (lane & 15) * 4;
            const size_t at = (size_t)(mby * 8 + (j >> 3));
            const uint32_t* crec = reinterpret_cast<const uint32_t*>(reinterpret_cast<const T*>(C.rec[1 + cc]) + at * C.cs + mbx * 8 + (j & 7));
            const uint32_t* csrc = reinterpret_cast<const uint32_t*>(reinterpret_cast<const T*>(C.src_c) + (size_t)cc * C.cw * C.ch + at * C.cw + mbx * 8 + (j & 7));
#pragma unroll
            for (int i = 0; i < B; i++) cv[i] = crec[i], cs[i] = csrc[i];
        }
#pragma unroll
        for (int i = 0; i < 2 * B; i++) {
            dst[lane * 2 * B + i] = v[i];
            ssd = squares(v[i], src[i], ssd);
        }
        if (chroma) {
#pragma unroll
            for (int i = 0; i < B; i++) {
                dst[64 * B + lane * B + i] = cv[i];
                cssd = squares(cv[i], cs[i], cssd);
            }
            cssd = warp_sum(cssd);
        }
        ssd = warp_sum(ssd);
    }
    if (lane == 0) {
        R.ssd[k] = (long long)(ssd + cssd);
        R.cssd[k] = (long long)cssd;
        R.valid[k] = 1;
    }
    __syncwarp();
}

// An intra candidate's chroma taken from another's (code_intra_chroma's outputs: mode, DC and AC levels, counts).
__device__ __forceinline__ void rd_chroma_copy(const ironav_mbcode& from, ironav_mbcode* o) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    const uint32_t* ac = reinterpret_cast<const uint32_t*>(from.res.cac);
    uint32_t* oc = reinterpret_cast<uint32_t*>(o->res.cac);
    for (int i = lane; i < (int)(sizeof(from.res.cac) / 4); i += 32) oc[i] = ac[i];
    if (lane < (int)(sizeof(from.res.cdc) / 4)) reinterpret_cast<uint32_t*>(o->res.cdc)[lane] = reinterpret_cast<const uint32_t*>(from.res.cdc)[lane];
    if (lane < (int)(sizeof(from.res.cnnz) / 4))
        reinterpret_cast<uint32_t*>(o->res.cnnz)[lane] = reinterpret_cast<const uint32_t*>(from.res.cnnz)[lane];
    if (lane == 0) o->chroma_mode = from.chroma_mode;
    __syncwarp();
}

// Candidate k priced on warp w (rd_cost, enc/frame.rs:1453-1457), from its own copy of the contexts.
template <class T, int W>
__device__ __forceinline__ void rd_price(RdSmem<T, W>& R, const cab::Slice& sl, const int* nbm, int k, int w) {
    const uint32_t bits = cab::price(R.live, R.cst[k], R.step, R.list[w], sl, &R.cand[k], R.nb[0], R.nb[1], nbm);
    if ((threadIdx.x & 31) == 0) R.bits[k] = bits;
    __syncwarp();
}

// Intra candidate k's chroma: Intra16x16's code, reconstruction and squared error (k's luma is coded).
template <class T, int W>
__device__ __forceinline__ void rd_take_chroma(RdSmem<T, W>& R, int k) {
    const int lane = threadIdx.x & 31;
    rd_chroma_copy(R.cand[3], &R.cand[k]);
    if (lane == 0) {
        R.cand[k].res.cbp |= (uint8_t)R.ccbp;
        R.ssd[k] += R.cssd[3];
    }
    for (int i = 256 + lane; i < 384; i += 32) R.crec[k][i] = R.crec[3][i];
    __syncwarp();
}

// The candidate of least SSD + lam2 * bits, the first of them in the reference's order (strict '<'), in f64 rounded as the reference's
// expression is (no fused multiply-add); on every lane.
template <class T, int W>
__device__ __forceinline__ int rd_best(const RdParams& P, const RdSmem<T, W>& R) {
    const int lane = threadIdx.x & 31;
    const bool in = lane < RD_CANDS && R.valid[lane < RD_CANDS ? lane : 0];
    double j = 0.0;
    if (in) j = __dadd_rn(__ll2double_rn(R.ssd[lane]), __dmul_rn(P.lam2, __dmul_rn((double)R.bits[lane], 0.00390625)));
    const unsigned valid = __ballot_sync(FULL, in);
    int best = -1;
    double bj = 0.0;
#pragma unroll
    for (int k = 0; k < RD_CANDS; k++) {
        const double jk = __shfl_sync(FULL, j, k);
        if (((valid >> k) & 1u) && (best < 0 || jk < bj)) best = k, bj = jk;
    }
    return best;
}

// The MbState of a coded candidate: the inter ones' from inter_tail (S.a.out), the intra ones' without motion.
template <class T, int W>
__device__ __forceinline__ void rd_state(RdSmem<T, W>& R, const DecideSmem<T>& S, int k, bool inter) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    uint32_t* d = reinterpret_cast<uint32_t*>(&R.state[k]);
    if (inter) {
        if (lane < 18) d[lane] = reinterpret_cast<const uint32_t*>(&S.a.out)[lane];
    } else {
        // inter 0, refs -1, pad 0, no motion (bytes 0-7, then the vectors)
        if (lane < 18) d[lane] = lane == 0 ? 0xFFFFFF00u : (lane == 1 ? 0x000000FFu : 0u);
    }
    __syncwarp();
}

// ---- one chain on five warps ----------------------------------------------------------------------------
// Few chains leave the chip idle, and a chain's time is the picture's, so each gets five warps:
//   - the P_Skip tests of five macroblocks at once (warp i the i-th, on the assumption that those before it in the group are
//     P_Skip: their states are then their skip vectors, a chain of a few instructions each). The leading ones that pass are
//     P_Skip, and the test of the first that does not pass is good too. Tested one by one, the P_Skip macroblocks (most of a P
//     picture's) took 12 us each;
//   - the candidates of a macroblock that does not pass, side by side: warp 0 best_inter and its partitioning with the 4x4
//     transform, into the picture; warp 4 P_Skip and then the partitioning with the 8x8 transform (best_inter's decision
//     handed over through named barrier 1); warp 1 Intra4x4, warp 2 Intra16x16 with the intra chroma, and warp 3 Intra8x8
//     (the chroma handed over through named barrier 2), warps 1 to 4 each into their own scratch planes (their edges read
//     from the picture, which warp 0 writes only inside the macroblock). Each warp prices what it coded;
//   - the commit of the kept one (code, reconstruction, contexts, state) by a warp each.
// The warps meet at CTA barriers (after the tests; after the P_Skip macroblocks' commits; and, when there are candidates, after
// them and after the commit), every warp at every one. An IDR and three P pictures at 1080p, 8 bands: 248 ms with three warps a
// chain (P_Skip tested one macroblock at a time, each candidate's bins walked by nine lanes), 118 ms in this form.
constexpr int RDW_WARPS = 5;

// skip_mv (enc/frame.rs:597-603) from a macroblock's table of neighbours, with its left neighbour's block a.
__device__ __forceinline__ int2 skip_mv_from(const Blk* ext, const Blk& a) {
    const Blk b = ext[1];
    Blk c = ext[5];
    if (!c.w) c = ext[0];
    if (!a.w || !b.w || (a.z == 0 && a.x == 0 && a.y == 0) || (b.z == 0 && b.x == 0 && b.y == 0)) return make_int2(0, 0);
    const int ra = a.z == 0, rb = b.z == 0, rc = c.z == 0;
    if (ra + rb + rc == 1) return ra ? make_int2(a.x, a.y) : (rb ? make_int2(b.x, b.y) : make_int2(c.x, c.y));
    return make_int2(median3_d(a.x, b.x, c.x), median3_d(a.y, b.y, c.y));
}

// The next macroblocks of the chain from (mbx0, mby) on: returns how many were decided (1 to RDW_WARPS).
template <class T>
__device__ int rd_group(const RdParams& P, const DecideParams* dw, RdSmem<T, RDW_WARPS>& R, const unsigned* i4tab, int mbx0, int mby) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const DecideParams& D = P.D;
    const AnalyseParams& A = D.C.A;
    const CodeParams& C = D.C;
    DecideSmem<T>& S = R.s[w];
    const bool ta = mby > A.band_start[mby];
    const cab::Slice sl = {D.intra ? 0 : 1, P.t8, D.intra ? 0 : A.nact};
    ironav_mbcode* cand = R.cand;
    const int mb0 = mby * A.mb_w + mbx0, n = D.intra ? 0 : min(RDW_WARPS, A.mb_w - mbx0);
    const bool la0 = mbx0 > 0, left_skip = la0 && R.done.skip;
    auto copy_nb = [&](cab::Nb* d, const cab::Nb* s) {  // zeros when s is nullptr
        if (lane < cab::NB_WORDS) reinterpret_cast<uint32_t*>(d)[lane] = s ? reinterpret_cast<const uint32_t*>(s)[lane] : 0u;
    };
    auto begin = [&](int x) {
        if (lane == 0) {
            S.a.mb = mby * A.mb_w + x;
            S.a.mbx = x;
            S.a.mby = mby;
        }
        __syncwarp();
        stage_source(A, S.a);
    };
    if (w < n) {
        begin(mbx0 + w);
        load_neighbours(A, S.a, A.states_out);
        copy_nb(&R.top[w], ta ? reinterpret_cast<const cab::Nb*>(P.nbs + (size_t)(mb0 + w - A.mb_w) * cab::NB_WORDS) : nullptr);
    } else if (n == 0 && w == 0) {
        copy_nb(&R.top[0], ta ? reinterpret_cast<const cab::Nb*>(P.nbs + (size_t)(mb0 - A.mb_w) * cab::NB_WORDS) : nullptr);
    }
    __syncthreads();  // every macroblock's table of neighbours
    if (w < n) {
        ironav_mbcode* out = &D.codes[mb0 + w];
        if (w > 0) {
            // the left neighbour is P_Skip by assumption, with the vector that the same assumption gives it (only the
            // tables' rows above are read from other warps, and only the left column is changed here)
            int2 sv = skip_mv_from(R.s[0].a.ext, R.s[0].a.ext[6]);
            for (int j = 1; j < w; j++) sv = skip_mv_from(R.s[j].a.ext, make_int4(sv.x, sv.y, 0, 1));
            if (lane < 4) S.a.ext[(lane + 1) * 6] = make_int4(sv.x, sv.y, 0, 1);
        }
        code_init(out);
        int2 sv = make_int2(0, 0);
        const bool skip = skip_tests_d<T>(D, S, mb0 + w, mbx0 + w, mby, out, &sv);
        if (lane == 0) {
            R.skip[w] = skip;
            R.sv[w] = sv;
        }
    }
    if (n > 0) __syncthreads();  // the verdicts
    int m = 0;
    while (m < n && R.skip[m]) m++;
    // the leading P_Skip macroblocks, and the neighbours of the one after them
    if (w < m) {
        const ironav_mbcode* out = &D.codes[mb0 + w];
        if (lane < 18) reinterpret_cast<uint32_t*>(&A.states_out[mb0 + w])[lane] = reinterpret_cast<const uint32_t*>(&S.a.out)[lane];
        cab::Nb* nb = w == m - 1 ? &R.done : &R.nbs[w];
        cab::nb_of_warp(out, nb);
        if (lane < cab::NB_WORDS) P.nbs[(size_t)(mb0 + w) * cab::NB_WORDS + lane] = reinterpret_cast<const uint32_t*>(nb)[lane];
        if (w == m - 1) copy_nb(&R.nb[0], nb);
    }
    if (w == 0 && lane == 0) {
        // their one bin each still moves the contexts (mb_skip_flag; the left one of all but the first is P_Skip)
        for (int j = 0; j < m; j++) {
            const int ctx = 11 + (j == 0 && la0 && !left_skip) + (R.top[j].avail && !R.top[j].skip);
            R.live[ctx] = (uint8_t)R.step[R.live[ctx] * 2 + 1];
        }
    }
    if (m < n || n == 0) {
        if (w == RDW_WARPS - 1) {
            copy_nb(&R.nb[1], &R.top[m]);
            if (lane < RD_CANDS) R.valid[lane] = 0;
        }
        if (w == 0 && m == 0) copy_nb(&R.nb[0], la0 ? &R.done : nullptr);
    }
    __syncthreads();
    if (n > 0 && m == n) return n;
    // the candidates of macroblock mb
    const int mb = mb0 + m, mbx = mbx0 + m;
    const bool la = mbx > 0, tra = ta && mbx + 1 < A.mb_w;
    begin(mbx);
    __syncwarp();
    if (w == 0) {
        if (!D.intra) {
            // best_inter, enc/frame.rs:839-849
            load_neighbours(A, S.a, A.states_out);
            int part = 0, cost = BIG, bestr = 0;
            uint32_t sub = 0;
            for (int r = 0; r < A.nact; r++) {
                const int4 bi = best_inter_or_learned(A, S.a, r);
                if (r == 0 || bi.x < cost) {
                    part = bi.y;
                    cost = bi.x;
                    bestr = r;
                    sub = (uint32_t)bi.z;
                    if (lane < 16) {
                        S.a.win_mvs[lane][0] = S.a.best_mvs[lane][0];
                        S.a.win_mvs[lane][1] = S.a.best_mvs[lane][1];
                    }
                    __syncwarp();
                }
            }
            ironav_interdec& Dd = *reinterpret_cast<ironav_interdec*>(S.c.dec);
            if (lane == 0) {
                Dd.mode = 2;
                Dd.part = (uint8_t)part;
                Dd.t8 = 0;
                for (int k = 0; k < 4; k++) {
                    Dd.sub[k] = (uint8_t)((sub >> (8 * k)) & 0xff);
                    Dd.refs[k] = (uint8_t)bestr;
                }
                R.try_t8 = P.t8 && sub == 0;
            }
            if (lane < 16) {
                Dd.mvs[lane][0] = S.a.win_mvs[lane][0];
                Dd.mvs[lane][1] = S.a.win_mvs[lane][1];
            }
            __syncwarp();
            if (P.t8) {
                for (int i = lane; i < 40; i += 32) R.idec[i] = S.c.dec[i];
                __threadfence_block();
                __syncwarp();
                asm volatile("bar.arrive 1, 64;" ::: "memory");
            }
            ironav_mbcode* o = &cand[1];
            code_init(o);
            const uint32_t cbp = code_inter_mb<T>(C, S.c, mb, &o->res);
            inter_tail(D, S, Dd, o);
            rd_state(R, S, 1, true);
            rd_take(C, R, S, 1, mbx, mby);
            // with nothing coded and the skip vector, it would be P_Skip at a higher price
            const int2 sv = R.sv[m];
            if (lane == 0 && cbp == 0 && part == 0 && Dd.mvs[0][0] == sv.x && Dd.mvs[0][1] == sv.y && bestr == 0) R.valid[1] = 0;
            __syncwarp();
            if (R.valid[1]) rd_price(R, sl, S.nbm, 1, w);
        }
    } else if (w == 1) {
        // Intra4x4 into warp 1's luma plane, with Intra16x16's chroma
        const DecideParams& Dw = dw[0];
        load_intra_neighbours(D, S, mb, mbx, mby, ta, la, tra);
        ironav_mbcode* o = &cand[4];
        code_init(o);
        code_i4_trial(Dw, S, i4tab, ta, la, tra);
        T* RY = reinterpret_cast<T*>(Dw.C.rec[0]);
        for (int i = lane; i < 256; i += 32) RY[(size_t)(mby * 16 + (i >> 4)) * Dw.C.ys + mbx * 16 + (i & 15)] = (T)S.i4rec[i];
        if (lane < 16) {
            uint32_t* lw = reinterpret_cast<uint32_t*>(o->res.luma[lane]);
            const uint32_t* src = reinterpret_cast<const uint32_t*>(S.i4lv[lane]);
#pragma unroll
            for (int k = 0; k < 8; k++) lw[k] = src[k];
            o->res.nnz[lane] = S.i4nnz[lane];
            o->modes[lane] = S.i4modes[lane];
        }
        const unsigned bal = __ballot_sync(FULL, lane < 16 && S.i4nnz[lane] > 0);
        uint32_t cbp = 0;
#pragma unroll
        for (int i8 = 0; i8 < 4; i8++)
            if (bal & (0x33u << ((i8 >> 1) * 8 + (i8 & 1) * 2))) cbp |= 1u << i8;
        if (lane == 0) {
            o->kind = KIND_I4;
            o->res.cbp = (uint8_t)cbp;
        }
        rd_state(R, S, 4, false);
        rd_take(Dw.C, R, S, 4, mbx, mby, false);
        asm volatile("bar.sync 2, 96;" ::: "memory");
        rd_take_chroma(R, 4);
        rd_price(R, sl, S.nbm, 4, w);
    } else if (w == 2) {
        // Intra16x16 in best_i16's mode with the intra chroma, into warp 2's planes
        const DecideParams& Dw = dw[1];
        load_intra_neighbours(D, S, mb, mbx, mby, ta, la, tra);
        const int2 i16 = best_i16_d(Dw, S, ta, la);
        ironav_mbcode* o = &cand[3];
        code_init(o);
        uint32_t cbp = code_i16_d(Dw, S, mbx, mby, i16.x, ta, la, o);
        const uint32_t ccbp = code_intra_chroma_d(Dw, S, mbx, mby, ta, la, o);
        cbp |= ccbp;
        if (lane == 0) {
            o->kind = KIND_I16;
            o->i16_mode = (uint8_t)i16.x;
            o->res.cbp = (uint8_t)cbp;
            R.ccbp = ccbp;
        }
        rd_state(R, S, 3, false);
        rd_take(Dw.C, R, S, 3, mbx, mby);
        __threadfence_block();
        __syncwarp();
        asm volatile("bar.arrive 2, 96;" ::: "memory");
        rd_price(R, sl, S.nbm, 3, w);
    } else if (w == 3) {
        // Intra8x8 into warp 3's luma plane (its edges from the picture), with Intra16x16's chroma
        const DecideParams& Dw = dw[2];
        if (P.t8) {
            load_intra_neighbours(D, S, mb, mbx, mby, ta, la, tra);
            ironav_mbcode* o = &cand[5];
            code_init(o);
            const uint32_t cbp = code_i8_d(D, S, R, mbx, mby, ta, la, tra, o, reinterpret_cast<T*>(Dw.C.rec[0]), Dw.C.ys);
            if (lane == 0) o->res.cbp = (uint8_t)cbp;
            rd_state(R, S, 5, false);
            rd_take(Dw.C, R, S, 5, mbx, mby, false);
        }
        asm volatile("bar.sync 2, 96;" ::: "memory");
        if (P.t8) {
            rd_take_chroma(R, 5);
            rd_price(R, sl, S.nbm, 5, w);
        }
    } else if (!D.intra) {
        // P_Skip: the skip vector's prediction is the reconstruction (put_inter_pred, 1391-1394), into warp 4's
        // planes; a P_Skip code carries no differences, its state the vector over the macroblock
        const DecideParams& Dw = dw[3];
        const int2 sv = R.sv[m];
        ironav_mbcode* o = &cand[0];
        code_init(o);
        ironav_interdec& Dd = *reinterpret_cast<ironav_interdec*>(S.c.dec);
        if (lane == 0) {
            Dd.mode = 1;
            Dd.part = 0;
            Dd.t8 = 0;
            for (int k = 0; k < 4; k++) Dd.sub[k] = Dd.refs[k] = 0;
            o->kind = KIND_INTER;
            o->skip = 1;
        }
        if (lane < 16) {
            Dd.mvs[lane][0] = (int16_t)sv.x;
            Dd.mvs[lane][1] = (int16_t)sv.y;
            o->mvs[lane][0] = (int16_t)sv.x;
            o->mvs[lane][1] = (int16_t)sv.y;
        }
        __syncwarp();
        code_inter_mb<T>(Dw.C, S.c, mb, &o->res);
        uint32_t* d = reinterpret_cast<uint32_t*>(&R.state[0]);
        if (lane < 18) d[lane] = lane == 0 ? 1u : (lane == 1 ? 0u : ((uint32_t)(uint16_t)sv.x | (uint32_t)(uint16_t)sv.y << 16));
        __syncwarp();
        rd_take(Dw.C, R, S, 0, mbx, mby);
        rd_price(R, sl, S.nbm, 0, w);
        if (P.t8) {
            // best_inter's partitioning with the 8x8 transform (when no 8x8 block is split; without luma levels it
            // would be the 4x4 candidate again), once warp 0 has handed its decision over
            load_neighbours(A, S.a, A.states_out);
            asm volatile("bar.sync 1, 64;" ::: "memory");
            if (R.try_t8) {
                for (int i = lane; i < 40; i += 32) S.c.dec[i] = R.idec[i];
                __syncwarp();
                if (lane == 0) Dd.t8 = 1;
                __syncwarp();
                o = &cand[2];
                code_init(o);
                code_inter_mb<T>(Dw.C, S.c, mb, &o->res);
                inter_tail(D, S, Dd, o);
                rd_state(R, S, 2, true);
                rd_take(Dw.C, R, S, 2, mbx, mby);
                if (lane == 0 && !o->res.t8x8) R.valid[2] = 0;
                __syncwarp();
                if (R.valid[2]) rd_price(R, sl, S.nbm, 2, w);
            }
        }
    }
    __syncthreads();
    // the least cost in order, and its commit
    const int b = rd_best(P, R);
    if (w == 0) {
        if (lane < 18) reinterpret_cast<uint32_t*>(&A.states_out[mb])[lane] = reinterpret_cast<const uint32_t*>(&R.state[b])[lane];
        cab::nb_of_warp(&cand[b], &R.done);
        if (lane < cab::NB_WORDS) P.nbs[(size_t)mb * cab::NB_WORDS + lane] = reinterpret_cast<const uint32_t*>(&R.done)[lane];
    } else if (w == 1) {
        const uint32_t* s32 = reinterpret_cast<const uint32_t*>(&cand[b]);
        uint32_t* d32 = reinterpret_cast<uint32_t*>(&D.codes[mb]);
        for (int i = lane; i < (int)(sizeof(ironav_mbcode) / 4); i += 32) d32[i] = s32[i];
    } else if (w == 2) {
        const int row = lane >> 1, half = lane & 1;
        const uint32_t* rec = reinterpret_cast<const uint32_t*>(R.crec[b]) + lane * 2 * (int)sizeof(T);
        uint32_t* d = reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(C.rec[0]) + (size_t)(mby * 16 + row) * C.ys + mbx * 16 + half * 8);
#pragma unroll
        for (int i = 0; i < 2 * (int)sizeof(T); i++) d[i] = rec[i];
    } else if (w == 3) {
        const int cc = lane >> 4, j = (lane & 15) * 4;
        const uint32_t* rec = reinterpret_cast<const uint32_t*>(R.crec[b]) + (64 + lane) * (int)sizeof(T);
        uint32_t* d = reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(C.rec[1 + cc]) + (size_t)(mby * 8 + (j >> 3)) * C.cs + mbx * 8 + (j & 7));
#pragma unroll
        for (int i = 0; i < (int)sizeof(T); i++) d[i] = rec[i];
    } else {
        const uint4* c16 = reinterpret_cast<const uint4*>(R.cst[b]);
        uint4* l16 = reinterpret_cast<uint4*>(R.live);
        l16[lane] = c16[lane];
        l16[lane + 32] = c16[lane + 32];
    }
    __syncthreads();
    return m + 1;
}

// A chain's set-up and walk for the parameters P (in parameter space or shared memory): warps 1 to 4's parameter
// copies writing into their scratch planes, the CTA's tables and contexts, then slice band `band` in raster order.
template <class T>
__device__ void rdw_chain(const RdParams& P, DecideParams* dw, RdSmem<T, RDW_WARPS>& R, unsigned* i4tab, int band) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w > 0) {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(&P.D);
        uint32_t* dst = reinterpret_cast<uint32_t*>(&dw[w - 1]);
        for (int k = lane; k < (int)(sizeof(DecideParams) / 4); k += 32) dst[k] = src[k];
        __syncwarp();
        if (lane == 0) {
            for (int k = 0; k < 3; k++) dw[w - 1].C.rec[k] = P.scr[3 * (w - 1) + k];
            dw[w - 1].C.ys = P.scr_ys;
            dw[w - 1].C.cs = P.scr_cs;
        }
    }
    fill_i4tab(i4tab);  // its __syncthreads also publishes dw
    const AnalyseParams& A = P.D.C.A;
    for (int i = threadIdx.x; i < cab::STEP_ENTRIES; i += blockDim.x) R.step[i] = P.step[i];
    for (int i = threadIdx.x; i < 9 * 64; i += blockDim.x) R.i8tab[i] = i8_entry(i >> 6, i & 7, (i >> 3) & 7);
    cab::init_states(R.live, P.D.intra != 0, 0, P.D.C.qp, threadIdx.x, blockDim.x);
    __syncthreads();
    for (int mby = P.band_rows[band]; mby < P.band_rows[band + 1]; mby++)
        for (int mbx = 0; mbx < A.mb_w;) mbx += rd_group<T>(P, dw, R, i4tab, mbx, mby);
}

// Decide mode under CABAC for one stream: CTA i walks slice band i.
template <class T>
__global__ void __launch_bounds__(RDW_WARPS * 32, 1) decide_rdw_kernel(const __grid_constant__ RdParams P) {
    extern __shared__ __align__(16) unsigned char rdw_smem[];
    __shared__ DecideParams dw[RDW_WARPS - 1];
    __shared__ unsigned i4tab[9 * 17];
    if ((int)blockIdx.x >= P.nbands) return;
    rdw_chain<T>(P, dw, *reinterpret_cast<RdSmem<T, RDW_WARPS>*>(rdw_smem), i4tab, blockIdx.x);
}

// The same for many streams' chains: CTA i walks chains[i] = stream << 16 | band with the stream's
// parameters from table[stream] (copied into shared memory). PER_SM: the CTAs an SM takes, one with 255 registers a thread or two
// with 168.
template <class T, int PER_SM>
__global__ void __launch_bounds__(RDW_WARPS * 32, PER_SM) decide_rdw_batch_kernel(const RdParams* __restrict__ table,
                                                                          const uint32_t* __restrict__ chains, int nchains) {
    extern __shared__ __align__(16) unsigned char rdw_smem[];
    __shared__ RdParams prm;
    __shared__ DecideParams dw[RDW_WARPS - 1];
    __shared__ unsigned i4tab[9 * 17];
    if ((int)blockIdx.x >= nchains) return;
    const uint32_t e = chains[blockIdx.x];
    const uint32_t* src = reinterpret_cast<const uint32_t*>(&table[e >> 16]);
    for (int k = threadIdx.x; k < (int)(sizeof(RdParams) / 4); k += blockDim.x) reinterpret_cast<uint32_t*>(&prm)[k] = src[k];
    __syncthreads();
    rdw_chain<T>(prm, dw, *reinterpret_cast<RdSmem<T, RDW_WARPS>*>(rdw_smem), i4tab, (int)(e & 0xFFFFu));
}

template <class T>
constexpr size_t rdw_smem_bytes() { return sizeof(RdSmem<T, RDW_WARPS>); }

// ---- the CABAC slice writer ---------------------------------------------------------------------------

// What the writer reads of a macroblock as a neighbour: its Nb, and the Intra NxN modes of its right column
// and bottom row (2 for a macroblock that is neither Intra4x4 nor Intra8x8), as pred_mode reads them.
struct WrNb {
    cab::Nb nb;
    int8_t rmodes[4], bmodes[4];
};
constexpr int WRNB_WORDS = (int)(sizeof(WrNb) / 4);
static_assert(sizeof(WrNb) % 4 == 0, "WrNb in whole words");

struct CabacWriteParams {
    const ironav_mbcode* codes;
    WrNb* nbs;              // per macroblock, filled by cabac_nb_kernel
    const int* band_rows;
    const uint32_t* step;
    uint32_t* out;          // slice i's data at out + i * region_words
    uint32_t region_words;
    uint32_t* slice_bytes;  // per slice: its data's bytes; [nbands]: set when a slice outgrew its region
    int mb_w, nmb, nbands, intra, t8, nref, qp;
    unsigned spins;         // polls of a shared-memory word before a warp gives up
};

// Every macroblock's WrNb, a warp a macroblock (grid-stride): the neighbours' side of the writer's walk,
// worked out for the whole picture at once.
static __global__ void __launch_bounds__(128) cabac_nb_kernel(const __grid_constant__ CabacWriteParams P) {
    const int lane = threadIdx.x & 31;
    const int warps = (int)(gridDim.x * blockDim.x) >> 5;
    for (int mb = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); mb < P.nmb; mb += warps) {
        const ironav_mbcode* k = &P.codes[mb];
        cab::nb_of_warp(k, &P.nbs[mb].nb);
        if (lane < 8) {
            const bool n = cab::nxn(k->kind);
            if (lane < 4) P.nbs[mb].rmodes[lane] = (int8_t)(n ? k->modes[lane * 4 + 3] : 2);
            else P.nbs[mb].bmodes[lane - 4] = (int8_t)(n ? k->modes[12 + lane - 4] : 2);
        }
        __syncwarp();
    }
}

// A slice band's data (FrameCoder::encode with write_mb_cabac, enc/frame.rs:461-486): each macroblock's bins
// (mb_bins) then end_of_slice_flag, arithmetic coded from the slice's contexts; the data starts on the byte
// that follows the header's cabac_alignment_one_bit (written on the host). CTA i walks slice band i, as a pipeline of warps:
//   - warps 2 and up list the macroblocks' bins, each every WR_LISTERS-th macroblock, in as many turns as its list needs;
//   - warp 1 takes the lists in order and looks up each bin's probability state (32 bins a turn; the bins of a context are a
//     chain, the contexts side by side), leaving what the coder needs of it in a ring;
//   - lane 0 of warp 0 runs the coder's own chain, the range, over the ring.
// One lane doing all three took 62 ms for an IDR and three P pictures at 1080p, the pipeline 27 ms with a branch on each bin's kind in
// the coder, now 14 (7 with the coder's arithmetic left out). Every wait is on shared memory and
// bounded; a warp that gives up stops the others, and the picture is reported like one that outgrew its region.
constexpr int WR_LISTERS = 6;
constexpr int WR_THREADS = (2 + WR_LISTERS) * 32;
constexpr int WR_CAP = 3328;   // bins a list holds: at least one piece's most (16 levels of up to 48 bins)
static_assert(16 * 48 <= WR_CAP, "one piece fits the list");
constexpr int WR_RING = 512;   // bins between the states and the coder

struct WrSmem {
    cab::CodeBin ring[WR_RING];
    cab::CodeBin entry[64];  // per probability state
    ironav_mbcode code[WR_LISTERS];
    WrNb nb[WR_LISTERS][2];
    uint32_t step[cab::STEP_ENTRIES];
    uint8_t st[1024];
    uint16_t list[WR_LISTERS][WR_CAP];
    uint8_t pre[32];                  // a turn's states before its bins
    unsigned count[WR_LISTERS];       // a list's bins, | WR_LAST when they are its macroblock's last
    unsigned listed[WR_LISTERS], taken[WR_LISTERS];  // turns of each lister
    unsigned head, tail;              // bins put into and taken from the ring
    unsigned stop;
};
constexpr unsigned WR_LAST = 1u << 31;

// Waits until the shared word is at least `need` (as a difference, the counts wrap); false when it gave up, after `spins` polls, or
// another warp did.
__device__ __forceinline__ bool wr_wait(WrSmem& S, unsigned spins, const unsigned* w, unsigned need) {
    for (unsigned i = 0;; i++) {
        if ((int)(ld_acquire_cta(w) - need) >= 0) return true;
        if ((i & 15) == 15) {
            if (ld_acquire_cta(&S.stop)) return false;
            if (i >= spins) {
                st_release_cta(&S.stop, 1u);
                return false;
            }
            __nanosleep(20);
        }
    }
}

static __global__ void __launch_bounds__(WR_THREADS) cabac_write_kernel(const __grid_constant__ CabacWriteParams P) {
    extern __shared__ __align__(16) unsigned char wr_smem[];
    WrSmem& S = *reinterpret_cast<WrSmem*>(wr_smem);
    const int chain = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (chain >= P.nbands) return;
    for (int i = threadIdx.x; i < cab::STEP_ENTRIES; i += WR_THREADS) S.step[i] = P.step[i];
    if (threadIdx.x < 64) S.entry[threadIdx.x] = cab::code_entry(threadIdx.x);
    if (threadIdx.x < WR_LISTERS) S.listed[threadIdx.x] = S.taken[threadIdx.x] = 0;
    if (threadIdx.x == 0) S.head = S.tail = S.stop = 0;
    cab::init_states(S.st, P.intra != 0, 0, P.qp, threadIdx.x, WR_THREADS);
    const cab::Slice sl = {P.intra ? 0 : 1, P.t8, P.intra ? 0 : P.nref};
    const int first = P.band_rows[chain] * P.mb_w, end = P.band_rows[chain + 1] * P.mb_w;
    __syncthreads();
    if (w == 0) {
        if (lane == 0) {
            cab::Coder k = {{P.out + (size_t)chain * P.region_words, P.region_words, 0, 0, 0, false, false}, 0ull, 510u, -1};
            unsigned at = 0, avail = 0;
            bool more = true;
            while (more) {
                if (at == avail) {
                    st_release_cta(&S.tail, at);
                    if (!wr_wait(S, P.spins, &S.head, at + 1)) break;
                    avail = ld_acquire_cta(&S.head);
                }
                if (avail - at >= 8u) {
                    // eight bins, read before the chain goes through them; the slice's last bin is the last of what there is
                    cab::CodeBin e[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) e[i] = S.ring[(at + i) % WR_RING];
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        k.code(e[i]);
                        k.code(e[i + 1]);
                        k.settle();
                    }
                    more = (e[7].ctl & cab::CODE_END) == 0;
                    at += 8;
                } else {
                    const cab::CodeBin e = S.ring[at % WR_RING];
                    k.code(e);
                    k.settle();
                    more = (e.ctl & cab::CODE_END) == 0;
                    at++;
                }
                if (at % (WR_RING / 4) < 8u) st_release_cta(&S.tail, at);  // room for the states' warp well before the ring runs dry
            }
            const uint32_t bytes = k.finish();
            P.slice_bytes[chain] = bytes;
            if (more || k.out.over) atomicOr(&P.slice_bytes[P.nbands], 1u);
        }
    } else if (w == 1) {
        unsigned head = 0, turns[WR_LISTERS] = {};
        for (int mb = first; mb < end; mb++) {
            const int l = (mb - first) % WR_LISTERS;
            unsigned n;
            do {
                unsigned turn = 0;
#pragma unroll
                for (int q = 0; q < WR_LISTERS; q++)
                    if (q == l) turn = ++turns[q];
                if (!__all_sync(FULL, wr_wait(S, P.spins, &S.listed[l], turn))) return;
                n = S.count[l];
                const int bins = (int)(n & ~WR_LAST);
                for (int i0 = 0; i0 < bins; i0 += 32) {
                    const bool in = i0 + lane < bins;
                    const uint32_t e = in ? S.list[l][i0 + lane] : cab::BIN_BYPASS;
                    const bool dec = (e & (cab::BIN_BYPASS | cab::BIN_TERMINATE)) == 0;
                    const int ctx = dec ? (int)(e & 1023u) : 1024 + lane;
                    uint32_t m = __match_any_sync(FULL, ctx);
                    const uint32_t ones = __ballot_sync(FULL, (e >> 10) & 1u);
                    if (dec && (m & ((1u << lane) - 1u)) == 0) {
                        uint32_t s = S.st[ctx];
                        do {
                            const int j = __ffs(m) - 1;
                            S.pre[j] = (uint8_t)s;
                            s = S.step[s * 2 + ((ones >> j) & 1u)] & 0xffu;
                            m &= m - 1;
                        } while (m);
                        S.st[ctx] = (uint8_t)s;
                    }
                    const int k = min(bins - i0, 32);
                    if (!__all_sync(FULL, wr_wait(S, P.spins, &S.tail, head + (unsigned)k - (unsigned)WR_RING))) return;
                    __syncwarp();
                    if (in) {
                        const uint32_t bin = (e >> 10) & 1u;
                        cab::CodeBin c = (e & cab::BIN_TERMINATE) ? cab::code_terminate(bin) : cab::code_bypass(bin);
                        if (dec) {
                            const uint32_t s = S.pre[lane];
                            c = S.entry[s >> 1];
                            c.ctl = (s & 1u) != bin ? cab::CODE_LOW | cab::CODE_ADD : 0u;
                        }
                        S.ring[(head + lane) % WR_RING] = c;
                    }
                    __syncwarp();
                    head += (unsigned)k;
                    if (lane == 0) st_release_cta(&S.head, head);
                }
                __syncwarp();
                if (lane == 0) st_release_cta(&S.taken[l], turn);
            } while (!(n & WR_LAST));
        }
    } else {
        const int l = w - 2;
        unsigned turn = 0;
        constexpr int W = (int)(sizeof(ironav_mbcode) / 4);
        ironav_mbcode* const code = &S.code[l];
        for (int mb = first + l; mb < end; mb += WR_LISTERS) {
            const int mbx = mb % P.mb_w;
            const bool la = mbx > 0, ta = mb - P.mb_w >= first;
            const uint32_t* g = reinterpret_cast<const uint32_t*>(&P.codes[mb]);
            for (int i = lane; i < W; i += 32) reinterpret_cast<uint32_t*>(code)[i] = g[i];
            uint32_t* d = reinterpret_cast<uint32_t*>(S.nb[l]);
            const uint32_t* gl = reinterpret_cast<const uint32_t*>(&P.nbs[la ? mb - 1 : mb]);
            const uint32_t* gt = reinterpret_cast<const uint32_t*>(&P.nbs[ta ? mb - P.mb_w : mb]);
            for (int i = lane; i < 2 * WRNB_WORDS; i += 32) d[i] = i < WRNB_WORDS ? (la ? gl[i] : 0u) : (ta ? gt[i - WRNB_WORDS] : 0u);
            __syncwarp();
            const WrNb &L = S.nb[l][0], &T = S.nb[l][1];
            int nbm[8];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                nbm[q] = la ? L.rmodes[q] : -1;
                nbm[4 + q] = ta ? T.bmodes[q] : -1;
            }
            // the pieces' bins, end_of_slice_flag after the last block's
            cab::BinCount h;
            cab::lane_head(h, sl, code, L.nb, T.nb, nbm);
            cab::ResPiece r;
            uint32_t bits;
            int nh;
            const int nr = cab::res_pieces<true>(r, code, L.nb, T.nb, &bits), oh = cab::warp_scan(h.n, &nh), total = nh + nr + 1;
            for (int base = 0; base < total;) {
                if (!__all_sync(FULL, wr_wait(S, P.spins, &S.taken[l], turn))) return;
                auto fits = [&](int at, int n) { return n > 0 && at >= base && at + n <= base + WR_CAP; };
                const bool fh = fits(oh, h.n), fm = fits(nh + r.os, r.ns), fl = fits(nh + r.ol, r.nl), ft = lane == 31 && fits(total - 1, 1);
                if (fh) {
                    cab::BinList c = {&S.list[l][oh - base]};
                    cab::lane_head(c, sl, code, L.nb, T.nb, nbm);
                }
                if (fm) {
                    cab::BinList c = {&S.list[l][nh + r.os - base]};
                    cab::list_map(c, r);
                }
                if (fl) {
                    cab::BinList c = {&S.list[l][nh + r.ol - base]};
                    cab::list_levels(c, r);
                }
                if (ft) {
                    cab::BinList c = {&S.list[l][total - 1 - base]};
                    c.terminate(mb + 1 == end);
                }
                const int to = __reduce_max_sync(FULL, max(max(fh ? oh + h.n : 0, fm ? nh + r.os + r.ns : 0), max(fl ? nh + r.ol + r.nl : 0, ft ? total : 0)));
                __syncwarp();
                turn++;
                if (lane == 0) {
                    S.count[l] = (unsigned)(to - base) | (to == total ? WR_LAST : 0u);
                    st_release_cta(&S.listed[l], turn);
                }
                base = to;
            }
        }
    }
}

}  // namespace ironav
