// cabac.cuh — CABAC on the device: the contexts of a slice, one macroblock's bins (mb_bins,
// enc/frame.rs:2028-2279, with write_block, enc/cabac.rs:194-250, and mvd_bins, enc/frame.rs:2393-2414), listed by the
// lanes of a warp, their price (CabacCost, enc/cabac.rs:150-192), and the arithmetic coder
// (CabacWriter, enc/cabac.rs:42-147).
//
// The walk reads the macroblock's code and what the contexts need of its left and top neighbours in the
// slice (Nb, the CABAC fields of MbState, enc/frame.rs:245-272). Only I and P slices are coded here.
#pragma once
#include <stdint.h>

#include "../../include/ironav_inter.h"
#include "cabac_tables.cuh"

namespace ironav {

namespace cab {

constexpr int KIND_I4 = 1, KIND_I8 = 2, KIND_I16 = 3, KIND_INTER = 5;  // Kind, h264/mb.rs:21-30

// The contexts' step table: for state s = pStateIdx * 2 + valMPS and bin b, entry [s * 2 + b] = the next
// state (next_state, enc/cabac.rs:32-40) | the bin's cost in 1/256 bits << 8 (entropy(), enc/cabac.rs:162-173,
// computed on the host with the reference's f64 formula and copied to the kernel's shared memory).
constexpr int STEP_ENTRIES = 256;

// The contexts of a slice (CabacWriter::new, enc/cabac.rs:54-64; 9.3.1.1): lanes share the 1024 entries.
__device__ __forceinline__ void init_states(uint8_t* st, bool intra, int idc, int slice_qp, int lane, int nlanes) {
    const int qp = min(max(slice_qp, 0), 51);
    for (int i = lane; i < 1024; i += nlanes) {
        const int m = intra ? CABAC_INIT_I[i][0] : CABAC_INIT_PB[idc][i][0];
        const int n = intra ? CABAC_INIT_I[i][1] : CABAC_INIT_PB[idc][i][1];
        const int pre = min(max(((m * qp) >> 4) + n, 1), 126);
        st[i] = (uint8_t)(pre <= 63 ? (63 - pre) << 1 : ((pre - 64) << 1) | 1);
    }
}

// The arithmetic coder's output: 32-bit pieces of the code value, MSB first, into the words of a region in global memory,
// stored so that the bytes read in order. A piece may carry into the ones before it, so the newest is held back, with a count of
// the 0xFFFFFFFF pieces after it that a carry would run through. A write beyond the region sets `over` and is dropped.
struct WordOut {
    uint32_t* words;
    uint32_t cap;  // words
    uint32_t nw;
    uint32_t held, ones;
    bool any, over;
    __device__ __forceinline__ void store(uint32_t v) {
        if (nw < cap) words[nw] = __byte_perm(v, 0, 0x0123);
        else over = true;
        nw++;
    }
    __device__ __forceinline__ void flush(uint32_t carry) {
        if (any) store(held + carry);
        for (; ones > 0; ones--) store(carry ? 0u : 0xFFFFFFFFu);
        any = false;
    }
    __device__ __forceinline__ void put(uint64_t v) {  // 32 bits and their carry
        if (v == 0xFFFFFFFFull && any) {
            ones++;
            return;
        }
        flush((uint32_t)(v >> 32));
        held = (uint32_t)v;
        any = true;
    }
    // the last k < 32 bits (and their carry), padded with zeros to a byte; returns the byte count
    __device__ __forceinline__ uint32_t finish(uint64_t v, int k) {
        flush((uint32_t)(v >> k));
        const uint32_t bytes = nw * 4 + (uint32_t)((k + 7) >> 3);
        if (k > 0) store((uint32_t)(v << (32 - k)));
        return bytes;
    }
};

// A bin as the coder takes it, every kind in one form: the range it takes off for each quarter of the range (a byte each: the LPS
// range of its state, 2 of a terminate bin, 0 of a bypass bin); what the range becomes when it is the low part (its low byte; the
// ninth bit is set) and by how many bits that shifts the code; and ctl.
enum CodeCtl : uint32_t {
    CODE_PRE = 1u,          // a bypass bin: the code shifts by one before the addition
    CODE_END = 2u,          // the slice's last bin
    CODE_LOW = 1u << 30,    // an LPS, or a terminate bin of 1: the range becomes the low part's
    CODE_ADD = 1u << 31     // the code goes up by the rest of the range
};
struct __align__(16) CodeBin {
    uint32_t lps, norm, shift, ctl;
};
static_assert(sizeof(CodeBin) == 16, "one 16-byte read");
// The entry of probability state p.
__device__ __forceinline__ CodeBin code_entry(int p) {
    CodeBin e = {0, 0, 0, 0};
    for (int q = 0; q < 4; q++) {
        const uint32_t r = LPS_RANGE[p][q], sh = (uint32_t)__clz((int)r) - 23u;
        e.lps |= r << (8 * q);
        e.norm |= ((r << sh) & 0xFFu) << (8 * q);
        e.shift |= sh << (8 * q);
    }
    return e;
}
__device__ __forceinline__ CodeBin code_bypass(uint32_t bin) { return {0u, 0u, 0u, CODE_PRE | (bin ? CODE_ADD : 0u)}; }
__device__ __forceinline__ CodeBin code_terminate(uint32_t bin) {
    return {0x02020202u, 0u, 0x07070707u, bin ? CODE_LOW | CODE_ADD | CODE_END : 0u};
}

// The arithmetic coder (9.3.4.2-9.3.4.5). Its serial chain is the range alone: a bin's probability state is looked up before it, and
// the code value is a plain sum, kept whole: `low` holds the 10 bits of the standard's codILow below the nb bits already shifted
// out of it, and a carry above them. nb begins at -1: the first bit of the code is not written (9.3.4.2). Every bin takes the same
// instructions, without a branch on its kind (the range's top bits pick the byte of its quarter: range >> 6 is 4 + the quarter, a
// byte permutation's selector): a branch a kind, on the writer's one coding lane, took some 240 cycles a bin.
struct Coder {
    WordOut out;
    uint64_t low;
    uint32_t range;
    int nb;
    // at most two bins (7 bits each) before settle(), from nb < 32: the code stays within 56 bits
    __device__ __forceinline__ void code(const CodeBin& e) {
        const uint32_t q = range >> 6, rest = range - __byte_perm(0u, e.lps, q), ms = rest < 256u, pre = e.ctl & CODE_PRE;
        const bool part = (e.ctl & CODE_LOW) != 0;
        const uint32_t sh = part ? __byte_perm(0u, e.shift, q) : ms;
        low = ((low << pre) + (rest & (uint32_t)((int)e.ctl >> 31))) << sh;
        nb += (int)(pre + sh);
        range = part ? 256u | __byte_perm(0u, e.norm, q) : rest << ms;
    }
    __device__ __forceinline__ void settle() {
        if (nb >= 32) {
            const int rest = nb - 22;  // 10 + nb - 32
            out.put(low >> rest);
            low &= (1ull << rest) - 1;
            nb -= 32;
        }
    }
    // after the last terminate bin: the flush's bit and two more, the last of them the rbsp_stop_one_bit
    __device__ __forceinline__ uint32_t finish() {
        uint64_t v = (low >> 7) | 1u;
        int k = nb + 3;
        if (k >= 32) {
            k -= 32;
            out.put(v >> k);
            v &= (1ull << k) - 1;
        }
        return out.finish(v, k);
    }
};

// What the contexts read of a neighbouring macroblock (finish_mb's MbState fields, enc/frame.rs:2281-2321).
struct Nb {
    uint8_t avail, skip, kind, inter, cbp, t8x8, chroma_mode, cbf_dc;
    int8_t r8[4];        // list 0 reference index per 8x8 block (-1: intra)
    uint8_t mvd[16][2];  // absolute vector differences per 4x4 block, capped at 64 (mvd_grid, enc/frame.rs:238-241)
    uint8_t nnz[16];
    uint8_t cnnz[2][4];
};

// The partition (rects order) that holds 4x4 block (bx, by) of a P macroblock.
__device__ __forceinline__ int part_index(int part, const uint8_t* sub, int bx, int by) {
    if (part == 0) return 0;
    if (part == 1) return by >> 1;
    if (part == 2) return bx >> 1;
    const int k = (by >> 1) * 2 + (bx >> 1);
    int n = 0;
    for (int q = 0; q < k; q++) n += sub[q] == 0 ? 1 : (sub[q] == 3 ? 4 : 2);
    const int s = sub[k];
    return n + (s == 0 ? 0 : s == 1 ? (by & 1) : s == 2 ? (bx & 1) : (by & 1) * 2 + (bx & 1));
}

// The origin of partition n (rects order) of a P macroblock; false beyond the last.
__device__ __forceinline__ bool part_origin(int part, const uint8_t* sub, int n, int* bx, int* by) {
    if (part < 3) {
        *bx = part == 2 ? 2 * n : 0;
        *by = part == 1 ? 2 * n : 0;
        return n < (part == 0 ? 1 : 2);
    }
    for (int k = 0; k < 4; k++) {
        const int s = sub[k], count = s == 0 ? 1 : (s == 3 ? 4 : 2);
        if (n < count) {
            *bx = (k & 1) * 2 + (s == 2 ? n : (s == 3 ? (n & 1) : 0));
            *by = (k >> 1) * 2 + (s == 1 ? n : (s == 3 ? (n >> 1) : 0));
            return true;
        }
        n -= count;
    }
    return false;
}

constexpr int NB_WORDS = (int)(sizeof(Nb) / 4);
static_assert(sizeof(Nb) % 4 == 0, "Nb in whole words");

// A neighbour's Nb from its code (in shared or global memory); every lane of the warp calls.
__device__ __forceinline__ void nb_of_warp(const ironav_mbcode* k, Nb* n) {
    const int lane = threadIdx.x & 31;
    const int kind = k->kind, skip = k->skip, cbp = k->res.cbp;
    const bool inter = kind == KIND_INTER;
    bool nz = false;
    if (lane < 16) nz = k->dc[lane] != 0;
    else if (lane < 24) nz = k->res.cdc[(lane - 16) >> 2][(lane - 16) & 3] != 0;
    const unsigned bal = __ballot_sync(0xffffffffu, nz);
    if (lane < 16) {
        n->nnz[lane] = k->res.nnz[lane];
        uint8_t ax = 0, ay = 0;
        if (inter && !skip) {
            const int q = part_index(k->part, k->sub, lane & 3, lane >> 2);
            ax = (uint8_t)min(abs((int)k->mvds[q][0]), 64);
            ay = (uint8_t)min(abs((int)k->mvds[q][1]), 64);
        }
        n->mvd[lane][0] = ax;
        n->mvd[lane][1] = ay;
    } else if (lane < 24) {
        n->cnnz[(lane - 16) >> 2][(lane - 16) & 3] = k->res.cnnz[(lane - 16) >> 2][(lane - 16) & 3];
    } else if (lane < 28) {
        const int b8 = lane - 24;
        n->r8[b8] = inter ? (int8_t)k->refs[k->part == 0 ? 0 : k->part == 1 ? b8 >> 1 : k->part == 2 ? (b8 & 1) : b8] : (int8_t)-1;
    } else if (lane == 28) {
        const int cbpc = cbp >> 4;
        n->avail = 1;
        n->skip = (uint8_t)skip;
        n->kind = (uint8_t)kind;
        n->inter = inter;
        n->cbp = (uint8_t)cbp;
        n->t8x8 = k->res.t8x8;
        n->chroma_mode = inter ? 0 : k->chroma_mode;
        n->cbf_dc = (uint8_t)((kind == KIND_I16 && (bal & 0xFFFFu)) | ((cbpc > 0 && (bal & 0xF0000u)) << 1) | ((cbpc > 0 && (bal & 0xF00000u)) << 2));
    }
    __syncwarp();
}

__device__ __forceinline__ bool nxn(int kind) { return kind == KIND_I4 || kind == KIND_I8; }

// pred_i4_mode, enc/frame.rs:619-627, with the neighbours' modes in nbm (left column then top row: a mode, 2
// for a macroblock that is neither Intra4x4 nor Intra8x8, -1 unavailable).
__device__ __forceinline__ int pred_mode(const int* nbm, const uint8_t* cur, int bx, int by) {
    const int a = bx > 0 ? cur[by * 4 + bx - 1] : nbm[by];
    const int b = by > 0 ? cur[(by - 1) * 4 + bx] : nbm[4 + bx];
    return (a >= 0 && b >= 0) ? min(a, b) : 2;
}

// mvd_bins, enc/frame.rs:2393-2414
template <class S>
__device__ __forceinline__ void mvd(S& c, int comp, int d, uint32_t sum) {
    const int base = comp == 0 ? 40 : 47, inc = sum < 3 ? 0 : sum > 32 ? 2 : 1;
    const uint32_t a = (uint32_t)abs(d);
    c.decision(base + inc, a > 0);
    if (a == 0) return;
    int ctx = base + 3;
    for (uint32_t k = 1; k < (a < 9 ? a : 9); k++) {
        c.decision(ctx, 1);
        if (ctx < base + 6) ctx++;
    }
    if (a < 9) c.decision(ctx, 0);
    else {
        uint32_t v = a - 9, k = 3;
        while (v >= (1u << k)) {
            c.bypass(1);
            v -= 1u << k;
            k++;
        }
        c.bypass(0);
        while (k > 0) {
            k--;
            c.bypass((v >> k) & 1);
        }
    }
    c.bypass(d < 0);
}

// The slice's parameters the walk reads.
struct Slice {
    int p_slice, t8, nref;
};

// mb_bins after mb_skip_flag and before the residual (enc/frame.rs:2046-2244), in three pieces in coding order, so that the
// middle one's parts can be walked side by side: mb_type (with an Intra NxN macroblock's transform_size_8x8_flag),
// sub_mb_type and ref_idx; the prediction modes or the vector differences; the rest.
template <class S>
__device__ __forceinline__ void head_first(S& c, const Slice& sl, const ironav_mbcode* code, const Nb& L, const Nb& T) {
    const bool la = L.avail, ta = T.avail;
    const int kind = code->kind, cbp = code->res.cbp, cbpl = cbp & 15, cbpc = cbp >> 4;
    // mb_type
    if (kind != KIND_INTER) {
        const int pre = sl.p_slice, base = pre ? 17 : 3;
        int first;
        if (pre) {
            c.decision(14, 1);
            first = 17;
        } else {
            first = 3 + (la && !nxn(L.kind)) + (ta && !nxn(T.kind));
        }
        if (nxn(kind)) {
            c.decision(first, 0);
            if (sl.t8) c.decision(399 + (la && L.t8x8) + (ta && T.t8x8), kind == KIND_I8);
        } else {
            c.decision(first, 1);
            c.terminate(0);  // not I_PCM
            c.decision(pre ? base + 1 : base + 3, cbpl != 0);
            c.decision(pre ? base + 2 : base + 4, cbpc != 0);
            if (cbpc) c.decision(pre ? base + 2 : base + 5, cbpc == 2);
            c.decision(pre ? base + 3 : base + 6, (code->i16_mode >> 1) == 1);
            c.decision(pre ? base + 3 : base + 7, code->i16_mode & 1);
        }
        return;
    }
    // P_L0_16x16 000, P_L0_L0_16x8 011, P_L0_L0_8x16 010, P_8x8 001
    const int b1 = code->part == 1 || code->part == 2, b2 = code->part == 1 || code->part == 3;
    c.decision(14, 0);
    c.decision(15, b1);
    c.decision(b1 ? 17 : 16, b2);
    // sub_mb_type of each 8x8 block of P_8x8 (Table 9-38: 1, 00, 011, 010; contexts 21 to 23)
    if (code->part == 3)
        for (int k = 0; k < 4; k++) {
            const int s = code->sub[k];
            c.decision(21, s == 0);
            if (s != 0) {
                c.decision(22, s != 1);
                if (s != 1) c.decision(23, s == 2);
            }
        }
    // ref_idx_l0 per partition (per 8x8 block for P_8x8), unary, with the contexts of 9.3.3.1.1.6
    if (sl.nref > 1) {
        uint8_t grid[4] = {0, 0, 0, 0};
        const int np = code->part == 0 ? 1 : code->part == 3 ? 4 : 2;
        for (int k = 0; k < np; k++) {
            int bx, by, w, h;
            if (code->part == 0) bx = 0, by = 0, w = 4, h = 4;
            else if (code->part == 1) bx = 0, by = 2 * k, w = 4, h = 2;
            else if (code->part == 2) bx = 2 * k, by = 0, w = 2, h = 4;
            else bx = (k & 1) * 2, by = (k >> 1) * 2, w = 2, h = 2;
            const int a = bx > 0 ? grid[(by / 2) * 2 + (bx - 1) / 2] > 0 : (la && L.r8[(by / 2) * 2 + 1] > 0);
            const int b = by > 0 ? grid[((by - 1) / 2) * 2 + bx / 2] > 0 : (ta && T.r8[2 + bx / 2] > 0);
            const int r = code->refs[k], base = 54 + a + 2 * b;
            for (int i = 0; i <= r; i++) c.decision(i == 0 ? base : i == 1 ? 58 : 59, i < r);
            for (int y8 = by / 2; y8 <= (by + h - 1) / 2; y8++)
                for (int x8 = bx / 2; x8 <= (bx + w - 1) / 2; x8++) grid[y8 * 2 + x8] = code->refs[k];
        }
    }
}

// Part n (0..15, in coding order) of the middle piece: the prediction mode of block n of an Intra NxN macroblock, or the
// vector difference of partition n of an inter one; nothing beyond the last. The modes of the blocks before it and the
// differences of the partitions before it are the code's own, so every part can be walked on its own.
template <class S>
__device__ __forceinline__ void head_part(S& c, const ironav_mbcode* code, const Nb& L, const Nb& T, const int* nbm, int n) {
    const int kind = code->kind;
    if (nxn(kind)) {
        const bool t8 = kind == KIND_I8;
        if (t8 && n >= 4) return;
        const int bx = t8 ? (n & 1) * 2 : ((n >> 2) & 1) * 2 + (n & 1);
        const int by = t8 ? (n >> 1) * 2 : ((n >> 3) & 1) * 2 + ((n >> 1) & 1);
        // the blocks to the left and above, at the origin of their 8x8 block for Intra8x8
        const int step = t8 ? 2 : 1;
        const int a = bx > 0 ? (int)code->modes[by * 4 + bx - step] : nbm[by], b = by > 0 ? (int)code->modes[(by - step) * 4 + bx] : nbm[4 + bx];
        const int mode = code->modes[by * 4 + bx], pred = (a >= 0 && b >= 0) ? min(a, b) : 2;
        c.decision(68, mode == pred);
        if (mode != pred) {
            const int rem = mode < pred ? mode : mode - 1;
            for (int k = 0; k < 3; k++) c.decision(69, (rem >> k) & 1);
        }
        return;
    }
    if (kind != KIND_INTER) return;
    int bx, by;
    if (!part_origin(code->part, code->sub, n, &bx, &by)) return;
    // the blocks left of and above a partition in the macroblock belong to earlier ones
    const int pl = bx > 0 ? part_index(code->part, code->sub, bx - 1, by) : 0, pt = by > 0 ? part_index(code->part, code->sub, bx, by - 1) : 0;
    for (int comp = 0; comp < 2; comp++) {
        const uint32_t a = bx > 0 ? (uint32_t)min(abs((int)code->mvds[pl][comp]), 64) : (L.avail ? L.mvd[by * 4 + 3][comp] : 0u);
        const uint32_t b = by > 0 ? (uint32_t)min(abs((int)code->mvds[pt][comp]), 64) : (T.avail ? T.mvd[12 + bx][comp] : 0u);
        mvd(c, comp, code->mvds[n][comp], a + b);
    }
}

template <class S>
__device__ __forceinline__ void head_last(S& c, const Slice& sl, const ironav_mbcode* code, const Nb& L, const Nb& T) {
    const bool la = L.avail, ta = T.avail;
    const int kind = code->kind, cbp = code->res.cbp, cbpl = cbp & 15, cbpc = cbp >> 4;
    if (kind != KIND_INTER) {
        const int m = code->chroma_mode;
        c.decision(64 + (la && !L.inter && L.chroma_mode != 0) + (ta && !T.inter && T.chroma_mode != 0), m > 0);
        if (m > 0) {
            c.decision(67, m > 1);
            if (m > 1) c.decision(67, m > 2);
        }
    }
    if (kind != KIND_I16) {
        int luma = 0;
        for (int b8 = 0; b8 < 4; b8++) {
            const int ca = (b8 & 1) ? ((luma >> (b8 - 1)) & 1) == 0 : (la && ((L.cbp >> (b8 + 1)) & 1) == 0);
            const int cb = b8 >= 2 ? ((luma >> (b8 - 2)) & 1) == 0 : (ta && ((T.cbp >> (b8 + 2)) & 1) == 0);
            const int bit = (cbpl >> b8) & 1;
            c.decision(73 + ca + 2 * cb, bit);
            luma |= bit << b8;
        }
        c.decision(77 + (la && (L.cbp >> 4) != 0) + 2 * (ta && (T.cbp >> 4) != 0), cbpc != 0);
        if (cbpc) c.decision(81 + (la && (L.cbp >> 4) == 2) + 2 * (ta && (T.cbp >> 4) == 2), cbpc == 2);
    }
    // transform_size_8x8_flag is absent from P_8x8 with any sub-partition smaller than 8x8
    if (kind == KIND_INTER && sl.t8 && cbpl && (code->part != 3 || !(code->sub[0] | code->sub[1] | code->sub[2] | code->sub[3])))
        c.decision(399 + (la && L.t8x8) + (ta && T.t8x8), code->res.t8x8);
    if (!cbp && kind != KIND_I16) return;
    c.decision(60, 0);  // mb_qp_delta 0, after a macroblock without a change
}

// The exclusive prefix sum of v over the warp; the total on every lane.
__device__ __forceinline__ int warp_scan(int v, int* total) {
    const int lane = threadIdx.x & 31;
    int x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    *total = __shfl_sync(0xffffffffu, x, 31);
    return x - v;
}

// The map contexts per scan position, a nibble each: a position's own number, or for the quarters of an 8x8 block significant_coeff_flag's
// and last_significant_coeff_flag's of Table 9-43 (frame coded).
constexpr unsigned long long MAP_OWN = 0xFEDCBA9876543210ull;
__device__ __forceinline__ unsigned long long map_sig8(int part) {
    return part == 0 ? 0x5544433445543210ull : part == 1 ? 0x789A987776334444ull : part == 2 ? 0xB689AE9876BDCB67ull : 0x0CAEBDCB9AE96BDCull;
}
__device__ __forceinline__ unsigned long long map_last8(int part) {
    return part == 0 ? 0x1111111111111110ull : part == 1 ? 0x2222222222222222ull : part == 2 ? 0x4444444433333333ull : 0x0888777766665555ull;
}

// A lane's share of a macroblock's residual bins (write_block, enc/cabac.rs:194-250: coded_block_flag, the significance map and the
// levels of a block): a block of up to 16 levels, or a quarter of an 8x8 block's 64. Its map bins lie together, and so do its level
// bins, which run from the last position down; `os` and `ol` are where in the macroblock's residual bins. Lane 0: the Intra16x16
// DC; 1-16: the luma blocks (4x4 in decoding order, or four lanes an 8x8 block); 17, 18: chroma DC; 19-26: chroma AC. What its
// bins hang on across the quarters is known from the block's masks of non-zero levels and of those above 1, so that the quarters
// are counted without a walk and listed side by side. (With a lane an 8x8 block, each block walked twice, the price of an
// Intra8x8 macroblock took 12 to 16 us, of an Intra4x4 one 10; with the quarters, the decide of an IDR and three P pictures at
// 1080p went from 126 to 118 ms.)
struct ResPiece {
    const int16_t* lv;           // its levels, in scan order
    unsigned long long sig, lst;  // its positions' map contexts
    int so, lo, ab, cbf;         // the contexts' bases; coded_block_flag's context (-1: none)
    int cnt, last;               // its positions in the map; the block's last non-zero position, from its first
    unsigned nz;                 // its non-zero levels
    int eq, gt;                  // the block's levels of 1 and above 1 after its own
    int capn;                    // contexts of a level's further bins
    int os, ns, ol, nl;
    bool coded;                  // the block has a non-zero level
};

// Every lane's share; BYP: the bypass bins count as bins, and otherwise as 256 of `bits` each. Returns all lanes' bins.
template <bool BYP>
__device__ __forceinline__ int res_pieces(ResPiece& r, const ironav_mbcode* code, const Nb& L, const Nb& T, uint32_t* bits) {
    const int i = threadIdx.x & 31;
    const bool la = L.avail, ta = T.avail;
    const int kind = code->kind, cbp = code->res.cbp, cbpl = cbp & 15, cbpc = cbp >> 4;
    const bool t8 = code->res.t8x8;
    // an unavailable neighbour counts as a coded block for an intra macroblock
    const int un = kind != KIND_INTER;
    int cat = 0, cbf = -1, max = 0, part = 0;
    const int16_t* lv = code->dc;
    if (code->skip || !(cbp || kind == KIND_I16)) {
    } else if (i == 0) {
        if (kind == KIND_I16) {
            max = 16;
            cbf = 85 + (la ? (L.cbf_dc & 1) != 0 : un) + 2 * (ta ? (T.cbf_dc & 1) != 0 : un);
        }
    } else if (i < 17) {
        const int n = i - 1;
        if (!(cbpl & (1 << (n >> 2)))) {
        } else if (t8) {
            part = n & 3;
            cat = 5, max = 16, lv = code->res.luma8[n >> 2] + 16 * part;
        } else {
            const int bx = ((n >> 2) & 1) * 2 + (n & 1), by = ((n >> 3) & 1) * 2 + ((n >> 1) & 1);
            const int fa = bx > 0 ? code->res.nnz[by * 4 + bx - 1] > 0 : (la ? L.nnz[by * 4 + 3] > 0 : un);
            const int fb = by > 0 ? code->res.nnz[(by - 1) * 4 + bx] > 0 : (ta ? T.nnz[12 + bx] > 0 : un);
            const bool i16 = kind == KIND_I16;
            cat = i16 ? 1 : 2, cbf = (i16 ? 89 : 93) + fa + 2 * fb, max = i16 ? 15 : 16;
            lv = code->res.luma[by * 4 + bx] + (i16 ? 1 : 0);
        }
    } else if (i < 19) {
        if (cbpc != 0) {
            const int comp = i - 17, m = 2 << comp;
            cat = 3, max = 4, lv = code->res.cdc[comp];
            cbf = 97 + (la ? (L.cbf_dc & m) != 0 : un) + 2 * (ta ? (T.cbf_dc & m) != 0 : un);
        }
    } else if (i < 27 && cbpc == 2) {
        const int comp = (i - 19) >> 2, blk = (i - 19) & 3, bx = blk & 1, by = blk >> 1;
        const uint8_t* cur = code->res.cnnz[comp];
        const int fa = bx > 0 ? cur[by * 2] > 0 : (la ? L.cnnz[comp][by * 2 + 1] > 0 : un);
        const int fb = by > 0 ? cur[bx] > 0 : (ta ? T.cnnz[comp][2 + bx] > 0 : un);
        cat = 4, max = 15, lv = code->res.cac[comp][blk] + 1, cbf = 101 + fa + 2 * fb;
    }
    // its own levels: which are there, which are above 1, and their bins (a level's context bins: its magnitude, 14 at most)
    unsigned nz = 0, big = 0;
    int dec = 0, byp = 0;
#pragma unroll
    for (int k = 0; k < 16; k++) {
        const int a = k < max ? abs((int)lv[k]) : 0;
        nz |= (unsigned)(a != 0) << k;
        big |= (unsigned)(a > 1) << k;
        dec += min(a, 14);
        if (a >= 15) byp += 2 * (31 - __clz(a - 14)) + 1;
    }
    byp += __popc(nz);
    const int len = BYP ? dec + byp : dec;
    // the block: its masks, and the level bins of the quarters after this one
    unsigned long long bnz = nz, bbig = big;
    int above = 0;
    const bool quarter = t8 && i >= 1 && i <= 16;
    const int head = quarter ? i - ((i - 1) & 3) : i;  // the block's first lane
    if (t8) {
        unsigned m[4];
        int l[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int from = quarter ? head + q : i;
            m[q] = __shfl_sync(0xffffffffu, nz | big << 16, from);
            l[q] = __shfl_sync(0xffffffffu, len, from);
        }
        if (quarter) {
            bnz = (unsigned long long)((m[0] & 0xffffu) | m[1] << 16) | (unsigned long long)((m[2] & 0xffffu) | m[3] << 16) << 32;
            bbig = (unsigned long long)(m[0] >> 16 | (m[1] & 0xffff0000u)) | (unsigned long long)(m[2] >> 16 | (m[3] & 0xffff0000u)) << 32;
#pragma unroll
            for (int q = 1; q < 4; q++) above += q > part ? l[q] : 0;
        }
    }
    const int p0 = 16 * part, last = 63 - __clzll((long long)bnz), all = cat == 5 ? 64 : max;
    const int maps = min(last + 1, all - 1);  // the block's positions in the map (the last position of all has no bins)
    const int mine = bnz ? min(max - (cat == 5 ? 0 : 1), maps - p0) : 0;
    auto below = [](unsigned long long m, int n) { return __popcll(n >= 64 ? m : m & ((1ull << n) - 1)); };  // of the first n positions
    const int flag = part == 0 && cbf >= 0, c0 = cbf >= 0;
    r.lv = lv;
    r.sig = cat == 5 ? map_sig8(part) : MAP_OWN;
    r.lst = cat == 5 ? map_last8(part) : MAP_OWN;
    r.so = SIG_OFF[0][cat];
    r.lo = LAST_OFF[0][cat];
    r.ab = ABS_OFF[cat];
    r.capn = 4 - (cat == 3);
    r.cbf = cbf;
    r.cnt = mine > 0 ? mine : 0;
    r.last = last - p0;
    r.nz = nz;
    const unsigned long long up = part == 3 || !quarter ? 0ull : bnz >> (p0 + 16), upb = part == 3 || !quarter ? 0ull : bbig >> (p0 + 16);
    r.gt = __popcll(upb);
    r.eq = __popcll(up) - r.gt;
    r.coded = bnz != 0;
    r.ns = flag + r.cnt + below(nz, r.cnt);
    r.nl = len;
    *bits = BYP ? 0u : 256u * (uint32_t)byp;
    int total;
    const int at = warp_scan(r.ns + r.nl, &total), base = __shfl_sync(0xffffffffu, at, head);
    // the map bins of the quarters before it; then, after all the block's, the level bins of the quarters after it
    const int maps_all = bnz ? maps : 0, before = min(p0, maps_all);
    r.os = base + (quarter ? before + below(bnz, before) : 0);
    r.ol = base + c0 + maps_all + below(bnz, maps_all) + above;
    return total;
}

template <class S>
__device__ __forceinline__ void list_map(S& c, const ResPiece& r) {
    if (r.ns > 0 && r.cbf >= 0) c.decision(r.cbf, r.coded);
    for (int k = 0; k < r.cnt; k++) {
        const int bit = (int)((r.nz >> k) & 1u);
        c.decision(r.so + (int)((r.sig >> (4 * k)) & 15u), bit);
        if (bit) c.decision(r.lo + (int)((r.lst >> (4 * k)) & 15u), k == r.last);
    }
}

template <class S>
__device__ __forceinline__ void list_levels(S& c, const ResPiece& r) {
    int eq1 = r.eq, gt1 = r.gt;
    for (unsigned nz = r.nz; nz;) {
        const int i = 31 - __clz((int)nz);
        nz ^= 1u << i;
        const int l = r.lv[i];
        const uint32_t a = (uint32_t)abs(l);
        const int inc0 = gt1 ? 0 : min(1 + eq1, 4);
        if (a == 1) {
            c.decision(r.ab + inc0, 0);
            eq1++;
        } else {
            c.decision(r.ab + inc0, 1);
            const int incn = r.ab + 5 + min(gt1, r.capn);
            // abs - 2 ones and a zero, the ones capped at 13 with the rest in an Exp-Golomb suffix
            const uint32_t ones = a - 2 < 13 ? a - 2 : 13;
            for (uint32_t k = 0; k < ones; k++) c.decision(incn, 1);
            if (a < 15) c.decision(incn, 0);
            else {
                uint32_t v = a - 15, k = 0;  // exp_golomb(abs - 15, 0), enc/cabac.rs:17-29
                while (v >= (1u << k)) {
                    c.bypass(1);
                    v -= 1u << k;
                    k++;
                }
                c.bypass(0);
                while (k > 0) {
                    k--;
                    c.bypass((v >> k) & 1);
                }
            }
            gt1++;
        }
        c.bypass(l < 0);
    }
}

// mb_skip_flag of a P slice's macroblock.
template <class S>
__device__ __forceinline__ void skip_bin(S& c, const ironav_mbcode* code, const Nb& L, const Nb& T) {
    c.decision(11 + (L.avail && !L.skip) + (T.avail && !T.skip), code->skip);
}

// The bins of a macroblock, mb_bins (enc/frame.rs:2028-2279) for I and P slices, are listed by a warp: a lane walks each piece (the
// head's pieces, then the residual's shares, all independent given the code and its neighbours) at the offset a scan of the
// pieces' counts gives. (One lane walking a macroblock's bins one by one spent 40 us on a
// coded macroblock's candidates and 49 us on writing an intra macroblock.) A listed bin: its context, bin << 10, and
// whether it is a bypass (or, with both, a terminate) bin.
constexpr uint32_t BIN_BYPASS = 1u << 11, BIN_TERMINATE = 1u << 12;

// What a piece holds: its bins and, where only contexts are listed (the price), the cost of the others.
struct PriceCount {
    int n = 0;
    uint32_t bits = 0;
    __device__ __forceinline__ void decision(int, int) { n++; }
    __device__ __forceinline__ void bypass(int) { bits += 256; }
    __device__ __forceinline__ void terminate(int bin) { bits += bin ? 7 * 256 : 1; }
};
struct PriceList {
    uint16_t* p;
    __device__ __forceinline__ void decision(int ctx, int bin) { *p++ = (uint16_t)(ctx | (bin != 0) << 10); }
    __device__ __forceinline__ void bypass(int) {}
    __device__ __forceinline__ void terminate(int) {}
};
struct BinCount {
    int n = 0;
    __device__ __forceinline__ void decision(int, int) { n++; }
    __device__ __forceinline__ void bypass(int) { n++; }
    __device__ __forceinline__ void terminate(int) { n++; }
};
struct BinList {
    uint16_t* p;
    __device__ __forceinline__ void decision(int ctx, int bin) { *p++ = (uint16_t)(ctx | (bin != 0) << 10); }
    __device__ __forceinline__ void bypass(int bin) { *p++ = (uint16_t)(BIN_BYPASS | (bin != 0) << 10); }
    __device__ __forceinline__ void terminate(int bin) { *p++ = (uint16_t)(BIN_TERMINATE | (bin != 0) << 10); }
};

// This lane's piece of a macroblock's head bins, in coding order over the lanes: lane 0 the skip flag and head_first, lanes 1-16 the
// parts, lane 17 head_last.
template <class S>
__device__ __forceinline__ void lane_head(S& c, const Slice& sl, const ironav_mbcode* code, const Nb& L, const Nb& T, const int* nbm) {
    const int lane = threadIdx.x & 31;
    if (lane == 0) {
        if (sl.p_slice) skip_bin(c, code, L, T);
        if (!code->skip) head_first(c, sl, code, L, T);
    } else if (!code->skip && lane <= 16) {
        head_part(c, code, L, T, nbm, lane - 1);
    } else if (!code->skip && lane == 17) {
        head_last(c, sl, code, L, T);
    }
}
// Bins a price's list holds. A piece never has more (a share's map bins, or its 16 levels of at most 14 context bins); a macroblock's
// pieces that together do are listed in several turns.
constexpr int PRICE_CAP = 1152;
static_assert(16 * 14 <= PRICE_CAP && 1 + 2 * 16 <= PRICE_CAP, "one piece fits the list");

// The cost in 1/256 bits of the listed decisions, their contexts advanced in st (CabacCost, enc/cabac.rs:150-192). 32 bins a
// turn, in order: the bins of a context form a chain, walked by its first lane, the contexts side by side.
__device__ __forceinline__ uint32_t price_list(const uint16_t* list, int n, uint8_t* st, const uint32_t* step) {
    const int lane = threadIdx.x & 31;
    uint32_t bits = 0;
    for (int i0 = 0; i0 < n; i0 += 32) {
        const bool in = i0 + lane < n;
        const uint32_t e = in ? list[i0 + lane] : 0u;
        const int ctx = in ? (int)(e & 1023u) : 1024 + lane;
        uint32_t m = __match_any_sync(0xffffffffu, ctx);
        const uint32_t ones = __ballot_sync(0xffffffffu, (e >> 10) & 1u);
        if (in && (m & ((1u << lane) - 1u)) == 0) {
            uint32_t s = st[ctx];
            do {
                const uint32_t v = step[s * 2 + ((ones >> (__ffs(m) - 1)) & 1u)];
                m &= m - 1;
                bits += v >> 8;
                s = v & 0xffu;
            } while (m);
            st[ctx] = (uint8_t)s;
        }
        __syncwarp();
    }
    return bits;
}

// The bits of macroblock `code` (1/256 bits, on every lane) from the contexts `live`, and the contexts after it in st. list: PRICE_CAP
// entries of the warp's own.
__device__ __forceinline__ uint32_t price(const uint8_t* live, uint8_t* st, const uint32_t* step, uint16_t* list, const Slice& sl,
                                          const ironav_mbcode* code, const Nb& L, const Nb& T, const int* nbm) {
    const int lane = threadIdx.x & 31;
    const uint4* s16 = reinterpret_cast<const uint4*>(live);
    uint4* d16 = reinterpret_cast<uint4*>(st);
    d16[lane] = s16[lane];
    d16[lane + 32] = s16[lane + 32];
    PriceCount h;
    lane_head(h, sl, code, L, T, nbm);
    ResPiece r;
    uint32_t bits;
    int nh;
    const int nr = res_pieces<false>(r, code, L, T, &bits), oh = warp_scan(h.n, &nh), total = nh + nr;
    bits += h.bits;
    __syncwarp();
    int base = 0;
    do {
        // the pieces that lie in [base, base + PRICE_CAP): a run of whole ones from base on
        auto fits = [&](int at, int n) { return n > 0 && at >= base && at + n <= base + PRICE_CAP; };
        const bool fh = fits(oh, h.n), fm = fits(nh + r.os, r.ns), fl = fits(nh + r.ol, r.nl);
        if (fh) {
            PriceList c = {list + (oh - base)};
            lane_head(c, sl, code, L, T, nbm);
        }
        if (fm) {
            PriceList c = {list + (nh + r.os - base)};
            list_map(c, r);
        }
        if (fl) {
            PriceList c = {list + (nh + r.ol - base)};
            list_levels(c, r);
        }
        const int end = __reduce_max_sync(0xffffffffu, max(fh ? oh + h.n : 0, max(fm ? nh + r.os + r.ns : 0, fl ? nh + r.ol + r.nl : 0)));
        __syncwarp();
        bits += price_list(list, end - base, st, step);
        base = end;
    } while (base < total);
    return __reduce_add_sync(0xffffffffu, bits);
}

}  // namespace cab

}  // namespace ironav
