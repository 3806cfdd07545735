/*
 * Encoder kernels for sm_103a (the forward transform is in jxs_fwd_dwt.cu).
 *
 *  rc_cost_kernel   per precinct row: GCLI histograms and the byte cost of
 *                   every (quantization, refinement) candidate.
 *                   The block that completes a slice then replays the
 *                   reference's sequential budget carry and binary searches
 *                   for that slice over the cost tables.
 *  pack_kernel      per precinct row: quantization and bit packing at
 *                   prefix-summed bit offsets into a shared-memory copy of the
 *                   precinct, then one coalesced copy to the codestream.
 *
 * Integer arithmetic follows the reference one to one (citations inline).
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <type_traits>

#include "jxs_core.h"
#include "jxs_kernels.cuh"

#define DEV __device__ __forceinline__

/* ------------------------------------------------------------------------ */
/* Rate control                                                              */
/* ------------------------------------------------------------------------ */
#define FULL 0xffffffffu
#define RC_THREADS 512
#define RC_WARPS (RC_THREADS / 32)
/* shared area of the rate control: 5 tables of 16 words per band line, 6
 * with sign handling */
#define RC_NOS 24
#define RC_SIG 46
#define RC_AREA_WORDS(signs) (((signs) ? 6 : 5) * JXS_MAXBLINES * 16)

/* binary_search_init / binary_search_next_step (BinarySearch.c:9-78) */
struct BSearch {
    int beg, end, step, best, last, below;
};
DEV void bs_init(BSearch& s, int beg, int end, int below, int step) {
    s.beg = beg; s.end = end; s.below = below; s.best = -1; s.last = -1;
    s.step = step ? step : (end - beg) / 2;
}
enum { BS_BEGIN = 0, BS_TOO_SMALL, BS_TOO_BIG, BS_OUT_OF_RANGE };
enum { BS_CONTINUE = 0, BS_FOUND, BS_ERROR };
DEV int bs_next(BSearch& s, int res, int* out) {
    if (res == BS_TOO_SMALL) {
        if (s.below && (s.best == -1 || s.best < s.last)) s.best = s.last;
        if (s.end >= s.last + 1) s.beg = s.last + 1;
        else {
            if (s.best == -1) return BS_ERROR;
            *out = s.best;
            return BS_FOUND;
        }
    } else if (res == BS_TOO_BIG || res == BS_OUT_OF_RANGE) {
        if (res == BS_TOO_BIG && !s.below && (s.best == -1 || s.best > s.last)) s.best = s.last;
        if (s.beg <= s.last - 1) s.end = s.last - 1;
        else {
            if (s.best == -1) return BS_ERROR;
            *out = s.best;
            return BS_FOUND;
        }
    }
    if (s.step > s.end - s.beg) s.step = (s.end - s.beg + 1) / 2;
    s.last = s.step + s.beg;
    *out = s.last;
    return BS_CONTINUE;
}

/* A slice's even split of its budget over its precincts
 * (PackStageProcess.c:600-684): mode 1 gives the first precinct 10 % more
 * (20 % with fast signs, :34-35). */
struct SliceSplit {
    uint32_t slice_budget, first_p, nprec, first_b, min_b, left;
};
DEV SliceSplit slice_split(const jxs_cfg_t* __restrict__ cfg, int s) {
    SliceSplit o;
    const int last_slice = (s + 1 == (int)cfg->nslices);
    o.slice_budget = cfg->slice_size[s] - 6 - (last_slice ? 2 : 0);
    o.first_p = cfg->pps * s;
    o.nprec = last_slice ? cfg->np - o.first_p : cfg->pps;
    o.min_b = o.slice_budget / o.nprec;
    o.left = o.slice_budget - o.min_b * o.nprec;
    o.first_b = o.min_b;
    if (cfg->rc_mode == 1) {
        o.first_b = min(o.slice_budget, o.first_b * (cfg->signs == 1 ? 120u : 110u) / 100);
        if (o.nprec > 1) {
            o.min_b = (o.slice_budget - o.first_b) / (o.nprec - 1);
            o.left = o.slice_budget - o.min_b * (o.nprec - 1) - o.first_b;
        } else {
            o.left = 0;
        }
    }
    return o;
}

/* What the searches of a slice read of the configuration, held in
 * registers by every lane of the searching warp. */
struct RcParams {
    int nr, max_q, max_r, rc_mode, signs;
    uint32_t hdrs0, hdrs1, np, empty; /* empty: lane q's word of cfg->empty */
};
DEV RcParams rc_params(const jxs_cfg_t* __restrict__ cfg) {
    RcParams P;
    P.nr = cfg->max_r + 1;
    P.max_q = cfg->max_q;
    P.max_r = cfg->max_r;
    P.rc_mode = (int)cfg->rc_mode;
    P.signs = (int)cfg->signs;
    P.hdrs0 = cfg->hdrs_bytes[0];
    P.hdrs1 = cfg->hdrs_bytes[1];
    P.np = cfg->np;
    P.empty = cfg->empty[threadIdx.x & 31];
    return P;
}
/* Both for a block's slice, in shared memory: read from the configuration
 * with its other tables, before the costs, so that the slice's selection, on
 * which a single frame waits, starts at once (3840x2160: the kernel 32.4 ->
 * 30.8 us). */
struct SliceInfo {
    RcParams P;
    SliceSplit sp;
    uint32_t begin, empty[32]; /* first byte after the slice header; per Q */
};
DEV void slice_info(const jxs_cfg_t* __restrict__ cfg, int s, SliceInfo* o) { /* by one warp */
    const RcParams P = rc_params(cfg);
    o->empty[threadIdx.x & 31] = P.empty;
    if ((threadIdx.x & 31) == 0) {
        o->P = P;
        o->sp = slice_split(cfg, s);
        o->begin = cfg->slice_begin[s] + 6;
    }
}

/* The reference's binary search (binary_search_next_step) over v in [0, n],
 * n <= 31, with the answers of every v known: bit v of `small` is "too
 * small" (the search moves up, the result with below = 1), of `big` "too
 * big" (it moves down, the result with below = 0), neither "out of range" (it
 * moves down).  Where exactly the lowest values are too small, every such
 * search ends at the border; other patterns (a cost that does not fall with
 * Q or grow with R) are searched step by step.  Returns the result or -1. */
DEV int mask_search(uint32_t small, uint32_t big, int n, int below, int step) {
    if (!(small & (small + 1u))) {
        const int border = __popc(small);
        if (below) {
            if (border > 0) return border - 1;
        } else if (border <= n && ((big >> border) & 1u)) {
            return border;
        }
    }
    BSearch bs;
    bs_init(bs, 0, n, below, step);
    int res, next = BS_BEGIN, v = 0;
    while ((res = bs_next(bs, next, &v)) == BS_CONTINUE)
        next = (small >> v) & 1u ? BS_TOO_SMALL : (big >> v) & 1u ? BS_TOO_BIG : BS_OUT_OF_RANGE;
    return res == BS_FOUND ? v : -1;
}

/* The precinct searches of rate_control_precinct (RateControl.c:1259-1333,
 * binary searches :889-1083), by one warp on tables in shared memory
 * ([q * ld + r]), a lane per candidate: the quantization by binary search on
 * T[q * ld]; with `scan` (full signs, vertical prediction) then lower
 * quantizations while TS fits, else the first higher one that fits
 * (:936-1015); the refinement by binary search on TS.  Returns an error
 * code, 0 when q, r and data (TS at (q, r)) are set; the same in every
 * lane. */
DEV int prec_search(const RcParams& P, const uint32_t* T, int ldt, const uint32_t* TS, int ld, int scan, uint32_t avail, int& q, int& r,
                    uint32_t& data) {
    const int lane = threadIdx.x & 31;
    const bool inq = lane <= P.max_q;
    const uint32_t none = __ballot_sync(FULL, inq && (P.empty & 1u)); /* every band truncated: out of range */
    const uint32_t fit = __ballot_sync(FULL, inq && T[lane * ldt] <= avail) & ~none;
    const uint32_t fulq = (2u << P.max_q) - 1u;
    q = mask_search(fulq & ~fit & ~none, fit, P.max_q, 0, 6 > P.max_q ? 0 : 6);
    if (q < 0) return JXS_E_ENC_FRAME;
    if (scan) {
        const uint32_t ok = __ballot_sync(FULL, inq && TS[lane * ld] <= avail) & ~none;
        const uint32_t low = (1u << q) - 1u, gaps = low & ~ok;
        const int run0 = gaps ? 32 - __clz((int)gaps) : 0; /* first of the run of fitting values that ends at q - 1 */
        if (run0 < q) q = run0;
        else if (ok & ~low) q = __ffs((int)(ok & ~low)) - 1;
        else return JXS_E_ENC_FRAME;
    }
    const bool inr = lane <= P.max_r;
    const uint32_t eq = __shfl_sync(FULL, P.empty, q);
    const uint32_t row = inr ? TS[q * ld + lane] : 0xffffffffu;
    const uint32_t fitr = __ballot_sync(FULL, inr && row <= avail) & ~eq;
    r = mask_search(fitr, __ballot_sync(FULL, inr) & ~fitr & ~eq, P.max_r, 1, 6 >= P.max_r ? 0 : 6);
    if (r < 0) return JXS_E_ENC_FRAME;
    data = __shfl_sync(FULL, row, r);
    return 0;
}

/* RC modes 2 and 3, per-slice common quantization (process_slice,
 * PackStageProcess.c:339-483; RateControl.c:1086-1209, 1336-1425): the
 * (fast-sign) data bytes of every (Q, R) summed over the slice's precincts
 * into `area`, one (Q, R) for the slice by the precinct searches, then the
 * budget of each precinct, kept in rc[p].total_bytes.  Run by a whole
 * block; returns the error (every thread). */
DEV int slice_common(const RcParams& P, int s, const SliceSplit& sp, const uint32_t* cost, uint32_t* area,
                     PrecRC* rc, int* status) {
    __shared__ int s_cerr;
    const int nr = P.nr, nt = (P.max_q + 1) * nr, rc_mode = P.rc_mode;
    const uint32_t np_all = P.np, hdrs0 = P.hdrs0, hdrs1 = P.hdrs1;
    const uint32_t first_p = sp.first_p, nprec = sp.nprec, slice_budget = sp.slice_budget;
    __syncthreads();
    for (int e = threadIdx.x; e < nt; e += blockDim.x) {
        const int q = e / nr, r = e - q * nr;
        uint32_t sum = 0;
        for (uint32_t i = 0; i < nprec; i++) sum += __ldcg(cost + (uint64_t)(first_p + i) * 1024 + q * 32 + r);
        area[e] = sum;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        int err = 0;
        uint32_t headers = 0;
        for (uint32_t i = 0; i < nprec; i++) headers += first_p + i + 1 >= np_all ? hdrs1 : hdrs0;
        if ((slice_budget + nprec - 1) / nprec > JXS_PREC_MAX_BYTES) err = JXS_E_ENC_FRAME;
        else if (slice_budget <= headers) err = JXS_E_UNDEFINED;
        int q = 0, r = 0;
        uint32_t dsum = 0;
        if (!err) err = prec_search(P, area, nr, area, nr, 0, slice_budget - headers, q, r, dsum);
        if (!err && threadIdx.x == 0) {
            /* each precinct its headers and data at (Q, R); the last also
             * the slice's remaining bytes */
            uint32_t pad_last = slice_budget - headers;
            for (uint32_t i = 0; i < nprec; i++) {
                const uint32_t p = first_p + i;
                const uint32_t d = __ldcg(cost + (uint64_t)p * 1024 + q * 32 + r);
                pad_last -= d;
                rc[p].total_bytes = (p + 1 >= np_all ? hdrs1 : hdrs0) + d;
            }
            rc[first_p + nprec - 1].total_bytes += pad_last;
            if (rc_mode == 3) {
                /* RC_CBR_PER_SLICE_COMMON_QUANT_MAX_RATE: no precinct below a
                 * quarter of the largest, padding excluded */
                uint32_t max_size = 0;
                for (uint32_t i = 0; i < nprec; i++)
                    max_size = max(max_size, rc[first_p + i].total_bytes - (i + 1 == nprec ? pad_last : 0u));
                const uint32_t min_size = max_size / 4;
                uint32_t need = 0;
                for (uint32_t i = 0; i < nprec; i++) {
                    const uint32_t ds = rc[first_p + i].total_bytes - (i + 1 == nprec ? pad_last : 0u);
                    if (ds < min_size) {
                        rc[first_p + i].total_bytes += min_size - ds;
                        need += min_size - ds;
                    }
                }
                if (need) {
                    if (pad_last >= need) {
                        pad_last -= need;
                        rc[first_p + nprec - 1].total_bytes -= need;
                    } else {
                        need -= pad_last;
                        rc[first_p + nprec - 1].total_bytes -= pad_last;
                        pad_last = 0;
                        /* the rest one byte at a time, round robin */
                        const uint32_t each = need / nprec, extra = need - each * nprec;
                        for (uint32_t i = 0; i < nprec; i++) rc[first_p + i].total_bytes -= each + (i < extra ? 1u : 0u);
                    }
                }
            }
            if (pad_last > 0) {
                /* the first precinct 10 % more (20 % with fast signs), the
                 * rest of the padding shared evenly */
                uint32_t add_first = rc[first_p].total_bytes * (P.signs == 1 ? 20u : 10u) / 100;
                if (add_first > pad_last) add_first = pad_last;
                pad_last -= add_first;
                rc[first_p + nprec - 1].total_bytes -= add_first;
                rc[first_p].total_bytes += add_first;
                if (pad_last) {
                    rc[first_p + nprec - 1].total_bytes -= pad_last;
                    const uint32_t each = pad_last / nprec, extra = pad_last - each * nprec;
                    for (uint32_t i = 0; i < nprec; i++) rc[first_p + i].total_bytes += each + (i < extra ? 1u : 0u);
                }
            }
        }
        if (err && threadIdx.x == 0) {
            printf("jxs rc: slice %d (common quantization): error 0x%x\n", s, (unsigned)err);
            JXS_STATUS_SET(status, err);
        }
        if (threadIdx.x == 0) s_cerr = err;
    }
    __syncthreads();
    return s_cerr;
}

/* One precinct's budget, searches and padding carry, by one warp.  `T` (row
 * stride ldt) is the table of the quantization search, `F` the exact-sign
 * table (fast signs: the bytes of the signs not sent are T - F at the chosen
 * (Q, R)), `TS` (row stride ld) the table of the scan and the refinement
 * search; all in shared memory.
 * Modes 1-3 carry the padding (and fast signs' unsent sign bytes) to the
 * next precinct of the slice; a slice's last precinct and mode 0 keep them
 * as zero bytes (PackStageProcess.c:293-333, 526-560,
 * PackPrecinct.c:513-536).  Returns an error code; that, the carry, the
 * running offset and q, r are the same in every lane. */
DEV int prec_select(const RcParams& P, int s, uint32_t i, const SliceSplit& sp, const uint32_t* T, const uint32_t* F, int ldt,
                    const uint32_t* TS, int ld, int scan, uint32_t& carry, uint32_t& run, int& q, int& r, PrecRC* rc,
                    int* status) {
    const uint32_t p = sp.first_p + i;
    const uint32_t budget = (P.rc_mode >= 2 ? rc[p].total_bytes : (i == 0 ? sp.first_b : sp.min_b) + (i < sp.left ? 1 : 0)) + carry;
    const uint32_t hdr = p + 1 >= P.np ? P.hdrs1 : P.hdrs0;
    int err = 0;
    if (budget > JXS_PREC_MAX_BYTES) err = JXS_E_ENC_FRAME;
    else if (budget <= hdr) err = JXS_E_UNDEFINED;
    q = r = 0;
    uint32_t data = 0;
    if (!err) err = prec_search(P, T, ldt, TS, ld, scan, budget - hdr, q, r, data);
    if (!err) {
        const uint32_t padding = budget - hdr - data;
        uint32_t total = budget;
        const uint32_t retrieve = P.signs == 1 ? T[q * ldt + r] - F[q * ldt + r] : 0u;
        if (P.rc_mode >= 1 && i + 1 < sp.nprec) {
            total -= padding + retrieve;
            carry = padding + retrieve;
        } else {
            carry = 0;
        }
        if ((threadIdx.x & 31) == 0) {
            PrecRC o;
            o.total_bytes = total;
            o.offset = run;
            o.data_bytes = data - retrieve; /* the sub-packet bytes packed */
            o.q = (uint8_t)q;
            o.r = (uint8_t)r;
            o.first_in_slice = (uint8_t)(i == 0);
            o.pad = 0;
            rc[p] = o;
        }
        run += total;
    } else if ((threadIdx.x & 31) == 0) {
        printf("jxs rc: slice %d precinct %u budget %u: error 0x%x\n", s, p, budget, (unsigned)err);
        JXS_STATUS_SET(status, err);
    }
    return err;
}

/* Words of one [Q][R] table in the selection's shared memory: 32 rows of 36
 * words, so that rows are written 16 bytes at a time and a column is read
 * with 4-way conflicts. */
#define RC_TLD 36
#define RC_TWORDS (32 * RC_TLD)

/* One slice's selection without vertical prediction, on the slice's cost
 * tables: as many precincts' tables as fit are read (through L2) into `area`
 * at a time by the whole block; one warp then runs their searches in order, a
 * lane per candidate.  With sign handling each precinct has two tables: signs
 * counted the fast way (every coefficient of a group above gtli) and
 * exactly; the quantization search runs on the fast one, the full strategy
 * then scans and searches the refinement on the exact one.
 *
 * A chain of one search after another, 4 per slice of 16 lines: by one
 * thread, step by step, 24,000 cycles of the slice's last block, alone on
 * the critical path of a single frame; now 5,000. */
DEV void select_slice(const SliceInfo& I, int s, const uint32_t* cost, uint32_t* area, uint32_t area_words,
                      PrecRC* rc, int* status) {
    __shared__ int s_err;
    RcParams P = I.P;
    P.empty = I.empty[threadIdx.x & 31];
    const SliceSplit sp = I.sp;
    uint32_t carry = 0, run = I.begin;
    if (threadIdx.x == 0) s_err = 0;
    __syncthreads();
    if (P.rc_mode >= 2 && slice_common(P, s, sp, cost, area, rc, status)) return;
    const uint32_t ntab = P.signs ? 2 : 1, chunk = area_words / (RC_TWORDS * ntab);
    for (uint32_t c0 = 0; c0 < sp.nprec; c0 += chunk) {
        const uint32_t cnt = min(chunk, sp.nprec - c0);
        __syncthreads();
        if (s_err) break;
        for (uint32_t e = threadIdx.x; e < cnt * ntab * 256; e += blockDim.x) {
            /* 16 bytes of row q of table tb of precinct i */
            const uint32_t i = e / (ntab * 256), tb = (e >> 8) - i * ntab, q = (e >> 3) & 31u, c = 4 * (e & 7u);
            *(uint4*)(area + (e >> 8) * RC_TWORDS + q * RC_TLD + c) =
                __ldcg((const uint4*)(cost + ((uint64_t)tb * P.np + sp.first_p + c0 + i) * 1024 + q * 32 + c));
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            int err = 0, q, r;
            for (uint32_t ii = 0; ii < cnt && !err; ii++) {
                const uint32_t* T = area + ii * RC_TWORDS * ntab;
                const uint32_t* F = P.signs ? T + RC_TWORDS : T; /* exact signs */
                err = prec_select(P, s, c0 + ii, sp, T, F, RC_TLD, P.signs == 2 ? F : T, RC_TLD, P.signs == 2, carry, run, q, r, rc,
                                  status);
            }
            if (err && threadIdx.x == 0) s_err = err;
        }
    }
}

/* Vertical prediction (RateControl.c:586-676): line tables stored by every
 * precinct's block for the ordered selection, and the shared regions of
 * that selection */
#define RC_LT_REGION (JXS_MAXBLINES * 16)
#define RC_LT_WORDS (5 * RC_LT_REGION) /* data, GCLI bits, GCLI bits with significance, fast / full sign bits */
#define RC_VP_REGIONS 12

/* Code lengths of two GCLIs c (16-bit halves) predicted from those above, tp,
 * as ones of the unary code (vlc_encode_get_bits, PackPrecinct.h:86-104) plus
 * VP_K - VP_ONE: with d the GCLI less its prediction mt, neither below t (t2: t in
 * both halves, G2: max(t, gtli above)), d < 0 takes -2 d - 1 ones, else 2 d or,
 * past mt - t, d + mt - t.  *off: zero where d is 0. */
#define VP_ONE 0x00010001u
#define VP_K 0x20002000u
DEV uint32_t vp_codes(uint32_t c, uint32_t tp, uint32_t t2, uint32_t G2, uint32_t* off) {
    const uint32_t mt = __vmaxu2(tp, G2), gv = __vmaxu2(c, t2);
    const uint32_t X = 2u * (gv - mt) + VP_K;
    *off = X ^ VP_K;
    return __vmaxu2(__vminu2(X, gv + (VP_K - t2)), (2u * VP_K - VP_ONE) - X);
}

/* Byte costs of a packet at quantization q for the refinements that lower the
 * gtli of its lines `chunk` of four (in the order of their priorities), as
 * changes at those refinements; the first chunk also the cost at R = 0.
 * tw: a line's word per gtli (fields at 0, RC_NOS and RC_SIG); ta, tb: sign
 * bits per line and gtli, each rounded on its own (SB tables: SB = 1 adds ta
 * to da, SB = 2 also keeps a second cost with tb in db, RateControl.c:745-756).
 * A chain of one line after another: by whole packets the first one, with most
 * of the lines, kept all warps waiting (a 256x64 block's costs 4,100 cycles,
 * 2,800 by four lines). */
template <int SB>
DEV void packet_costs(int q, uint32_t chunk, uint32_t b0, uint32_t nb, uint32_t raw, uint32_t nr, const uint32_t* opk,
                      const uint64_t (*tw)[16], const uint32_t (*ta)[16], const uint32_t (*tb)[16], uint32_t (*da)[33],
                      uint32_t (*db)[33]) {
    /* sums of the words plus 7 in each field; bytes of the fields */
    uint64_t S = 7u | (uint64_t)7u << RC_NOS | (uint64_t)7u << RC_SIG;
    auto bytes = [&](uint64_t v) {
        return ((uint32_t)v << (32 - RC_NOS) >> (35 - RC_NOS)) +
               min(raw, (uint32_t)(v >> (RC_SIG + 3)) + ((uint32_t)(v >> (RC_NOS + 3)) & ((1u << (RC_SIG - RC_NOS - 3)) - 1u)));
    };
    uint32_t fb = 7, zb = 7;
#pragma unroll 4
    for (uint32_t i = b0; i < b0 + nb; i++) {
        const uint32_t w = opk[i], x = w & 255u;
        const int t = min(max(q - (int)((w >> 8) & 255u), 0), 15);
        S += tw[x][t];
        if (SB > 0) fb += ta[x][t];
        if (SB > 1) zb += tb[x][t];
    }
    auto lower = [&](uint32_t w) { /* the line's gtli drops by one */
        const uint32_t x = w & 255u;
        const int d = q - (int)((w >> 8) & 255u);
        const int t0 = min(max(d, 0), 15), t1 = min(max(d - 1, 0), 15);
        S += tw[x][t1] - tw[x][t0];
        if (SB > 0) fb += ta[x][t1] - ta[x][t0];
        if (SB > 1) zb += tb[x][t1] - tb[x][t0];
    };
    const uint32_t i0 = b0 + 4 * chunk, i1 = min(b0 + nb, i0 + 4);
    for (uint32_t i = b0; i < i0; i++) {
        const uint32_t w = opk[i];
        if ((w >> 16) >= nr) return;
        lower(w);
    }
    const uint32_t base = bytes(S);
    uint32_t c = base + (SB > 0 ? fb >> 3 : 0u), cf = base + (zb >> 3);
    if (chunk == 0) {
        atomicAdd(&da[q][0], c);
        if (SB > 1) atomicAdd(&db[q][0], cf);
    }
    uint32_t w = opk[i0];
    for (uint32_t i = i0; i < i1; i++) {
        const uint32_t rf = w >> 16; /* the first R at which it has dropped */
        if (rf >= nr) break;
        lower(w);
        w = opk[i + 1]; /* the next line's before its turn */
        const uint32_t base1 = bytes(S), c1 = base1 + (SB > 0 ? fb >> 3 : 0u), cf1 = base1 + (zb >> 3);
        atomicAdd(&da[q][rf], c1 - c);
        if (SB > 1) atomicAdd(&db[q][rf], cf1 - cf);
        c = c1;
        cf = cf1;
    }
}
/* What packet_costs reads of the precinct kind's tables: the order's lines, and
 * the packets' chunks (packet | chunk << 8, their number last).  By a block. */
#define RC_MAXITEM (JXS_MAXBLINES / 4 + JXS_MAXPK)
DEV void cost_items(uint32_t nbl, uint32_t npk, const uint8_t* order, const uint8_t* gain, const uint8_t* prio, const uint8_t* pknbl,
                    uint32_t* opk, uint16_t* items) {
    for (uint32_t x = threadIdx.x; x < nbl; x += blockDim.x) {
        const uint32_t y = order[x];
        opk[x] = y | (uint32_t)gain[y] << 8 | (prio[y] + 1u) << 16;
    }
    if ((threadIdx.x >> 5) == RC_WARPS - 1) {
        const uint32_t lane = threadIdx.x & 31, n = lane < npk ? (pknbl[lane] + 3u) >> 2 : 0u;
        uint32_t e = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, e, o);
            if (lane >= (uint32_t)o) e += y;
        }
        for (uint32_t c = 0; c < n; c++) items[e - n + c] = (uint16_t)(lane | c << 8);
        if (lane == 31) items[RC_MAXITEM] = (uint16_t)e;
    }
}

/* One slice's selection with vertical prediction, precinct after precinct
 * (the costs of a row depend on the gtli chosen for the row above,
 * RateControl.c:586-676), by the block that completes the slice.  Per
 * precinct:
 *   tables   its line tables and (fast-sign) cost tables from the other
 *            blocks;
 *   vpred    warp per segment: for every gtli t, the unary bits of each
 *            GCLI coded from the line above (line 0: the band's last line
 *            in the row above, with that row's gtli) and the bits the
 *            significance groups without code save (run mode Rm: groups
 *            with every GCLI <= t; else groups predicted exactly);
 *   methods  per band and t: no significance, significance, prediction,
 *            prediction with significance; a later one only if strictly
 *            cheaper;
 *   costs    as in the parallel pass, with those methods and exact signs
 *            for the full strategy;
 *   search   warp 0: quantization on the plain table, then the scan and
 *            refinement on the prediction table (:909-1083).
 * A chain of a slice's precincts with few blocks at work, bound by the vpred
 * part.  Two GCLIs to an instruction and two gtli values to a warp, with the
 * coding choice as minima and maxima, take it from 65,000 to 18,000 cycles
 * per precinct (1279x717 4:4:4), the costs by a warp per packet from 13,000
 * to 5,500; the kernel from 231 to 102 us, 88 us with what came after (gtli
 * values above every GCLI without the loop, costs by chunks of lines).  Two
 * blocks per SM: with registers for three (40) the loop spilled (114 us
 * against 102). */
template <typename Stage>
DEV void select_slice_vpred(const jxs_cfg_t* __restrict__ cfg, const SliceInfo& I, int s, const uint8_t* gcli,
                            const uint32_t* cost, uint32_t* area, PrecRC* rc,
                            int* status, Stage& stage_kind, const uint8_t* lgain, const uint8_t* lprio,
                            const uint8_t* lfb, const uint32_t* lsig, const uint32_t* lraw, const jxs_bline_t* bls,
                            const jxs_seg_t* segs, const uint8_t* s_pkbl0, const uint8_t* s_pknbl, const uint8_t* s_order, uint32_t* opk,
                            uint16_t* items) {
    __shared__ int s_err;
    __shared__ uint8_t s_gtop[JXS_MAXBL], s_bl0[JXS_MAXBL], s_bl1[JXS_MAXBL];
    uint32_t(*vtfs)[16] = (uint32_t(*)[16])area;
    uint32_t(*dV)[33] = (uint32_t(*)[33])(area + RC_LT_REGION);
    static_assert(32 * 33 <= RC_LT_REGION, "rows of 33 words: a lane per Q adds at one R");
    uint32_t(*vtdat)[16] = (uint32_t(*)[16])(area + 2 * RC_LT_REGION);
    uint32_t(*vtnos)[16] = (uint32_t(*)[16])(area + 3 * RC_LT_REGION);
    uint32_t(*vtsig)[16] = (uint32_t(*)[16])(area + 4 * RC_LT_REGION);
    uint32_t(*vtnz)[16] = (uint32_t(*)[16])(area + 5 * RC_LT_REGION);
    uint32_t(*vnos)[16] = (uint32_t(*)[16])(area + 6 * RC_LT_REGION);
    uint32_t(*vred)[16] = (uint32_t(*)[16])(area + 7 * RC_LT_REGION);
    uint32_t* Ts = area + 8 * RC_LT_REGION;
    uint32_t* Fs = area + 9 * RC_LT_REGION;
    uint64_t(*tw)[16] = (uint64_t(*)[16])(area + 10 * RC_LT_REGION);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = lane >> 4;
    RcParams P = I.P;
    P.empty = I.empty[threadIdx.x & 31];
    const SliceSplit sp = I.sp;
    uint32_t carry = 0, run = I.begin; /* of warp 0 */
    if (threadIdx.x == 0) s_err = 0;
    const int nq = cfg->max_q + 1, nr = cfg->max_r + 1, nt = nq * nr;
    const uint32_t np_all = cfg->np, signs = cfg->signs, fs = cfg->fs, SG = cfg->seg_groups, npk = cfg->npk;
    const uint32_t nbands = cfg->nbands, sig = cfg->sig;
    const int rm = cfg->rm;
    uint32_t(*vtz)[16] = signs == 2 ? vtnz : vtfs; /* sign bits */
    __syncthreads();
    if (P.rc_mode >= 2 && slice_common(P, s, sp, cost, Ts, rc, status)) return;
    int kind_staged = -1;
    for (uint32_t i = 0; i < sp.nprec; i++) {
        const uint32_t p = sp.first_p + i;
        const int kind = (p + 1 >= np_all);
        __syncthreads();
        if (s_err) break;
        if (kind != kind_staged) {
            stage_kind(kind);
            kind_staged = kind;
            __syncthreads();
        }
        const uint32_t nbl = cfg->nbline[kind], nseg = cfg->nseg[kind];
        /* the lines of each band (at most two per precinct row) */
        for (uint32_t fb = threadIdx.x; fb < nbands; fb += blockDim.x) {
            s_bl0[fb] = 0xff;
            s_bl1[fb] = 0xff;
        }
        __syncthreads();
        for (uint32_t x = threadIdx.x; x < nbl; x += blockDim.x) {
            if (bls[x].line == 0) s_bl0[bls[x].fb] = (uint8_t)x;
            else s_bl1[bls[x].fb] = (uint8_t)x;
        }
        /* this row's tables from the other blocks */
        const uint32_t* lt = cost + (uint64_t)np_all * 1024 * (fs ? 2 : 1) + (uint64_t)p * RC_LT_WORDS;
        for (uint32_t k = threadIdx.x; k < nbl * 16; k += blockDim.x) {
            const uint32_t x = k >> 4, t = k & 15;
            vtdat[x][t] = __ldcg(lt + k);
            vtnos[x][t] = __ldcg(lt + RC_LT_REGION + k);
            vtsig[x][t] = __ldcg(lt + 2 * RC_LT_REGION + k);
            if (fs) {
                vtfs[x][t] = __ldcg(lt + 3 * RC_LT_REGION + k);
                vtnz[x][t] = __ldcg(lt + 4 * RC_LT_REGION + k);
            }
            vnos[x][t] = 0;
            vred[x][t] = 0;
        }
        for (int e = threadIdx.x; e < nt; e += blockDim.x) {
            const int q = e / nr, r = e - q * nr;
            Ts[e] = __ldcg(cost + (uint64_t)p * 1024 + q * 32 + r);
            if (fs) Fs[e] = __ldcg(cost + ((uint64_t)np_all + p) * 1024 + q * 32 + r);
        }
        for (int e = threadIdx.x; e < nq * 33; e += blockDim.x) (&dV[0][0])[e] = 0;
        cost_items(nbl, npk, s_order, lgain, lprio, s_pknbl, opk, items);
        __syncthreads();
        /* vertical prediction costs of every line, for every t */
        if (i > 0) {
            for (uint32_t sidx = warp; sidx < nseg; sidx += RC_WARPS) {
                const jxs_seg_t sg = segs[sidx];
                const uint32_t x = sg.bl;
                const jxs_bline_t B = bls[x];
                const jxs_band_t& bd = cfg->band[B.fb];
                const uint8_t* cur = gcli + bd.gcli_off + (uint64_t)(p * bd.lines + B.line) * bd.gpitch;
                const uint8_t* top = cur - bd.gpitch; /* the row above: the previous line, for line 0 in the row above */
                const int gtt = B.line ? -1 : (int)s_gtop[B.fb];
                const uint32_t gend = min(sg.g0 + SG, B.gcli_w);
                uint32_t acc = 0; /* lane t: bits at t; lane 16 + t: those that significance groups save */
                for (uint32_t base = sg.g0; base < gend; base += 128) {
                    /* a significance group of 8 GCLIs per lane, in both
                     * halves of the warp; pairs of GCLIs in 16-bit halves */
                    const uint32_t g = base + 8 * (lane & 15);
                    const uint32_t nv = g < gend ? min(8u, gend - g) : 0u;
                    const uint32_t E = 0x00ff00ffu;
                    uint32_t wc[2] = {0, 0}, wt[2] = {0, 0}, c[4], tp[4], pv[4], kc = 0;
                    if (nv) {
                        wc[0] = *(const uint32_t*)(cur + g);
                        wt[0] = *(const uint32_t*)(top + g);
                    }
                    if (nv > 4) {
                        wc[1] = *(const uint32_t*)(cur + g + 4);
                        wt[1] = *(const uint32_t*)(top + g + 4);
                    }
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int n = min(max((int)nv - 4 * (k >> 1), 0), 4), sh = 8 * (k & 1);
                        const uint32_t vm = n == 4 ? 0xffffffffu : (1u << (8 * n)) - 1u;
                        pv[k] = ((vm >> sh) & E) * 0x101u;
                        c[k] = (wc[k >> 1] >> sh) & E & pv[k];
                        tp[k] = (wt[k >> 1] >> sh) & E;
                        kc += (VP_K - VP_ONE) & pv[k];
                    }
                    uint32_t m8 = __vmaxu2(__vmaxu2(c[0], c[1]), __vmaxu2(c[2], c[3]));
                    m8 = max(m8 & 0xffffu, m8 >> 16);
                    /* from the largest GCLI of both rows on, every GCLI is at t
                     * and its prediction at max(t, gtt): without the loop */
                    uint32_t top8 = __vmaxu2(__vmaxu2(tp[0] & pv[0], tp[1] & pv[1]), __vmaxu2(tp[2] & pv[2], tp[3] & pv[3]));
                    top8 = max(m8, max(top8 & 0xffffu, top8 >> 16));
                    const int its = (int)min((__reduce_max_sync(FULL, top8) + 1) >> 1, 8u);
                    {
                        const int t = lane & 15, G = max(t, gtt);
                        const uint32_t n = min(128u, gend - base);
                        const uint32_t bits = G == t ? n : 2u * (uint32_t)(G - t) * n;
                        if (t >= 2 * its) acc += lane < 16 || rm ? bits : G == t ? n : 0u;
                    }
#pragma unroll 2
                    for (int it = 0; it < its; it++) {
                        const int t = 2 * it + half;
                        const uint32_t t2 = t * VP_ONE, G2 = max(t, gtt) * VP_ONE;
                        uint32_t sum = 0, off = 0;
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            uint32_t x;
                            sum += vp_codes(c[k], tp[k], t2, G2, &x) & pv[k];
                            off |= x & pv[k];
                        }
                        sum -= kc; /* and the code's closing zero */
                        sum = (sum & 0xffffu) + (sum >> 16);
                        const uint32_t red = (rm ? m8 <= (uint32_t)t : off == 0) ? sum : 0u;
                        const uint32_t a = __reduce_add_sync(FULL, sum << (16 * half)), b = __reduce_add_sync(FULL, red << (16 * half));
                        if (((lane & 15) >> 1) == it) acc += ((lane < 16 ? a : b) >> (16 * (lane & 1))) & 0xffffu;
                    }
                }
                if (acc) atomicAdd(lane < 16 ? &vnos[x][lane] : &vred[x][lane - 16], acc);
            }
        }
        __syncthreads();
        /* coding method per band and t (RateControl.c:526-676) */
        for (uint32_t e = threadIdx.x; e < nbands * 16; e += blockDim.x) {
            const uint32_t fb = e >> 4, t = e & 15;
            const uint32_t x0 = s_bl0[fb], x1 = s_bl1[fb];
            if (x0 == 0xff) continue;
            const bool two = x1 != 0xff;
            uint32_t cnv = vtnos[x0][t], csv = vtsig[x0][t] + lsig[x0], vn = vnos[x0][t], vs = vnos[x0][t] - vred[x0][t] + lsig[x0];
            if (two) {
                cnv += vtnos[x1][t];
                csv += vtsig[x1][t] + lsig[x1];
                vn += vnos[x1][t];
                vs += vnos[x1][t] - vred[x1][t] + lsig[x1];
            }
            uint32_t m = 0, best = cnv;
            if (sig && best > csv) {
                m = 2;
                best = csv;
            }
            if (i > 0) {
                if (best > vn) {
                    m = 1;
                    best = vn;
                }
                if (sig && best > vs) m = 3;
            }
            for (uint32_t x = x0, k = 0; k < (two ? 2u : 1u); x = x1, k++) {
                const uint32_t bits = m == 0 ? vtnos[x][t] : m == 2 ? vtsig[x][t] : vnos[x][t] - (m == 3 ? vred[x][t] : 0u);
                tw[x][t] = vtdat[x][t] | (uint64_t)bits << RC_NOS | (uint64_t)(m & 2u ? lsig[x] : 0u) << RC_SIG;
            }
        }
        __syncthreads();
        /* costs with those methods, as in the parallel pass */
        for (uint32_t it = warp; it < items[RC_MAXITEM]; it += RC_WARPS) {
            const uint32_t e = items[it], k = e & 255u;
            if (lane >= nq) continue;
            if (signs) packet_costs<1>(lane, e >> 8, s_pkbl0[k], s_pknbl[k], lraw[k], nr, opk, tw, vtz, nullptr, dV, nullptr);
            else packet_costs<0>(lane, e >> 8, s_pkbl0[k], s_pknbl[k], lraw[k], nr, opk, tw, nullptr, nullptr, dV, nullptr);
        }
        __syncthreads();
        for (int q = warp; q < nq; q += RC_WARPS) {
            uint32_t c = dV[q][lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, c, o);
                if (lane >= o) c += y;
            }
            dV[q][lane] = c;
        }
        __syncthreads();
        if (warp == 0) {
            int q, r;
            const int err = prec_select(P, s, i, sp, Ts, fs ? Fs : Ts, nr, &dV[0][0], 33, 1, carry, run, q, r, rc, status);
            if (err) {
                if (lane == 0) s_err = err;
            } else {
                for (uint32_t fb = lane; fb < nbands; fb += 32)
                    s_gtop[fb] = jxs_truncation(cfg->band[fb].gain, cfg->band[fb].prio, (uint8_t)q, (uint8_t)r);
            }
        }
    }
}

/* Number of gtli values t (from 0 up) at which a coefficient of magnitude m
 * in a group with GCLI g stays non-zero after quantization
 * (rate_control_lut_fill, RateControl.c:124-137, and
 * rate_control_sign_coding_get_sum_nonzero_coeff_c, :366-455): the bits of
 * m for deadzone quantization; for uniform quantization the value
 * ((m << (g - t + 1)) - m + 2^g) >> (g + 1) falls as t grows and is non-zero
 * while m (2^(g-t+1) - 1) >= 2^g, which for m of b <= g bits holds at
 * t = b - 1, never at t = b + 1. */
DEV uint32_t nz_levels(uint32_t m, uint32_t g, uint32_t uniform) {
    const uint32_t b = 32u - __clz(m);
    return b + (uniform && (m << (g - b + 1u)) - m >= (1u << g));
}

/* Byte cost of every (quantization, refinement) candidate of one precinct
 * row: rate_control_lut_fill, rate_control_calculate_band_best_method and
 * precinct_get_budget_bytes (RateControl.c:18-154, 457-781).
 *   histograms  warp per segment: GCLI histogram of every band line
 *               (warp-aggregated shared atomics) and the line's groups by
 *               the maximum GCLI of their significance group; each segment's
 *               own two histograms also go to device memory for packing
 *               (segments of at most 128 groups);
 *   tables      thread per band line: for every gtli t, data bits, GCLI bits
 *               without significance and with it (suffix sums over the
 *               histogram); per band, significance coding at t only if
 *               strictly cheaper over all its lines;
 *   costs       per packet, data / significance / GCLI bytes rounded
 *               separately, raw fallback when cheaper; summed over packets
 *               for every (Q, R). */
/* a << n, 0 for n >= 32 (the machine's shift, for which C++ has no
 * expression without a comparison) */
DEV uint32_t shl_or_0(uint32_t a, uint32_t n) {
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(n));
    return r;
}

template <bool SIGNS, bool VPRED>
__device__ __forceinline__ void rc_cost_body(const jxs_cfg_t* __restrict__ cfg, const uint8_t* gcli,
                                             const uint16_t* coef, uint32_t* cost,
                                             uint32_t* slice_done, PrecRC* rc,
                                             int* status, const int p) {
    /* per band line: GCLI and significance-maximum histograms (with sign
     * handling also the coefficients by non-zero levels), then per gtli data
     * / GCLI bits without and with significance and the sign bits; the area
     * is reused by the slice selection at the end (with vertical prediction
     * it is dynamic shared memory of RC_VP_REGIONS regions) */
    __shared__ __align__(16) uint32_t s_area_st[VPRED ? 4 : RC_AREA_WORDS(SIGNS)];
    extern __shared__ __align__(16) uint32_t rc_dyn[];
    uint32_t* s_area = VPRED ? rc_dyn : s_area_st;
    uint32_t(*hist)[16] = (uint32_t(*)[16])s_area;                          /* later: fast sign bits per t */
    uint32_t(*shist)[16] = (uint32_t(*)[16])(s_area + JXS_MAXBLINES * 16);  /* groups by significance-group maximum; later: full-sign cost changes */
    uint32_t(*tdat)[16] = (uint32_t(*)[16])(s_area + 2 * JXS_MAXBLINES * 16);
    uint32_t(*tnos)[16] = (uint32_t(*)[16])(s_area + 3 * JXS_MAXBLINES * 16);
    uint32_t(*tsig)[16] = (uint32_t(*)[16])(s_area + 4 * JXS_MAXBLINES * 16);
    uint32_t(*nzh)[16] = (uint32_t(*)[16])(s_area + (SIGNS ? 5 : 0) * JXS_MAXBLINES * 16); /* later: full sign bits per t */
    uint32_t(*tfs)[16] = hist;
    uint32_t(*tnz)[16] = nzh;
    uint32_t(*dF)[33] = (uint32_t(*)[33])shist;
    /* SIGNS: the launch may hold frames with sign handling; VPRED: with
     * vertical prediction (compiled out otherwise) */
    const uint32_t fs = SIGNS ? cfg->fs : 0u, uniform = cfg->qpih;
    __shared__ uint32_t cn[JXS_MAXBL][16], cs[JXS_MAXBL][16];
    __shared__ uint8_t lgain[JXS_MAXBLINES], lprio[JXS_MAXBLINES], lfb[JXS_MAXBLINES];
    __shared__ uint32_t lsig[JXS_MAXBLINES], lraw[JXS_MAXPK];
    /* per Q: cost at R = 0, then its changes at each R; rows of 33 words, a
     * lane per Q adds at one R (rows of 32 would put all lanes in one bank) */
    __shared__ uint32_t dC[32][33];
    /* this precinct kind's tables, staged from the configuration */
    __shared__ jxs_seg_t s_seg[JXS_MAXSEG];
    __shared__ jxs_bline_t s_bl[JXS_MAXBLINES];
    __shared__ uint64_t s_grow[JXS_MAXBLINES];
    __shared__ uint8_t s_pkbl0[JXS_MAXPK], s_pknbl[JXS_MAXPK], s_order[JXS_MAXBLINES];
    __shared__ uint32_t s_opk[JXS_MAXBLINES + 1]; /* the order's lines: number | gain << 8 | first R that lowers its gtli << 16 */
    __shared__ uint16_t s_item[RC_MAXITEM + 1];
    uint64_t(*tw)[16] = (uint64_t(*)[16])(s_area + (SIGNS ? 2 : 0) * JXS_MAXBLINES * 16); /* in place of hist and shist, or tdat and tnos */

    const int last = (p + 1 >= (int)cfg->np);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t nbl = cfg->nbline[last], nseg = cfg->nseg[last], SG = cfg->seg_groups;
    const jxs_bline_t* bls = s_bl;
    const jxs_seg_t* segs = s_seg;
    /* the tables of a precinct kind (normal / last row) */
    auto stage_kind = [&](int kind) {
        const uint32_t nb = cfg->nbline[kind], ns = cfg->nseg[kind];
        for (uint32_t i = threadIdx.x; i < ns * (sizeof(jxs_seg_t) / 4); i += blockDim.x)
            ((uint32_t*)s_seg)[i] = ((const uint32_t*)cfg->seg[kind])[i];
        for (uint32_t i = threadIdx.x; i < nb * (sizeof(jxs_bline_t) / 4); i += blockDim.x)
            ((uint32_t*)s_bl)[i] = ((const uint32_t*)cfg->bline[kind])[i];
        for (uint32_t k = threadIdx.x; k < cfg->npk; k += blockDim.x) {
            s_pkbl0[k] = cfg->pk_bl0[kind][k];
            s_pknbl[k] = cfg->pk_nbl[kind][k];
            lraw[k] = cfg->raw_bytes[kind][k];
        }
        for (uint32_t x = threadIdx.x; x < nb; x += blockDim.x) {
            const jxs_bline_t& B = cfg->bline[kind][x];
            const jxs_band_t& bd = cfg->band[B.fb];
            lgain[x] = bd.gain;
            lprio[x] = bd.prio;
            lfb[x] = B.fb;
            lsig[x] = B.sig_w;
            s_order[x] = cfg->pk_order[kind][x];
        }
    };
    __shared__ SliceInfo s_info;
    if (warp == RC_WARPS - 1) slice_info(cfg, (int)((uint32_t)p / cfg->pps), &s_info);
    stage_kind(last);
    for (uint32_t i = threadIdx.x; i < nbl * 16; i += blockDim.x) {
        hist[i >> 4][i & 15] = 0;
        shist[i >> 4][i & 15] = 0;
        if (SIGNS) nzh[i >> 4][i & 15] = 0;
    }
    for (uint32_t i = threadIdx.x; i < cfg->nbands * 16; i += blockDim.x) {
        cn[i >> 4][i & 15] = 0;
        cs[i >> 4][i & 15] = 0;
    }
    for (uint32_t x = threadIdx.x; x < nbl; x += blockDim.x) {
        const jxs_bline_t& B = cfg->bline[last][x];
        const jxs_band_t& bd = cfg->band[B.fb];
        s_grow[x] = bd.gcli_off + (uint64_t)(p * bd.lines + B.line) * bd.gpitch;
    }
    dep_wait(); /* up to here configuration only */
    __syncthreads();

    /* histograms: each lane 4 consecutive groups (one 4-byte load) in 4-bit
     * counters, one per GCLI value (at most 4, or 8 for a significance
     * group's weight), values 0..7 in one word and 8..15 in another, each
     * counter reached by a shift that gives 0 past the word; widened to
     * bytes and summed over the warp per 128 groups (at most 128 per bin);
     * then lane b < 16 holds the count of GCLI b and lane 16 + b that of
     * significance-group maximum b, adds it to the band line's histogram
     * and, for a segment of at most 128 groups, stores it as byte b / 16 + b
     * of the segment's histograms for packing.  Groups without a GCLI of 8 or
     * more skip the upper word.  Bound by instruction issue: 58 warp
     * instructions per 128 groups fewer than counters picked by comparisons and
     * 8-byte maxima (8 4K frames: 143 -> 132 us). */
    uint32_t* seghist = cost + jxs_seghist_word(cfg) + (uint64_t)p * jxs_seg_cap(cfg) * JXS_SEGHIST_WORDS;
    static_assert(JXS_SEGHIST_WORDS * 4 == 32, "a segment's histograms: one byte per lane");
    const bool export_hist = SG <= 128;
    /* this lane's bin: byte (b >> 1) & 3 of word 2 (b >= 8) + (b & 1) of the
     * value (lanes 0..15) or significance (16..31) words */
    const uint32_t hb = lane & 15u, hsh = 8u * ((hb >> 1) & 3u);
    uint32_t* htab = (lane < 16 ? &hist[0][0] : &shist[0][0]) + hb;
    for (uint32_t sidx = warp; sidx < nseg; sidx += RC_WARPS) {
        const jxs_seg_t sg = segs[sidx];
        const uint32_t x = sg.bl;
        const uint8_t* grow = gcli + s_grow[x];
        const uint32_t gend = min(sg.g0 + SG, bls[x].gcli_w);
        const uint16_t* crow = nullptr;
        if (fs) {
            const jxs_band_t& bd = cfg->band[lfb[x]];
            crow = coef + bd.coef_off + (uint64_t)(p * bd.lines + bls[x].line) * bd.pitch;
        }
        for (uint32_t base = sg.g0; base < gend; base += 128) {
            const uint32_t g = base + 4 * lane;
            const uint32_t nv = g < gend ? min(4u, gend - g) : 0u;
            uint32_t w4 = nv ? *(const uint32_t*)(grow + g) : 0u;
            /* GCLIs past the line's end read as 0 and are taken off bin 0 */
            w4 &= nv >= 4 ? 0xffffffffu : (1u << (8 * nv)) - 1u;
            /* significance group: 8 groups in lanes 2i, 2i+1; its groups
             * (8, or fewer at the end of a line) counted at its maximum */
            uint32_t m = __vmaxu2(w4 & 0x00ff00ffu, (w4 >> 8) & 0x00ff00ffu);
            m = __vmaxu2(m, m >> 16);
            const uint32_t mx = __vmaxu2(m, __shfl_xor_sync(FULL, m, 1)) & 255u;
            const uint32_t left = gend - base; /* groups of the segment from base on */
            const uint32_t nvp = (lane & 1) || g >= gend ? 0u : min(8u, left - 4 * lane);
            /* 4 GCLI per byte */
            const uint32_t a4 = 4u * w4;
            const uint32_t M = 0x0f0f0f0fu;
            const uint32_t lo = nv - 4u + shl_or_0(1u, a4 & 255u) + shl_or_0(1u, __byte_perm(a4, 0u, 0x4441)) +
                                shl_or_0(1u, __byte_perm(a4, 0u, 0x4442)) + shl_or_0(1u, a4 >> 24); /* bin 0 starts at -(4 - nv) */
            const uint32_t slo = shl_or_0(nvp, 4u * mx);
            const uint32_t v0 = __reduce_add_sync(FULL, lo & M), v1 = __reduce_add_sync(FULL, (lo >> 4) & M);
            const uint32_t s0 = __reduce_add_sync(FULL, slo & M), s1 = __reduce_add_sync(FULL, (slo >> 4) & M);
            const uint32_t even = lane < 16 ? v0 : s0, odd = lane < 16 ? v1 : s1;
            uint32_t word = hb >= 8 ? 0u : hb & 1 ? odd : even;
            if (__any_sync(FULL, w4 & 0x08080808u)) {
                /* the same for values 8..15 (shifts less 32) */
                const uint32_t b4 = a4 ^ 0x20202020u; /* 4 v - 32 per byte, 32 or more below 8 */
                const uint32_t hi = shl_or_0(1u, b4 & 255u) + shl_or_0(1u, __byte_perm(b4, 0u, 0x4441)) +
                                    shl_or_0(1u, __byte_perm(b4, 0u, 0x4442)) + shl_or_0(1u, b4 >> 24);
                const uint32_t shi = shl_or_0(nvp, 4u * mx - 32u);
                const uint32_t v2 = __reduce_add_sync(FULL, hi & M), v3 = __reduce_add_sync(FULL, (hi >> 4) & M);
                const uint32_t s2 = __reduce_add_sync(FULL, shi & M), s3 = __reduce_add_sync(FULL, (shi >> 4) & M);
                if (hb >= 8) word = lane < 16 ? (hb & 1 ? v3 : v2) : (hb & 1 ? s3 : s2);
            }
            const uint32_t c = (word >> hsh) & 255u;
            if (c) atomicAdd(htab + 16 * x, c);
            if (export_hist) ((uint8_t*)(seghist + sidx * JXS_SEGHIST_WORDS))[lane] = (uint8_t)c;
            if (fs) {
                /* sign handling: the lane's 16 coefficients (inside the band
                 * width) by the number of gtli values at which they stay
                 * non-zero, counted like the GCLIs, 8 coefficients to 4-bit
                 * counters and 16 to 8-bit ones, by a loop per quantizer
                 * (8 4K frames with signs: 0.096 -> 0.094 ms each) */
                uint4 c0 = make_uint4(0, 0, 0, 0), c1 = c0;
                if (nv) {
                    c0 = *(const uint4*)(crow + 4 * g);
                    c1 = *(const uint4*)(crow + 4 * g + 8);
                }
                uint32_t cw[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
                const int left16 = min((int)bls[x].w - 4 * (int)g, 4 * (int)nv);
                if (left16 < 16) {
#pragma unroll
                    for (int i = 0; i < 8; i++) cw[i] &= 2 * i + 1 < left16 ? 0xffffffffu : 2 * i < left16 ? 0xffffu : 0u;
                }
                const bool large = __any_sync(FULL, w4 & 0x08080808u);
                uint32_t za[4] = {0, 0, 0, 0}; /* levels 0, 2, 4, 6; 1, 3, 5, 7; the same of 8..15 */
                auto count = [&](auto uq) {
#pragma unroll
                    for (int i0 = 0; i0 < 16; i0 += 8) {
                        uint32_t zl = 0, zg = 0;
#pragma unroll
                        for (int i = i0; i < i0 + 8; i++) {
                            const uint32_t m = cw[i >> 1] >> (16 * (i & 1)) & 0x7fffu;
                            const uint32_t n = nz_levels(m, (w4 >> (8 * (i >> 2))) & 255u, decltype(uq)::value);
                            zl += shl_or_0(1u, 4 * n);
                            if (large) zg += shl_or_0(1u, 4 * n - 32u);
                        }
                        za[0] += zl & M;
                        za[1] += (zl >> 4) & M;
                        za[2] += zg & M;
                        za[3] += (zg >> 4) & M;
                    }
                };
                if (uniform) count(std::true_type());
                else count(std::false_type());
                const uint32_t M2 = 0x00ff00ffu;
                uint32_t zw = 0; /* of lane b < 16: levels b & 11 and (b & 11) + 4 in its halves */
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (i >= 2 && !large) break;
                    const uint32_t e = __reduce_add_sync(FULL, za[i] & M2), o = __reduce_add_sync(FULL, (za[i] >> 8) & M2);
                    if ((lane >> 3) == (i >> 1) && (lane & 1) == (i & 1)) zw = lane & 2 ? o : e;
                }
                const uint32_t zn = (zw >> (16 * ((lane >> 2) & 1))) & 0xffffu;
                if (lane < 16 && zn) atomicAdd(&nzh[x][lane], zn);
            }
        }
    }
    __syncthreads();

    /* per band line and gtli t: data bits, GCLI bits without / with
     * significance coding; half a warp per line, a lane per t, the sums over
     * the larger and smaller GCLIs by shuffles */
    for (uint32_t x0 = 2 * warp; x0 < nbl; x0 += 2 * RC_WARPS) {
        const uint32_t x = min(x0 + (lane >> 4), nbl - 1);
        const int t = lane & 15;
        const int h = (int)hist[x][t], th = t * h;
        const uint32_t zh = SIGNS ? nzh[x][t] : 0u;
        int S0 = h, S1 = th;
        uint32_t Z = shist[x][t], Z1 = zh;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const int a0 = __shfl_down_sync(FULL, S0, o, 16), a1 = __shfl_down_sync(FULL, S1, o, 16);
            const uint32_t az = __shfl_up_sync(FULL, Z, o, 16);
            if (t + o < 16) {
                S0 += a0;
                S1 += a1;
            }
            if (t >= o) Z += az; /* groups in significance groups whose maximum is <= t: no GCLI codes */
            if (SIGNS) {
                const uint32_t a2 = __shfl_down_sync(FULL, Z1, o, 16);
                if (t + o < 16) Z1 += a2;
            }
        }
        S0 -= h; /* over v > t */
        S1 -= th;
        const int dsum = S1 - (t - 1) * S0; /* sum over v > t of (v - t + 1) h[v] */
        if (x == x0 + (lane >> 4)) {
            /* with sign handling the data leave out the sign nibbles
             * (RateControl.c:156-210): fast signs count 4 per group above
             * t, full signs the coefficients that stay non-zero */
            const uint32_t nos = (uint32_t)dsum + bls[x].gcli_w - (uint32_t)S0, fb = lfb[x];
            tdat[x][t] = 4u * (uint32_t)(dsum - (fs ? S0 : 0));
            tnos[x][t] = nos;
            tsig[x][t] = nos - Z;
            if (SIGNS) {
                tfs[x][t] = 4u * (uint32_t)S0;
                tnz[x][t] = Z1 - zh;
            }
            atomicAdd(&cn[fb][t], nos);
            atomicAdd(&cs[fb][t], nos - Z + lsig[x]);
        }
    }
    __syncthreads();
    if (VPRED && cfg->vpred) {
        /* the line tables, for the slice's selection in precinct order */
        uint32_t* lt = cost + (uint64_t)cfg->np * 1024 * (cfg->fs ? 2 : 1) + (uint64_t)p * RC_LT_WORDS;
        for (uint32_t i = threadIdx.x; i < nbl * 16; i += blockDim.x) {
            const uint32_t x = i >> 4, t = i & 15;
            lt[i] = tdat[x][t];
            lt[RC_LT_REGION + i] = tnos[x][t];
            lt[2 * RC_LT_REGION + i] = tsig[x][t];
            if (fs) {
                lt[3 * RC_LT_REGION + i] = tfs[x][t];
                lt[4 * RC_LT_REGION + i] = tnz[x][t];
            }
        }
    }
    /* coding method per band and t: significance only if strictly cheaper
     * (RateControl.c:528-575).  Per line and t one word: data bits, from bit
     * RC_NOS the GCLI bits of the method chosen, from bit RC_SIG its
     * significance flags; a packet's sums stay within these fields, at most
     * 4 * 16384 groups of 64 data and 16 GCLI bits */
    const int nq = cfg->max_q + 1, nr = cfg->max_r + 1;
    const uint32_t sig = cfg->sig;
    static_assert(JXS_MAXBLINES * 16 <= 3 * RC_THREADS, "three words per thread");
    uint64_t word[3] = {0, 0, 0};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint32_t i = threadIdx.x + k * RC_THREADS, x = i >> 4, t = i & 15;
        if (i < nbl * 16) {
            const uint32_t fb = lfb[x];
            const bool m = sig && cn[fb][t] > cs[fb][t];
            word[k] = tdat[x][t] | (uint64_t)(m ? tsig[x][t] : tnos[x][t]) << RC_NOS | (uint64_t)(m ? lsig[x] : 0u) << RC_SIG;
        }
    }
    if (SIGNS) __syncthreads(); /* the words take the place of tdat and tnos */
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint32_t i = threadIdx.x + k * RC_THREADS;
        if (i < nbl * 16) tw[i >> 4][i & 15] = word[k];
    }
    cost_items(nbl, cfg->npk, s_order, lgain, lprio, s_pknbl, s_opk, s_item);
    /* costs: band priorities are distinct, so raising R by one lowers the
     * gtli of one band only; each (Q, packet) thread adds its packet's cost
     * at R = 0 and its change at every R where one of its band lines drops,
     * and the table is a prefix sum over R */
    if (SIGNS) __syncthreads(); /* dF takes the place of shist */
    for (int e = threadIdx.x; e < nq * 33; e += blockDim.x) {
        (&dC[0][0])[e] = 0;
        if (SIGNS) (&dF[0][0])[e] = 0;
    }
    __syncthreads();
    /* with sign handling each packet adds its sign sub-packet, rounded on
     * its own: fast signs in dC, full signs in dF (RateControl.c:745-756) */
    /* a warp per packet's chunk, a lane per Q (at most 32) */
    for (uint32_t it = warp; it < s_item[RC_MAXITEM]; it += RC_WARPS) {
        const uint32_t e = s_item[it], k = e & 255u;
        if (lane >= nq) continue;
        if (SIGNS && fs) packet_costs<2>(lane, e >> 8, s_pkbl0[k], s_pknbl[k], lraw[k], nr, s_opk, tw, tfs, tnz, dC, dF);
        else packet_costs<0>(lane, e >> 8, s_pkbl0[k], s_pknbl[k], lraw[k], nr, s_opk, tw, nullptr, nullptr, dC, nullptr);
    }
    __syncthreads();
    /* a warp per Q, a lane per R */
    uint32_t* out = cost + (uint64_t)p * 32 * 32;
    uint32_t* outf = cost + ((uint64_t)cfg->np + p) * 32 * 32;
    for (int q = warp; q < nq; q += RC_WARPS) {
        uint32_t c = dC[q][lane], f = SIGNS && fs ? dF[q][lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, c, o);
            if (lane >= o) c += y;
            if (SIGNS) {
                const uint32_t yf = __shfl_up_sync(FULL, f, o);
                if (lane >= o) f += yf;
            }
        }
        if (lane < nr) {
            out[q * 32 + lane] = c;
            if (SIGNS && fs) outf[q * 32 + lane] = f;
        }
    }
    /* the block that completes a slice runs the slice's selection: tables
     * published with a fence, blocks counted per slice */
    __shared__ int s_last;
    __syncthreads();
    const uint32_t s = (uint32_t)p / cfg->pps, nprec = s_info.sp.nprec;
    if (threadIdx.x == 0) {
        __threadfence(); /* the block's writes, ordered before by the barrier */
        s_last = atomicAdd(&slice_done[s], 1u) + 1 == nprec;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    if constexpr (VPRED) {
        if (cfg->vpred) select_slice_vpred(cfg, s_info, (int)s, gcli, cost, s_area, rc, status, stage_kind, lgain, lprio, lfb, lsig,
                                           lraw, s_bl, s_seg, s_pkbl0, s_pknbl, s_order, s_opk, s_item);
        else select_slice(s_info, (int)s, cost, s_area, RC_VP_REGIONS * RC_LT_REGION, rc, status);
    } else {
        select_slice(s_info, (int)s, cost, s_area, RC_AREA_WORDS(SIGNS), rc, status);
    }
    if (threadIdx.x == 0) slice_done[s] = 0; /* ready for the next frame */
}

/* ------------------------------------------------------------------------ */
/* Packing                                                                   */
/* ------------------------------------------------------------------------ */
#define PK_THREADS 512
#define PK_WARPS (PK_THREADS / 32)

/* Next entry of a block's shared work queue for a warp. */
__device__ __forceinline__ uint32_t queue_next(uint32_t* ctr, int lane) {
    uint32_t v = 0;
    if (lane == 0) v = atomicAdd(ctr, 1u);
    return __shfl_sync(0xffffffffu, v, 0);
}

/* The precinct being packed is a bit string in 32-bit words, first bit in
 * the most significant position; its bytes are swapped when it is copied
 * out.  OR the low `n` bits (1..64) of `v` into it at bit `pos`.  Bits past
 * the buffer's `nw` words are not written and set `ovf` (the sizes would
 * disagree with the rate control). */
DEV void put_bits(uint32_t* buf, uint32_t nw, uint32_t pos, uint64_t v, uint32_t n, int& ovf) {
    if (((pos + n - 1) >> 5) >= nw) {
        ovf = 1;
        return;
    }
    const uint64_t a = v << (64 - n); /* left-aligned */
    const uint32_t hi = (uint32_t)(a >> 32), lo = (uint32_t)a;
    const uint32_t w = pos >> 5, sh = pos & 31;
    atomicOr(&buf[w], hi >> sh);
    if (sh + n > 32) atomicOr(&buf[w + 1], __funnelshift_r(lo, hi, sh));
    if (sh + n > 64) atomicOr(&buf[w + 2], lo << (32 - sh));
}
/* The same for at most 32 bits, left-aligned in `a` (zeros after them), that
 * are known to lie inside the buffer. */
DEV void put_left32(uint32_t* buf, uint32_t pos, uint32_t a) {
    const uint32_t w = pos >> 5, sh = pos & 31, lo = __funnelshift_r(0u, a, sh);
    atomicOr(&buf[w], a >> sh);
    if (lo) atomicOr(&buf[w + 1], lo);
}
/* all ones in every byte whose top bit is set */
DEV uint32_t sign_bytes(uint32_t x) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %1, 0xba98;" : "=r"(r) : "r"(x));
    return r;
}
/* byte i of the bit string */
DEV uint8_t& byte_at(uint32_t* buf, uint32_t i) { return ((uint8_t*)buf)[i ^ 3u]; }

/* Inclusive sum over the lanes up to this one (the shuffle's own predicate
 * says whether there is a lane to add). */
DEV uint32_t warp_incl_scan(uint32_t x) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
        asm volatile("{.reg .u32 r; .reg .pred p; shfl.sync.up.b32 r|p, %0, %1, 0, 0xffffffff; @p add.u32 %0, %0, r;}"
                     : "+r"(x)
                     : "r"(o));
    return x;
}
DEV uint32_t warp_excl_scan(uint32_t x, uint32_t* total) {
    const uint32_t inc = warp_incl_scan(x);
    *total = __shfl_sync(FULL, inc, 31);
    return inc - x;
}

/* Inverse of the 8 x 4 bit-matrix transpose: byte 3 - c holds the 8 plane
 * bits of coefficient c; bit k of it moves to bit 4k + 3 - c (nibble k =
 * plane k, coefficient 0 in its most significant bit).  Masked delta swaps
 * of index bits (1,0), (2,1), (3,0), (4,1). */
DEV uint32_t dswap(uint32_t x, int d, uint32_t m) {
    const uint32_t t = ((x >> d) ^ x) & m;
    return x ^ t ^ (t << d);
}
DEV uint32_t coefs_to_planes(uint32_t x) {
    x = dswap(x, 1, 0x22222222u);
    x = dswap(x, 2, 0x0c0c0c0cu);
    x = dswap(x, 7, 0x00aa00aau);
    return dswap(x, 14, 0x0000ccccu);
}

/* A group's (pack_data_c, PackPrecinct.c:128-198; quantization, Quant.c:9-45,
 * is skipped for t = 0 like the reference, QuantStageProcess.c:18-31)
 * quantized magnitudes as 16-bit pairs (coefficients 0 | 1 << 16 and 2 | 3 <<
 * 16) with the sign of every coefficient that stays non-zero as
 * plane v - t, above the magnitude: one transpose then gives the sign nibble
 * and the planes.  For signs with the data and a group whose coefficients
 * past the band width are stored as zero; uq: uniform quantization, t > 0
 * (t = 0 is not quantized, and a deadzone shift by 0 is the same). */
DEV void quantize_signed(uint2 raw4, uint32_t v, uint32_t t, bool uq, uint32_t& P01, uint32_t& P23) {
    const uint32_t c01 = raw4.x, c23 = raw4.y, np = v - t;
    if (!uq) {
        const uint32_t keep = (0x7fffu >> t) * 0x00010001u;
        P01 = (c01 >> t) & keep;
        P23 = (c23 >> t) & keep;
    } else {
        uint32_t q[4];
        const uint32_t c[4] = {c01 & 0xffffu, c01 >> 16, c23 & 0xffffu, c23 >> 16};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t m = c[k] & 0x7fffu;
            const uint32_t u = (((m << (v - t + 1)) - m + (1u << v)) >> (v + 1)) & 0xffffu;
            q[k] = ((u << t) & 0xffffu) >> t;
        }
        P01 = q[0] | (q[1] << 16);
        P23 = q[2] | (q[3] << 16);
    }
    /* magnitudes stay below 2^15: adding 0x7fff sets bit 15 of the non-zero
     * ones; the sign moves to bit np (<= 15) */
    P01 |= ((P01 + 0x7fff7fffu) & c01 & 0x80008000u) >> (15 - np);
    P23 |= ((P23 + 0x7fff7fffu) & c23 & 0x80008000u) >> (15 - np);
}

/* Bits 15 and 31 where the quantized magnitudes of two coefficients are not
 * zero: under deadzone quantization m >= 2^t, under uniform quantization
 * m (2^(v-t+1) - 1) >= 2^v. */
DEV uint32_t nonzero_flags(uint32_t c, uint32_t v, uint32_t t, bool uq) {
    if (!uq) return (((c >> t) & (0x7fffu >> t) * 0x00010001u) + 0x7fff7fffu) & 0x80008000u;
    const uint32_t k = (2u << (v - t)) - 1u, least = 1u << v;
    return ((c & 0x7fffu) * k >= least ? 0x8000u : 0u) | (((c >> 16) & 0x7fffu) * k >= least ? 0x80000000u : 0u);
}

/* A segment as pass B reads it: bit positions of its first GCLI code and
 * data bit, first group and group count, gtli | method << 4 | raw << 6 | band
 * line << 8. */
struct PkSeg {
    uint32_t vpos, dpos, g0n, info;
};

/* pack_precinct (PackPrecinct.c:235-572) for one precinct row.
 *
 * The precinct is assembled in shared memory, `lead` bytes into the buffer
 * so that buffer byte i lands on the 16-byte aligned address
 * out + offset - lead + i, then copied out.  Band lines are split into
 * segments of seg_groups groups, one warp per segment:
 *   pass A  each segment's data bits, VLC bits and groups lying in
 *           insignificant significance groups, at the precinct's gtli: from
 *           the segment's histograms that the rate control stored (thread
 *           per segment), or, with sign handling, vertical prediction or
 *           segments of more than 128 groups, from the GCLIs (warp per
 *           segment);
 *   layout  band totals (thread per segment); coding method per band
 *           (significance only if strictly cheaper), running sums over the
 *           segments and lines in packet order, packet headers, raw
 *           fallback, packet positions; then each segment's positions
 *           (thread per segment): a segment's start in its sub-packet is the
 *           running sum up to it less that at its packet's first segment;
 *   pass B  each lane 4 groups: significance flags and the unary GCLI
 *           codes at positions from a warp prefix sum; the groups above
 *           gtli listed per warp, each lane then packing one listed group's
 *           data bits; everything OR-ed into the buffer.
 * SIGNS: the launch may hold frames with sign handling; VPRED: with vertical
 * prediction (both compiled out otherwise); BATCH: a launch of many frames.  With vertical prediction a
 * precinct row below another of its slice also sums, per segment, the
 * codes of its GCLIs predicted from the line above at its gtli (line 0:
 * from the row above, with that row's gtli) and the groups that need no
 * code; the layout chooses among the four codings per band like the rate
 * control (RateControl.c:526-676), and pass B writes the prediction codes
 * (pack_bitplane_count_vpred_*, PackPrecinct.c:47-74). */
template <bool SIGNS, bool VPRED, bool BATCH>
__device__ __forceinline__ void pack_body(const jxs_cfg_t* __restrict__ cfg, const uint16_t* coef,
                                          const uint8_t* gcli, const PrecRC* rc,
                                          const uint32_t* cost, uint8_t* out, uint32_t cap_words,
                                          int* status, const int p) {
    extern __shared__ __align__(16) uint32_t buf[];
    /* per segment: data bits, VLC bits, groups without codes, signs, then
     * running sums; in pass B the same words hold each warp's list of
     * significant groups */
    __shared__ uint32_t s_segw[4][JXS_MAXSEG + 4];
    uint32_t* s_data = s_segw[0];
    uint32_t* s_vlc = s_segw[1];
    uint32_t* s_zero = s_segw[2];
    uint32_t* s_nz = s_segw[3];
    static_assert(4 * JXS_MAXSEG >= 128 * PK_WARPS, "a list of 128 groups per warp");
    __shared__ __align__(16) PkSeg s_desc[JXS_MAXSEG];
    __shared__ uint32_t s_nst[SIGNS ? JXS_MAXSEG : 1];                 /* per segment: first sign bit */
    __shared__ uint8_t s_meth[JXS_MAXBL];
    __shared__ uint32_t s_cn[JXS_MAXBL], s_cs[JXS_MAXBL];
    __shared__ uint32_t s_vn[VPRED ? JXS_MAXSEG : 1], s_vr[VPRED ? JXS_MAXSEG : 1]; /* per segment: prediction bits */
    __shared__ uint32_t s_cv[VPRED ? JXS_MAXBL : 1], s_cvs[VPRED ? JXS_MAXBL : 1];   /* per band: prediction totals */
    __shared__ int8_t s_gtt[VPRED ? JXS_MAXBLINES : 1];                            /* per line: gtli of the line above (-1: this row's) */
    __shared__ uint32_t s_gp[VPRED ? JXS_MAXBLINES : 1];                           /* per line: GCLI row pitch */
    __shared__ uint32_t s_part[SIGNS ? 3 : 2][JXS_MAXSEG / 32 + 1]; /* per 32 segments: data, GCLI, sign bits, then those before */
    __shared__ uint32_t s_lsx[JXS_MAXBLINES + 1], s_lrx[JXS_MAXBLINES + 1]; /* per line: significance / raw GCLI bits before it */
    __shared__ uint32_t s_pks[JXS_MAXPK], s_pkg[JXS_MAXPK], s_pkd[JXS_MAXPK], s_pkn[JXS_MAXPK]; /* per packet: sub-packet starts less the running sums there */
    __shared__ uint8_t s_pkr[JXS_MAXPK];
    /* this precinct kind's tables, staged from the configuration */
    __shared__ jxs_seg_t s_seg[JXS_MAXSEG];
    __shared__ uint16_t s_ord[JXS_MAXSEG];                              /* work order of the segments */
    __shared__ uint32_t s_q[2];                                         /* work queues of passes A and B */
    __shared__ jxs_bline_t s_bl[JXS_MAXBLINES];
    __shared__ uint64_t s_grow[JXS_MAXBLINES], s_crow[JXS_MAXBLINES]; /* per line: GCLI / coefficient row offsets */
    __shared__ uint32_t s_sigp[JXS_MAXBLINES];                         /* per line: bit position of its significance flags */
    __shared__ uint8_t s_lt[JXS_MAXBLINES];                            /* per line: gtli */
    __shared__ uint16_t s_lgp[BATCH ? 1 : JXS_MAXBLINES];              /* per line: band gain | priority << 8 */
    __shared__ uint8_t s_pkbl0[JXS_MAXPK], s_pknbl[JXS_MAXPK];
    __shared__ uint32_t s_praw[JXS_MAXPK];
    __shared__ uint8_t s_g2f[JXS_MAXBL];                               /* global band -> flat band */
    __shared__ uint8_t s_blines[JXS_MAXBL];                            /* lines of each band in this precinct kind */
    /* configuration scalars of the layout, loaded with the tables so that the
     * single-warp layout waits on no device-memory read */
    __shared__ uint32_t s_nbands, s_nbands_all, s_npk, s_sig, s_short, s_phb, s_hdrs, s_nbl;
    __shared__ int s_ok;

    const int last = (p + 1 >= (int)cfg->np);
    const uint32_t nbl = cfg->nbline[last];
    PrecRC R;
    uint32_t total = 0, lead = 0, words = 0;
    int ovf = 0, vp = 0;
    const int rmode = VPRED ? (int)cfg->rm : 0;
    /* the precinct's record and the buffer's size; false: nothing to pack */
    auto begin = [&]() {
        R = rc[p];
        /* nothing to pack once the rate control failed somewhere in the
         * frame; the flag is read once so that the whole block takes the same
         * branch */
        if (threadIdx.x == 0) s_ok = *(volatile int*)status == 0;
        __syncthreads();
        if (!s_ok) return false;
        total = R.total_bytes;
        lead = (uint32_t)((uintptr_t)(out + R.offset) & 15);
        words = ((lead + total + 15) >> 4) << 2;
        if (words > cap_words) {
            if (threadIdx.x == 0) {
                printf("jxs pack: precinct %d needs %u words, buffer holds %u\n", p, words, cap_words);
                JXS_STATUS_SET(status, JXS_E_ENC_FRAME);
            }
            return false;
        }
        for (uint32_t i = threadIdx.x; i < words >> 2; i += blockDim.x) ((uint4*)buf)[i] = make_uint4(0u, 0u, 0u, 0u);
        /* vertical prediction applies below the first row of a slice */
        vp = VPRED && cfg->vpred && !R.first_in_slice;
        return true;
    };
    /* a line's gtli, and that of the line above where it is in the row above */
    auto line_gtli = [&](uint32_t x, uint8_t gain, uint8_t prio, uint32_t line) {
        s_lt[x] = jxs_truncation(gain, prio, R.q, R.r);
        if (VPRED) s_gtt[x] = (int8_t)(vp && line == 0 ? jxs_truncation(gain, prio, rc[p - 1].q, rc[p - 1].r) : -1);
    };
    /* BATCH: an ordinary launch, the record first; else the tables first, and
     * the record once the rate control is done */
    if (BATCH && !begin()) return;
    {
        const uint32_t ns = cfg->nseg[last];
        for (uint32_t i = threadIdx.x; i < ns * (sizeof(jxs_seg_t) / 4); i += blockDim.x)
            ((uint32_t*)s_seg)[i] = ((const uint32_t*)cfg->seg[last])[i];
        for (uint32_t i = threadIdx.x; i < nbl * (sizeof(jxs_bline_t) / 4); i += blockDim.x)
            ((uint32_t*)s_bl)[i] = ((const uint32_t*)cfg->bline[last])[i];
        for (uint32_t i = threadIdx.x; i < ns; i += blockDim.x) s_ord[i] = cfg->seg_ord[last][i];
        if (threadIdx.x < 2) s_q[threadIdx.x] = 0;
        for (uint32_t x = threadIdx.x; x < nbl; x += blockDim.x) {
            const jxs_bline_t& B = cfg->bline[last][x];
            const jxs_band_t& bd = cfg->band[B.fb];
            const uint64_t row = (uint64_t)(p * bd.lines + B.line);
            s_grow[x] = bd.gcli_off + row * bd.gpitch;
            s_crow[x] = bd.coef_off + row * bd.pitch;
            if (BATCH) line_gtli(x, bd.gain, bd.prio, B.line);
            else s_lgp[x] = (uint16_t)(bd.gain | (bd.prio << 8));
            if (VPRED) s_gp[x] = bd.gpitch;
        }
        for (uint32_t k = threadIdx.x; k < cfg->npk; k += blockDim.x) {
            s_pkbl0[k] = cfg->pk_bl0[last][k];
            s_pknbl[k] = cfg->pk_nbl[last][k];
            s_praw[k] = cfg->raw_bytes[last][k];
        }
        for (uint32_t gb = threadIdx.x; gb < cfg->nbands_all; gb += blockDim.x) s_g2f[gb] = cfg->g2f[gb];
        for (uint32_t fb = threadIdx.x; fb < cfg->nbands; fb += blockDim.x) {
            s_blines[fb] = (uint8_t)(last ? cfg->band[fb].last_lines : cfg->band[fb].lines);
            s_cn[fb] = 0;
            s_cs[fb] = 0;
            if (VPRED) {
                s_cv[fb] = 0;
                s_cvs[fb] = 0;
            }
        }
    }
    if (threadIdx.x == 0) {
        s_nbands = cfg->nbands;
        s_nbands_all = cfg->nbands_all;
        s_npk = cfg->npk;
        s_sig = cfg->sig;
        s_short = cfg->short_hdr;
        s_phb = cfg->prec_hdr_bytes;
        s_hdrs = cfg->hdrs_bytes[last];
        s_nbl = nbl;
    }
    if (!BATCH) {
        dep_wait(); /* up to here configuration only */
        if (!begin()) return;
        for (uint32_t x = threadIdx.x; x < nbl; x += blockDim.x)
            line_gtli(x, (uint8_t)(s_lgp[x] & 255u), (uint8_t)(s_lgp[x] >> 8), s_bl[x].line);
    }
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t nseg = cfg->nseg[last], SG = cfg->seg_groups;
    const jxs_seg_t* segs = s_seg;
    const jxs_bline_t* bls = s_bl;

    /* pass A: each lane 4 consecutive groups (one 4-byte GCLI load), a warp
     * 128 groups per step; with sign handling also the non-zero quantized
     * coefficients, whose signs go to the sign sub-packets */
    const uint32_t fs = SIGNS ? cfg->fs : 0u, uniform = cfg->qpih;
    if (!VPRED && !fs && SG <= 128) {
        /* from the rate control's histograms: data bits 4 (v - t + 1) and
         * codes of v - t + 1 bits for groups with GCLI v > t, 1-bit codes
         * for the others; no codes for the groups of significance groups
         * whose maximum is <= t */
        const uint32_t* hist = cost + jxs_seghist_word(cfg) + (uint64_t)p * jxs_seg_cap(cfg) * JXS_SEGHIST_WORDS;
        for (uint32_t i = threadIdx.x; i < nseg; i += blockDim.x) {
            const uint4 gh = __ldcg((const uint4*)(hist + i * JXS_SEGHIST_WORDS));
            const uint4 zh = __ldcg((const uint4*)(hist + i * JXS_SEGHIST_WORDS + 4));
            const uint32_t t = s_lt[segs[i].bl];
            const uint32_t gw[4] = {gh.x, gh.y, gh.z, gh.w}, zw[4] = {zh.x, zh.y, zh.z, zh.w};
            uint32_t d = 0, v = 0, z = 0;
#pragma unroll
            for (uint32_t b = 0; b < 16; b++) {
                const uint32_t c = (gw[b >> 2] >> (8 * (b & 3))) & 255u, cz = (zw[b >> 2] >> (8 * (b & 3))) & 255u;
                if (b > t) {
                    d += (b - t + 1) * c;
                    v += (b - t + 1) * c;
                } else {
                    v += c;
                    z += cz;
                }
            }
            s_data[i] = 4 * d;
            s_vlc[i] = v;
            s_zero[i] = z;
            s_nz[i] = 0;
        }
    } else
    for (uint32_t qi = queue_next(&s_q[0], lane); qi < nseg; qi = queue_next(&s_q[0], lane)) {
        const uint32_t sidx = s_ord[qi];
        const jxs_seg_t sg = segs[sidx];
        const uint32_t t = s_lt[sg.bl];
        const uint8_t* grow = gcli + s_grow[sg.bl];
        const uint16_t* crow = coef + s_crow[sg.bl];
        const uint32_t gend = min(sg.g0 + SG, bls[sg.bl].gcli_w);
        uint32_t dsum = 0, vsum = 0, zsum = 0, nsum = 0, pnsum = 0, prsum = 0;
        for (uint32_t base = sg.g0; base < gend; base += 128) {
            const uint32_t g = base + 4 * lane;
            const uint32_t nv = g < gend ? min(4u, gend - g) : 0u;
            const uint32_t keep = nv >= 4 ? 0xffffffffu : (1u << (8 * nv)) - 1u;
            const uint32_t w4 = nv ? *(const uint32_t*)(grow + g) & keep : 0u;
            if (VPRED && vp) {
                /* GCLIs predicted from the line above: code bits, and the
                 * groups of 8 that need none (lanes 2j, 2j + 1) */
                const uint32_t wt = nv ? *(const uint32_t*)(grow - s_gp[sg.bl] + g) : 0u;
                const uint32_t t2 = t * VP_ONE, G2 = (uint32_t)max((int)t, (int)s_gtt[sg.bl]) * VP_ONE;
                uint32_t two = 0, off = 0;
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const uint32_t pv = ((keep >> (8 * k)) & 0x00ff00ffu) * 0x101u;
                    uint32_t x;
                    two += (vp_codes((w4 >> (8 * k)) & 0x00ff00ffu, (wt >> (8 * k)) & 0x00ff00ffu, t2, G2, &x) - (VP_K - VP_ONE)) & pv;
                    off |= x & pv;
                }
                const uint32_t sum = (two & 0xffffu) + (two >> 16);
                const uint32_t flag = rmode ? (((w4 | 0x80808080u) - (t + 1) * 0x01010101u) & 0x80808080u) == 0u : off == 0u;
                const uint32_t f2 = flag & __shfl_xor_sync(FULL, flag, 1), s2 = sum + __shfl_xor_sync(FULL, sum, 1);
                pnsum += sum;
                prsum += (!(lane & 1) && f2) ? s2 : 0u;
            }
            /* per byte: all ones for a group above gtli t, and its v - t - 1 */
            const uint32_t y = (w4 | 0x80808080u) - (t + 1) * 0x01010101u;
            const uint32_t above = sign_bytes(y), na = __popc(above & 0x01010101u);
            const uint32_t dd = __dp4a(y & above & 0x7f7f7f7fu, 0x01010101u, 0u);
            const uint32_t some = above | __shfl_xor_sync(FULL, above, 1); /* significance group: 2 lanes */
            dsum += 4 * (dd + (2 - fs) * na);
            vsum += dd + na + nv;
            zsum += some ? 0u : nv;
            if (fs && above) {
                const uint4 c0 = *(const uint4*)(crow + 4 * g), c1 = *(const uint4*)(crow + 4 * g + 8);
                const uint32_t cw[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t v = (w4 >> (8 * k)) & 255u;
                    if (k < (int)nv && v > t) nsum += __popc(nonzero_flags(cw[2 * k], v, t, uniform && t) | nonzero_flags(cw[2 * k + 1], v, t, uniform && t) >> 1);
                }
            }
        }
        dsum = __reduce_add_sync(FULL, dsum);
        vsum = __reduce_add_sync(FULL, vsum);
        zsum = __reduce_add_sync(FULL, zsum);
        nsum = __reduce_add_sync(FULL, nsum);
        if (VPRED) {
            pnsum = __reduce_add_sync(FULL, pnsum);
            prsum = __reduce_add_sync(FULL, prsum);
        }
        if (lane == 0) {
            s_data[sidx] = dsum;
            s_vlc[sidx] = vsum;
            s_zero[sidx] = zsum;
            s_nz[sidx] = nsum;
            if (VPRED) {
                s_vn[sidx] = pnsum;
                s_vr[sidx] = prsum;
            }
        }
    }
    __syncthreads();

    /* layout: band totals of every coding */
    for (uint32_t i = threadIdx.x; i < nseg; i += blockDim.x) {
        const jxs_bline_t& B = bls[segs[i].bl];
        const uint32_t sw = segs[i].g0 ? 0u : B.sig_w;
        atomicAdd(&s_cn[B.fb], s_vlc[i]);
        atomicAdd(&s_cs[B.fb], s_vlc[i] - s_zero[i] + sw);
        if (VPRED && vp) {
            atomicAdd(&s_cv[B.fb], s_vn[i]);
            atomicAdd(&s_cvs[B.fb], s_vn[i] - s_vr[i] + sw);
        }
    }
    __syncthreads();
    /* coding method of a band, D[p,b] (bit 1 significance, bit 0 prediction):
     * a later one only if strictly cheaper (RateControl.c:526-676) */
    auto data_at = [&](uint32_t i) { return s_data[i] + s_part[0][i >> 5]; };
    auto vlc_at = [&](uint32_t i) { return s_vlc[i] + s_part[1][i >> 5]; };
    auto nz_at = [&](uint32_t i) { return s_nz[i] + s_part[SIGNS ? 2 : 0][i >> 5]; };
    auto method = [&](uint32_t fb) {
        uint32_t m = 0, best = s_cn[fb];
        if (s_sig && best > s_cs[fb]) {
            m = 2;
            best = s_cs[fb];
        }
        if (VPRED && vp) {
            if (best > s_cv[fb]) {
                m = 1;
                best = s_cv[fb];
            }
            if (s_sig && best > s_cvs[fb]) m = 3;
        }
        return m;
    };
    if (warp == PK_WARPS - 1) {
        /* significance flags and raw GCLI bits before every line, each lane a
         * run of them */
        const uint32_t nbl = s_nbl, per = (nbl + 31) >> 5, x0 = min(nbl, per * lane), x1 = min(nbl, x0 + per);
        uint32_t sg = 0, rw = 0;
        for (uint32_t x = x0; x < x1; x++) {
            sg += (method(bls[x].fb) & 2) ? bls[x].sig_w : 0u;
            rw += 4 * bls[x].gcli_w;
        }
        uint32_t tsg, trw;
        sg = warp_excl_scan(sg, &tsg);
        rw = warp_excl_scan(rw, &trw);
        for (uint32_t x = x0; x < x1; x++) {
            s_lsx[x] = sg;
            s_lrx[x] = rw;
            sg += (method(bls[x].fb) & 2) ? bls[x].sig_w : 0u;
            rw += 4 * bls[x].gcli_w;
        }
        if (lane == 0) {
            s_lsx[nbl] = tsg;
            s_lrx[nbl] = trw;
        }
    } else if (warp == PK_WARPS - 2) {
        for (uint32_t fb = lane; fb < s_nbands; fb += 32) s_meth[fb] = (uint8_t)method(fb);
        /* precinct header: Lprc, Q, R as bytes first, then the 2-bit band
         * coding modes D[p,b] of every existing band */
        if (lane == 0) {
            const uint32_t lprc = total - s_phb;
            byte_at(buf, lead) = (uint8_t)(lprc >> 16);
            byte_at(buf, lead + 1) = (uint8_t)(lprc >> 8);
            byte_at(buf, lead + 2) = (uint8_t)lprc;
            byte_at(buf, lead + 3) = R.q;
            byte_at(buf, lead + 4) = R.r;
        }
        __syncwarp();
        uint32_t idx0 = 0;
        for (uint32_t gb0 = 0; gb0 < s_nbands_all; gb0 += 32) {
            const uint32_t gb = gb0 + lane;
            const int fb = gb < s_nbands_all ? s_g2f[gb] : JXS_NOBAND;
            const bool ex = fb != JXS_NOBAND;
            const uint32_t bal = __ballot_sync(FULL, ex);
            if (ex && s_blines[fb] > 0 && s_meth[fb])
                put_bits(buf, words, lead * 8 + 40 + 2 * (idx0 + __popc(bal & ((1u << lane) - 1))), s_meth[fb], 2, ovf);
            idx0 += __popc(bal);
        }
    }
    /* data, GCLI and sign bits before every segment, in its warp's part of 32
     * (into s_data, s_vlc, s_nz), and those of the parts; the warps from the
     * first on hold the segments, the lines are the last's in a precinct of
     * few */
    for (uint32_t i0 = 32 * warp; i0 < nseg; i0 += 32 * PK_WARPS) {
        const uint32_t i = i0 + lane;
        uint32_t d = 0, g = 0, n = 0;
        if (i < nseg) {
            const uint32_t m = method(bls[segs[i].bl].fb);
            d = s_data[i];
            g = m == 0 ? s_vlc[i] : m == 2 ? s_vlc[i] - s_zero[i] : m == 1 ? s_vn[VPRED ? i : 0] : s_vn[VPRED ? i : 0] - s_vr[VPRED ? i : 0];
            if (SIGNS) n = s_nz[i];
        }
        uint32_t td, tg, tn = 0;
        d = warp_excl_scan(d, &td);
        g = warp_excl_scan(g, &tg);
        if (SIGNS) n = warp_excl_scan(n, &tn);
        if (i < nseg) {
            s_data[i] = d;
            s_vlc[i] = g;
            if (SIGNS) s_nz[i] = n;
        }
        if (lane == 0) {
            s_part[0][i0 >> 5] = td;
            s_part[1][i0 >> 5] = tg;
            if (SIGNS) s_part[2][i0 >> 5] = tn;
        }
    }
    __syncthreads();
    if (warp == 0) {
        /* the parts' running sums: bits before segment i are its own in
         * s_data[i] and those of the parts before, s_part[0][i >> 5] */
        static_assert(JXS_MAXSEG / 32 < 32, "a lane per part, and the end");
        {
            const uint32_t parts = (nseg + 31) >> 5;
            uint32_t td, tg, tn = 0;
            const uint32_t d = warp_excl_scan(lane < parts ? s_part[0][lane] : 0u, &td);
            const uint32_t g = warp_excl_scan(lane < parts ? s_part[1][lane] : 0u, &tg);
            const uint32_t n = SIGNS ? warp_excl_scan(lane < parts ? s_part[2][lane] : 0u, &tn) : 0u;
            if (lane <= parts) {
                s_part[0][lane] = d;
                s_part[1][lane] = g;
                if (SIGNS) s_part[2][lane] = n;
            }
            /* the end, in the last part or the first place of the next */
            if (lane == (nseg >> 5)) {
                s_data[nseg] = td - d;
                s_vlc[nseg] = tg - g;
                if (SIGNS) s_nz[nseg] = tn - n;
            }
        }
        __syncwarp();
        /* one lane per packet: sub-packet sizes, raw fallback, header */
        const uint32_t k = lane;
        const uint32_t nb = k < s_npk ? s_pknbl[k] : 0u, b0 = k < s_npk ? s_pkbl0[k] : 0u;
        uint32_t db = 0, gbits = 0, sbits = 0, nbits = 0, i0 = 0;
        if (nb) {
            i0 = bls[b0].seg0;
            const uint32_t i1 = bls[b0 + nb - 1].seg0 + bls[b0 + nb - 1].nseg;
            db = data_at(i1) - data_at(i0);
            gbits = vlc_at(i1) - vlc_at(i0);
            sbits = s_lsx[b0 + nb] - s_lsx[b0];
            if (SIGNS) nbits = nz_at(i1) - nz_at(i0);
        }
        const uint32_t dB = (db + 7) >> 3, gB = (gbits + 7) >> 3, sB = (sbits + 7) >> 3, nB = (nbits + 7) >> 3;
        const uint32_t rawB = nb ? s_praw[k] : 0u;
        const int raw = nb && sB + gB > rawB;
        const uint32_t gcl_bytes = raw ? rawB : gB;
        const uint32_t hb = nb ? (s_short ? 5u : 7u) : 0u;
        const uint32_t pk_bytes = nb ? hb + (raw ? rawB : sB + gB) + dB + nB : 0u;
        uint32_t pk_total;
        const uint32_t hdr = s_phb;
        const uint32_t start = lead + hdr + warp_excl_scan(pk_bytes, &pk_total);
        const int fits = start + hb <= words * 4;
        if (nb && fits) {
            /* packet header (PackHeaders.c:98-127) */
            if (s_short) {
                byte_at(buf, start) = (uint8_t)((raw << 7) | ((dB >> 8) & 0x7f));
                byte_at(buf, start + 1) = (uint8_t)dB;
                byte_at(buf, start + 2) = (uint8_t)(gcl_bytes >> 5);
                byte_at(buf, start + 3) = (uint8_t)(((gcl_bytes & 0x1f) << 3) | ((nB >> 8) & 7));
                byte_at(buf, start + 4) = (uint8_t)nB;
            } else {
                byte_at(buf, start) = (uint8_t)((raw << 7) | ((dB >> 13) & 0x7f));
                byte_at(buf, start + 1) = (uint8_t)(dB >> 5);
                byte_at(buf, start + 2) = (uint8_t)(((dB & 0x1f) << 3) | ((gcl_bytes >> 17) & 7));
                byte_at(buf, start + 3) = (uint8_t)(gcl_bytes >> 9);
                byte_at(buf, start + 4) = (uint8_t)(gcl_bytes >> 1);
                byte_at(buf, start + 5) = (uint8_t)(((gcl_bytes & 1) << 7) | ((nB >> 8) & 0x7f));
                byte_at(buf, start + 6) = (uint8_t)nB;
            }
            /* sub-packet starts (significance, GCLIs, data, signs) less the
             * running sums at the packet's first segment or line */
            const uint32_t p0 = (start + hb) * 8, pd = p0 + (raw ? rawB : sB + gB) * 8;
            s_pks[k] = p0 - s_lsx[b0];
            s_pkg[k] = raw ? p0 - s_lrx[b0] : p0 + sB * 8 - vlc_at(i0);
            s_pkd[k] = pd - data_at(i0);
            if (SIGNS) s_pkn[k] = pd + dB * 8 - nz_at(i0);
            s_pkr[k] = (uint8_t)raw;
        }
        /* the packed size must be what the rate control paid for */
        const int all_fit = __all_sync(FULL, fits || !nb);
        if (lane == 0) {
            const uint32_t end = hdr + pk_total;
            s_ok = all_fit && end <= total && end == s_hdrs + R.data_bytes;
            if (!s_ok) {
                printf("jxs pack: precinct %d packs to %u bytes, rate control paid %u + %u bytes (total %u)\n", p, end,
                       s_hdrs, R.data_bytes, total);
                JXS_STATUS_SET(status, JXS_E_ENC_FRAME);
            }
        }
    }
    __syncthreads();
    if (!s_ok) return;
    /* every segment's positions */
    for (uint32_t i = threadIdx.x; i < nseg; i += blockDim.x) {
        const jxs_seg_t sg = segs[i];
        const jxs_bline_t& B = bls[sg.bl];
        const uint32_t m = s_meth[B.fb], raw = s_pkr[B.pk];
        PkSeg D;
        D.vpos = s_pkg[B.pk] + (raw ? s_lrx[sg.bl] + 4 * sg.g0 : vlc_at(i));
        D.dpos = s_pkd[B.pk] + data_at(i);
        D.g0n = sg.g0 | (min(SG, B.gcli_w - sg.g0) << 16);
        D.info = s_lt[sg.bl] | (m << 4) | (raw << 6) | ((uint32_t)sg.bl << 8);
        s_desc[i] = D;
        if (SIGNS) s_nst[i] = s_pkn[B.pk] + nz_at(i);
    }
    for (uint32_t x = threadIdx.x; x < s_nbl; x += blockDim.x) s_sigp[x] = s_pks[bls[x].pk] + s_lsx[x];
    __syncthreads();

    if constexpr (!SIGNS && !VPRED) {
        /* pass B.  Bound by instruction issue; per 128 groups about 200 warp
         * instructions, of them 90 for the groups above gtli. */
        uint32_t* list = &s_segw[0][0] + 128 * warp;
        for (uint32_t qi = queue_next(&s_q[1], lane); qi < nseg; qi = queue_next(&s_q[1], lane)) {
            const uint32_t sidx = s_ord[qi];
            const PkSeg D = s_desc[sidx];
            const bool uq = uniform && (D.info & 15u);
            const uint32_t line = D.info >> 8, t = D.info & 15u, n = D.g0n >> 16;
            const uint8_t* grow = gcli + s_grow[line] + (D.g0n & 0xffffu);
            const uint16_t* crow = coef + s_crow[line] + 4 * (D.g0n & 0xffffu);
            uint32_t vpos = D.vpos, dpos = D.dpos;
            if ((D.info & 64u) && vpos + 4 * n > words * 32) {
                ovf = 1;
                continue;
            }
            for (uint32_t base = 0; base < n; base += 128) {
                const uint32_t g = base + 4 * lane;
                const uint32_t nv = g < n ? min(4u, n - g) : 0u;
                /* the lane's GCLIs, one per byte (0 past the line's end) */
                uint32_t w4 = nv ? *(const uint32_t*)(grow + g) : 0u;
                const uint32_t keep = nv >= 4 ? 0xffffffffu : (1u << (8 * nv)) - 1u;
                w4 &= keep;
                /* per byte: all ones for a group above gtli (v > t), and its
                 * planes above gtli d = v - t */
                const uint32_t y = (w4 | 0x80808080u) - (t + 1) * 0x01010101u;
                const uint32_t above = sign_bytes(y), ones = above & 0x01010101u;
                const uint32_t d4 = (y & above & 0x7f7f7f7fu) + ones;
                /* code bits d + 1 of every group up to and with each byte's,
                 * data nibbles d + 1 of every group above gtli likewise */
                const uint32_t codes = (d4 + (keep & 0x01010101u)) * 0x01010101u, nibs = (d4 + ones) * 0x01010101u;
                uint32_t vl = 0;
                if (D.info & 64u) {
                    /* raw GCLIs: the lane's nibbles in one write */
                    const uint32_t h = ((w4 & 0x000f000fu) << 4) | ((w4 >> 8) & 0x000f000fu);
                    if (nv) put_left32(buf, vpos + 4 * g, (h << 24) | (h & 0x00ff0000u));
                } else {
                    vl = codes >> 24;
                    if (D.info & 32u) {
                        /* significance flags, 1 = insignificant, of the groups
                         * of 8 in lanes 2i, 2i + 1: the even votes compacted (bit
                         * i: group of 8 number i), then reversed, group 0 first */
                        const uint32_t bal = __ballot_sync(FULL, above != 0u), some = bal | (bal >> 1);
                        if (lane == 0) {
                            const uint32_t nsg = min(16u, (n - base + 7) >> 3), pos = s_sigp[line] + (((D.g0n & 0xffffu) + base) >> 3);
                            uint32_t x = ~some & 0x55555555u;
                            x = (x | (x >> 1)) & 0x33333333u;
                            x = (x | (x >> 2)) & 0x0f0f0f0fu;
                            x = (x | (x >> 4)) & 0x00ff00ffu;
                            x = (x | (x >> 8)) & 0x0000ffffu;
                            const uint32_t bits = (__brev(x) >> (32 - nsg)) << (32 - nsg);
                            if (pos + nsg > words * 32) ovf = 1;
                            else put_left32(buf, pos, bits);
                        }
                        if (!((some >> (lane & 30)) & 1u)) vl = 0;
                    }
                }
                /* one scan for three running sums: data nibbles (12 bits), code
                 * bits (12 bits), listed groups */
                const uint32_t own = (nibs >> 24) | (vl << 12) | ((uint32_t)__popc(ones) << 24);
                const uint32_t inc = warp_incl_scan(own), ex = inc - own, tot = __shfl_sync(FULL, inc, 31);
                const uint32_t tot_d = (tot & 0xfffu) << 2, tot_v = (tot >> 12) & 0xfffu, cnt = tot >> 24;
                if (max(vpos + tot_v, dpos + tot_d) > words * 32) {
                    ovf = 1;
                    break;
                }
                if (vl) {
                    /* unary codes: d ones then a zero for each present group
                     * (PackPrecinct.h:25-39) */
                    const uint32_t pos = vpos + ((ex >> 12) & 0xfffu);
                    if (vl <= 32) {
                        /* ones, and a zero where each code ends (absent groups
                         * repeat the last end) */
                        const uint32_t f = 0x20202020u - codes;
                        const uint32_t z = (1u << (f & 255u)) | (1u << __byte_perm(f, 0u, 0x4441)) | (1u << __byte_perm(f, 0u, 0x4442)) |
                                           (1u << (f >> 24));
                        put_left32(buf, pos, (uint32_t)((int32_t)0x80000000 >> (vl - 1)) & ~z);
                    } else {
                        /* up to 64 bits, first code at the top */
                        uint64_t z = 0;
#pragma unroll
                        for (int k = 0; k < 4; k++) z |= 1ull << (64 - ((codes >> (8 * k)) & 255u));
                        const uint64_t a = (uint64_t)((int64_t)0x8000000000000000ll >> (vl - 1)) & ~z;
                        put_bits(buf, words, pos, a >> (64 - vl), vl, ovf);
                    }
                }
                /* the warp lists its groups above gtli (nibble offset in the
                 * warp's data, group, GCLI), then each lane packs one listed
                 * group at a time, its sign nibble and planes in one write of
                 * at most 64 bits; the coefficients of the other groups are
                 * never read */
                {
                    const uint32_t po = nibs << 8, pi = ones * 0x01010100u; /* before each byte's group */
                    const uint32_t e0 = ((ex & 0xfffu) << 16) | ((uint32_t)lane << 6);
                    uint32_t* slot = list + (ex >> 24);
                    if (ones & 0x00000001u) slot[0] = e0 + (w4 & 255u);
                    if (ones & 0x00000100u) slot[(pi >> 8) & 255u] = e0 + 0x10u + __byte_perm(w4, po, 0x4541);
                    if (ones & 0x00010000u) slot[(pi >> 16) & 255u] = e0 + 0x20u + __byte_perm(w4, po, 0x4642);
                    if (ones & 0x01000000u) slot[pi >> 24] = e0 + 0x30u + __byte_perm(w4, po, 0x4743);
                }
                __syncwarp();
                for (uint32_t r = lane; r < cnt; r += 32) {
                    const uint32_t e = list[r];
                    const uint32_t gi = base + ((e >> 4) & 127u), np = (e & 15u) - t, pos = dpos + 4 * (e >> 16);
                    /* the coefficients past the band width are stored as zero */
                    const uint2 raw4 = *(const uint2*)(crow + 4 * gi);
                    uint32_t P01, P23;
                    quantize_signed(raw4, e & 15u, t, uq, P01, P23);
                    /* up to 8 planes with the sign's in one word, left-aligned;
                     * the upper ones only where the warp has a group with more */
                    const uint32_t low = coefs_to_planes(__byte_perm(P01, P23, 0x0246));
                    const uint32_t w = pos >> 5, sh = pos & 31;
                    uint32_t hi = low << ((28 - 4 * np) & 31);
                    if (__any_sync(__activemask(), np >= 8)) {
                        const uint32_t high = coefs_to_planes(__byte_perm(P01, P23, 0x1357));
                        uint32_t lo = 0u;
                        if (np >= 8) {
                            hi = __funnelshift_l(low, high, 60 - 4 * np); /* 4 (np + 1) bits of high : low */
                            lo = low << (60 - 4 * np);
                        }
                        const uint32_t w2 = __funnelshift_r(0u, lo, sh);
                        if (w2) atomicOr(&buf[w + 2], w2);
                        const uint32_t w1 = __funnelshift_r(lo, hi, sh);
                        if (w1) atomicOr(&buf[w + 1], w1);
                    } else {
                        const uint32_t w1 = __funnelshift_r(0u, hi, sh);
                        if (w1) atomicOr(&buf[w + 1], w1);
                    }
                    atomicOr(&buf[w], hi >> sh);
                }
                __syncwarp();
                vpos += tot_v;
                dpos += tot_d;
            }
        }
    } else {
        /* pass B with signs in a sub-packet of their own or predicted codes:
         * each lane 4 consecutive groups; its unary codes are joined into one
         * write, then a listed group's data and signs into one each */
        for (uint32_t qi = queue_next(&s_q[1], lane); qi < nseg; qi = queue_next(&s_q[1], lane)) {
            const uint32_t sidx = s_ord[qi];
            const jxs_seg_t sg = segs[sidx];
            const jxs_bline_t B = bls[sg.bl];
            const PkSeg D = s_desc[sidx];
            const uint32_t t = D.info & 15u, meth = (D.info >> 4) & 3u, raw = (D.info >> 6) & 1u;
            const uint8_t* grow = gcli + s_grow[sg.bl];
            const uint16_t* crow = coef + s_crow[sg.bl];
            const uint32_t gend = min(sg.g0 + SG, B.gcli_w);
            uint32_t vpos = D.vpos, dpos = D.dpos, npos = s_nst[SIGNS ? sidx : 0];
            for (uint32_t base = sg.g0; base < gend; base += 128) {
                const uint32_t g = base + 4 * lane;
                const uint32_t nv = g < gend ? min(4u, gend - g) : 0u;
                /* the lane's GCLIs, one per byte (0 past the line's end) */
                uint32_t w4 = nv ? *(const uint32_t*)(grow + g) : 0u;
                w4 &= nv >= 4 ? 0xffffffffu : (1u << (8 * nv)) - 1u;
                /* per byte: all ones for a group above gtli, and its planes
                 * above gtli */
                const uint32_t y = (w4 | 0x80808080u) - (t + 1) * 0x01010101u;
                const uint32_t s4 = sign_bytes(y), d4 = (y & s4 & 0x7f7f7f7fu) + (s4 & 0x01010101u);
                const uint32_t dsum = __dp4a(d4, 0x01010101u, 0u), nsig = __popc(s4 & 0x01010101u);
                uint32_t v[4];
#pragma unroll
                for (int k = 0; k < 4; k++) v[k] = (w4 >> (8 * k)) & 255u;
                const uint32_t some = s4 | __shfl_xor_sync(FULL, s4, 1);
                /* a significance group without codes: all GCLIs <= gtli, or with
                 * prediction the group's flag */
                bool insig = !some;
                uint32_t n4[4] = {0, 0, 0, 0}; /* prediction: each GCLI's code length */
                uint64_t vacc = 0;             /* otherwise: the lane's codes joined */
                uint32_t vl = 0;
                if (VPRED && (meth & 1) && !raw) {
                    /* codes predicted from the line above (vlc_encode,
                     * PackPrecinct.h:41-65) */
                    const uint32_t wt = nv ? *(const uint32_t*)(grow - s_gp[VPRED ? sg.bl : 0] + g) : 0u;
                    const uint32_t t2 = t * VP_ONE, G2 = (uint32_t)max((int)t, (int)s_gtt[VPRED ? sg.bl : 0]) * VP_ONE;
                    uint32_t off = 0;
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        const uint32_t pv = (k < (int)nv ? 0xffffu : 0u) | (k + 2 < (int)nv ? 0xffff0000u : 0u);
                        uint32_t x;
                        const uint32_t two = (vp_codes((w4 >> (8 * k)) & 0x00ff00ffu, (wt >> (8 * k)) & 0x00ff00ffu, t2, G2, &x) - (VP_K - VP_ONE)) & pv;
                        off |= x & pv;
                        n4[k] = two & 0xffffu;
                        n4[k + 2] = two >> 16;
                    }
                    const uint32_t flag = rmode ? s4 == 0u : off == 0u;
                    insig = (flag & __shfl_xor_sync(FULL, flag, 1)) != 0;
                }
                if (raw) {
                    /* raw GCLIs: the lane's nibbles in one write */
                    if (nv) put_bits(buf, words, D.vpos + 4 * (g - sg.g0), ((v[0] << 12) | (v[1] << 8) | (v[2] << 4) | v[3]) >> (4 * (4 - nv)), 4 * nv, ovf);
                } else {
                    if (meth & 2) {
                        /* significance flags, 1 = insignificant: even lanes lead a group of 8 */
                        const uint32_t bal = __ballot_sync(FULL, nv && !(lane & 1) && insig);
                        if (lane == 0) {
                            /* the even lanes' votes compacted (bit i: group of 8
                             * number i), then reversed: group 0 first */
                            const uint32_t nsg = min(16u, (gend - base + 7) >> 3);
                            uint32_t x = bal & 0x55555555u;
                            x = (x | (x >> 1)) & 0x33333333u;
                            x = (x | (x >> 2)) & 0x0f0f0f0fu;
                            x = (x | (x >> 4)) & 0x00ff00ffu;
                            x = (x | (x >> 8)) & 0x0000ffffu;
                            const uint32_t bits = __brev(x) >> (32 - nsg);
                            if (bits) put_bits(buf, words, s_sigp[sg.bl] + (base >> 3), bits, nsg, ovf);
                        }
                    }
                    if (!((meth & 2) && insig)) {
                        if (VPRED && (meth & 1)) {
#pragma unroll
                            for (int k = 0; k < 4; k++) vl += n4[k];
                        } else {
                            /* unary codes: d ones then a zero for each present
                             * group (PackPrecinct.h:25-39), two groups per word */
                            uint32_t n[4], c[4];
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                const uint32_t dk = (d4 >> (8 * k)) & 255u;
                                n[k] = k < (int)nv ? dk + 1 : 0u;
                                c[k] = ((1u << dk) - 1u) << 1;
                            }
                            const uint32_t l23 = n[2] + n[3];
                            vacc = ((uint64_t)((c[0] << n[1]) | c[1]) << l23) | ((c[2] << n[3]) | c[3]);
                            vl = dsum + nv;
                        }
                    }
                }
                /* data bits of the groups above gtli: 4 (d + 1) each (the sign
                 * nibble, unless signs go to their own sub-packet) */
                const uint32_t dl4 = dsum + (fs ? 0u : nsig);
                /* one scan for three running sums: data bits / 4 (12 bits), code
                 * bits (13 bits), listed groups (the exclusive sums, at most 124,
                 * in the top 7 bits) */
                uint32_t tot;
                const uint32_t ex = warp_excl_scan(dl4 | (vl << 12) | (nsig << 25), &tot);
                const uint32_t ex_d = (ex & 0xfffu) << 2, ex_v = (ex >> 12) & 0x1fffu;
                const uint32_t tot_d = (tot & 0xfffu) << 2, tot_v = (tot >> 12) & 0x1fffu;
                if (vl) {
                    if (VPRED && (meth & 1)) {
                        /* prediction codes (up to 31 bits each): n - 1 ones then
                         * a zero, joined while they fit 64 bits */
                        uint32_t pos = vpos + ex_v, an = 0;
                        uint64_t acc = 0;
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const uint32_t n = n4[k];
                            if (n) {
                                if (an + n > 64) {
                                    put_bits(buf, words, pos, acc, an, ovf);
                                    pos += an;
                                    acc = 0;
                                    an = 0;
                                }
                                acc = (acc << n) | (((1ull << (n - 1)) - 1) << 1);
                                an += n;
                            }
                        }
                        if (an) put_bits(buf, words, pos, acc, an, ovf);
                    } else {
                        put_bits(buf, words, vpos + ex_v, vacc, vl, ovf);
                    }
                }
                /* the warp lists its groups above gtli (bit offset in the warp's
                 * data, group, GCLI), then each lane packs one listed group at a
                 * time; the coefficients of the other groups are never read */
                uint32_t* list = &s_segw[0][0] + 128 * warp;
                const uint32_t cnt = __reduce_add_sync(FULL, nsig);
                {
                    /* per byte: 1 for a listed group, and its data nibbles v -
                     * t + 1 (v - t with separate signs); their exclusive prefix
                     * sums over the lane's bytes give each entry's slot and
                     * offset */
                    const uint32_t one = s4 & 0x01010101u, dd = fs ? d4 : d4 + one;
                    const uint32_t po = dd * 0x01010100u, pi = one * 0x01010100u;
                    const uint32_t e0 = (ex_d << 11) | ((uint32_t)lane << 6), i0 = ex >> 25;
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if ((one >> (8 * k)) & 1u)
                            list[i0 + ((pi >> (8 * k)) & 255u)] = e0 + (((po >> (8 * k)) & 255u) << 13) + ((uint32_t)k << 4) + v[k];
                }
                __syncwarp();
                for (uint32_t r0 = 0; r0 < cnt; r0 += 32) {
                    const bool have = r0 + lane < cnt;
                    uint32_t sbits = 0, sn = 0;
                    if (have) {
                        const uint32_t e = list[r0 + lane];
                        const uint32_t gi = base + ((e >> 4) & 127u), vv = e & 15u, np = vv - t;
                        /* the coefficients past the band width are stored as zero */
                        const uint2 raw4 = *(const uint2*)(crow + 4 * gi);
                        uint32_t P01, P23;
                        quantize_signed(fs ? make_uint2(raw4.x & 0x7fff7fffu, raw4.y & 0x7fff7fffu) : raw4, vv, t, uniform && t, P01, P23);
                        uint64_t planes = coefs_to_planes(__byte_perm(P01, P23, 0x0246));
                        if (np >= 8) planes |= (uint64_t)coefs_to_planes(__byte_perm(P01, P23, 0x1357)) << 32;
                        put_bits(buf, words, dpos + (e >> 11), planes, 4 * (np + 1 - fs), ovf);
                        if (fs) {
                            /* the signs of the non-zero magnitudes (pack_sign_c,
                             * PackPrecinct.c:200-233), coefficient 0 first */
                            const uint32_t z01 = (P01 + 0x7fff7fffu) & 0x80008000u, z23 = (P23 + 0x7fff7fffu) & 0x80008000u;
#pragma unroll
                            for (int j = 0; j < 4; j++) {
                                const uint32_t at = 15 + 16 * (j & 1), on = ((j < 2 ? z01 : z23) >> at) & 1u;
                                sbits = (sbits << on) | (on & ((j < 2 ? raw4.x : raw4.y) >> at));
                                sn += on;
                            }
                        }
                    }
                    if (fs) {
                        uint32_t stot;
                        const uint32_t sx = warp_excl_scan(sn, &stot);
                        if (sn) put_bits(buf, words, npos + sx, sbits, sn, ovf);
                        npos += stot;
                    }
                }
                __syncwarp();
                vpos += tot_v;
                dpos += tot_d;
            }
        }
    }
    if (__syncthreads_or(ovf)) {
        if (threadIdx.x == 0) {
            printf("jxs pack: precinct %d wrote past its %u words\n", p, words);
            JXS_STATUS_SET(status, JXS_E_ENC_FRAME);
        }
        return;
    }
    /* copy out: whole 16-byte chunks where the precinct covers them, single
     * bytes at its two ends; slice header, codestream header and EOC around */
    uint8_t* gbase = out + R.offset - lead;
    const uint32_t nbytes = lead + total;
    for (uint32_t c = threadIdx.x; c < (nbytes + 15) >> 4; c += blockDim.x) {
        const uint32_t b0 = c << 4;
        if (b0 >= lead && b0 + 16 <= nbytes) {
            const uint4 v = *(const uint4*)(buf + 4 * c);
            *(uint4*)(gbase + b0) = make_uint4(__byte_perm(v.x, 0u, 0x0123), __byte_perm(v.y, 0u, 0x0123),
                                               __byte_perm(v.z, 0u, 0x0123), __byte_perm(v.w, 0u, 0x0123));
        } else {
            for (uint32_t i = max(b0, lead); i < min(b0 + 16, nbytes); i++) gbase[i] = byte_at(buf, i);
        }
    }
    if (threadIdx.x == 0) {
        uint8_t* dst = out + R.offset;
        if (R.first_in_slice) {
            const uint32_t s = p / cfg->pps;
            uint8_t* sh = dst - 6;
            sh[0] = 0xff; sh[1] = 0x20; sh[2] = 0; sh[3] = 4;
            sh[4] = (uint8_t)(s >> 8); sh[5] = (uint8_t)s;
        }
        if (p + 1 == (int)cfg->np) {
            dst[total] = 0xff;
            dst[total + 1] = 0x11;
        }
    }
    if (p == 0)
        for (uint32_t i = threadIdx.x; i < cfg->hdr_len; i += blockDim.x) out[i] = cfg->hdr[i];
}

/* ------------------------------------------------------------------------ */
/* kernels: one frame, or a batch of frames (block -> frame by its first block) */
/* ------------------------------------------------------------------------ */
template <bool SIGNS, bool VPRED>
__global__ void __launch_bounds__(RC_THREADS, VPRED ? 2 : SIGNS ? 3 : 4) rc_cost_kernel(const jxs_cfg_t* __restrict__ cfg, const uint8_t* gcli,
                                                           const uint16_t* coef, uint32_t* cost,
                                                           uint32_t* slice_done, PrecRC* rc,
                                                           int* status) {
    rc_cost_body<SIGNS, VPRED>(cfg, gcli, coef, cost, slice_done, rc, status, (int)blockIdx.x);
}

template <bool SIGNS, bool VPRED>
__global__ void __launch_bounds__(RC_THREADS, VPRED ? 2 : SIGNS ? 3 : 4) rc_cost_batch_kernel(const __grid_constant__ EncPrecLaunch L) {
    const EncPrecFrame& F = L.job[find_job<JXS_BATCH_FRAMES>(L.job, L.nframes, (int)blockIdx.x)];
    rc_cost_body<SIGNS, VPRED>(F.cfg, F.gcli, F.coef, F.cost, F.slice_done, F.rc, F.status, (int)blockIdx.x - F.first_block);
}

template <bool SIGNS, bool VPRED>
__global__ void __launch_bounds__(PK_THREADS, VPRED ? 3 : 4) pack_kernel(const jxs_cfg_t* __restrict__ cfg, const uint16_t* coef,
                                                          const uint8_t* gcli, const PrecRC* rc,
                                                          const uint32_t* cost, uint8_t* out,
                                                          uint32_t cap_words, int* status) {
    pack_body<SIGNS, VPRED, false>(cfg, coef, gcli, rc, cost, out, cap_words, status, (int)blockIdx.x);
}

template <bool SIGNS, bool VPRED>
__global__ void __launch_bounds__(PK_THREADS, VPRED ? 3 : 4) pack_batch_kernel(const __grid_constant__ EncPrecLaunch L, uint32_t cap_words) {
    const EncPrecFrame& F = L.job[find_job<JXS_BATCH_FRAMES>(L.job, L.nframes, (int)blockIdx.x)];
    pack_body<SIGNS, VPRED, true>(F.cfg, F.coef, F.gcli, F.rc, F.cost, F.out, cap_words, F.status, (int)blockIdx.x - F.first_block);
}

/* ------------------------------------------------------------------------ */
/* host-side launchers                                                       */
/* ------------------------------------------------------------------------ */
/* The rate-control variants: `modes` bit 0 = a frame of the launch has
 * sign handling, bit 1 = vertical prediction (dynamic shared memory for
 * the ordered selection). */
#define RC_VP_SMEM (RC_VP_REGIONS * RC_LT_REGION * 4)
template <bool S, bool V>
static cudaError_t rc_one(const jxs_cfg_t* dcfg, uint32_t np, const uint8_t* gcli, const uint16_t* coef, uint32_t* cost,
                          uint32_t* slice_done, PrecRC* rc, int* status, cudaStream_t st) {
    if (V) {
        static std::atomic<int> attr[JXS_MAX_DEV];
        cudaError_t e = jxs_smem_attr(rc_cost_kernel<S, V>, RC_VP_SMEM, attr);
        if (e != cudaSuccess) return e;
    }
    return jxs_launch(rc_cost_kernel<S, V>, dim3(np), RC_THREADS, V ? RC_VP_SMEM : 0, st, dcfg, gcli, coef, cost, slice_done, rc, status);
}
template <bool S, bool V>
static cudaError_t rc_batch_one(const EncPrecLaunch* L, cudaStream_t st) {
    if (V) {
        static std::atomic<int> attr[JXS_MAX_DEV];
        cudaError_t e = jxs_smem_attr(rc_cost_batch_kernel<S, V>, RC_VP_SMEM, attr);
        if (e != cudaSuccess) return e;
    }
    rc_cost_batch_kernel<S, V><<<L->nblocks, RC_THREADS, V ? RC_VP_SMEM : 0, st>>>(*L);
    return cudaGetLastError();
}

extern "C" cudaError_t jxs_launch_rc(const jxs_cfg_t* dcfg, uint32_t np, uint32_t nslices, const uint8_t* gcli,
                                     const uint16_t* coef, uint32_t* cost, uint32_t* slice_done, PrecRC* rc, int* status,
                                     int modes, cudaStream_t st) {
    (void)nslices;
    switch (modes & 3) {
    case 0: return rc_one<false, false>(dcfg, np, gcli, coef, cost, slice_done, rc, status, st);
    case 1: return rc_one<true, false>(dcfg, np, gcli, coef, cost, slice_done, rc, status, st);
    case 2: return rc_one<false, true>(dcfg, np, gcli, coef, cost, slice_done, rc, status, st);
    default: return rc_one<true, true>(dcfg, np, gcli, coef, cost, slice_done, rc, status, st);
    }
}

template <bool S, bool V>
static cudaError_t pack_one(const jxs_cfg_t* dcfg, uint32_t np, const uint16_t* coef, const uint8_t* gcli, const PrecRC* rc,
                            const uint32_t* cost, uint8_t* out, uint32_t cap_words, int* status, cudaStream_t st) {
    const size_t smem = (size_t)cap_words * 4;
    static std::atomic<int> attr[JXS_MAX_DEV];
    cudaError_t e = jxs_smem_attr(pack_kernel<S, V>, (int)smem, attr);
    if (e != cudaSuccess) return e;
    return jxs_launch(pack_kernel<S, V>, dim3(np), PK_THREADS, smem, st, dcfg, coef, gcli, rc, cost, out, cap_words, status);
}

/* `modes` as for the rate control */
extern "C" cudaError_t jxs_launch_pack(const jxs_cfg_t* dcfg, uint32_t np, const uint16_t* coef, const uint8_t* gcli,
                                       const PrecRC* rc, const uint32_t* cost, uint8_t* out, uint32_t cap_words, int* status,
                                       int modes, cudaStream_t st) {
    if (modes & 2) return pack_one<true, true>(dcfg, np, coef, gcli, rc, cost, out, cap_words, status, st);
    if (modes & 1) return pack_one<true, false>(dcfg, np, coef, gcli, rc, cost, out, cap_words, status, st);
    return pack_one<false, false>(dcfg, np, coef, gcli, rc, cost, out, cap_words, status, st);
}

extern "C" cudaError_t jxs_launch_rc_batch(const EncPrecLaunch* L, int modes, cudaStream_t st) {
    if (L->nblocks <= 0) return cudaSuccess;
    switch (modes & 3) {
    case 0: return rc_batch_one<false, false>(L, st);
    case 1: return rc_batch_one<true, false>(L, st);
    case 2: return rc_batch_one<false, true>(L, st);
    default: return rc_batch_one<true, true>(L, st);
    }
}

template <bool S, bool V>
static cudaError_t pack_batch_one(const EncPrecLaunch* L, uint32_t cap_words, cudaStream_t st) {
    const size_t smem = (size_t)cap_words * 4;
    static std::atomic<int> attr[JXS_MAX_DEV];
    cudaError_t e = jxs_smem_attr(pack_batch_kernel<S, V>, (int)smem, attr);
    if (e != cudaSuccess) return e;
    if (L->nblocks <= 0) return cudaSuccess;
    pack_batch_kernel<S, V><<<L->nblocks, PK_THREADS, smem, st>>>(*L, cap_words);
    return cudaGetLastError();
}

extern "C" cudaError_t jxs_launch_pack_batch(const EncPrecLaunch* L, uint32_t cap_words, int modes, cudaStream_t st) {
    if (modes & 2) return pack_batch_one<true, true>(L, cap_words, st);
    if (modes & 1) return pack_batch_one<true, false>(L, cap_words, st);
    return pack_batch_one<false, false>(L, cap_words, st);
}
