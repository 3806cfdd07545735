/*
 * Inverse 5/3 wavelet transform for sm_103a.
 *
 *  inv_h_kernel  the horizontal-only levels, deepest first: one warp per
 *                chunk of a row combines the final LL band with the high band
 *                of each level (in registers) and writes the row of the last
 *                vertical level's low band, or, for a component without
 *                vertical levels, the output samples.
 *  inv_v_kernel  one vertical level: each warp streams down a strip of 240
 *                output columns (8 per lane, plus one halo lane on either
 *                side) for a few row pairs.  Every step rebuilds a low row (LL +
 *                HL) and a high row (LH + HH) by inverse horizontal lifting
 *                across the warp, lifts vertically in registers and writes
 *                two rows of the next level's int32 low band or, for level 0,
 *                of the output samples with the linear output scaling fused.
 *
 * Arithmetic (bit-exact with the reference): coefficients are int16 two's
 * complement scaled by << Fq (Definitions.h:128); inverse lifting
 * x[2i] = s[i] - ((d[i-1] + d[i] + 2) >> 2), x[2i+1] = d[i] + ((x[2i] +
 * x[2i+2]) >> 1) with whole-sample symmetric extension (Idwt.c:11-53,
 * :186-263); linear output scaling v += 2^(Bw-1), v = (v + 2^(zeta-1)) >>
 * zeta, clamp to [0, 2^d - 1], zeta = Bw - d (NltDec.c:242-264).
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "jxs_core.h"
#include "jxs_kernels.cuh"

#define DEV __device__ __forceinline__
#define FULL 0xffffffffu

/* linear_output_scaling (NltDec.c:242-264).  The reference adds 2^(Bw-1) in
 * int32, then rounds (v + 2^(zeta-1)) >> zeta in int64 and clamps to
 * [0, 2^d - 1].  With u = q 2^zeta + r (0 <= r < 2^zeta) the rounded value is
 * q + ((r + 2^(zeta-1)) >> zeta), so everything stays in 32 bits; the
 * constants of a launch are computed once (OutScale). */
struct OutScale {
    uint32_t half_bw, mask_z, half_z;
    int zeta, m;
};
DEV OutScale out_scale(int bw, int depth) {
    OutScale s;
    s.zeta = bw - depth;
    s.half_bw = (uint32_t)((1ull << bw) >> 1);
    s.mask_z = (1u << s.zeta) - 1u;
    s.half_z = (1u << s.zeta) >> 1;
    s.m = (1 << depth) - 1;
    return s;
}
DEV uint32_t out_sample(int32_t v, const OutScale& s) {
    const int32_t u = (int32_t)((uint32_t)v + s.half_bw);
    const int32_t t = (u >> s.zeta) + (int32_t)((((uint32_t)u & s.mask_z) + s.half_z) >> s.zeta);
    return (uint32_t)min(max(t, 0), s.m);
}

/* One band row of int16 coefficients as int32 << fq; index i < width. */
struct CoefRow {
    const int16_t* row;
    int w;
};
DEV CoefRow coef_row(const jxs_band_t& bd, int r, const int16_t* coef) {
    CoefRow c;
    c.row = coef + bd.coef_off + (uint64_t)r * bd.pitch;
    c.w = (int)bd.w;
    return c;
}

/* ------------------------------------------------------------------------ */
/* horizontal-only levels                                                    */
/* ------------------------------------------------------------------------ */
/* A warp rebuilds one chunk of one row through every level in registers:
 * lane l ends with the 16 output columns c0 = first - 16 halo + 16 l .. c0 +
 * 15, so that a level takes 8, 4, 2, 1 low and high values per lane and, at
 * level 5, one pair per two lanes.  A sample needs the high value before its
 * pair (left lane) and the next pair's even sample (right lane), which in
 * turn needs only the first values of that lane and the high value before
 * them: one halo lane on either side, or two where level 5 pairs lanes.  A
 * chunk yields 480 or 448 columns.
 *
 * Bound by memory: 2 bytes read and 4 written per column.  The form before
 * kept whole rows in shared memory, one warp per row, which left few warps
 * on an SM for wide rows: 8 8K frames with one vertical level (3840-column
 * rows) took 1050 us, now 225 (1.2 GB; that step took their decode from 3081
 * to 2249 us). */
#define IH_MAX_WARPS 4
#define IH_COLS 16

static inline __host__ __device__ int ih_halo_lanes(int nh) { return nh >= 5 ? 2 : 1; }
static inline __host__ __device__ int ih_net_cols(int nh) { return IH_COLS * (32 - 2 * ih_halo_lanes(nh)); }

/* K coefficients j .. j + K - 1 of a band row (j a multiple of K) as int32
 * << fq; indices outside the band read as 0 or as row padding (ih_level
 * never lets them into a result). */
template <int K, bool EDGE>
DEV void ih_load(const CoefRow& b, int j, int fq, int32_t* v) {
    uint32_t w[(K + 1) / 2];
#pragma unroll
    for (int k = 0; k < (K + 1) / 2; k++) w[k] = 0u;
    if constexpr (K >= 8) {
        /* rows are padded to a multiple of 8 */
#pragma unroll
        for (int h = 0; h < K; h += 8)
            if (!EDGE || (j >= 0 && j + h < b.w)) {
                const uint4 a = *(const uint4*)(b.row + j + h);
                w[h / 2] = a.x;
                w[h / 2 + 1] = a.y;
                w[h / 2 + 2] = a.z;
                w[h / 2 + 3] = a.w;
            }
    } else if (!EDGE || (j >= 0 && j < b.w)) {
        if constexpr (K == 4) {
            const uint2 a = *(const uint2*)(b.row + j);
            w[0] = a.x;
            w[1] = a.y;
        } else if constexpr (K == 2) {
            w[0] = *(const uint32_t*)(b.row + j);
        } else {
            w[0] = (uint16_t)b.row[j];
        }
    }
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = (k & 1) ? (int32_t)(w[k >> 1] & 0xffff0000u) >> (16 - fq) : (int32_t)(w[k >> 1] << 16) >> (16 - fq);
}

/* One level: the lane's P low and high values (pairs j0 .. j0 + P - 1 of n1
 * even and n2 odd samples) to its 2 P samples.  EDGE: the chunk touches an
 * end of the row, where the symmetric extension holds: high values past
 * either end are the nearest one, past the last even sample it is its own
 * right neighbour. */
template <int P, bool EDGE>
DEV void ih_level(const int32_t* s, int32_t* d, int j0, int n1, int n2, int32_t* x) {
    int32_t dm = __shfl_up_sync(FULL, d[P - 1], 1);
    if (EDGE) {
        if (j0 == 0) dm = n2 > 0 ? d[0] : 0;
#pragma unroll
        for (int q = 0; q < P; q++)
            if (j0 + q >= n2) d[q] = q ? d[q - 1] : dm;
    }
#pragma unroll
    for (int q = 0; q < P; q++) x[2 * q] = s[q] - (((q ? d[q - 1] : dm) + d[q] + 2) >> 2);
    const int32_t xn = __shfl_down_sync(FULL, x[0], 1);
#pragma unroll
    for (int q = 0; q < P; q++) {
        int32_t next = q + 1 < P ? x[2 * q + 2] : xn;
        if (EDGE && j0 + q + 1 >= n1) next = x[2 * q];
        x[2 * q + 1] = d[q] + ((x[2 * q] + next) >> 1);
    }
}
/* The level with one pair (index j) per lanes 2k, 2k + 1, held by both: lane
 * 2k gets the even sample, lane 2k + 1 the odd one. */
template <bool EDGE>
DEV int32_t ih_level_lanes(int32_t s, int32_t d, int j, int n1, int n2) {
    int32_t dm = __shfl_up_sync(FULL, d, 2);
    if (EDGE) {
        if (j == 0) dm = n2 > 0 ? d : 0;
        if (j >= n2) d = dm;
    }
    const int32_t xe = s - ((dm + d + 2) >> 2);
    int32_t next = __shfl_down_sync(FULL, xe, 2);
    if (EDGE && j + 1 >= n1) next = xe;
    return (threadIdx.x & 1) ? d + ((xe + next) >> 1) : xe;
}

/* The lane's 16 samples of row `row` from column c0 (c0 < w). */
template <int OUT, bool EDGE>
DEV void ih_store(const InvHJob& J, int row, int c0, const int32_t* x, const OutScale& os) {
    if constexpr (OUT == 0) {
        /* rows are padded to a multiple of 4 */
        int32_t* dst = (int32_t*)J.dst + (size_t)row * J.dst_pitch + c0;
#pragma unroll
        for (int k = 0; k < IH_COLS; k += 4)
            if (!EDGE || c0 + k < J.w) *(int4*)(dst + k) = make_int4(x[k], x[k + 1], x[k + 2], x[k + 3]);
    } else {
        /* samples: vector stores where the rows are aligned */
        const int esz = OUT;
        uint8_t* dst = (uint8_t*)J.dst + ((size_t)row * J.dst_pitch + c0) * esz;
        const bool vec = (((uintptr_t)J.dst | ((size_t)J.dst_pitch * esz)) & 15) == 0;
        uint32_t o[16];
#pragma unroll
        for (int k = 0; k < IH_COLS; k++) o[k] = out_sample(x[k], os);
        if (vec && (!EDGE || c0 + IH_COLS <= J.w)) {
            uint32_t w[4 * OUT];
#pragma unroll
            for (int k = 0; k < 4 * OUT; k++)
                w[k] = OUT == 1 ? o[4 * k] | (o[4 * k + 1] << 8) | (o[4 * k + 2] << 16) | (o[4 * k + 3] << 24)
                                : o[2 * k] | (o[2 * k + 1] << 16);
#pragma unroll
            for (int k = 0; k < 4 * OUT; k += 4) *(uint4*)(dst + 4 * k) = make_uint4(w[k], w[k + 1], w[k + 2], w[k + 3]);
        } else {
#pragma unroll
            for (int k = 0; k < IH_COLS; k++) {
                if (EDGE && c0 + k >= J.w) break;
                if constexpr (OUT == 1) dst[k] = (uint8_t)o[k];
                else ((uint16_t*)dst)[k] = (uint16_t)o[k];
            }
        }
    }
}

template <int OUT, bool EDGE>
DEV void ih_chunk(const InvHJob& J, int row, int c0, bool out_lane, const OutScale& os) {
    const int fq = J.fq, nh = J.nh;
    auto brow = [&](int b) { return coef_row(J.bands[b], row, J.coef); };
    int m[6]; /* the row's length at every level */
    m[0] = J.w;
#pragma unroll
    for (int e = 0; e < 5; e++) m[e + 1] = (m[e] + 1) >> 1;
    int32_t x[16];
    if (nh == 0) {
        ih_load<16, EDGE>(brow(J.b_ll), c0, fq, x);
    } else {
        int32_t d1[8], s1[8];
        ih_load<8, EDGE>(brow(J.b_hf[0]), c0 >> 1, fq, d1);
        if (nh == 1) {
            ih_load<8, EDGE>(brow(J.b_ll), c0 >> 1, fq, s1);
        } else {
            int32_t d2[4], s2[4];
            ih_load<4, EDGE>(brow(J.b_hf[1]), c0 >> 2, fq, d2);
            if (nh == 2) {
                ih_load<4, EDGE>(brow(J.b_ll), c0 >> 2, fq, s2);
            } else {
                int32_t d3[2], s3[2];
                ih_load<2, EDGE>(brow(J.b_hf[2]), c0 >> 3, fq, d3);
                if (nh == 3) {
                    ih_load<2, EDGE>(brow(J.b_ll), c0 >> 3, fq, s3);
                } else {
                    int32_t d4[1], s4[1];
                    ih_load<1, EDGE>(brow(J.b_hf[3]), c0 >> 4, fq, d4);
                    if (nh == 4) {
                        ih_load<1, EDGE>(brow(J.b_ll), c0 >> 4, fq, s4);
                    } else {
                        int32_t d5[1], s5[1];
                        ih_load<1, EDGE>(brow(J.b_hf[4]), c0 >> 5, fq, d5);
                        ih_load<1, EDGE>(brow(J.b_ll), c0 >> 5, fq, s5);
                        s4[0] = ih_level_lanes<EDGE>(s5[0], d5[0], c0 >> 5, m[5], m[4] >> 1);
                    }
                    ih_level<1, EDGE>(s4, d4, c0 >> 4, m[4], m[3] >> 1, s3);
                }
                ih_level<2, EDGE>(s3, d3, c0 >> 3, m[3], m[2] >> 1, s2);
            }
            ih_level<4, EDGE>(s2, d2, c0 >> 2, m[2], m[1] >> 1, s1);
        }
        ih_level<8, EDGE>(s1, d1, c0 >> 1, m[1], m[0] >> 1, x);
    }
    if (out_lane) ih_store<OUT, EDGE>(J, row, c0, x, os);
}

template <int OUT, int NJ>
__global__ void __launch_bounds__(IH_MAX_WARPS * 32) inv_h_kernel(const __grid_constant__ InvHLaunchN<NJ> L) {
    if (NJ <= JXS_MAXC) dep_wait();
    const InvHJob& J = L.job[find_job<NJ>(L.job, L.njobs, (int)blockIdx.x)];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = (blockIdx.x - J.first_block) * L.rows_per_block + warp;
    const int row = unit / J.chunks, ch = unit - row * J.chunks;
    if (row >= J.h) return; /* the whole warp */
    const int halo = ih_halo_lanes(J.nh), first = ch * ih_net_cols(J.nh) - IH_COLS * halo;
    const int c0 = first + IH_COLS * lane;
    const bool out_lane = lane >= halo && lane < 32 - halo && c0 < J.w;
    const OutScale os = out_scale(J.bw, J.depth);
    if (first >= 0 && first + 32 * IH_COLS <= J.w) ih_chunk<OUT, false>(J, row, c0, out_lane, os);
    else ih_chunk<OUT, true>(J, row, c0, out_lane, os);
}

/* ------------------------------------------------------------------------ */
/* vertical level                                                            */
/* ------------------------------------------------------------------------ */
/* A block is one warp, working on a strip of IV_COLS columns x rp row pairs
 * of the level's output.  Lane l holds the 8 output columns c0 = first - 8 +
 * 8 l .. c0 + 7 (band pairs j0 = c0 / 2 .. j0 + 3, one group of every band):
 * lanes 1 to 30 produce the strip, lanes 0 and 31 are the halo the lifting
 * needs on either side.  Each step rebuilds the next low row (LL + HL) and
 * high row (LH + HH) by inverse horizontal lifting across the warp (the
 * neighbours by two shuffles), lifts vertically in registers (the last even
 * row and high row are kept) and writes two output rows.  The band rows of
 * the step after are loaded while this one computes.  No shared memory, no
 * barrier; with one warp per block every row address is the same for the
 * whole block and stays out of the lanes' registers. */
#define IV_COLS 240                          /* output columns of a strip: lanes 1..30, 8 each */

DEV int clampi(int i, int n) { return i < 0 ? 0 : (i >= n ? n - 1 : i); }

/* Raw band values of the lane's pairs j0 .. j0 + 3 of a low row (int32 low
 * band) and a high row (LH coefficients), each with its high-pass
 * coefficients (HL, HH), two per word. */
struct IvRaw {
    int4 s;
    uint2 hl, lh, hh;
};
/* four int16 values of two words */
DEV void unpack4(uint2 w, int32_t* v) {
    v[0] = (int16_t)(w.x & 0xffffu);
    v[1] = (int32_t)w.x >> 16;
    v[2] = (int16_t)(w.y & 0xffffu);
    v[3] = (int32_t)w.y >> 16;
}

/* The lane's neighbours at the ends of a row (EDGE: the strip touches one):
 * the high value before its first is the first one at the row's start, high
 * values past the last are the last one. */
template <bool EDGE>
DEV int32_t iv_high_edge(int32_t* d, int j0, int w2) {
    int32_t dm = __shfl_up_sync(FULL, d[3], 1);
    if (EDGE) {
        if (j0 == 0) dm = w2 > 0 ? d[0] : 0;
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (j0 + q >= w2) d[q] = q ? d[q - 1] : dm;
    }
    return dm;
}

/* linear_output_scaling with zeta >= 2: the rounded value (u + 2^(zeta-1))
 * >> zeta (u = v + 2^(Bw-1), wrapping like the reference's int32 addition)
 * equals ((u >> 1) + 2^(zeta-2)) >> (zeta-1), which cannot overflow; then the
 * clamp to [0, 2^d - 1] */
struct OutScale8 {
    uint32_t half_bw;
    int32_t q;
    int zm1, m, general;
    OutScale os;
};
DEV OutScale8 out_scale8(int bw, int depth) {
    OutScale8 s;
    s.os = out_scale(bw, depth);
    s.half_bw = s.os.half_bw;
    s.general = s.os.zeta < 2;
    s.zm1 = s.os.zeta - 1;
    s.q = s.general ? 0 : 1 << (s.os.zeta - 2);
    s.m = s.os.m;
    return s;
}
DEV uint32_t out_sample8(int32_t v, const OutScale8& s) {
    if (s.general) return out_sample(v, s.os);
    const int32_t u = (int32_t)((uint32_t)v + s.half_bw);
    return (uint32_t)min(max(((u >> 1) + s.q) >> s.zm1, 0), s.m);
}

/* How a strip writes its rows. */
enum {
    ST_ALL = 0,     /* every lane's 8 columns inside the row, aligned rows */
    ST_WHOLE = 1,   /* every lane's 8 columns inside the row or all outside it, aligned rows */
    ST_ANY = 2      /* sample by sample */
};

/* The lane's 8 columns c0 .. c0 + 7 (c0 < w) of output row y; samples already
 * scaled. */
template <int OUT, int ST>
DEV void iv_store8(const InvVJob& J, int y, uint32_t c0, int left, const int32_t* x) {
    if constexpr (OUT == 0) {
        /* rows are padded to a multiple of 4 */
        int32_t* d = (int32_t*)J.dst + (size_t)y * J.dst_pitch + c0;
        *(int4*)d = make_int4(x[0], x[1], x[2], x[3]);
        if (ST == ST_ALL || left > 4) *(int4*)(d + 4) = make_int4(x[4], x[5], x[6], x[7]);
    } else if constexpr (OUT == 1) {
        uint8_t* d = (uint8_t*)J.dst + (size_t)y * J.dst_pitch + c0;
        if constexpr (ST != ST_ANY) {
            const uint32_t a = __byte_perm(__byte_perm(x[0], x[1], 0x0040), __byte_perm(x[2], x[3], 0x0040), 0x5410);
            const uint32_t b = __byte_perm(__byte_perm(x[4], x[5], 0x0040), __byte_perm(x[6], x[7], 0x0040), 0x5410);
            *(uint2*)d = make_uint2(a, b);
        } else {
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (q < left) d[q] = (uint8_t)x[q];
        }
    } else {
        uint16_t* d = (uint16_t*)J.dst + (size_t)y * J.dst_pitch + c0;
        if constexpr (ST != ST_ANY) {
            *(uint4*)d = make_uint4(__byte_perm(x[0], x[1], 0x5410), __byte_perm(x[2], x[3], 0x5410), __byte_perm(x[4], x[5], 0x5410),
                                    __byte_perm(x[6], x[7], 0x5410));
        } else {
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (q < left) d[q] = (uint16_t)x[q];
        }
    }
}

/* One warp's strip: row pairs r0 .. rend - 1 of output columns c0 (this
 * lane) of job J.
 *
 * EXACT (Fq 6 or 8): the coefficients are multiples of 2^Fq and no rounding
 * happens where only they meet, so that the high rows are kept as exact
 * multiples, even columns E = 4 lh - (hh' + hh) of 2^(Fq-2) and odd ones O =
 * 8 hh + E + E' of 2^(Fq-3), and the updates subtract their plain sums.  The
 * output scaling's offset 2^(Bw-1) + 2^(zeta-1) is added once to the four low
 * values of a lane: every lifting step passes a constant of the low band to
 * all samples unchanged.  Nothing can overflow: with |c| < 2^15 the levels
 * reach less than 16 2^(15+Fq) <= 2^27.  Otherwise (Fq 0) in the order of
 * the standard, rounding at every step.
 *
 * Bound by memory latency at 24 warps per SM: 29 -> 19.6 thread
 * instructions per sample against rounding at every step in 64-bit row
 * pointers, and 8 4K 4:2:2 10-bit frames in 118 us instead of 174 (560 MB of
 * DRAM traffic, 4.8 TB/s). */
template <int OUT, int ST, bool EXACT>
DEV void iv_strip(const InvVJob& J, int r0, int rend, int c0) {
    constexpr bool EDGE = ST != ST_ALL;
    const int lane = threadIdx.x & 31;
    const int w = J.w, h = J.h, fq = J.fq;
    const int n2 = h >> 1, w1 = (w + 1) >> 1, w2 = w >> 1;
    const int j0 = c0 >> 1, left = w - c0;
    const bool have = c0 >= 0 && left > 0, have2 = have && j0 < w2;
    const bool out_lane = lane >= 1 && lane <= 30 && left > 0;
    const jxs_band_t& bHL = J.bands[J.b_hl];
    const jxs_band_t& bLH = J.bands[J.b_lh];
    const jxs_band_t& bHH = J.bands[J.b_hh];
    const int16_t* hl = J.coef + bHL.coef_off;
    const int16_t* lh = J.coef + bLH.coef_off;
    const int16_t* hh = J.coef + bHH.coef_off;
    const uint32_t hl_p = bHL.pitch, lh_p = bLH.pitch, hh_p = bHH.pitch;
    const int32_t* llb = J.ll;
    const int ll_p = J.ll_pitch;
    const OutScale8 os = out_scale8(J.bw, J.depth);
    const int zeta = os.os.zeta, maxv = os.m;
    const int32_t offset = EXACT && OUT != 0 ? (int32_t)(os.half_bw + os.os.half_z) : 0;
    /* exact: scales of a coefficient, of E and O, and of their sums' quarters */
    const int32_t kc = 1 << fq, kc4 = EXACT ? kc >> 2 : 1, ke = kc4, ko = EXACT ? kc >> 3 : 1, ke4 = EXACT ? kc >> 4 : 1,
                  ko4 = EXACT ? kc >> 5 : 1;

    /* raw loads of low row i (i < (h + 1) / 2) and high row i (clamped into [0, n2),
     * n2 > 0) */
    auto ld_low = [&](int i, IvRaw& r) {
        r.s = make_int4(0, 0, 0, 0);
        r.hl = make_uint2(0u, 0u);
        if (!EDGE || have) r.s = *(const int4*)(llb + (size_t)i * ll_p + (uint32_t)j0);
        if (!EDGE || have2) r.hl = *(const uint2*)(hl + (size_t)i * hl_p + (uint32_t)j0);
    };
    auto ld_high = [&](int i, IvRaw& r) {
        i = clampi(i, n2);
        r.lh = make_uint2(0u, 0u);
        r.hh = make_uint2(0u, 0u);
        if (!EDGE || have) r.lh = *(const uint2*)(lh + (size_t)i * lh_p + (uint32_t)j0);
        if (!EDGE || have2) r.hh = *(const uint2*)(hh + (size_t)i * hh_p + (uint32_t)j0);
    };
    /* a low row's 8 samples */
    auto build_low = [&](const IvRaw& r, int32_t* x) {
        const int32_t s[4] = {r.s.x + offset, r.s.y + offset, r.s.z + offset, r.s.w + offset};
        int32_t d[4];
        unpack4(r.hl, d);
        if constexpr (!EXACT) {
#pragma unroll
            for (int q = 0; q < 4; q++) d[q] = (int32_t)((uint32_t)d[q] << fq);
        }
        const int32_t dm = iv_high_edge<EDGE>(d, j0, w2);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int32_t t = (q ? d[q - 1] : dm) + d[q];
            x[2 * q] = EXACT ? s[q] - t * kc4 : s[q] - ((t + 2) >> 2);
        }
        const int32_t xn = __shfl_down_sync(FULL, x[0], 1);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            int32_t next = q < 3 ? x[2 * q + 2] : xn;
            if (EDGE && j0 + q + 1 >= w1) next = x[2 * q];
            x[2 * q + 1] = (EXACT ? d[q] * kc : d[q]) + ((x[2 * q] + next) >> 1);
        }
    };
    /* a high row's 8 values (exact: scaled down by ke and ko) */
    auto build_high = [&](const IvRaw& r, int32_t* x) {
        int32_t s[4], d[4];
        unpack4(r.lh, s);
        unpack4(r.hh, d);
        if constexpr (!EXACT) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                s[q] = (int32_t)((uint32_t)s[q] << fq);
                d[q] = (int32_t)((uint32_t)d[q] << fq);
            }
        }
        const int32_t dm = iv_high_edge<EDGE>(d, j0, w2);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int32_t t = (q ? d[q - 1] : dm) + d[q];
            x[2 * q] = EXACT ? 4 * s[q] - t : s[q] - ((t + 2) >> 2);
        }
        const int32_t xn = __shfl_down_sync(FULL, x[0], 1);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            int32_t next = q < 3 ? x[2 * q + 2] : xn;
            if (EDGE && j0 + q + 1 >= w1) next = x[2 * q];
            x[2 * q + 1] = EXACT ? 8 * d[q] + (x[2 * q] + next) : d[q] + ((x[2 * q] + next) >> 1);
        }
    };
    auto update = [&](int k, int32_t low, int32_t ha, int32_t hb) { /* an even row's sample */
        return EXACT ? low - (ha + hb) * ((k & 1) ? ko4 : ke4) : low - ((ha + hb + 2) >> 2);
    };
    auto high = [&](int k, int32_t v) { return EXACT ? v * ((k & 1) ? ko : ke) : v; };
    auto store = [&](int y, const int32_t* x) {
        if constexpr (OUT == 0) {
            iv_store8<OUT, ST>(J, y, (uint32_t)c0, left, x);
        } else {
            int32_t o[8];
#pragma unroll
            for (int k = 0; k < 8; k++) o[k] = EXACT ? __vimin_s32_relu(x[k] >> zeta, maxv) : (int32_t)out_sample8(x[k], os);
            iv_store8<OUT, ST>(J, y, (uint32_t)c0, left, o);
        }
    };

    /* x[2 r0] = low[r0] - ((high[r0 - 1] + high[r0] + 2) >> 2) */
    int32_t xe[8], hc[8];
    IvRaw nx; /* the next step's low and high rows, in flight */
    {
        IvRaw a, b;
        ld_low(r0, a);
        if (n2) {
            ld_high(r0 - 1, b);
            ld_high(r0, a);
        }
        if (2 * r0 + 2 < h) {
            ld_low(r0 + 1, nx);
            if (n2) ld_high(r0 + 1, nx);
        }
        int32_t hp[8];
        build_low(a, xe);
        if (n2) {
            build_high(b, hp);
            build_high(a, hc);
        } else {
#pragma unroll
            for (int k = 0; k < 8; k++) hp[k] = hc[k] = 0;
        }
#pragma unroll
        for (int k = 0; k < 8; k++) xe[k] = update(k, xe[k], hp[k], hc[k]);
    }
#pragma unroll 2
    for (int i = r0; i < rend; i++) {
        const int y = 2 * i;
        int32_t xo[8], xn[8];
        if (y + 2 < h) {
            /* x[2i + 2] from the next low and high rows */
            int32_t hn[8];
            build_low(nx, xn);
            if (n2) {
                build_high(nx, hn);
            } else {
#pragma unroll
                for (int k = 0; k < 8; k++) hn[k] = 0;
            }
            if (i + 1 < rend && y + 4 < h) {
                ld_low(i + 2, nx);
                if (n2) ld_high(i + 2, nx);
            }
#pragma unroll
            for (int k = 0; k < 8; k++) {
                xn[k] = update(k, xn[k], hc[k], hn[k]);
                xo[k] = high(k, hc[k]) + ((xe[k] + xn[k]) >> 1);
                hc[k] = hn[k];
            }
        } else {
            /* the last even row is its own lower neighbour */
#pragma unroll
            for (int k = 0; k < 8; k++) {
                xn[k] = xe[k];
                xo[k] = high(k, hc[k]) + xe[k];
            }
        }
        if (out_lane) {
            store(y, xe);
            if (y + 1 < h) store(y + 1, xo);
        }
#pragma unroll
        for (int k = 0; k < 8; k++) xe[k] = xn[k];
    }
}

template <int OUT, int ST>
DEV void iv_strip_any(const InvVJob& J, int r0, int rend, int c0) {
    if (J.fq >= 6) iv_strip<OUT, ST, true>(J, r0, rend, c0);
    else iv_strip<OUT, ST, false>(J, r0, rend, c0);
}

template <int OUT, int NJ>
__global__ void __launch_bounds__(32, 24) inv_v_kernel(const __grid_constant__ InvVLaunchN<NJ> L) {
    if (NJ <= JXS_MAXC) dep_wait();
    const InvVJob& J = L.job[find_job<NJ>(L.job, L.njobs, (int)blockIdx.x)];
    const int t = blockIdx.x - J.first_block;
    const int ty = t / J.col_tiles, tx = t - ty * J.col_tiles;
    const int n1 = (J.h + 1) >> 1;
    const int r0 = ty * J.rp, rend = min(r0 + J.rp, n1);
    const int first = tx * IV_COLS, c0 = first - 8 + 8 * (int)threadIdx.x;
    const int esz = OUT == 0 ? 4 : OUT;
    const bool vec = (((uintptr_t)J.dst | ((size_t)J.dst_pitch * esz)) & (8 * esz - 1) & 15) == 0;
    /* the strip's 256 columns first - 8 .. first + 247 (band pairs up to
     * first / 2 + 123) all inside, aligned rows: the whole warp takes the
     * path without checks */
    const bool inner = first >= 8 && first + IV_COLS + 8 <= J.w;
    if (OUT == 0) {
        if (inner) iv_strip_any<OUT, ST_ALL>(J, r0, rend, c0);
        else iv_strip_any<OUT, ST_WHOLE>(J, r0, rend, c0);
    } else if (vec && inner) {
        iv_strip_any<OUT, ST_ALL>(J, r0, rend, c0);
    } else if (vec && (J.w & 7) == 0) {
        iv_strip_any<OUT, ST_WHOLE>(J, r0, rend, c0);
    } else {
        iv_strip_any<OUT, ST_ANY>(J, r0, rend, c0);
    }
}

/* ------------------------------------------------------------------------ */
/* launchers                                                                 */
/* ------------------------------------------------------------------------ */
extern "C" int jxs_inv_v_tile_cols(void) { return IV_COLS; }
extern "C" int jxs_inv_h_max_rows_per_block(void) { return IH_MAX_WARPS; }
extern "C" int jxs_inv_h_chunk_cols(int nh) { return ih_net_cols(nh); }

template <int OUT, int NJ>
static cudaError_t launch_iv(const InvVLaunchN<NJ>* L, int nblocks, cudaStream_t st) {
    if (nblocks <= 0) return cudaSuccess;
    if (NJ > JXS_MAXC) {
        inv_v_kernel<OUT, NJ><<<nblocks, 32, 0, st>>>(*L);
        return cudaGetLastError();
    }
    return jxs_launch(inv_v_kernel<OUT, NJ>, dim3((unsigned)nblocks), (unsigned)(32), 0, st, *L);
}

extern "C" cudaError_t jxs_launch_inv_v(const InvVLaunch* L, int out_kind, int nblocks, cudaStream_t st) {
    if (out_kind == 0) return launch_iv<0, JXS_MAXC>(L, nblocks, st);
    if (out_kind == 1) return launch_iv<1, JXS_MAXC>(L, nblocks, st);
    return launch_iv<2, JXS_MAXC>(L, nblocks, st);
}
extern "C" cudaError_t jxs_launch_inv_v_batch(const InvVLaunchB* L, int out_kind, int nblocks, cudaStream_t st) {
    if (out_kind == 0) return launch_iv<0, JXS_BATCH_JOBS>(L, nblocks, st);
    if (out_kind == 1) return launch_iv<1, JXS_BATCH_JOBS>(L, nblocks, st);
    return launch_iv<2, JXS_BATCH_JOBS>(L, nblocks, st);
}

template <int OUT, int NJ>
static cudaError_t launch_ih(const InvHLaunchN<NJ>* L, int nblocks, cudaStream_t st) {
    if (nblocks <= 0) return cudaSuccess;
    if (NJ > JXS_MAXC) {
        inv_h_kernel<OUT, NJ><<<nblocks, L->rows_per_block * 32, 0, st>>>(*L);
        return cudaGetLastError();
    }
    return jxs_launch(inv_h_kernel<OUT, NJ>, dim3((unsigned)nblocks), (unsigned)(L->rows_per_block * 32), 0, st, *L);
}

extern "C" cudaError_t jxs_launch_inv_h(const InvHLaunch* L, int out_kind, int nblocks, cudaStream_t st) {
    if (out_kind == 0) return launch_ih<0, JXS_MAXC>(L, nblocks, st);
    if (out_kind == 1) return launch_ih<1, JXS_MAXC>(L, nblocks, st);
    return launch_ih<2, JXS_MAXC>(L, nblocks, st);
}
extern "C" cudaError_t jxs_launch_inv_h_batch(const InvHLaunchB* L, int out_kind, int nblocks, cudaStream_t st) {
    if (out_kind == 0) return launch_ih<0, JXS_BATCH_JOBS>(L, nblocks, st);
    if (out_kind == 1) return launch_ih<1, JXS_BATCH_JOBS>(L, nblocks, st);
    return launch_ih<2, JXS_BATCH_JOBS>(L, nblocks, st);
}

/* ------------------------------------------------------------------------ */
/* Colour transform and output non-linearity                                 */
/* ------------------------------------------------------------------------ */
/* Streams with a colour transform (Cpih = 1) or an NLT marker: the last
 * inverse level writes int32 planes, and this kernel turns them into
 * samples.  Cpih = 1: the inverse reversible colour transform of
 * components 0-2 (inverse_rct, Mct.c:137-153); then every component's
 * output scaling (nlt_inverse_transform_line_*, NltDec.c:22-194, 366-406):
 * linear, quadratic (Tnlt = 1) or extended (Tnlt = 2), with the first
 * component's depth.  One thread per sample column x, rows over grid.y. */
DEV int32_t nlt_clamp64(int64_t v, int32_t m) { return (int32_t)(v > m ? m : v < 0 ? 0 : v); }

DEV int32_t nlt_sample(const NltOut& P, int64_t v) {
    const int32_t bw = P.bw, depth = P.depth, m = (1 << depth) - 1, clampv = (1 << bw) - 1;
    v += ((int64_t)1 << bw) >> 1;
    if (P.tnlt == 1) {
        const int32_t zeta = 2 * bw - depth;
        const int64_t q = (int64_t)nlt_clamp64(v, clampv);
        return nlt_clamp64(((q * q + (((int64_t)1 << zeta) >> 1)) >> zeta) + P.dco, m);
    }
    if (P.tnlt == 2) {
        const int32_t zeta = 2 * bw - depth;
        if (v < P.t1) {
            const int64_t q = nlt_clamp64((int64_t)P.b1 - v, clampv);
            v = P.a1 - q * q;
        } else if (v < P.t2) {
            v = v * ((int64_t)1 << (bw - P.e)) + P.b2;
        } else {
            const int64_t q = nlt_clamp64(v - P.b3, clampv);
            v = P.a3 + q * q;
        }
        return nlt_clamp64((v + (((int64_t)1 << zeta) >> 1)) >> zeta, m);
    }
    const int32_t zeta = bw - depth;
    return nlt_clamp64((v + (((int64_t)1 << zeta) >> 1)) >> zeta, m);
}

__global__ void __launch_bounds__(256) nlt_out_kernel(const __grid_constant__ NltOut P) {
    dep_wait();
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    int32_t v[JXS_MAXC];
#pragma unroll
    for (int k = 0; k < JXS_MAXC; k++)
        v[k] = (k < P.nc && x < P.w[k] && y < P.h[k]) ? P.in[k][(size_t)y * P.in_pitch[k] + x] : 0;
    if (P.cpih == 1 && x < P.w[0] && y < P.h[0]) {
        const int32_t o1 = v[0] - ((v[1] + v[2]) >> 2);
        const int32_t o0 = o1 + v[2], o2 = o1 + v[1];
        v[0] = o0;
        v[1] = o1;
        v[2] = o2;
    }
#pragma unroll
    for (int k = 0; k < JXS_MAXC; k++) {
        if (k >= P.nc || x >= P.w[k] || y >= P.h[k]) continue;
        const int32_t o = nlt_sample(P, v[k]);
        if (P.bps == 1) ((uint8_t*)P.out[k])[(size_t)y * P.out_pitch[k] + x] = (uint8_t)o;
        else ((uint16_t*)P.out[k])[(size_t)y * P.out_pitch[k] + x] = (uint16_t)o;
    }
}

extern "C" cudaError_t jxs_launch_nlt_out(const NltOut* P, cudaStream_t st) {
    int wmax = 1, hmax = 1;
    for (int k = 0; k < P->nc; k++) {
        wmax = max(wmax, P->w[k]);
        hmax = max(hmax, P->h[k]);
    }
    return jxs_launch(nlt_out_kernel, dim3((unsigned)((wmax + 255) / 256), (unsigned)hmax), 256, 0, st, *P);
}

/* Inverse Star-Tetrix (Cpih = 3; ISO/IEC 21122-1 Annex F, Mct.c:14-136) on
 * the int32 planes of the four components, before nlt_out_kernel.  Each of
 * the four steps updates components that none of its reads touch (the
 * access function always lands on another component), so one launch per
 * step is exact in any thread order:
 *   step 0  average: c0 -= (four diagonal neighbours) >> 3
 *   step 1  delta:   c3 += (four diagonal neighbours) >> 2
 *   step 2  Y:       c0, c3 -= (2^e2 (horizontal pair) + 2^e1 (vertical pair)) >> 3
 *   step 3  CbCr:    c1, c2 += (four direct neighbours) >> 2
 * then components 0 <-> 2 and 1 <-> 3 (done by the caller's plane order). */
__constant__ int8_t c_st_disp[2][4][2] = {{{0, 1}, {1, 1}, {0, 0}, {1, 0}}, {{1, 1}, {0, 1}, {1, 0}, {0, 0}}}; /* Table F.10 */
__constant__ uint8_t c_st_comp[2][2][2] = {{{2, 0}, {3, 1}}, {{3, 1}, {2, 0}}};                            /* Table F.11 */

/* Table F.12: mirrored at the picture edges and, for Cf = 3, within a line
 * pair */
DEV int32_t st_access(const StParams& P, int c, int x, int y, int rx, int ry) {
    const int dx = c_st_disp[P.ct][c][0], dy = c_st_disp[P.ct][c][1];
    if (2 * x + rx + dx < 0 || 2 * x + rx + dx >= 2 * P.w) rx = -rx;
    if ((P.cf == 3 && (ry + dy < 0 || ry + dy > 1)) || 2 * y + ry + dy < 0 || 2 * y + ry + dy >= 2 * P.h) ry = -ry;
    const int xx = (2 * x + rx + dx) / 2, yy = (2 * y + ry + dy) / 2;
    return P.c[c_st_comp[P.ct][(2 + rx + dx) % 2][(2 + ry + dy) % 2]][(long long)yy * P.pitch + xx];
}

/* products in 32-bit wrap-around arithmetic like the reference's int */
DEV int32_t st_mul(int32_t k, int32_t v) { return (int32_t)((uint32_t)k * (uint32_t)v); }

__global__ void __launch_bounds__(256) star_tetrix_kernel(const __grid_constant__ StParams P, int step) {
    dep_wait();
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= P.w || y >= P.h) return;
    const long long i = (long long)y * P.pitch + x;
#define ACC(c, rx, ry) st_access(P, c, x, y, rx, ry)
    if (step == 0) {
        P.c[0][i] -= (ACC(0, -1, -1) + ACC(0, 1, -1) + ACC(0, -1, 1) + ACC(0, 1, 1)) >> 3;
    } else if (step == 1) {
        P.c[3][i] += (ACC(3, -1, -1) + ACC(3, 1, -1) + ACC(3, -1, 1) + ACC(3, 1, 1)) >> 2;
    } else if (step == 2) {
        const int32_t k1 = 1 << P.e1, k2 = 1 << P.e2;
        P.c[0][i] -= (st_mul(k2, ACC(0, -1, 0) + ACC(0, 1, 0)) + st_mul(k1, ACC(0, 0, -1) + ACC(0, 0, 1))) >> 3;
        P.c[3][i] -= (st_mul(k2, ACC(3, 0, -1) + ACC(3, 0, 1)) + st_mul(k1, ACC(3, -1, 0) + ACC(3, 1, 0))) >> 3;
    } else {
        P.c[1][i] += (ACC(1, -1, 0) + ACC(1, 1, 0) + ACC(1, 0, -1) + ACC(1, 0, 1)) >> 2;
        P.c[2][i] += (ACC(2, -1, 0) + ACC(2, 1, 0) + ACC(2, 0, -1) + ACC(2, 0, 1)) >> 2;
    }
#undef ACC
}

extern "C" cudaError_t jxs_launch_star_tetrix(const StParams* P, cudaStream_t st) {
    const dim3 grid((unsigned)((P->w + 255) / 256), (unsigned)P->h);
    for (int step = 0; step < 4; step++) {
        const cudaError_t e = jxs_launch(star_tetrix_kernel, grid, 256, 0, st, *P, step);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
