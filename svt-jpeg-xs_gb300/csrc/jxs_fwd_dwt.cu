/*
 * Forward 5/3 wavelet transform for sm_103a.
 *
 *  fwd_v_kernel  one vertical level and the horizontal level that follows
 *                it.  Each warp streams down a strip of 240 columns (8 per
 *                lane, plus one halo lane on either side) for 8 row pairs:
 *                vertical lifting in registers, then horizontal lifting
 *                across the warp with shuffles.  Outputs: the HL, LH and HH
 *                bands as 16-bit sign-magnitude coefficients with the GCLI of
 *                every 4-coefficient group (one group per lane and band row),
 *                and the int32 LL plane for the next level.
 *  fwd_h_kernel  the horizontal-only levels below the last vertical level
 *                (or all levels of a component without vertical
 *                decomposition): one warp per chunk of a row, every level in
 *                registers, the high band of each level and the final LL
 *                band emitted as coefficients + GCLIs.
 *
 * Arithmetic (bit-exact with the reference):
 *  - input scaling: v = ((x & (2^d - 1)) << (20 - d)) - 2^19 (NltEnc.c:33-72);
 *  - lifting: d[i] = x[2i+1] - ((x[2i] + x[2i+2]) >> 1),
 *    s[i] = x[2i] + ((d[i-1] + d[i] + 2) >> 2), with whole-sample symmetric
 *    extension at both ends (Dwt.c:15-40 horizontally, :337-398 vertically;
 *    the reference's edge special cases are what the mirrored samples give);
 *  - vertical before horizontal at every level, the low band of a level
 *    being the next level's input (Dwt.c:550-1142, frame form);
 *  - sign-magnitude with Fq = 8: m = (|v| + 128) >> 8, no negative zero
 *    (NltEnc.c:12-31);
 *  - GCLI = bit length of the OR of a group's magnitudes
 *    (GcStageProcess.c:42-68).
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "jxs_core.h"
#include "jxs_kernels.cuh"

#define DEV __device__ __forceinline__
#define FULL 0xffffffffu

/* ------------------------------------------------------------------------ */
/* helpers                                                                   */
/* ------------------------------------------------------------------------ */
/* whole-sample symmetric extension of index i into [0, n) */
DEV int mirror_idx(int i, int n) {
    if ((unsigned)i < (unsigned)n) return i;
    if (n == 1) return 0;
    const int p = 2 * (n - 1);
    i %= p;
    if (i < 0) i += p;
    return i < n ? i : p - i;
}

/* The same for the indices a strip reads (-n < i < 2n - 1: one reflection)
 * without a division; other indices (levels of one or two samples) take the
 * general form out of line, so that the division is never inlined into the
 * loops. */
__device__ __noinline__ int mirror_far(int i, int n) { return mirror_idx(i, n); }
DEV int mirror1(int i, int n) {
    const int a = i < 0 ? -i : i;
    const int m = a < n ? a : 2 * (n - 1) - a;
    return (unsigned)m < (unsigned)n ? m : mirror_far(i, n);
}

/* Two values as 16-bit sign-magnitude, the first in the low half: m = (|v| +
 * 128) >> 8 (bytes 1 and 2 of the sum), the sign only where m is not zero.
 * m stays below 2^15, so that m + 0x7fff has bit 15 set exactly where m > 0. */
DEV uint32_t sm_pair(int32_t v0, int32_t v1) {
    const uint32_t m = __byte_perm((uint32_t)abs(v0) + 128u, (uint32_t)abs(v1) + 128u, 0x6521);
    const uint32_t sign = __byte_perm((uint32_t)v0, (uint32_t)v1, 0x7733);
    return m | ((m + 0x7fff7fffu) & sign & 0x80008000u);
}
/* GCLI of a group of two pairs */
DEV uint32_t gcli_of(uint32_t c01, uint32_t c23) {
    const uint32_t o = c01 | c23;
    return 32u - (uint32_t)__clz((int)((o | (o >> 16)) & 0x7fffu));
}

/* One lane's 4-coefficient group of a band row: coefficients j..j+3 (j a
 * multiple of 4) as sign-magnitude plus the group's GCLI.  crow / grow are
 * the band row's coefficient and GCLI rows; w its width, gw its groups.
 * Coefficients past the width are written as zero; nothing past the last
 * group. */
struct BandRow {
    uint16_t* crow;
    uint8_t* grow;
    int w, gw;
};
DEV BandRow band_row(const jxs_band_t& bd, int row, uint16_t* coef, uint8_t* gcli) {
    BandRow r;
    r.crow = coef + bd.coef_off + (uint64_t)row * bd.pitch;
    r.grow = gcli + bd.gcli_off + (uint64_t)row * bd.gpitch;
    r.w = (int)bd.w;
    r.gw = (int)bd.gcli_w;
    return r;
}
DEV void emit4(const BandRow& b, int j, int32_t v0, int32_t v1, int32_t v2, int32_t v3) {
    if ((j >> 2) >= b.gw) return;
    const uint32_t c01 = sm_pair(v0, j + 1 < b.w ? v1 : 0), c23 = sm_pair(j + 2 < b.w ? v2 : 0, j + 3 < b.w ? v3 : 0);
    *(uint2*)(b.crow + j) = make_uint2(c01, c23);
    b.grow[j >> 2] = (uint8_t)gcli_of(c01, c23);
}

/* ------------------------------------------------------------------------ */
/* vertical level + one horizontal level                                     */
/* ------------------------------------------------------------------------ */
/* A tile is FV_COLS columns x FV_ROWPAIRS row pairs of the level input; its
 * warps are stacked vertically, each working alone on FV_WROWPAIRS row pairs
 * of the tile's column strip.  Lane l holds the 8 columns c0 = first - 8 +
 * 8 l .. c0 + 7: lanes 1 to 30 produce the strip, lanes 0 and 31 are the
 * halo the horizontal lifting needs on either side.  Each lane streams down
 * its 8 columns: two input rows per step, the vertical lifting in registers
 * (the previous even row and high value are kept), then the horizontal
 * lifting of the new low and high rows across the warp (the neighbours by
 * two shuffles).  Every lane's 4 output pairs are one 4-coefficient group of
 * each band.  No shared memory, no block barrier. */
#define FV_WARPS 4
#define FV_THREADS (32 * FV_WARPS)
#define FV_COLS 240          /* level-input columns of a strip: lanes 1..30, 8 each */
#define FV_WROWPAIRS 8       /* row pairs per warp */
#define FV_ROWPAIRS (FV_WROWPAIRS * FV_WARPS)

/* Raw samples of one input row for a lane's 8 columns: 16-bit sources hold
 * two samples per word (column 2k in the low half of word k), int32 sources
 * one per word. */
template <int SRC> struct FvRaw { static const int N = 4; };
template <> struct FvRaw<SRC_I32> { static const int N = 8; };

/* raw value of column x (0 <= x < w) of a row */
template <int SRC>
DEV uint32_t raw1(const void* row, int chan, int x) {
    if (SRC == SRC_I32) return (uint32_t)((const int32_t*)row)[x];
    if (SRC == SRC_U8) return ((const uint8_t*)row)[x];
    if (SRC == SRC_U16) return ((const uint16_t*)row)[x];
    if (SRC == SRC_PK8) return ((const uint8_t*)row)[3 * x + chan];
    return ((const uint16_t*)row)[3 * x + chan];
}

template <int SRC> DEV size_t src_elem() { return SRC == SRC_I32 ? 4 : (SRC == SRC_U16 || SRC == SRC_PK16) ? 2 : 1; }

/* A strip's input: base, row pitch in bytes, width and channel, held in
 * registers for the whole strip. */
struct FvSrc {
    const char* base;
    size_t pitch;
    int w, chan;
};

/* Loads row y (in range) for the lane's columns c0 .. c0 + 7: one or two
 * vector loads when the lane's 8 columns are inside and the rows aligned
 * (`fast`; always so in a FAST strip), else one load per column with the
 * symmetric extension. */
template <int SRC, bool FAST>
DEV void fv_load(const FvSrc& S, int y, int c0, bool fast, uint32_t* r) {
    const char* row = S.base + (size_t)y * S.pitch;
    if constexpr (SRC == SRC_I32) {
        if (FAST || fast) {
            const int4 a = *(const int4*)((const int32_t*)row + c0), b = *(const int4*)((const int32_t*)row + c0 + 4);
            r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
            r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
        } else {
#pragma unroll
            for (int k = 0; k < 8; k++) r[k] = raw1<SRC>(row, 0, mirror1(c0 + k, S.w));
        }
    } else if ((FAST || fast) && SRC == SRC_U16) {
        const uint4 q = *(const uint4*)((const uint16_t*)row + c0);
        r[0] = q.x; r[1] = q.y; r[2] = q.z; r[3] = q.w;
    } else if ((FAST || fast) && SRC == SRC_U8) {
        const uint2 q = *(const uint2*)((const uint8_t*)row + c0);
        r[0] = __byte_perm(q.x, 0, 0x4140);
        r[1] = __byte_perm(q.x, 0, 0x4342);
        r[2] = __byte_perm(q.y, 0, 0x4140);
        r[3] = __byte_perm(q.y, 0, 0x4342);
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++)
            r[k] = raw1<SRC>(row, S.chan, mirror1(c0 + 2 * k, S.w)) | (raw1<SRC>(row, S.chan, mirror1(c0 + 2 * k + 1, S.w)) << 16);
    }
}

/* The scaled samples of a raw row: ((x & (2^d - 1)) << (20 - d)) - 2^19 as
 * one multiply-add (mul = 2^(20 - d)). */
template <int SRC>
DEV void fv_decode(const uint32_t* r, uint32_t mask, int32_t mul, int32_t* v) {
    if constexpr (SRC == SRC_I32) {
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = (int32_t)r[k];
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[2 * k] = (int32_t)(r[k] & mask) * mul - (1 << 19);
            v[2 * k + 1] = (int32_t)((r[k] >> 16) & mask) * mul - (1 << 19);
        }
    }
}

/* Horizontal lifting of one row across the warp: v holds the lane's 8
 * samples x[2j0 .. 2j0 + 7]; s / d receive its 4 low / high outputs.  The
 * right neighbour's first sample and the left neighbour's last high value
 * come by shuffles (lanes 0 and 31 get values only their neighbours use). */
DEV void fv_hlift(const int32_t* v, int32_t* s, int32_t* d) {
    const int32_t nx = __shfl_down_sync(FULL, v[0], 1);
    d[0] = v[1] - ((v[0] + v[2]) >> 1);
    d[1] = v[3] - ((v[2] + v[4]) >> 1);
    d[2] = v[5] - ((v[4] + v[6]) >> 1);
    d[3] = v[7] - ((v[6] + nx) >> 1);
    const int32_t dm = __shfl_up_sync(FULL, d[3], 1);
    s[0] = v[0] + ((dm + d[0] + 2) >> 2);
    s[1] = v[2] + ((d[0] + d[1] + 2) >> 2);
    s[2] = v[4] + ((d[1] + d[2] + 2) >> 2);
    s[3] = v[6] + ((d[2] + d[3] + 2) >> 2);
}

/* One band's output of a strip: coefficient and GCLI rows advanced by one
 * band row per step. */
struct FvBand {
    uint16_t* crow;
    uint8_t* grow;
    uint32_t pitch, gpitch;
    int w, gw;
};
DEV FvBand fv_band(const jxs_band_t& bd, int row, uint16_t* coef, uint8_t* gcli) {
    FvBand b;
    b.pitch = bd.pitch;
    b.gpitch = bd.gpitch;
    b.crow = coef + bd.coef_off + (uint64_t)row * bd.pitch;
    b.grow = gcli + bd.gcli_off + (uint64_t)row * bd.gpitch;
    b.w = (int)bd.w;
    b.gw = (int)bd.gcli_w;
    return b;
}
template <bool FAST>
DEV void fv_emit(const FvBand& b, int j, const int32_t* v) {
    if constexpr (FAST) {
        /* the whole group inside the band */
        const uint32_t c01 = sm_pair(v[0], v[1]), c23 = sm_pair(v[2], v[3]);
        *(uint2*)(b.crow + j) = make_uint2(c01, c23);
        b.grow[j >> 2] = (uint8_t)gcli_of(c01, c23);
    } else {
        emit4(BandRow{b.crow, b.grow, b.w, b.gw}, j, v[0], v[1], v[2], v[3]);
    }
}
DEV void fv_next(FvBand& b) {
    b.crow += b.pitch;
    b.grow += b.gpitch;
}

/* One warp's strip: row pairs r0 .. rend - 1 of columns c0 (this lane) of
 * job J.  FAST: the strip is away from the level's left and right edges
 * (every lane's 8 columns and every output group inside), so that no load
 * or store needs a check. */
template <int SRC, bool FAST>
DEV void fv_strip(const FwdVJob& J, int r0, int rend, int c0) {
    const int lane = threadIdx.x & 31;
    const int h = J.h, n2 = h >> 1;
    const FvSrc S{(const char*)J.src, (size_t)J.src_pitch * src_elem<SRC>(), J.w, J.chan};
    const bool fast = J.vec && c0 >= 0 && c0 + 8 <= J.w;
    const uint32_t mask = (1u << J.depth) - 1u;
    const int32_t mul = 1 << (20 - J.depth);
    /* output: pairs jj .. jj + 3 of the level's bands (one group), lanes 1..30 */
    const int jj = c0 >> 1, w1 = (J.w + 1) >> 1;
    const bool out_lane = lane >= 1 && lane <= 30 && c0 < J.w;
    FvBand bhl = fv_band(J.bands[J.b_hl], r0, J.coef, J.gcli);
    FvBand blh = fv_band(J.bands[J.b_lh], r0, J.coef, J.gcli);
    FvBand bhh = fv_band(J.bands[J.b_hh], r0, J.coef, J.gcli);
    const int ll_pitch = J.ll_pitch;
    int32_t* ll = J.ll + (size_t)r0 * ll_pitch + jj;
    const int N = FvRaw<SRC>::N;

    /* x[2 r0] and d[r0 - 1] (rows 2 r0 - 2, 2 r0 - 1 mirrored at the top);
     * rows 2 r0 + 1, 2 r0 + 2 already in flight */
    int32_t xe[8], dp[8];
    uint32_t ra[N], rb[N];
    {
        uint32_t q0[N], q1[N], q2[N];
        fv_load<SRC, FAST>(S, mirror1(2 * r0 - 2, h), c0, fast, q0);
        fv_load<SRC, FAST>(S, mirror1(2 * r0 - 1, h), c0, fast, q1);
        fv_load<SRC, FAST>(S, 2 * r0, c0, fast, q2);
        fv_load<SRC, FAST>(S, mirror1(2 * r0 + 1, h), c0, fast, ra);
        fv_load<SRC, FAST>(S, mirror1(2 * r0 + 2, h), c0, fast, rb);
        int32_t xa[8], xb[8];
        fv_decode<SRC>(q0, mask, mul, xa);
        fv_decode<SRC>(q1, mask, mul, xb);
        fv_decode<SRC>(q2, mask, mul, xe);
#pragma unroll
        for (int k = 0; k < 8; k++) dp[k] = xb[k] - ((xa[k] + xe[k]) >> 1);
    }
    for (int i = r0; i < rend; i++) {
        int32_t xo[8], xn[8];
        fv_decode<SRC>(ra, mask, mul, xo);
        fv_decode<SRC>(rb, mask, mul, xn);
        if (i + 1 < rend) {
            /* rows 2i + 3, 2i + 4, mirrored past the bottom */
            const int ya = 2 * i + 3, yb = 2 * i + 4;
            fv_load<SRC, FAST>(S, ya < h ? ya : mirror1(ya, h), c0, fast, ra);
            fv_load<SRC, FAST>(S, yb < h ? yb : mirror1(yb, h), c0, fast, rb);
        }
        /* vertical lifting: high d[i], low s[i] */
        int32_t d[8], s[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            d[k] = xo[k] - ((xe[k] + xn[k]) >> 1);
            s[k] = xe[k] + ((dp[k] + d[k] + 2) >> 2);
            xe[k] = xn[k];
            dp[k] = d[k];
        }
        /* low row i: LL (int32, next level) and HL */
        int32_t hs[4], hd[4];
        fv_hlift(s, hs, hd);
        if (out_lane) {
            fv_emit<FAST>(bhl, jj, hd);
            if (FAST || jj + 3 < w1) {
                *(int4*)ll = make_int4(hs[0], hs[1], hs[2], hs[3]);
            } else {
                for (int q = 0; q < 4; q++)
                    if (jj + q < w1) ll[q] = hs[q];
            }
        }
        /* high row i: LH and HH */
        if (i < n2) {
            fv_hlift(d, hs, hd);
            if (out_lane) {
                fv_emit<FAST>(blh, jj, hs);
                fv_emit<FAST>(bhh, jj, hd);
            }
        }
        fv_next(bhl);
        fv_next(blh);
        fv_next(bhh);
        ll += ll_pitch;
    }
}

template <int SRC, int NJ>
__global__ void __launch_bounds__(FV_THREADS) fwd_v_kernel(const __grid_constant__ FwdVLaunchN<NJ> L) {
    const FwdVJob& J = L.job[find_job<NJ>(L.job, L.njobs, (int)blockIdx.x)];
    const int u = blockIdx.x - J.first_block;
    const int ty = u / J.col_tiles, tx = u - ty * J.col_tiles;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n1 = (J.h + 1) >> 1;
    const int r0 = (ty * FV_WARPS + warp) * FV_WROWPAIRS;
    if (r0 >= n1) return; /* the whole warp */
    const int rend = min(r0 + FV_WROWPAIRS, n1);
    const int first = tx * FV_COLS, c0 = first - 8 + 8 * lane;
    /* the strip's 256 columns first - 8 .. first + 247 all inside: the
     * whole warp takes the path without checks */
    if (J.vec && first >= 8 && first + FV_COLS + 8 <= J.w) fv_strip<SRC, true>(J, r0, rend, c0);
    else fv_strip<SRC, false>(J, r0, rend, c0);
}

/* ------------------------------------------------------------------------ */
/* horizontal-only levels                                                    */
/* ------------------------------------------------------------------------ */
/* A warp transforms one chunk of one row through every level in registers:
 * lane l holds the 16 input columns c0 = first - 16 halo + 16 l .. c0 + 15,
 * so that a level leaves 8, 4, 2, 1 low and high values per lane and, at
 * level 5, one pair per two lanes.  The neighbours come by shuffles.  A low
 * value of level e reaches 2^(e+1) - 2 input columns to either side, so the
 * outer 1 (up to 3 levels), 2 (4 levels) or 4 lanes (5 levels) on each side
 * are halo, and a chunk yields 480, 448 or 384 columns, always whole
 * 4-coefficient groups of every band.
 *
 * Bound by memory: 4 bytes read and 2 1/4 written per column.  The form
 * before kept whole rows in shared memory, one warp per row, which left 8
 * warps on an SM for the 3840-column rows of an 8K frame with one vertical
 * level: 8 such frames took 650 us, now 250 (1.24 GB; encode 3308 -> 2907
 * us). */
#define FH_MAX_WARPS 4
#define FH_COLS 16

/* columns a warp's chunk yields */
static inline __host__ __device__ int fh_halo_lanes(int nh) { return nh >= 5 ? 4 : nh == 4 ? 2 : 1; }
static inline __host__ __device__ int fh_net_cols(int nh) { return FH_COLS * (32 - 2 * fh_halo_lanes(nh)); }

/* One level over the lane's N inputs x (the row's samples i0 .. i0 + N - 1,
 * `rel` = row length - i0): N / 2 low and high values.  EDGE: the chunk
 * touches an end of the row, where the symmetric extension holds: past the
 * last pair's even sample the sample itself, before the first high value
 * the first and past the last one the last. */
template <int N, bool EDGE>
DEV void fh_level(const int32_t* x, int i0, int rel, int32_t* s, int32_t* d) {
    const int P = N / 2;
    const int32_t nx = __shfl_down_sync(FULL, x[0], 1);
#pragma unroll
    for (int q = 0; q < P; q++) {
        int32_t next = q + 1 < P ? x[2 * q + 2] : nx;
        if (EDGE && 2 * q + 2 >= rel) next = x[2 * q];
        d[q] = x[2 * q + 1] - ((x[2 * q] + next) >> 1);
    }
    int32_t dm = __shfl_up_sync(FULL, d[P - 1], 1);
    if (EDGE) {
        if (i0 == 0) dm = rel > 1 ? d[0] : 0;
#pragma unroll
        for (int q = 0; q < P; q++)
            if (2 * q + 1 >= rel) d[q] = q ? d[q - 1] : dm;
    }
#pragma unroll
    for (int q = 0; q < P; q++) s[q] = x[2 * q] + (((q ? d[q - 1] : dm) + d[q] + 2) >> 2);
}
/* The level with one input per lane: the pairs are lanes 2k, 2k + 1 and the
 * results belong to lane 2k. */
template <bool EDGE>
DEV void fh_level_lanes(int32_t x, int i0, int rel, int32_t& s, int32_t& d) {
    const int32_t xo = __shfl_down_sync(FULL, x, 1);
    int32_t next = __shfl_down_sync(FULL, x, 2);
    if (EDGE && 2 >= rel) next = x;
    d = xo - ((x + next) >> 1);
    int32_t dm = __shfl_up_sync(FULL, d, 2);
    if (EDGE) {
        if (i0 == 0) dm = rel > 1 ? d : 0;
        if (1 >= rel) d = dm;
    }
    s = x + ((dm + d + 2) >> 2);
}

/* K coefficients j .. j + K - 1 of a band row per lane (j a multiple of K)
 * with the GCLIs of their groups.  Lanes that share a group OR their
 * magnitudes down to the group's first lane.  Coefficients past the band
 * width are zero, nothing is written past the last group. */
template <int K, bool EDGE>
DEV void fh_emit(const BandRow& b, int j, const int32_t* v, bool out_lane) {
    int32_t t[K];
#pragma unroll
    for (int q = 0; q < K; q++) t[q] = !EDGE || j + q < b.w ? v[q] : 0;
    const int g = j >> 2;
    const bool ok = out_lane && (!EDGE || g < b.gw);
    if constexpr (K >= 4) {
#pragma unroll
        for (int h = 0; h < K; h += 8) {
            const uint32_t c0 = sm_pair(t[h], t[h + 1]), c1 = sm_pair(t[h + 2], t[h + 3]);
            if constexpr (K >= 8) {
                const uint32_t c2 = sm_pair(t[h + 4], t[h + 5]), c3 = sm_pair(t[h + 6], t[h + 7]);
                const int gh = g + (h >> 2);
                if (out_lane && (!EDGE || gh + 1 < b.gw)) {
                    *(uint4*)(b.crow + j + h) = make_uint4(c0, c1, c2, c3);
                    *(uint16_t*)(b.grow + gh) = (uint16_t)(gcli_of(c0, c1) | (gcli_of(c2, c3) << 8));
                } else if (EDGE && out_lane && gh < b.gw) {
                    *(uint2*)(b.crow + j + h) = make_uint2(c0, c1);
                    b.grow[gh] = (uint8_t)gcli_of(c0, c1);
                }
            } else if (ok) {
                *(uint2*)(b.crow + j) = make_uint2(c0, c1);
                b.grow[g] = (uint8_t)gcli_of(c0, c1);
            }
        }
    } else if constexpr (K == 2) {
        const uint32_t c = sm_pair(t[0], t[1]);
        const uint32_t m = c | __shfl_down_sync(FULL, c, 1);
        if (ok) {
            *(uint32_t*)(b.crow + j) = c;
            if (!(j & 3)) b.grow[g] = (uint8_t)gcli_of(m, 0u);
        }
    } else {
        const uint32_t c = sm_pair(t[0], 0);
        uint32_t m = c | __shfl_down_sync(FULL, c, 1);
        m |= __shfl_down_sync(FULL, m, 2);
        if (ok) {
            b.crow[j] = (uint16_t)c;
            if (!(j & 3)) b.grow[g] = (uint8_t)gcli_of(m, 0u);
        }
    }
}
/* one coefficient j per lane 2k */
template <bool EDGE>
DEV void fh_emit_lanes(const BandRow& b, int j, int32_t v, bool out_lane) {
    const uint32_t c = sm_pair(!EDGE || j < b.w ? v : 0, 0);
    uint32_t m = c | __shfl_down_sync(FULL, c, 2);
    m |= __shfl_down_sync(FULL, m, 4);
    if (out_lane && !(threadIdx.x & 1) && (!EDGE || (j >> 2) < b.gw)) {
        b.crow[j] = (uint16_t)c;
        if (!(j & 3)) b.grow[j >> 2] = (uint8_t)gcli_of(m, 0u);
    }
}

/* The lane's 16 input columns; columns outside the row read as anything
 * in it or as 0 (fh_level never lets them into a result). */
template <int SRC, bool EDGE>
DEV void fh_load(const FwdHJob& J, int row, int c0, int32_t* x) {
    if constexpr (SRC == SRC_I32) {
        /* rows are padded to a multiple of 4 */
        const int32_t* r = (const int32_t*)J.src + (size_t)row * J.src_pitch;
#pragma unroll
        for (int k = 0; k < FH_COLS; k += 4) {
            int4 a = make_int4(0, 0, 0, 0);
            if (!EDGE || (c0 >= 0 && c0 + k < J.w)) a = *(const int4*)(r + c0 + k);
            x[k] = a.x;
            x[k + 1] = a.y;
            x[k + 2] = a.z;
            x[k + 3] = a.w;
        }
    } else {
        const FvSrc S{(const char*)J.src, (size_t)J.src_pitch * src_elem<SRC>(), J.w, J.chan};
        const uint32_t mask = (1u << J.depth) - 1u;
        const int32_t mul = 1 << (20 - J.depth);
#pragma unroll
        for (int k = 0; k < FH_COLS; k += 8) {
            const int c = c0 + k;
            uint32_t q[4];
            fv_load<SRC, false>(S, row, EDGE ? min(max(c, 0), J.w - 1) : c, J.vec && c >= 0 && c + 8 <= J.w, q);
            fv_decode<SRC>(q, mask, mul, x + k);
        }
    }
}

template <int SRC, bool EDGE>
DEV void fh_chunk(const FwdHJob& J, int row, int c0, bool out_lane) {
    const int nh = J.nh;
    int32_t x[16];
    fh_load<SRC, EDGE>(J, row, c0, x);
    int m = J.w, b = J.b_ll;
    if (nh == 0) {
        fh_emit<16, EDGE>(band_row(J.bands[b], row, J.coef, J.gcli), c0, x, out_lane);
        return;
    }
    int32_t s1[8], d1[8];
    fh_level<16, EDGE>(x, c0, m - c0, s1, d1);
    fh_emit<8, EDGE>(band_row(J.bands[J.b_hf[0]], row, J.coef, J.gcli), c0 >> 1, d1, out_lane);
    m = (m + 1) >> 1;
    if (nh == 1) {
        fh_emit<8, EDGE>(band_row(J.bands[b], row, J.coef, J.gcli), c0 >> 1, s1, out_lane);
        return;
    }
    int32_t s2[4], d2[4];
    fh_level<8, EDGE>(s1, c0 >> 1, m - (c0 >> 1), s2, d2);
    fh_emit<4, EDGE>(band_row(J.bands[J.b_hf[1]], row, J.coef, J.gcli), c0 >> 2, d2, out_lane);
    m = (m + 1) >> 1;
    if (nh == 2) {
        fh_emit<4, EDGE>(band_row(J.bands[b], row, J.coef, J.gcli), c0 >> 2, s2, out_lane);
        return;
    }
    int32_t s3[2], d3[2];
    fh_level<4, EDGE>(s2, c0 >> 2, m - (c0 >> 2), s3, d3);
    fh_emit<2, EDGE>(band_row(J.bands[J.b_hf[2]], row, J.coef, J.gcli), c0 >> 3, d3, out_lane);
    m = (m + 1) >> 1;
    if (nh == 3) {
        fh_emit<2, EDGE>(band_row(J.bands[b], row, J.coef, J.gcli), c0 >> 3, s3, out_lane);
        return;
    }
    int32_t s4[1], d4[1];
    fh_level<2, EDGE>(s3, c0 >> 3, m - (c0 >> 3), s4, d4);
    fh_emit<1, EDGE>(band_row(J.bands[J.b_hf[3]], row, J.coef, J.gcli), c0 >> 4, d4, out_lane);
    m = (m + 1) >> 1;
    if (nh == 4) {
        fh_emit<1, EDGE>(band_row(J.bands[b], row, J.coef, J.gcli), c0 >> 4, s4, out_lane);
        return;
    }
    int32_t s5, d5;
    fh_level_lanes<EDGE>(s4[0], c0 >> 4, m - (c0 >> 4), s5, d5);
    fh_emit_lanes<EDGE>(band_row(J.bands[J.b_hf[4]], row, J.coef, J.gcli), c0 >> 5, d5, out_lane);
    fh_emit_lanes<EDGE>(band_row(J.bands[b], row, J.coef, J.gcli), c0 >> 5, s5, out_lane);
}

template <int SRC, int NJ>
__global__ void __launch_bounds__(FH_MAX_WARPS * 32) fwd_h_kernel(const __grid_constant__ FwdHLaunchN<NJ> L) {
    const FwdHJob& J = L.job[find_job<NJ>(L.job, L.njobs, (int)blockIdx.x)];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = (blockIdx.x - J.first_block) * L.rows_per_block + warp;
    const int row = unit / J.chunks, ch = unit - row * J.chunks;
    if (row >= J.h) return; /* the whole warp */
    const int halo = fh_halo_lanes(J.nh), first = ch * fh_net_cols(J.nh) - FH_COLS * halo;
    const int c0 = first + FH_COLS * lane;
    const bool out_lane = lane >= halo && lane < 32 - halo && c0 < J.w;
    if (first >= 0 && first + 32 * FH_COLS <= J.w) fh_chunk<SRC, false>(J, row, c0, out_lane);
    else fh_chunk<SRC, true>(J, row, c0, out_lane);
}

/* ------------------------------------------------------------------------ */
/* launchers                                                                 */
/* ------------------------------------------------------------------------ */
extern "C" int jxs_fwd_v_tile_rows(void) { return FV_ROWPAIRS; }
extern "C" int jxs_fwd_v_tile_cols(void) { return FV_COLS; }
extern "C" int jxs_fwd_h_max_rows_per_block(void) { return FH_MAX_WARPS; }
extern "C" int jxs_fwd_h_chunk_cols(int nh) { return fh_net_cols(nh); }

template <int SRC, int NJ>
static cudaError_t launch_v(const FwdVLaunchN<NJ>* L, int grid_per_sm, cudaStream_t st) {
    (void)grid_per_sm; /* one block per tile */
    if (L->ntiles <= 0) return cudaSuccess;
    fwd_v_kernel<SRC, NJ><<<L->ntiles, FV_THREADS, 0, st>>>(*L);
    return cudaGetLastError();
}

template <int NJ>
static cudaError_t launch_v_kind(const FwdVLaunchN<NJ>* L, int src_kind, int grid_per_sm, cudaStream_t st) {
    switch (src_kind) {
    case SRC_I32: return launch_v<SRC_I32, NJ>(L, grid_per_sm, st);
    case SRC_U8: return launch_v<SRC_U8, NJ>(L, grid_per_sm, st);
    case SRC_U16: return launch_v<SRC_U16, NJ>(L, grid_per_sm, st);
    case SRC_PK8: return launch_v<SRC_PK8, NJ>(L, grid_per_sm, st);
    default: return launch_v<SRC_PK16, NJ>(L, grid_per_sm, st);
    }
}

extern "C" cudaError_t jxs_launch_fwd_v(const FwdVLaunch* L, int src_kind, int grid_per_sm, cudaStream_t st) {
    return launch_v_kind<JXS_MAXC>(L, src_kind, grid_per_sm, st);
}
extern "C" cudaError_t jxs_launch_fwd_v_batch(const FwdVLaunchB* L, int src_kind, int grid_per_sm, cudaStream_t st) {
    return launch_v_kind<JXS_BATCH_JOBS>(L, src_kind, grid_per_sm, st);
}

template <int SRC, int NJ>
static cudaError_t launch_h(const FwdHLaunchN<NJ>* L, int nblocks, cudaStream_t st) {
    if (nblocks <= 0) return cudaSuccess;
    fwd_h_kernel<SRC, NJ><<<nblocks, L->rows_per_block * 32, 0, st>>>(*L);
    return cudaGetLastError();
}

template <int NJ>
static cudaError_t launch_h_kind(const FwdHLaunchN<NJ>* L, int src_kind, int nblocks, cudaStream_t st) {
    switch (src_kind) {
    case SRC_I32: return launch_h<SRC_I32, NJ>(L, nblocks, st);
    case SRC_U8: return launch_h<SRC_U8, NJ>(L, nblocks, st);
    case SRC_U16: return launch_h<SRC_U16, NJ>(L, nblocks, st);
    case SRC_PK8: return launch_h<SRC_PK8, NJ>(L, nblocks, st);
    default: return launch_h<SRC_PK16, NJ>(L, nblocks, st);
    }
}

extern "C" cudaError_t jxs_launch_fwd_h(const FwdHLaunch* L, int src_kind, int nblocks, cudaStream_t st) {
    return launch_h_kind<JXS_MAXC>(L, src_kind, nblocks, st);
}
extern "C" cudaError_t jxs_launch_fwd_h_batch(const FwdHLaunchB* L, int src_kind, int nblocks, cudaStream_t st) {
    return launch_h_kind<JXS_BATCH_JOBS>(L, src_kind, nblocks, st);
}
