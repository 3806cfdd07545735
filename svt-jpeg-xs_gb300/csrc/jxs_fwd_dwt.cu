/*
 * Forward 5/3 wavelet transform for sm_103a.
 *
 *  fwd_v_kernel  one vertical level and the horizontal level that follows
 *                it.  Each warp streams down a strip of 240 columns (8 per
 *                lane, plus one halo lane on either side) for a few row
 *                pairs: vertical lifting in registers, then horizontal
 *                lifting across the warp with shuffles.  Outputs: the HL, LH and HH
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
/* whole-sample symmetric extension of row y (-3 < y < h + 2) into [0, h) */
DEV int fold_row(int y, int h) {
    const int a = y < 0 ? -y : y;
    return a < h ? a : max(2 * (h - 1) - a, 0);
}

/* Two values as 16-bit sign-magnitude, the first in the low half: m =
 * (|v| * mul + 128) >> 8 (bytes 1 and 2 of the sum), the sign only where m is
 * not zero.  m stays below 2^15, so that m + 0x7fff has bit 15 set exactly
 * where m > 0. */
DEV uint32_t sm_pair(int32_t v0, int32_t v1, uint32_t mul) {
    const uint32_t m = __byte_perm((uint32_t)abs(v0) * mul + 128u, (uint32_t)abs(v1) * mul + 128u, 0x6521);
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
/* ------------------------------------------------------------------------ */
/* horizontal lifting across a warp, and the output of coefficients          */
/* ------------------------------------------------------------------------ */
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

/* A level of exact values, scaled instead of divided: of the lane's 8 inputs
 * x the high values 2 x[2q+1] - x[2q] - x[2q+2] (twice their size) and the low
 * values 8 x[2q] + d[q-1] + d[q] (8 times).  EDGE as for fh_level. */
template <bool EDGE>
DEV void fx_level(const int32_t* x, int i0, int rel, int32_t* s, int32_t* d) {
    const int32_t nx = __shfl_down_sync(FULL, x[0], 1);
#pragma unroll
    for (int q = 0; q < 4; q++) {
        int32_t next = q < 3 ? x[2 * q + 2] : nx;
        if (EDGE && 2 * q + 2 >= rel) next = x[2 * q];
        d[q] = 2 * x[2 * q + 1] - (x[2 * q] + next);
    }
    int32_t dm = __shfl_up_sync(FULL, d[3], 1);
    if (EDGE) {
        if (i0 == 0) dm = rel > 1 ? d[0] : 0;
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (2 * q + 1 >= rel) d[q] = q ? d[q - 1] : dm;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) s[q] = 8 * x[2 * q] + ((q ? d[q - 1] : dm) + d[q]);
}

/* K coefficients j .. j + K - 1 (values v * mul) of a band row per lane (j a
 * multiple of K) with the GCLIs of their groups.  Lanes that share a group OR their
 * magnitudes down to the group's first lane.  Coefficients past the band
 * width are zero, nothing is written past the last group. */
template <int K, bool EDGE>
DEV void fh_emit(const BandRow& b, int j, const int32_t* v, bool out_lane, uint32_t mul = 1u) {
    int32_t t[K];
#pragma unroll
    for (int q = 0; q < K; q++) t[q] = !EDGE || j + q < b.w ? v[q] : 0;
    const int g = j >> 2;
    const bool ok = out_lane && (!EDGE || g < b.gw);
    if constexpr (K >= 4) {
#pragma unroll
        for (int h = 0; h < K; h += 8) {
            const uint32_t c0 = sm_pair(t[h], t[h + 1], mul), c1 = sm_pair(t[h + 2], t[h + 3], mul);
            if constexpr (K >= 8) {
                const uint32_t c2 = sm_pair(t[h + 4], t[h + 5], mul), c3 = sm_pair(t[h + 6], t[h + 7], mul);
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
        const uint32_t c = sm_pair(t[0], t[1], mul);
        const uint32_t m = c | __shfl_down_sync(FULL, c, 1);
        if (ok) {
            *(uint32_t*)(b.crow + j) = c;
            if (!(j & 3)) b.grow[g] = (uint8_t)gcli_of(m, 0u);
        }
    } else {
        const uint32_t c = sm_pair(t[0], 0, mul);
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
    const uint32_t c = sm_pair(!EDGE || j < b.w ? v : 0, 0, 1u);
    uint32_t m = c | __shfl_down_sync(FULL, c, 2);
    m |= __shfl_down_sync(FULL, m, 4);
    if (out_lane && !(threadIdx.x & 1) && (!EDGE || (j >> 2) < b.gw)) {
        b.crow[j] = (uint16_t)c;
        if (!(j & 3)) b.grow[j >> 2] = (uint8_t)gcli_of(m, 0u);
    }
}

/* ------------------------------------------------------------------------ */
/* vertical level + one horizontal level                                     */
/* ------------------------------------------------------------------------ */
/* A block is one warp, working on a strip of FV_COLS columns x rp row pairs
 * of the level input.  Lane l holds the 8 columns c0 = first - 8 + 8 l .. c0 +
 * 7: lanes 1 to 30 produce the strip, lanes 0 and 31 are the halo the
 * horizontal lifting needs on either side.  Each lane streams down its 8
 * columns: two input rows per step, the vertical lifting in registers (the
 * previous even row and high value are kept), then the horizontal lifting of
 * the new low and high rows across the warp (the neighbours by two
 * shuffles).  Every lane's 4 output pairs are one 4-coefficient group of each
 * band.  No shared memory, no barrier; with one warp per block every row
 * address is the same for the whole block and stays out of the lanes'
 * registers, which lets 28 to 32 warps share an SM (20 with four warps per
 * block). */
#define FV_COLS 240          /* level-input columns of a strip: lanes 1..30, 8 each */

template <int SRC> DEV size_t src_elem() { return SRC == SRC_I32 ? 4 : (SRC == SRC_U16 || SRC == SRC_PK16) ? 2 : 1; }
/* bytes from one sample of a component to the next */
template <int SRC> DEV int src_step() { return SRC == SRC_PK8 ? 3 : SRC == SRC_PK16 ? 6 : SRC == SRC_U16 ? 2 : 1; }

/* Byte i (0 .. 23) of six words / half h (0 .. 23) of twelve, paired into one
 * word. */
template <int I0, int I1> DEV uint32_t pick_bytes(const uint32_t* w) {
    return __byte_perm(w[I0 >> 2], w[I1 >> 2], (I0 & 3) | ((4 + (I1 & 3)) << 8)) & 0x00ff00ffu;
}
template <int H0, int H1> DEV uint32_t pick_halves(const uint32_t* w) {
    return __byte_perm(w[H0 >> 1], w[H1 >> 1], ((H0 & 1) ? 0x32 : 0x10) | ((H1 & 1) ? 0x7600 : 0x5400));
}

/* 8 samples of a component from address p (packed: of channel 0), two per
 * word (sample 2k in the low half of word k), by vector loads. */
template <int SRC>
DEV void load_samples8(const char* p, int chan, uint32_t* r) {
    if constexpr (SRC == SRC_U16) {
        const uint4 q = *(const uint4*)p;
        r[0] = q.x; r[1] = q.y; r[2] = q.z; r[3] = q.w;
    } else if constexpr (SRC == SRC_U8) {
        const uint2 q = *(const uint2*)p;
        r[0] = __byte_perm(q.x, 0, 0x4140);
        r[1] = __byte_perm(q.x, 0, 0x4342);
        r[2] = __byte_perm(q.y, 0, 0x4140);
        r[3] = __byte_perm(q.y, 0, 0x4342);
    } else if constexpr (SRC == SRC_PK8) {
        const uint2 a = *(const uint2*)p, b = *(const uint2*)(p + 8), c = *(const uint2*)(p + 16);
        const uint32_t w[6] = {a.x, a.y, b.x, b.y, c.x, c.y};
        if (chan == 0) {
            r[0] = pick_bytes<0, 3>(w); r[1] = pick_bytes<6, 9>(w); r[2] = pick_bytes<12, 15>(w); r[3] = pick_bytes<18, 21>(w);
        } else if (chan == 1) {
            r[0] = pick_bytes<1, 4>(w); r[1] = pick_bytes<7, 10>(w); r[2] = pick_bytes<13, 16>(w); r[3] = pick_bytes<19, 22>(w);
        } else {
            r[0] = pick_bytes<2, 5>(w); r[1] = pick_bytes<8, 11>(w); r[2] = pick_bytes<14, 17>(w); r[3] = pick_bytes<20, 23>(w);
        }
    } else {
        const uint4 a = *(const uint4*)p, b = *(const uint4*)(p + 16), c = *(const uint4*)(p + 32);
        const uint32_t w[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
        if (chan == 0) {
            r[0] = pick_halves<0, 3>(w); r[1] = pick_halves<6, 9>(w); r[2] = pick_halves<12, 15>(w); r[3] = pick_halves<18, 21>(w);
        } else if (chan == 1) {
            r[0] = pick_halves<1, 4>(w); r[1] = pick_halves<7, 10>(w); r[2] = pick_halves<13, 16>(w); r[3] = pick_halves<19, 22>(w);
        } else {
            r[0] = pick_halves<2, 5>(w); r[1] = pick_halves<8, 11>(w); r[2] = pick_halves<14, 17>(w); r[3] = pick_halves<20, 23>(w);
        }
    }
}

/* How a strip reads its rows. */
enum {
    LD_ALL = 0,     /* every lane's 8 columns inside the row, aligned rows */
    LD_WHOLE = 1,   /* every lane's 8 columns inside the row or all outside it, aligned rows */
    LD_ANY = 2      /* sample by sample */
};

/* A strip's input rows: the same for every lane but for off and left. */
struct FvLane {
    const char* base;   /* row 0 */
    size_t pitch;       /* bytes */
    uint32_t off;       /* of sample column c0 (packed: of channel 0; sample by sample: of the component) */
    int chan, left;     /* columns of the row from c0 on; <= 0: none */
};
template <int SRC, int LD>
DEV FvLane fv_lane(const void* src, long long pitch, int chan, int w, int c0) {
    FvLane S;
    S.base = (const char*)src;
    S.pitch = (size_t)pitch * src_elem<SRC>();
    S.off = (uint32_t)(c0 * src_step<SRC>() + (LD == LD_ANY ? chan * (int)src_elem<SRC>() : 0));
    S.chan = chan;
    S.left = c0 >= 0 ? w - c0 : 0;
    return S;
}
/* Row y's raw samples of the lane's columns, two per word; columns outside
 * the row read as 0 (the horizontal lifting never lets them into a result). */
template <int SRC, int LD>
DEV void fv_load(const FvLane& S, int y, uint32_t* r) {
    const char* p = S.base + (size_t)y * S.pitch + S.off;
    if constexpr (LD == LD_ALL) {
        load_samples8<SRC>(p, S.chan, r);
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++) r[k] = 0u;
        if constexpr (LD == LD_WHOLE) {
            if (S.left > 0) load_samples8<SRC>(p, S.chan, r);
        } else {
            const bool wide = SRC == SRC_U16 || SRC == SRC_PK16;
            uint32_t v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const char* a = p + k * src_step<SRC>();
                v[k] = 0u;
                if (k < S.left) v[k] = wide ? (uint32_t)*(const uint16_t*)a : (uint32_t)*(const uint8_t*)a;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) r[k] = v[2 * k] | (v[2 * k + 1] << 16);
        }
    }
}

/* One band's output of a strip: coefficient and GCLI rows advanced by one
 * band row per step (the same for every lane). */
struct FvBand {
    BandRow b;
    uint32_t pitch, gpitch;
};
DEV FvBand fv_band(const jxs_band_t& bd, int row, uint16_t* coef, uint8_t* gcli) {
    FvBand f;
    f.b = band_row(bd, row, coef, gcli);
    f.pitch = bd.pitch;
    f.gpitch = bd.gpitch;
    return f;
}
DEV void fv_next(FvBand& f) {
    f.b.crow += f.pitch;
    f.b.grow += f.gpitch;
}
/* The lane's group of a band row: coefficients j .. j + 3 (values v * mul);
 * see fh_emit. */
template <bool EDGE>
DEV void fv_emit(const FvBand& f, uint32_t j, const int32_t* v, uint32_t mul) {
    const uint32_t g = j >> 2;
    uint32_t c0, c1;
    if constexpr (EDGE) {
        const int left = f.b.w - (int)j;
        if ((int)g >= f.b.gw) return;
        c0 = sm_pair(v[0], left > 1 ? v[1] : 0, mul);
        c1 = sm_pair(left > 2 ? v[2] : 0, left > 3 ? v[3] : 0, mul);
    } else {
        c0 = sm_pair(v[0], v[1], mul);
        c1 = sm_pair(v[2], v[3], mul);
    }
    *(uint2*)(f.b.crow + j) = make_uint2(c0, c1);
    f.b.grow[g] = (uint8_t)gcli_of(c0, c1);
}

/* The first level of integer samples, in exact integers without a shift.
 * The scaled input v = X 2^(20-d) - 2^19 (d <= 14) has 20 - d >= 6 trailing
 * zero bits and this level's lifting divides by 2 and 4 once in each
 * direction, so that no rounding ever happens and
 *   D = 2 X[2i+1] - X[2i] - X[2i+2]    is the vertical high row x 2^(21-d),
 *   S = 8 X[2i] + D[i-1] + D[i]        the low row x 2^(17-d),
 * and the same again horizontally: HL x 2^(16-d), LL x 2^(14-d) (plus the
 * offset), HH x 2^(18-d), LH x 2^(16-d).  The vertical step works on two
 * columns per word: with a bias of 2 M (M = 2^d - 1) D lies in [0, 4 M], and
 * S then carries 4 M and lies in [2 M, 14 M], inside 16 bits up to d = 12;
 * deeper samples (WIDE) form S in 32 bits.
 *
 * Bound by memory once the integer pipes are relieved: 29 -> 21.5 thread
 * instructions per sample against lifting in 32 bits with shifts, and 8 4K
 * 4:2:2 10-bit frames in 106 us instead of 160 (580 MB of DRAM traffic, 5.4
 * TB/s).  Packed input is read 8 pixels at a time too, its three components
 * in strips of their own that share the lines in L2: 16 4K frames took 755
 * us sample by sample. */
template <int SRC, int LD, bool WIDE>
DEV void fv_strip_samples(const FwdVJob& J, int r0, int rend, int c0) {
    constexpr bool EDGE = LD != LD_ALL;
    const int lane = threadIdx.x & 31;
    const int h = J.h, n2 = h >> 1, d = J.depth;
    const FvLane S = fv_lane<SRC, LD>(J.src, J.src_pitch, J.chan, J.w, c0);
    const uint32_t M = (1u << d) - 1u, mask2 = M * 0x00010001u, bias = 2u * mask2;
    const bool masked = SRC == SRC_U16 || SRC == SRC_PK16; /* 8-bit samples have no bits above the depth */
    /* output: pairs jj .. jj + 3 of the level's bands (one group), lanes 1..30 */
    const uint32_t jj = (uint32_t)(c0 >> 1);
    const int rel = J.w - c0;
    const bool out_lane = lane >= 1 && lane <= 30 && rel > 0;
    const uint32_t mul4 = 1u << (16 - d), mul2 = 1u << (18 - d);
    const int32_t llmul = 1 << (14 - d), lloff = -(1 << 19) - 32 * (int32_t)M * llmul;
    FvBand bhl = fv_band(J.bands[J.b_hl], r0, J.coef, J.gcli);
    FvBand blh = fv_band(J.bands[J.b_lh], r0, J.coef, J.gcli);
    FvBand bhh = fv_band(J.bands[J.b_hh], r0, J.coef, J.gcli);
    const int ll_pitch = J.ll_pitch;
    int32_t* ll = J.ll + (size_t)r0 * ll_pitch;

    /* X[2 r0] and D[r0 - 1]; rows 2 r0 + 1, 2 r0 + 2 already in flight */
    uint32_t xe[4], ra[4], rb[4];
    uint32_t dp[WIDE ? 8 : 4];
    {
        uint32_t q0[4], q1[4];
        fv_load<SRC, LD>(S, fold_row(2 * r0 - 2, h), q0);
        fv_load<SRC, LD>(S, fold_row(2 * r0 - 1, h), q1);
        fv_load<SRC, LD>(S, 2 * r0, xe);
        fv_load<SRC, LD>(S, fold_row(2 * r0 + 1, h), ra);
        fv_load<SRC, LD>(S, fold_row(2 * r0 + 2, h), rb);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (masked) {
                q0[k] &= mask2;
                q1[k] &= mask2;
                xe[k] &= mask2;
            }
            const uint32_t t = 2u * q1[k] + (bias - q0[k] - xe[k]);
            if constexpr (WIDE) {
                dp[2 * k] = t & 0xffffu;
                dp[2 * k + 1] = t >> 16;
            } else {
                dp[k] = t;
            }
        }
    }
#pragma unroll 2
    for (int i = r0; i < rend; i++) {
        int32_t sv[8], dv[8];
        uint32_t xn[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t xo = masked ? ra[k] & mask2 : ra[k];
            xn[k] = masked ? rb[k] & mask2 : rb[k];
            const uint32_t t = 2u * xo + (bias - xe[k] - xn[k]);
            dv[2 * k] = (int32_t)(t & 0xffffu);
            dv[2 * k + 1] = (int32_t)(t >> 16);
            if constexpr (WIDE) {
                sv[2 * k] = 8 * (int32_t)(xe[k] & 0xffffu) + ((int32_t)dp[2 * k] + dv[2 * k]);
                sv[2 * k + 1] = 8 * (int32_t)(xe[k] >> 16) + ((int32_t)dp[2 * k + 1] + dv[2 * k + 1]);
                dp[2 * k] = (uint32_t)dv[2 * k];
                dp[2 * k + 1] = (uint32_t)dv[2 * k + 1];
            } else {
                const uint32_t u = 8u * xe[k] + (dp[k] + t);
                sv[2 * k] = (int32_t)(u & 0xffffu);
                sv[2 * k + 1] = (int32_t)(u >> 16);
                dp[k] = t;
            }
            xe[k] = xn[k];
        }
        if (i + 1 < rend) {
            fv_load<SRC, LD>(S, fold_row(2 * i + 3, h), ra);
            fv_load<SRC, LD>(S, fold_row(2 * i + 4, h), rb);
        }
        /* low row i: LL (int32, next level) and HL; high row i: LH and HH */
        int32_t lo[4], hi[4], lo2[4], hi2[4];
        fx_level<EDGE>(sv, c0, rel, lo, hi);
        fx_level<EDGE>(dv, c0, rel, lo2, hi2);
        if (out_lane) {
            fv_emit<EDGE>(bhl, jj, hi, mul4);
            /* rows are padded to a multiple of 4 */
            *(int4*)(ll + jj) =
                make_int4(lo[0] * llmul + lloff, lo[1] * llmul + lloff, lo[2] * llmul + lloff, lo[3] * llmul + lloff);
            if (i < n2) {
#pragma unroll
                for (int q = 0; q < 4; q++) lo2[q] -= 16 * (int32_t)M;
                fv_emit<EDGE>(blh, jj, lo2, mul4);
                fv_emit<EDGE>(bhh, jj, hi2, mul2);
            }
        }
        fv_next(bhl);
        fv_next(blh);
        fv_next(bhh);
        ll += ll_pitch;
    }
}

/* The lane's 8 columns of an int32 low band row (rows padded to a multiple
 * of 4). */
template <bool EDGE>
DEV void fv_load_i32(const int32_t* base, size_t pitch, int y, uint32_t c0, int left, int32_t* x) {
    const int32_t* p = base + (size_t)y * pitch + c0;
    int4 a = make_int4(0, 0, 0, 0), b = a;
    if (!EDGE || left > 0) a = *(const int4*)p;
    if (!EDGE || left > 4) b = *(const int4*)(p + 4);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}

/* A deeper level, on the int32 low band of the one above, where the lifting
 * rounds. */
template <bool EDGE>
DEV void fv_strip_i32(const FwdVJob& J, int r0, int rend, int c0) {
    const int lane = threadIdx.x & 31;
    const int h = J.h, n2 = h >> 1;
    const int32_t* src = (const int32_t*)J.src;
    const size_t pitch = (size_t)J.src_pitch;
    const uint32_t jj = (uint32_t)(c0 >> 1);
    const int rel = J.w - c0, left = c0 >= 0 ? rel : 0;
    const bool out_lane = lane >= 1 && lane <= 30 && rel > 0;
    FvBand bhl = fv_band(J.bands[J.b_hl], r0, J.coef, J.gcli);
    FvBand blh = fv_band(J.bands[J.b_lh], r0, J.coef, J.gcli);
    FvBand bhh = fv_band(J.bands[J.b_hh], r0, J.coef, J.gcli);
    const int ll_pitch = J.ll_pitch;
    int32_t* ll = J.ll + (size_t)r0 * ll_pitch;

    int32_t xe[8], dp[8], ra[8], rb[8];
    {
        int32_t q0[8], q1[8];
        fv_load_i32<EDGE>(src, pitch, fold_row(2 * r0 - 2, h), (uint32_t)c0, left, q0);
        fv_load_i32<EDGE>(src, pitch, fold_row(2 * r0 - 1, h), (uint32_t)c0, left, q1);
        fv_load_i32<EDGE>(src, pitch, 2 * r0, (uint32_t)c0, left, xe);
        fv_load_i32<EDGE>(src, pitch, fold_row(2 * r0 + 1, h), (uint32_t)c0, left, ra);
        fv_load_i32<EDGE>(src, pitch, fold_row(2 * r0 + 2, h), (uint32_t)c0, left, rb);
#pragma unroll
        for (int k = 0; k < 8; k++) dp[k] = q1[k] - ((q0[k] + xe[k]) >> 1);
    }
#pragma unroll 2
    for (int i = r0; i < rend; i++) {
        int32_t dv[8], sv[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            dv[k] = ra[k] - ((xe[k] + rb[k]) >> 1);
            sv[k] = xe[k] + ((dp[k] + dv[k] + 2) >> 2);
            xe[k] = rb[k];
            dp[k] = dv[k];
        }
        if (i + 1 < rend) {
            fv_load_i32<EDGE>(src, pitch, fold_row(2 * i + 3, h), (uint32_t)c0, left, ra);
            fv_load_i32<EDGE>(src, pitch, fold_row(2 * i + 4, h), (uint32_t)c0, left, rb);
        }
        int32_t lo[4], hi[4], lo2[4], hi2[4];
        fh_level<8, EDGE>(sv, c0, rel, lo, hi);
        fh_level<8, EDGE>(dv, c0, rel, lo2, hi2);
        if (out_lane) {
            fv_emit<EDGE>(bhl, jj, hi, 1u);
            *(int4*)(ll + jj) = make_int4(lo[0], lo[1], lo[2], lo[3]);
            if (i < n2) {
                fv_emit<EDGE>(blh, jj, lo2, 1u);
                fv_emit<EDGE>(bhh, jj, hi2, 1u);
            }
        }
        fv_next(bhl);
        fv_next(blh);
        fv_next(bhh);
        ll += ll_pitch;
    }
}

template <int SRC, int LD>
DEV void fv_strip(const FwdVJob& J, int r0, int rend, int c0) {
    if constexpr (SRC == SRC_I32) {
        fv_strip_i32<LD != LD_ALL>(J, r0, rend, c0);
    } else if constexpr (SRC == SRC_U16 || SRC == SRC_PK16) {
        if (J.depth > 12) fv_strip_samples<SRC, LD, true>(J, r0, rend, c0);
        else fv_strip_samples<SRC, LD, false>(J, r0, rend, c0);
    } else {
        fv_strip_samples<SRC, LD, false>(J, r0, rend, c0);
    }
}

template <int SRC, int NJ>
__global__ void __launch_bounds__(32, SRC == SRC_I32 ? 28 : 32) fwd_v_kernel(const __grid_constant__ FwdVLaunchN<NJ> L) {
    if (NJ <= JXS_MAXC) dep_wait();
    const FwdVJob& J = L.job[find_job<NJ>(L.job, L.njobs, (int)blockIdx.x)];
    const int u = blockIdx.x - J.first_block;
    const int ty = u / J.col_tiles, tx = u - ty * J.col_tiles;
    const int n1 = (J.h + 1) >> 1;
    const int r0 = ty * J.rp, rend = min(r0 + J.rp, n1);
    const int first = tx * FV_COLS, c0 = first - 8 + 8 * (int)threadIdx.x;
    /* the strip's 256 columns first - 8 .. first + 247 all inside: the
     * whole warp takes the path without checks */
    const bool inner = first >= 8 && first + FV_COLS + 8 <= J.w;
    if (SRC == SRC_I32) {
        if (inner) fv_strip<SRC, LD_ALL>(J, r0, rend, c0);
        else fv_strip<SRC, LD_WHOLE>(J, r0, rend, c0);
    } else if (J.vec && inner) {
        fv_strip<SRC, LD_ALL>(J, r0, rend, c0);
    } else if (J.vec && (J.w & 7) == 0) {
        fv_strip<SRC, LD_WHOLE>(J, r0, rend, c0);
    } else {
        fv_strip<SRC, LD_ANY>(J, r0, rend, c0);
    }
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
 * level: 8 such frames took 650 us, now 283 (1.24 GB; that step took their
 * encode from 3308 to 2907 us). */
#define FH_MAX_WARPS 4
#define FH_COLS 16

/* columns a warp's chunk yields */
static inline __host__ __device__ int fh_halo_lanes(int nh) { return nh >= 5 ? 4 : nh == 4 ? 2 : 1; }
static inline __host__ __device__ int fh_net_cols(int nh) { return FH_COLS * (32 - 2 * fh_halo_lanes(nh)); }

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
        const uint32_t mask = (1u << J.depth) - 1u;
        const int32_t mul = 1 << (20 - J.depth);
#pragma unroll
        for (int k = 0; k < FH_COLS; k += 8) {
            uint32_t q[4];
            if (J.vec && (J.w & 7) == 0) fv_load<SRC, LD_WHOLE>(fv_lane<SRC, LD_WHOLE>(J.src, J.src_pitch, J.chan, J.w, c0 + k), row, q);
            else fv_load<SRC, LD_ANY>(fv_lane<SRC, LD_ANY>(J.src, J.src_pitch, J.chan, J.w, c0 + k), row, q);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                x[k + 2 * i] = (int32_t)(q[i] & mask) * mul - (1 << 19);
                x[k + 2 * i + 1] = (int32_t)((q[i] >> 16) & mask) * mul - (1 << 19);
            }
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
    if (NJ <= JXS_MAXC) dep_wait();
    const FwdHJob& J = L.job[find_job<NJ>(L.job, L.njobs, (int)blockIdx.x)];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = (blockIdx.x - J.first_block) * L.rows_per_block + warp;
    const int row = unit / J.chunks, ch = unit - row * J.chunks;
    if (row >= J.h) return; /* the whole warp */
    const int halo = fh_halo_lanes(J.nh), first = ch * fh_net_cols(J.nh) - FH_COLS * halo;
    const int c0 = first + FH_COLS * lane;
    /* lanes past the row's end too: the last group of a deeper band, which
     * several lanes share, ends in theirs with zeros */
    const bool out_lane = lane >= halo && lane < 32 - halo;
    if (first >= 0 && first + 32 * FH_COLS <= J.w) fh_chunk<SRC, false>(J, row, c0, out_lane);
    else fh_chunk<SRC, true>(J, row, c0, out_lane);
}

/* ------------------------------------------------------------------------ */
/* launchers                                                                 */
/* ------------------------------------------------------------------------ */
extern "C" int jxs_fwd_v_tile_cols(void) { return FV_COLS; }
extern "C" int jxs_fwd_h_max_rows_per_block(void) { return FH_MAX_WARPS; }
extern "C" int jxs_fwd_h_chunk_cols(int nh) { return fh_net_cols(nh); }

template <int SRC, int NJ>
static cudaError_t launch_v(const FwdVLaunchN<NJ>* L, int grid_per_sm, cudaStream_t st) {
    (void)grid_per_sm; /* one block per tile */
    if (L->ntiles <= 0) return cudaSuccess;
    if (NJ > JXS_MAXC) {
        fwd_v_kernel<SRC, NJ><<<L->ntiles, 32, 0, st>>>(*L);
        return cudaGetLastError();
    }
    return jxs_launch(fwd_v_kernel<SRC, NJ>, dim3((unsigned)L->ntiles), (unsigned)(32), 0, st, *L);
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
    if (NJ > JXS_MAXC) {
        fwd_h_kernel<SRC, NJ><<<nblocks, L->rows_per_block * 32, 0, st>>>(*L);
        return cudaGetLastError();
    }
    return jxs_launch(fwd_h_kernel<SRC, NJ>, dim3((unsigned)nblocks), (unsigned)(L->rows_per_block * 32), 0, st, *L);
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
