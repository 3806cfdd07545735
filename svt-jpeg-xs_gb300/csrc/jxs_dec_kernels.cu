/*
 * Decoder kernels for sm_103a.
 *
 *  unpack_kernel   per precinct row: copies the precinct into shared memory,
 *                  parses its header and packet headers, decodes GCLIs (raw
 *                  nibbles or unary codes found by a block-wide scan of zero
 *                  bits), then all data groups at prefix-summed bit offsets,
 *                  dequantizes and writes int16 coefficients
 *                  (unpack_precinct, Packing.c:513-868; Dequant.c:9-57;
 *                  Precinct.c:9-29).
 *  walk_*_kernel   precinct offsets of a device-resident codestream.
 * The inverse transform is in jxs_inv_dwt.cu.
 */
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "jxs_core.h"
#include "jxs_kernels.cuh"

#define DEV __device__ __forceinline__

#define UK_THREADS 512
#define UK_WARPS (UK_THREADS / 32)
#define FULL 0xffffffffu
static_assert(JXS_MAXSEG <= UK_THREADS, "one thread per segment");
static_assert(UK_LIST_BYTES == 4 * 128 * UK_WARPS, "a list of 128 groups per warp");

/* Per band line of the precinct being unpacked. */
struct UkLine {
    uint8_t t, meth, vp, pk;    /* vp: GCLIs predicted from the line above */
};
/* Per packet. */
struct UkPk {
    uint32_t spos;              /* first bit after the packet header */
    uint32_t gpos, gbits;       /* GCLI sub-packet: bit position and length */
    uint32_t dpos, dbits;       /* data sub-packet */
    uint32_t sgpos, sgbits;     /* sign sub-packet (separate signs, Fs = 1) */
    uint32_t wbase, nwords;     /* its 32-bit words in the concatenated GCLI word list (VLC packets) */
    uint32_t zbase, nzero;      /* rank of its first zero bit among all VLC zeros; zeros in its range */
    uint32_t ncoded;            /* unary codewords */
    uint32_t rbase;             /* codewords with ones among all VLC zeros before it */
    uint32_t raw, present;
};
/* A segment as the warp passes read it: rank of its first codeword's zero
 * bit (raw packets: bit position of its first 4-bit GCLI), bit position of its
 * first significance flag, its first group's place among the precinct's
 * GCLIs, and group count | gtli << 16 | significance << 20 | raw << 21 |
 * predicted << 22 | band line << 24. */
struct UkSeg {
    uint32_t vpos, sig, z, info;
};

/* The precinct's bytes are kept as a bit string in 32-bit words, first bit in
 * the most significant position (bytes swapped once, when it is copied in):
 * 32 bits from bit `pos`, readable 8 bytes past pos / 8, and byte i. */
DEV uint32_t bits32_at(const uint32_t* b, uint32_t pos) {
    const uint32_t wi = pos >> 5;
    return __funnelshift_l(b[wi + 1], b[wi], pos & 31);
}
DEV uint32_t byte_of(const uint32_t* b, uint32_t i) { return ((const uint8_t*)b)[i ^ 3u]; }
DEV uint32_t shl_or_0(uint32_t a, uint32_t n) { /* 0 for n >= 32 */
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(n));
    return r;
}
/* all ones in every byte whose top bit is set */
DEV uint32_t sign_bytes(uint32_t x) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %1, 0xba98;" : "=r"(r) : "r"(x));
    return r;
}

/* Transpose of the 8 x 4 bit matrix in a word: bit 4k + j moves to bit
 * 8j + k (k: nibble = bit-plane, j: bit in the nibble), so that byte 3 - c
 * collects the 8 plane bits of coefficient c.  Four swaps of index bits
 * ((4,1), (3,0), (2,1), (1,0)) as masked delta swaps. */
DEV uint32_t dswap(uint32_t x, int d, uint32_t m) {
    const uint32_t t = ((x >> d) ^ x) & m;
    return x ^ (t * ((1u << d) + 1u)); /* t and t << d have no bit in common */
}
DEV uint32_t planes_to_coefs(uint32_t x) {
    x = dswap(x, 14, 0x0000ccccu);
    x = dswap(x, 7, 0x00aa00aau);
    x = dswap(x, 2, 0x0c0c0c0cu);
    return dswap(x, 1, 0x22222222u);
}

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

/* Block-wide exclusive scan of one counter; returns the block total.  ws is
 * free for another scan once every thread has passed a later barrier. */
DEV uint32_t block_scan1(uint32_t a, uint32_t* ea, uint32_t* ws) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t ia = warp_incl_scan(a);
    if (lane == 31) ws[warp] = ia;
    __syncthreads();
    /* every warp adds up the totals of the 16 */
    const uint32_t w = warp_incl_scan(lane < UK_WARPS ? ws[lane] : 0u);
    *ea = (warp ? __shfl_sync(FULL, w, warp - 1) : 0u) + ia - a;
    return __shfl_sync(FULL, w, 31);
}

/* Next segment for a warp from a shared queue (the warps balance segments
 * of different lengths between them). */
DEV uint32_t next_seg(uint32_t* ctr, int lane) {
    uint32_t v = 0;
    if (lane == 0) v = atomicAdd(ctr, 1u);
    return __shfl_sync(FULL, v, 0);
}

/* Per-packet exclusive running sums of one count per segment.  Segments
 * are numbered in packet order, so a segment's base inside its packet is the
 * block-wide exclusive sum up to it minus that of its packet's first
 * segment.  Thread i holds segment i's count and band line (nseg <=
 * blockDim.x) and gets its base; ex[0 .. nseg] receives the block-wide
 * exclusive sums, and threads k < npk get packet k's total in *sum (0 without
 * segments). */
DEV uint32_t seg_bases(uint32_t cnt, uint32_t bl, uint32_t nseg, uint32_t npk, const jxs_bline_t* bls, const uint8_t* pkbl0,
                       const uint8_t* pknbl, uint32_t* ex, uint32_t* ws, uint32_t* sum) {
    const uint32_t i = threadIdx.x;
    uint32_t e;
    const uint32_t total = block_scan1(i < nseg ? cnt : 0u, &e, ws);
    if (i < nseg) ex[i] = e;
    if (i == 0) ex[nseg] = total;
    __syncthreads();
    *sum = 0;
    if (i < npk && pknbl[i]) {
        const uint32_t b0 = pkbl0[i], lb = b0 + pknbl[i] - 1;
        *sum = ex[bls[lb].seg0 + bls[lb].nseg] - ex[bls[b0].seg0];
    }
    return i < nseg ? e - ex[bls[pkbl0[bls[bl].pk]].seg0] : 0u;
}

/* Data nibbles of a VLC packet's first n codewords (signs with the data): a
 * codeword of r > 0 ones stands for a group of r planes and its signs, so
 * they are the ones before the n-th zero bit and the codewords among them
 * that have ones (a zero bit after a one).  zpre / rpre: zeros and codewords
 * with ones before each thread's `per` words of the zeros pass. */
DEV uint32_t vlc_nibbles(const uint32_t* b, const UkPk& P, uint32_t n, const uint32_t* zpre, const uint32_t* rpre, uint32_t per) {
    if (!n) return 0;
    const uint32_t Z = P.zbase + n; /* the zero bits of all packets up to the n-th */
    uint32_t T = 0;
#pragma unroll 1
    for (uint32_t step = UK_THREADS / 2; step; step >>= 1)
        if (zpre[T + step] < Z) T += step;
    uint32_t i = 0, zeros = P.zbase, runs = P.rbase;
    if (T * per > P.wbase) {
        i = T * per - P.wbase;
        zeros = zpre[T];
        runs = rpre[T];
    }
    uint32_t z, before;
    for (;; i++) {
        const uint32_t at = P.gpos + 32 * i;
        z = ~bits32_at(b, at);
        before = i ? bits32_at(b, at - 1) : ~z >> 1; /* the bit before each */
        const uint32_t nz = __popc(z);
        if (zeros + nz >= Z || i + 1 >= P.nwords) break;
        zeros += nz;
        runs += __popc(z & before);
    }
    /* place of the last one in the word, by halves */
    uint32_t left = Z - zeros, y = z, pos = 0;
#pragma unroll
    for (int s = 16; s; s >>= 1) {
        const uint32_t c = __popc(y >> (32 - s));
        if (left > c) {
            left -= c;
            pos += s;
            y <<= s;
        }
    }
    runs += __popc(z & before & ~(0x7fffffffu >> pos));
    return 32 * i + pos + 1 - n + (runs - P.rbase);
}

/* Packet header fields (get_packet_header, ParseHeader.c:20-44): raw flag,
 * data, GCLI and sign sub-packet lengths in bytes; short (5-byte) or long
 * (7-byte) form. */
DEV void pk_header(const uint32_t* b, uint32_t at, int long_hdr, uint32_t& raw, uint32_t& dlen, uint32_t& glen, uint32_t& slen) {
    /* bytes 0-3 and 3-6 (or 1-4) */
    const uint32_t h = bits32_at(b, 8 * at), l = bits32_at(b, 8 * (at + (long_hdr ? 3 : 1)));
    raw = h >> 31;
    if (long_hdr) {
        /* 1 raw, 20 data, 20 GCLI, 15 sign bits */
        dlen = (h >> 11) & 0xfffffu;
        glen = ((h & 0x7ffu) << 9) | ((l >> 15) & 0x1ffu);
        slen = l & 0x7fffu;
    } else {
        /* 1 raw, 15 data, 13 GCLI, 11 sign bits */
        dlen = (h >> 16) & 0x7fffu;
        glen = (h >> 3) & 0x1fffu;
        slen = l & 0x7ffu;
    }
}

/* One group's coefficients from its data bits (unpack_data_c,
 * Packing.c:134-219): sign nibble (coefficient 0 in the most significant
 * bit), then bit-planes gcli-1 .. gtli; planes placed at << gtli
 * (Packing.c:117-132), deadzone or uniform dequantization (Dequant.c:9-57)
 * and sign-magnitude to two's complement (inv_sign_c, Precinct.c:9-14).
 * Returns the four int16 results packed two per word, coefficient 0 in the
 * low half of .x; coefficients at or past `wl` (remaining width) are 0. */
DEV uint2 group_finish(uint32_t A, uint32_t B, uint32_t sgn, uint32_t uniform, int wl);

/* The dequantized magnitudes of a group's four coefficients from its plane
 * bits, as 16-bit pairs: coefficients 0 | 1 << 16 in *A, 2 | 3 << 16 in *B.
 * The plane bits are planes v-1 .. gtli as nibbles, coefficient 0 in each
 * nibble's most significant bit (Packing.c:117-132), placed at << gtli, then
 * deadzone or uniform dequantization (Dequant.c:9-57).  Returns the mask of
 * non-zero magnitudes (bit 3 - c for coefficient c). */
DEV uint32_t group_mags(uint64_t planes, uint32_t np, uint32_t t, uint32_t gv, uint32_t uniform, uint32_t* A, uint32_t* B) {
    /* the plane bits of coefficients 0, 1 / 2, 3 as 16-bit pairs */
    const uint32_t tl = planes_to_coefs((uint32_t)planes);
    uint32_t P01 = __byte_perm(tl, 0u, 0x4243), P23 = __byte_perm(tl, 0u, 0x4041);
    if (np > 8) {
        const uint32_t th = planes_to_coefs((uint32_t)(planes >> 32));
        P01 |= __byte_perm(th, 0u, 0x4243) << 8;
        P23 |= __byte_perm(th, 0u, 0x4041) << 8;
    }
    const uint32_t nz01 = __vcmpne2(P01, 0u), nz23 = __vcmpne2(P23, 0u);
    const uint32_t nz = ((nz01 & 1u) << 3) | ((nz01 >> 16 & 1u) << 2) | ((nz23 & 1u) << 1) | (nz23 >> 16 & 1u);
    if (!uniform || t == 0) {
        /* two coefficients per word: m << t stays below 2^15 */
        uint32_t a = P01 << t, b = P23 << t;
        if (t > 0) {
            const uint32_t half = (1u << (t - 1)) * 0x00010001u;
            a |= __vcmpne2(a, 0u) & half;
            b |= __vcmpne2(b, 0u) & half;
        }
        *A = a;
        *B = b;
        return nz;
    }
    const uint32_t m[4] = {P01 & 0xffffu, P01 >> 16, P23 & 0xffffu, P23 >> 16};
    uint32_t o[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
        uint32_t mag = (m[c] << t) & 0xffffu;
        if (mag & 0x7fffu) {
            /* inv_quant_uniform (Dequant.c:23-43) */
            uint32_t val = mag & 0x7fffu, acc = 0;
            const uint32_t sc = gv - t + 1;
            for (; val > 0; val >>= sc) acc = (acc + val) & 0xffffu;
            mag = acc;
        }
        o[c] = mag;
    }
    *A = o[0] | (o[1] << 16);
    *B = o[2] | (o[3] << 16);
    return nz;
}

/* Sign-magnitude to two's complement (inv_sign_c, Precinct.c:9-14): sign
 * bit 3 - c of `sgn` for coefficient c; coefficients at or past `wl`
 * (remaining width) are 0.  Returns the four int16 results packed two per
 * word, coefficient 0 in the low half of .x. */
DEV uint2 group_finish(uint32_t A, uint32_t B, uint32_t sgn, uint32_t uniform, int wl) {
    const uint32_t keepA = (wl > 1 ? 0xffff0000u : 0u) | 0xffffu, keepB = (wl > 2 ? 0xffffu : 0u) | (wl > 3 ? 0xffff0000u : 0u);
    if (!uniform) {
        /* deadzone magnitudes stay below 2^15 */
        const uint32_t nA = ((sgn & 8u) ? 0xffffu : 0u) | ((sgn & 4u) ? 0xffff0000u : 0u);
        const uint32_t nB = ((sgn & 2u) ? 0xffffu : 0u) | ((sgn & 1u) ? 0xffff0000u : 0u);
        A = (A & ~nA) | (__vsub2(0u, A) & nA);
        B = (B & ~nB) | (__vsub2(0u, B) & nB);
        return make_uint2(A & keepA, B & keepB);
    }
    const uint32_t mg[4] = {A & 0xffffu, A >> 16, B & 0xffffu, B >> 16};
    uint32_t o[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const uint32_t sm = (mg[c] | (((sgn >> (3 - c)) & 1u) << 15)) & 0xffffu;
        o[c] = (uint32_t)((sm & 0x8000u) ? -(int32_t)(sm & 0x7fffu) : (int32_t)sm) & 0xffffu;
    }
    return make_uint2((o[0] | (o[1] << 16)) & keepA, (o[2] | (o[3] << 16)) & keepB);
}

/* One group's coefficients from its data bits with the signs joined to the
 * data (unpack_data_c, Packing.c:134-219): the sign nibble (coefficient 0 in
 * its most significant bit), then the plane nibbles. */
DEV uint2 decode_group(uint64_t chunk, uint32_t np, uint32_t t, uint32_t gv, uint32_t uniform, int wl) {
    const uint32_t sgn = (uint32_t)(chunk >> (4 * np)) & 15u;
    uint32_t A, B;
    group_mags(chunk & ((1ull << (4 * np)) - 1), np, t, gv, uniform, &A, &B);
    return group_finish(A, B, sgn, uniform && t != 0, wl);
}

/* Two coefficients of a group under deadzone quantization from their plane
 * bits P (16-bit halves, the sign as bit np above the magnitude), without a
 * comparison: `mag` has the np magnitude bits of both halves, `half` half a
 * step, 2^(t-1) (0 for t = 0), in both.  Magnitudes stay below 2^15, so that
 * adding 0x7fff sets bit 15 of the non-zero ones; a sign counts for those
 * only. */
DEV uint32_t dequant_pair(uint32_t P, uint32_t np, uint32_t t, uint32_t mag, uint32_t half) {
    uint32_t a = (P & mag) << t;
    const uint32_t u = a + 0x7fff7fffu;
    a |= (u >> (16 - t)) & half; /* deadzone reconstruction (Dequant.c:9-21) */
    const uint32_t neg = (P >> np) & (u >> 15) & 0x00010001u;
    return (a ^ (neg * 0xffffu)) + neg; /* two's complement (Precinct.c:9-14) */
}
DEV uint32_t be24(const uint8_t* p) { return ((uint32_t)p[0] << 16) | ((uint32_t)p[1] << 8) | p[2]; }

/* Offset of precinct p of a device codestream: its slice is expected where
 * the constant-bit-rate split of Lcod puts it (EncHandle.c:760-809), and the
 * 24-bit precinct lengths lead from there to p, three steps at most in slices
 * of 16 lines with two vertical levels.  False if the slice is not there. */
DEV bool find_precinct(const jxs_cfg_t* __restrict__ cfg, const uint8_t* bs, uint32_t size, uint32_t phb, uint32_t p,
                       uint32_t* out) {
    const uint32_t per = cfg->pps * cfg->ncol, s = p / per;
    uint64_t off = cfg->slice_begin[s];
    *out = 0;
    if (off + 6 > size) return false;
    /* its six bytes at once: byte after byte, each load would wait for the
     * comparison before it (2 % of a 3840x2160 frame's time) */
    const uint8_t* h = bs + off;
    const uint32_t at = ((uint32_t)h[0] << 24) | ((uint32_t)h[1] << 16) | ((uint32_t)h[2] << 8) | h[3], num = ((uint32_t)h[4] << 8) | h[5];
    if (at != 0xff200004u || num != s) return false;
    off += 6;
    for (uint32_t i = s * per; i < p; i++) {
        if (off + phb > size) return false;
        const uint32_t lprc = be24(bs + off);
        if (lprc > JXS_PREC_MAX_BYTES) return false;
        off += phb + lprc;
    }
    if (off + phb > size) return false;
    *out = (uint32_t)off;
    return true;
}
/* The same for the end of a slice's last precinct p: the next slice, or the
 * end of the codestream (true for the other precincts). */
DEV bool slice_ends(const jxs_cfg_t* __restrict__ cfg, const uint8_t* bs, uint32_t size, uint32_t p, uint64_t end) {
    const uint32_t per = cfg->pps * cfg->ncol, s = p / per;
    if (p + 1 == cfg->nprec) return end + 2 <= size && (((uint32_t)bs[end] << 8) | bs[end + 1]) == 0xff11u;
    return p + 1 != (s + 1) * per || end == cfg->slice_begin[s + 1];
}

/* unpack_precinct (Packing.c:513-868) for one precinct.  FS: the launch may
 * hold frames with separate sign sub-packets; VP: slice-ordered decoding,
 * which resolves vertical prediction (otherwise a precinct with predicted
 * bands reports JXS_E_DEC_VPRED); both compiled out otherwise.  BATCH: a
 * launch of many frames.
 *
 * Dynamic shared memory: see uk_layout.
 *
 *   copy    the precinct's bytes into shared memory as big-endian words;
 *   parse   warp 0: precinct header, band modes, packet headers, sub-packet
 *           positions with the reference's length checks, running sums of
 *           the lines' significance and raw GCLI bits;
 *   counts  thread per segment: groups with a unary codeword (the
 *           significance flags drop the insignificant ones);
 *   zeros   block pass over the VLC sub-packets: codeword c of a packet ends
 *           at the c-th zero bit of its sub-packet (unpack_pred_zero_gclis_*,
 *           Packing.c:435-511); its value, the ones before that bit, goes to
 *           byte c of a table;
 *   bases   signs with the data, no prediction: thread per segment, the data
 *           nibbles before it by a search in the unary codes' bits;
 *   pass 2  otherwise, warp per segment: GCLI = gtli + codeword value, or raw;
 *           prediction; data bits; running sums of these;
 *   pass 3  warp per segment: GCLIs (bases), data bits at warp-scanned
 *           offsets, decoded and written as int16 coefficients (8 bytes per
 *           lane, coalesced).
 *
 * Bound by instruction issue.  Segments are described once, a 16-byte record
 * each, instead of by every warp that takes one; codeword values are read 4
 * at a time instead of 5 zero positions; bytes are swapped once.  8 4K 4:2:2
 * 10-bit frames: 263 us before, 223 us so; 203 us with the segments' data
 * positions from the codes' bits instead of from a pass over all GCLIs. */
template <bool FS, bool VP, bool BATCH>
__device__ __forceinline__ void unpack_body(const jxs_cfg_t* __restrict__ cfg, const uint8_t* bs, uint32_t bs_size,
                                            const uint32_t* prec_off, int16_t* coef,
                                            uint32_t cap_bytes, uint32_t cap_groups, uint32_t cap_seg, int* status, const int p,
                                            uint8_t* top_gcl, uint8_t* top_t, const int vp_ok, const int rank = 0,
                                            const int turns = 0) {
    extern __shared__ __align__(16) uint8_t dsm[];
    /* signs with the data, no prediction: the segments' data positions come
     * from the unary codes' bits and the GCLIs are read in the data pass */
    constexpr bool LEAN = !FS && !VP;
    const UkLayout UL = uk_layout(cap_bytes, cap_groups, cap_seg, LEAN);
    uint32_t* pbuf = (uint32_t*)dsm;
    uint8_t* gcl = dsm + UL.gcl;
    uint8_t* zval = dsm + UL.zval;
    uint32_t* zpre = (uint32_t*)(dsm + UL.list); /* LEAN, until the data pass: see vlc_nibbles */
    uint32_t* rpre = zpre + UK_THREADS;
    /* zero bits: one per codeword plus up to 7 padding bits per packet */
    const uint32_t zcap = UK_ZCAP(cap_groups);
    __shared__ UkLine ln[JXS_MAXBLINES];
    __shared__ UkPk pk[JXS_MAXPK];
    __shared__ uint8_t s_mode[JXS_MAXBL];
    __shared__ uint32_t s_hpos[JXS_MAXPK];
    __shared__ uint32_t s_next[2]; /* segment queues of the two warp passes */
    /* per segment (dynamic: sized for the launch's largest segment count) */
    uint16_t* s_ord = (uint16_t*)(dsm + UL.ord);
    UkSeg* s_desc = (UkSeg*)(dsm + UL.desc);
    uint32_t* s_cnt = (uint32_t*)(dsm + UL.cnt);   /* data bits (LEAN: of raw packets); separate signs: then signs */
    uint32_t* s_base = (uint32_t*)(dsm + UL.base); /* bit position of the data */
    uint32_t* s_ex = (uint32_t*)(dsm + UL.ex);
    uint32_t* s_sgb = (uint32_t*)(dsm + UL.sgb);   /* separate signs: bit position of the signs */
    /* this precinct kind's tables, staged from the configuration */
    __shared__ jxs_bline_t s_bl[JXS_MAXBLINES];
    __shared__ uint64_t s_crow[JXS_MAXBLINES]; /* per line: coefficient row offset, less 4 times the line's first group */
    __shared__ uint32_t s_wend[JXS_MAXBLINES]; /* per line: coefficients, plus 4 times the line's first group */
    __shared__ uint32_t s_lsx[JXS_MAXBLINES + 1], s_lrx[JXS_MAXBLINES + 1]; /* per line: significance / raw GCLI bits before it */
    __shared__ uint8_t s_pkbl0[JXS_MAXPK], s_pknbl[JXS_MAXPK];
    __shared__ uint32_t ws[UK_WARPS], ws2[UK_WARPS];
    __shared__ int s_err;
    __shared__ uint32_t s_total, s_lead, s_tw, s_off;
    __shared__ uint8_t s_g2f[JXS_MAXBL];          /* global band -> flat band */
    __shared__ uint16_t s_lgp[JXS_MAXBLINES];      /* per line: band gain | priority << 8 */
    __shared__ uint32_t s_sc[9];                   /* nbands_all, npk, long headers, separate signs, precinct header bytes,
                                                      band lines, segments, groups per segment, run mode */
    __shared__ uint8_t s_topbl[VP ? JXS_MAXBLINES : 1], s_topprev[VP ? JXS_MAXBLINES : 1]; /* vertical prediction: the line above */
    __shared__ uint32_t s_topg[VP ? JXS_MAXBLINES : 1];
    __shared__ int s_hasvp, s_hasraw;

    /* the precinct kind's tables (last row / last of several columns) */
    const int last = jxs_pkind(cfg, (uint32_t)p);
    const uint32_t prow = (uint32_t)p / cfg->ncol, pcol = (uint32_t)p - prow * cfg->ncol;
    const int one_col = cfg->ncol == 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    /* the frame's status and the precinct's length field, by a warp that has
     * little to stage */
    auto begin = [&]() {
        if (threadIdx.x == UK_THREADS - 32) {
            /* the precinct's offset and length field are read in bounds before
             * the frame status, so that the three loads do not wait in turn */
            const uint32_t phb = cfg->prec_hdr_bytes;
            uint32_t off;
            bool lost = false;
            if (BATCH || prec_off) off = prec_off[p];
            else lost = !find_precinct(cfg, bs, bs_size, phb, (uint32_t)p, &off);
            s_off = off; /* read once: the offsets may be in host memory */
            const bool inb = (uint64_t)off + phb <= bs_size;
            const uint32_t lprc = inb ? ((uint32_t)bs[off] << 16) | ((uint32_t)bs[off + 1] << 8) | bs[off + 2] : 0u;
            if (!BATCH && !prec_off && (lost || !slice_ends(cfg, bs, bs_size, (uint32_t)p, (uint64_t)off + phb + lprc))) {
                /* the frame is decoded again, its precincts located first */
                atomicExch(status + 1, 1);
                s_err = -1;
                return;
            }
            int err = *(volatile int*)status; /* set: the precinct offsets could not be found */
            if (!err) {
                if (!inb) {
                    err = JXS_E_DEC_SHORT;
                } else {
                    s_total = phb + lprc;
                    s_lead = (uint32_t)((uintptr_t)(bs + off) & 15);
                    if (lprc > JXS_PREC_MAX_BYTES || s_total + 48 > cap_bytes) err = JXS_E_DEC_BITSTREAM;
                    else if ((uint64_t)off + s_total > bs_size) err = JXS_E_DEC_SHORT;
                }
                if (err) JXS_STATUS_SET(status, err);
            } else {
                err = -1; /* already reported */
            }
            s_err = err;
        }
    };
    /* BATCH: an ordinary launch, these first; else the tables first, which need
     * not wait for the kernel before */
    if (BATCH) begin();
    /* every thread stages this precinct kind's tables and the scalars the
     * parse needs, so that no single-warp phase waits on device memory */
    if (threadIdx.x == 0) {
        s_sc[0] = cfg->nbands_all;
        s_sc[1] = cfg->npk;
        s_sc[2] = cfg->lh || !cfg->short_hdr;
        s_sc[3] = cfg->fs;
        s_sc[4] = cfg->prec_hdr_bytes;
        s_sc[5] = cfg->nbline[last];
        s_sc[6] = cfg->nseg[last];
        s_sc[7] = cfg->seg_groups;
        s_sc[8] = cfg->rm;
        s_hasvp = 0;
    }
    if (threadIdx.x < 2) s_next[threadIdx.x] = 0;
    jxs_seg_t myseg; /* thread i: segment i */
    myseg.bl = 0;
    myseg.g0 = 0;
    {
        const uint32_t ns = cfg->nseg[last], nl = cfg->nbline[last];
        if (threadIdx.x < ns) {
            myseg = cfg->seg[last][threadIdx.x];
            s_ord[threadIdx.x] = cfg->seg_ord[last][threadIdx.x];
        }
        for (uint32_t i = threadIdx.x; i < nl * (sizeof(jxs_bline_t) / 4); i += blockDim.x)
            ((uint32_t*)s_bl)[i] = ((const uint32_t*)cfg->bline[last])[i];
        for (uint32_t x = threadIdx.x; x < nl; x += blockDim.x) {
            const jxs_bline_t& B = cfg->bline[last][x];
            const jxs_band_t& bd = cfg->band[B.fb];
            s_crow[x] = bd.coef_off + (uint64_t)(prow * bd.lines + B.line) * bd.pitch + (uint64_t)pcol * bd.cwn - 4 * (uint64_t)B.gbase;
            s_wend[x] = B.w + 4 * B.gbase;
            s_lgp[x] = (uint16_t)(bd.gain | (bd.prio << 8));
            if (VP) {
                s_topbl[x] = cfg->top_bl[last][x];
                s_topprev[x] = cfg->top_prev[last][x];
                s_topg[x] = cfg->top_gbase[last][x];
            }
        }
        for (uint32_t k = threadIdx.x; k < cfg->npk; k += blockDim.x) {
            s_pkbl0[k] = cfg->pk_bl0[last][k];
            s_pknbl[k] = cfg->pk_nbl[last][k];
        }
        for (uint32_t gb = threadIdx.x; gb < cfg->nbands_all; gb += blockDim.x) s_g2f[gb] = cfg->g2f[gb];
    }
    /* up to here configuration only */
    if (!BATCH) {
        dep_wait();
        begin();
    }
    __syncthreads();
    /* VP: a row that fails before its turn leaves it, and the others', in step */
    auto leave = [&]() {
        if constexpr (VP)
            for (int i = 0; i < turns; i++) cooperative_groups::this_cluster().sync();
    };
    if (s_err) {
        leave();
        return;
    }
    const uint32_t off = s_off;
    const uint32_t total = s_total, lead = s_lead;
    {
        /* aligned 16-byte chunks inside the precinct, single bytes at its
         * ends; 32 zero bytes after it for the bit readers */
        const uint8_t* gsrc = bs + off - lead;
        const uint32_t nbytes = lead + total, nch = (nbytes + 15) >> 4;
        for (uint32_t c = threadIdx.x; c < nch + 2; c += blockDim.x) {
            const uint32_t b0 = c << 4;
            if (b0 >= lead && b0 + 16 <= nbytes) {
                const uint4 v = *(const uint4*)(gsrc + b0);
                *(uint4*)(pbuf + 4 * c) = make_uint4(__byte_perm(v.x, 0u, 0x0123), __byte_perm(v.y, 0u, 0x0123),
                                                     __byte_perm(v.z, 0u, 0x0123), __byte_perm(v.w, 0u, 0x0123));
            } else {
                for (uint32_t i = b0; i < b0 + 16; i++) ((uint8_t*)pbuf)[i ^ 3u] = (i >= lead && i < nbytes) ? gsrc[i] : 0;
            }
        }
    }
    __syncthreads();

    const uint32_t nbl = s_sc[5], nseg = s_sc[6], SG = s_sc[7], npk = s_sc[1];
    const jxs_bline_t* bls = s_bl;
    /* parse, by warp 0: band modes and per-line fields in parallel, the
     * packet headers in order by lane 0 */
    if (warp == 0) {
        const uint32_t q = byte_of(pbuf, lead + 3), r = byte_of(pbuf, lead + 4);
        int err = 0, vp_seen = 0;
        /* band coding modes D[p,b], 2 bits per existing band */
        uint32_t idx0 = 0;
        const uint32_t nbands_all = s_sc[0];
        for (uint32_t gb0 = 0; gb0 < nbands_all; gb0 += 32) {
            const uint32_t gb = gb0 + lane;
            const int fb = gb < nbands_all ? s_g2f[gb] : JXS_NOBAND;
            const bool ex = fb != JXS_NOBAND;
            const uint32_t bal = __ballot_sync(FULL, ex);
            if (ex) {
                const uint32_t pos = 8 * lead + 40 + 2 * (idx0 + __popc(bal & ((1u << lane) - 1)));
                s_mode[fb] = (uint8_t)((pbuf[pos >> 5] >> (30 - (pos & 31))) & 3);
                /* vertical prediction: resolved here when the precinct row
                 * above is known (slice-ordered decoding), else the frame is
                 * decoded again that way; never in a slice's first row */
                if (s_mode[fb] & 1) vp_seen = 1;
            }
            idx0 += __popc(bal);
        }
        __syncwarp();
        /* per line, each lane a run of them: gtli and method, and the
         * significance flags and raw GCLI bits before it */
        {
            const uint32_t per = (nbl + 31) >> 5, x0 = min(nbl, per * lane), x1 = min(nbl, x0 + per);
            uint32_t sg = 0, rw = 0;
            for (uint32_t x = x0; x < x1; x++) {
                const uint32_t m = s_mode[bls[x].fb];
                ln[x].t = jxs_truncation((uint8_t)(s_lgp[x] & 255u), (uint8_t)(s_lgp[x] >> 8), (uint8_t)q, (uint8_t)r);
                ln[x].meth = (m & 2) ? 1 : 0;
                ln[x].vp = (m & 1) ? 1 : 0;
                ln[x].pk = bls[x].pk;
                sg += (m & 2) ? bls[x].sig_w : 0u;
                rw += 4 * bls[x].gcli_w;
            }
            uint32_t tsg, trw;
            sg = warp_excl_scan(sg, &tsg);
            rw = warp_excl_scan(rw, &trw);
            for (uint32_t x = x0; x < x1; x++) {
                s_lsx[x] = sg;
                s_lrx[x] = rw;
                sg += ln[x].meth ? bls[x].sig_w : 0u;
                rw += 4 * bls[x].gcli_w;
            }
            if (lane == 0) {
                s_lsx[nbl] = tsg;
                s_lrx[nbl] = trw;
            }
        }
        __syncwarp();
        /* per packet: significance bytes and raw GCLI bits it must hold */
        const bool here = lane < (int)npk && s_pknbl[lane];
        uint32_t sB = 0, rb = 0;
        if (here) {
            const uint32_t b0 = s_pkbl0[lane], b1 = b0 + s_pknbl[lane];
            sB = (s_lsx[b1] - s_lsx[b0] + 7) >> 3;
            rb = s_lrx[b1] - s_lrx[b0];
        }
        /* packet headers: the warp follows the chain of header positions
         * only; one lane per packet then reads its header again and derives
         * its sub-packet positions with the reference's checks (every check
         * bounds the running position, so testing each packet's own end
         * against the precinct's end is equivalent) */
        const int long_hdr = (int)s_sc[2];
        const uint32_t hb = long_hdr ? 7u : 5u, pend_max = lead + total;
        {
            const uint32_t have = __ballot_sync(FULL, here);
            uint32_t bpos = lead + s_sc[4], mine = 0; /* bytes */
            for (uint32_t left = have; left; left &= left - 1) {
                const int k = __ffs((int)left) - 1;
                if (bpos + hb > pend_max) {
                    err = JXS_E_DEC_BITSTREAM;
                    break;
                }
                uint32_t raw, dlen, glen, slen;
                pk_header(pbuf, bpos, long_hdr, raw, dlen, glen, slen);
                if (lane == k) mine = bpos;
                const uint32_t sBk = __shfl_sync(FULL, sB, k);
                bpos += hb + (raw ? 0u : sBk) + glen + dlen + slen;
            }
            if (lane < JXS_MAXPK) s_hpos[lane] = mine;
        }
        uint32_t nwords = 0;
        if (lane < (int)npk) {
            UkPk& P = pk[lane];
            P.present = 0;
            P.gbits = P.dbits = P.ncoded = P.nzero = 0;
            P.raw = 0;
            if (!err && here) {
                uint32_t raw, dlen, glen, slen;
                const uint32_t b = s_hpos[lane] + hb;
                pk_header(pbuf, s_hpos[lane], long_hdr, raw, dlen, glen, slen);
                uint32_t gp = b;
                if (raw) {
                    if (rb > glen * 8) err = JXS_E_DEC_BITSTREAM;
                } else {
                    gp += sB;
                    /* unary codes longer than this are refused */
                    if (glen * 8 > 65535u) err = JXS_E_DEC_BITSTREAM;
                }
                if ((uint64_t)gp + glen + dlen + slen > pend_max) err = JXS_E_DEC_BITSTREAM;
                P.raw = raw;
                P.spos = b * 8;
                P.gpos = gp * 8;
                P.gbits = glen * 8;
                P.dpos = (gp + glen) * 8;
                P.dbits = dlen * 8;
                P.sgpos = (gp + glen + dlen) * 8;
                P.sgbits = slen * 8;
                P.present = 1;
                if (!raw) nwords = (P.gbits + 31) >> 5;
            }
        }
        {
            uint32_t tw;
            const uint32_t wb = warp_excl_scan(nwords, &tw);
            if (lane < (int)npk) {
                pk[lane].wbase = wb;
                pk[lane].nwords = nwords;
            }
            if (lane == 0) s_tw = tw;
        }
        if (LEAN) {
            const bool any_raw = __any_sync(FULL, lane < (int)npk && pk[min(lane, JXS_MAXPK - 1)].raw);
            if (lane == 0) s_hasraw = any_raw;
        }
        err = __reduce_or_sync(FULL, (uint32_t)err) ? JXS_E_DEC_BITSTREAM : 0;
        if (!err && __any_sync(FULL, vp_seen)) {
            if (!VP) err = JXS_E_DEC_VPRED;
            else if (!vp_ok) err = JXS_E_DEC_BITSTREAM; /* no precinct row above to predict from */
        }
        __syncwarp();
        if (VP && !err) {
            bool hv = false;
            for (uint32_t x = lane; x < nbl; x += 32) {
                if (pk[ln[x].pk].raw) ln[x].vp = 0;
                hv |= ln[x].vp != 0;
            }
            if (__any_sync(FULL, hv) && lane == 0) s_hasvp = 1;
        }
        if (lane == 0) s_err = err;
    }
    __syncthreads();
    if (s_err) {
        if (threadIdx.x == 0) JXS_STATUS_SET(status, s_err);
        leave();
        return;
    }

    /* codewords of every segment, one thread each: its groups minus those
     * in insignificant significance groups (flags: 1 = insignificant); then
     * the codeword base of every segment inside its packet */
    const uint32_t tw = s_tw;
    uint32_t cwbase, sigpos = 0;
    {
        uint32_t cnt = 0;
        if (threadIdx.x < nseg) {
            const jxs_bline_t& B = bls[myseg.bl];
            const UkPk& P = pk[B.pk];
            const uint32_t gend = min(myseg.g0 + SG, B.gcli_w);
            if (!P.raw) {
                cnt = gend - myseg.g0;
                if (ln[myseg.bl].meth) {
                    sigpos = P.spos + s_lsx[myseg.bl] - s_lsx[s_pkbl0[B.pk]] + (myseg.g0 >> 3);
                    for (uint32_t s0 = myseg.g0 >> 3; s0 < ((gend + 7) >> 3); s0 += 32) {
                        const uint32_t ns = min(32u, ((gend + 7) >> 3) - s0);
                        const uint32_t fl = bits32_at(pbuf, sigpos + s0 - (myseg.g0 >> 3)) >> (32 - ns);
                        cnt -= 8 * __popc(fl);
                        /* a flagged partial last group counts its own size */
                        if ((fl & 1u) && 8 * (s0 + ns) > B.gcli_w) cnt += 8 * (s0 + ns) - B.gcli_w;
                    }
                }
            }
        }
        uint32_t ncoded;
        cwbase = seg_bases(cnt, myseg.bl, nseg, npk, bls, s_pkbl0, s_pknbl, s_ex, ws, &ncoded);
        if (threadIdx.x < npk) pk[threadIdx.x].ncoded = ncoded;
        __syncthreads();
    }

    /* zero bits of the VLC sub-packets: count, scan, record the codeword
     * values.  A thread's first word finds its packet by binary search over
     * the packets' word ranges (contiguous, in packet order; a packet without
     * VLC words has an empty range), later words step forward. */
    const uint32_t per = (tw + blockDim.x - 1) / blockDim.x;
    const uint32_t wa = min(tw, threadIdx.x * per), we = min(tw, wa + per);
    uint32_t k0 = 0;
    if (wa < we) {
        uint32_t lo = 0, hi = npk - 1; /* the first packet whose range ends past wa */
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (pk[mid].wbase + pk[mid].nwords > wa) hi = mid;
            else lo = mid + 1;
        }
        k0 = lo;
    }
    uint32_t zc = 0, nc = 0; /* zeros; of them after a one */
    {
        uint32_t k = k0;
        for (uint32_t wi = wa; wi < we; wi++) {
            while (k + 1 < npk && wi >= pk[k].wbase + pk[k].nwords) k++;
            const uint32_t i = wi - pk[k].wbase;
            const uint32_t valid = min(32u, pk[k].gbits - 32 * i);
            uint32_t z = ~bits32_at(pbuf, pk[k].gpos + 32 * i);
            const uint32_t before = !LEAN ? 0u : i ? bits32_at(pbuf, pk[k].gpos + 32 * i - 1) : ~z >> 1;
            if (valid < 32) z &= ~(0xffffffffu >> valid);
            if (LEAN && i == 0) pk[k].rbase = nc;
            zc += __popc(z);
            nc += __popc(z & before);
        }
    }
    uint32_t z0, r0 = 0;
    const uint32_t ztotal = block_scan1(zc, &z0, ws);
    if (LEAN) {
        (void)block_scan1(nc, &r0, ws2);
        zpre[threadIdx.x] = z0;
        rpre[threadIdx.x] = r0;
    }
    {
        uint32_t k = k0, ones = 0; /* ones since the last zero bit */
        for (uint32_t wi = wa; wi < we; wi++) {
            while (k + 1 < npk && wi >= pk[k].wbase + pk[k].nwords) k++;
            const uint32_t i = wi - pk[k].wbase, at = pk[k].gpos + 32 * i;
            if (i == 0) {
                pk[k].zbase = z0;
                if (LEAN) pk[k].rbase += r0;
                ones = 0;
            } else if (wi == wa) {
                /* the end of the word before (32 ones: no valid codeword is
                 * that long) */
                const uint32_t zp = ~bits32_at(pbuf, at - 32);
                ones = zp ? (uint32_t)__ffs((int)zp) - 1 : 32u;
            }
            const uint32_t valid = min(32u, pk[k].gbits - 32 * i);
            uint32_t z = ~bits32_at(pbuf, at);
            if (valid < 32) z &= ~(0xffffffffu >> valid);
            const uint32_t tail = z ? (uint32_t)__ffs((int)z) - 1 : min(ones + 32u, 64u);
            const uint32_t nz = __popc(z);
            uint8_t* o = zval + z0;
            for (uint32_t k2 = z0 < zcap ? min(nz, zcap - z0) : 0u; k2; k2--) {
                const uint32_t run = __clz((int)z);
                *o++ = (uint8_t)(ones + run);
                ones = 0;
                z = shl_or_0(z, run + 1);
            }
            z0 += nz;
            ones = tail;
        }
    }
    __syncthreads();
    if (warp == 0) {
        /* zeros of each VLC packet: up to the next VLC packet's first zero */
        const uint32_t k = lane;
        const bool vlc = k < npk && pk[k].present && !pk[k].raw && pk[k].nwords;
        const uint32_t zb = vlc ? pk[k].zbase : 0u;
        const uint32_t later = __ballot_sync(FULL, vlc) & ~((2u << k) - 1u);
        const uint32_t zn = __shfl_sync(FULL, zb, later ? __ffs(later) - 1 : 0);
        const uint32_t znext = later ? zn : ztotal;
        bool bad_pk = false;
        if (k < npk && pk[k].present && !pk[k].raw) {
            UkPk& P = pk[k];
            if (!P.nwords) {
                P.zbase = 0;
                P.nzero = 0;
            } else {
                P.nzero = znext - P.zbase;
            }
            bad_pk = P.ncoded > P.nzero || (P.ncoded && P.zbase + P.ncoded > zcap);
        }
        if (lane == 0) s_err = 0;
        __syncwarp();
        if (__any_sync(FULL, bad_pk) && lane == 0) s_err = JXS_E_DEC_BITSTREAM;
    }
    __syncthreads();
    if (s_err) {
        if (threadIdx.x == 0) JXS_STATUS_SET(status, s_err);
        leave();
        return;
    }
    /* the segments' records */
    if (threadIdx.x < nseg) {
        const jxs_bline_t& B = bls[myseg.bl];
        const UkLine L = ln[myseg.bl];
        const UkPk& P = pk[B.pk];
        UkSeg D;
        D.vpos = P.raw ? P.spos + s_lrx[myseg.bl] - s_lrx[s_pkbl0[B.pk]] + 4 * myseg.g0 : P.zbase + cwbase;
        D.sig = sigpos;
        D.z = B.gbase + myseg.g0;
        D.info = min(SG, B.gcli_w - myseg.g0) | ((uint32_t)L.t << 16) | ((P.raw ? 0u : (uint32_t)L.meth) << 20) | (P.raw << 21) |
                 (VP ? (uint32_t)L.vp << 22 : 0u) | ((uint32_t)myseg.bl << 24);
        s_desc[threadIdx.x] = D;
    }
    int bad = 0;
    if constexpr (LEAN) {
        /* data position of every segment, then of every packet's end */
        bool bad_pk = false;
        for (uint32_t j = threadIdx.x; j < nseg + npk; j += UK_THREADS) {
            const uint32_t k = j < nseg ? bls[myseg.bl].pk : j - nseg;
            const UkPk& P = pk[k];
            const bool vlc = P.present && !P.raw;
            const uint32_t bits = vlc ? 4 * vlc_nibbles(pbuf, P, j < nseg ? cwbase : P.ncoded, zpre, rpre, per) : 0u;
            if (j < nseg) s_base[j] = P.dpos + bits;
            else bad_pk |= vlc && bits > P.dbits;
        }
        if (__syncthreads_or(bad_pk)) {
            if (threadIdx.x == 0) JXS_STATUS_SET(status, JXS_E_DEC_BITSTREAM);
            return;
        }
        if (s_hasraw) {
            /* raw packets: from their GCLIs, a warp per segment */
            for (uint32_t sidx = warp; sidx < nseg; sidx += UK_WARPS) {
                const UkSeg D = s_desc[sidx];
                const uint32_t n = D.info & 0xffffu, t = (D.info >> 16) & 15u;
                uint32_t nib = 0;
                if ((D.info >> 21) & 1u)
                    for (uint32_t g = lane; g < n; g += 32) {
                        const uint32_t v = bits32_at(pbuf, D.vpos + 4 * g) >> 28;
                        nib += v > t ? v - t + 1 : 0u;
                    }
                nib = __reduce_add_sync(FULL, nib);
                if (lane == 0) s_cnt[sidx] = 4 * nib;
            }
            __syncthreads();
            uint32_t dbits;
            const uint32_t b = seg_bases(threadIdx.x < nseg ? s_cnt[threadIdx.x] : 0u, myseg.bl, nseg, npk, bls, s_pkbl0, s_pknbl, s_ex,
                                         ws, &dbits);
            if (threadIdx.x < nseg && pk[bls[myseg.bl].pk].raw) s_base[threadIdx.x] = pk[bls[myseg.bl].pk].dpos + b;
            if (__syncthreads_or(threadIdx.x < npk && pk[threadIdx.x].present && pk[threadIdx.x].raw && dbits > pk[threadIdx.x].dbits)) {
                if (threadIdx.x == 0) JXS_STATUS_SET(status, JXS_E_DEC_BITSTREAM);
                return;
            }
        }
    }
    const uint32_t lt_mask = (1u << lane) - 1u;
    /* a group's data: its sign nibble (signs with the data) and its planes */
    const uint32_t fs = FS ? s_sc[3] : 0u;
    if constexpr (!LEAN) {
    __syncthreads();

    /* pass 2: GCLIs from codeword values; data bits per segment.  Each lane
     * takes 4 consecutive groups: they share one significance flag, so
     * either all of them carry a codeword or none (only the segment's last
     * lane may hold fewer than 4 groups, and no lane after it holds any). */
    for (uint32_t qi = next_seg(&s_next[0], lane); qi < nseg; qi = next_seg(&s_next[0], lane)) {
        const uint32_t sidx = s_ord[qi];
        const UkSeg D = s_desc[sidx];
        const uint32_t n = D.info & 0xffffu, t = (D.info >> 16) & 15u;
        const bool raw = (D.info >> 21) & 1u, sig = (D.info >> 20) & 1u, vp = VP && ((D.info >> 22) & 1u);
        uint32_t cw = D.vpos, dsum = 0;
        for (uint32_t base = 0; base < n; base += 128) {
            const uint32_t g = base + 4 * lane;
            const uint32_t nv = g < n ? min(4u, n - g) : 0u;
            const uint32_t keep = nv >= 4 ? 0xffffffffu : (1u << (8 * nv)) - 1u, t4 = t * 0x01010101u;
            uint32_t v4;
            if (raw) {
                /* 4 raw 4-bit GCLIs, the first in the top nibble */
                const uint32_t w = nv ? bits32_at(pbuf, D.vpos + 4 * g) : 0u;
                v4 = (w >> 28) | ((w >> 16) & 0x00000f00u) | ((w >> 4) & 0x000f0000u) | ((w << 8) & 0x0f000000u);
            } else {
                /* the groups of 8 in lanes 2i, 2i + 1 share flag i */
                bool coded = nv != 0;
                if (sig) coded = coded && !((bits32_at(pbuf, D.sig + (base >> 3)) >> (31 - (lane >> 1))) & 1u);
                const uint32_t bal = __ballot_sync(FULL, coded);
                /* predicted lines keep the codeword value (0xff: no
                 * codeword) until the line above is known */
                v4 = vp ? 0xffffffffu : t4;
                if (coded) {
                    const uint32_t c = cw + 4 * __popc(bal & lt_mask);
                    const uint32_t* zw = (const uint32_t*)(zval + (c & ~3u));
                    const uint32_t r4 = __funnelshift_r(zw[0], zw[1], 8 * (c & 3u)) & keep;
                    /* GCLI = gtli + value, at most 15 (31 for a predicted
                     * line's codeword value; values are below 128) */
                    const uint32_t room = vp ? 31u : 15u - t;
                    v4 = vp ? r4 : r4 + t4;
                    if ((r4 + (127u - room) * 0x01010101u) & 0x80808080u) {
                        bad = 1;
                        v4 = t4;
                    }
                }
                if (base + 128 < n) cw += 4 * __popc(bal);
            }
            if (nv) *(uint32_t*)(gcl + D.z + g) = v4; /* lines are padded to a multiple of 4 */
            if (!vp) {
                /* data bits: 4 (v - t + 1) per group above gtli (4 (v - t)
                 * with separate signs) */
                const uint32_t y = ((v4 & keep) | 0x80808080u) - (t + 1) * 0x01010101u;
                const uint32_t above = sign_bytes(y), one = above & 0x01010101u;
                dsum += __dp4a((y & above & 0x7f7f7f7fu) + (fs ? one : 2u * one), 0x01010101u, 0u);
            }
        }
        dsum = __reduce_add_sync(FULL, dsum);
        if (lane == 0) s_cnt[sidx] = 4 * dsum;
    }
    __syncthreads();
    if constexpr (VP) {
        /* the slice's rows in their order: each resolves its own and hands its
         * GCLIs and gtlis to the block of the next */
        cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
        for (int turn = 0; turn < turns; turn++) {
            if (turn == rank) {
                if (s_hasvp) {
                /* vertical prediction (unpack_verical_pred_gclis_*, Packing.c:267-431):
                 * GCLI = the predictor max(top, max(gtli_top, gtli)) moved by the
                 * codeword value; without a codeword (insignificant group) the
                 * predictor, or gtli in run mode.  Line levels in order: line l reads
                 * line l - 1 of its band (line 0: the row above, top_gcl). */
                    const uint32_t rm = s_sc[8];
                    for (uint32_t lvl = 0;; lvl++) {
                        bool more = false; /* lines below this level */
                        for (uint32_t sidx = warp; sidx < nseg; sidx += UK_WARPS) {
                            const UkSeg D = s_desc[sidx];
                            const uint32_t bl = D.info >> 24, n = D.info & 0xffffu, lt = (D.info >> 16) & 15u;
                            if (!((D.info >> 22) & 1u)) continue;
                            more |= bls[bl].line > lvl;
                            if (bls[bl].line != lvl) continue;
                            const uint32_t tb = s_topbl[bl];
                            const int from_prev = s_topprev[bl];
                            /* in both rows a line starts at a multiple of 4 */
                            const uint8_t* src = (from_prev ? top_gcl : gcl) + s_topg[bl] + (D.z - bls[bl].gbase);
                            const uint32_t tt = max(from_prev ? (uint32_t)top_t[tb] : (uint32_t)ln[tb].t, lt);
                            uint32_t dsum = 0;
                            for (uint32_t g = 4 * lane; g < n; g += 128) {
                                const uint32_t x4 = *(const uint32_t*)(gcl + D.z + g), m4 = *(const uint32_t*)(src + g);
                                uint32_t v4 = 0;
#pragma unroll
                                for (int k = 0; k < 2; k++) {
                                    /* two GCLIs in 16-bit halves: x > 2 thr moves the
                                     * predictor by x - thr, a smaller odd x by -(x + 1)
                                     * / 2, an even one by x / 2 */
                                    const uint32_t x = (x4 >> (8 * k)) & 0x00ff00ffu;
                                    const uint32_t mt = __vmaxu2((m4 >> (8 * k)) & 0x00ff00ffu, tt * 0x00010001u);
                                    const uint32_t up = __vcmpgtu2(x, 2u * (mt - lt * 0x00010001u)), none = __vcmpeq2(x, 0x00ff00ffu);
                                    const uint32_t odd = (x & 0x00010001u) * 0xffffu, half = (x >> 1) & 0x007f007fu;
                                    const uint32_t moved = __vadd2(mt, half ^ odd), far = x + lt * 0x00010001u;
                                    const uint32_t v = (none & (rm ? lt * 0x00010001u : mt)) | (~none & ((up & far) | (~up & moved)));
                                    bad |= (__vcmpgtu2(v, 0x000f000fu) & (g + k + 2 < n ? 0xffffffffu : g + k < n ? 0xffffu : 0u)) != 0u;
                                    v4 |= __vminu2(v, 0x000f000fu) << (8 * k);
                                }
                                const uint32_t nv = min(4u, n - g), keep = nv >= 4 ? 0xffffffffu : (1u << (8 * nv)) - 1u;
                                *(uint32_t*)(gcl + D.z + g) = v4;
                                const uint32_t y = ((v4 & keep) | 0x80808080u) - (lt + 1) * 0x01010101u;
                                const uint32_t above = sign_bytes(y), one = above & 0x01010101u;
                                dsum += __dp4a((y & above & 0x7f7f7f7fu) + (fs ? one : 2u * one), 0x01010101u, 0u);
                            }
                            dsum = __reduce_add_sync(FULL, dsum);
                            if (lane == 0) s_cnt[sidx] = 4 * dsum;
                        }
                        if (!__syncthreads_or(more)) break;
                    }
                }
                const int next = rank + 1 == turns ? 0 : rank + 1;
                uint32_t* to = cl.map_shared_rank((uint32_t*)top_gcl, next);
                uint8_t* tot = cl.map_shared_rank(top_t, next);
                for (uint32_t i = threadIdx.x; i < (cap_groups >> 2); i += blockDim.x) to[i] = ((const uint32_t*)gcl)[i];
                for (uint32_t x = threadIdx.x; x < nbl; x += blockDim.x) tot[x] = ln[x].t;
            }
            cl.sync();
        }
    }
    {
        /* data position of every segment */
        uint32_t dbits;
        const uint32_t b = seg_bases(threadIdx.x < nseg ? s_cnt[threadIdx.x] : 0u, myseg.bl, nseg, npk, bls, s_pkbl0, s_pknbl, s_ex, ws,
                                     &dbits);
        if (threadIdx.x < nseg) s_base[threadIdx.x] = pk[bls[myseg.bl].pk].dpos + b;
        const int bad_pk = threadIdx.x < npk && pk[threadIdx.x].present && dbits > pk[threadIdx.x].dbits;
        if (__syncthreads_or(bad_pk)) {
            if (threadIdx.x == 0) JXS_STATUS_SET(status, JXS_E_DEC_BITSTREAM);
            return;
        }
    }

    } /* !LEAN */

    /* pass 3: data */
    const uint32_t uniform = cfg->qpih;
    if (FS && fs) {
        /* separate signs (unpack_sign, Packing.c:221-247): a sign bit for
         * every non-zero magnitude, band lines of the packet in order and each
         * line in coefficient order (the last group's padding coefficients
         * last).  Count them per segment, give each segment its first sign
         * bit in the packet's sign sub-packet, then decode with the signs. */
        for (uint32_t qi = next_seg(&s_next[1], lane); qi < nseg; qi = next_seg(&s_next[1], lane)) {
            const uint32_t sidx = s_ord[qi];
            const UkSeg D = s_desc[sidx];
            const uint32_t n = D.info & 0xffffu, t = (D.info >> 16) & 15u;
            uint32_t dpos = s_base[sidx], nzs = 0;
            for (uint32_t base = 0; base < n; base += 32) {
                const uint32_t g = base + lane;
                const uint32_t v = g < n ? gcl[D.z + g] : 0u;
                const uint32_t np = v > t ? v - t : 0u;
                const uint32_t len = 4 * np;
                uint32_t tot;
                const uint32_t ex = warp_excl_scan(len, &tot);
                if (len) {
                    const uint32_t pos = dpos + ex;
                    const uint64_t win = ((uint64_t)bits32_at(pbuf, pos) << 32) | bits32_at(pbuf, pos + 32);
                    uint32_t A, B2;
                    nzs += __popc(group_mags(win >> (64 - len), np, t, v, uniform, &A, &B2));
                }
                dpos += tot;
            }
            nzs = __reduce_add_sync(FULL, nzs);
            if (lane == 0) s_cnt[sidx] = nzs;
        }
        __syncthreads();
        /* first sign bit of every segment */
        uint32_t sbits;
        const uint32_t b = seg_bases(threadIdx.x < nseg ? s_cnt[threadIdx.x] : 0u, myseg.bl, nseg, npk, bls, s_pkbl0, s_pknbl, s_ex, ws,
                                     &sbits);
        if (threadIdx.x < nseg) s_sgb[threadIdx.x] = pk[bls[myseg.bl].pk].sgpos + b;
        const int bad_pk = threadIdx.x < npk && pk[threadIdx.x].present && sbits > pk[threadIdx.x].sgbits;
        if (threadIdx.x == 0) s_next[1] = 0;
        if (__syncthreads_or(bad_pk)) {
            if (threadIdx.x == 0) JXS_STATUS_SET(status, JXS_E_DEC_BITSTREAM);
            return;
        }
    }
    for (uint32_t qi = next_seg(&s_next[1], lane); qi < nseg; qi = next_seg(&s_next[1], lane)) {
        const uint32_t sidx = s_ord[qi];
        const UkSeg D = s_desc[sidx];
        const uint32_t n = D.info & 0xffffu, t = (D.info >> 16) & 15u, bl = D.info >> 24;
        int16_t* crow = coef + (s_crow[bl] + 4 * (uint64_t)D.z);
        const int wend = (int)(s_wend[bl] - 4 * D.z); /* coefficients of the line from the segment on */
        uint32_t dpos = s_base[sidx];
        if (!FS || !fs) {
            /* signs with the data: each lane 4 consecutive groups.  The lane
             * writes zeros for its groups, then the warp lists the groups
             * with data (nibble offset in the warp's data, group, GCLI) and
             * each lane decodes one listed group at a time, so that the decode
             * work follows the groups that have data */
            uint32_t* list = (uint32_t*)(dsm + UL.list) + 128 * warp;
            uint32_t cw = D.vpos;
            for (uint32_t base = 0; base < n; base += 128) {
                const uint32_t g = base + 4 * lane;
                const uint32_t nv = g < n ? min(4u, n - g) : 0u;
                const uint32_t keep = nv >= 4 ? 0xffffffffu : (1u << (8 * nv)) - 1u;
                uint32_t v4;
                if constexpr (LEAN) {
                    if ((D.info >> 21) & 1u) {
                        /* 4 raw 4-bit GCLIs, the first in the top nibble */
                        const uint32_t w = nv ? bits32_at(pbuf, D.vpos + 4 * g) : 0u;
                        v4 = (w >> 28) | ((w >> 16) & 0x00000f00u) | ((w >> 4) & 0x000f0000u) | ((w << 8) & 0x0f000000u);
                    } else {
                        /* the groups of 8 in lanes 2i, 2i + 1 share flag i, so
                         * that a lane's groups all carry a codeword or none
                         * (only the segment's last lane may hold fewer than 4) */
                        bool coded = nv != 0;
                        if ((D.info >> 20) & 1u) coded = coded && !((bits32_at(pbuf, D.sig + (base >> 3)) >> (31 - (lane >> 1))) & 1u);
                        const uint32_t bal = __ballot_sync(FULL, coded);
                        v4 = t * 0x01010101u;
                        if (coded) {
                            const uint32_t c = cw + 4 * __popc(bal & lt_mask);
                            const uint32_t* zw = (const uint32_t*)(zval + (c & ~3u));
                            const uint32_t r4 = __funnelshift_r(zw[0], zw[1], 8 * (c & 3u)) & keep;
                            /* GCLI = gtli + value, at most 15 (values are below 128) */
                            if ((r4 + (112u + t) * 0x01010101u) & 0x80808080u) bad = 1;
                            else v4 += r4;
                        }
                        cw += 4 * __popc(bal);
                    }
                    v4 &= keep;
                } else {
                    v4 = nv ? *(const uint32_t*)(gcl + D.z + g) & keep : 0u;
                }
                /* per byte: v > t, and the data nibbles of such a group (v - t
                 * + 1); running sums over the lane's bytes, then one scan for
                 * the nibbles and the listed groups */
                const uint32_t y = (v4 | 0x80808080u) - (t + 1) * 0x01010101u;
                const uint32_t above = sign_bytes(y), one = above & 0x01010101u;
                const uint32_t nibs = ((y & above & 0x7f7f7f7fu) + 2u * one) * 0x01010101u;
                const uint32_t own = (nibs >> 24) | ((uint32_t)__popc(one) << 24);
                const uint32_t inc = warp_incl_scan(own), ex = inc - own, tot = __shfl_sync(FULL, inc, 31), cnt = tot >> 24;
                /* zeros for the lane's groups (those with data are written
                 * again below, after the warp barrier) */
                if (one_col) {
                    if (nv == 4) {
                        *(uint4*)(crow + 4 * g) = make_uint4(0u, 0u, 0u, 0u);
                        *(uint4*)(crow + 4 * g + 8) = make_uint4(0u, 0u, 0u, 0u);
                    } else {
                        for (uint32_t q = 0; q < nv; q++) *(uint2*)(crow + 4 * (g + q)) = make_uint2(0u, 0u);
                    }
                } else {
                    /* a column starts anywhere in the row and ends where the
                     * next begins: the groups' coefficients inside it only */
                    for (int c = 0; c < 4 * (int)nv && c < wend - 4 * (int)g; c++)
                        if (!((one >> (8 * (c >> 2))) & 1u)) crow[4 * g + c] = 0;
                }
                {
                    const uint32_t po = nibs << 8, pi = one * 0x01010100u; /* before each byte's group */
                    const uint32_t e0 = ((ex & 0xffffu) << 16) | ((uint32_t)lane << 6);
                    uint32_t* slot = list + (ex >> 24);
                    if (one & 0x00000001u) slot[0] = e0 + (v4 & 255u);
                    if (one & 0x00000100u) slot[(pi >> 8) & 255u] = e0 + 0x10u + __byte_perm(v4, po, 0x4541);
                    if (one & 0x00010000u) slot[(pi >> 16) & 255u] = e0 + 0x20u + __byte_perm(v4, po, 0x4642);
                    if (one & 0x01000000u) slot[pi >> 24] = e0 + 0x30u + __byte_perm(v4, po, 0x4743);
                }
                __syncwarp();
                for (uint32_t r = lane; r < cnt; r += 32) {
                    const uint32_t e = list[r];
                    const uint32_t gi = base + ((e >> 4) & 127u), v = e & 15u, np = v - t, pos = dpos + 4 * (e >> 16);
                    const int wl = wend - 4 * (int)gi;
                    const uint32_t win = bits32_at(pbuf, pos);
                    uint2 ov;
                    if (uniform) {
                        const uint64_t w2 = (((uint64_t)win << 32) | bits32_at(pbuf, pos + 32)) >> (60 - 4 * np);
                        ov = decode_group(w2, np, t, v, uniform, wl);
                    } else {
                        /* the sign nibble is transposed with the planes, as the
                         * plane above the np magnitude planes, 8 at a time; the
                         * upper ones only where the warp has a group with more
                         * than 7 planes.  Coefficients past the band width come
                         * out as the stream has them: they go to the row's
                         * padding, or nowhere */
                        const uint32_t more = np >= 8 ? 4 * np - 28 : 0u; /* bits past the first 32 */
                        uint32_t low = np >= 8 ? win : win >> ((28 - 4 * np) & 31), high = 0u;
                        const bool any8 = __any_sync(__activemask(), np >= 8);
                        if (any8) {
                            low = __funnelshift_lc(bits32_at(pbuf, pos + 32), low, more);
                            high = more ? win >> (32 - more) : 0u;
                        }
                        const uint32_t tl = planes_to_coefs(low);
                        uint32_t P01 = __byte_perm(tl, 0u, 0x4243), P23 = __byte_perm(tl, 0u, 0x4041);
                        if (any8) {
                            const uint32_t th = planes_to_coefs(high);
                            P01 |= __byte_perm(th, 0u, 0x2434);
                            P23 |= __byte_perm(th, 0u, 0x0414);
                        }
                        const uint32_t mag = ((1u << np) - 1u) * 0x00010001u, half = ((1u << t) >> 1) * 0x00010001u;
                        ov = make_uint2(dequant_pair(P01, np, t, mag, half), dequant_pair(P23, np, t, mag, half));
                    }
                    if (one_col) {
                        *(uint2*)(crow + 4 * gi) = ov;
                    } else {
                        const uint32_t vv[2] = {ov.x, ov.y};
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            if (c < wl) crow[4 * gi + c] = (int16_t)((vv[c >> 1] >> (16 * (c & 1))) & 0xffffu);
                    }
                }
                __syncwarp();
                dpos += 4 * (tot & 0xffffu);
            }
            continue;
        }
        uint32_t spos = s_sgb[sidx];
        for (uint32_t base = 0; base < n; base += 32) {
            const uint32_t g = base + lane;
            const bool valid = g < n;
            const uint32_t v = valid ? gcl[D.z + g] : 0u;
            const uint32_t np = v > t ? v - t : 0u;
            const uint32_t len = 4 * np; /* separate signs: planes only */
            uint32_t tot;
            const uint32_t ex = warp_excl_scan(len, &tot);
            uint2 o = make_uint2(0u, 0u);
            {
                uint32_t A = 0, B2 = 0, nz = 0;
                if (len) {
                    const uint32_t pos = dpos + ex;
                    const uint64_t win = ((uint64_t)bits32_at(pbuf, pos) << 32) | bits32_at(pbuf, pos + 32);
                    nz = group_mags(win >> (64 - len), np, t, v, uniform, &A, &B2);
                }
                /* this group's sign bits follow those of the lanes before it */
                uint32_t stot;
                const uint32_t sex = warp_excl_scan(__popc(nz), &stot);
                uint32_t sgn = 0;
                if (nz) {
                    const uint32_t sw = bits32_at(pbuf, spos + sex);
                    uint32_t k = 0;
#pragma unroll
                    for (int c = 3; c >= 0; c--) {
                        if (nz & (1u << c)) {
                            sgn |= ((sw >> (31 - k)) & 1u) << c;
                            k++;
                        }
                    }
                }
                if (len) o = group_finish(A, B2, sgn, uniform && t != 0, wend - 4 * (int)g);
                spos += stot;
            }
            if (valid) {
                if (one_col) {
                    *(uint2*)(crow + 4 * g) = o; /* the band row's padding takes the last group's tail */
                } else {
                    /* a column starts anywhere in the row and ends where the
                     * next begins: the group's coefficients inside it only */
                    const int wl = wend - 4 * (int)g;
                    crow[4 * g] = (int16_t)(o.x & 0xffffu);
                    if (wl > 1) crow[4 * g + 1] = (int16_t)(o.x >> 16);
                    if (wl > 2) crow[4 * g + 2] = (int16_t)(o.y & 0xffffu);
                    if (wl > 3) crow[4 * g + 3] = (int16_t)(o.y >> 16);
                }
            }
            dpos += tot;
        }
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) JXS_STATUS_SET(status, JXS_E_DEC_BITSTREAM);
}

/* ------------------------------------------------------------------------ */
/* Precinct offsets of a device-resident codestream                          */
/* ------------------------------------------------------------------------ */
/* One thread per slice: the slice is expected where the constant-bit-rate
 * split of Lcod puts it (EncHandle.c:760-809); its precincts are found by
 * following the 24-bit precinct lengths, and the walk must end exactly at
 * the next slice (or at EOC).  False if anything is not so. */
DEV bool walk_slice(const jxs_cfg_t* __restrict__ cfg, const uint8_t* bs, uint32_t size,
                    uint32_t* prec_off, const uint32_t s) {
    if (cfg->max_slice_budget == 0) return false;
    uint64_t off = cfg->slice_begin[s];
    if (off + 6 > size || bs[off] != 0xff || bs[off + 1] != 0x20 || bs[off + 2] != 0 || bs[off + 3] != 4 ||
        (((uint32_t)bs[off + 4] << 8) | bs[off + 5]) != s) return false;
    off += 6;
    /* the slice's precincts: rows x columns, row after row */
    const uint32_t first = s * cfg->pps * cfg->ncol,
                   n = ((s + 1 == cfg->nslices) ? cfg->np - s * cfg->pps : cfg->pps) * cfg->ncol;
    for (uint32_t i = 0; i < n; i++) {
        if (off + cfg->prec_hdr_bytes > size) return false;
        const uint32_t lprc = be24(bs + off);
        if (lprc > JXS_PREC_MAX_BYTES) return false;
        prec_off[first + i] = (uint32_t)off;
        off += cfg->prec_hdr_bytes + lprc;
    }
    const int ok = (s + 1 < cfg->nslices) ? off == cfg->slice_begin[s + 1]
                                          : (off + 2 <= size && bs[off] == 0xff && bs[off + 1] == 0x11);
    return ok;
}

/* Fallback when the prediction failed: one thread walks the whole codestream
 * from the header (get_slice_size, DecThreadInit.c:35-131). */
DEV void walk_sequential(const jxs_cfg_t* __restrict__ cfg, const uint8_t* bs, uint32_t size,
                         uint32_t* prec_off, int* status) {
    uint64_t off = cfg->hdr_len;
    for (uint32_t s = 0; s < cfg->nslices; s++) {
        if (off + 6 > size) {
            JXS_STATUS_SET(status, JXS_E_DEC_SHORT);
            return;
        }
        if (bs[off] != 0xff || bs[off + 1] != 0x20 || bs[off + 2] != 0 || bs[off + 3] != 4 ||
            (((uint32_t)bs[off + 4] << 8) | bs[off + 5]) != s) {
            JXS_STATUS_SET(status, JXS_E_DEC_BITSTREAM);
            return;
        }
        off += 6;
        const uint32_t first = s * cfg->pps * cfg->ncol,
                       n = ((s + 1 == cfg->nslices) ? cfg->np - s * cfg->pps : cfg->pps) * cfg->ncol;
        for (uint32_t i = 0; i < n; i++) {
            if (off + cfg->prec_hdr_bytes > size) {
                JXS_STATUS_SET(status, JXS_E_DEC_SHORT);
                return;
            }
            const uint32_t lprc = be24(bs + off);
            if (lprc > JXS_PREC_MAX_BYTES) {
                JXS_STATUS_SET(status, JXS_E_DEC_BITSTREAM);
                return;
            }
            prec_off[first + i] = (uint32_t)off;
            off += cfg->prec_hdr_bytes + lprc;
        }
    }
    if (off + 2 > size) JXS_STATUS_SET(status, JXS_E_DEC_SHORT);
    else if (bs[off] != 0xff || bs[off + 1] != 0x11) JXS_STATUS_SET(status, JXS_E_DEC_BITSTREAM);
}

/* A frame's precincts, by one block: a thread per slice (or more slices),
 * then one thread in order if any slice is not where it is expected.  Bound by
 * the latency of a handful of loads that wait for one another; the second step
 * as a launch of its own cost 5 us, taken or not. */
#define WALK_THREADS 512
DEV void walk_frame(const jxs_cfg_t* __restrict__ cfg, const uint8_t* bs, uint32_t size, uint32_t* prec_off,
                    int* status) {
    bool lost = false;
    for (uint32_t s = threadIdx.x; s < cfg->nslices; s += blockDim.x) lost |= !walk_slice(cfg, bs, size, prec_off, s);
    if (__syncthreads_or(lost) && threadIdx.x == 0) walk_sequential(cfg, bs, size, prec_off, status);
}

/* ------------------------------------------------------------------------ */
/* kernels: one frame, or a batch of frames                                  */
/* ------------------------------------------------------------------------ */
/* 4 blocks of 512 threads per SM where the shared memory allows it (32
 * registers) */
template <bool FS>
__global__ void __launch_bounds__(UK_THREADS, 4) unpack_kernel(const jxs_cfg_t* __restrict__ cfg, const uint8_t* bs,
                                                               uint32_t bs_size, const uint32_t* prec_off,
                                                               int16_t* coef, uint32_t cap_bytes, uint32_t cap_groups,
                                                               uint32_t cap_seg, int* status) {
    unpack_body<FS, false, false>(cfg, bs, bs_size, prec_off, coef, cap_bytes, cap_groups, cap_seg, status, (int)blockIdx.x, nullptr, nullptr,
                           0);
}

/* cap_bytes / cap_groups / cap_seg: the largest of the batch's frames
 * (shared-memory layout of the launch) */
template <bool FS>
__global__ void __launch_bounds__(UK_THREADS, 4) unpack_batch_kernel(const __grid_constant__ DecPrecLaunch L, uint32_t cap_bytes,
                                                                     uint32_t cap_groups, uint32_t cap_seg) {
    const DecPrecFrame& F = L.job[find_job<JXS_BATCH_FRAMES>(L.job, L.nframes, (int)blockIdx.x)];
    unpack_body<FS, false, true>(F.cfg, F.bs, F.bs_size, F.prec_off, F.coef, cap_bytes, cap_groups, cap_seg, F.status,
                           (int)blockIdx.x - F.first_block, nullptr, nullptr, 0);
}

/* Streams with vertical prediction: a cluster of blocks per slice, a
 * precinct row each (more rows than blocks: in rounds).  Only the GCLIs
 * depend on the row above; parsing, codeword values and coefficients of the
 * slice's rows run side by side, the GCLIs in turns with a cluster barrier
 * after each, handed on through the next block's shared memory (after the
 * codeword values: cap_groups bytes).  With several precinct columns, column
 * after column (the precinct above is in the same column).  Every block takes
 * the same number of barriers, failed rows and rows past the slice's end
 * included.  Bound by the latency of one precinct and the turns, which take
 * two GCLIs to an instruction: 1279x717 4:4:4 with slices of 4 rows 116 us
 * with a block per slice and a GCLI per lane, 48 us now. */
__global__ void __launch_bounds__(UK_THREADS) unpack_vpred_kernel(const jxs_cfg_t* __restrict__ cfg, const uint8_t* bs,
                                                                  uint32_t bs_size, const uint32_t* prec_off,
                                                                  int16_t* coef, uint32_t cap_bytes,
                                                                  uint32_t cap_groups, uint32_t cap_seg, int* status) {
    extern __shared__ __align__(16) uint8_t dsm[];
    __shared__ uint8_t top_t[JXS_MAXBLINES];
    uint8_t* top_gcl = dsm + uk_layout(cap_bytes, cap_groups, cap_seg, false).top;
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const uint32_t turns = cl.num_blocks(), rank = cl.block_rank();
    const uint32_t s = blockIdx.x / turns, ncol = cfg->ncol;
    const uint32_t first = s * cfg->pps, end = min(cfg->np, first + cfg->pps);
    cl.sync(); /* every block runs before another writes to it */
    for (uint32_t col = 0; col < ncol; col++) {
        for (uint32_t row0 = first; row0 < end; row0 += turns) {
            const uint32_t row = row0 + rank;
            if (row < end) {
                unpack_body<true, true, false>(cfg, bs, bs_size, prec_off, coef, cap_bytes, cap_groups, cap_seg, status,
                                               (int)(row * ncol + col), top_gcl, top_t, row != first, (int)rank, (int)turns);
                __syncthreads();
            } else {
                for (uint32_t i = 0; i < turns; i++) cl.sync();
            }
        }
    }
    cl.sync(); /* and until none does any more */
}

__global__ void __launch_bounds__(WALK_THREADS) walk_kernel(const jxs_cfg_t* __restrict__ cfg, const uint8_t* bs,
                                                            uint32_t size, uint32_t* prec_off, int* status) {
    dep_wait();
    walk_frame(cfg, bs, size, prec_off, status);
}

/* one block per frame of the batch */
__global__ void __launch_bounds__(WALK_THREADS) walk_batch_kernel(const __grid_constant__ DecPrecLaunch L) {
    const DecPrecFrame& F = L.job[blockIdx.x];
    walk_frame(F.cfg, F.bs, F.bs_size, F.prec_off, F.status);
}

/* ------------------------------------------------------------------------ */
/* host-side launchers                                                       */
/* ------------------------------------------------------------------------ */
extern "C" cudaError_t jxs_launch_walk(const jxs_cfg_t* dcfg, const uint8_t* bs, uint32_t size, uint32_t* prec_off, int* status,
                                       cudaStream_t st) {
    return jxs_launch(walk_kernel, dim3(1), WALK_THREADS, 0, st, dcfg, bs, size, prec_off, status);
}

template <bool FS>
static cudaError_t unpack_one(const jxs_cfg_t* dcfg, const uint8_t* bs, uint32_t bs_size, const uint32_t* prec_off, int16_t* coef,
                              uint32_t np, uint32_t cap_bytes, uint32_t cap_groups, uint32_t cap_seg, int* status, cudaStream_t st) {
    const size_t smem = uk_layout(cap_bytes, cap_groups, cap_seg, !FS).end;
    static std::atomic<int> attr[JXS_MAX_DEV];
    cudaError_t e = jxs_smem_attr(unpack_kernel<FS>, (int)smem, attr);
    if (e != cudaSuccess) return e;
    return jxs_launch(unpack_kernel<FS>, dim3(np), UK_THREADS, smem, st, dcfg, bs, bs_size, prec_off, coef, cap_bytes, cap_groups,
                      cap_seg, status);
}
/* fs: the frame has separate sign sub-packets (batch: some frame has).
 * prec_off may be NULL for a device codestream whose slices are expected at
 * the constant-bit-rate split: every block then finds its own precinct (a 4K
 * frame: 100 -> 89 us against locating all of them in two launches
 * first), and status[1] is set where that fails. */
extern "C" cudaError_t jxs_launch_unpack(const jxs_cfg_t* dcfg, const uint8_t* bs, uint32_t bs_size, const uint32_t* prec_off,
                                         int16_t* coef, uint32_t np, uint32_t cap_bytes, uint32_t cap_groups, uint32_t cap_seg,
                                         int fs, int* status, cudaStream_t st) {
    if (fs) return unpack_one<true>(dcfg, bs, bs_size, prec_off, coef, np, cap_bytes, cap_groups, cap_seg, status, st);
    return unpack_one<false>(dcfg, bs, bs_size, prec_off, coef, np, cap_bytes, cap_groups, cap_seg, status, st);
}

extern "C" cudaError_t jxs_launch_walk_batch(const DecPrecLaunch* L, cudaStream_t st) {
    if (L->nframes <= 0) return cudaSuccess;
    walk_batch_kernel<<<L->nframes, WALK_THREADS, 0, st>>>(*L);
    return cudaGetLastError();
}

template <bool FS>
static cudaError_t unpack_batch_one(const DecPrecLaunch* L, uint32_t cap_bytes, uint32_t cap_groups, uint32_t cap_seg, cudaStream_t st) {
    const size_t smem = uk_layout(cap_bytes, cap_groups, cap_seg, !FS).end;
    static std::atomic<int> attr[JXS_MAX_DEV];
    cudaError_t e = jxs_smem_attr(unpack_batch_kernel<FS>, (int)smem, attr);
    if (e != cudaSuccess) return e;
    if (L->nblocks <= 0) return cudaSuccess;
    unpack_batch_kernel<FS><<<L->nblocks, UK_THREADS, smem, st>>>(*L, cap_bytes, cap_groups, cap_seg);
    return cudaGetLastError();
}
extern "C" cudaError_t jxs_launch_unpack_batch(const DecPrecLaunch* L, uint32_t cap_bytes, uint32_t cap_groups, uint32_t cap_seg,
                                               int fs, cudaStream_t st) {
    return fs ? unpack_batch_one<true>(L, cap_bytes, cap_groups, cap_seg, st)
              : unpack_batch_one<false>(L, cap_bytes, cap_groups, cap_seg, st);
}

extern "C" cudaError_t jxs_launch_unpack_vpred(const jxs_cfg_t* dcfg, const uint8_t* bs, uint32_t bs_size, const uint32_t* prec_off,
                                               int16_t* coef, uint32_t nslices, uint32_t pps, uint32_t cap_bytes,
                                               uint32_t cap_groups, uint32_t cap_seg, int* status, cudaStream_t st) {
    const size_t smem = uk_layout(cap_bytes, cap_groups, cap_seg, false).top_end;
    static std::atomic<int> attr[JXS_MAX_DEV];
    cudaError_t e = jxs_smem_attr(unpack_vpred_kernel, (int)smem, attr);
    if (e != cudaSuccess) return e;
    /* a block per row of a slice, up to the 8 that every device takes, while
     * the blocks are all resident (2 to an SM by their registers, fewer by
     * their shared memory): beyond that they wait in place of others' work.
     * 1, 2, 4, 8 blocks: 1279x717 in 45 slices of 4 rows 123, 92, 83 us,
     * 3840x2160 in 135 158, 131, 146 us, in 34 of 16 rows 419, 283, 211,
     * 359 us, 7680x4320 in 270 of 4 rows 283, 302, 337 us */
    const unsigned resident = 152 * (2 * (smem + UK_STATIC_SMEM) <= 228 * 1024 ? 2 : 1);
    unsigned cluster = 8;
    while (cluster > 1 && nslices * (cluster < pps ? cluster : pps) > resident) cluster >>= 1;
    if (cluster > pps) cluster = pps;
    return jxs_launch_cluster(unpack_vpred_kernel, dim3((unsigned)nslices), cluster, UK_THREADS, smem, st, dcfg, bs, bs_size, prec_off,
                              coef, cap_bytes, cap_groups, cap_seg, status);
}
