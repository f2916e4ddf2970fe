/*
 * gs_fm.cuh -- FM-index primitives on the device.
 *
 * The occurrence table in HBM: one 64-byte block per 64 rows of the BWT (its
 * $ row included), a 16-byte slot per base c: {L2[c] + 1 + count of c before
 * the block, the block's rows that hold c as a 64-bit mask (two words, row i
 * at bit i & 31 of word i >> 5), 0}.  The $ row is set in no mask.  A step's
 * bound with base c is then one 16-byte load, and the new bound is the
 * slot's count plus the set bits of its mask below the bound's row: no
 * counting of two-bit fields, no selection of the base's count, no
 * correction for the $ row, no base offset to add.  The loader makes the
 * blocks from the file's checkpoints and packed words once (gs_index.cu).
 * Results are the reference's integers (seed_gen.cu:195-216 occ, :329-368
 * occ pair, :455-484 LF).
 *
 * The walk pass executes such queries without end and is bound by fills and by
 * instructions, so a bound is one load of one 64-byte fill.  Against 32 bytes
 * for 64 rows, four counts and bit-sliced bases, also one fill but two loads
 * and about 30 instructions, this form takes twice the HBM (3.1 GB at 3.1 Gbp)
 * and reaches half as far in L2, and a whole pass (the walk in brackets) takes,
 * with steps of one base, 15.5 ms instead of 16.3 for 2 M reads on 3.1 Gbp (8.7
 * of 9.5), 7.3 instead of 7.7 for 1 M on 100 Mbp (3.6 of 4.1), 6.9 instead of
 * 7.1 for 40,000 long reads.
 */
#ifndef GS_FM_CUH
#define GS_FM_CUH

#include "gs_internal.h"

/* one random read-only word with a 64-byte L2 fill (the default fills 128) */
__device__ __forceinline__ uint32_t gs_ld64(const uint32_t *p)
{
    uint32_t v;
    asm("ld.global.nc.L2::64B.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ uint32_t gs_sel4(uint32_t c, uint32_t a0, uint32_t a1, uint32_t a2,
                                            uint32_t a3)
{
    return c == 0 ? a0 : c == 1 ? a1 : c == 2 ? a2 : a3;
}

/* base c's slot of a row's block */
struct GsSlot {
    uint32_t cnt, m0, m1;
};

/* rows & ~63 is the byte offset of a row's 64-byte block */
__device__ __forceinline__ const char *gs_slot_at(const uint4 *occ, uint32_t row, uint32_t c)
{
    return (const char *)occ + (size_t)(row & ~63u) + (c << 4);
}

__device__ __forceinline__ GsSlot gs_load_slot(const uint4 *occ, uint32_t row, uint32_t c)
{
    GsSlot s;
    [[maybe_unused]] uint32_t pad;
    asm("ld.global.nc.L2::64B.v4.u32 {%0,%1,%2,%3}, [%4];"
        : "=r"(s.cnt), "=r"(s.m0), "=r"(s.m1), "=r"(pad)
        : "l"(gs_slot_at(occ, row, c)));
    return s;
}

/* the same when `yes`, as a predicated load instead of a branch; else the
 * slot is left undefined.  Of a table whose blocks have 4 << sh slots. */
__device__ __forceinline__ GsSlot gs_load_slot_if(bool yes, const uint4 *occ, uint32_t row, uint32_t c,
                                                  uint32_t sh)
{
    GsSlot s;
    [[maybe_unused]] uint32_t pad;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t"
        "@q ld.global.nc.L2::64B.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
        : "=r"(s.cnt), "=r"(s.m0), "=r"(s.m1), "=r"(pad)
        : "l"((const char *)occ + ((size_t)(row & ~63u) << sh) + (c << 4)), "r"((int)yes));
    return s;
}

/* a with `s`, else b */
__device__ __forceinline__ GsSlot gs_slot_sel(bool s, const GsSlot &a, const GsSlot &b)
{
    GsSlot r;
    r.cnt = s ? a.cnt : b.cnt;
    r.m0 = s ? a.m0 : b.m0;
    r.m1 = s ? a.m1 : b.m1;
    return r;
}

/* L2[c] + 1 + occurrences of c in rows [0, row): with the bits of the masks
 * below row & 63 (PTX bmsk and shr clamp counts of 32 and more) */
__device__ __forceinline__ uint32_t gs_slot_rank(const GsSlot &s, uint32_t row)
{
    const uint32_t j = row & 63u;
    uint32_t w0, w1;
    asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(w0) : "r"(j));
    asm("shr.u32 %0, 0xffffffff, %1;" : "=r"(w1) : "r"(64u - j));
    return s.cnt + __popc(s.m0 & w0) + __popc(s.m1 & w1);
}

/* One backward-search step with base c in [0,3]: [l,u] -> [l',u'].
 * Returns the number of 32-byte blocks of 64 rows of the $-removed string
 * that the canonical walk reads for it (0..2). */
__device__ __forceinline__ int gs_step(const GsDevIndex &I, uint32_t &l, uint32_t &u, uint32_t c)
{
    const bool lz = (l == 0);            /* occ(-1) = 0 */
    const bool uf = (u == I.seq_len);    /* occ(seq_len) = total */
    uint32_t la = l - 1u;
    la -= (la >= I.primary) ? 1u : 0u;
    const uint32_t ua = u - ((u >= I.primary) ? 1u : 0u);
    const int nb = (uf ? 0 : 1) + ((!lz && (uf || (la >> 6) != (ua >> 6))) ? 1 : 0);
    const GsSlot A = gs_load_slot(I.occ, l, c);
    const GsSlot E = gs_load_slot(I.occ, u + 1u, c);
    l = gs_slot_rank(A, l);
    u = gs_slot_rank(E, u + 1u) - 1u;
    return nb;
}

/* how many distinct values among those of a..d that are valid */
__device__ __forceinline__ int gs_distinct4(uint32_t a, bool va, uint32_t b, bool vb, uint32_t c,
                                            bool vc, uint32_t d, bool vd)
{
    return (int)va + (int)(vb && !(va && b == a)) + (int)(vc && !(va && c == a) && !(vb && c == b)) +
           (int)(vd && !(va && d == a) && !(vb && d == b) && !(vc && d == c));
}

/* What one step of gs_step_pair touched, for the work counters: slots
 * loaded, those for J alone, and the distinct lines of 256 and 384 rows its
 * bounds fall in. */
struct GsStepTouch {
    int blocks, jblocks, lines256, lines384;
};

/* A table of blocks of 4 << sh slots, and a slot: one base of occ (sh 0), or
 * a base and the next of occ2 (sh 2) */
struct GsStepBy {
    const uint4 *occ;
    uint32_t sh, c;
};

/* One backward step of an interval I = [l,e) (only when doI) and of an
 * interval J = [jl,je) (jl >= je: none; left unchanged): e and je are one
 * past the last row.  With `within`, J lies within I and both step by the same
 * slot: J's bounds lie between I's, so a slot is loaded only where its block
 * differs from those of the bounds before it.  Predicated loads, all of which
 * issue before any is used. */
template <int COUNT>
__device__ __forceinline__ void gs_step_pair(const GsStepBy &by_i, const GsStepBy &by_j, bool within,
                                             uint32_t &l, uint32_t &e, uint32_t &jl, uint32_t &je, bool doI,
                                             GsStepTouch &touch)
{
    const bool jn = jl < je;
    const uint32_t bl = l >> 6, be = e >> 6, bj = jl >> 6, bk = je >> 6;
    const bool one = be == bl;                             /* I within a block: J too */
    const bool jL = within && bj == bl, jE = within && bj == be;
    const bool kL = within && bk == bl, kE = within && bk == be, kJ = bk == bj;
    const bool n0 = doI, n1 = doI && !one, n2 = jn && !jL && !jE, n3 = jn && !kL && !kE && !kJ;
    const GsSlot A = gs_load_slot_if(n0, by_i.occ, l, by_i.c, by_i.sh);
    GsSlot E = gs_load_slot_if(n1, by_i.occ, e, by_i.c, by_i.sh);
    GsSlot P = gs_load_slot_if(n2, by_j.occ, jl, by_j.c, by_j.sh);
    GsSlot Q = gs_load_slot_if(n3, by_j.occ, je, by_j.c, by_j.sh);
    E = gs_slot_sel(one, A, E);
    P = gs_slot_sel(jL, A, gs_slot_sel(jE, E, P));
    Q = gs_slot_sel(kL, A, gs_slot_sel(kE, E, gs_slot_sel(kJ, P, Q)));
    if (COUNT) {
        touch.blocks = (int)n0 + (int)n1 + (int)n2 + (int)n3;
        touch.jblocks = (int)n2 + (int)n3;
        touch.lines256 = gs_distinct4(e >> 8, doI, l >> 8, doI, je >> 8, jn, jl >> 8, jn);
        touch.lines384 = gs_distinct4(e / 384u, doI, l / 384u, doI, je / 384u, jn, jl / 384u, jn);
    }
    const uint32_t nl = gs_slot_rank(A, l), ne = gs_slot_rank(E, e);
    const uint32_t njl = gs_slot_rank(P, jl), nje = gs_slot_rank(Q, je);
    l = doI ? nl : l;
    e = doI ? ne : e;
    jl = jn ? njl : jl;
    je = jn ? nje : je;
}

/* a whole block: every base's slot */
struct GsBlk {
    GsSlot s[4];
};

__device__ __forceinline__ GsBlk gs_load_block(const uint4 *occ, uint32_t row)
{
    GsBlk b;
    const char *p = (const char *)occ + (size_t)(row & ~63u);
    [[maybe_unused]] uint32_t z0, z1;
    asm("ld.global.nc.L2::64B.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(b.s[0].cnt), "=r"(b.s[0].m0), "=r"(b.s[0].m1), "=r"(z0), "=r"(b.s[1].cnt),
          "=r"(b.s[1].m0), "=r"(b.s[1].m1), "=r"(z1)
        : "l"(p));
    asm("ld.global.nc.L2::64B.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(b.s[2].cnt), "=r"(b.s[2].m0), "=r"(b.s[2].m1), "=r"(z0), "=r"(b.s[3].cnt),
          "=r"(b.s[3].m0), "=r"(b.s[3].m1), "=r"(z1)
        : "l"(p + 32));
    return b;
}

/* the base of a row that is not the $ row, given its block */
__device__ __forceinline__ uint32_t gs_block_base(const GsBlk &b, uint32_t row)
{
    const uint32_t sh = row & 31u;
    const bool hi = (row & 32u) != 0;
    const uint32_t m1 = hi ? b.s[1].m1 : b.s[1].m0, m2 = hi ? b.s[2].m1 : b.s[2].m0,
                   m3 = hi ? b.s[3].m1 : b.s[3].m0;
    return (((m1 | m3) >> sh) & 1u) | ((((m2 | m3) >> sh) & 1u) << 1);
}

/* LF of a row whose base is c, given its block */
__device__ __forceinline__ uint32_t gs_block_lf(const GsBlk &b, uint32_t row, uint32_t c)
{
    GsSlot s;
    s.cnt = gs_sel4(c, b.s[0].cnt, b.s[1].cnt, b.s[2].cnt, b.s[3].cnt);
    s.m0 = gs_sel4(c, b.s[0].m0, b.s[1].m0, b.s[2].m0, b.s[3].m0);
    s.m1 = gs_sel4(c, b.s[0].m1, b.s[1].m1, b.s[2].m1, b.s[3].m1);
    return gs_slot_rank(s, row);
}

/* LF of a BWT row (bwt_inv_psi_gpu, seed_gen.cu:455-484).  lf_mode
 * GS_LF_GPUSEED reproduces its return of 0 for row primary+1; GS_LF_BWA
 * computes LF there as bwa does (seed_gen.cu:448-453). */
__device__ __forceinline__ uint32_t gs_lf(const GsDevIndex &I, uint32_t k, int lf_mode)
{
    if (k == I.primary) return 0;
    if (lf_mode == GS_LF_GPUSEED && k == I.primary + 1u) return 0;
    const GsBlk B = gs_load_block(I.occ, k);
    return gs_block_lf(B, k, gs_block_base(B, k));
}

#endif
