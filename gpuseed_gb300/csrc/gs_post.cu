/*
 * gs_post.cu -- per-read filtering, ordering and the sampled-SA locate.
 *
 * Replaces, for one batch, the reference's compaction (DeviceSelect::Flagged,
 * seed_gen.cu:3400-3401), the SMEM/MEM filters and counts (:865-1251), the
 * segmented sorts by begin (:1233, :3570) and the expansion + locate kernels
 * (:555-724):
 *
 *   gs_finalize_count  lane per read (warp per long read): compacts the
 *                      read's candidate slots in place and counts the
 *                      seeds/positions the filters keep;
 *   gs_finalize_emit   thread per read: its offsets, and merges the forward (ascending end)
 *                      and reverse (ascending start) records by begin --
 *                      equal begins keep forward first, as the reference's
 *                      stable sort does -- and writes the output seeds;
 *   gs_locate          position -> seed map, and each position's row by an
 *                      LF walk to a sampled row (or the full suffix array).
 *
 * Filter rules on the per-strand record lists (ascending end / start):
 *   SMEM forward: keep a record unless the next one has the same begin
 *        (:1000-1006); reverse: keep unless the previous has the same end
 *        (:1013-1019).
 *   MEM  forward: drop a record whose next record has the same begin and the
 *        same interval size (:1114-1120); its positions are its rows minus the
 *        rows of that next same-begin record's interval (:933-953, :624-667);
 *        reverse: the same toward the previous record with the same end.
 */
#include "gs_fm.cuh"
#include "gs_scan.cuh"



__device__ __forceinline__ uint32_t gs_size(const GsRec &r) { return r.u - r.l + 1u; }

/* decision for forward record R whose next record (when has_next) is N */
__device__ __forceinline__ void gs_fwd_rule_v(const GsRec &R, const GsRec &N, bool has_next,
                                              int smem, uint32_t max_occ, bool &keep,
                                              uint32_t &cnt, uint32_t &xl, uint32_t &xu)
{
    const bool same = has_next && N.x == R.x;
    uint32_t sz = gs_size(R);
    xl = 1; xu = 0;
    if (smem) {
        keep = !same;
        cnt = sz;
    } else {
        uint32_t nsz = same ? gs_size(N) : 0u;
        keep = !(same && nsz == sz);
        cnt = sz - nsz;
        if (same) { xl = N.l; xu = N.u; }
    }
    if (max_occ && sz > max_occ) keep = false;
}

/* decision for forward record o of list F[0..nf) */
__device__ __forceinline__ void gs_fwd_rule(const GsRec *F, uint32_t nf, uint32_t o, int smem,
                                            uint32_t max_occ, bool &keep, uint32_t &cnt,
                                            uint32_t &xl, uint32_t &xu)
{
    GsRec N;
    N.l = 1; N.u = 0; N.x = 0; N.y = 0;
    if (o + 1 < nf) N = F[o + 1];
    gs_fwd_rule_v(F[o], N, o + 1 < nf, smem, max_occ, keep, cnt, xl, xu);
}

/* decision for reverse record R whose previous record (when has_prev) is P */
__device__ __forceinline__ void gs_rev_rule_v(const GsRec &R, const GsRec &P, bool has_prev,
                                              int smem, uint32_t max_occ, bool &keep,
                                              uint32_t &cnt, uint32_t &xl, uint32_t &xu)
{
    const bool same = has_prev && P.y == R.y;
    uint32_t sz = gs_size(R);
    xl = 1; xu = 0;
    if (smem) {
        keep = !same;
        cnt = sz;
    } else {
        uint32_t psz = same ? gs_size(P) : 0u;
        keep = !(same && psz == sz);
        cnt = sz - psz;
        if (same) { xl = P.l; xu = P.u; }
    }
    if (max_occ && sz > max_occ) keep = false;
}

__device__ __forceinline__ void gs_rev_rule(const GsRec *Rv, uint32_t nr, uint32_t o, int smem,
                                            uint32_t max_occ, bool &keep, uint32_t &cnt,
                                            uint32_t &xl, uint32_t &xu)
{
    (void)nr;
    GsRec P;
    P.l = 1; P.u = 0; P.x = 0; P.y = 0;
    if (o > 0) P = Rv[o - 1];
    gs_rev_rule_v(Rv[o], P, o > 0, smem, max_occ, keep, cnt, xl, xu);
}

/* Compacts the records among slots s0..s0+n (flagged in the record mask;
 * the other slots were never written) to the front, in order; returns the
 * count.  Per 1024 slots: one round of mask words (a lane each, scanned
 * across the warp), then the records, 32 at a time -- lane j finds the j-th
 * set bit by binary lifting over the scan and __fns within its word.  A
 * record's target is never beyond its source, and a group's loads all come
 * before its writes, so compacting in place is safe. */
__device__ __forceinline__ uint32_t gs_warp_compact(GsRec *slots, const uint32_t *mask, uint64_t s0,
                                                    uint32_t n, int lane)
{
    uint32_t cnt = 0;
    if (n == 0) return 0;
    const uint64_t s1 = s0 + n;
    const uint64_t w0 = s0 >> 5, wend = (s1 + 31) >> 5;
    for (uint64_t wc = w0; wc < wend; wc += 32) {
        const uint64_t w = wc + (uint64_t)lane;
        uint32_t m = 0;
        if (w < wend) {
            m = mask[w];
            const uint64_t lo = w << 5;
            if (lo < s0) m &= 0xffffffffu << (uint32_t)(s0 - lo);
            if (lo + 32 > s1) m &= 0xffffffffu >> (uint32_t)(lo + 32 - s1);
        }
        const uint32_t c = __popc(m);
        uint32_t inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
        for (uint32_t g = 0; g < total; g += 32) {
            const uint32_t j = g + (uint32_t)lane;
            const uint32_t jj = j < total ? j : total - 1u;
            int L = 0;   /* first lane whose inclusive count exceeds jj */
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1) {
                uint32_t x = __shfl_sync(0xffffffffu, inc, L + step - 1);
                if (x <= jj) L += step;
            }
            const uint32_t word = __shfl_sync(0xffffffffu, m, L);
            const uint32_t before = __shfl_sync(0xffffffffu, inc - c, L);
            const uint32_t bit = __fns(word, 0, (int)(jj - before) + 1);
            GsRec rec;
            const bool v = j < total;
            if (v) rec = slots[((wc + (uint64_t)L) << 5) + bit];
            __syncwarp();
            if (v) slots[s0 + cnt + j] = rec;
            __syncwarp();
        }
        cnt += total;
    }
    return cnt;
}

/* Both strands of a read at once when their 2n slots fit one 1024-slot
 * round: forward records (slots s0..s0+n) go to s0 + rank, reverse ones
 * (s0+n..s0+2n) to s0 + n + rank -- one round of mask words, one of
 * records, for both.  Every target is at or before its source and earlier
 * records' targets lie before later records' sources, so in place is safe.
 * mine: lane j's record among the first 32 (forward, then reverse). */
__device__ __forceinline__ void gs_warp_compact_both(GsRec *slots, const uint32_t *mask, uint64_t s0,
                                                     uint32_t n, int lane, uint32_t &nf,
                                                     uint32_t &nr, GsRec &mine)
{
    const uint64_t s1 = s0 + n, s2 = s0 + 2ull * n;
    const uint64_t w0 = s0 >> 5, wend = (s2 + 31) >> 5;   /* at most 32 words */
    mine.x = mine.y = 0;
    mine.l = 1u;
    mine.u = 0u;
    const uint64_t w = w0 + (uint64_t)lane;
    uint32_t mf = 0, mr = 0;
    if (w < wend) {
        uint32_t m = mask[w];
        const uint64_t lo = w << 5;
        if (lo < s0) m &= 0xffffffffu << (uint32_t)(s0 - lo);
        if (lo + 32 > s2) m &= 0xffffffffu >> (uint32_t)(lo + 32 - s2);
        /* bits below s1 are forward slots */
        const uint32_t fmask = s1 <= lo ? 0u : (s1 >= lo + 32 ? 0xffffffffu
                                                              : ~(0xffffffffu << (uint32_t)(s1 - lo)));
        mf = m & fmask;
        mr = m & ~fmask;
    }
    const uint32_t cf = __popc(mf), cr = __popc(mr);
    uint32_t incf = cf, incr = cr;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t tf = __shfl_up_sync(0xffffffffu, incf, o);
        uint32_t tr = __shfl_up_sync(0xffffffffu, incr, o);
        if (lane >= o) {
            incf += tf;
            incr += tr;
        }
    }
    nf = __shfl_sync(0xffffffffu, incf, 31);
    nr = __shfl_sync(0xffffffffu, incr, 31);
    const uint32_t total = nf + nr;
    for (uint32_t g = 0; g < total; g += 32) {
        const uint32_t j = g + (uint32_t)lane;
        const bool v = j < total;
        const bool rev = j >= nf;
        const uint32_t jj = !v ? 0u : (rev ? j - nf : j);
        int L = 0;   /* first lane whose inclusive count (of this strand) exceeds jj */
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
            const uint32_t xf = __shfl_sync(0xffffffffu, incf, L + step - 1);
            const uint32_t xr = __shfl_sync(0xffffffffu, incr, L + step - 1);
            if ((rev ? xr : xf) <= jj) L += step;
        }
        const uint32_t wf = __shfl_sync(0xffffffffu, mf, L);
        const uint32_t wr = __shfl_sync(0xffffffffu, mr, L);
        const uint32_t bf = __shfl_sync(0xffffffffu, incf - cf, L);
        const uint32_t br = __shfl_sync(0xffffffffu, incr - cr, L);
        GsRec rec;
        rec.x = rec.y = 0;
        rec.l = 1u;
        rec.u = 0u;
        if (v) {
            const uint32_t word = rev ? wr : wf;
            const uint32_t bit = __fns(word, 0, (int)(jj - (rev ? br : bf)) + 1);
            rec = slots[((w0 + (uint64_t)L) << 5) + bit];
        }
        if (g == 0) mine = rec;
        __syncwarp();
        if (v) slots[(rev ? s1 : s0) + jj] = rec;
        __syncwarp();
    }
}

/* One strand of a read -- slots s0..s0+n -- compacted in place by one
 * thread: each flagged record moves to s0 + (its rank), in order, and the
 * rule decides it once its neighbour is known (forward: the next record,
 * one record behind; reverse: the previous one).  Adds the kept seeds and
 * their positions; returns the record count. */
__device__ __forceinline__ uint32_t gs_lane_compact(GsRec *slots, const uint32_t *mask, uint64_t s0,
                                                    uint32_t n, bool fwd, int smem,
                                                    uint32_t max_occ, uint64_t &seeds,
                                                    uint64_t &npos)
{
    const uint64_t s1 = s0 + n;
    uint32_t cnt = 0;
    GsRec prev;
    prev.x = prev.y = 0;
    prev.l = 1u;
    prev.u = 0u;
    bool keep;
    uint32_t c, xl, xu;
    for (uint64_t lo = s0 & ~31ull; lo < s1; lo += 32) {
        uint32_t m = mask[lo >> 5];
        if (lo < s0) m &= 0xffffffffu << (uint32_t)(s0 - lo);
        if (lo + 32 > s1) m &= 0xffffffffu >> (uint32_t)(lo + 32 - s1);
        while (m) {
            const uint32_t b = (uint32_t)__ffs(m) - 1u;
            m &= m - 1u;
            const GsRec rec = slots[lo + b];
            slots[s0 + cnt] = rec;   /* at or before its source: read already */
            if (fwd) {
                if (cnt) gs_fwd_rule_v(prev, rec, true, smem, max_occ, keep, c, xl, xu);
            } else {
                gs_rev_rule_v(rec, prev, cnt > 0, smem, max_occ, keep, c, xl, xu);
            }
            if ((!fwd || cnt) && keep && c) {
                seeds++;
                npos += c;
            }
            prev = rec;
            cnt++;
        }
    }
    if (fwd && cnt) {
        gs_fwd_rule_v(prev, prev, false, smem, max_occ, keep, c, xl, xu);
        if (keep && c) {
            seeds++;
            npos += c;
        }
    }
    return cnt;
}

/* reads whose two strands span at most this many slots are compacted by one
 * lane; longer ones by the whole warp */
#define GS_LANE_SLOTS 512u

/* a read compacted and counted by the whole warp (long reads); lane 0 adds
 * its seeds and positions to the sums */
__device__ __noinline__ void gs_finalize_read_warp(const GsBatch &B, uint32_t r, uint64_t base,
                                                   uint64_t next, int lane, uint64_t &sum_s,
                                                   uint64_t &sum_p)
{
    uint32_t n = (uint32_t)((next - base) >> 1);
    GsRec *F = B.slots + base;
    GsRec *Rv = F + n;
    uint32_t nf, nr;
    uint64_t seeds = 0, npos = 0;
    bool done = false;
    if (2u * n + 31u <= 1024u) {
        GsRec mine;
        gs_warp_compact_both(B.slots, B.recmask, base, n, lane, nf, nr, mine);
        if (nf + nr <= 32u) {
            /* lane j holds record j of [forward | reverse]: the rules'
             * neighbours are lanes j+1 (forward) and j-1 (reverse) */
            GsRec up, dn;
            up.x = __shfl_down_sync(0xffffffffu, mine.x, 1);
            up.y = __shfl_down_sync(0xffffffffu, mine.y, 1);
            up.l = __shfl_down_sync(0xffffffffu, mine.l, 1);
            up.u = __shfl_down_sync(0xffffffffu, mine.u, 1);
            dn.x = __shfl_up_sync(0xffffffffu, mine.x, 1);
            dn.y = __shfl_up_sync(0xffffffffu, mine.y, 1);
            dn.l = __shfl_up_sync(0xffffffffu, mine.l, 1);
            dn.u = __shfl_up_sync(0xffffffffu, mine.u, 1);
            const uint32_t j = (uint32_t)lane;
            bool keep = false;
            uint32_t cnt = 0, xl, xu;
            if (j < nf)
                gs_fwd_rule_v(mine, up, j + 1 < nf, B.smem, B.max_occ, keep, cnt, xl, xu);
            else if (j < nf + nr)
                gs_rev_rule_v(mine, dn, j > nf, B.smem, B.max_occ, keep, cnt, xl, xu);
            if (keep && cnt) {
                seeds = 1;
                npos = cnt;
            }
            done = true;
        }
    } else {
        nf = gs_warp_compact(B.slots, B.recmask, base, n, lane);
        nr = gs_warp_compact(B.slots, B.recmask, base + n, n, lane);
    }
    for (uint32_t o = lane; !done && o < nf; o += 32) {
        bool keep; uint32_t cnt, xl, xu;
        gs_fwd_rule(F, nf, o, B.smem, B.max_occ, keep, cnt, xl, xu);
        if (keep && cnt) { seeds++; npos += cnt; }
    }
    for (uint32_t o = lane; !done && o < nr; o += 32) {
        bool keep; uint32_t cnt, xl, xu;
        gs_rev_rule(Rv, nr, o, B.smem, B.max_occ, keep, cnt, xl, xu);
        if (keep && cnt) { seeds++; npos += cnt; }
    }
    for (int off = 16; off; off >>= 1) {
        seeds += __shfl_xor_sync(0xffffffffu, seeds, off);
        npos += __shfl_xor_sync(0xffffffffu, npos, off);
    }
    if (lane == 0) {
        B.rd_nf[r] = nf;
        B.rd_nr[r] = nr;
        B.rd_nseeds[r] = seeds;
        B.rd_npos[r] = npos;
        sum_s += seeds;
        sum_p += npos;
    }
}

/* Tiles of 256 reads, 32 consecutive ones per warp: a lane compacts and
 * counts its own read when it spans at most GS_LANE_SLOTS slots (few
 * instructions a read, the warp's loads spread over 32 reads); the warp then
 * takes its longer reads one at a time.  Small batches have tiles of 8 reads
 * and the warp takes its one read whatever its length (gs_finalize_tile).
 * The blocks' sums become the offsets of gs_finalize_emit. */
__global__ void __launch_bounds__(GS_SCAN_THREADS) gs_finalize_count(GsBatch B, uint32_t tile)
{
    gs_after_previous();
    const int lane = threadIdx.x & 31;
    const uint32_t per_warp = tile / (GS_SCAN_THREADS / 32u);
    uint32_t first, last;
    gs_part_reads(B.n_reads, tile, blockIdx.x, gridDim.x, first, last);
    uint64_t sum_s = 0, sum_p = 0;
    for (uint32_t r0 = first + (threadIdx.x >> 5) * per_warp; r0 < last; r0 += tile) {
        const uint32_t r = r0 + (uint32_t)lane;
        uint64_t base = 0, next = 0;
        bool longr = false;
        if (r < last && lane < (int)per_warp) {
            base = B.slot_off[r];
            next = B.slot_off[r + 1];
            if (next > B.slot_cap) {
                /* a replayed pass whose input needs more slots than it was
                 * sized for: nothing of this read is there; the host
                 * re-sizes */
                B.rd_nf[r] = 0;
                B.rd_nr[r] = 0;
                B.rd_nseeds[r] = 0;
                B.rd_npos[r] = 0;
                atomicOr(B.queue + 1, GS_FLAG_OVERFLOW);
            } else if (next - base > GS_LANE_SLOTS || per_warp == 1u) {
                longr = true;
            } else {
                const uint32_t n = (uint32_t)((next - base) >> 1);
                uint64_t seeds = 0, npos = 0;
                const uint32_t nf = gs_lane_compact(B.slots, B.recmask, base, n, true, B.smem,
                                                    B.max_occ, seeds, npos);
                const uint32_t nr = gs_lane_compact(B.slots, B.recmask, base + n, n, false,
                                                    B.smem, B.max_occ, seeds, npos);
                B.rd_nf[r] = nf;
                B.rd_nr[r] = nr;
                B.rd_nseeds[r] = seeds;
                B.rd_npos[r] = npos;
                sum_s += seeds;
                sum_p += npos;
            }
        }
        uint32_t lm = __ballot_sync(0xffffffffu, longr);
        while (lm) {
            const int src = __ffs(lm) - 1;
            lm &= lm - 1u;
            const uint64_t b0 = __shfl_sync(0xffffffffu, base, src);
            const uint64_t b1 = __shfl_sync(0xffffffffu, next, src);
            gs_finalize_read_warp(B, r0 + (uint32_t)src, b0, b1, lane, sum_s, sum_p);
        }
    }
    GsPart sum, total;
    gs_block_scan(sum_s, sum_p, sum);
    if (gs_parts_publish(B.parts, 1, sum, total) && threadIdx.x == 0) {
        B.totals[2] = total.a;
        B.totals[3] = total.b;
        if (B.h_totals) {
            B.h_totals[2] = total.a;
            B.h_totals[3] = total.b;
        }
    }
}

/* an output seed and, at the tiles of 32 positions that begin in it, its number */
__device__ __forceinline__ void gs_put_seed(const GsBatch &B, uint64_t *seed_pos, uint64_t s, uint64_t p,
                                            const gs_seed_rec &o)
{
    if (s >= B.seed_cap) return;
    B.seeds[s] = o;
    seed_pos[s] = p;
    for (uint64_t m = (p + 31u) >> 5; (m << 5) < p + o.n_pos && (m << 5) < B.pos_cap; m++)
        B.tile_seed[m] = (uint32_t)s;
}

/* A read's seeds from place s and position p, merged by begin by one thread,
 * from records a and b on. */
__device__ __forceinline__ void gs_emit_lane(const GsBatch &B, uint64_t *seed_pos, const GsRec *F, uint32_t nf,
                                             const GsRec *Rv, uint32_t nr, uint32_t a, uint32_t b,
                                             uint64_t s, uint64_t p)
{
    /* each record loaded once: the forward list's current and next, the
     * reverse list's current and previous */
    GsRec none;
    none.x = none.y = 0;
    none.l = 1u;
    none.u = 0u;
    GsRec fc = a < nf ? F[a] : none, fn = a + 1 < nf ? F[a + 1] : none;
    GsRec rc = b < nr ? Rv[b] : none, rp = b ? Rv[b - 1] : none;
    while (a < nf || b < nr) {
        bool take_f;
        if (a >= nf) take_f = false;
        else if (b >= nr) take_f = true;
        else take_f = ((uint32_t)fc.x & 0x7fffffffu) <= ((uint32_t)rc.x & 0x7fffffffu);
        bool keep; uint32_t cnt, xl, xu;
        GsRec R;
        if (take_f) {
            gs_fwd_rule_v(fc, fn, a + 1 < nf, B.smem, B.max_occ, keep, cnt, xl, xu);
            R = fc;
            a++;
            fc = fn;
            fn = a + 1 < nf ? F[a + 1] : none;
        } else {
            gs_rev_rule_v(rc, rp, b > 0, B.smem, B.max_occ, keep, cnt, xl, xu);
            R = rc;
            b++;
            rp = rc;
            rc = b < nr ? Rv[b] : none;
        }
        if (keep && cnt) {
            gs_seed_rec o;
            o.x = R.x; o.y = R.y; o.l = R.l; o.u = R.u;
            o.xl = xl; o.xu = xu; o.n_pos = cnt; o.pad = 0;
            gs_put_seed(B, seed_pos, s, p, o);
            s++;
            p += cnt;
        }
    }
}

/* how many of the warp's values, ascending by lane, are below v (or_equal: at
 * most v) */
__device__ __forceinline__ uint32_t gs_warp_below(uint32_t value, uint32_t v, bool or_equal)
{
    uint32_t k = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
        const uint32_t x = __shfl_sync(0xffffffffu, value, k + step - 1);
        if (or_equal ? x <= v : x < v) k += step;
    }
    const uint32_t x = __shfl_sync(0xffffffffu, value, k);
    return k + ((or_equal ? x <= v : x < v) ? 1u : 0u);
}

/* ... by the warp, 32 merged records a round: a record of the next 32 of its
 * list has its rank in the round by its lane and the other list's records
 * before it.  Both lists ascend by begin wherever a match has no longer one
 * ending before it; a round whose lists do not goes on with one thread. */
__device__ __forceinline__ void gs_emit_warp(const GsBatch &B, uint64_t *seed_pos, const GsRec *F, uint32_t nf,
                                             const GsRec *Rv, uint32_t nr, uint64_t s, uint64_t p, int lane,
                                             gs_seed_rec *round)
{
    uint32_t a = 0, b = 0;
    GsRec none;
    none.x = none.y = 0;
    none.l = 1u;
    none.u = 0u;
    while (a < nf || b < nr) {
        const uint32_t i = a + (uint32_t)lane, j = b + (uint32_t)lane;
        const bool hf = i < nf, hr = j < nr;
        const GsRec f = hf ? F[i] : none, fn = i + 1u < nf ? F[i + 1u] : none;
        const GsRec r = hr ? Rv[j] : none, rp = hr && j ? Rv[j - 1u] : none;
        const uint32_t fx = hf ? (uint32_t)f.x & 0x7fffffffu : 0xffffffffu;
        const uint32_t rx = hr ? (uint32_t)r.x & 0x7fffffffu : 0xffffffffu;
        const bool down = __shfl_up_sync(0xffffffffu, fx, 1) > fx || __shfl_up_sync(0xffffffffu, rx, 1) > rx;
        if (__any_sync(0xffffffffu, down)) {
            if (lane == 0) gs_emit_lane(B, seed_pos, F, nf, Rv, nr, a, b, s, p);
            return;
        }
        const uint32_t fk = (uint32_t)lane + gs_warp_below(rx, fx, false);
        const uint32_t rk = (uint32_t)lane + gs_warp_below(fx, rx, true);
        const bool tf = hf && fk < 32u, tr = hr && rk < 32u;
        bool keep; uint32_t cnt;
        gs_seed_rec o;
        o.pad = 0;
        if (tf) {
            gs_fwd_rule_v(f, fn, i + 1u < nf, B.smem, B.max_occ, keep, cnt, o.xl, o.xu);
            o.x = f.x; o.y = f.y; o.l = f.l; o.u = f.u;
            o.n_pos = keep ? cnt : 0u;
            round[fk] = o;
        }
        if (tr) {
            gs_rev_rule_v(r, rp, j > 0, B.smem, B.max_occ, keep, cnt, o.xl, o.xu);
            o.x = r.x; o.y = r.y; o.l = r.l; o.u = r.u;
            o.n_pos = keep ? cnt : 0u;
            round[rk] = o;
        }
        __syncwarp();
        const uint32_t na = (uint32_t)__popc(__ballot_sync(0xffffffffu, tf));
        const uint32_t nb = (uint32_t)__popc(__ballot_sync(0xffffffffu, tr));
        const bool in = (uint32_t)lane < na + nb;
        if (in) o = round[lane];
        const uint32_t n = in ? o.n_pos : 0u;
        unsigned long long sum = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long x = __shfl_up_sync(0xffffffffu, sum, d);
            if (lane >= d) sum += x;
        }
        const uint32_t kept = __ballot_sync(0xffffffffu, n != 0u);
        if (n) gs_put_seed(B, seed_pos, s + (uint32_t)__popc(kept & ((1u << lane) - 1u)), p + sum - n, o);
        s += (uint32_t)__popc(kept);
        p += __shfl_sync(0xffffffffu, sum, 31);
        a += na;
        b += nb;
        __syncwarp();
    }
}

/* A thread per read, or a warp where the tile has one a warp: its seeds' and
 * positions' offsets, and its seeds merged by begin. */
template <bool WARP>
__global__ void __launch_bounds__(GS_SCAN_THREADS) gs_finalize_emit(GsBatch B, uint64_t *seed_pos,
                                                                    uint32_t tile)
{
    gs_after_previous();
    __shared__ gs_seed_rec rounds[WARP ? GS_SCAN_THREADS : 1u];
    uint32_t first, last;
    gs_part_reads(B.n_reads, tile, blockIdx.x, gridDim.x, first, last);
    GsPart run = B.parts.part[blockIdx.x];
    if (last == B.n_reads && threadIdx.x == 0) {
        B.seed_off[B.n_reads] = B.totals[2] + B.base_s;
        B.pos_off[B.n_reads] = B.totals[3] + B.base_p;
    }
    /* the offsets of all the block's reads first: the merges below then need
     * no barrier, and a warp of short lists does not wait for one of long */
    for (uint32_t r0 = first; r0 < last; r0 += tile) {
        const uint32_t r = r0 + threadIdx.x;
        const bool in = r < last && threadIdx.x < tile;
        GsPart t;
        const GsPart x = gs_block_scan(in ? B.rd_nseeds[r] : 0ull, in ? B.rd_npos[r] : 0ull, t);
        if (in) {
            B.seed_off[r] = run.a + x.a + B.base_s;
            B.pos_off[r] = run.b + x.b + B.base_p;
        }
        run.a += t.a;
        run.b += t.b;
    }
    if (WARP) __syncthreads();   /* another thread's offsets */
    const uint32_t at = WARP ? threadIdx.x >> 5 : threadIdx.x;
    for (uint32_t r = at < tile ? first + at : last; r < last; r += tile) {
        const uint64_t s = B.seed_off[r] - B.base_s, p = B.pos_off[r] - B.base_p;
        const uint64_t base = B.slot_off[r];
        const uint32_t n = (uint32_t)((B.slot_off[r + 1] - base) >> 1);
        const GsRec *F = B.slots + base;
        const uint32_t nf = B.rd_nf[r], nr = B.rd_nr[r];
        if (WARP) gs_emit_warp(B, seed_pos, F, nf, F + n, nr, s, p, threadIdx.x & 31, rounds + (threadIdx.x & ~31u));
        else gs_emit_lane(B, seed_pos, F, nf, F + n, nr, 0, 0, s, p);
    }
}

/* GS_MEM_NEXT_GPUSEED (MEM mode).  seeds_to_threads_mem (seed_gen.cu:635-650)
 * looks for a kept record's exclusion interval among the compacted records
 * that follow it (forward: same begin) or precede it (reverse: same end),
 * and its scan does not stop at the read's end, while the count kernel's
 * does (:927-989).  Inside the read the scan finds the filters' own
 * neighbour.  It leaves the read only from the read's last forward record
 * when the read has no reverse record -- into the next read that has
 * records, whose first record is then forward -- and from the read's first
 * reverse record when the read has no forward record, into the previous
 * read's last record.  The record it meets heads (ends) a run whose last
 * (first) record is kept, and a dropped record has the interval of the
 * record it was dropped for, so the interval found is that of the other
 * read's first forward (last reverse) output seed, when the begin (end)
 * matches.  The seed keeps its count and its rows become the first n_pos
 * rows from l outside that interval.  Thread per read, after the emit. */
__global__ void __launch_bounds__(128) gs_mem_next_kernel(GsBatch B)
{
    gs_after_previous();
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= B.n_reads) return;
    const uint64_t s0 = B.seed_off[r], s1 = B.seed_off[r + 1];
    if (s0 == s1 || s1 > B.seed_cap) return;
    uint64_t last_f = s1, first_r = s1;
    for (uint64_t s = s0; s < s1; s++) {
        if ((uint32_t)B.seeds[s].y >> 31) {
            if (first_r == s1) first_r = s;
        } else {
            last_f = s;
        }
    }
    if (last_f < s1 && first_r == s1) {
        /* the next read with seeds; its first seed in output order is
         * forward exactly when it has forward records */
        uint32_t q = r + 1;
        while (q < B.n_reads && B.seed_off[q + 1] == B.seed_off[q]) q++;
        if (q < B.n_reads && B.seed_off[q + 1] <= B.seed_cap) {
            for (uint64_t s = B.seed_off[q]; s < B.seed_off[q + 1]; s++) {
                const gs_seed_rec N = B.seeds[s];
                if ((uint32_t)N.y >> 31) continue;
                if (N.x == B.seeds[last_f].x) {
                    B.seeds[last_f].xl = N.l;
                    B.seeds[last_f].xu = N.u;
                }
                break;
            }
        }
    }
    if (first_r < s1 && last_f == s1 && r > 0) {
        uint32_t q = r - 1;
        while (q > 0 && B.seed_off[q + 1] == B.seed_off[q]) q--;
        if (B.seed_off[q + 1] > B.seed_off[q] && B.seed_off[q + 1] <= B.seed_cap) {
            for (uint64_t s = B.seed_off[q + 1]; s-- > B.seed_off[q];) {
                const gs_seed_rec P = B.seeds[s];
                if (!((uint32_t)P.y >> 31)) continue;
                if (P.y == B.seeds[first_r].y) {
                    B.seeds[first_r].xl = P.l;
                    B.seeds[first_r].xu = P.u;
                }
                break;
            }
        }
    }
}

/* Positions: a warp takes a tile of them, 32 a round (they span at most 32
 * seeds, as every seed has a position), from the seed of the round's first
 * position, which gs_finalize_emit noted.  It writes the position -> seed map
 * for the text records and resolves each row.  A seed of many positions is
 * spread over many warps.  Tiles of 32 to 256, so that few positions spread
 * over many warps.
 *
 * With the full suffix array a row is one read.  Else it is a chain of LF
 * steps, up to sa_intv - 1 of them, whose latency bounds the kernel: a tile's
 * rows go through shared memory, and a lane whose row is resolved takes the
 * next, so that a warp does not wait for the longest chain of each 32 (1 M
 * reads on 100 Mbp, 2.3 M positions 246 -> 208 us; 150,001 reads 166 -> 131).
 * A tile of one round has nothing to hand out: each lane runs its own chain
 * (10,000 reads on 1 Mbp 35 us, 47 through shared memory). */
#define GS_LOCATE_MOST 256u

/* the row of position p (in the round from pb), and its seed */
__device__ __forceinline__ uint32_t gs_position_row(const GsBatch &B, uint64_t pb, uint64_t p, bool in,
                                                    uint64_t n_seeds, int lane)
{
    /* plain loads: the kernel before this one, which may not have ended when
     * this one starts, writes all of these */
    const uint64_t s0 = B.tile_seed[pb >> 5];
    /* first positions of seeds s0+1 .. s0+32 */
    const uint64_t at = s0 + 1u + (uint64_t)lane;
    const uint64_t next = at < n_seeds ? B.seed_pos[at] : ~0ull;
    int k = 0;   /* how many of them are at or before p */
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1)
        if (__shfl_sync(0xffffffffu, next, k + step - 1) <= p) k += step;
    if (__shfl_sync(0xffffffffu, next, k) <= p) k++;
    const uint64_t s = s0 + (uint64_t)k;
    if (!in) return 0u;
    const uint4 *rec = reinterpret_cast<const uint4 *>(B.seeds + s);
    const uint4 S = rec[0], T = rec[1];   /* x y l u, xl xu n_pos pad */
    /* the (p - first)-th row from l outside [xl, xu] */
    uint32_t row = S.z + (uint32_t)(p - B.seed_pos[s]);
    B.pmap[p] = (uint32_t)s;
    const uint32_t x0 = T.x > S.z ? T.x : S.z;
    if (T.x <= T.y && T.y >= x0 && row >= x0) row += T.y - x0 + 1u;
    return row;
}

template <bool SAF>
__global__ void __launch_bounds__(256, 8) gs_locate(GsDevIndex I, GsBatch B)
{
    __shared__ uint32_t rows[SAF ? 1 : 8][GS_LOCATE_MOST];
    gs_after_previous();
    /* a replayed pass with more output than it was sized for: the host sees
     * the totals and sizes it again */
    const uint64_t n_pos = B.totals[3], n_seeds = B.totals[2];
    if (n_pos > B.pos_cap || n_seeds > B.seed_cap || n_seeds == 0) return;
    const int lane = threadIdx.x & 31;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint32_t cap = I.seq_len + 2u;
    const uint64_t share = ((n_pos + nwarps - 1) / nwarps + 31u) & ~31ull;
    const uint64_t tile = share < GS_LOCATE_MOST ? share : GS_LOCATE_MOST;
    for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * tile < n_pos;
         w += nwarps) {
        const uint64_t p0 = w * tile;
        const uint32_t n = (uint32_t)(p0 + tile < n_pos ? tile : n_pos - p0);
        if (SAF) {
            /* the chain's result is SA[row], except that the LF quirk sends
             * the rows whose chain passes row primary+1 to row 0, where
             * sa[0] = -1 gives the steps taken minus one: position -
             * quirk_lo. */
            for (uint32_t i0 = 0; i0 < n; i0 += 32) {
                const uint64_t p = p0 + i0 + (uint32_t)lane;
                const bool in = i0 + (uint32_t)lane < n;
                const uint32_t row = gs_position_row(B, p0 + i0, p, in, n_seeds, lane);
                if (!in) continue;
                uint32_t v = gs_ld64(&I.saf[row]);
                if (B.lf_mode == GS_LF_GPUSEED && v - I.quirk_lo < I.quirk_n) v -= I.quirk_lo;
                B.pos[p] = v;
            }
            if (B.work && lane == 0) atomicAdd(&B.work[3], (unsigned long long)n);
            continue;
        }
        /* locate_seeds_gpu (:668-684): LF until a sampled row; a consistent
         * index reaches one within seq_len+1 steps */
        unsigned long long all = 0;
        const auto resolve = [&](uint64_t p, uint32_t row, uint32_t steps) {
            uint32_t v = 0xffffffffu;
            if (steps > cap) atomicOr(B.queue + 1, GS_FLAG_WALK);
            else v = __ldg(&I.sa[row / I.sa_intv]) + steps;
            B.pos[p] = v;
            all += steps;
        };
        if (n <= 32u) {
            const uint64_t p = p0 + (uint32_t)lane;
            uint32_t row = gs_position_row(B, p0, p, (uint32_t)lane < n, n_seeds, lane), steps = 0;
            if ((uint32_t)lane < n) {
                while (row % I.sa_intv && steps <= cap) {
                    row = gs_lf(I, row, B.lf_mode);
                    steps++;
                }
                resolve(p, row, steps);
            }
        } else {
            uint32_t *list = rows[threadIdx.x >> 5];
            for (uint32_t i0 = 0; i0 < n; i0 += 32) {
                const uint32_t i = i0 + (uint32_t)lane;
                const uint32_t row = gs_position_row(B, p0 + i0, p0 + i, i < n, n_seeds, lane);
                if (i < n) list[i] = row;
            }
            __syncwarp();
            uint32_t i = 0, row = 0, steps = 0, taken = 0;
            bool have = false;
            for (;;) {
                const uint32_t need = __ballot_sync(0xffffffffu, !have);
                if (need && taken < n) {
                    if (!have) {
                        i = taken + (uint32_t)__popc(need & ((1u << lane) - 1u));
                        have = i < n;
                        if (have) {
                            row = list[i];
                            steps = 0;
                        }
                    }
                    taken += (uint32_t)__popc(need);
                } else if (need == 0xffffffffu) {
                    break;
                }
                if (have) {
                    if (row % I.sa_intv == 0 || steps > cap) {
                        resolve(p0 + i, row, steps);
                        have = false;
                    } else {
                        row = gs_lf(I, row, B.lf_mode);
                        steps++;
                    }
                }
            }
            __syncwarp();
        }
        if (B.work) {
            for (int off = 16; off; off >>= 1) all += __shfl_xor_sync(0xffffffffu, all, off);
            if (lane == 0) {
                atomicAdd(&B.work[2], all);
                atomicAdd(&B.work[3], (unsigned long long)n);
            }
        }
    }
}

/* Reads of a block of gs_finalize_count and _emit: a warp's each, or a lane's.
 * A lane's way through its read's mask words and records is one chain of
 * loads: 34 us for the count of 300 reads of 100 to 250 bases and 17 for
 * their merges, against 9 and 6 by the warp.  10,000 reads of 100 keep enough
 * lanes busy (13 and 7 us, 19 and 13 by the warp), so the line lies between.
 * Long reads are a warp's work in any number, by their average, 16 items of a
 * strand's candidates (about GS_LANE_SLOTS): 40,000 reads of 2 kbp, blocks of
 * 256 on an SM each, 409 -> 186 us and 355 -> 110. */
#define GS_WARP_READS 4096u

static bool gs_finalize_by_warp(const GsBatch &B)
{
    return B.n_reads <= GS_WARP_READS || (uint64_t)B.item_cap * (B.paired ? 2u : 1u) > 16ull * B.n_reads;
}

static uint32_t gs_finalize_tile(const GsBatch &B)
{
    return gs_finalize_by_warp(B) ? GS_SCAN_THREADS / 32u : GS_SCAN_THREADS;
}

int gs_launch_finalize_count(const GsDevIndex &I, GsBatch &B, cudaStream_t st)
{
    (void)I;
    const uint32_t tile = gs_finalize_tile(B);
    GS_CUDA(gs_launch_after(gs_finalize_count, gs_parts_of(B.n_reads, tile), GS_SCAN_THREADS, st, B, tile));
    return GS_OK;
}

int gs_launch_finalize_emit(const GsDevIndex &I, GsBatch &B, cudaStream_t st)
{
    (void)I;
    const uint32_t tile = gs_finalize_tile(B);
    void (*emit)(GsBatch, uint64_t *, uint32_t) =
        gs_finalize_by_warp(B) ? gs_finalize_emit<true> : gs_finalize_emit<false>;
    GS_CUDA(gs_launch_after(emit, gs_parts_of(B.n_reads, tile), GS_SCAN_THREADS, st, B, B.seed_pos, tile));
    if (B.n_reads && !B.smem && B.mem_next == GS_MEM_NEXT_GPUSEED) {
        gs_mem_next_kernel<<<(B.n_reads + 127) / 128, 128, 0, st>>>(B);
        GS_CUDA(cudaGetLastError());
    }
    return GS_OK;
}

int gs_launch_locate(const GsDevIndex &I, GsBatch &B, uint64_t n_pos, cudaStream_t st)
{
    if (B.n_reads == 0 || B.seed_cap == 0 || B.pos_cap == 0 || n_pos == 0) return GS_OK;
    uint64_t n = n_pos < B.pos_cap ? n_pos : B.pos_cap;
    /* eight warps a block, a round of positions each, at most what is
     * resident, 8 blocks an SM (twice that where a position is one read) */
    const uint64_t most = 152ull * (I.saf ? 16u : 8u);
    uint64_t grid = (n + 255) / 256;
    if (grid > most) grid = most;
    GS_CUDA(gs_launch_after(I.saf ? gs_locate<true> : gs_locate<false>, (unsigned)grid, 256, st, I, B));
    return GS_OK;
}
