/*
 * gs_search.cu -- seed-interval search (the hot path).
 *
 * Semantics (restated from find_seed_intervals_gpu, seed_gen.cu:2087-2413):
 *   forward candidate e (end):   13-mer R[e-12..e] from the k-mer table, then
 *                                extend left while the interval stays valid;
 *                                record ([b, e+1), I) if e+1-b >= k;
 *   reverse candidate s (start): complement codes, 13-mer at s, extend right;
 *                                record ([s, x+1) | bit 31, I) if x+1-s >= k.
 * A candidate may stop early once its interval has the same size as that of
 * its neighbour toward the longer match (e+1 forward, s-1 reverse) at the
 * same far end: both filters drop such a record, so it need not be produced.
 * The reference prunes with 30 warp shuffles per step over uninitialised
 * flags (:2100-2204); this file uses a defined rule with three launch forms:
 *
 *   GS_KERNEL_BATCHED (default): gs_search_start + gs_search_walk (+
 *     gs_search_text, gs_search_leftover).  Each candidate carries the
 *     interval of its neighbour's string at its own far end and stops
 *     exactly where the rule says; candidates are started a warp per work
 *     item and walked one per lane (see "batched search").
 *   GS_KERNEL_LOCKSTEP: gs_search_lockstep + gs_search_tail.  Persistent
 *     CTAs; each warp takes work items (read, strand, 31 candidates + 1
 *     helper lane) from a global queue and steps its 32 candidates in
 *     lockstep, comparing with the nearest still-extending lane to the right
 *     from a GS_HIST-deep own history; the last candidates of a warp go to a
 *     tail pass.
 *   GS_KERNEL_PLAIN: gs_search_plain, one thread per read, candidates one
 *     after another, containment history in a per-read global array.
 */
#include "gs_fm.cuh"
#include "gs_scan.cuh"



/* ------------------------------------------------------------------ */
/* 13-mer interval table (pre_calc_seed_intervals_gpu, seed_gen.cu:2648) */

/* The intervals of all strings of LV more bases than one whose interval is
 * [l,u], each from the string one base shorter: an absent string keeps the
 * empty interval at which it ended.  put(ext, l, u) gets each, the base
 * processed first at bits 0-1 of ext. */
template <int LV, class F>
__device__ __forceinline__ void gs_kmer_expand(const GsDevIndex &I, uint32_t l, uint32_t u, int at,
                                               uint32_t ext, const F &put)
{
    if constexpr (LV == 0) {
        put(ext, l, u);
    } else {
        for (uint32_t c = 0; c < 4; c++) {
            uint32_t cl = l, cu = u;
            if (l <= u) gs_step(I, cl, cu, c);
            gs_kmer_expand<LV - 1>(I, cl, cu, at + 1, ext | (c << (2 * at)), put);
        }
    }
}

/* A thread per 10-mer: its interval, then its 64 13-mers, 94 steps instead
 * of 13 for each (loading a 400 Mbp index, with its 15-mer table made the
 * same way: 139 -> 102 ms) */
__global__ void __launch_bounds__(256) gs_kmer_kernel(GsDevIndex I, uint2 *table)
{
    const int head = GS_K0 - 3;
    const uint32_t patt = blockIdx.x * blockDim.x + threadIdx.x;
    if (patt >= (1u << (2 * head))) return;
    uint32_t l = 0, u = I.seq_len;
    for (int i = 0; i < head; i++) {
        gs_step(I, l, u, (patt >> (i << 1)) & 3u);
        if (l > u) break;
    }
    gs_kmer_expand<3>(I, l, u, 0, 0u, [&](uint32_t ext, uint32_t cl, uint32_t cu) {
        table[patt | (ext << (2 * head))] = make_uint2(cl, cu);
    });
}

int gs_build_kmer_table(const GsDevIndex &I, uint2 *table, cudaStream_t st)
{
    gs_kmer_kernel<<<(1u << (2 * (GS_K0 - 3))) / 256, 256, 0, st>>>(I, table);
    GS_CUDA(cudaGetLastError());
    return GS_OK;
}

/* Start table, built in four passes over all kx-mers (base j at
 * bits 2j, processed first, i.e. the string's last character sits at bits
 * 0-1):
 *   1. (l,u) from the 13-mer prefix interval plus kx-13 steps;
 *   2. what follows each kx-mer X: the forced right extension, i.e. the base
 *      c with count(Xc) == count(X) > 0, if any; for an X of one to three
 *      rows, the base after each row's X.  Xc's interval is one step with X's
 *      first character from the kx-mer table entry of (X without its first
 *      character)·c;
 *   3. packing: entry.x = l, entry.y = the size, the forced base and what the
 *      rows' left contexts are (gs_entry_* below);
 *   4. entry.z, entry.w = the packed entry of gs_kmer_rc(X), the kx-mer of
 *      X's reverse complement in the same bit order.
 * A candidate whose kx-mer is always followed by its neighbour's next base is
 * contained in that neighbour (see the file comment) and needs no walk;
 * gs_search_plain stops such candidates at their start.  A read's window
 * R[s..s+kx-1] is the start string of its forward candidate ending at
 * s+kx-1 and, as complement codes, of its reverse candidate starting at s:
 * the two keys are X and gs_kmer_rc(X), so one 16-byte entry starts both. */
__device__ __forceinline__ uint32_t gs_kmer_rc(uint32_t X, int kx)
{
    /* complement every base (3 - c = c ^ 3), then reverse the order of the
     * kx 2-bit groups */
    const uint32_t b = __brev(~X);
    return (((b >> 1) & 0x55555555u) | ((b & 0x55555555u) << 1)) >> (32 - 2 * kx);
}

/* a thread per 13-mer: the intervals of its 4^(kx-13) kx-mers */
template <int LV>
__global__ void __launch_bounds__(256) gs_kmerx_kernel(GsDevIndex I, uint4 *table)
{
    const uint32_t patt = blockIdx.x * blockDim.x + threadIdx.x;
    const uint2 iv = __ldg(&I.kmer[patt]);
    gs_kmer_expand<LV>(I, iv.x, iv.y, 0, 0u, [&](uint32_t ext, uint32_t l, uint32_t u) {
        table[patt | ((uint64_t)ext << (2 * GS_K0))] = make_uint4(l, u, 0u, 0u);
    });
}

/* What follows X = [l,u] (pass 2): c with count(Xc) == count(X) > 0, or 4;
 * for one to three rows whose X all have a base after them, GS_RIGHTS | the
 * rows' bases in row order (rows are sorted by what follows X), 2 bits each.
 * raw(Y): the interval of a kx-mer. */
#define GS_RIGHTS 0x40u
#define GS_ROWS_MOST 3u

template <class F>
__device__ __forceinline__ uint32_t gs_right_code(const GsDevIndex &I, uint64_t X, int kx, uint32_t l,
                                                  uint32_t u, const F &raw)
{
    if (l > u) return 4u;
    const uint64_t mask = (1ull << (2 * kx)) - 1u;
    const uint32_t size = u - l + 1u, first = (uint32_t)(X >> (2 * (kx - 1))) & 3u;   /* X's first character */
    const bool few = size <= GS_ROWS_MOST;
    uint32_t forced = 4u, rows = 0u, rights = 0u;
    for (uint32_t c = 0; c < 4; c++) {
        uint2 y = raw(((X << 2) | c) & mask);
        /* as many rows as X's at most come before the step */
        if (y.x > y.y || (!few && y.y - y.x + 1u < size)) continue;
        gs_step(I, y.x, y.y, first);
        const uint32_t n = y.x <= y.y ? y.y - y.x + 1u : 0u;
        if (n == size) forced = c;
        if (!few) {
            if (n == size) break;
            continue;
        }
        for (uint32_t i = 0; i < n; i++) rights |= c << (2u * (rows + i));
        rows += n;
    }
    return few && rows == size ? GS_RIGHTS | rights : forced;
}

/* The X of a block's GS_DENSE that occur, dense: most kx-mers of a table of
 * about as many entries as the text has bases occur nowhere, and the chains
 * of loads of the others, which bound these kernels, would hold warps of a few
 * busy lanes.  entry(X): the interval; none(X, iv) and some(X, iv): what is
 * done for either.  The 13-mer entries of ten million bases, 1.6 ms with a
 * thread per entry, take 0.77 in blocks of 32 registers a thread, 8 an SM, and
 * 0.87 in 5 an SM; one round of blocks after another overlaps one's chains
 * with the next's entries, where blocks, or warps, that stay and keep what is
 * left over for their next entries take 1.2 and 1.0 ms. */
#define GS_DENSE 2048u

template <class E, class N, class S>
__device__ __forceinline__ void gs_dense(const E &entry, const N &none, const S &some)
{
    __shared__ uint16_t list[GS_DENSE];
    __shared__ uint32_t count;
    const uint64_t X0 = (uint64_t)blockIdx.x * GS_DENSE;
    const uint32_t lane = threadIdx.x & 31u;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < GS_DENSE; i += 256u) {
        const uint2 iv = entry(X0 + i);
        const bool occurs = iv.x <= iv.y;
        if (!occurs) none(X0 + i, iv);
        const uint32_t m = __ballot_sync(0xffffffffu, occurs);
        uint32_t at = 0;
        if (lane == 0 && m) at = atomicAdd(&count, (uint32_t)__popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (occurs) list[at + __popc(m & ((1u << lane) - 1u))] = (uint16_t)i;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < count; i += 256u) {
        const uint64_t X = X0 + list[i];
        some(X, entry(X));
    }
}

__global__ void __launch_bounds__(256, 8) gs_kmerx_code_kernel(GsDevIndex I, const uint4 *table, int kx,
                                                            uint8_t *code)
{
    const auto entry = [&](uint64_t X) {
        const uint4 e = table[X];
        return make_uint2(e.x, e.y);
    };
    gs_dense(
        entry, [&](uint64_t X, uint2) { code[X] = 4u; },
        [&](uint64_t X, uint2 iv) { code[X] = (uint8_t)gs_right_code(I, X, kx, iv.x, iv.y, entry); });
}

/* A packed half entry's second word (the first is l).  Bits 0-2:
 *   5, 6, 7  one, two, three rows, each with the bases before its X (nearest
 *            in the high bits) and the base after: six before, 14 bits a
 *            row from bit 3 (one and two rows), or three, 8 bits (three);
 *   0-3, 4   the forced base, or none, and
 *     bit 3 set: at most GS_EXT_ROWS rows, and
 *       bits 4-11  the size
 *       bits 12-15 base c: exactly one row of X is preceded by c
 *       bits 16-31 bit 4*c + d: some row of X is preceded by c, and that by d
 *     bit 3 clear: bits 4-31 the size (4 and size 0: it does not fit).
 * (Rows whose context reaches an end of the text take the second form.)
 * A candidate whose extension by the bases its read has next does not occur
 * can reach no minimum length past it, and one whose extension is a single
 * row that its neighbour's string shares is contained there: both end at
 * their start, without a walk.  A walk is a chain of dependent loads, and most
 * are of strings that a chance hit keeps alive for a base or two.  What the
 * forms are worth: the extensions (with the item's bases loaded by the warp,
 * and its read from a map) 7.6 of 24.2 ms of a 2 M-read SMEM pass on 3.1 Gbp,
 * 3.2 of 10.4 of a 40,000-read (2 kbp) MEM pass, 2.6 of 10.5 of a 1 M-read pass
 * on 100 Mbp; the few rows' contexts, by which a start plays its walk out over
 * up to six bases, its neighbour's with it, a quarter (3.1 Gbp) to half (100
 * Mbp) of the walkers that are left, 1.17, 0.44 and 0.75 ms of the same three.
 * 255 rows is what the size's byte holds. */
#define GS_EXT_ROWS 255u
#define GS_ENTRY_EXT 8u
#define GS_ENTRY_WIDE 4u

__device__ __forceinline__ uint32_t gs_entry_rows(uint32_t y) { return (y & 7u) > 4u ? (y & 7u) - 4u : 0u; }

__device__ __forceinline__ uint32_t gs_entry_size(uint32_t y)
{
    const uint32_t rows = gs_entry_rows(y);
    return rows ? rows : (y & GS_ENTRY_EXT) ? (y >> 4) & 255u : y >> 4;
}

/* row i's context in an entry of n rows: the bases before it in 12 bits (the
 * last six 0 where there are three), and the base after */
__device__ __forceinline__ void gs_entry_row(uint32_t y, uint32_t n, uint32_t i, uint32_t &left,
                                             uint32_t &right)
{
    const bool six = n < 3u;
    const uint32_t f = y >> (3u + i * (six ? 14u : 8u));
    left = six ? f & 0xfffu : (f & 0x3fu) << 6;
    right = (six ? f >> 12 : f >> 6) & 3u;
}

/* the forced base, or 4 */
__device__ __forceinline__ uint32_t gs_entry_forced(uint32_t y)
{
    const uint32_t n = gs_entry_rows(y);
    if (!n) return y & 7u;
    uint32_t left, first, right;
    gs_entry_row(y, n, 0u, left, first);
    uint32_t forced = first;
    for (uint32_t i = 1; i < n; i++) {
        gs_entry_row(y, n, i, left, right);
        if (right != first) forced = 4u;
    }
    return forced;
}

/* The second word of X = [l,u] from what follows it (gs_right_code).  Rows
 * l..u are read in order (their blocks, and those of their LF rows, are
 * shared by neighbouring entries, whose strings and so whose rows are
 * adjacent). */
__device__ __forceinline__ uint32_t gs_entry_word(const GsDevIndex &I, uint32_t l, uint32_t u,
                                                  uint32_t code)
{
    const uint32_t size = l <= u ? u - l + 1u : 0u;
    if (size >= (1u << 28)) return GS_ENTRY_WIDE;
    if (code & GS_RIGHTS) {
        const bool six = size < 3u;
        uint32_t y = 4u + size;
        bool end = false;
        for (uint32_t i = 0; i < size && !end; i++) {
            uint32_t row = l + i, left = 0;
            for (int at = six ? 10 : 4; at >= 0 && !end; at -= 2) {
                end = row == I.primary;   /* the text begins here */
                if (end) break;
                const GsBlk B = gs_load_block(I.occ, row);
                const uint32_t c = gs_block_base(B, row);
                left |= c << at;
                if (at) row = gs_block_lf(B, row, c);
            }
            const uint32_t right = (code >> (2u * i)) & 3u;
            y |= (left | right << (six ? 12 : 6)) << (3u + i * (six ? 14u : 8u));
        }
        if (!end) return y;
        /* all rows followed by one base: forced */
        uint32_t forced = code & 3u;
        for (uint32_t i = 1; i < size; i++)
            if (((code >> (2u * i)) & 3u) != (code & 3u)) forced = 4u;
        code = forced;
    }
    if (size > GS_EXT_ROWS) return code | (size << 4);
    uint32_t seen = 0, multi = 0, two = 0, at = 0xffffffffu;
    GsBlk B;
    for (uint32_t i = 0; i < size; i++) {
        const uint32_t row = l + i;
        if (row == I.primary) continue;   /* the text starts with X */
        if ((row >> 6) != at) {
            at = row >> 6;
            B = gs_load_block(I.occ, row);
        }
        const uint32_t c = gs_block_base(B, row);
        multi |= seen & (1u << c);
        seen |= 1u << c;
        const uint32_t prev = gs_block_lf(B, row, c);
        if (prev == I.primary) continue;   /* ... with cX */
        const GsBlk P = gs_load_block(I.occ, prev);
        two |= 1u << (4u * c + gs_block_base(P, prev));
    }
    return code | GS_ENTRY_EXT | (size << 4) | ((seen & ~multi) << 12) | (two << 16);
}

#define GS_ENTRY_NONE (4u | GS_ENTRY_EXT)   /* no rows */

__global__ void __launch_bounds__(256, 8) gs_kmerx_pack_kernel(GsDevIndex I, uint4 *table, const uint8_t *code)
{
    gs_dense(
        [&](uint64_t X) {
            const uint4 e = table[X];
            return make_uint2(e.x, e.y);
        },
        [&](uint64_t X, uint2 iv) { table[X] = make_uint4(iv.x, GS_ENTRY_NONE, 0u, 0u); },
        [&](uint64_t X, uint2 iv) {
            table[X] = make_uint4(iv.x, gs_entry_word(I, iv.x, iv.y, code[X]), 0u, 0u);
        });
}

/* Passes 1 to 3 at once for kx = 13, whose raw intervals are the 13-mer
 * table's.  (Pass 4 follows.)  Texts of up to 2^26 bases start from this
 * table: nearly every 13-mer of theirs is forced or dead at once, where the
 * plain table left every candidate to the walk (10,000 reads on 1 Mbp, a
 * replayed pass: 430 -> 373 us), for 1 GiB and about 1.5 ms at load. */
__global__ void __launch_bounds__(256, 8) gs_kmer13_entries_kernel(GsDevIndex I, uint4 *table)
{
    const auto entry = [&](uint64_t X) { return __ldg(&I.kmer[X]); };
    gs_dense(
        entry, [&](uint64_t X, uint2 iv) { table[X] = make_uint4(iv.x, GS_ENTRY_NONE, 0u, 0u); },
        [&](uint64_t X, uint2 iv) {
            const uint32_t code = gs_right_code(I, X, GS_K0, iv.x, iv.y, entry);
            table[X] = make_uint4(iv.x, gs_entry_word(I, iv.x, iv.y, code), 0u, 0u);
        });
}

/* Pass 4: each entry's second half from the packed first half of its reverse
 * complement's entry.
 *
 * A transposition: with the first and last three bases free and the others
 * fixed to M, 64 x 64 entries in runs of 64 by the last three, whose partners
 * are those of M's reverse complement, by the first three.  A block holds
 * both tiles' first halves and writes both tiles' entries, all by the run.
 * Bound by HBM, an entry read and written once: 1 GiB (kx = 13) in 0.53 ms,
 * 4.1 TB/s, where one 8-byte read at a random place per entry took 1.67 ms.
 * A tile's row is kept where the reverse complement of its first bases says,
 * so that what a run of the other tile takes lies one row apart, and a row is
 * one entry longer than the run, so that those lie in different banks. */
#define GS_PAIR_RUN 64u
#define GS_PAIR_PITCH (GS_PAIR_RUN + 1u)
#define GS_PAIR_SHARED (2u * GS_PAIR_RUN * GS_PAIR_PITCH * (uint32_t)sizeof(uint2))

__global__ void __launch_bounds__(256) gs_kmerx_pair_kernel(uint4 *table, int kx)
{
    extern __shared__ uint2 tile[];
    const uint32_t nm = 1u << (2 * (kx - 6));
    for (uint32_t M = blockIdx.x; M < nm; M += gridDim.x) {
        const uint32_t RM = gs_kmer_rc(M, kx - 6);
        if (RM < M) continue;   /* its partner's */
        const uint32_t tiles = RM == M ? 1u : 2u;   /* its own partner */
        for (uint32_t i = threadIdx.x; i < tiles * 4096u; i += 256u) {
            const uint32_t q = i >> 12, h = (i >> 6) & 63u, l = i & 63u;
            const uint64_t X = ((uint64_t)h << (2 * (kx - 3))) | ((uint64_t)(q ? RM : M) << 6) | l;
            tile[(q * GS_PAIR_RUN + gs_kmer_rc(h, 3)) * GS_PAIR_PITCH + l] =
                *reinterpret_cast<const uint2 *>(table + X);
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < tiles * 4096u; i += 256u) {
            const uint32_t q = i >> 12, h = (i >> 6) & 63u, l = i & 63u, rh = gs_kmer_rc(h, 3);
            const uint64_t X = ((uint64_t)h << (2 * (kx - 3))) | ((uint64_t)(q ? RM : M) << 6) | l;
            const uint2 a = tile[(q * GS_PAIR_RUN + rh) * GS_PAIR_PITCH + l];
            const uint2 b = tile[((tiles - 1u - q) * GS_PAIR_RUN + l) * GS_PAIR_PITCH + rh];
            table[X] = make_uint4(a.x, a.y, b.x, b.y);
        }
        __syncthreads();
    }
}

static cudaError_t gs_kmerx_pair(uint4 *table, int kx, cudaStream_t st)
{
    cudaError_t e = cudaFuncSetAttribute(gs_kmerx_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)GS_PAIR_SHARED);
    if (e != cudaSuccess) return e;
    gs_kmerx_pair_kernel<<<152 * 3, 256, GS_PAIR_SHARED, st>>>(table, kx);
    return cudaGetLastError();
}

int gs_build_kmerx_table(const GsDevIndex &I, uint4 *table, int kx, cudaStream_t st)
{
    const uint64_t n = 1ull << (2 * kx);
    const uint32_t n13 = 1u << (2 * GS_K0);
    if (kx == GS_K0) {
        gs_kmer13_entries_kernel<<<n13 / GS_DENSE, 256, 0, st>>>(I, table);
        GS_CUDA(cudaGetLastError());
        GS_CUDA(gs_kmerx_pair(table, kx, st));
        return GS_OK;
    }
    void (*expand)(GsDevIndex, uint4 *) = kx == 14   ? gs_kmerx_kernel<1>
                                          : kx == 15 ? gs_kmerx_kernel<2>
                                                     : gs_kmerx_kernel<3>;
    expand<<<n13 / 256, 256, 0, st>>>(I, table);
    GS_CUDA(cudaGetLastError());
    uint8_t *code = NULL;
    GS_CUDA(cudaMallocAsync(&code, n, st));
    gs_kmerx_code_kernel<<<(unsigned)(n / GS_DENSE), 256, 0, st>>>(I, table, kx, code);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) {
        gs_kmerx_pack_kernel<<<(unsigned)(n / GS_DENSE), 256, 0, st>>>(I, table, code);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = gs_kmerx_pair(table, kx, st);
    cudaFreeAsync(code, st);
    if (e != cudaSuccess) return gs_cuda_fail(e, "k-mer start table");
    return GS_OK;
}

/* a start-table entry: one random 8-byte load whose L2 fill is 64 bytes
 * (the default fills 128 for random loads; the table's lookups are bound by
 * the DRAM access rate, and the start pass also streams the walker buffer) */
__device__ __forceinline__ uint2 gs_ld_entry(const uint2 *p)
{
    uint2 v;
    asm("ld.global.nc.L2::64B.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

/* both halves of a paired start-table entry: one 16-byte load, the same
 * 64-byte L2 fill */
__device__ __forceinline__ uint4 gs_ld_pair(const uint4 *p)
{
    uint4 v;
    asm("ld.global.nc.L2::64B.v4.u32 {%0,%1,%2,%3}, [%4];"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p));
    return v;
}

/* The start from the 13-mer table: the interval of the first 13 bases,
 * then steps up to KT bases (a non-ACGT base is a wildcard, or stops the
 * start under GS_N_STOP) */
template <int NSTOP>
__device__ __forceinline__ void gs_start_from13(const GsDevIndex &I, const unsigned char *seq,
                                                int anchor, int dir, bool fwd, int KT, uint32_t pat,
                                                uint32_t &l, uint32_t &u, int &pos, bool &alive,
                                                unsigned long long &w_blk)
{
    uint2 iv = gs_ld_entry(&I.kmer[pat & ((1u << (2 * GS_K0)) - 1u)]);
    l = iv.x;
    u = iv.y;
    alive = l <= u;
    pos = anchor + dir * (GS_K0 - 1);
    for (int j = GS_K0; j < KT && alive; j++) {
        int np = pos + dir;
        unsigned char ch = seq[np];
        uint32_t c = fwd ? gs_fwd_code(ch) : gs_comp_code(ch);
        if (c > 3u) {
            if (NSTOP) alive = false;
            else pos = np;
        } else {
            uint32_t nl = l, nu = u;
            w_blk += (unsigned long long)gs_step(I, nl, nu, c);
            if (nl > nu) {
                alive = false;
            } else {
                l = nl;
                u = nu;
                pos = np;
            }
        }
    }
}

/* Start of a candidate: the interval of its first KT bases (forward: the
 * bases anchor, anchor-1, ...; reverse: the complement codes anchor,
 * anchor+1, ...; the first base at bits 0-1).  Returns false when one of the
 * first 13 bases is not ACGT (no search, seed_gen.cu:2132-2143).  A non-ACGT
 * base at positions 13..KT-1 takes the 13-mer start and steps over it like
 * the main loop does.  pos = far end reached; alive = interval non-empty;
 * contained (FORCED only) = the start string is always followed by the
 * neighbour's next base (the candidate needs no walk and produces no record);
 * fcode = the start table's forced-extension code (0-3, or 4: none/unknown). */
template <int NSTOP, bool FORCED>
__device__ __forceinline__ bool gs_start(const GsDevIndex &I, const unsigned char *seq, int anchor,
                                         int dir, bool fwd, int KT, int iL, uint32_t &l,
                                         uint32_t &u, int &pos, bool &alive, bool &contained,
                                         uint32_t &fcode, unsigned long long &w_kmer,
                                         unsigned long long &w_blk)
{
    uint32_t pat = 0;
    int first_bad = KT;
#pragma unroll
    for (int j = 0; j < 16; j++) {
        if (j < KT) {
            unsigned char ch = seq[anchor + dir * j];
            uint32_t c = fwd ? gs_fwd_code(ch) : gs_comp_code(ch);
            if (c > 3u && first_bad == KT) first_bad = j;
            pat |= (c & 3u) << (j << 1);
        }
    }
    l = 1;
    u = 0;
    alive = false;
    contained = false;
    fcode = 4;
    pos = anchor + dir * (GS_K0 - 1);
    if (first_bad < GS_K0) return false;
    w_kmer++;
    if (first_bad == KT) {
        if (KT == GS_K0) {
            uint2 iv = gs_ld_entry(&I.kmer[pat]);
            l = iv.x;
            u = iv.y;
            pos = anchor + dir * (KT - 1);
            alive = l <= u;
            return true;
        }
        uint2 iv = gs_ld_entry(reinterpret_cast<const uint2 *>(&I.kmerx[pat]));
        if (iv.y != GS_ENTRY_WIDE) {
            const uint32_t code = gs_entry_forced(iv.y), size = gs_entry_size(iv.y);
            fcode = code;
            l = iv.x;
            u = size ? iv.x + size - 1u : iv.x - 1u;
            pos = anchor + dir * (KT - 1);
            alive = size != 0;
            /* neighbour toward the longer match: e+1 (forward), s-1 (reverse) */
            int nb = anchor - dir;
            if (FORCED && alive && code < 4u && nb >= 0 && nb < iL) {
                unsigned char ch = seq[nb];
                uint32_t c = fwd ? gs_fwd_code(ch) : gs_comp_code(ch);
                contained = (c == code);
            }
            return true;
        }
        /* interval too wide to pack: the 13-mer start below */
    }
    gs_start_from13<NSTOP>(I, seq, anchor, dir, fwd, KT, pat, l, u, pos, alive, w_blk);
    return true;
}

/* start-table length used for minimum seed length k */
__host__ __device__ __forceinline__ int gs_start_len(const GsDevIndex &I, int k)
{
    return (I.kx > GS_K0 && k > I.kx) ? I.kx : GS_K0;
}

/* one candidate's start as gs_start reports it */
struct GsStart {
    uint32_t l, u, fcode;
    int pos;
    bool ok, alive;
};

/* gs_start of one candidate: the rare starts of a paired window (a
 * non-ACGT base in it, or an interval too wide to pack) */
template <int NSTOP>
__device__ __forceinline__ GsStart gs_start_apart(const GsDevIndex &I, const unsigned char *seq,
                                               int anchor, bool fwd, int KT, int iL)
{
    GsStart S;
    bool contained;
    unsigned long long w_kmer = 0, w_blk = 0;
    S.ok = gs_start<NSTOP, false>(I, seq, anchor, fwd ? -1 : 1, fwd, KT, iL, S.l, S.u, S.pos,
                                  S.alive, contained, S.fcode, w_kmer, w_blk);
    return S;
}

/* The bases around a lane's read window, from one 64-byte stretch of the
 * read that the warp loads a word a lane: lane i gets the 2-bit codes of
 * bases b0 + i .. b0 + i + 28 (the first at bits 0-1 of lo, the 17th at bits
 * 0-1 of hi) and bit j of `odd` set when base b0 + i + j lies outside the
 * read or is no plain base.  Plain letters are those whose complement code
 * is 3 - code; the nibble tables give some other letters code 0 on both
 * strands, which the callers look up one by one.  A word is loaded only if
 * it holds a byte of the read. */
__device__ __forceinline__ void gs_warp_bases(const unsigned char *seq, int iL, int b0, int lane,
                                              uint32_t &lo, uint32_t &hi, uint32_t &odd)
{
    const uintptr_t a0 = (uintptr_t)seq + (uintptr_t)(intptr_t)b0;
    const int d = (int)(a0 & 3u);
    const int p0 = b0 - d + 4 * lane;   /* read position of this lane's word */
    uint32_t t = 0x000f0000u;
    if (lane < 16 && p0 + 3 >= 0 && p0 < iL) {
        const uint32_t b = __ldg((const uint32_t *)(a0 - (uintptr_t)d) + lane);
        const uint32_t idx = b & 0x07070707u;
        const uint32_t sel = (idx & 7u) | ((idx >> 4) & 0x70u) | ((idx >> 8) & 0x700u) |
                             ((idx >> 12) & 0x7000u);
        /* letter & 7: A 0, C 1, G 2, T 3, others 4 */
        const uint32_t c = __byte_perm(0x01040004u, 0x02040403u, sel);
        uint32_t v = c & 0x03030303u;
        v = (v | (v >> 6)) & 0x000f000fu;
        uint32_t iv = (c >> 2) & 0x01010101u;
        iv = (iv | (iv >> 7)) & 0x00030003u;
        iv = (iv | (iv >> 14)) & 0xfu;
        if (p0 < 0) iv |= (1u << -p0) - 1u;
        if (p0 + 4 > iL) iv |= 0xfu << (iL - p0);
        t = ((v | (v >> 12)) & 0xffu) | ((iv & 0xfu) << 16);
    }
    /* words j..j+3 at lane j: 16 codes and 16 flags */
    uint32_t n = __shfl_down_sync(0xffffffffu, t, 1);
    t = (t & 0xffu) | ((n & 0xffu) << 8) | (t & 0xf0000u) | ((n & 0xf0000u) << 4);
    n = __shfl_down_sync(0xffffffffu, t, 2);
    const uint32_t c16 = (t & 0xffffu) | (n << 16);
    uint32_t v = (t >> 16) | ((n >> 16) << 8);
    v |= __shfl_down_sync(0xffffffffu, v, 4) << 16;
    const int q = (lane + d) >> 2, sh = (lane + d) & 3;
    const uint32_t x0 = __shfl_sync(0xffffffffu, c16, q);
    const uint32_t x1 = __shfl_sync(0xffffffffu, c16, q + 4);
    lo = __funnelshift_r(x0, x1, 2 * sh);
    hi = x1 >> (2 * sh);
    odd = __shfl_sync(0xffffffffu, v, q) >> sh;
}

/* What a start's entry says about the candidate's next bases, for the
 * candidate itself and, by a shuffle, for the one it may contain. */
#define GS_START_ALIVE 1u
#define GS_START_ONE 2u     /* its string extended by the next base is one row */
#define GS_START_TWO 4u     /* extended by the next two it occurs ... */
#define GS_START_KNOWN 8u   /* ... or, with this and not _TWO, does not */
#define GS_CODE_UNKNOWN 5u  /* forced code of a start that no packed entry gave */
#define GS_START_DEAD 16u   /* it ends before length k: no record */
#define GS_START_ROWS 32u   /* its few rows' contexts settle J: */
#define GS_START_IN 64u     /*   contained in its neighbour */
#define GS_START_J 128u     /*   walks with its neighbour's interval */

/* walk: the next six bases of the walk, the nearest at bits 10-11, nv of them
 * plain; cn: the neighbour's base (4 or more: none); more: bases that the
 * start lacks to length k, at least 1.
 *
 * With the rows' contexts the walk is played out: each row stays for as many
 * bases as match, and is one of J's rows if the neighbour's base follows.
 * a, b: how far J's rows and the others get, of the `cap` bases known.  The
 * candidate is contained where the last of the others has gone and a J row
 * is left (a > b); it has no use for J where that cannot be (a < b, or both
 * end at the same base); otherwise both last as far as is known. */
__device__ __forceinline__ uint32_t gs_start_flags(uint32_t y, uint32_t walk, int nv, uint32_t cn,
                                                   int more)
{
    const uint32_t n = gs_entry_rows(y);
    uint32_t f = GS_START_ALIVE;
    if (n) {
        const int cap = min(nv, n < 3u ? 6 : 3);
        int a = -1, b = -1;
#pragma unroll
        for (uint32_t i = 0; i < GS_ROWS_MOST; i++) {
            if (i < n) {
                uint32_t left, right;
                gs_entry_row(y, n, i, left, right);
                const int m = min(__clz((left ^ walk) << 20) >> 1, cap);
                if (right == cn) a = max(a, m);
                else b = max(b, m);
            }
        }
        const int m = max(a, b);
        f |= GS_START_ROWS;
        if (m < cap && m < more) f |= GS_START_DEAD;
        if (cap >= 2) f |= GS_START_KNOWN;
        if (m >= 2) f |= GS_START_TWO;
        if (a > b) f |= GS_START_IN;
        else if (a == b && a == cap) f |= GS_START_J;
        return f;
    }
    if (!(y & GS_ENTRY_EXT)) return f;
    if (!((y >> 4) & 255u)) return 0u;
    if (nv >= 1) {
        const uint32_t c = (walk >> 10) & 3u, d = (walk >> 8) & 3u;
        const uint32_t two = y >> (16u + 4u * c);
        const bool one = (y >> (12u + c)) & 1u;
        if (one) f |= GS_START_ONE;
        if (!one && !(two & 15u)) f |= GS_START_DEAD;
        if (nv >= 2) {
            f |= GS_START_KNOWN;
            if ((two >> d) & 1u) f |= GS_START_TWO;
            else if (more >= 2) f |= GS_START_DEAD;
        }
    }
    return f;
}

/* ------------------------------------------------------------------ */
/* per-batch preparation: candidate slots and work items per read */

__device__ __forceinline__ void gs_put_totals(const GsBatch &B, int at, const GsPart &t)
{
    if (threadIdx.x) return;
    B.totals[at] = t.a;
    B.totals[at + 1] = t.b;
    if (B.h_totals) {
        B.h_totals[at] = t.a;
        B.h_totals[at + 1] = t.b;
    }
}

/* the pass's counters and record mask, where the host left that to the
 * first kernel */
__device__ __forceinline__ void gs_clear(const GsBatch &B)
{
    if (!B.clear) return;
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 8) B.queue[t] = 0u;
    for (uint64_t i = t; i < B.clear_words; i += (uint64_t)gridDim.x * blockDim.x) B.recmask[i] = 0u;
}

__global__ void __launch_bounds__(GS_SCAN_THREADS) gs_prepare_sum(GsBatch B, int paired_kt)
{
    gs_after_previous();
    gs_clear(B);
    uint32_t first, last;
    gs_part_reads(B.n_reads, GS_SCAN_THREADS, blockIdx.x, gridDim.x, first, last);
    unsigned long long a = 0, b = 0;
    for (uint32_t r = first + threadIdx.x; r < last; r += GS_SCAN_THREADS) {
        uint32_t slots, items;
        gs_read_counts(B.lengths[r], B.k, paired_kt, slots, items);
        a += slots;
        b += items;
    }
    GsPart sum, total;
    gs_block_scan(a, b, sum);
    if (gs_parts_publish(B.parts, 0, sum, total)) gs_put_totals(B, 0, total);
}

/* Offsets of the reads' slots and work items, and the read of each work
 * item, so that the start pass need not search item_off for it (a thread per
 * read, or the warp for a read of many items). */
__global__ void __launch_bounds__(GS_SCAN_THREADS) gs_prepare_scan(GsBatch B, int paired_kt)
{
    gs_after_previous();
    const int lane = threadIdx.x & 31;
    if (gridDim.x == 1) gs_clear(B);
    uint32_t first, last;
    gs_part_reads(B.n_reads, GS_SCAN_THREADS, blockIdx.x, gridDim.x, first, last);
    GsPart run = {0ull, 0ull};
    if (gridDim.x > 1) run = B.parts.part[blockIdx.x];
    for (uint32_t r0 = first; r0 < last; r0 += GS_SCAN_THREADS) {
        const uint32_t r = r0 + threadIdx.x;
        uint32_t slots = 0, items = 0;
        if (r < last) gs_read_counts(B.lengths[r], B.k, paired_kt, slots, items);
        GsPart t;
        const GsPart x = gs_block_scan(slots, items, t);
        const uint32_t a = (uint32_t)(run.b + x.b), e = a + items;
        if (r < last) {
            B.slot_off[r] = run.a + x.a;
            B.item_off[r] = a;
        }
        if (B.item_read) {
            const bool big = items > 16u;
            if (!big)
                for (uint32_t i = a; i < e; i++)
                    if (i < B.item_read_cap) B.item_read[i] = r;
            uint32_t m = __ballot_sync(0xffffffffu, big);
            while (m) {
                const int src = __ffs(m) - 1;
                m &= m - 1u;
                const uint32_t a1 = __shfl_sync(0xffffffffu, a, src), e1 = __shfl_sync(0xffffffffu, e, src);
                for (uint32_t i = a1 + (uint32_t)lane; i < e1; i += 32)
                    if (i < B.item_read_cap) B.item_read[i] = r - (uint32_t)lane + (uint32_t)src;
            }
        }
        run.a += t.a;
        run.b += t.b;
    }
    if (last == B.n_reads && (first < last || blockIdx.x == 0)) {
        /* the block that holds the last read */
        if (threadIdx.x == 0) {
            B.slot_off[B.n_reads] = run.a;
            B.item_off[B.n_reads] = (uint32_t)run.b;
        }
        if (gridDim.x == 1) gs_put_totals(B, 0, run);
    }
}

int gs_launch_prepare(const GsDevIndex &I, GsBatch &b, int kernel, cudaStream_t st)
{
    const int kt = gs_paired_len(I, kernel, b.k);
    b.paired = kt != 0;
    const uint32_t parts = gs_parts_of(b.n_reads, GS_SCAN_THREADS);
    if (b.clear && !gs_clear_in_kernel(b.n_reads, GS_SCAN_THREADS, b.clear_words)) {
        GS_CUDA(cudaMemsetAsync(b.recmask, 0, b.clear_words * sizeof(uint32_t), st));
        b.clear_words = 0;
    }
    if (parts > 1) {
        gs_prepare_sum<<<parts, GS_SCAN_THREADS, 0, st>>>(b, kt);
        GS_CUDA(cudaGetLastError());
    }
    if (parts > 1) {
        GS_CUDA(gs_launch_after(gs_prepare_scan, parts, GS_SCAN_THREADS, st, b, kt));
    } else {
        /* the pass's first kernel: after all that the stream holds */
        gs_prepare_scan<<<parts, GS_SCAN_THREADS, 0, st>>>(b, kt);
        GS_CUDA(cudaGetLastError());
    }
    return GS_OK;
}

/* ------------------------------------------------------------------ */
/* lockstep search */

/* one extension step of a candidate; false when it cannot extend further
 * (read end, empty interval, or a non-ACGT base under GS_N_STOP) */
template <int NSTOP, int COUNT>
__device__ __forceinline__ bool gs_advance(const GsDevIndex &I, const unsigned char *seq, int iL,
                                           bool fwd, int dir, uint32_t &l, uint32_t &u, int &pos,
                                           unsigned long long &w_blk)
{
    int np = pos + dir;
    if (np < 0 || np >= iL) return false;
    uint32_t c = fwd ? gs_fwd_code(seq[np]) : gs_comp_code(seq[np]);
    if (c > 3u) {
        if (NSTOP) return false;
        pos = np;   /* wildcard: interval unchanged */
        return true;
    }
    uint32_t nl = l, nu = u;
    int blocks = gs_step(I, nl, nu, c);
    if (COUNT) w_blk += (unsigned long long)blocks;
    if (nl > nu) return false;
    l = nl;
    u = nu;
    pos = np;
    return true;
}

/* record of a finished candidate (seed_gen.cu:2259-2264, :2398-2404) */
__device__ __forceinline__ void gs_write_record(const GsBatch &B, uint32_t r, uint32_t n, bool fwd,
                                                int anchor, int pos, uint32_t l, uint32_t u,
                                                bool ok, bool killed)
{
    const int k = B.k;
    GsRec rec;
    rec.x = 0; rec.y = 0; rec.l = l; rec.u = u;
    if (!killed) {
        if (fwd) {
            /* length e - beg with beg = pos-1; a 13-mer that is absent still
             * counts 13 (the k == 13 case of :2259) */
            if (ok && anchor - pos + 1 >= k) {
                rec.x = pos;
                rec.y = anchor + 1;
            }
        } else if (ok && l <= u && pos + 1 - anchor >= k) {
            rec.x = (int32_t)((uint32_t)anchor | 0x80000000u);
            rec.y = (int32_t)((uint32_t)(pos + 1) | 0x80000000u);
        }
    }
    if (rec.y == 0) return;   /* no record: the slot stays unflagged and unwritten */
    uint64_t slot = B.slot_off[r] + (fwd ? (uint64_t)(anchor - (k - 1)) : (uint64_t)n + (uint64_t)anchor);
    if (slot < B.slot_cap) {
        B.slots[slot] = rec;
        atomicOr(B.recmask + (slot >> 5), 1u << (slot & 31u));
    } else {
        atomicOr(B.queue + 1, GS_FLAG_OVERFLOW);
    }
}

template <int NSTOP, int COUNT>
__device__ __forceinline__ void gs_lockstep_item(const GsDevIndex &I, const GsBatch &B, uint32_t r,
                                             uint32_t local, int lane, unsigned long long &wk,
                                             unsigned long long &wb)
{
    const uint32_t L = B.lengths[r];
    const int k = B.k;
    const uint32_t n = L - (uint32_t)k + 1u;
    const uint32_t nch = (n + GS_CHUNK - 1) / GS_CHUNK;
    const bool fwd = local < nch;
    const uint32_t chunk = fwd ? local : local - nch;
    const uint32_t ci = chunk * GS_CHUNK + (uint32_t)lane;
    const bool in_range = ci < n;
    /* lane 31 only starts the next item's first candidate (which that item
     * owns: ceil(n / GS_CHUNK) items cover every candidate) */
    const bool owned = in_range && lane < GS_CHUNK;
    const unsigned char *seq = (const unsigned char *)B.seqs + B.offsets[r];
    const int iL = (int)L;

    /* anchor: e = k-1+ci (fwd), s = n-1-ci (rev); the containing neighbour
     * of every lane is lane+1 */
    int anchor = fwd ? (k - 1 + (int)ci) : ((int)n - 1 - (int)ci);
    const int dir = fwd ? -1 : 1;
    uint32_t l = 1, u = 0;
    int pos = anchor;
    bool alive = false, ok = false;
    bool killed = false;
    /* The start table's forced extensions are not used here.  A lockstep warp
     * lasts as long as its longest owned walk; a forced lane dies at step 1
     * by the neighbour rule anyway, and its step-1 size is what lane-1 is
     * compared with at step 1 (and lane 31, which nothing kills, is lane 30's
     * partner for the whole walk).  Stopping forced lanes at their start
     * saved 4% of the DRAM reads but, after keeping exactly those two
     * roles, still cost 2.5% of the time (config 3, 10M reads). */
    if (in_range) {
        bool contained = false;
        uint32_t fcode = 4;
        ok = gs_start<NSTOP, false>(I, seq, anchor, dir, fwd, gs_start_len(I, k), iL, l, u, pos,
                                    alive, contained, fcode, wk, wb);
    }

    uint32_t hist[GS_HIST];
#pragma unroll
    for (int m = 0; m < GS_HIST; m++) hist[m] = 0;
    uint32_t cur = alive ? u - l + 1u : 0u;
    int t = 0;
    const uint32_t owned_mask = __ballot_sync(0xffffffffu, owned);

    bool pushed = false;
    while (__ballot_sync(0xffffffffu, alive) & owned_mask) {
        if (alive) alive = gs_advance<NSTOP, COUNT>(I, seq, iL, fwd, dir, l, u, pos, wb);
        t++;
        uint32_t pub = alive ? u - l + 1u : 0u;
        /* containment: own size d steps ago vs the nearest extending lane
         * d to the right, which now stands at the same far end */
        uint32_t right = __ballot_sync(0xffffffffu, pub != 0u) & ~((2u << lane) - 1u);
        int j = right ? __ffs(right) - 1 : lane;
        uint32_t v = __shfl_sync(0xffffffffu, pub, j);
        int d = j - lane;
        if (alive && right && d <= GS_HIST && d <= t) {
            /* cur = own size one step ago, hist[m] = m+2 steps ago */
            uint32_t h = cur;
#pragma unroll
            for (int m = 0; m < GS_HIST - 1; m++) h = (d == m + 2) ? hist[m] : h;
            if (h == v) {
                alive = false;
                killed = true;
            }
        }
#pragma unroll
        for (int m = GS_HIST - 1; m > 0; m--) hist[m] = hist[m - 1];
        hist[0] = cur;
        cur = pub;
        /* few candidates left: hand them to the tail pass, which walks them
         * without lockstep, and free the warp */
        if (B.cont && t >= B.handoff_steps) {
            uint32_t left = __ballot_sync(0xffffffffu, alive) & owned_mask;
            if (__popc(left) <= B.handoff_lanes) {
                bool push = alive && owned;
                uint32_t base = 0;
                if (lane == 0 && left) base = atomicAdd(B.queue + 2, (uint32_t)__popc(left));
                base = __shfl_sync(0xffffffffu, base, 0);
                if (push && base + __popc(left & ((1u << lane) - 1u)) >= B.cont_cap) {
                    atomicOr(B.queue + 1, GS_FLAG_OVERFLOW);
                    push = false;
                }
                if (push) {
                    GsCont cst;
                    cst.r = r;
                    cst.anchor = anchor;
                    cst.pos = pos;
                    cst.l = l;
                    cst.u = u;
                    cst.fwd = fwd ? 1u : 0u;
                    B.cont[base + __popc(left & ((1u << lane) - 1u))] = cst;
                    pushed = true;
                }
                break;
            }
        }
    }

    if (owned && !pushed) gs_write_record(B, r, n, fwd, anchor, pos, l, u, ok, killed);
}

/* executed-work counters (count_work with the batched kernel): a warp sum,
 * one atomic per warp */
__device__ __forceinline__ void gs_add_work(const GsBatch &B, unsigned long long wk,
                                            unsigned long long wb)
{
    for (int o = 16; o > 0; o >>= 1) {
        wk += __shfl_xor_sync(0xffffffffu, wk, o);
        wb += __shfl_xor_sync(0xffffffffu, wb, o);
    }
    if ((threadIdx.x & 31) == 0 && B.work) {
        atomicAdd(&B.work[0], wk);
        atomicAdd(&B.work[1], wb);
    }
}

/* Tail pass: the candidates handed over by gs_search_lockstep, one per lane;
 * a lane takes the next one as soon as its own is finished. */
template <int NSTOP, int COUNT>
__global__ void __launch_bounds__(256) gs_search_tail(GsDevIndex I, GsBatch B)
{
    const int lane = threadIdx.x & 31;
    unsigned long long wb = 0;
    uint32_t n_cont = *(volatile uint32_t *)(B.queue + 2);
    if (n_cont > B.cont_cap) n_cont = (uint32_t)B.cont_cap;
    bool have = false, exhausted = false;
    uint32_t r = 0, l = 0, u = 0, n = 0;
    int anchor = 0, pos = 0, iL = 0, dir = 0;
    bool fwd = false;
    const unsigned char *seq = NULL;
    for (;;) {
        uint32_t need = __ballot_sync(0xffffffffu, !have && !exhausted);
        if (need) {
            int leader = __ffs(need) - 1;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(B.queue + 3, (uint32_t)__popc(need));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (!have && !exhausted) {
                uint32_t idx = base + __popc(need & ((1u << lane) - 1u));
                if (idx < n_cont) {
                    GsCont c = B.cont[idx];
                    r = c.r;
                    anchor = c.anchor;
                    pos = c.pos;
                    l = c.l;
                    u = c.u;
                    fwd = c.fwd != 0;
                    dir = fwd ? -1 : 1;
                    uint32_t L = B.lengths[r];
                    iL = (int)L;
                    n = L - (uint32_t)B.k + 1u;
                    seq = (const unsigned char *)B.seqs + B.offsets[r];
                    have = true;
                } else {
                    exhausted = true;
                }
            }
        }
        if (!__ballot_sync(0xffffffffu, have)) break;
        if (have && !gs_advance<NSTOP, COUNT>(I, seq, iL, fwd, dir, l, u, pos, wb)) {
            gs_write_record(B, r, n, fwd, anchor, pos, l, u, true, false);
            have = false;
        }
    }
    if (COUNT) gs_add_work(B, 0, wb);
}

template <int NSTOP, int COUNT>
__global__ void __launch_bounds__(256, 5) gs_search_lockstep(GsDevIndex I, GsBatch B, int queue_chunk)
{
    const int lane = threadIdx.x & 31;
    unsigned long long wk = 0, wb = 0;
    const uint32_t n_items = B.item_off[B.n_reads];
    if (n_items > B.item_cap) {
        /* the hand-over buffer was sized for fewer items (a captured pass
         * replayed on larger input): report, do nothing */
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(B.queue + 1, GS_FLAG_OVERFLOW);
        return;
    }
    for (;;) {
        uint32_t first = 0;
        if (lane == 0) first = atomicAdd(B.queue, (uint32_t)queue_chunk);
        first = __shfl_sync(0xffffffffu, first, 0);
        if (first >= n_items) break;
        uint32_t last = min(first + (uint32_t)queue_chunk, n_items);
        /* read of the first item: largest r with item_off[r] <= first */
        uint32_t lo = 0, hi = B.n_reads;
        while (lo + 1 < hi) {
            uint32_t mid = (lo + hi) >> 1;
            if (B.item_off[mid] <= first) lo = mid; else hi = mid;
        }
        uint32_t r = lo;
        for (uint32_t it = first; it < last; it++) {
            while (B.item_off[r + 1] <= it) r++;
            gs_lockstep_item<NSTOP, COUNT>(I, B, r, it - B.item_off[r], lane, wk, wb);
        }
    }
    if (COUNT) gs_add_work(B, wk, wb);
}

/* ------------------------------------------------------------------ */
/* batched search
 *
 * Candidate e is contained in e+1 at far end p exactly when
 * count(R[p..e]) == count(R[p..e+1]) (sizes only fall along the chain
 * e, e+1, ..., so this is the nearest-extending-candidate rule of the file
 * comment).  R[p..e+1]'s interval J is nested in R[p..e]'s interval I, so a
 * candidate can carry J itself and stop at the canonical step without
 * seeing its neighbour: no lockstep, no helper lane walking, no history.
 * J's bounds share occurrence blocks with I's whenever I is narrow.
 *
 *   gs_search_start: a warp per work item, one round of start-table
 *     lookups.  With the longer start table (k > kx) an item is 30 read
 *     windows (+ a helper window on each side) and one paired entry starts
 *     a window's forward and reverse candidate (gs_start_pair_item); else
 *     31 candidates of one strand + the next item's first, started for its
 *     interval only (gs_start_item).  The forced-extension code settles J
 *     where it can (forced to the neighbour's base: contained, stop; forced
 *     elsewhere: no J); otherwise the walker carries its neighbour's start
 *     interval and its first step in the walk pass extends that to I's far
 *     end.  Survivors go to the walker buffer in per-warp reserved chunks
 *     (unused entries marked r = ~0); a walker that finds the buffer full is
 *     left in its record slot for gs_search_leftover.
 *   gs_search_walk: one walker per lane, each lane refilled as soon as its
 *     walker ends, from a per-warp window of the buffer; walkers that reach
 *     one row without J go to gs_search_text. */

#define GS_WALKER_CHUNK 512u      /* most buffer entries a warp reserves at a time */
#define GS_WALK_WINDOW 512u       /* ... and a walk-pass warp takes */

/* Buffer entries a start-pass warp reserves at a time, a multiple of 16: a
 * 32nd of its share of the capacity, 32 to 512.  The capacity is all
 * candidates, of which a tenth or so become walkers, so what stays unused of
 * the last reservations counts against them (each warp a 16th: 2.9 M entries
 * for 1.6 M walkers); less than an item's walkers is a reservation an item
 * (16 entries at 60,007 short reads: start pass 85 -> 104 us). */
static uint32_t gs_walker_chunk(uint64_t cap, uint32_t warps)
{
    const uint64_t v = cap / ((uint64_t)warps * 32u) & ~15ull;
    return v < 32u ? 32u : v > GS_WALKER_CHUNK ? GS_WALKER_CHUNK : (uint32_t)v;
}

/* Buffer entries a walk-pass warp takes at a time: an eighth of its share of
 * the entries in use, 32 to 512, so that the walks spread over every warp
 * (sized by the buffer's capacity, 100,000 reads of 150 were 3,100 windows
 * of 512 for 4,900 warps: walk pass 538 -> 456 us on 100 Mbp; 150,001
 * reads, 740 -> 622). */
__device__ __forceinline__ uint32_t gs_walk_window(uint32_t n_w, uint32_t warps)
{
    return min(max((n_w / (warps * 8u)) & ~31u, 32u), GS_WALK_WINDOW);
}
/* entries of a list that a walk-pass warp reserves at a time: an eighth of
 * its share of the capacity, 1 to 32 */
static uint32_t gs_list_chunk(uint64_t cap, uint32_t warps)
{
    const uint64_t v = cap / ((uint64_t)warps * 8u);
    return v < 1u ? 1u : v > 32u ? 32u : (uint32_t)v;
}

/* Text mode.  A walker whose interval is one row [l,l] and whose J is
 * empty can no longer be contained: its walk only extends one occurrence,
 * at text position q = SA[l], while the read goes on matching T[q-1],
 * T[q-2], ...  It ends where the read and the text differ, the read or the
 * text ends, or (GS_N_STOP) a non-ACGT base comes; its record is the row of
 * the suffix at that position.  Text mode finds that position by comparing
 * 16 bases a round and takes its row from the inverse-SA sample at or above
 * it, with at most GS_ISA_STEP-1 LF steps over the text bases in between.
 * Under GS_N_WILDCARD a non-ACGT base hands the walker back to the
 * interval walk, which skips the base.  The walker's J words hold the
 * state: jl = GS_TEXT_MARK | phase << 26 | flags, ju = a text position. */
#define GS_TM_MOVED (1u << 25)   /* the compare advanced past the entry position */
#define GS_TM_CONT (1u << 24)    /* a wildcard base follows: back to the interval walk */

/* The 2-bit codes (forward or complement table) and the non-ACGT flags of 4
 * ASCII bytes: a byte-permute lookup of the nibble table, indexed by ch & 7 */
__device__ __forceinline__ void gs_codes4(uint32_t b, bool fwd, uint32_t &packed, uint32_t &inv)
{
    const uint32_t idx = b & 0x07070707u;
    const uint32_t sel = (idx & 7u) | ((idx >> 4) & 0x70u) | ((idx >> 8) & 0x700u) |
                         ((idx >> 12) & 0x7000u);
    /* bytes 0..7 = code of ch & 7: forward A0 C1 G2 T3 N4 others 0/5, complement */
    const uint32_t c = fwd ? __byte_perm(0x01000005u, 0x02040003u, sel)
                           : __byte_perm(0x02000305u, 0x01040000u, sel);
    uint32_t v = c & 0x03030303u;
    v = (v | (v >> 6)) & 0x000f000fu;
    packed = (v | (v >> 12)) & 0xffu;
    uint32_t iv = (c >> 2) & 0x01010101u;   /* codes 4 and 5 */
    iv = (iv | (iv >> 7)) & 0x00030003u;
    inv = (iv | (iv >> 14)) & 0xfu;
}

/* The read's next `avail` (1..16) bases in walk order from pos: the first at
 * bits 30-31 of *wr (2-bit codes), and *inv with bit 31 - i set when the
 * i-th is not ACGT.  Loads the aligned words that hold the bytes, each of
 * which holds at least one byte of the read. */
__device__ __forceinline__ void gs_read_window(const unsigned char *seq, int pos, bool fwd,
                                               int avail, uint32_t &wr, uint32_t &inv32)
{
    const unsigned char *lo = seq + (fwd ? pos - avail : pos + 1);
    const uintptr_t a = (uintptr_t)lo;
    const uint32_t *wp = (const uint32_t *)(a & ~(uintptr_t)3);
    const uint32_t off = (uint32_t)(a & 3u);
    const uint32_t nw = (off + (uint32_t)avail + 3u) >> 2;   /* 1..5 */
    uint32_t w[5];
#pragma unroll
    for (int k = 0; k < 5; k++) w[k] = (uint32_t)k < nw ? __ldg(wp + k) : 0u;
    uint32_t wr16 = 0, inv16 = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        uint32_t p, iv;
        gs_codes4(__funnelshift_r(w[k], w[k + 1], off * 8u), fwd, p, iv);
        wr16 |= p << (8 * k);
        inv16 |= iv << (4 * k);
    }
    if (fwd) {
        /* memory order ends with the first base of the walk (pos-1) */
        wr = wr16 << (2 * (16 - avail));
        inv32 = inv16 << (32 - avail);
    } else {
        /* memory order starts with it (pos+1): reverse the 2-bit groups */
        uint32_t x = __brev(wr16);
        wr = ((x >> 1) & 0x55555555u) | ((x & 0x55555555u) << 1);
        inv32 = __brev(inv16) & (0xffffffffu << (32 - avail));
    }
}

template <int COUNT>
__device__ __forceinline__ bool gs_text_round(const GsDevIndex &I, const unsigned char *seq, int iL,
                                              bool fwd, int dir, uint32_t &l, uint32_t &u,
                                              uint32_t &jl, uint32_t &ju, int &pos, int nstop,
                                              unsigned long long &wb)
{
    const uint32_t ph = (jl >> 26) & 3u;
    (void)wb;
    if (ph == 0) {
        ju = gs_ld64(&I.saf[l]);
        jl = GS_TEXT_MARK | (1u << 26);
        return true;
    }
    bool cont;
    if (ph == 1) {
        const uint32_t q = ju;
        const int rem = fwd ? pos : iL - 1 - pos;
        int avail = rem < 16 ? rem : 16;
        if ((uint32_t)avail > q) avail = (int)q;
        int m = 0, bad = avail;
        if (avail > 0) {
            /* T[q-16..q-1], T[q-1] at bits 30-31 */
            uint32_t wt;
            if (q >= 16) {
                const uint32_t b = q - 16u;
                wt = __funnelshift_r(gs_ld64(&I.text[b >> 4]), gs_ld64(&I.text[(b >> 4) + 1]),
                                     (b & 15u) << 1);
            } else {
                wt = __ldg(&I.text[0]) << ((16u - q) << 1);
            }
            /* the read's next bases in walk order, the first at bits 30-31 */
            uint32_t wr, inv32;
            gs_read_window(seq, pos, fwd, avail, wr, inv32);
            if (inv32) bad = __clz(inv32);
            m = (int)(__clz(wr ^ wt) >> 1);
            if (m > bad) m = bad;
            pos += dir * m;
            ju = q - (uint32_t)m;
            if (m) jl |= GS_TM_MOVED;
            if (m == avail && avail < rem && ju > 0u) return true;
        }
        cont = !nstop && m == bad && bad < avail;
        if (!(jl & GS_TM_MOVED)) {
            /* still at the entry row */
            if (!cont) return false;
            jl = 1u;
            ju = 0u;
            return true;
        }
        jl = GS_TEXT_MARK | (2u << 26) | (cont ? GS_TM_CONT : 0u);
        return true;
    }
    cont = (jl & GS_TM_CONT) != 0;
    {
        /* the row of position qs from the sample at qp >= qs (position
         * seq_len is row 0), and T[qs..qs+3] for the LF steps down to qs */
        const uint32_t qs = ju;
        uint32_t qp = (qs + GS_ISA_STEP - 1u) & ~(GS_ISA_STEP - 1u);
        uint32_t row = 0;
        if (qp > I.seq_len) qp = I.seq_len;
        else row = gs_ld64(&I.isa[qp / GS_ISA_STEP]);
        const uint32_t w = __funnelshift_r(gs_ld64(&I.text[qs >> 4]), gs_ld64(&I.text[(qs >> 4) + 1]),
                                           (qs & 15u) << 1);
        l = u = row;
        const uint32_t d = qp - qs;
        jl = GS_TEXT_MARK | (3u << 26) | (jl & GS_TM_CONT) | (d << 16) | (w & 0xffu);
        if (d) return true;
    }
    /* phase 3, the LF steps, is the interval walk's own step (gs_walk_step) */
    if (!cont) return false;
    jl = 1u;
    ju = 0u;
    return true;
}

/* One iteration of a walk: normally a step of I and J with the next
 * base; for a walker whose J is still one base short (jpend), the J-only
 * step with the base at pos that brings J to I's far end -- the same call,
 * so the lanes of a warp take one memory round per iteration either way.
 * Returns false when the walk is over (killed: it ended by containment).
 * A step that leaves the walker eligible for text mode sets jl to
 * GS_TEXT_MARK. */
/* walk-pass counters of a count_work pass (gs_ctx_last_walk_counts) */
struct GsWalkCounts {
    unsigned long long steps, jsteps, jblocks, jshrank, jwalkers, lines256, lines384;
};

/* Steps of two bases (the walk pass).  A walk is a chain of dependent steps,
 * each of which waits for slots at random places of the occurrence table.
 * occ2 has a slot for each base and the base after, so one step by a slot of
 * the same form goes two bases.
 *   - At odd read positions only: the neighbour's walk, a base ahead or
 *     behind in the same warp, then comes by the same strings, and so the same
 *     slots, as this one's J.  Without that nearly every slot was a fill
 *     of its own: 2 M reads on 3.1 Gbp 13.9 GB of DRAM reads, 17.4 without.
 *   - J's step to I's far end goes on with I's first step, J by two bases and
 *     I by the second of them, at the parity that makes it the neighbour's own
 *     first step of two (11.7 GB).
 *   - Contained at the first base is contained at the second, unless I ends
 *     between: an empty I is not taken, and the next step is with the first
 *     base alone (or J's alone) and the walk's last.
 * Walk pass before and after: 2 M reads 7.26 -> 5.18 ms, 40,000 long reads
 * 2.77 -> 2.19, 1 M reads on 100 Mbp 2.72 -> 2.32, 300 reads 89 -> 63 us.
 *
 * The walk pass's bases ahead: those of the next step and of the one after
 * (0, no base, past the read), here before they are needed; alone: the two
 * together end the walk. */
struct GsAhead {
    unsigned char first, second;
    bool alone;
};

template <int NSTOP, int COUNT, int TEXT, bool PRE = false>
__device__ __forceinline__ bool gs_walk_step(const GsDevIndex &I, const unsigned char *seq, int iL,
                                             bool fwd, int dir, uint32_t &l, uint32_t &u,
                                             uint32_t &jl, uint32_t &ju, int &pos, bool &jpend,
                                             bool &killed, unsigned long long &wb,
                                             GsWalkCounts *wc = nullptr,
                                             GsAhead *pre = nullptr)
{
    const bool text = TEXT == GS_TEXT_RUN && gs_text_mode(TEXT, jl);
    bool settle = false, two = false, fused = false;
    int np = pos;
    uint32_t c;
    if (text) {
        if (((jl >> 26) & 3u) != 3u)
            return gs_text_round<COUNT>(I, seq, iL, fwd, dir, l, u, jl, ju, pos, NSTOP, wb);
        /* text mode's LF step with base T[qs + d - 1]; J stays empty */
        c = (jl >> ((((jl >> 16) & 15u) - 1u) << 1)) & 3u;
    } else {
        settle = jpend;
        jpend = false;
        np = settle ? pos : pos + dir;
        if (np < 0 || np >= iL) return false;
        const unsigned char ch = PRE ? pre->first : seq[np];
        c = fwd ? gs_fwd_code(ch) : gs_comp_code(ch);
        /* PRE: this step's bases are here already, the next step's come while
         * this one waits for its slots (1 M reads on 100 Mbp 7.27 -> 7.08 ms,
         * 2 M on 3.1 Gbp 15.34 -> 15.28, 300 reads' walk -5 us) */
        if (PRE) {
            const uint32_t d = fwd ? gs_fwd_code(pre->second) : gs_comp_code(pre->second);
            const bool both = I.occ2 && !pre->alone && c <= 3u && d <= 3u;
            two = both && !settle && (np & 1);
            fused = both && settle && (np & 1);
            const bool ahead = two || fused;
            const int n1 = np + dir + dir, n2 = n1 + dir;
            const unsigned char x = n1 >= 0 && n1 < iL ? seq[n1] : 0;
            const unsigned char y = ahead && n2 >= 0 && n2 < iL ? seq[n2] : 0;
            pre->first = ahead ? x : pre->second;
            pre->second = ahead ? y : x;
            if (ahead) {
                np += dir;
                c = c << 2 | d;
            }
        }
    }
    const bool doI = !settle || fused;
    if (!two && !fused && c > 3u) {
        if (!settle) {
            if (NSTOP) return false;
            pos = np;   /* wildcard: both intervals unchanged, so no new equality */
            return true;
        }
        /* settle over a wildcard: J unchanged */
    } else {
        uint32_t nl = l, ne = u + 1u, je = ju + 1u;
        const bool had_j = jl <= ju;
        GsStepTouch touch;
        uint32_t njl = jl;
        const GsStepBy by_i = {two ? I.occ2 : I.occ, two ? 2u : 0u, fused ? c & 3u : c};
        const GsStepBy by_j = {two || fused ? I.occ2 : I.occ, two || fused ? 2u : 0u, c};
        gs_step_pair<COUNT>(by_i, by_j, !settle, nl, ne, njl, je, doI, touch);
        const uint32_t nu = ne - 1u;
        if (COUNT) wb += (unsigned long long)touch.blocks;
        if (COUNT && wc) {
            wc->steps++;
            wc->lines256 += (unsigned long long)touch.lines256;
            wc->lines384 += (unsigned long long)touch.lines384;
            if (had_j) {
                wc->jsteps++;
                wc->jblocks += (unsigned long long)touch.jblocks;
                if (doI && nl <= nu && nu - nl < u - l) wc->jshrank++;
            }
        }
        if (PRE && (two || fused) && nl > nu) {
            /* it ends at one of the two: by the first alone */
            pre->alone = true;
            pre->first = seq[np - dir];
            jpend = fused;
            return true;
        }
        jl = njl;
        ju = je - 1u;
        if (text) {
            l = nl;
            u = nu;
            const uint32_t d = ((jl >> 16) & 15u) - 1u;
            jl = (jl & ~(15u << 16)) | (d << 16);
            if (d) return true;
            if (!(jl & GS_TM_CONT)) return false;
            jl = 1u;
            ju = 0u;
            return true;
        }
        if (doI) {
            if (nl > nu) return false;   /* natural end at pos */
            l = nl;
            u = nu;
            pos = np;
        }
    }
    if (jl <= ju && ju - jl == u - l) {
        killed = true;
        return false;
    }
    if (PRE && pre->alone) return false;   /* the second base ends it */
    /* one row and no J: count the steps taken so (J's words are free);
     * after text_min of them the occurrence is no chance hit, and with 16
     * bases or more left the walker enters text mode */
    if (TEXT != GS_TEXT_NONE && I.text_min && l == u && jl > ju) {
        if (jl < GS_REGIME_MARK) {
            jl = GS_REGIME_MARK;
            ju = 0u;
        } else if ((jl += two ? 2u : 1u) - GS_REGIME_MARK >= (uint32_t)I.text_min &&
                   (fwd ? pos : iL - 1 - pos) >= 16) {
            jl = GS_TEXT_MARK;
        }
    }
    return true;
}

/* A walk that found no room in the walker buffer: its start interval goes
 * to its own record slot under GS_LEFTOVER_MARK (no record has x = y = ~0),
 * and gs_search_leftover walks it after the other passes (its start and J
 * made again from the read). */
#define GS_LEFTOVER_MARK 0xffffffffu

__device__ __forceinline__ void gs_write_leftover(const GsBatch &B, uint32_t r, uint32_t n, bool fwd,
                                                  int anchor, uint32_t l, uint32_t u)
{
    const uint64_t slot = B.slot_off[r] + (fwd ? (uint64_t)(anchor - (B.k - 1))
                                               : (uint64_t)n + (uint64_t)anchor);
    if (slot < B.slot_cap) {
        GsRec rec;
        rec.x = (int32_t)GS_LEFTOVER_MARK;
        rec.y = (int32_t)GS_LEFTOVER_MARK;
        rec.l = l;
        rec.u = u;
        B.slots[slot] = rec;
        atomicOr(B.recmask + (slot >> 5), 1u << (slot & 31u));
        atomicOr(B.queue + 1, GS_FLAG_LEFTOVER);
    } else {
        atomicOr(B.queue + 1, GS_FLAG_OVERFLOW);
    }
}

/* per-warp reservation of walker-buffer entries: [next, end); full once a
 * reservation came back past the capacity (no further atomics, so the
 * 32-bit counter cannot wrap) */
struct GsReserve {
    uint32_t next, end, full;
};

/* Room for an item's cnt walkers beyond the rem entries left: a new
 * reservation of walker_chunk entries, or of all it needs.  Its first entry
 * (walker_cap: none to be had) and size. */
__device__ __forceinline__ uint32_t gs_reserve(const GsBatch &B, GsReserve &res, uint32_t cnt,
                                               uint32_t rem, int lane, uint32_t &take)
{
    uint32_t g = 0;
    take = 0;
    if (rem >= cnt) return g;
    take = max(B.walker_chunk, cnt - rem);
    if (res.full) return (uint32_t)B.walker_cap;
    if (lane == 0) g = atomicAdd(B.queue + 2, take);
    g = __shfl_sync(0xffffffffu, g, 0);
    if ((uint64_t)g + take >= B.walker_cap) res.full = 1u;
    return g;
}

/* ... and the reservation after them */
__device__ __forceinline__ void gs_reserved(const GsBatch &B, GsReserve &res, uint32_t cnt, uint32_t rem,
                                            uint32_t g, uint32_t take)
{
    if (rem >= cnt) {
        res.next += cnt;
        return;
    }
    res.next = (uint32_t)min((uint64_t)g + (cnt - rem), B.walker_cap);
    res.end = (uint32_t)min((uint64_t)g + take, B.walker_cap);
    if (res.next > res.end) res.next = res.end;
}

/* one walker-buffer entry of a warp's reservation (rank among the warp's
 * walkers of this item); false when the buffer is full (or the read too
 * long for the entry's anchor bits): the walk is then left over */
__device__ __forceinline__ bool gs_push_walker(const GsBatch &B, const GsReserve &res, uint32_t g,
                                               uint32_t take, uint32_t rem, uint32_t rank,
                                               uint32_t r, bool fwd,
                                               int anchor, uint32_t l, uint32_t u, uint32_t jl,
                                               uint32_t ju, bool jpend, int iL)
{
    uint64_t idx;
    if (rank < rem) idx = res.next + rank;
    else idx = (uint64_t)g + (rank - rem);
    const uint64_t cap_end = rank < rem ? res.end : min((uint64_t)g + take, B.walker_cap);
    return gs_put_walker(B.walkers, idx, cap_end, r, fwd, anchor, l, u, jl, ju, jpend, iL);
}

template <int NSTOP, int COUNT>
__device__ __forceinline__ void gs_start_item(const GsDevIndex &I, const GsBatch &B, uint32_t r,
                                             uint32_t local, uint32_t L, uint64_t off, int lane,
                                             GsReserve &res, unsigned long long &wk,
                                             unsigned long long &wb)
{
    const int k = B.k;
    const uint32_t n = L - (uint32_t)k + 1u;
    const uint32_t nch = (n + GS_CHUNK - 1) / GS_CHUNK;
    const bool fwd = local < nch;
    const uint32_t chunk = fwd ? local : local - nch;
    const uint32_t ci = chunk * GS_CHUNK + (uint32_t)lane;
    const bool in_range = ci < n;
    /* lane 31 only starts the next item's first candidate (which that item
     * owns: ceil(n / GS_CHUNK) items cover every candidate) */
    const bool owned = in_range && lane < GS_CHUNK;
    const unsigned char *seq = (const unsigned char *)B.seqs + off;
    const int iL = (int)L;
    const int anchor = fwd ? (k - 1 + (int)ci) : ((int)n - 1 - (int)ci);
    const int dir = fwd ? -1 : 1;

    uint32_t l = 1, u = 0, fcode = 4;
    int pos = anchor;
    bool alive = false, ok = false, contained = false;
    if (in_range)
        ok = gs_start<NSTOP, false>(I, seq, anchor, dir, fwd, gs_start_len(I, k), iL, l, u, pos,
                                    alive, contained, fcode, wk, wb);
    /* lane+1 holds the neighbour toward the longer match (e+1 forward, s-1
     * reverse), started at far end pos - dir */
    const uint32_t nl = __shfl_down_sync(0xffffffffu, l, 1);
    const uint32_t nu = __shfl_down_sync(0xffffffffu, u, 1);
    const int nalive = __shfl_down_sync(0xffffffffu, alive ? 1 : 0, 1);

    bool killed = false, jpend = false;
    uint32_t jl = 1, ju = 0;
    if (owned && alive && ci + 1u < n) {
        const int nb = anchor - dir;
        const uint32_t cn = fwd ? gs_fwd_code(seq[nb]) : gs_comp_code(seq[nb]);
        if (cn <= 3u) {
            if (fcode < 4u) {
                killed = (fcode == cn);   /* otherwise X·cn does not occur: no J */
            } else if (nalive) {
                jl = nl;
                ju = nu;
                jpend = true;
            }
        }
        /* cn not ACGT: the candidates to the right never started; this one
         * walks without J and, if the rule would have stopped it, its record
         * is one the filters drop */
    }

    const bool walker = owned && alive && !killed;
    const uint32_t wm = __ballot_sync(0xffffffffu, walker);
    if (owned && !walker) gs_write_record(B, r, n, fwd, anchor, pos, l, u, ok, killed);
    if (!wm) return;
    /* entries for this item's walkers: the rest of the reservation, then a
     * new chunk */
    const uint32_t cnt = (uint32_t)__popc(wm);
    const uint32_t rank = (uint32_t)__popc(wm & ((1u << lane) - 1u));
    const uint32_t rem = res.end - res.next;
    uint32_t take;
    const uint32_t g = gs_reserve(B, res, cnt, rem, lane, take);
    if (walker && !gs_push_walker(B, res, g, take, rem, rank, r, fwd, anchor, l, u, jl, ju, jpend, iL))
        gs_write_leftover(B, r, n, fwd, anchor, l, u);
    gs_reserved(B, res, cnt, rem, g, take);
}

/* Whether a candidate that is to walk is contained in its neighbour at the
 * start already (walk cleared), and whether it carries the neighbour's start
 * interval as J, one base short.  cn: the neighbour's base; f, nf: the
 * candidate's and the neighbour's GS_START_* flags. */
__device__ __forceinline__ void gs_start_settle(uint32_t cn, uint32_t fcode, uint32_t f, uint32_t nf,
                                                bool &walk, bool &j)
{
    if (f & GS_START_ROWS) {
        walk = !(f & GS_START_IN);
        j = (f & GS_START_J) != 0u;
        return;
    }
    if (cn > 3u) return;   /* the candidates beyond never started: no J */
    if (fcode < 4u) {
        walk = fcode != cn;   /* forced elsewhere: the neighbour's string does not occur */
        return;
    }
    if (!(nf & GS_START_ALIVE)) return;
    if (!(nf & GS_START_KNOWN)) {
        j = true;
    } else if (nf & GS_START_TWO) {
        if (f & GS_START_ONE) walk = false;
        else j = true;
    } else if (fcode != 4u) {
        j = true;   /* the sizes may be equal at the start already */
    }
}

/* A paired work item: the windows s = GS_PCHUNK*local - 1 + lane of a read
 * (lanes 1..GS_PCHUNK own theirs; lanes 0 and 31 start their windows only
 * for the neighbours' J), each window's forward candidate (ending at
 * s+KT-1, neighbour e+1 = lane+1) and reverse candidate (starting at s,
 * neighbour s-1 = lane-1) from one start-table entry: its two keys are the
 * window and its reverse complement.  A window that holds another letter
 * than a plain base, or whose entry is too wide to pack, starts each
 * candidate on its own.  No record is written here: a start is KT < k bases
 * long.
 *
 * Which candidates walk.  Not those whose next one or two bases make a
 * string that does not occur, where that keeps them below length k
 * (GS_START_DEAD).  Not those contained in their neighbour: by their few
 * rows' contexts (gs_start_flags), forced to its base, or a single row after one base where the neighbour's string, one
 * base longer, still occurs (its own two-base extension: the same bases).
 * Of the others, those whose neighbour's string no longer occurs after one
 * base walk without J (at the start itself the sizes differ: no forced
 * code). */
template <int NSTOP>
__device__ __forceinline__ void gs_start_pair_item(const GsDevIndex &I, const GsBatch &B, uint32_t r,
                                                   uint32_t local, int iL, uint64_t off, int lane,
                                                   GsReserve &res, unsigned long long &wk)
{
    const int k = B.k, KT = I.kx;
    const int s = (int)(local * GS_PCHUNK) - 1 + lane;
    const bool in_range = s >= 0 && s <= iL - KT;
    const bool owned = in_range && lane >= 1 && lane <= GS_PCHUNK;
    const bool vf = in_range && s >= k - KT;   /* forward candidate s+KT-1 >= k-1 */
    const bool vr = in_range && s <= iL - k;   /* reverse candidate s <= L-k */
    const unsigned char *seq = (const unsigned char *)B.seqs + off;
    const int ef = s + KT - 1;
    uint32_t lo, hi, odd;
    gs_warp_bases(seq, iL, s - lane - 6, lane, lo, hi, odd);
    /* the walks' next six bases, the nearest at bits 10-11: s-1, s-2, ...
     * forward, the complements of s+KT, s+KT+1, ... reverse; how many are
     * plain; and the neighbours' bases, s+KT and s-1 */
    const uint32_t before = lo & 0xfffu;
    const uint32_t after = (uint32_t)((((uint64_t)hi << 32) | lo) >> (2 * (KT + 6))) & 0xfffu;
    const uint32_t rev = __brev(~after << 20);   /* the 12 bits reversed */
    const uint32_t rwalk = ((rev >> 1) & 0x555u) | ((rev & 0x555u) << 1);
    const uint32_t ob = odd << 26, oa = (odd >> (KT + 6)) & 0x3fu;
    const int fnv = ob ? __clz(ob) : 6, rnv = oa ? __ffs(oa) - 1 : 6;
    uint32_t fcn = 4u, rcn = 4u;
    if (ef + 1 < iL && in_range) fcn = rnv > 0 ? after & 3u : gs_fwd_code(seq[ef + 1]);
    if (s >= 1 && in_range) rcn = fnv > 0 ? 3u - (before >> 10) : gs_comp_code(seq[s - 1]);

    uint32_t fl = 1u, fu = 0u, ff = 0u, fcode = 4u, rl = 1u, ru = 0u, rf = 0u, rcode = 4u;
    if (vf || vr) {
        bool apart = ((odd >> 6) & ((1u << KT) - 1u)) != 0u;
        if (!apart) {
            /* the reverse key: complement codes, R[s] at bits 0-1; the forward
             * key (R[s+KT-1] at bits 0-1) is its reverse complement */
            const uint32_t pr = ~__funnelshift_r(lo, hi, 12) & (0xffffffffu >> (32 - 2 * KT));
            const uint4 e = gs_ld_pair(&I.kmerx[gs_kmer_rc(pr, KT)]);
            fcode = e.y & 7u;
            rcode = e.w & 7u;
            apart = (vf && e.y == GS_ENTRY_WIDE) || (vr && e.w == GS_ENTRY_WIDE);
            if (vf) {
                fl = e.x;
                fu = e.x + gs_entry_size(e.y) - 1u;
                ff = gs_start_flags(e.y, before, fnv, fcn, k - KT);
            }
            if (vr) {
                rl = e.z;
                ru = e.z + gs_entry_size(e.w) - 1u;
                rf = gs_start_flags(e.w, rwalk, rnv, rcn, k - KT);
            }
        }
        wk += (vf ? 1u : 0u) + (vr ? 1u : 0u);   /* entries: a paired one is two */
        if (apart) {
            if (vf) {
                const GsStart S = gs_start_apart<NSTOP>(I, seq, ef, true, KT, iL);
                fl = S.l; fu = S.u; fcode = S.fcode < 4u ? S.fcode : GS_CODE_UNKNOWN;
                ff = S.alive ? GS_START_ALIVE : 0u;
            }
            if (vr) {
                const GsStart S = gs_start_apart<NSTOP>(I, seq, s, false, KT, iL);
                rl = S.l; ru = S.u; rcode = S.fcode < 4u ? S.fcode : GS_CODE_UNKNOWN;
                rf = S.alive ? GS_START_ALIVE : 0u;
            }
        }
    }
    const uint32_t nff = __shfl_down_sync(0xffffffffu, ff, 1);
    const uint32_t nrf = __shfl_up_sync(0xffffffffu, rf, 1);
    bool wf = owned && (ff & (GS_START_ALIVE | GS_START_DEAD)) == GS_START_ALIVE;
    bool wr = owned && (rf & (GS_START_ALIVE | GS_START_DEAD)) == GS_START_ALIVE;
    bool fj = false, rj = false;
    if (wf) gs_start_settle(fcn, fcode, ff, nff, wf, fj);
    if (wr) gs_start_settle(rcn, rcode, rf, nrf, wr, rj);
    const uint32_t mf = __ballot_sync(0xffffffffu, wf), mr = __ballot_sync(0xffffffffu, wr);
    if (!(mf | mr)) return;
    const uint32_t fnl = __shfl_down_sync(0xffffffffu, fl, 1);
    const uint32_t fnu = __shfl_down_sync(0xffffffffu, fu, 1);
    const uint32_t rnl = __shfl_up_sync(0xffffffffu, rl, 1);
    const uint32_t rnu = __shfl_up_sync(0xffffffffu, ru, 1);
    const uint32_t n = (uint32_t)(iL - k + 1);   /* candidates per strand (the item exists: L >= k) */
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t cnt = (uint32_t)(__popc(mf) + __popc(mr));
    const uint32_t rem = res.end - res.next;
    uint32_t take;
    const uint32_t g = gs_reserve(B, res, cnt, rem, lane, take);
    if (wf && !gs_push_walker(B, res, g, take, rem, (uint32_t)__popc(mf & lt), r, true, ef, fl, fu,
                              fj ? fnl : 1u, fj ? fnu : 0u, fj, iL))
        gs_write_leftover(B, r, n, true, ef, fl, fu);
    if (wr && !gs_push_walker(B, res, g, take, rem, (uint32_t)(__popc(mf) + __popc(mr & lt)), r, false,
                              s, rl, ru, rj ? rnl : 1u, rj ? rnu : 0u, rj, iL))
        gs_write_leftover(B, r, n, false, s, rl, ru);
    gs_reserved(B, res, cnt, rem, g, take);
}

/* 5 CTAs of 256 per SM (48 registers, no spills): more lookups in flight
 * than 4 or 3 (config-3 search 101.1 / 101.8 / 104.5 ms) */
#define GS_START_CTAS 5

template <int NSTOP, int COUNT, bool PAIRED>
__global__ void __launch_bounds__(256, GS_START_CTAS) gs_search_start(GsDevIndex I, GsBatch B, int queue_chunk)
{
    gs_after_previous();
    const int lane = threadIdx.x & 31;
    unsigned long long wk = 0, wb = 0;
    GsReserve res = {0u, 0u, B.walker_cap == 0 ? 1u : 0u};
    const uint32_t n_items = B.item_off[B.n_reads];
    if (n_items > B.item_read_cap) {
        /* a captured pass replayed on larger input: report, do nothing */
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(B.queue + 1, GS_FLAG_OVERFLOW);
        return;
    }
    for (;;) {
        uint32_t first = 0;
        if (lane == 0) first = atomicAdd(B.queue, (uint32_t)queue_chunk);
        first = __shfl_sync(0xffffffffu, first, 0);
        if (first >= n_items) break;
        const uint32_t last = min(first + (uint32_t)queue_chunk, n_items);
        /* up to 32 items at a time, each lane looking up one item's read */
        for (uint32_t it = first; it < last; it += 32) {
            const int m = (int)min(last - it, 32u);
            uint32_t ir = 0, il = 0, iLen = 0;
            uint64_t ioff = 0;
            if (lane < m) {
                ir = B.item_read[it + (uint32_t)lane];
                il = it + (uint32_t)lane - B.item_off[ir];
                iLen = B.lengths[ir];
                ioff = B.offsets[ir];
            }
            for (int j = 0; j < m; j++) {
                const uint32_t r = __shfl_sync(0xffffffffu, ir, j);
                const uint32_t local = __shfl_sync(0xffffffffu, il, j);
                const uint32_t L = __shfl_sync(0xffffffffu, iLen, j);
                const uint64_t off = __shfl_sync(0xffffffffu, ioff, j);
                if (PAIRED) gs_start_pair_item<NSTOP>(I, B, r, local, (int)L, off, lane, res, wk);
                else gs_start_item<NSTOP, COUNT>(I, B, r, local, L, off, lane, res, wk, wb);
            }
        }
    }
    /* unused entries of the last reservation: holes */
    for (uint32_t i = res.next + (uint32_t)lane; i < res.end; i += 32) B.walkers[i].r = GS_WALKER_HOLE;
    if (COUNT) gs_add_work(B, wk, wb);
}

#define GS_WALK_WARPS 4
#define GS_WALK_CTAS 8

/* A warp's part [next, end) of a list that all warps append to, in shared
 * memory; full once the list gave no more room (no further atomics, so that
 * the 32-bit counter cannot wrap) */
struct GsListPart {
    uint32_t next, end, full, used;
};

/* Places for the lanes of m in a list of `cap` entries with counter *count
 * (at or past cap: no room): the rest of the warp's part, then a new part of
 * `chunk` entries or more -- one atomic a part instead of one a push, on an
 * address that every warp of the grid takes turns at. */
__device__ __forceinline__ uint32_t gs_list_room(GsListPart &part, uint32_t *count, uint32_t chunk,
                                                 uint32_t cap, uint32_t m, int lane)
{
    const uint32_t cnt = (uint32_t)__popc(m), rank = (uint32_t)__popc(m & ((1u << lane) - 1u));
    const uint32_t at = part.next, rem = part.end - at, full = part.full;
    __syncwarp();
    uint32_t g = cap;
    if (rem < cnt && !full) {
        const uint32_t take = max(chunk, cnt - rem);
        if (lane == 0) g = atomicAdd(count, take);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (lane == 0) {
            part.full = (uint64_t)g + take >= cap;
            part.next = (uint32_t)min((uint64_t)g + (cnt - rem), (uint64_t)cap);
            part.end = (uint32_t)min((uint64_t)g + take, (uint64_t)cap);
        }
    } else if (lane == 0) {
        part.next = rem < cnt ? part.end : at + cnt;
    }
    __syncwarp();
    const uint64_t j = rank < rem ? (uint64_t)at + rank : (uint64_t)g + (rank - rem);
    return (uint32_t)min(j, (uint64_t)cap);
}

template <int NSTOP, int COUNT, int TEXT>
__global__ void __launch_bounds__(GS_WALK_WARPS * 32, GS_WALK_CTAS) gs_search_walk(GsDevIndex I, GsBatch B)
{
    gs_after_previous();
    __shared__ GsListPart s_text[GS_WALK_WARPS];
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    GsListPart &text = s_text[threadIdx.x >> 5];
    if (lane == 0) {
        text.next = text.end = text.used = 0u;
        text.full = B.text_cap == 0;
    }
    __syncwarp();
    unsigned long long wb = 0;
    /* walker indices fit 32 bits: the buffer holds at most 2^31 entries */
    uint32_t n_w = *(volatile uint32_t *)(B.queue + 2);
    if (n_w > B.walker_cap) n_w = (uint32_t)B.walker_cap;
    const uint32_t wsz = gs_walk_window(n_w, gridDim.x * GS_WALK_WARPS);
    uint32_t win = 0, win_end = 0;   /* warp-uniform window of walker indices */
    bool have = false, exhausted = false, killed = false, jpend = false;
    uint32_t r = 0, l = 0, u = 0, jl = 0, ju = 0, n = 0;
    int anchor = 0, pos = 0, iL = 0, dir = 0;
    bool fwd = false;
    const unsigned char *seq = NULL;
    GsAhead pre = {0, 0, false};
    GsWalkCounts wc = {0ull, 0ull, 0ull, 0ull, 0ull, 0ull, 0ull};
    for (;;) {
        uint32_t need = __ballot_sync(0xffffffffu, !have);
        while (need && !exhausted) {
            if (win == win_end) {
                uint32_t g = 0;
                if (lane == 0) g = atomicAdd(B.queue + 3, wsz);
                g = __shfl_sync(0xffffffffu, g, 0);
                if (g >= n_w) {
                    exhausted = true;
                    break;
                }
                win = g;
                win_end = min(g + wsz, n_w);
            }
            const uint32_t take = min((uint32_t)__popc(need), win_end - win);
            const uint32_t rank = __popc(need & lt);
            if (((need >> lane) & 1u) && rank < take) {
                GsWalker w = B.walkers[win + rank];
                if (w.r != GS_WALKER_HOLE) {
                    r = w.r;
                    fwd = (w.anchor & GS_WALKER_FWD) != 0;
                    anchor = (int)(w.anchor & (GS_WALKER_JPEND - 1u));
                    dir = fwd ? -1 : 1;
                    pos = anchor + dir * (gs_start_len(I, B.k) - 1);
                    l = w.l;
                    u = w.u;
                    jl = w.jl;
                    ju = w.ju;
                    dir = fwd ? -1 : 1;
                    const uint32_t Lr = B.lengths[r];
                    iL = (int)Lr;
                    n = Lr - (uint32_t)B.k + 1u;
                    seq = (const unsigned char *)B.seqs + B.offsets[r];
                    have = true;
                    killed = false;
                    jpend = (w.anchor & GS_WALKER_JPEND) != 0;
                    const int np = jpend ? pos : pos + dir, nn = np + dir;
                    pre.first = np >= 0 && np < iL ? seq[np] : 0;
                    pre.second = nn >= 0 && nn < iL ? seq[nn] : 0;
                    pre.alone = false;
                    if (COUNT && (jpend || jl <= ju)) wc.jwalkers++;
                }
            }
            win += take;
            need = __ballot_sync(0xffffffffu, !have);
        }
        if (!__ballot_sync(0xffffffffu, have)) {
            if (exhausted) break;
            continue;
        }
        if (have && !gs_walk_step<NSTOP, COUNT, TEXT, true>(I, seq, iL, fwd, dir, l, u, jl, ju, pos,
                                                             jpend, killed, wb, &wc, &pre)) {
            gs_write_record(B, r, n, fwd, anchor, pos, l, u, true, killed);
            have = false;
        }
        /* walkers that entered text mode go to the text pass, so that no
         * lane of this pass runs the compare; without room they walk on
         * (gs_text_mode written out: compiled through it, a pass over long
         * reads took 1 % more) */
        const bool tx = TEXT != GS_TEXT_NONE && have && jl >= GS_TEXT_MARK;
        const uint32_t tm = __ballot_sync(0xffffffffu, tx);
        if (tm) {
            const uint32_t cap = (uint32_t)B.text_cap;
            const uint32_t j = gs_list_room(text, B.queue + 4, B.text_chunk, cap, tm, lane);
            if (tx) {
                if (j < cap) {
                    atomicAdd(&text.used, 1u);
                    GsTextJob t;
                    t.r = r;
                    t.anchor = (uint32_t)anchor | (fwd ? GS_WALKER_FWD : 0u);
                    t.pos = (uint32_t)pos;
                    t.l = l;
                    B.text_jobs[j] = t;
                    have = false;
                } else {
                    jl = 1u;
                    ju = 0u;
                }
            }
        }
    }
    /* what the warp reserved and did not fill */
    __syncwarp();
    for (uint32_t j = text.next + (uint32_t)lane; j < text.end; j += 32)
        B.text_jobs[j].r = GS_WALKER_HOLE;
    if (lane == 0 && text.used) atomicAdd(B.queue + 5, text.used);
    if (COUNT) {
        gs_add_work(B, 0, wb);
        unsigned long long v[7] = {wc.steps, wc.jsteps, wc.jblocks, wc.jshrank, wc.jwalkers,
                                   wc.lines256, wc.lines384};
        for (int i = 0; i < 7; i++) {
            for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
            if (lane == 0) atomicAdd(&B.work[4 + i], v[i]);
        }
    }
}

/* Text pass: the walkers the walk pass handed over, one per thread, each
 * run to its end in text mode (and back in the interval walk after a
 * wildcard base). */
template <int NSTOP, int COUNT>
__global__ void __launch_bounds__(256) gs_search_text(GsDevIndex I, GsBatch B)
{
    gs_after_previous();
    uint64_t n_jobs = B.queue[4];
    if (n_jobs > B.text_cap) n_jobs = B.text_cap;
    unsigned long long wb = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n_jobs; j += stride) {
        const GsTextJob t = B.text_jobs[j];
        const uint32_t r = t.r;
        if (r == GS_WALKER_HOLE) continue;
        const bool fwd = (t.anchor & GS_WALKER_FWD) != 0;
        const int anchor = (int)(t.anchor & ~GS_WALKER_FWD);
        const int dir = fwd ? -1 : 1;
        const uint32_t Lr = B.lengths[r];
        const int iL = (int)Lr;
        const unsigned char *seq = (const unsigned char *)B.seqs + B.offsets[r];
        int pos = (int)t.pos;
        uint32_t l = t.l, u = t.l, jl = GS_TEXT_MARK, ju = 0u;
        bool jpend = false, killed = false;
        while (gs_walk_step<NSTOP, COUNT, GS_TEXT_RUN>(I, seq, iL, fwd, dir, l, u, jl, ju, pos, jpend,
                                                killed, wb)) {
        }
        gs_write_record(B, r, Lr - (uint32_t)B.k + 1u, fwd, anchor, pos, l, u, true, killed);
    }
    if (COUNT) gs_add_work(B, 0, wb);
}

/* ------------------------------------------------------------------ */
/* plain search: one read per thread */

/* Leftover pass: the walks the start pass left in their record slots
 * (GS_LEFTOVER_MARK), a warp per read, each slot's walk on one lane, started
 * again with its J as the start pass would have made it; the slot gets the
 * walk's record, or loses its record bit.  Returns at once when the start
 * pass left none. */
template <int NSTOP, int COUNT, int TEXT>
__global__ void __launch_bounds__(256) gs_search_leftover(GsDevIndex I, GsBatch B)
{
    gs_after_previous();
    if (!(*(volatile uint32_t *)(B.queue + 1) & GS_FLAG_LEFTOVER)) return;
    const int lane = threadIdx.x & 31;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const int k = B.k, KT = gs_start_len(I, k);
    unsigned long long wk = 0, wb = 0;
    for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < B.n_reads; r += nwarps) {
        const uint64_t base = B.slot_off[r], end = B.slot_off[r + 1];
        if (end > B.slot_cap) continue;
        const uint32_t n = (uint32_t)((end - base) >> 1);
        const int iL = (int)B.lengths[r];
        const unsigned char *seq = (const unsigned char *)B.seqs + B.offsets[r];
        for (uint32_t j = (uint32_t)lane; j < 2u * n; j += 32) {
            const uint64_t slot = base + j;
            if (!((B.recmask[slot >> 5] >> (slot & 31u)) & 1u)) continue;
            const GsRec rec = B.slots[slot];
            if ((uint32_t)rec.x != GS_LEFTOVER_MARK || (uint32_t)rec.y != GS_LEFTOVER_MARK) continue;
            const bool fwd = j < n;
            /* slot j: forward e = k-1+j, reverse s = j-n (gs_write_record) */
            const int anchor = fwd ? k - 1 + (int)j : (int)(j - n);
            const int dir = fwd ? -1 : 1;
            /* the walker as the start pass made it: its start, and J from
             * the start of its neighbour toward the longer match (gs_start_item) */
            uint32_t l, u, fcode, jl = 1u, ju = 0u;
            int pos;
            bool alive, contained, jpend = false, killed = false;
            gs_start<NSTOP, false>(I, seq, anchor, dir, fwd, KT, iL, l, u, pos, alive, contained,
                                   fcode, wk, wb);
            const int nb = anchor - dir;
            if (alive && fcode >= 4u && nb >= 0 && nb < iL &&
                (fwd ? gs_fwd_code(seq[nb]) : gs_comp_code(seq[nb])) <= 3u) {
                uint32_t nl, nu, nfc;
                int npos;
                bool nalive, ncont;
                gs_start<NSTOP, false>(I, seq, nb, dir, fwd, KT, iL, nl, nu, npos, nalive, ncont,
                                       nfc, wk, wb);
                if (nalive) {
                    jl = nl;
                    ju = nu;
                    jpend = true;
                }
            }
            while (alive && gs_walk_step<NSTOP, COUNT, TEXT>(I, seq, iL, fwd, dir, l, u, jl, ju, pos,
                                                             jpend, killed, wb)) {
            }
            /* no record: drop the slot's bit (gs_write_record leaves it) */
            atomicAnd(B.recmask + (slot >> 5), ~(1u << (slot & 31u)));
            gs_write_record(B, r, n, fwd, anchor, pos, l, u, true, killed);
        }
    }
    if (COUNT) gs_add_work(B, wk, wb);
}

template <int NSTOP>
__global__ void __launch_bounds__(128) gs_search_plain(GsDevIndex I, GsBatch B)
{
    uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= B.n_reads) return;
    const uint32_t L = B.lengths[r];
    const int k = B.k;
    if (L < (uint32_t)k) return;
    const uint32_t n = L - (uint32_t)k + 1u;
    const unsigned char *seq = (const unsigned char *)B.seqs + B.offsets[r];
    uint32_t *H = B.hist + B.offsets[r];
    GsRec *slots = B.slots + B.slot_off[r];
    const int iL = (int)L;
    unsigned long long w_kmer = 0, w_blk = 0;
    const int KT = gs_start_len(I, k);

    for (int strand = 0; strand < 2; strand++) {
        const bool fwd = strand == 0;
        for (uint32_t q = 0; q < L; q++) H[q] = 0;
        for (uint32_t ci = 0; ci < n; ci++) {
            /* forward: e from L-1 down; reverse: s from 0 up */
            int anchor = fwd ? iL - 1 - (int)ci : (int)ci;
            const int dir = fwd ? -1 : 1;
            uint32_t l = 1, u = 0;
            int pos = anchor;
            bool alive = false;
            bool contained = false;
            uint32_t fcode = 4;
            bool ok = gs_start<NSTOP, true>(I, seq, anchor, dir, fwd, KT, iL, l, u, pos, alive, contained,
                                            fcode, w_kmer, w_blk);
            bool killed = contained;
            if (contained) {
                /* it reached its start level: the candidates to its left may
                 * compare with it there */
                H[pos] = u - l + 1u;
                alive = false;
            }
            if (alive) {
                uint32_t sz = u - l + 1u;
                uint32_t h = H[pos];
                H[pos] = sz;
                killed = (h == sz);
                while (!killed) {
                    int np = pos + dir;
                    if (np < 0 || np >= iL) break;
                    uint32_t c = fwd ? gs_fwd_code(seq[np]) : gs_comp_code(seq[np]);
                    uint32_t nl = l, nu = u;
                    if (c > 3u) {
                        if (NSTOP) break;
                    } else {
                        w_blk += (unsigned long long)gs_step(I, nl, nu, c);
                        if (nl > nu) break;
                    }
                    l = nl;
                    u = nu;
                    pos = np;
                    sz = u - l + 1u;
                    h = H[pos];
                    H[pos] = sz;
                    killed = (h == sz);
                }
            }
            GsRec rec;
            rec.x = 0; rec.y = 0; rec.l = l; rec.u = u;
            if (!killed && ok) {
                if (fwd) {
                    if (anchor - pos + 1 >= k) { rec.x = pos; rec.y = anchor + 1; }
                } else if (l <= u && pos + 1 - anchor >= k) {
                    rec.x = (int32_t)((uint32_t)anchor | 0x80000000u);
                    rec.y = (int32_t)((uint32_t)(pos + 1) | 0x80000000u);
                }
            }
            if (rec.y != 0) {
                const uint64_t slot = B.slot_off[r] + (fwd ? (uint64_t)(anchor - (k - 1))
                                                           : (uint64_t)n + (uint64_t)anchor);
                slots[slot - B.slot_off[r]] = rec;
                atomicOr(B.recmask + (slot >> 5), 1u << (slot & 31u));
            }
        }
    }
    if (B.work) {
        atomicAdd(&B.work[0], w_kmer);
        atomicAdd(&B.work[1], w_blk);
    }
}

/* ------------------------------------------------------------------ */

static int gs_launch_batched(const GsDevIndex &I, GsBatch &B, int queue_chunk, int ctas_per_sm,
                            uint32_t n_items, cudaStream_t st)
{
    int dev = 0, sms = 0;
    GS_CUDA(cudaGetDevice(&dev));
    GS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const bool cnt = B.work != NULL, nstop = B.n_mode == GS_N_STOP;
    void (*start)(GsDevIndex, GsBatch, int) =
        B.paired ? (nstop ? (cnt ? gs_search_start<1, 1, true> : gs_search_start<1, 0, true>)
                          : (cnt ? gs_search_start<0, 1, true> : gs_search_start<0, 0, true>))
                 : (nstop ? (cnt ? gs_search_start<1, 1, false> : gs_search_start<1, 0, false>)
                          : (cnt ? gs_search_start<0, 1, false> : gs_search_start<0, 0, false>));
    void (*walk)(GsDevIndex, GsBatch) =
        I.text_min ? (nstop ? (cnt ? gs_search_walk<1, 1, GS_TEXT_GIVEN> : gs_search_walk<1, 0, GS_TEXT_GIVEN>)
                            : (cnt ? gs_search_walk<0, 1, GS_TEXT_GIVEN> : gs_search_walk<0, 0, GS_TEXT_GIVEN>))
                   : (nstop ? (cnt ? gs_search_walk<1, 1, GS_TEXT_NONE> : gs_search_walk<1, 0, GS_TEXT_NONE>)
                            : (cnt ? gs_search_walk<0, 1, GS_TEXT_NONE> : gs_search_walk<0, 0, GS_TEXT_NONE>));
    if (ctas_per_sm <= 0) ctas_per_sm = GS_START_CTAS;
    uint32_t grid = (uint32_t)sms * (uint32_t)ctas_per_sm;
    /* a captured pass knows its items only on the device: as many as the
     * pass it was sized by */
    const uint32_t items = n_items ? n_items : B.item_cap;
    if (queue_chunk <= 0) {
        /* a warp's share of the items, 1 to GS_QUEUE_CHUNK_MAX: items take
         * alike long, and each grab is a chain of three dependent accesses
         * (60,007 short reads, 17 items a warp: start pass 123 -> 79 us
         * against an eighth of a share) */
        const uint32_t share = items / (grid * 8u);
        queue_chunk = share < 1u ? 1 : share > GS_QUEUE_CHUNK_MAX ? GS_QUEUE_CHUNK_MAX : (int)share;
    }
    if (n_items) {
        uint32_t need = (n_items + (uint32_t)queue_chunk - 1) / (uint32_t)queue_chunk;
        if (need < grid * 8) grid = (need + 7) / 8;
    }
    if (grid == 0) grid = 1;
    B.walker_chunk = gs_walker_chunk(B.walker_cap, grid * 8u);
    GS_CUDA(gs_launch_after(start, grid, 256, st, I, B, queue_chunk));
    if (B.walker_cap) {
        /* no more warps than the items can have walkers for, 32 each */
        uint32_t wgrid = (uint32_t)sms * GS_WALK_CTAS;
        const uint64_t most = (uint64_t)items * (2u * GS_PCHUNK) / (GS_WALK_WARPS * 32u) + 1u;
        if (most < wgrid) wgrid = (uint32_t)most;
        B.text_chunk = gs_list_chunk(B.text_cap, wgrid * GS_WALK_WARPS);
        GS_CUDA(gs_launch_after(walk, wgrid, GS_WALK_WARPS * 32, st, I, B));
        if (B.text_cap) {
            void (*text)(GsDevIndex, GsBatch) =
                nstop ? (cnt ? gs_search_text<1, 1> : gs_search_text<1, 0>)
                      : (cnt ? gs_search_text<0, 1> : gs_search_text<0, 0>);
            uint32_t tgrid = (uint32_t)sms * 8u;
            if (B.text_cap < (uint64_t)tgrid * 256u) tgrid = (uint32_t)(B.text_cap / 256u) + 1u;
            GS_CUDA(gs_launch_after(text, tgrid, 256, st, I, B));
        }
    }
    void (*leftover)(GsDevIndex, GsBatch) =
        I.text_min
            ? (nstop ? (cnt ? gs_search_leftover<1, 1, GS_TEXT_RUN> : gs_search_leftover<1, 0, GS_TEXT_RUN>)
                     : (cnt ? gs_search_leftover<0, 1, GS_TEXT_RUN> : gs_search_leftover<0, 0, GS_TEXT_RUN>))
            : (nstop ? (cnt ? gs_search_leftover<1, 1, GS_TEXT_NONE> : gs_search_leftover<1, 0, GS_TEXT_NONE>)
                     : (cnt ? gs_search_leftover<0, 1, GS_TEXT_NONE> : gs_search_leftover<0, 0, GS_TEXT_NONE>));
    uint32_t lgrid = (uint32_t)sms * 8u;
    if (B.n_reads < lgrid * 8u) lgrid = B.n_reads / 8u + 1u;
    GS_CUDA(gs_launch_after(leftover, lgrid, 256, st, I, B));
    return GS_OK;
}

int gs_launch_search(const GsDevIndex &I, GsBatch &B, int kernel, int queue_chunk, int ctas_per_sm,
                     uint32_t n_items, cudaStream_t st)
{
    if (B.n_reads == 0) return GS_OK;
    if (kernel == GS_KERNEL_BATCHED) return gs_launch_batched(I, B, queue_chunk, ctas_per_sm, n_items, st);
    if (kernel == GS_KERNEL_PLAIN) {
        uint32_t nb = (B.n_reads + 127) / 128;
        if (B.n_mode == GS_N_STOP) gs_search_plain<1><<<nb, 128, 0, st>>>(I, B);
        else gs_search_plain<0><<<nb, 128, 0, st>>>(I, B);
        GS_CUDA(cudaGetLastError());
        return GS_OK;
    }
    int dev = 0, sms = 0;
    GS_CUDA(cudaGetDevice(&dev));
    GS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (queue_chunk <= 0) queue_chunk = GS_QUEUE_CHUNK;
    /* count_work: instances that also count the lookups they execute */
    const bool cnt = B.work != NULL, nstop = B.n_mode == GS_N_STOP;
    void (*batched)(GsDevIndex, GsBatch, int) =
        nstop ? (cnt ? gs_search_lockstep<1, 1> : gs_search_lockstep<1, 0>)
              : (cnt ? gs_search_lockstep<0, 1> : gs_search_lockstep<0, 0>);
    void (*tail)(GsDevIndex, GsBatch) = nstop ? (cnt ? gs_search_tail<1, 1> : gs_search_tail<1, 0>)
                                              : (cnt ? gs_search_tail<0, 1> : gs_search_tail<0, 0>);
    if (ctas_per_sm <= 0) {
        int occ = 0;
        GS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, batched, 256, 0));
        ctas_per_sm = occ > 0 ? occ : 1;
    }
    uint32_t grid = (uint32_t)sms * (uint32_t)ctas_per_sm;
    if (n_items) {
        uint32_t need = (n_items + (uint32_t)queue_chunk - 1) / (uint32_t)queue_chunk;
        uint32_t warps = grid * 8;
        if (need < warps) grid = (need + 7) / 8;
    }
    if (grid == 0) grid = 1;
    GS_CUDA(cudaMemsetAsync(B.queue, 0, sizeof(uint32_t), st));
    if (B.cont) GS_CUDA(cudaMemsetAsync(B.queue + 2, 0, 2 * sizeof(uint32_t), st));
    batched<<<grid, 256, 0, st>>>(I, B, queue_chunk);
    GS_CUDA(cudaGetLastError());
    if (B.cont) {
        int tocc = 0;
        GS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&tocc, tail, 256, 0));
        uint32_t tgrid = (uint32_t)sms * (uint32_t)(tocc > 0 ? tocc : 4);
        tail<<<tgrid, 256, 0, st>>>(I, B);
        GS_CUDA(cudaGetLastError());
    }
    return GS_OK;
}
