/*
 * gs_build.cu -- index construction on the GPU.
 *
 * Replaces build_index.sh (bwa index -b sa -r R, then bwa index -b bwt with
 * OCC_INTERVAL 0x40; build_index.sh:36-75), whose bwa fork is not available:
 * it produces the .bwt/.sa pair in the layout the reference reads
 * (seed_gen.cu:2685-2736, :52-58) for a forward-strand text.
 *
 *   suffix array  prefix doubling over 32-bit ranks, a rank being the first
 *                 place of its group: initial keys pack the first 17 (20)
 *                 characters in base 5 ($ = 0 < A..T); each later round sorts
 *                 (rank[i], rank[i+h]) with a 64-bit LSD radix sort for the
 *                 suffixes whose rank is still shared, and only those;
 *   BWT           B[row] = T[SA[row]-1], the $ row dropped (primary), packed
 *                 into blocks of 64 rows: counts of A,C,G,T before the block
 *                 (a scan of the blocks' counts) + 4 words of 16 bases, MSB
 *                 first;
 *   sampled SA    SA[i * sa_intv] for i >= 1.
 *
 * The blocks stay on the device for the index that is returned; they go to
 * the host for the files alone.
 *
 * Bound by the first sort's five passes and the start table's kernels, not
 * by the host.  Ten million bases (an eighth of repeats), built, seeded with
 * and freed: 6.6 ms, of which sorting is 1.7 (0.9 in the first round).  Six
 * rounds over all suffixes, the host's pass over the codes and the blocks'
 * round trip over the host took 16.5 ms, of which 4.4 were the sorts.
 *
 * Memory: about 33 bytes per base on the device (keys and values double
 * buffered, ranks, suffix array, text); a 3.1 Gbp text needs ~103 GB of HBM.
 */
#include "gs_internal.h"

#include <cub/cub.cuh>

#include <stdlib.h>
#include <string.h>

/* what a round leaves for the host */
struct GsSaState {
    uint32_t left;       /* suffixes whose rank is shared */
    uint32_t pad;
    unsigned long long bad;   /* first code that is not 0..3, or ~0 */
};

/* keys of the first H characters, by 5 (0: past the end) */
template <int H>
static __global__ void init_keys(const uint8_t *__restrict__ T, uint64_t n, uint64_t *keys, uint32_t *vals,
                                 GsSaState *st)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t k = 0;
        if (i < n && T[i] > 3) atomicMin(&st->bad, (unsigned long long)i);
#pragma unroll
        for (int j = 0; j < H; j++) {
            uint64_t p = i + (uint64_t)j;
            uint64_t c = p < n ? (uint64_t)T[p] + 1u : 0u;
            k = k * 5u + c;
        }
        keys[i] = k;
        vals[i] = (uint32_t)i;
    }
}

/* Of the sorted keys, per place: where its group of this round's ranks (key
 * >> shift) and its group of equal keys begin, once the marks (a place that
 * begins one, else 0) are scanned by the larger of each half. */
static __global__ void group_marks(const uint64_t *keys, uint64_t N, int shift, uint64_t *marks)
{
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < N;
         j += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t k = keys[j], before = j ? keys[j - 1] : k;
        marks[j] = ((k >> shift) != (before >> shift) ? j << 32 : 0u) | (k != before ? j : 0u);
    }
}

struct GsMarkMax {
    __host__ __device__ __forceinline__ uint64_t operator()(uint64_t a, uint64_t b) const
    {
        const uint64_t ah = a >> 32, bh = b >> 32, al = a & 0xffffffffu, bl = b & 0xffffffffu;
        return ((ah > bh ? ah : bh) << 32) | (al > bl ? al : bl);
    }
};

/* Places and ranks from the sorted keys, and the suffixes whose rank is
 * still shared, in any order.  A group's places begin at its rank, key >>
 * shift (the first round's one group at 0).  One count per warp and block
 * goes to the list's end: the addition per warp alone took longer than the
 * ranks' scattered writes. */
static __global__ void __launch_bounds__(256)
settle_ranks(const uint64_t *keys, const uint32_t *vals, const uint64_t *marks, uint64_t N, int shift,
             uint32_t *sa, uint32_t *rank, uint32_t *next, GsSaState *st)
{
    __shared__ uint32_t cnt[8];
    __shared__ uint32_t base;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t j0 = (uint64_t)blockIdx.x * blockDim.x; j0 < N; j0 += stride) {
        const uint64_t j = j0 + threadIdx.x;
        bool shared = false;
        uint32_t s = 0;
        if (j < N) {
            const uint64_t m = marks[j];
            const uint64_t first = m & 0xffffffffu, at = (keys[j] >> shift) - (m >> 32);
            s = vals[j];
            sa[at + j] = s;
            rank[s] = (uint32_t)(at + first);
            shared = first != j || (j + 1 < N && (marks[j + 1] & 0xffffffffu) == first);
        }
        const uint32_t votes = __ballot_sync(0xffffffffu, shared);
        if (lane == 0) cnt[warp] = __popc(votes);
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t sum = 0;
            for (int w = 0; w < 8; w++) {
                const uint32_t c = cnt[w];
                cnt[w] = sum;
                sum += c;
            }
            base = sum ? atomicAdd(&st->left, sum) : 0u;
        }
        __syncthreads();
        if (shared) next[base + cnt[warp] + __popc(votes & ((1u << lane) - 1u))] = s;
        __syncthreads();
    }
}

/* a suffix shorter than h has its $ among its first h characters, so its
 * rank is not shared: those listed have a suffix h further on */
static __global__ void pair_keys(const uint32_t *rank, const uint32_t *list, uint64_t left, uint64_t n,
                                 uint64_t h, int b, uint64_t *keys)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < left;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t s = list[i];
        keys[i] = ((uint64_t)rank[s] << b) | (s + h <= n ? rank[s + h] : 0u);
    }
}

/* the even bits of the result from the low 16 of x */
__device__ __forceinline__ uint32_t even_bits(uint32_t x)
{
    x = (x | (x << 8)) & 0x00ff00ffu;
    x = (x | (x << 4)) & 0x0f0f0f0fu;
    x = (x | (x << 2)) & 0x33333333u;
    return (x | (x << 1)) & 0x55555555u;
}

/* A warp per 64-row block of the $-removed string: its 4 packed words and its
 * base counts; cnt[nblk] = 0.  Two rows a lane, a word from half a ballot of
 * each bit of the bases (one thread per block, reading bytes that a pass
 * before it had written, left sectors of 64 blocks to each load). */
static __global__ void pack_blocks(const uint8_t *__restrict__ T, const uint32_t *__restrict__ sa,
                                   uint64_t n, const uint32_t *rank, uint32_t *occ, uint4 *cnt,
                                   uint64_t nblk)
{
    const uint32_t lane = threadIdx.x & 31u, primary = rank[0];   /* the row of the whole text */
    const uint64_t stride = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t b = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; b <= nblk; b += stride) {
        uint32_t in[2], lo[2], hi[2];
        for (int q = 0; q < 2; q++) {
            const uint64_t s = b * 64 + q * 32 + lane;
            const bool ok = s < n;
            const uint32_t c = ok ? T[sa[s + (s >= primary ? 1u : 0u)] - 1u] : 0u;
            in[q] = __ballot_sync(0xffffffffu, ok);
            lo[q] = __ballot_sync(0xffffffffu, c & 1u);
            hi[q] = __ballot_sync(0xffffffffu, c & 2u);
        }
        if (lane == 0) {
            uint4 v = make_uint4(0, 0, 0, 0);
            for (int q = 0; q < 2; q++) {
                v.x += __popc(in[q] & ~hi[q] & ~lo[q]);
                v.y += __popc(lo[q] & ~hi[q]);
                v.z += __popc(hi[q] & ~lo[q]);
                v.w += __popc(hi[q] & lo[q]);
            }
            cnt[b] = v;
        }
        if (lane < 4 && b < nblk) {
            const uint32_t half = lane & 1u;   /* base i of a word at bits 2*(15-i) */
            const uint32_t rl = __brev(lane < 2 ? lo[0] : lo[1]), rh = __brev(lane < 2 ? hi[0] : hi[1]);
            occ[b * GS_BLOCK_WORDS + 4 + lane] =
                even_bits((half ? rl : rl >> 16) & 0xffffu) | (even_bits((half ? rh : rh >> 16) & 0xffffu) << 1);
        }
    }
}

struct GsCountSum {
    __host__ __device__ __forceinline__ uint4 operator()(const uint4 &a, const uint4 &b) const
    {
        return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
    }
};

static __global__ void write_counts(const uint4 *scan, uint64_t nblk, uint32_t *occ)
{
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nblk;
         b += (uint64_t)gridDim.x * blockDim.x)
        *reinterpret_cast<uint4 *>(occ + b * GS_BLOCK_WORDS) = scan[b];
}

static __global__ void gather_samples(const uint32_t *sa, uint64_t n_samples, uint32_t intv,
                                      uint32_t *out)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_samples;
         i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = sa[(i + 1) * intv];
}

static unsigned grid_for(uint64_t n)
{
    uint64_t g = (n + 255) / 256;
    return (unsigned)(g > 152ull * 64 ? 152ull * 64 : (g ? g : 1));
}

/* One device allocation, dealt out in pieces. */
struct DevMem {
    uint8_t *p;
    size_t used;
    DevMem() : p(NULL), used(0) {}
    ~DevMem() { release(); }
    void release()
    {
        cudaFree(p);
        p = NULL;
    }
    cudaError_t alloc(size_t bytes)
    {
        used = 0;
        return cudaMalloc(&p, bytes);
    }
    static size_t room(size_t bytes) { return (bytes + 271) & ~(size_t)255; }
    template <class T>
    void take(T *&ptr, size_t count)
    {
        ptr = (T *)(p + used);
        used += room(count * sizeof(T));
    }
};

#define BCUDA(x)                                               \
    do {                                                       \
        cudaError_t _e = (x);                                  \
        if (_e != cudaSuccess) return gs_cuda_fail(_e, #x);    \
    } while (0)

/* the built index on the device: blocks in the file's layout, of which the
 * last may be part used, and samples */
struct GsBuilt {
    uint32_t primary, tot[4], L2[4];   /* L2: cumulative counts */
    uint32_t *d_occ, *d_smp;
    uint64_t nblk, n_samples;
    DevMem mem;
};

static int build_device(const uint8_t *codes, uint64_t n, uint32_t sa_intv, GsBuilt &o)
{
    const uint64_t N = n + 1;
    const uint64_t nblk = o.nblk = (n + 63) / 64;
    o.n_samples = n / sa_intv;   /* rows intv, 2 intv, ... <= n */
    cub::DoubleBuffer<uint64_t> keys;
    cub::DoubleBuffer<uint32_t> vals;
    uint64_t *k0, *k1;
    uint32_t *v0, *v1, *rank, *sa;
    uint8_t *T, *tmp;
    GsSaState *st;
    size_t sort_bytes = 0, scan_bytes = 0, sum_bytes = 0;
    BCUDA(cub::DeviceRadixSort::SortPairs(NULL, sort_bytes, keys, vals, N, 0, 64));
    BCUDA(cub::DeviceScan::InclusiveScan(NULL, scan_bytes, (uint64_t *)NULL, (uint64_t *)NULL,
                                         GsMarkMax(), N));
    BCUDA(cub::DeviceScan::ExclusiveScan(NULL, sum_bytes, (uint4 *)NULL, (uint4 *)NULL, GsCountSum(),
                                         make_uint4(0, 0, 0, 0), nblk + 1));
    size_t tmp_bytes = sort_bytes > scan_bytes ? sort_bytes : scan_bytes;
    if (sum_bytes > tmp_bytes) tmp_bytes = sum_bytes;
    DevMem m;
    BCUDA(m.alloc(2 * DevMem::room(N * 8) + 4 * DevMem::room(N * 4) + DevMem::room(n) +
                  DevMem::room(tmp_bytes) + DevMem::room(sizeof(GsSaState))));
    m.take(k0, N);
    m.take(k1, N);
    m.take(v0, N);
    m.take(v1, N);
    m.take(rank, N);
    m.take(sa, N);
    m.take(T, n);
    m.take(tmp, tmp_bytes);
    m.take(st, 1);
    keys = cub::DoubleBuffer<uint64_t>(k0, k1);
    vals = cub::DoubleBuffer<uint32_t>(v0, v1);

    GsSaState h_st = {0, 0, ~0ull};
    BCUDA(cudaMemcpyAsync(T, codes, n, cudaMemcpyHostToDevice, 0));
    BCUDA(cudaMemcpyAsync(st, &h_st, sizeof(h_st), cudaMemcpyHostToDevice, 0));
    int b = 1;
    while (b < 32 && (1ull << b) < N) b++;
    /* as many characters as five or six passes of 8 bits sort (5^17 < 2^40,
     * 5^20 < 2^47): 17 tell apart all but the repeats of texts well below 4^17
     * (21 took a seventh pass: the first sort of ten million bases .82 ms) */
    const bool few = n < (1ull << 29);
    if (few) init_keys<17><<<grid_for(N), 256>>>(T, n, keys.Current(), vals.Current(), st);
    else init_keys<20><<<grid_for(N), 256>>>(T, n, keys.Current(), vals.Current(), st);
    BCUDA(cudaGetLastError());
    int end_bit = few ? 40 : 47, shift = 63;   /* one group */
    uint64_t h = few ? 17 : 20, left = N;
    for (int round = 0; left; round++) {
        if (round == 40) {
            gs_set_error("suffix sorting did not converge");
            return GS_EINVAL;
        }
        /* a smaller sort may be of another kind, with its own needs */
        size_t need = 0;
        BCUDA(cub::DeviceRadixSort::SortPairs(NULL, need, keys, vals, left, 0, end_bit));
        DevMem more;
        if (need > tmp_bytes) BCUDA(more.alloc(need));
        BCUDA(cub::DeviceRadixSort::SortPairs(need > tmp_bytes ? more.p : tmp, need, keys, vals, left, 0,
                                              end_bit));
        uint64_t *marks = keys.Alternate();
        group_marks<<<grid_for(left), 256>>>(keys.Current(), left, shift, marks);
        BCUDA(cudaGetLastError());
        need = scan_bytes;
        BCUDA(cub::DeviceScan::InclusiveScan(tmp, need, marks, marks, GsMarkMax(), left));
        BCUDA(cudaMemsetAsync(&st->left, 0, 4, 0));
        settle_ranks<<<grid_for(left), 256>>>(keys.Current(), vals.Current(), marks, left, shift, sa, rank,
                                              vals.Alternate(), st);
        BCUDA(cudaGetLastError());
        BCUDA(cudaMemcpy(&h_st, st, sizeof(h_st), cudaMemcpyDeviceToHost));
        if (h_st.bad != ~0ull) return GS_EINVAL;   /* the caller names the code */
        left = h_st.left;
        vals.selector ^= 1;
        shift = b;
        end_bit = 2 * b;
        if (left) pair_keys<<<grid_for(left), 256>>>(rank, vals.Current(), left, n, h, b, keys.Current());
        BCUDA(cudaGetLastError());
        h *= 2;
    }

    uint4 *cnt;
    BCUDA(o.mem.alloc(DevMem::room((nblk + 1) * GS_BLOCK_WORDS * 4) + DevMem::room((o.n_samples + 1) * 4) +
                      DevMem::room((nblk + 1) * 16)));
    o.mem.take(o.d_occ, (nblk + 1) * GS_BLOCK_WORDS);
    o.mem.take(o.d_smp, o.n_samples + 1);
    o.mem.take(cnt, nblk + 1);
    pack_blocks<<<grid_for((nblk + 1) * 32), 256>>>(T, sa, n, rank, o.d_occ, cnt, nblk);
    BCUDA(cudaGetLastError());
    BCUDA(cub::DeviceScan::ExclusiveScan(tmp, sum_bytes, cnt, cnt, GsCountSum(), make_uint4(0, 0, 0, 0),
                                         nblk + 1));
    write_counts<<<grid_for(nblk), 256>>>(cnt, nblk, o.d_occ);
    BCUDA(cudaGetLastError());
    if (o.n_samples) {
        gather_samples<<<grid_for(o.n_samples), 256>>>(sa, o.n_samples, sa_intv, o.d_smp);
        BCUDA(cudaGetLastError());
    }
    BCUDA(cudaMemcpy(&o.primary, rank, 4, cudaMemcpyDeviceToHost));
    BCUDA(cudaMemcpy(o.tot, cnt + nblk, 16, cudaMemcpyDeviceToHost));
    for (uint32_t c = 0, sum = 0; c < 4; c++) o.L2[c] = sum += o.tot[c];
    return GS_OK;
}

/* The file's .bwt words and .sa samples on the host: whole blocks, the last
 * block's used words, final counts. */
static int download(const GsBuilt &o, uint64_t n, uint32_t **bwt_out, uint64_t *bwt_words_out,
                    uint32_t **samples_out)
{
    const uint64_t nblk = o.nblk;
    uint64_t words = 4 * (nblk + 1) + (n + 15) / 16;
    uint32_t *occ = (uint32_t *)malloc((nblk + 1) * GS_BLOCK_WORDS * 4);
    uint32_t *bwt = (uint32_t *)malloc(words * 4 + 16);
    uint32_t *smp = (uint32_t *)malloc(o.n_samples * 4 + 16);
    if (!occ || !bwt || !smp) {
        free(occ); free(bwt); free(smp);
        return GS_ENOMEM;
    }
    cudaError_t e = cudaMemcpy(occ, o.d_occ, nblk * GS_BLOCK_WORDS * 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && o.n_samples)
        e = cudaMemcpy(smp, o.d_smp, o.n_samples * 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        free(occ); free(bwt); free(smp);
        return gs_cuda_fail(e, "index download");
    }
    uint64_t k = 0;
    for (uint64_t bl = 0; bl < nblk; bl++) {
        const uint32_t *ob = occ + bl * GS_BLOCK_WORDS;
        uint64_t rows = n - bl * 64 < 64 ? n - bl * 64 : 64;
        uint64_t nw = (rows + 15) / 16;
        memcpy(bwt + k, ob, 16);
        memcpy(bwt + k + 4, ob + 4, nw * 4);
        k += 4 + nw;
    }
    memcpy(bwt + k, o.tot, 16);
    k += 4;
    free(occ);
    *bwt_out = bwt;
    *bwt_words_out = k;
    *samples_out = smp;
    return GS_OK;
}

static int write_files(const char *prefix, uint32_t primary, const uint32_t L2[4], const uint32_t *bwt,
                       uint64_t words, uint32_t sa_intv, uint32_t seq_len, const uint32_t *smp,
                       uint64_t n_samples)
{
    size_t pl = strlen(prefix);
    char *fn = (char *)malloc(pl + 8);
    if (!fn) return GS_ENOMEM;
    memcpy(fn, prefix, pl);
    strcpy(fn + pl, ".bwt");
    FILE *fp = fopen(fn, "wb");
    int ok = fp != NULL;
    if (ok) {
        ok = fwrite(&primary, 4, 1, fp) == 1 && fwrite(L2, 4, 4, fp) == 4 &&
             fwrite(bwt, 4, words, fp) == words;
        ok = (fclose(fp) == 0) && ok;
    }
    if (ok) {
        strcpy(fn + pl, ".sa");
        fp = fopen(fn, "wb");
        ok = fp != NULL;
        if (ok) {
            ok = fwrite(&primary, 4, 1, fp) == 1 && fwrite(L2, 4, 4, fp) == 4 &&
                 fwrite(&sa_intv, 4, 1, fp) == 1 && fwrite(&seq_len, 4, 1, fp) == 1 &&
                 fwrite(smp, 4, n_samples, fp) == n_samples;
            ok = (fclose(fp) == 0) && ok;
        }
    }
    if (!ok) gs_set_error("cannot write %s", fn);
    free(fn);
    return ok ? GS_OK : GS_EIO;
}

static int build(const uint8_t *codes, uint64_t n, uint32_t sa_intv, int device, const char *prefix,
                 gs_index **out)
{
    GS_ON_DEVICE(device);
    GsBuilt o;
    int rc = build_device(codes, n, sa_intv, o);   /* its sort buffers are freed on return */
    if (rc == GS_OK && prefix) {
        uint32_t *bwt = NULL, *smp = NULL;
        uint64_t words = 0;
        rc = download(o, n, &bwt, &words, &smp);
        if (rc == GS_OK)
            rc = write_files(prefix, o.primary, o.L2, bwt, words, sa_intv, (uint32_t)n, smp, o.n_samples);
        free(bwt);
        free(smp);
    }
    if (rc == GS_OK && out)
        rc = gs_index_from_device(o.primary, o.L2, o.d_occ, sa_intv, o.d_smp, o.n_samples, device, out);
    return rc;
}

extern "C" int gs_index_build(const uint8_t *codes, uint64_t n, uint32_t sa_intv, int device,
                              const char *prefix, gs_index **out)
{
    if (!codes || n == 0 || n >= 0xfffffffeull || sa_intv == 0 || (!prefix && !out)) {
        gs_set_error("gs_index_build: need 1 <= n < 2^32-1 codes, sa_intv > 0 and an output");
        return GS_EINVAL;
    }
    const int rc = build(codes, n, sa_intv, device, prefix, out);
    /* the device looks at the codes; a failure of any kind is put down to a
     * bad one first */
    for (uint64_t i = 0; rc != GS_OK && i < n; i++)
        if (codes[i] > 3) {
            gs_set_error("gs_index_build: code %u at %llu is not 0..3", codes[i], (unsigned long long)i);
            return GS_EINVAL;
        }
    return rc;
}
