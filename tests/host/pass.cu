/*
 * pass.cu -- the host code of the seeding context (gs_api.cu) and the serving
 * loop (gs_server.cu) on the fake runtime.
 * The launchers here stand for the kernels: they count slots and work items
 * as those do, raise the overflow flag where a batch does not fit, and
 * give each read the seeds and positions that the test asks for.
 */
#include "../../gpuseed_gb300/csrc/gs_api.cu"
#include "../../gpuseed_gb300/csrc/gs_server.cu"

#include "fake_cuda.h"

struct gs_index {
    GsDevIndex dev;
};

/* the last pass's sizes, for the test */
struct FakePass {
    uint64_t passes, n_items, item_cap, item_read_cap, slot_cap, walker_cap, clear_words, mask_words, items, slots;
    uint64_t seeds_a_read, pos_a_read;
};
static FakePass pass;
static gs_index the_index;

const GsDevIndex *gs_index_dev(const gs_index *idx) { return &idx->dev; }
int gs_index_device(const gs_index *) { return 0; }
uint32_t gs_index_generation(const gs_index *) { return 0; }
float gs_index_l2_ratio(const gs_index *) { return 0.f; }
size_t gs_index_occ_bytes(const gs_index *) { return 0; }

int gs_launch_prepare(const GsDevIndex &I, GsBatch &b, int kernel, cudaStream_t)
{
    const int kt = gs_paired_len(I, kernel, b.k);
    b.paired = kt != 0;
    uint64_t slots = 0, items = 0;
    for (uint32_t r = 0; r < b.n_reads; r++) {
        uint32_t s, i;
        gs_read_counts(b.lengths[r], b.k, kt, s, i);
        slots += s;
        items += i;
    }
    pass.slots = slots;
    pass.items = items;
    if (b.clear) {
        fake_set(b.queue, 0, 32);
        fake_set(b.recmask, 0, b.clear_words * 4);
    }
    pass.clear_words = b.clear ? b.clear_words : 0;
    b.totals[0] = b.h_totals[0] = slots;
    b.totals[1] = b.h_totals[1] = items;
    return GS_OK;
}

int gs_launch_search(const GsDevIndex &, GsBatch &b, int, int, int, uint32_t n_items, cudaStream_t)
{
    pass.passes++;
    pass.n_items = n_items;
    pass.item_cap = b.item_cap;
    pass.item_read_cap = b.item_read_cap;
    pass.slot_cap = b.slot_cap;
    pass.walker_cap = b.walker_cap;
    pass.mask_words = fake_room(b.recmask) / 4;
    if (pass.items > b.item_read_cap || pass.slots > b.slot_cap) b.queue[1] |= GS_FLAG_OVERFLOW;
    /* as many walkers as there is room for, where a warp had 16 an item */
    const uint64_t walkers = pass.items * 16u;
    b.queue[2] = (uint32_t)(walkers < b.walker_cap ? walkers : b.walker_cap);
    if (b.slots && b.slot_cap * sizeof(GsRec) > fake_room(b.slots)) fake_bad++;
    if (b.recmask && (b.slot_cap + 31) / 32 > pass.mask_words) fake_bad++;
    return GS_OK;
}

int gs_launch_finalize_count(const GsDevIndex &, GsBatch &b, cudaStream_t)
{
    b.totals[2] = b.h_totals[2] = pass.seeds_a_read * b.n_reads;
    b.totals[3] = b.h_totals[3] = pass.pos_a_read * b.n_reads;
    return GS_OK;
}

int gs_launch_finalize_emit(const GsDevIndex &, GsBatch &b, cudaStream_t)
{
    if (b.seed_cap * sizeof(gs_seed_rec) > fake_room(b.seeds) || b.seed_cap * 8 > fake_room(b.seed_pos)) fake_bad++;
    return GS_OK;
}

int gs_launch_locate(const GsDevIndex &, GsBatch &b, uint64_t, cudaStream_t)
{
    if (b.pos_cap * 4 > fake_room(b.pos) || b.pos_cap * 4 > fake_room(b.pmap)) fake_bad++;
    return GS_OK;
}

int gs_launch_text_lengths(const GsTextArgs &, cudaStream_t) { return GS_OK; }
int gs_launch_text_write(const GsTextArgs &, cudaStream_t) { return GS_OK; }

static void fake_kernel(const std::string &name, void **args)
{
    if (name.find("gs_copy_out_kernel") != std::string::npos) {
        const GsBatch &B = *(const GsBatch *)args[0];
        memcpy(*(uint32_t **)args[7], B.queue, 32);
    } else if (name.find("gs_fetch_small_kernel") != std::string::npos) {
        memcpy(*(uint32_t **)args[0], *(const uint32_t **)args[1], 4u * *(uint32_t *)args[2]);
    } else if (name.find("gs_max_end_kernel") != std::string::npos) {
        const uint64_t *off = *(const uint64_t **)args[0];
        const uint32_t *len = *(const uint32_t **)args[1], n = *(uint32_t *)args[2];
        unsigned long long *out = *(unsigned long long **)args[3];
        for (uint32_t r = 0; r < n; r++)
            if (off[r] + len[r] > out[0]) out[0] = off[r] + len[r];
    }
}

extern "C" {
/* whether a pass captured now would be replayed once buffer `which`, where it
 * lies, has room for 100 entries more; -1: there is no such buffer */
int fake_replayed_when_larger(gs_ctx *c, int which)
{
    size_t *const cap[] = {&c->cap_slots, &c->cap_item_read, &c->cap_recmask, &c->cap_walkers, &c->cap_seeds,
                           &c->cap_seed_pos, &c->cap_pos, &c->cap_pmap, &c->cap_tile_seed};
    if (which >= (int)(sizeof(cap) / sizeof(cap[0]))) return -1;
    *cap[which] += 100;
    const int same = same_graph(c, c->g_seqs, c->g_offs, c->g_lens, c->g_n, &c->g_params);
    *cap[which] -= 100;
    return same;
}

FakePass *fake_pass(void) { return &pass; }
gs_index *fake_index(void)
{
    static const uint4 start_table = {0, 0, 0, 0};   /* there is one; nothing reads it */
    the_index.dev.seq_len = 1000000;
    the_index.dev.kmerx = &start_table;
    the_index.dev.kx = 13;
    return &the_index;
}
}
