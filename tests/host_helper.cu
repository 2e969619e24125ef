// Host-side pieces of the library for tests that run without a GPU.

// A handle without tables that claims to live on device `device`: the entry points have to refuse it before they touch anything.
#include "../apr-cnn_b200/csrc/apr_device.cuh"

extern "C" aprnet_apr* fake_handle(int device) {
    aprnet_apr* a = new aprnet_apr();
    a->device = device;
    a->meta = LevelMeta();
    a->meta.level_min = 1; a->meta.level_max = 2;
    for (int l = 0; l < APRNET_MAX_LEVELS; ++l) a->meta.z_num[l] = a->meta.x_num[l] = a->meta.y_num[l] = 1;
    for (int l = 0; l <= APRNET_MAX_LEVELS; ++l) { a->meta.lvl_begin[l] = l < 2 ? 0 : 8 * (l - 1); a->meta.tlvl_begin[l] = l; }
    a->n_particles = 16; a->n_tree = 2;
    a->plans[0].n = 16; a->plans[0].tree_size = 2;          // "cached", so that nothing that would check builds them
    a->edge_plans[0]; a->run_plans[0];
    return a;
}

// passes over a chunk map whose largest chunks are as large as the plan makes them, with the workspace the library asks for: the largest
// number of rows of one pass minus what the workspace holds (> 0: refused)
extern "C" long long vrow_worst_pass(long long n_vrows, long long row_bytes) {
    std::vector<long long> v;
    for (long long k = 0; k * APRNET_VROW_GRANULE < n_vrows; ++k) v.push_back(std::min(n_vrows, k ? k * APRNET_VROW_GRANULE + 26 * (k & 1) : 0));
    if (v.empty() || v.back() != n_vrows) v.push_back(n_vrows);
    const long long cap = aprnet_vrow_workspace_bytes(n_vrows, row_bytes) / row_bytes - 1;      // (the rows start at a multiple of a row)
    long long worst = 0, seen = 0;
    const int nk = (int) v.size() - 1;
    for (int k0 = 0, k1; k0 < nk; k0 = k1) {
        k1 = aprnet_vrow_pass_end(v, k0, cap);
        worst = std::max(worst, v[k1] - v[k0]);
        seen += v[k1] - v[k0];
    }
    return seen == n_vrows ? worst - cap : 1ll << 60;
}
extern "C" void set_vrows(aprnet_apr* a, long long n) { a->edge_plans[0].n_vrows = n; }
extern "C" void set_particles(aprnet_apr* a, long long n) { for (int l = 3; l <= APRNET_MAX_LEVELS; ++l) a->meta.lvl_begin[l] = n; }
extern "C" long long vrow_chunk() { return APRNET_VROW_CHUNK; }

extern "C" int rows_overflow(aprnet_apr* a, long long particles, long long nodes) {
    const LevelMeta kept = a->meta;
    for (int l = 2; l <= APRNET_MAX_LEVELS; ++l) { a->meta.lvl_begin[l] = particles; a->meta.tlvl_begin[l] = nodes; }
    const int over = aprnet_rows_overflow(a, 0);
    a->meta = kept;
    return over;
}

extern "C" int f32_few_blocks(int tile_channels, int forward) { return aprnet_f32_few_blocks(tile_channels, forward != 0); }
extern "C" int run_max_height(int nt) { return aprnet_run_max_height(nt); }
extern "C" int f32_many_blocks(int tile_channels, int source_channels, long long blocks) { return aprnet_f32_many_blocks(tile_channels, source_channels, blocks); }
