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
