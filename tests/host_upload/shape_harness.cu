/*
 * shape_harness.cu -- TEST INFRASTRUCTURE ONLY.
 *
 * harness.cu with the default kernel shape and the step kernel's form in
 * sight, for tests/test_kernel_shape_host.py.
 */
#include "harness.cu"

HU_API int hs_create(int block_size, fn_ctx** out) {
    fn_config cfg = {0, 64, 64, 1, 0, block_size, 0, 0.0, 1};
    return fn_create(&cfg, out);
}
/* 0 one thread per bead, 1 staged, 2 five warps per 28 beads */
HU_API int hs_form(fn_ctx* c) { return c->staged ? 1 : c->wide ? 2 : 0; }
HU_API int hs_set_shape(fn_ctx* c, int block, int items) { return fn_set_kernel_shape(c, block, items); }
HU_API void hs_shape(fn_ctx* c, int* block_items2) {
    fn_stats st;
    fn_get_stats(c, &st);
    block_items2[0] = st.block_size;
    block_items2[1] = st.items_per_thread;
}
