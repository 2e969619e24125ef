// Drivers of the 3x3x3 convolution over packed rows (float32 tensors), in either arithmetic: exact fp32 on the CUDA cores
// (conv333_f32.cu) or bf16 operands with fp32 accumulation on the tensor cores (conv333_tc.cu, conv333_tc_dw.cu, edge_plan.cu).
//
// forward:   tree means of the input -> packed rows (particles, tree means, zero row) at the start of the workspace -> gather
//            product with the level's stencils.
// backward:  from the packed rows that the forward call left (nothing of the fp32 input is needed): packed rows of grad_output
//            -> weight gradient -> same-level input gradient -> cross-level part -> tree adjoint.
// For Cin <= 4 the rows area holds an fp32 channel-major copy instead (conv333_small.cu), in both arithmetics.
// Reference: pyapr/aprnet/src/conv.hpp:83-195 (forward), :289-481 (backward).
#include "apr_device.cuh"
#include <algorithm>

typedef long long ll;

int aprnet_tc_pack_rows(const float* x, ll ld_x, ll n, const float* tree, ll ld_tree, ll t, int c, int cpad, void* out, cudaStream_t st);
int aprnet_tc_pack_rows_pair(const float* x0, ll ld0, int c0, const float* x1, ll ld1, ll n, const float* tree, ll ld_tree, ll t, int c, int cpad, void* out, cudaStream_t st);
int aprnet_tc_pack_rows_sums(const float* x, ll ld_x, ll n, int c, int cpad, void* out, double* sums, float* sums_out, cudaStream_t st);
size_t aprnet_tc_pack_sums_bytes(int c);
int aprnet_f32_pack_pair(const aprnet_apr* a, int dl, int cin, const float* in0, ll ld0, int c0, const float* in1, ll ld1, const float* tree, ll ld_tree, void* rows, cudaStream_t st);
int aprnet_fill_tree_mean_pair(const aprnet_apr* a, int dl, int C, const float* in0, ll ld0, int c0, const float* in1, ll ld1, float* tree, ll ld_tree, cudaStream_t st);
int aprnet_tc_gather_conv(aprnet_apr* a, int dl, int backward, int cin, int cout, int slots, const void* rows, int kpad,
                          ll tree_base, ll zero_row, const float* w, void* wp_ws, const float* bias, float* out, ll ld_out, cudaStream_t st);

namespace {

inline bool is_bf16(int precision) { return precision == APRNET_PREC_BF16; }

size_t grad_bytes(const aprnet_apr* a, int dl, int precision, int cin, int cout, int slots) {
    if (!is_bf16(precision)) return aprnet_f32_backward_bytes(a, dl, cin, cout, slots);
    return aprnet_tc_rows_bytes(a->number_parts(dl) + 1, cout) + aprnet_tc_weight_bytes(cout, cin, slots) + (size_t) aprnet_edge_workspace_bytes(a, dl, cout);
}

int pack_input(const aprnet_apr* a, int dl, int precision, int cin, const float* in, ll ld_in, const float* tree, ll ld_tree, void* rows, cudaStream_t st) {
    const ll n = a->number_parts(dl), t = a->tree_size(dl);
    if (aprnet_small_cin(cin)) return aprnet_small_stage(in, ld_in, n, tree, ld_tree, t, cin, (float*) rows, st);
    return is_bf16(precision) ? aprnet_tc_pack_rows(in, ld_in, n, tree, ld_tree, t, cin, aprnet_tc_pad(cin), rows, st)
                              : aprnet_f32_pack_input(a, dl, cin, in, ld_in, tree, ld_tree, rows, st);
}

// forward product from the packed rows at the start of `workspace`
int product(aprnet_apr* a, int dl, int precision, int cin, int cout, int slots, const float* w, const float* bias, float* out, ll ld_out, void* workspace, cudaStream_t st) {
    if (!is_bf16(precision) || aprnet_small_cin(cin)) return aprnet_f32_forward(a, dl, cin, cout, slots, w, bias, out, ld_out, workspace, st);
    const ll n = a->number_parts(dl), t = a->tree_size(dl);
    void* wp = (char*) workspace + aprnet_tc_rows_bytes(n + t + 1, cin);
    return aprnet_tc_gather_conv(a, dl, 0, cin, cout, slots, workspace, aprnet_tc_pad(cin), n, n + t, w, wp, bias, out, ld_out, st);
}

int forward_rows(aprnet_apr* a, int dl, int precision, int cin, int cout, int slots, const float* in, ll ld_in, const float* w, const float* bias,
                 float* out, ll ld_out, float* tree, ll ld_tree, bool tree_valid, void* workspace, cudaStream_t st) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && cin > 0 && cout > 0 && slots > 0 && in && w && out && tree && workspace, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_out >= a->number_parts(dl) && ld_tree >= a->tree_size(dl), "leading dimension too small");
    int rc = tree_valid ? APRNET_OK : aprnet_fill_tree_mean_forward(a, dl, APRNET_F32, cin, in, ld_in, tree, ld_tree, st);
    if (rc) return rc;
    if ((rc = pack_input(a, dl, precision, cin, in, ld_in, tree, ld_tree, workspace, st))) return rc;
    return product(a, dl, precision, cin, cout, slots, w, bias, out, ld_out, workspace, st);
}

// `ws`: grad_bytes() bytes.  gout == null: `ws` starts with the packed rows of grad_output already (bf16, Cin > 4).  gin == null: no input gradient; gw == null: no weight gradient; fold_tree: grad_tree is folded into gin
int backward_rows(aprnet_apr* a, int dl, int precision, int cin, int cout, int slots, const void* rows, const float* gout, ll ld_out, const float* w,
                  float* gin, ll ld_in, float* gw, int accumulate, float* gtree, ll ld_tree, float* partial, void* ws, bool fold_tree, cudaStream_t st, float* gbias = nullptr) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && cin > 0 && cout > 0 && slots > 0 && (gout || (is_bf16(precision) && !aprnet_small_cin(cin) && 27 * a->number_parts(dl) + 1 < (1ll << 31))) && (gin || gw) && (!gin || (w && gtree)) && ws && (!gw || (rows && partial)), "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_out >= a->number_parts(dl) && (!gin || (ld_in >= a->number_parts(dl) && ld_tree >= a->tree_size(dl))), "leading dimension too small");
    const ll n = a->number_parts(dl);
    const int gpad = aprnet_tc_pad(cout);
    const bool bf16 = is_bf16(precision);
    int rc;
    // the weight gradient of a first layer reads grad_output itself
    if (gout && (gin || !aprnet_small_cin(cin))) {
        // (the sums' buffer is the weight gradient's, which comes afterwards)
        rc = gbias ? aprnet_tc_pack_rows_sums(gout, ld_out, n, cout, gpad, ws, (double*) partial, gbias, st)
           : bf16 ? aprnet_tc_pack_rows(gout, ld_out, n, nullptr, 0, 0, cout, gpad, ws, st) : aprnet_f32_pack_grad(a, dl, cout, gout, ld_out, ws, st);
        if (rc) return rc;
    }
    if (gw) {
        rc = bf16 && !aprnet_small_cin(cin) ? aprnet_tc_backward_weights(a, dl, cin, cout, slots, rows, aprnet_tc_pad(cin), ws, gpad, gw, accumulate, partial, st)
                                            : aprnet_f32_backward_weights(a, dl, cin, cout, slots, rows, gout, ld_out, ws, gw, accumulate, partial, st);
        if (rc) return rc;
    }
    if (!gin) return APRNET_OK;
    if (!bf16) return aprnet_f32_backward_input(a, dl, cin, cout, slots, gout, ld_out, w, gin, ld_in, gtree, ld_tree, ws, fold_tree, st);
    void* wp = (char*) ws + aprnet_tc_rows_bytes(n + 1, cout);
    if ((rc = aprnet_tc_gather_conv(a, dl, 1, cin, cout, slots, ws, gpad, n, n, w, wp, nullptr, gin, ld_in, st))) return rc;
    void* edge_ws = (char*) wp + aprnet_tc_weight_bytes(cout, cin, slots);
    if (27 * n + 1 >= (1ll << 31)) {
        // more than 79.5 M locations: the 32-bit edge ids of the edge plan run out.  The cross-level part then runs on the
        // fp32 scatter kernel (atomic adds: correct, but the summation order is no longer fixed).
        if (!fold_tree) { aprnet_set_error("the split backward form needs the edge plan, which supports up to 79.5 M locations"); return APRNET_ERR_UNSUPPORTED; }
        return aprnet_conv333_backward_input_cross_level(a, dl, APRNET_F32, cin, cout, slots, gout, ld_out, w, gin, ld_in, gtree, ld_tree, st);
    }
    return aprnet_cross_level_tc(a, dl, cin, cout, slots, ws, gpad, w, gin, ld_in, gtree, ld_tree, wp, edge_ws,
                                 aprnet_edge_workspace_bytes(a, dl, cout), st, fold_tree);
}

inline bool precision_ok(int precision) { return precision == APRNET_PREC_F32 || precision == APRNET_PREC_BF16; }

} // namespace

// ---- either arithmetic --------------------------------------------------------------------------------
extern "C" int64_t aprnet_conv333_rows_bytes(const aprnet_apr* a, int dl, int precision, int cin) {
    if (!a || !a->valid_dl(dl) || cin <= 0 || !precision_ok(precision)) return -1;
    const ll rows = a->number_parts(dl) + a->tree_size(dl) + 1;
    return (int64_t) (is_bf16(precision) && !aprnet_small_cin(cin) ? aprnet_tc_rows_bytes(rows, cin) : aprnet_f32_rows_bytes(a, dl, cin));
}

extern "C" int64_t aprnet_conv333_rows_forward_workspace_bytes(const aprnet_apr* a, int dl, int precision, int cin, int cout, int slots) {
    if (!a || !a->valid_dl(dl) || cin <= 0 || cout <= 0 || !precision_ok(precision)) return -1;
    if (is_bf16(precision) && !aprnet_small_cin(cin)) return aprnet_conv333_tc_forward_workspace_bytes(a, dl, cin, cout, slots);
    return (int64_t) aprnet_f32_forward_bytes(a, dl, cin, cout, slots);
}

extern "C" int64_t aprnet_conv333_rows_backward_workspace_bytes(const aprnet_apr* a, int dl, int precision, int cin, int cout, int slots, int with_grad_input) {
    if (!a || !a->valid_dl(dl) || cin <= 0 || cout <= 0 || !precision_ok(precision)) return -1;
    if (with_grad_input) return (int64_t) grad_bytes(a, dl, precision, cin, cout, slots);
    if (aprnet_small_cin(cin)) return 256;
    const ll rows = a->number_parts(dl) + 1;
    return (int64_t) (is_bf16(precision) ? aprnet_tc_rows_bytes(rows, cout) : (size_t) rows * ((cout + 3) / 4 * 4) * sizeof(float));
}

extern "C" int64_t aprnet_conv333_rows_partial_elems(int precision, int cin, int cout) {
    if (cin <= 0 || cout <= 0 || !precision_ok(precision)) return -1;
    return is_bf16(precision) ? aprnet_conv333_tc_dw_partial_elems(cin, cout) : aprnet_f32_partial_elems(cin, cout);
}

extern "C" int aprnet_conv333_rows_forward(aprnet_apr* a, int dl, int precision, int cin, int cout, int slots, const float* in, int64_t ld_in, const float* w,
                                           const float* bias, float* out, int64_t ld_out, float* tree, int64_t ld_tree, int tree_is_valid, void* workspace, void* stream) {
    APRNET_ARG_CHECK(precision_ok(precision), "unknown precision");
    return forward_rows(a, dl, precision, cin, cout, slots, in, ld_in, w, bias, out, ld_out, tree, ld_tree, tree_is_valid != 0, workspace, (cudaStream_t) stream);
}

// Forward pass over the concatenation of two tensors of cin0 and cin - cin0 channels, which is never written out: tree means and packed rows are made from both.
extern "C" int aprnet_conv333_rows_forward_pair(aprnet_apr* a, int dl, int precision, int cin, int cout, int slots, const float* in0, int64_t ld0, int cin0, const float* in1, int64_t ld1,
                                                const float* w, const float* bias, float* out, int64_t ld_out, float* tree, int64_t ld_tree, void* workspace, void* stream) {
    APRNET_ARG_CHECK(precision_ok(precision), "unknown precision");
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && cin > 0 && cout > 0 && slots > 0 && in0 && in1 && w && out && tree && workspace, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(cin0 > 0 && cin0 < cin && cin0 % 4 == 0 && !aprnet_small_cin(cin), "the first tensor's channels must be a multiple of four, both together more than four");
    const ll n = a->number_parts(dl), t = a->tree_size(dl);
    APRNET_ARG_CHECK(ld0 >= n && ld1 >= n && ld_out >= n && ld_tree >= t, "leading dimension too small");
    cudaStream_t st = (cudaStream_t) stream;
    int rc = aprnet_fill_tree_mean_pair(a, dl, cin, in0, ld0, cin0, in1, ld1, tree, ld_tree, st);
    if (rc) return rc;
    rc = is_bf16(precision) ? aprnet_tc_pack_rows_pair(in0, ld0, cin0, in1, ld1, n, tree, ld_tree, t, cin, aprnet_tc_pad(cin), workspace, st)
                            : aprnet_f32_pack_pair(a, dl, cin, in0, ld0, cin0, in1, ld1, tree, ld_tree, workspace, st);
    return rc ? rc : product(a, dl, precision, cin, cout, slots, w, bias, out, ld_out, workspace, st);
}

extern "C" int aprnet_conv333_rows_pack(aprnet_apr* a, int dl, int precision, int cin, const float* in, int64_t ld_in, float* tree, int64_t ld_tree, int tree_is_valid,
                                        void* rows, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && cin > 0 && in && tree && rows && precision_ok(precision), "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_tree >= a->tree_size(dl), "leading dimension too small");
    const int rc = tree_is_valid ? APRNET_OK : aprnet_fill_tree_mean_forward(a, dl, APRNET_F32, cin, in, ld_in, tree, ld_tree, stream);
    return rc ? rc : pack_input(a, dl, precision, cin, in, ld_in, tree, ld_tree, rows, (cudaStream_t) stream);
}

extern "C" int aprnet_conv333_rows_backward(aprnet_apr* a, int dl, int precision, int cin, int cout, int slots, const void* rows, const float* gout, int64_t ld_out,
                                            const float* w, float* gin, int64_t ld_in, float* gw, int accumulate, float* gtree, int64_t ld_tree, int fold_tree,
                                            float* partial, void* workspace, void* stream) {
    APRNET_ARG_CHECK(precision_ok(precision), "unknown precision");
    APRNET_ARG_CHECK(gout, "bad argument");
    return backward_rows(a, dl, precision, cin, cout, slots, rows, gout, ld_out, w, gin, ld_in, gw, accumulate, gtree, ld_tree, partial, workspace, fold_tree != 0, (cudaStream_t) stream);
}

// The backward pass in bf16 arithmetic (cin > 4) with the sums of grad_output over the structure's locations, the gradient of a bias, in grad_bias (cout): taken along where
// grad_output is packed.  partial: aligned to 8 bytes
extern "C" int aprnet_conv333_rows_backward_bias(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* rows, const float* gout, int64_t ld_out, const float* w,
                                                 float* gin, int64_t ld_in, float* gw, float* gtree, int64_t ld_tree, float* gbias, float* partial, void* workspace, void* stream) {
    APRNET_ARG_CHECK(gout && gw && gbias && partial && (reinterpret_cast<uintptr_t>(partial) & 7) == 0 && cin > 0 && !aprnet_small_cin(cin) && cout > 0, "bad argument");
    if (aprnet_tc_pack_sums_bytes(cout) > (size_t) aprnet_conv333_tc_dw_partial_elems(cin, cout) * sizeof(float)) { aprnet_set_error("%s: the weight gradient's buffer is too small for the sums", __func__); return APRNET_ERR_UNSUPPORTED; }
    return backward_rows(a, dl, APRNET_PREC_BF16, cin, cout, slots, rows, gout, ld_out, w, gin, ld_in, gw, 0, gtree, ld_tree, partial, workspace, true, (cudaStream_t) stream, gbias);
}

// ---- the tensor-core entry points ------------------------------------------------------------------------
// forward: out = conv(in) with bf16 operands / fp32 accumulation; tree_scratch receives the fp32 tree means
extern "C" int aprnet_conv333_forward_tc(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* in, int64_t ld_in,
                                         const float* w, float* out, int64_t ld_out, float* tree, int64_t ld_tree,
                                         void* workspace, void* stream) {
    return forward_rows(a, dl, APRNET_PREC_BF16, cin, cout, slots, in, ld_in, w, nullptr, out, ld_out, tree, ld_tree, false, workspace, (cudaStream_t) stream);
}

// Split form (see aprnet_conv333_forward_pretree): the tree means are taken as given.
extern "C" int aprnet_conv333_forward_tc_pretree(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* in, int64_t ld_in,
                                                 const float* w, float* out, int64_t ld_out, const float* tree, int64_t ld_tree,
                                                 void* workspace, void* stream) {
    return forward_rows(a, dl, APRNET_PREC_BF16, cin, cout, slots, in, ld_in, w, nullptr, out, ld_out, const_cast<float*>(tree), ld_tree, true, workspace, (cudaStream_t) stream);
}

extern "C" int64_t aprnet_conv333_tc_packed_rows_bytes(const aprnet_apr* a, int dl, int cin) {
    if (!a || !a->valid_dl(dl)) return -1;
    return (int64_t) aprnet_tc_rows_bytes(a->number_parts(dl) + a->tree_size(dl) + 1, cin);
}

// workspace: aprnet_conv333_tc_workspace_bytes() bytes; its leading part (packed input rows) is not touched, so the forward
// workspace itself may be passed as packed_input_rows
static void* grad_area(const aprnet_apr* a, int dl, int cin, void* workspace) {
    return workspace && a && a->valid_dl(dl) ? (char*) workspace + aprnet_tc_rows_bytes(a->number_parts(dl) + a->tree_size(dl) + 1, cin) : nullptr;
}

extern "C" int aprnet_conv333_backward_tc_rows(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* packed_input_rows,
                                               const float* gout, int64_t ld_out, const float* w, float* gin, int64_t ld_in, float* gw,
                                               float* gtree, int64_t ld_tree, float* partial, void* workspace, void* stream) {
    APRNET_ARG_CHECK(gw && gout, "bad argument");
    return backward_rows(a, dl, APRNET_PREC_BF16, cin, cout, slots, packed_input_rows, gout, ld_out, w, gin, ld_in, gw, 1, gtree, ld_tree, partial,
                         grad_area(a, dl, cin, workspace), true, (cudaStream_t) stream);
}

// Split form: grad_input holds the direct contributions only and grad_tree the gradient of the tree means; the
// caller folds them with aprnet_fill_tree_mean_backward after it has exchanged the halo parts.
extern "C" int aprnet_conv333_backward_tc_rows_pretree(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* packed_input_rows,
                                                       const float* gout, int64_t ld_out, const float* w, float* gin, int64_t ld_in, float* gw,
                                                       float* gtree, int64_t ld_tree, float* partial, void* workspace, void* stream) {
    APRNET_ARG_CHECK(gw && gout, "bad argument");
    return backward_rows(a, dl, APRNET_PREC_BF16, cin, cout, slots, packed_input_rows, gout, ld_out, w, gin, ld_in, gw, 1, gtree, ld_tree, partial,
                         grad_area(a, dl, cin, workspace), false, (cudaStream_t) stream);
}

// Complete backward pass from the fp32 input: fills the tree means (unless tree_valid), packs the input
// rows into the workspace and continues as aprnet_conv333_backward_tc_rows.
extern "C" int aprnet_conv333_backward_tc(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* in, int64_t ld_in,
                                          const float* gout, int64_t ld_out, const float* w, float* gin, float* gw,
                                          float* tree, int tree_valid, float* gtree, int64_t ld_tree, float* partial,
                                          void* workspace, void* stream) {
    APRNET_ARG_CHECK(cout > 0 && slots > 0 && gout && w && gw && gtree && partial, "bad argument");
    const int rc = aprnet_conv333_rows_pack(a, dl, APRNET_PREC_BF16, cin, in, ld_in, tree, ld_tree, tree_valid, workspace, stream);
    if (rc) return rc;
    return aprnet_conv333_backward_tc_rows(a, dl, cin, cout, slots, workspace, gout, ld_out, w, gin, ld_in, gw, gtree, ld_tree, partial, workspace, stream);
}

// GroupNorm + ReLU and the convolution in front of it, backward in one call for one batch item (float32 tensors, bf16 arithmetic, Cin > 4): conv_out is the
// output of the convolution, n its row length; the gradient of it exists only as packed rows in `workspace`
// (aprnet_conv333_rows_backward_workspace_bytes()).  norm_ws: aprnet_groupnorm_workspace_bytes(1, cout, groups)
int aprnet_groupnorm_relu_backward_rows(int C, ll n, ll n_rows, int groups, const float* x, const float* dy, const float* gamma, const float* beta,
                                        const float* mean, const float* rstd, float* dgamma, float* dbeta, int cpad, void* rows_out, double* ws, int relu, cudaStream_t st);

extern "C" int aprnet_conv333_norm_backward(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* rows, const float* conv_out, int64_t n, int groups,
                                            const float* gamma, const float* beta, const float* mean, const float* rstd, int relu, const float* grad_y, const float* w,
                                            float* gin, int64_t ld_in, float* gw, float* gtree, int64_t ld_tree, float* dgamma, float* dbeta, float* partial,
                                            void* workspace, void* norm_ws, void* stream) {
    // all of it before the first launch, which overwrites grad_gamma, grad_beta and the workspace
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && cin > 0 && cout > 0 && slots > 0 && !aprnet_small_cin(cin) && rows && conv_out && n > 0 && groups > 0 && cout % groups == 0 &&
                     mean && rstd && grad_y && gw && (!gin || (w && gtree)) && dgamma && dbeta && partial && workspace && norm_ws, "bad argument");
    APRNET_ARG_CHECK(((reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(workspace)) & 15) == 0, "packed rows and workspace must be 16-byte aligned");
    const ll parts = a->number_parts(dl);
    APRNET_ARG_CHECK(n >= parts && (!gin || (ld_in >= parts && ld_tree >= a->tree_size(dl))), "leading dimension too small");
    if (27 * parts + 1 >= (1ll << 31)) { aprnet_set_error("%s: supports up to 79.5 M locations", __func__); return APRNET_ERR_UNSUPPORTED; }
    APRNET_DEVICE_CHECK(a);
    cudaStream_t st = (cudaStream_t) stream;
    const int rc = aprnet_groupnorm_relu_backward_rows(cout, n, a->number_parts(dl), groups, conv_out, grad_y, gamma, beta, mean, rstd, dgamma, dbeta,
                                                       aprnet_tc_pad(cout), workspace, (double*) norm_ws, relu, st);
    if (rc) return rc;
    return backward_rows(a, dl, APRNET_PREC_BF16, cin, cout, slots, rows, nullptr, n, w, gin, ld_in, gw, 0, gtree, ld_tree, partial, workspace, true, st);
}
