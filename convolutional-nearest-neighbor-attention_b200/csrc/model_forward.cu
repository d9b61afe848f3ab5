// The whole ViT forward as one native call: the chain of entry points that vit.py issues one binding call at a
// time, over one workspace.  No kernel of its own.
//
// Why: at batch sizes up to ~100 images a ViT-Tiny forward was bound by the host, 1.14 ms per forward for 64
// launches, of which the library's own share was a fifth; the rest was argument handling, allocation of the
// intermediates and shape logic in Python between them.
#include "common.cuh"

using namespace convnn;

namespace {

size_t up(size_t n) { return (n + 255) & ~(size_t)255; }
size_t most(size_t a, size_t b) { return a > b ? a : b; }

// Buffers of one forward.  x and x1 alternate as the rows between blocks (block input in x, after the attention
// layer in x1, block output in x again); everything in `scratch` lives inside one phase (embedding, attention, MLP).
struct Plan {
    size_t x, x1, mom, mom1, scratch, total;      // byte offsets into the workspace
    size_t cols, proj;                             // embedding phase, offsets into scratch
    size_t xn, cat, layer_ws, h;                   // block phases
    size_t other_ws, least;                        // the other half's own workspace, if it is to run beside; bytes without it
};

int planes_of(int D) {
    return (int)most((size_t)convnn_b200_moment_planes(D), (size_t)convnn_b200_prenorm_mlp_moment_planes());
}

bool plan_of(const convnn_model* m, Plan* p) {
    const size_t elt = m->dtype == CONVNN_F32 ? 4 : 2;
    const size_t rows = (size_t)m->B * m->T, row_bytes = up(rows * m->D * elt);
    const size_t patches = (size_t)m->B * (m->T - 1);
    size_t off = 0;
    auto take = [&](size_t n) { const size_t r = off; off += up(n); return r; };
    size_t h = 0, layer = 0, other = 0, cat = 0, planes = 1;
    for (int i = 0; i < m->n_blocks; ++i) {
        const convnn_block& b = m->blocks[i];
        const size_t ws = convnn_b200_workspace_bytes(&b.layer);
        if (ws == 0) return false;
        layer = most(layer, ws);
        const int rest = m->D - b.layer.D;
        if (b.kind == CONVNN_BLOCK_BRANCH_ATTENTION)
            other = most(other, convnn_b200_attention_workspace_bytes(m->dtype, m->B, m->T, rest));
        else if (b.kind == CONVNN_BLOCK_BRANCH_CONV1D)
            other = most(other, convnn_b200_conv1d_attention_workspace_bytes(m->dtype, m->B, m->T, rest, b.kernel_size));
        if (b.kind != CONVNN_BLOCK_CONVNN) cat = row_bytes;
        h = most(h, rows * (size_t)b.d_mlp * elt);
        planes = most(planes, (size_t)planes_of(m->D));
    }
    const size_t mom = planes * (size_t)convnn_b200_moment_stride((int64_t)rows) * 8;
    p->x = take(row_bytes);
    p->x1 = take(row_bytes);
    p->mom = take(mom);
    p->mom1 = take(mom);
    p->scratch = off;
    p->cols = 0;
    p->proj = up(patches * (size_t)m->channels * m->patch * m->patch * elt);
    const size_t embed = p->proj + up(patches * m->D * elt);
    p->xn = 0;
    p->cat = row_bytes;
    p->layer_ws = row_bytes + cat;
    p->h = row_bytes;
    p->least = off + most(embed, most(p->layer_ws + up(most(layer, other)), p->h + up(h)));
    p->other_ws = p->layer_ws + up(layer);
    // (float32 kernels are started one after the other whatever the order: nothing to run beside)
    p->total = m->dtype == CONVNN_BF16 ? most(p->least, off + p->other_ws + up(other)) : p->least;
    return true;
}

// Whether the other half's entry point would take these arguments (it reports what it refuses, stage() does not look).
bool half_ok(const convnn_block& b, const OtherHalf& h) {
    return h.D >= 1 && h.D % h.H == 0 && h.w_in && h.w_out && (!h.conv1d || (h.w_conv && b.kernel_size >= 1)) &&
           (long long)h.B * h.T * h.D < (1ll << 31);
}

// One encoder block (vit.py:262-269): rows in x, result in x again, the rows in between in x1.  `mom` / `planes`:
// moments of x, 0 planes where no kernel has produced them; on return those of the result (if `want_moments`).
int block_forward(const convnn_model* m, const convnn_block& b, char* ws, const Plan& p, bool beside, int* planes,
                  bool want_moments, void* stream) {
    const int64_t D = m->D, rows = (int64_t)m->B * m->T;
    const size_t elt = m->dtype == CONVNN_F32 ? 4 : 2;
    char *x = ws + p.x, *x1 = ws + p.x1, *scratch = ws + p.scratch;
    char *xn = scratch + p.xn, *layer_ws = scratch + p.layer_ws;
    const size_t layer_bytes = p.least - p.scratch - p.layer_ws;
    float *mom = reinterpret_cast<float*>(ws + p.mom), *mom1 = reinterpret_cast<float*>(ws + p.mom1);
    const bool fold_mlp = b.fc1_folded != nullptr;
    int planes1 = 0, rc;
    if (b.w_qkv_folded) {
        if (*planes == 0) {
            if ((rc = convnn_b200_row_moments(x, D, rows, (int32_t)D, mom, stream))) return rc;
            *planes = 1;
        }
        if ((rc = prenorm_forward(&b.layer, x, D, mom, *planes, b.eps1, b.w_qkv_folded, b.w_qkv_extra, b.w_conv, b.w_pw, b.w_o, x,
                                  D, x1, D, fold_mlp ? mom1 : nullptr, layer_ws, layer_bytes, true, stream)))
            return rc;
        if (fold_mlp) planes1 = convnn_b200_moment_planes((int32_t)D);
    } else {
        if ((rc = convnn_b200_layernorm(m->dtype, x, D, b.norm1_w, b.norm1_b, b.eps1, xn, D, rows, (int32_t)D, stream))) return rc;
        if (b.kind == CONVNN_BLOCK_CONVNN) {
            if ((rc = layer_forward(&b.layer, xn, D, b.w_qkv, b.w_conv, b.w_pw, b.w_o, b.cand, x, D, x1, D, layer_ws, layer_bytes,
                                    true, stream)))
                return rc;
        } else {
            // both branches read their channel slice of xn and write theirs of the concat buffer
            const int64_t dc = b.layer.D, rest = D - dc;
            char* cat = scratch + p.cat;
            const char* xr = xn + dc * elt;
            char* cr = cat + dc * elt;
            const bool conv1d = b.kind == CONVNN_BLOCK_BRANCH_CONV1D;
            const OtherHalf half{conv1d, xr, b.branch_w_in, conv1d ? b.branch_b_in : nullptr, b.branch_w_conv, b.branch_b_conv,
                                 b.branch_w_out, conv1d ? b.branch_b_out : nullptr, cr, scratch + p.other_ws, D, D, m->B, m->T,
                                 (int32_t)rest, b.layer.H, b.kernel_size, m->dtype};
            if ((rc = layer_forward(&b.layer, xn, D, b.w_qkv, b.w_conv, b.w_pw, b.w_o, b.cand, nullptr, 0, cat, D, layer_ws,
                                    layer_bytes, true, stream, beside && half_ok(b, half) ? &half : nullptr)))
                return rc;
            if (!(beside && half_ok(b, half))) rc = b.kind == CONVNN_BLOCK_BRANCH_ATTENTION
                     ? softmax_attention(m->dtype, xr, D, b.branch_w_in, b.branch_w_out, cr, D, m->B, m->T, (int32_t)rest,
                                         b.layer.H, layer_ws, layer_bytes, true, stream)
                     : conv1d_attention(m->dtype, xr, D, b.branch_w_in, b.branch_b_in, b.branch_w_conv, b.branch_b_conv,
                                        b.branch_w_out, b.branch_b_out, cr, D, m->B, m->T, (int32_t)rest, b.layer.H,
                                        b.kernel_size, layer_ws, layer_bytes, true, stream);
            if (rc) return rc;
            if ((rc = linear(m->dtype, cat, D, b.pointwise_w, b.pointwise_b, x, D, x1, D, rows, (int32_t)D, (int32_t)D, 0, true,
                             stream)))
                return rc;
        }
    }
    const int32_t dm = b.d_mlp;
    char* h = scratch + p.h;
    *planes = 0;
    if (fold_mlp) {
        if (planes1 == 0) {
            if ((rc = convnn_b200_row_moments(x1, D, rows, (int32_t)D, mom1, stream))) return rc;
            planes1 = 1;
        }
        if (b.fuse_mlp && convnn_b200_prenorm_mlp_supported((int32_t)D, dm, planes1)) {
            if (want_moments) *planes = convnn_b200_prenorm_mlp_moment_planes();
            return prenorm_mlp(x1, D, mom1, planes1, b.eps2, b.fc1_folded, b.fc1_extra, b.fc2_w, b.fc2_b, x, D, rows, (int32_t)D,
                               dm, want_moments ? mom : nullptr, true, stream);
        }
        if ((rc = prenorm_linear(x1, D, mom1, planes1, b.eps2, b.fc1_folded, b.fc1_extra, h, dm, rows, dm, (int32_t)D, 1, true,
                                 stream)))
            return rc;
    } else {
        if ((rc = convnn_b200_layernorm(m->dtype, x1, D, b.norm2_w, b.norm2_b, b.eps2, xn, D, rows, (int32_t)D, stream))) return rc;
        if ((rc = linear(m->dtype, xn, D, b.fc1_w, b.fc1_b, nullptr, 0, h, dm, rows, dm, (int32_t)D, 1, true, stream))) return rc;
    }
    if (want_moments && m->dtype == CONVNN_BF16) {
        *planes = convnn_b200_moment_planes((int32_t)D);
        return linear_moments(h, dm, b.fc2_w, b.fc2_b, x1, D, x, D, rows, (int32_t)D, dm, mom, true, stream);
    }
    return linear(m->dtype, h, dm, b.fc2_w, b.fc2_b, x1, D, x, D, rows, (int32_t)D, dm, 0, true, stream);
}

int check(const convnn_model* m) {
    if (!m || (m->n_blocks > 0 && !m->blocks)) return set_error(CONVNN_E_NULL, "model_forward: the model or its block list is NULL");
    if ((m->dtype != CONVNN_F32 && m->dtype != CONVNN_BF16) || m->B < 1 || m->T < 2 || m->D < 1 || m->n_blocks < 0 ||
        m->classes < 1 || m->channels < 1 || m->patch < 1 || m->height % m->patch != 0 || m->width % m->patch != 0 ||
        (m->height / m->patch) * (m->width / m->patch) + 1 != m->T)
        return set_error(CONVNN_E_INVALID, "model_forward: bad shape (B=%d T=%d D=%d, %d x %d images, patch %d)", m->B, m->T,
                         m->D, m->height, m->width, m->patch);
    for (int i = 0; i < m->n_blocks; ++i) {
        const convnn_block& b = m->blocks[i];
        const bool branch = b.kind == CONVNN_BLOCK_BRANCH_ATTENTION || b.kind == CONVNN_BLOCK_BRANCH_CONV1D;
        if ((!branch && b.kind != CONVNN_BLOCK_CONVNN) || b.layer.B != m->B || b.layer.T != m->T ||
            b.layer.dtype != m->dtype || (branch ? b.layer.D >= m->D : b.layer.D != m->D) || b.d_mlp < 1 ||
            (b.kind == CONVNN_BLOCK_BRANCH_CONV1D && b.kernel_size < 1))
            return set_error(CONVNN_E_INVALID, "model_forward: block %d does not fit the model", i);
    }
    return CONVNN_OK;
}

}  // namespace

extern "C" {

size_t convnn_b200_model_workspace_bytes(const convnn_model* m) {
    Plan p;
    if (check(m) || !plan_of(m, &p)) return 0;
    return p.total;
}

size_t convnn_b200_model_workspace_least_bytes(const convnn_model* m) {
    Plan p;
    if (check(m) || !plan_of(m, &p)) return 0;
    return p.least;
}

int convnn_b200_model_forward(const convnn_model* m, const void* images, void* logits, void* workspace,
                              size_t workspace_bytes, void* stream) {
    int rc = check(m);
    if (rc) return rc;
    if (!images || !logits || !workspace) return set_error(CONVNN_E_NULL, "model_forward: a buffer is NULL");
    if (!aligned16(workspace)) return set_error(CONVNN_E_ALIGN, "workspace must be 16-byte aligned");
    Plan p;
    if (!plan_of(m, &p)) return CONVNN_E_INVALID;                 // the layer's own message stands
    if (workspace_bytes < p.least)
        return set_error(CONVNN_E_WORKSPACE, "workspace has %zu bytes, %zu needed", workspace_bytes, p.least);
    const bool beside = p.total > p.least && workspace_bytes >= p.total;       // the halves of a block side by side
    char *ws = static_cast<char*>(workspace), *cols = ws + p.scratch + p.cols, *proj = ws + p.scratch + p.proj;
    const int32_t np = m->T - 1, pix = m->channels * m->patch * m->patch;
    if (m->images_u8)
        rc = convnn_b200_patchify_u8(m->dtype, static_cast<const uint8_t*>(images), m->pixel_mean, m->pixel_inv_std, cols, m->B,
                                     m->channels, m->height, m->width, m->patch, stream);
    else
        rc = convnn_b200_patchify(m->dtype, images, cols, m->B, m->channels, m->height, m->width, m->patch, stream);
    if (rc) return rc;
    if ((rc = linear(m->dtype, cols, pix, m->patch_w, m->patch_b, nullptr, 0, proj, m->D, (int64_t)m->B * np, m->D, pix, 0, true,
                     stream)))
        return rc;
    const bool first_folds = m->n_blocks > 0 && m->blocks[0].w_qkv_folded;
    if ((rc = convnn_b200_embed_tokens_moments(m->dtype, proj, m->embed_norm_w, m->embed_norm_b, m->embed_eps, m->cls, m->pe,
                                               ws + p.x, m->B, np, m->D,
                                               first_folds ? reinterpret_cast<float*>(ws + p.mom) : nullptr, stream)))
        return rc;
    int planes = first_folds ? 1 : 0;
    for (int i = 0; i < m->n_blocks; ++i) {
        const bool want = i + 1 < m->n_blocks && m->blocks[i + 1].w_qkv_folded;
        if ((rc = block_forward(m, m->blocks[i], ws, p, beside, &planes, want, stream))) return rc;
    }
    return linear(m->dtype, ws + p.x, (int64_t)m->T * m->D, m->head_w, m->head_b, nullptr, 0, logits, m->classes, m->B,
                  m->classes, m->D, 0, true, stream);
}

}  // extern "C"
