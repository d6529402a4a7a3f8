// Module-level compositions of the shape-generic kernels (fp32 validation mode, and bf16
// storage for shapes without a tcgen05 kernel). Each function restates one reference module
// as a short chain of kernels on fp32 intermediates in the caller's workspace; with
// `ws.base == nullptr` it only measures the workspace it would use.
#include "modules.cuh"
#include "generic_ops.cuh"

namespace of3 {
namespace generic {

#define TRY(x)                  \
    do {                        \
        int _rc = (x);          \
        if (_rc) return _rc;    \
    } while (0)

// ------------------------------------------------------------------ triangle multiplication
template <typename T>
int trimul(const T* z, const T* mask, T* out, int B, int N, int c_z, int c_h, int flags,
           const of3_trimul_params* p, Arena& ws, cudaStream_t st) {
    const long long rows = (long long)B * N * N;
    const int cm = c_z > c_h ? c_z : c_h;
    float* zn = (float*)ws.take(rows * c_z * sizeof(float));
    float* t1 = (float*)ws.take(rows * cm * sizeof(float));
    float* t2 = (float*)ws.take(rows * cm * sizeof(float));
    float* a = (float*)ws.take(rows * cm * sizeof(float));
    float* b = (float*)ws.take(rows * cm * sizeof(float));
    float* x = (float*)ws.take(rows * c_h * sizeof(float));
    if (!ws.base) return OF3_OK;
    OF3_REQUIRE(ws.ok(), OF3_ERR_WORKSPACE, "trimul: workspace too small (%zu needed)", ws.off);
    const bool outgoing = (flags & OF3_FLAG_OUTGOING) != 0;
    typedef const T* P;
    const RowMap dense = dense_rows(rows, c_z);
    TRY((layernorm<T, T>(z, (P)p->ln_in_w, (P)p->ln_in_b, zn, rows, c_z, 1e-5f, dense, st)));
    {   // gated projections as channel planes a[c][i][k], b[c][j][k] (incoming: a[c][k][i], b[c][k][j])
        const P wp[2] = {(P)p->w_a_p, (P)p->w_b_p}, wg[2] = {(P)p->w_a_g, (P)p->w_b_g};
        float* const ab[2] = {a, b};
        TRY(linear_gated_planes<T>(zn, 2, wp, wg, mask, ab, rows, c_h, c_z, st));
    }
    for (int s = 0; s < B; ++s) {
        const long long off = (long long)s * N * N;
        TRY(contract_planes(a + off, b + off, x + off, c_h, N, rows, !outgoing, st));
    }
    TRY(layernorm_planes<T>(x, (P)p->ln_out_w, (P)p->ln_out_b, t1, rows, c_h, 1e-5f, st));
    TRY(linear<T>(zn, (P)p->w_g, nullptr, t2, rows, c_z, c_z, st));
    return linear_final<T>(t1, (P)p->w_z, t2, (flags & OF3_FLAG_ADD_RESIDUAL) ? z : nullptr, nullptr, out, rows, c_z, c_h,
                           dense, st);
}

// ------------------------------------------------------------------ triangle attention
template <typename T>
int triattn(const T* z, const T* mask, T* out, int B, int N, int c_z, int H, int d, float inf,
            int flags, const of3_triattn_params* p, Arena& ws, cudaStream_t st) {
    const long long rows = (long long)N * N;  // one sample at a time
    const int hd = H * d;
    float* xn = (float*)ws.take(rows * c_z * sizeof(float));
    float* q = (float*)ws.take(rows * hd * sizeof(float));
    float* k = (float*)ws.take(rows * hd * sizeof(float));
    float* v = (float*)ws.take(rows * hd * sizeof(float));
    float* g = (float*)ws.take(rows * hd * sizeof(float));
    float* tb = (float*)ws.take(rows * H * sizeof(float));
    if (!ws.base) return OF3_OK;
    OF3_REQUIRE(ws.ok(), OF3_ERR_WORKSPACE, "triattn: workspace too small (%zu needed)", ws.off);
    const bool tr = (flags & OF3_FLAG_TRANSPOSED) != 0;
    typedef const T* P;
    // row r = (i', j') of the (possibly transposed) view: source element z[j', i'] when transposed
    const RowMap view{N, tr ? c_z : (long long)N * c_z, tr ? (long long)N * c_z : c_z};
    const float scale = 1.0f / sqrtf((float)d);
    for (int s = 0; s < B; ++s) {
        const T* zs = z + (long long)s * rows * c_z;
        T* os = out + (long long)s * rows * c_z;
        const T* ms = mask ? mask + (long long)s * rows : nullptr;
        TRY((layernorm<T, T>(zs, (P)p->ln_w, (P)p->ln_b, xn, rows, c_z, 1e-5f, view, st, (P)p->w_bias, H, tb)));
        const P w4[4] = {(P)p->w_q, (P)p->w_k, (P)p->w_v, (P)p->w_g};
        float* const qkvg[4] = {q, k, v, g};
        TRY(linear_multi<T>(xn, 4, w4, nullptr, qkvg, rows, hd, c_z, st));
        TRY(attention<T>(q, k, v, g, ms, tr ? 1 : N, tr ? N : 1, inf, tb, g, N, N, H, d, scale, N, st));
        TRY(linear_final<T>(g, (P)p->w_o, nullptr, (flags & OF3_FLAG_ADD_RESIDUAL) ? zs : nullptr, nullptr, os, rows, c_z,
                            hd, view, st));
    }
    return OF3_OK;
}

// ------------------------------------------------------------------ SwiGLU transition
template <typename T>
int transition(const T* x, const T* mask, T* out, long long rows, int c, int n, int flags,
               const of3_transition_params* p, Arena& ws, cudaStream_t st) {
    const int hid = n * c;
    float* xn = (float*)ws.take(rows * c * sizeof(float));
    float* a = (float*)ws.take(rows * hid * sizeof(float));
    if (!ws.base) return OF3_OK;
    OF3_REQUIRE(ws.ok(), OF3_ERR_WORKSPACE, "transition: workspace too small (%zu needed)", ws.off);
    typedef const T* P;
    const RowMap dense = dense_rows(rows, c);
    TRY((layernorm<T, T>(x, (P)p->ln_w, (P)p->ln_b, xn, rows, c, 1e-5f, dense, st)));
    TRY(linear_swiglu<T>(xn, (P)p->w_a, (P)p->w_b, a, rows, hid, c, st));
    return linear_final<T>(a, (P)p->w_out, nullptr, (flags & OF3_FLAG_ADD_RESIDUAL) ? x : nullptr, mask, out, rows, c, hid,
                           dense, st);
}

// adaptive LayerNorm: dst = sigmoid(W_g LN_s(s) + b_g) * LN(a) + W_s LN_s(s); also returns nothing else
template <typename T>
static int ada_ln(const T* a, const T* s, float* dst, float* sn, float* t1, float* t2,
                  long long rows, int c_a, int c_s, const T* ln_s_w, const T* w_g, const T* b_g,
                  const T* w_s, cudaStream_t st) {
    TRY((layernorm<T, T>(a, nullptr, nullptr, dst, rows, c_a, 1e-5f, dense_rows(rows, c_a), st)));
    TRY((layernorm<T, T>(s, ln_s_w, nullptr, sn, rows, c_s, 1e-5f, dense_rows(rows, c_s), st)));
    const T *w2[2] = {w_g, w_s}, *b2[2] = {b_g, nullptr};
    float* const t12[2] = {t1, t2};
    TRY(linear_multi<T>(sn, 2, w2, b2, t12, rows, c_a, c_s, st));
    TRY(ada_combine(t1, dst, t2, dst, rows * c_a, st));
    return OF3_OK;
}

// ------------------------------------------------------------------ attention with pair bias
template <typename T>
int attn_pair_bias(const T* a, const T* z, const T* s, const T* mask, T* out, int Ba, int Bz, int N,
                   int c_a, int c_s, int c_z, int H, int d, float inf, int flags,
                   const of3_attn_pair_bias_params* p, Arena& ws, cudaStream_t st, const float* pair_bias) {
    const long long rows = (long long)Ba * N;
    const long long zrows = (long long)Bz * N * N;
    const int hd = H * d;
    const bool ada = (flags & OF3_FLAG_ADA_LN) != 0;
    float* an = (float*)ws.take(rows * c_a * sizeof(float));
    float* q = (float*)ws.take(rows * hd * sizeof(float));
    float* k = (float*)ws.take(rows * hd * sizeof(float));
    float* v = (float*)ws.take(rows * hd * sizeof(float));
    float* g = (float*)ws.take(rows * hd * sizeof(float));
    float* zb = pair_bias ? nullptr : (float*)ws.take(zrows * H * sizeof(float));
    float* sn = ada ? (float*)ws.take(rows * c_s * sizeof(float)) : nullptr;
    float* t1 = ada ? (float*)ws.take(rows * c_a * sizeof(float)) : nullptr;
    float* t2 = ada ? (float*)ws.take(rows * c_a * sizeof(float)) : nullptr;
    float* zp = (!pair_bias && Bz > 1) ? (float*)ws.take(zrows * H * sizeof(float)) : zb;
    if (!ws.base) return OF3_OK;
    OF3_REQUIRE(ws.ok(), OF3_ERR_WORKSPACE, "attn_pair_bias: workspace too small (%zu needed)", ws.off);
    OF3_REQUIRE(Bz > 0 && Ba % Bz == 0, OF3_ERR_SHAPE, "attn_pair_bias: Ba %d not a multiple of Bz %d",
                Ba, Bz);
    if (ada) {
        OF3_REQUIRE(s != nullptr, OF3_ERR_ARG, "attn_pair_bias: AdaLN needs s");
        TRY(ada_ln<T>(a, s, an, sn, t1, t2, rows, c_a, c_s, (const T*)p->ada_ln_s_w,
                      (const T*)p->ada_w_g, (const T*)p->ada_b_g, (const T*)p->ada_w_s, st));
    } else {
        TRY((layernorm<T, T>(a, (const T*)p->ln_a_w, (const T*)p->ln_a_b, an, rows, c_a, 1e-5f, dense_rows(rows, c_a),
                             st)));
    }
    if (pair_bias != nullptr) {
        zb = const_cast<float*>(pair_bias);
    } else if (c_z == 128 && H == 16 && ((uintptr_t)z & 15) == 0) {
        // one pass over z: LayerNorm statistics and all 16 head projections per pair position
        TRY(pair_bias_c128_h16<T>(z, (const T*)p->ln_z_w, (const T*)p->ln_z_b, (const T*)p->w_z, zb, Bz,
                                      (long long)N * N, st));
    } else {
        TRY((layernorm<T, T>(z, (const T*)p->ln_z_w, (const T*)p->ln_z_b, nullptr, zrows, c_z, 1e-5f,
                             dense_rows(zrows, c_z), st, (const T*)p->w_z, H, zp)));
        if (Bz > 1) TRY(swap_heads(zp, zb, Bz, N, H, st));
    }
    {
        const T* w4[4] = {(const T*)p->w_q, (const T*)p->w_k, (const T*)p->w_v, (const T*)p->w_g};
        const T* b4[4] = {(const T*)p->b_q, nullptr, nullptr, nullptr};
        float* const qkvg[4] = {q, k, v, g};
        TRY(linear_multi<T>(an, 4, w4, b4, qkvg, rows, hd, c_a, st));
    }
    TRY(attention<T>(q, k, v, g, mask, N, 1, inf, zb, g, Ba, N, H, d, 1.0f / sqrtf((float)d), Ba / Bz, st));
    const float* gate = nullptr;
    if (ada) {
        TRY(to_f32<T>(s, sn, rows * c_s, st));
        TRY(linear<T>(sn, (const T*)p->w_ada_out, (const T*)p->b_ada_out, t1, rows, c_a, c_s, st));
        gate = t1;
    }
    return linear_final<T>(g, (const T*)p->w_o, gate, (flags & OF3_FLAG_ADD_RESIDUAL) ? a : nullptr, nullptr, out, rows,
                           c_a, hd, dense_rows(rows, c_a), st);
}

// ------------------------------------------------------------------ conditioned transition
template <typename T>
int cond_transition(const T* a, const T* s, const T* mask, T* out, long long rows, int c_a, int c_s,
                    int n, int flags, const of3_cond_transition_params* p, Arena& ws,
                    cudaStream_t st) {
    const int hid = n * c_a;
    float* an = (float*)ws.take(rows * c_a * sizeof(float));
    float* sn = (float*)ws.take(rows * c_s * sizeof(float));
    float* t1 = (float*)ws.take(rows * c_a * sizeof(float));
    float* t2 = (float*)ws.take(rows * c_a * sizeof(float));
    float* ha = (float*)ws.take(rows * hid * sizeof(float));
    if (!ws.base) return OF3_OK;
    OF3_REQUIRE(ws.ok(), OF3_ERR_WORKSPACE, "cond_transition: workspace too small (%zu needed)", ws.off);
    TRY(ada_ln<T>(a, s, an, sn, t1, t2, rows, c_a, c_s, (const T*)p->ada_ln_s_w, (const T*)p->ada_w_g,
                  (const T*)p->ada_b_g, (const T*)p->ada_w_s, st));
    TRY(linear_swiglu<T>(an, (const T*)p->w_a, (const T*)p->w_b, ha, rows, hid, c_a, st));
    TRY(to_f32<T>(s, sn, rows * c_s, st));
    TRY(linear<T>(sn, (const T*)p->w_g, (const T*)p->b_g, t2, rows, c_a, c_s, st));
    return linear_final<T>(ha, (const T*)p->w_out, t2, (flags & OF3_FLAG_ADD_RESIDUAL) ? a : nullptr, mask, out, rows, c_a,
                           hid, dense_rows(rows, c_a), st);
}

#define INSTANTIATE(T)                                                                               \
    template int trimul<T>(const T*, const T*, T*, int, int, int, int, int, const of3_trimul_params*, \
                           Arena&, cudaStream_t);                                                    \
    template int triattn<T>(const T*, const T*, T*, int, int, int, int, int, float, int,             \
                            const of3_triattn_params*, Arena&, cudaStream_t);                        \
    template int transition<T>(const T*, const T*, T*, long long, int, int, int,                     \
                               const of3_transition_params*, Arena&, cudaStream_t);                  \
    template int attn_pair_bias<T>(const T*, const T*, const T*, const T*, T*, int, int, int, int,   \
                                   int, int, int, int, float, int, const of3_attn_pair_bias_params*, \
                                   Arena&, cudaStream_t, const float*);                                          \
    template int cond_transition<T>(const T*, const T*, const T*, T*, long long, int, int, int, int, \
                                    const of3_cond_transition_params*, Arena&, cudaStream_t);
INSTANTIATE(float)
INSTANTIATE(__nv_bfloat16)

}  // namespace generic
}  // namespace of3
