/* geoflac_fno.h -- tensor-core kernels of the learned surrogate (Fourier
 * neural operator) that screens and fast-forwards ensemble members.
 *
 * No reference counterpart: GeoFLAC has no learned component.  Device
 * pointers throughout; every call is asynchronous on `stream` (a
 * cudaStream_t, NULL = default stream).
 */
#ifndef GEOFLAC_FNO_H
#define GEOFLAC_FNO_H

#ifdef __cplusplus
extern "C" {
#endif

#define GF_FNO_OK 0
#define GF_FNO_ERR_CUDA (-1)
#define GF_FNO_ERR_ARG (-2)
#define GF_FNO_ERR_ALIGN (-3)   /* TMA needs 16-byte aligned bases and strides */
#define GF_FNO_ERR_TIMEOUT (-6) /* a bounded wait inside a kernel gave up */

/* C[z][m][n] = alpha * sum_k A[z][m][k] * B[z][n][k] + beta * C[z][m][n] + bias[n]
 * A: BF16, row stride lda, batch stride sA (elements); B: BF16, ldb, sB;
 * C: FP32 (c_bf16 = 0) or BF16 (c_bf16 = 1, beta must be 0), ldc, sC
 * (sA/sB/sC = 0: dense batches).  K % 8 == 0, lda and ldb multiples of 8.
 * tcgen05 MMA with FP32 accumulation in tensor memory, TMA operand loads. */
int gf_gemm_bf16(const void *A, const void *B, void *C, int batch, int M, int N, int K, long long lda, long long sA,
                 long long ldb, long long sB, long long ldc, long long sC, int c_bf16, float alpha, float beta,
                 const float *bias, void *stream);
/* The same with three extensions: sA = -1 shares one A among all batches;
 * (FP32 C only) aux, if not NULL, receives a BF16 copy of the final C
 * (act = 0) or of GELU(C) (act = 1) in the same layout; and c_bf16 = 2
 * (with aux) leaves C unwritten: C is then only read, for beta != 0, or
 * may be NULL with beta = 0 (inference, where only the BF16 activation
 * is kept). */
int gf_gemm_bf16_ex(const void *A, const void *B, void *C, int batch, int M, int N, int K, long long lda,
                    long long sA, long long ldb, long long sB, long long ldc, long long sC, int c_bf16, float alpha,
                    float beta, const float *bias, void *aux, int act, void *stream);
/* GF_FNO_ERR_TIMEOUT if a GEMM kernel gave up a wait since the last call. */
int gf_gemm_error(void);

/* Element types below: 0 = FP32, 1 = BF16. */
/* dst[b][c][r] = src[b][r][c] for batch matrices of rows x cols. */
int gf_fno_transpose(const void *src, void *dst, int batch, long long rows, int cols, int src_bf16, int dst_bf16,
                     void *stream);
int gf_fno_cast(const void *src, void *dst, long long n, int src_bf16, int dst_bf16, void *stream);
/* a = GELU(z) (erf form); dz = da * GELU'(z), with an optional BF16 copy. */
int gf_fno_gelu(const float *z, void *a, long long n, int a_bf16, void *stream);
int gf_fno_gelu_bwd(const float *z, const void *da, int da_bf16, float *dz, void *dz_bf16, long long n, void *stream);
/* Complex bookkeeping of the truncated 2-D DFT.  Y[(b, c, kp)][q]: for the
 * W-transformed row kp (kp < m2 real part, kp >= m2 imaginary part of W-mode
 * kp mod m2), cosine (q < Q) and sine (q >= Q) sums over the rows h of the Q
 * kept H-modes.  U[(k2, q)][b][(c, re|im)] (BF16) is the 2-D DFT coefficient;
 * the _bwd form maps dU (FP32, same layout) back to dY (BF16). */
int gf_fno_spec_combine(const float *Y, void *U, int B, int C, int m2, int Q, void *stream);
int gf_fno_spec_combine_bwd(const float *dU, void *dY, int B, int C, int m2, int Q, void *stream);
/* Complex mode weights R[mode][i][o][re, im] (FP32) to the real 2C x 2C
 * blocks Rm[mode][(o, part)][(i, part)] and RmT = transpose (BF16), and the
 * gradient of R from the gradient of Rm. */
int gf_fno_expand_modes(const float *R, void *Rm, void *RmT, int modes, int C, void *stream);
int gf_fno_modes_grad(const float *dRm, float *dR, int modes, int C, void *stream);
/* out[c] (+)= sum_r X[r][c]; dst[i] (+)= sum_b src[b][i]. */
int gf_fno_colsum(const float *X, float *out, long long rows, int cols, int accum, void *stream);
int gf_fno_colsum_bf16(const void *X, float *out, long long rows, int cols, int accum, void *stream);
/* X in blocks of 32 rows x 8 columns, [rows / 32][cols / 8][32][8] (rows >= 4096,
 * a multiple of 32; cols a multiple of 8 that divides 256): gf_fno_colsum's sums. */
int gf_fno_colsum_blocked(const float *X, float *out, long long rows, int cols, int accum, void *stream);
/* The same sums with the caller's scratch of 1024 x cols floats (the others
 * allocate theirs in the stream's order): layout 0 gf_fno_colsum, 1
 * gf_fno_colsum_bf16, 2 gf_fno_colsum_blocked. */
int gf_fno_colsum_with(const void *X, int layout, float *part, float *out, long long rows, int cols, int accum,
                       void *stream);
int gf_fno_sum_batches(const float *src, float *dst, int nb, long long n, int accum, void *stream);
/* Adam (bias-corrected, decoupled from the loss scale), step counts from 1. */
int gf_fno_adam(float *p, const float *g, float *m, float *v, long long n, float lr, float b1, float b2, float eps,
                int step, float weight_decay, void *stream);
/* loss += mean((pred - target)^2); dpred = scale * 2 (pred - target) / n. */
int gf_fno_mse(const float *pred, const float *target, void *dpred, int dpred_bf16, double *loss, long long n,
               float scale, void *stream);
/* Surrogate input from a sampled grid raw [n][H][W][9] and member
 * parameters [n][4]: (raw - mean) / std per channel, (params - pmean) /
 * pstd, two grid coordinates in [-1, 1], one zero channel -> BF16
 * [n][H][W][16].  stats = {mean[9], std[9], pmean[4], pstd[4]}. */
int gf_fno_pack_input(const float *raw, const float *params, const float *stats, void *out, int n, int H, int W,
                      void *stream);
/* Training target from the later grid y and the earlier x: (y - x - mean_d) /
 * std_d in channels 0..8 of 16 (FP32); stats_d = {mean_d[9], std_d[9]}. */
int gf_fno_pack_target(const float *y, const float *x, const float *stats_d, float *out, long long points,
                       void *stream);
/* dst[r] = src[idx[r]] for nrows rows of row_bytes bytes (idx on the device). */
int gf_fno_gather_rows(const void *src, void *dst, const long long *idx, int nrows, long long row_bytes,
                       void *stream);
/* Prediction back to fields: y = x + mean_d + std_d * pred. */
int gf_fno_unpack(const float *pred, const float *x, const float *stats_d, float *y, long long points, void *stream);
/* The same with weights: term i weighted by w[(i / w_period) % w_len]. */
int gf_fno_mse_weighted(const float *pred, const float *target, void *dpred, int dpred_bf16, double *loss,
                        long long n, float scale, const float *w, long long w_period, int w_len, void *stream);
/* out = x + y (y may be NULL), FP32 and/or BF16 outputs. */
int gf_fno_add(const float *x, const float *y, float *out, void *out_bf16, long long n, void *stream);

/* ---- the forward pass in fused kernels (64 channels) ----
 * gf_fno_layer_ok: 1 if the shapes fit them (C = 64, W = 128, 256 or 384,
 * H = 64 or 128, 2 m2 and Q multiples of 16 up to 64, cin a multiple of 16 up
 * to 64, P = 128, cout = 16).  Their results equal the products above, bit for
 * bit.  BF16 unless said otherwise; K2 = 2 m2; DFT matrices as in
 * geoflac_gb300/fno.py.
 * gf_fno_row: rows of W points, z = v Wl^T + bias + IW Z (v [rows W][kin], Wl
 * [64][kin], bias FP32; Z [rows][K2][64] with rows (k2, re|im), NULL: no such
 * term); z (FP32, may be NULL) and vout [rows W][64] = GELU(z) (act = 1) or z
 * are written, and Xw [rows][K2][64] = FW vout (rows: real, then imaginary
 * parts; NULL: not computed).
 * gf_fno_fwd_h: Xw [B][H][K2][64] -> U[(k2, q)][b][(c, re|im)].
 * gf_fno_modes: V[mode][b][re|im][o] from U and the FP32 weights
 * R[mode][i][o][re, im].
 * gf_fno_inv_h: V -> Z [B][H][(k2, re|im)][64].
 * gf_fno_proj: out (FP32 [rows W][16]) = GELU(v P1^T + b1) P2^T + b2; zp (FP32)
 * and h [rows W][128], if not NULL, receive the pre-activations and GELU(zp). */
int gf_fno_layer_ok(int H, int W, int C, int m2, int Q, int cin, int P, int cout);
int gf_fno_row(const void *v, int kin, const void *Z, const void *IW, const void *Wl, const float *bias, int act,
               const void *FW, float *z, void *vout, void *Xw, int rows, int W, int K2, void *stream);
int gf_fno_fwd_h(const void *Xw, const void *FH, void *U, int B, int H, int m2, int Q, void *stream);
int gf_fno_modes(const void *U, const float *R, void *V, int B, int modes, void *stream);
/* and keeps R in BF16, Rb[mode][i][o][re, im], as the products took it */
int gf_fno_modes_keep(const void *U, const float *R, void *V, void *Rb, int B, int modes, void *stream);
int gf_fno_inv_h(const void *V, const void *IH, void *Z, int B, int H, int m2, int Q, void *stream);
int gf_fno_proj(const void *v, const void *P1, const float *b1, const void *P2, const float *b2, float *zp, void *h,
                float *out, int rows, int W, void *stream);

/* ---- the backward pass in fused kernels, under the same shapes ----
 * Gradients BF16, and (df1, df) FP32 for the bias gradients, in gf_fno_colsum_blocked's
 * layout.
 * gf_fno_proj_bwd: dzp [rows W][128] = (dout P2) GELU'(zp), dzo [rows W][64] =
 * dzp P1, dZ [rows][K2][64] = IWT dzo.
 * gf_fno_row_bwd: dzo = (dz Wl + FW^T dXw) GELU'(z) (z NULL: no factor), dZ =
 * IWT dzo (NULL: not computed).
 * gf_fno_inv_h_bwd: dZ -> dV[(k2, q)][b][(c, re|im)].
 * gf_fno_modes_bwd: dU[mode][b][re|im][c] and dR (FP32) from dV and U.
 * gf_fno_fwd_h_bwd: dU -> dXw [B][H][K2][64].
 * gf_fno_wgrad: part[s][j][n] = sum over the s-th of `chunks` equal chunks
 * (multiples of 128 points) of A[m][j] B[m][n], A [M][na = 64 or 128], B
 * [M][nb]; transposed (nb = 16): part[s][n][j]. */
int gf_fno_proj_bwd(const void *dout, const float *zp, const void *P1, const void *P2, const void *IWT, void *dzp,
                    float *df1, void *dzo, float *df, void *dZ, int rows, int W, int K2, void *stream);
int gf_fno_row_bwd(const void *dz, const void *dXw, const void *FW, const void *Wl, const float *z, const void *IWT,
                   void *dzo, float *df, void *dZ, int rows, int W, int K2, void *stream);
int gf_fno_inv_h_bwd(const void *dZ, const void *IHT, void *dV, int B, int H, int m2, int Q, void *stream);
int gf_fno_modes_bwd(const void *dV, const void *U, const float *R, void *dU, float *dR, int B, int modes,
                     void *stream);
/* the same from gf_fno_modes_keep's Rb */
int gf_fno_modes_bwd_kept(const void *dV, const void *U, const void *Rb, void *dU, float *dR, int B, int modes,
                          void *stream);
int gf_fno_fwd_h_bwd(const void *dU, const void *FHT, void *dXw, int B, int H, int m2, int Q, void *stream);
int gf_fno_wgrad(const void *A, int na, const void *B, int nb, int transposed, float *part, long long M, int chunks,
                 void *stream);

#ifdef __cplusplus
}
#endif

#endif /* GEOFLAC_FNO_H */
