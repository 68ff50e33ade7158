// Transition log-probabilities ("links") of the PCFG-NAT decoder from the projected link features,
// max_left == 1: extract_links() of the reference model after its three link projections
// (fs_plugins/models/glat_decomposed_with_link_two_hands_tri_pcfg.py:163-199) in three launches, and its
// gradient with respect to the link features and the gate logits in two more.
//
// The reference forms, per sentence b, node a, head h (chunk of the decoder dimension):
//     ab[a][k][h]    = q[a][h] . kl[left(a,k)][h] / sqrt(D)     left(a,0) = 0 (no left child), left(a,1) = a - 1
//     bc[a][k][c][h] = kl[left(a,k)][h] . kr[c][h] / sqrt(D)
//     ac[a][c][h]    = q[a][h] . kr[c][h] / sqrt(D)
// masks ab where left(a,k) is padding or outside a's left subtree and ac where c is padding, outside a's right
// subtree or not a main-chain node, normalises (ab + bc) + ac jointly over (k, c) per head (log-softmax), mixes
// the heads with log-softmax(gate logits) by log-sum-exp, and sets the whole row to -inf when a has no admissible
// left or no admissible right child.  That is ~30 element-wise / gather / roll / softmax launches over
// [B, L, 2, L, heads] tensors.  Only main-chain nodes have right children and only main-chain nodes are right
// children, so here
//   links_gather_kernel        packs the features of the M main-chain nodes (and of their left options) as the
//                              float32 operands of the GEMMs:  qm, krm [B][H][M][D], klm [B][H][M+1][D];
//   links_scores_kernel        ac [B][H][M][M] = qm krm^T,  bc [B][H][M+1][M] = klm krm^T, unscaled (small batched
//                              float32 products, one block per sentence, head and 64 x 64 tile);
//   links_from_scores_kernel   one block per (sentence, node) does the rest.
// Backward (training): links_grad [B][L][2][L] ->
//   links_scores_grad_kernel   one block per (sentence, node): the row's forward quantities once more, then the
//                              gradient of every logit (k, c, head) as X0, X1 [B][H][M][M] (left option 0 / 1,
//                              scaled), their row sums (gradient of ab) and the gradient of the gate logits;
//   links_features_grad_kernel the small products that turn X0, X1 into the gradients of q, kl, kr at the main-chain
//                              nodes and their left options, 64 x 64 tiles per (sentence, head).
#include <cuda_fp16.h>

#include "common.cuh"

namespace pcfgnat {

namespace {

constexpr int kLinkThreads = 128;
constexpr int kMaxHeads = 32;

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ float feat(const void *p, bool half, size_t i) {
    return half ? __half2float(static_cast<const __half *>(p)[i]) : static_cast<const float *>(p)[i];
}

// q, kl, kr [B][L][H][D] (f16 or f32); nodes [M] = ids of the main-chain nodes, ascending.
//   qm = q[nodes], krm = kr[nodes]; klm row 0 = kl[0] (no left child), row 1 + s = kl[nodes[s] - 1].
__global__ void links_gather_kernel(const void *__restrict__ q, const void *__restrict__ kl, const void *__restrict__ kr,
                                    int is_half, const int *__restrict__ nodes, int M, int L, int H, int D, float *qm,
                                    float *klm, float *krm) {
    const int b = blockIdx.y, r = blockIdx.x;  // r = 0 .. M: row of klm; rows 1 .. M are also rows r - 1 of qm, krm
    const int HD = H * D;
    const int left = r == 0 ? 0 : max(nodes[r - 1] - 1, 0);
    for (int i = threadIdx.x; i < HD; i += blockDim.x) {
        const int h = i / D, d = i - h * D;
        klm[(((size_t)b * H + h) * (M + 1) + r) * D + d] = feat(kl, is_half, ((size_t)b * L + left) * HD + i);
        if (r > 0) {
            const size_t src = ((size_t)b * L + nodes[r - 1]) * HD + i;
            const size_t dst = (((size_t)b * H + h) * M + (r - 1)) * D + d;
            qm[dst] = feat(q, is_half, src);
            krm[dst] = feat(kr, is_half, src);
        }
    }
}

// HT: number of heads known at compile time (the terms of a cell stay in registers between the two reductions
// over the heads), or 0 for any number up to kMaxHeads.
// gates [B][L][H] f32 (logits); nonpad [B][L] u8; left_mask, right_mask [L][L] u8 (1 = not allowed); main_chain [L]
// u8; slot_of [L] = index of a node among the main-chain nodes or -1; nodes [M] its inverse.
template <int HT>
__global__ void __launch_bounds__(kLinkThreads)
    links_from_scores_kernel(const float *__restrict__ ac, const float *__restrict__ bc, const float *__restrict__ qm,
                             const float *__restrict__ klm, const float *__restrict__ gates,
                             const uint8_t *__restrict__ nonpad, const uint8_t *__restrict__ left_mask,
                             const uint8_t *__restrict__ right_mask, const uint8_t *__restrict__ main_chain,
                             const int *__restrict__ slot_of, const int *__restrict__ nodes, int M, int L, int H, int D,
                             float scale, float *__restrict__ links) {
    extern __shared__ uint8_t s_right_ok[];  // [M] right child nodes[s] admissible for this node
    __shared__ float s_ab[2][kMaxHeads], s_lse[kMaxHeads], s_lg[kMaxHeads];
    const int a = blockIdx.x, b = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = kLinkThreads / 32;
    const uint8_t *np = nonpad + (size_t)b * L;
    float *out = links + ((size_t)b * L + a) * 2 * L;
    for (int i = tid; i < 2 * L; i += kLinkThreads) out[i] = neg_inf();  // admissible cells are overwritten below
    const int sa = slot_of[a];
    if (sa < 0) return;  // not on the main chain: no right child at max_left == 1
    // admissible children of a at all?  (the reference's link_left_nouse_mask / link_right_nouse_mask)
    int any_left = 0, any_right = 0;
    for (int j = tid; j < L; j += kLinkThreads) any_left |= np[j] && !left_mask[(size_t)a * L + j];
    for (int s = tid; s < M; s += kLinkThreads) {
        const int c = nodes[s];
        const bool r_ok = np[c] && !right_mask[(size_t)a * L + c] && main_chain[c];
        s_right_ok[s] = r_ok;
        any_right |= r_ok;
    }
    any_left = __syncthreads_or(any_left);
    any_right = __syncthreads_or(any_right);  // also: s_right_ok is written, and so is the -inf fill of this row
    if (!any_left || !any_right) return;
    const int left1 = a >= 1 ? a - 1 : 0;  // the reference's _max_left_index[a][1]
    const bool ok_left0 = np[0] && !left_mask[(size_t)a * L + 0];
    const bool ok_left1 = np[left1] && !left_mask[(size_t)a * L + left1];
    // ab[k][h]: one warp per head at a time, lanes over the chunk dimension
    for (int h = warp; h < H; h += n_warps) {
        const float *qa = qm + (((size_t)b * H + h) * M + sa) * D;
        const float *k0 = klm + (((size_t)b * H + h) * (M + 1) + 0) * D;
        const float *k1 = klm + (((size_t)b * H + h) * (M + 1) + 1 + sa) * D;
        float d0 = 0.f, d1 = 0.f;
        for (int d = lane; d < D; d += 32) {
            const float x = qa[d];
            d0 = fmaf(x, k0[d], d0);
            d1 = fmaf(x, k1[d], d1);
        }
        d0 = warp_sum_f(d0);
        d1 = warp_sum_f(d1);
        if (lane == 0) {
            s_ab[0][h] = ok_left0 ? d0 * scale : neg_inf();
            s_ab[1][h] = ok_left1 ? d1 * scale : neg_inf();
        }
    }
    if (warp == n_warps - 1) {  // log-softmax of the gate logits over the heads
        const float gt = lane < H ? gates[((size_t)b * L + a) * H + lane] : neg_inf();
        const float mx = warp_max_f(gt);
        const float sum = warp_sum_f(lane < H ? expf(gt - mx) : 0.f);
        if (lane < H) s_lg[lane] = gt - (mx + logf(sum));
    }
    __syncthreads();
    // logit of (left option k, right child slot s) for head h: (ab + bc) + ac
    auto logit = [&](int h, int k, int s) {
        const float vac = ac[(((size_t)b * H + h) * M + sa) * M + s] * scale;
        const float vbc = bc[(((size_t)b * H + h) * (M + 1) + (k ? 1 + sa : 0)) * M + s] * scale;
        return (s_ab[k][h] + vbc) + vac;
    };
    // pass 1: log-sum-exp over (k, c) per head
    for (int h = warp; h < H; h += n_warps) {
        float mx = neg_inf(), sum = 0.f;
        for (int s = lane; s < M; s += 32) {
            if (!s_right_ok[s]) continue;
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float v = logit(h, k, s);
                if (v > mx) {
                    sum = sum * expf(mx - v) + 1.f;  // exp(-inf - v) = 0 on the first finite value
                    mx = v;
                } else if (v > neg_inf()) {
                    sum += expf(v - mx);
                }
            }
        }
        const float top = warp_max_f(mx);
        sum = isinf(mx) ? 0.f : sum * expf(mx - top);
        sum = warp_sum_f(sum);
        if (lane == 0) s_lse[h] = isinf(top) ? top : top + logf(sum);
    }
    __syncthreads();
    // pass 2: mix the heads
    for (int i = tid; i < 2 * M; i += kLinkThreads) {
        const int k = i / M, s = i - k * M;
        if (!s_right_ok[s]) continue;
        float res = neg_inf();
        if (HT > 0) {
            float term[HT > 0 ? HT : 1];
            float mx = neg_inf();
#pragma unroll
            for (int h = 0; h < HT; h++) {
                term[h] = (logit(h, k, s) - s_lse[h]) + s_lg[h];
                mx = fmaxf(mx, term[h]);  // fmaxf drops NaN
            }
            if (!isinf(mx)) {
                float sum = 0.f;
#pragma unroll
                for (int h = 0; h < HT; h++)
                    if (term[h] > neg_inf()) sum += expf(term[h] - mx);
                res = mx + logf(sum);
            }
        } else {
            float mx = neg_inf();
            for (int h = 0; h < H; h++) mx = fmaxf(mx, (logit(h, k, s) - s_lse[h]) + s_lg[h]);
            if (!isinf(mx)) {
                float sum = 0.f;
                for (int h = 0; h < H; h++) {
                    const float t = (logit(h, k, s) - s_lse[h]) + s_lg[h];
                    if (t > neg_inf()) sum += expf(t - mx);
                }
                res = mx + logf(sum);
            }
        }
        out[(size_t)k * L + nodes[s]] = res;
    }
}

// C[b][h] = A[b][h] krm[b][h]^T for the rows of A = qm (M rows -> ac) and A = klm (M + 1 rows -> bc): float32, 64 x 64
// output tiles, the D axis walked in chunks of 16 through shared memory.
constexpr int kScoreTile = 64, kScoreK = 16;
__global__ void __launch_bounds__(256)
    links_scores_kernel(const float *__restrict__ qm, const float *__restrict__ klm, const float *__restrict__ krm, int M,
                        int D, float *__restrict__ ac, float *__restrict__ bc) {
    __shared__ float sa[kScoreK][kScoreTile + 1], sb[kScoreK][kScoreTile + 1];
    const int bh = blockIdx.z;
    const int tiles_m = (M + kScoreTile - 1) / kScoreTile, tiles_r = (2 * M + 1 + kScoreTile - 1) / kScoreTile;
    const int tr = blockIdx.y, tc = blockIdx.x;  // row tile over the 2 M + 1 stacked rows (qm then klm), column tile over M
    if (tr >= tiles_r || tc >= tiles_m) return;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;  // 16 x 16 threads, 4 x 4 outputs each
    float acc[4][4] = {};
    const float *qb = qm + (size_t)bh * M * D, *klb = klm + (size_t)bh * (M + 1) * D, *krb = krm + (size_t)bh * M * D;
    for (int k0 = 0; k0 < D; k0 += kScoreK) {
        for (int i = threadIdx.x; i < kScoreTile * kScoreK; i += 256) {
            const int r = i / kScoreK, k = i - r * kScoreK;
            const int row = tr * kScoreTile + r, col = tc * kScoreTile + r;
            float va = 0.f, vb = 0.f;
            if (k0 + k < D) {
                if (row < M) va = qb[(size_t)row * D + k0 + k];
                else if (row < 2 * M + 1) va = klb[(size_t)(row - M) * D + k0 + k];
                if (col < M) vb = krb[(size_t)col * D + k0 + k];
            }
            sa[k][r] = va;
            sb[k][r] = vb;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kScoreK; k++) {
            float a4[4], b4[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                a4[i] = sa[k][ty * 4 + i];
                b4[i] = sb[k][tx * 4 + i];
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a4[i], b4[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = tr * kScoreTile + ty * 4 + i;
        if (row >= 2 * M + 1) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int col = tc * kScoreTile + tx * 4 + j;
            if (col >= M) continue;
            if (row < M) ac[((size_t)bh * M + row) * M + col] = acc[i][j];
            else bc[((size_t)bh * (M + 1) + (row - M)) * M + col] = acc[i][j];
        }
    }
}

// Gradient of the logits of one (sentence, node) row.  With G = links_grad[a][k][c], res = links[a][k][c],
//   term[h] = logit[h] - lse[h] + lg[h],  w[h] = exp(term[h] - res)             (share of head h in the mixture)
//   d lp[k][c][h] = G w[h],   Gs[h] = sum_{k,c} d lp[k][c][h]  (= d lg[h]),
//   d logit[k][c][h] = d lp[k][c][h] - exp(logit[k][c][h] - lse[h]) Gs[h]
// written scaled by 1/sqrt(D) (the logits are scaled dot products) as X0 (k = 0) and X1 (k = 1) [B][H][M][M] at row
// slot(a); dab [B][H][M][2] = their row sums; dgates[a][h] = Gs[h] - softmax(gates)[h] sum_h' Gs[h'].  Rows of nodes
// that are not on the main chain, or have no admissible child, are zero (X rows) / zero (dgates).
__global__ void __launch_bounds__(kLinkThreads)
    links_scores_grad_kernel(const float *__restrict__ links_grad, const float *__restrict__ ac, const float *__restrict__ bc,
                             const float *__restrict__ qm, const float *__restrict__ klm, const float *__restrict__ gates,
                             const uint8_t *__restrict__ nonpad, const uint8_t *__restrict__ left_mask,
                             const uint8_t *__restrict__ right_mask, const uint8_t *__restrict__ main_chain,
                             const int *__restrict__ slot_of, const int *__restrict__ nodes, int M, int L, int H, int D,
                             float scale, float *__restrict__ X0, float *__restrict__ X1, float *__restrict__ dab,
                             float *__restrict__ dgates) {
    extern __shared__ uint8_t s_right_ok[];
    __shared__ float s_ab[2][kMaxHeads], s_lse[kMaxHeads], s_lg[kMaxHeads], s_gs[kMaxHeads], s_red[kMaxHeads][4];
    const int a = blockIdx.x, b = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = kLinkThreads / 32;
    const uint8_t *np = nonpad + (size_t)b * L;
    float *dg = dgates + ((size_t)b * L + a) * H;
    for (int h = tid; h < H; h += kLinkThreads) dg[h] = 0.f;
    const int sa = slot_of[a];
    if (sa < 0) return;
    // this node's rows of X0, X1 and dab start at zero
    for (int i = tid; i < H * M; i += kLinkThreads) {
        const int h = i / M, s = i - h * M;
        X0[(((size_t)b * H + h) * M + sa) * M + s] = 0.f;
        X1[(((size_t)b * H + h) * M + sa) * M + s] = 0.f;
    }
    for (int i = tid; i < 2 * H; i += kLinkThreads) dab[(((size_t)b * H + i / 2) * M + sa) * 2 + (i & 1)] = 0.f;
    int any_left = 0, any_right = 0;
    for (int j = tid; j < L; j += kLinkThreads) any_left |= np[j] && !left_mask[(size_t)a * L + j];
    for (int s = tid; s < M; s += kLinkThreads) {
        const int c = nodes[s];
        const bool r_ok = np[c] && !right_mask[(size_t)a * L + c] && main_chain[c];
        s_right_ok[s] = r_ok;
        any_right |= r_ok;
    }
    any_left = __syncthreads_or(any_left);
    any_right = __syncthreads_or(any_right);
    if (!any_left || !any_right) return;
    const int left1 = a >= 1 ? a - 1 : 0;
    const bool ok_left0 = np[0] && !left_mask[(size_t)a * L + 0];
    const bool ok_left1 = np[left1] && !left_mask[(size_t)a * L + left1];
    for (int h = warp; h < H; h += n_warps) {
        const float *qa = qm + (((size_t)b * H + h) * M + sa) * D;
        const float *k0 = klm + (((size_t)b * H + h) * (M + 1) + 0) * D;
        const float *k1 = klm + (((size_t)b * H + h) * (M + 1) + 1 + sa) * D;
        float d0 = 0.f, d1 = 0.f;
        for (int d = lane; d < D; d += 32) {
            const float x = qa[d];
            d0 = fmaf(x, k0[d], d0);
            d1 = fmaf(x, k1[d], d1);
        }
        d0 = warp_sum_f(d0);
        d1 = warp_sum_f(d1);
        if (lane == 0) {
            s_ab[0][h] = ok_left0 ? d0 * scale : neg_inf();
            s_ab[1][h] = ok_left1 ? d1 * scale : neg_inf();
        }
    }
    float gate_p = 0.f;  // softmax(gates)[lane] in the last warp
    if (warp == n_warps - 1) {
        const float gt = lane < H ? gates[((size_t)b * L + a) * H + lane] : neg_inf();
        const float mx = warp_max_f(gt);
        const float sum = warp_sum_f(lane < H ? expf(gt - mx) : 0.f);
        if (lane < H) {
            s_lg[lane] = gt - (mx + logf(sum));
            gate_p = expf(s_lg[lane]);
        }
    }
    __syncthreads();
    auto logit = [&](int h, int k, int s) {
        const float vac = ac[(((size_t)b * H + h) * M + sa) * M + s] * scale;
        const float vbc = bc[(((size_t)b * H + h) * (M + 1) + (k ? 1 + sa : 0)) * M + s] * scale;
        return (s_ab[k][h] + vbc) + vac;
    };
    for (int h = warp; h < H; h += n_warps) {
        float mx = neg_inf(), sum = 0.f;
        for (int s = lane; s < M; s += 32) {
            if (!s_right_ok[s]) continue;
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float v = logit(h, k, s);
                if (v > mx) {
                    sum = sum * expf(mx - v) + 1.f;
                    mx = v;
                } else if (v > neg_inf()) {
                    sum += expf(v - mx);
                }
            }
        }
        const float top = warp_max_f(mx);
        sum = isinf(mx) ? 0.f : sum * expf(mx - top);
        sum = warp_sum_f(sum);
        if (lane == 0) s_lse[h] = isinf(top) ? top : top + logf(sum);
    }
    for (int i = tid; i < kMaxHeads * 4; i += kLinkThreads) s_red[i / 4][i & 3] = 0.f;
    __syncthreads();
    // pass A: Gs[h] = sum over the row's cells of G w[h]; every thread walks its cells, heads in registers
    const float *grow = links_grad + ((size_t)b * L + a) * 2 * L;
    float gs_part[kMaxHeads];
    for (int h = 0; h < H; h++) gs_part[h] = 0.f;
    for (int i = tid; i < 2 * M; i += kLinkThreads) {
        const int k = i / M, s = i - k * M;
        if (!s_right_ok[s]) continue;
        const float G = grow[(size_t)k * L + nodes[s]];
        if (G == 0.f) continue;
        float mx = neg_inf();
        for (int h = 0; h < H; h++) mx = fmaxf(mx, (logit(h, k, s) - s_lse[h]) + s_lg[h]);
        if (isinf(mx)) continue;  // the cell is -inf: no gradient
        float sum = 0.f;
        for (int h = 0; h < H; h++) {
            const float t = (logit(h, k, s) - s_lse[h]) + s_lg[h];
            if (t > neg_inf()) sum += expf(t - mx);
        }
        const float inv = G / sum;
        for (int h = 0; h < H; h++) {
            const float t = (logit(h, k, s) - s_lse[h]) + s_lg[h];
            if (t > neg_inf()) gs_part[h] += expf(t - mx) * inv;
        }
    }
    for (int h = 0; h < H; h++) {
        const float v = warp_sum_f(gs_part[h]);
        if (lane == 0) s_red[h][warp] = v;
    }
    __syncthreads();
    if (tid < H) s_gs[tid] = (s_red[tid][0] + s_red[tid][1]) + (s_red[tid][2] + s_red[tid][3]);
    __syncthreads();
    if (warp == n_warps - 1) {  // gate logits: d lg - softmax(gates) sum d lg
        const float tot = warp_sum_f(lane < H ? s_gs[lane] : 0.f);
        if (lane < H) dg[lane] = s_gs[lane] - gate_p * tot;
    }
    // pass B: d logit of every cell and head, and the row sums per left option
    float ab_part[2][kMaxHeads];
    for (int h = 0; h < H; h++) ab_part[0][h] = ab_part[1][h] = 0.f;
    for (int i = tid; i < 2 * M; i += kLinkThreads) {
        const int k = i / M, s = i - k * M;
        if (!s_right_ok[s]) continue;
        const float G = grow[(size_t)k * L + nodes[s]];
        float mx = neg_inf(), sum = 0.f;
        for (int h = 0; h < H; h++) mx = fmaxf(mx, (logit(h, k, s) - s_lse[h]) + s_lg[h]);
        if (!isinf(mx))
            for (int h = 0; h < H; h++) {
                const float t = (logit(h, k, s) - s_lse[h]) + s_lg[h];
                if (t > neg_inf()) sum += expf(t - mx);
            }
        float *X = k ? X1 : X0;
        for (int h = 0; h < H; h++) {
            const float lgt = logit(h, k, s);
            float d = 0.f;
            if (lgt > neg_inf()) {
                const float t = (lgt - s_lse[h]) + s_lg[h];
                const float dlp = (G != 0.f && !isinf(mx)) ? G * expf(t - mx) / sum : 0.f;
                d = (dlp - expf(lgt - s_lse[h]) * s_gs[h]) * scale;
            }
            X[(((size_t)b * H + h) * M + sa) * M + s] = d;
            ab_part[k][h] += d;
        }
    }
    __syncthreads();  // s_red is reused
    for (int k = 0; k < 2; k++) {
        for (int h = 0; h < H; h++) {
            const float v = warp_sum_f(ab_part[k][h]);
            if (lane == 0) s_red[h][warp] = v;
        }
        __syncthreads();
        if (tid < H) dab[(((size_t)b * H + tid) * M + sa) * 2 + k] = (s_red[tid][0] + s_red[tid][1]) + (s_red[tid][2] + s_red[tid][3]);
        __syncthreads();
    }
}

// Gradients of the packed features from X0, X1 and dab:
//   dqm[a]      = dab[a][0] klm[0] + dab[a][1] klm[1 + a] + sum_s (X0 + X1)[a][s] krm[s]
//   dklm[1 + a] = dab[a][1] qm[a] + sum_s X1[a][s] krm[s]
//   dklm[0]     = sum_a ( dab[a][0] qm[a] + sum_s X0[a][s] krm[s] )
//   dkrm[s]     = sum_a ( (X0 + X1)[a][s] qm[a] + X0[a][s] klm[0] + X1[a][s] klm[1 + a] )
// and scattered to the nodes: dq[nodes[a]], dkr[nodes[s]], dkl[nodes[a] - 1] and dkl[0] (which also takes row 1 of the
// first main-chain node, whose left option 1 is node 0 again).  dq, dkl, dkr [B][L][H][D] f32 were zero-filled.
//
// Four float32 matrix products, M x M x D each, per (sentence, head).  A block makes 64 rows x 64 columns of d of the
// parents' two products (role 0) or of the children's two (role 1), 4 x 4 outputs of both per thread, the summed index
// walked in chunks of 32 through 27 / 33 KB of shared memory: three 16-byte shared-memory loads per 32 FMAs, so the
// FMA pipe is what bounds it, and no shape is too large for it.  The X matrices are zero wherever a child is not
// admissible (all children at or below the parent, padding): a chunk whose X are all zero is skipped, unless the
// features beside it are not finite (0 x inf stays NaN).  90 sentences, M = 161, 8 x 64 features: 366 us; 3 095 us
// with one thread per output reading its operands from global memory, as it was.
constexpr int kFgThreads = 256, kFgTile = 64, kFgChunk = 32, kFgPitch = kFgChunk + 4;
constexpr int kFgSmemFloats = 4 * kFgChunk * kFgTile + 4 * kFgTile;  // role 1, the larger of the two

__device__ __forceinline__ bool not_finite(float x) { return !(fabsf(x) < CUDART_INF_F); }

// rows r0 .. r0 + 31 (< rows), columns d0 .. d0 + 63 (< D) of src [rows][D] into dst [32][64], zero outside
__device__ __forceinline__ bool stage_features(const float *__restrict__ src, int r0, int rows, int d0, int D, bool vec,
                                               float *dst) {
    bool odd = false;
    if (vec) {
        for (int i = threadIdx.x; i < kFgChunk * kFgTile / 4; i += kFgThreads) {
            const int r = r0 + i / (kFgTile / 4), d = d0 + i % (kFgTile / 4) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < rows && d < D) v = __ldg(reinterpret_cast<const float4 *>(src + (size_t)r * D + d));
            odd |= not_finite(v.x) || not_finite(v.y) || not_finite(v.z) || not_finite(v.w);
            reinterpret_cast<float4 *>(dst)[i] = v;
        }
    } else {
        for (int i = threadIdx.x; i < kFgChunk * kFgTile; i += kFgThreads) {
            const int r = r0 + i / kFgTile, d = d0 + i % kFgTile;
            const float v = r < rows && d < D ? __ldg(src + (size_t)r * D + d) : 0.f;
            odd |= not_finite(v);
            dst[i] = v;
        }
    }
    return odd;
}

__device__ __forceinline__ float part(const float4 &v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; }

// vec: D a multiple of 4 and the feature matrices on 16-byte boundaries
__global__ void __launch_bounds__(kFgThreads, 2)
    links_features_grad_kernel(const float *__restrict__ X0, const float *__restrict__ X1, const float *__restrict__ dab,
                               const float *__restrict__ qm, const float *__restrict__ klm, const float *__restrict__ krm,
                               const int *__restrict__ nodes, int M, int L, int H, int D, int vec, float *__restrict__ dq,
                               float *__restrict__ dkl, float *__restrict__ dkr) {
    __shared__ __align__(16) float smem[kFgSmemFloats];
    const int role = blockIdx.x & 1, r0 = (blockIdx.x >> 1) * kFgTile, d0 = blockIdx.y * kFgTile;
    const size_t bh = blockIdx.z;
    const int b = blockIdx.z / H, h = blockIdx.z - b * H;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const float *x0 = X0 + bh * M * M, *x1 = X1 + bh * M * M;
    const float *q = qm + bh * M * D, *kl = klm + bh * (M + 1) * D, *kr = krm + bh * M * D;
    const size_t pitch = (size_t)H * D, base = (size_t)b * L * pitch + (size_t)h * D;
    float acc0[4][4] = {}, acc1[4][4] = {};
    if (role == 0) {  // rows are parents a; summed over the children s
        float *sx0 = smem, *sx1 = sx0 + kFgTile * kFgPitch, *sk = sx1 + kFgTile * kFgPitch;
        for (int s0 = 0; s0 < M; s0 += kFgChunk) {
            bool work = false;
#pragma unroll 4
            for (int i = tid; i < kFgTile * kFgChunk; i += kFgThreads) {
                const int r = i / kFgChunk, s = i % kFgChunk;
                float v0 = 0.f, v1 = 0.f;
                if (r0 + r < M && s0 + s < M) {
                    v0 = __ldg(x0 + (size_t)(r0 + r) * M + s0 + s);
                    v1 = __ldg(x1 + (size_t)(r0 + r) * M + s0 + s);
                }
                work |= v0 != 0.f || v1 != 0.f;
                sx0[r * kFgPitch + s] = v0;
                sx1[r * kFgPitch + s] = v1;
            }
            work |= stage_features(kr, s0, M, d0, D, vec, sk);
            if (__syncthreads_or(work)) {
#pragma unroll 2
                for (int s = 0; s < kFgChunk; s += 4) {
                    float4 x0v[4], x1v[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        x0v[i] = *reinterpret_cast<const float4 *>(sx0 + (4 * ty + i) * kFgPitch + s);
                        x1v[i] = *reinterpret_cast<const float4 *>(sx1 + (4 * ty + i) * kFgPitch + s);
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float4 kv = *reinterpret_cast<const float4 *>(sk + (s + j) * kFgTile + 4 * tx);
#pragma unroll
                        for (int i = 0; i < 4; i++)
#pragma unroll
                            for (int c = 0; c < 4; c++) {
                                acc0[i][c] = fmaf(part(x0v[i], j), part(kv, c), acc0[i][c]);
                                acc1[i][c] = fmaf(part(x1v[i], j), part(kv, c), acc1[i][c]);
                            }
                    }
                }
            }
            __syncthreads();
        }
        float kl0_part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = r0 + 4 * ty + i;
            if (r >= M) continue;
            const float w0 = dab[(bh * M + r) * 2], w1 = dab[(bh * M + r) * 2 + 1];
            const int node = nodes[r], left = node - 1 > 0 ? node - 1 : 0;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int d = d0 + 4 * tx + c;
                if (d >= D) continue;
                const float qv = q[(size_t)r * D + d];
                dq[base + node * pitch + d] = w0 * kl[d] + w1 * kl[(size_t)(1 + r) * D + d] + (acc0[i][c] + acc1[i][c]);
                const float g = w1 * qv + acc1[i][c];  // left option 1 of node r: a row of its own, but for node 0's
                if (left > 0) dkl[base + left * pitch + d] = g;
                else kl0_part[c] += g;
                kl0_part[c] += w0 * qv + acc0[i][c];  // this node's part of the "no left child" row
            }
        }
        // the block's part of row 0 of kl: all parents share that row
        float *red = smem;
#pragma unroll
        for (int c = 0; c < 4; c++) red[ty * kFgTile + 4 * tx + c] = kl0_part[c];
        __syncthreads();
        if (tid < kFgTile && d0 + tid < D) {
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 16; i++) sum += red[i * kFgTile + tid];
            atomicAdd(dkl + base + d0 + tid, sum);
        }
    } else {  // rows are children s; summed over the parents a
        float *sxs = smem, *sx1 = sxs + kFgChunk * kFgTile, *sq = sx1 + kFgChunk * kFgTile, *sk = sq + kFgChunk * kFgTile;
        float *sums = sk + kFgChunk * kFgTile;  // [4][64]
        const int s_own = r0 + (tid & 63);      // the column whose X this thread stages
        float x0sum = 0.f;                      // its sum of X0 over a = tid / 64 + 4 j
        for (int a0 = 0; a0 < M; a0 += kFgChunk) {
            bool work = false;
#pragma unroll
            for (int j = 0; j < kFgChunk / 4; j++) {
                const int a = (tid >> 6) + 4 * j;
                float v0 = 0.f, v1 = 0.f;
                if (a0 + a < M && s_own < M) {
                    v0 = __ldg(x0 + (size_t)(a0 + a) * M + s_own);
                    v1 = __ldg(x1 + (size_t)(a0 + a) * M + s_own);
                }
                work |= v0 != 0.f || v1 != 0.f;
                x0sum += v0;
                sxs[a * kFgTile + (tid & 63)] = v0 + v1;
                sx1[a * kFgTile + (tid & 63)] = v1;
            }
            work |= stage_features(q, a0, M, d0, D, vec, sq);
            work |= stage_features(kl + D, a0, M, d0, D, vec, sk);
            if (__syncthreads_or(work)) {
#pragma unroll 4
                for (int a = 0; a < kFgChunk; a++) {
                    const float4 xs = *reinterpret_cast<const float4 *>(sxs + a * kFgTile + 4 * ty);
                    const float4 xb = *reinterpret_cast<const float4 *>(sx1 + a * kFgTile + 4 * ty);
                    const float4 qv = *reinterpret_cast<const float4 *>(sq + a * kFgTile + 4 * tx);
                    const float4 kv = *reinterpret_cast<const float4 *>(sk + a * kFgTile + 4 * tx);
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            acc0[i][c] = fmaf(part(xs, i), part(qv, c), acc0[i][c]);
                            acc1[i][c] = fmaf(part(xb, i), part(kv, c), acc1[i][c]);
                        }
                }
            }
            __syncthreads();
        }
        sums[(tid >> 6) * kFgTile + (tid & 63)] = x0sum;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = r0 + 4 * ty + i;
            if (r >= M) continue;
            const int t = 4 * ty + i;
            const float w = (sums[t] + sums[kFgTile + t]) + (sums[2 * kFgTile + t] + sums[3 * kFgTile + t]);
            const size_t at = base + nodes[r] * pitch;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int d = d0 + 4 * tx + c;
                if (d < D) dkr[at + d] = fmaf(w, kl[d], acc0[i][c] + acc1[i][c]);
            }
        }
    }
}

}  // namespace

int launch_links_scores(const float *qm, const float *klm, const float *krm, int M, int B, int H, int D, float *ac,
                        float *bc, cudaStream_t st) {
    if (B == 0 || M == 0) return PCFGNAT_OK;
    const dim3 grid((M + kScoreTile - 1) / kScoreTile, (2 * M + 1 + kScoreTile - 1) / kScoreTile, B * H);
    links_scores_kernel<<<grid, 256, 0, st>>>(qm, klm, krm, M, D, ac, bc);
    return cuda_rc(cudaGetLastError());
}

int launch_links_backward(const float *links_grad, const float *ac, const float *bc, const float *qm, const float *klm,
                          const float *krm, const float *gates, const uint8_t *nonpad, const uint8_t *left_mask,
                          const uint8_t *right_mask, const uint8_t *main_chain, const int *slot_of, const int *nodes, int M,
                          int B, int L, int H, int D, float *X0, float *X1, float *dab, float *dq, float *dkl, float *dkr,
                          float *dgates, cudaStream_t st) {
    if (B == 0) return PCFGNAT_OK;
    if (H > kMaxHeads) return PCFGNAT_ERR_TOO_LARGE;
    const float scale = 1.f / sqrtf((float)D);
    const size_t smem = (size_t)(M + 16) / 16 * 16;
    if (smem > 40 * 1024) return PCFGNAT_ERR_TOO_LARGE;
    links_scores_grad_kernel<<<dim3(L, B), kLinkThreads, smem, st>>>(links_grad, ac, bc, qm, klm, gates, nonpad, left_mask,
                                                                     right_mask, main_chain, slot_of, nodes, M, L, H, D, scale,
                                                                     X0, X1, dab, dgates);
    if (cudaGetLastError() != cudaSuccess) return PCFGNAT_ERR_CUDA;
    if (M == 0) return PCFGNAT_OK;
    const bool vec = D % 4 == 0 && ((reinterpret_cast<uintptr_t>(qm) | reinterpret_cast<uintptr_t>(klm) |
                                     reinterpret_cast<uintptr_t>(krm)) & 15) == 0;
    const dim3 grid(2 * ((M + kFgTile - 1) / kFgTile), (D + kFgTile - 1) / kFgTile, B * H);
    links_features_grad_kernel<<<grid, kFgThreads, 0, st>>>(X0, X1, dab, qm, klm, krm, nodes, M, L, H, D, vec, dq, dkl, dkr);
    return cuda_rc(cudaGetLastError());
}

int launch_links_gather(const void *q, const void *kl, const void *kr, int is_half, const int *nodes, int M, int B, int L,
                        int H, int D, float *qm, float *klm, float *krm, cudaStream_t st) {
    if (B == 0) return PCFGNAT_OK;
    links_gather_kernel<<<dim3(M + 1, B), 256, 0, st>>>(q, kl, kr, is_half, nodes, M, L, H, D, qm, klm, krm);
    return cuda_rc(cudaGetLastError());
}

int launch_links_from_scores(const float *ac, const float *bc, const float *qm, const float *klm, const float *gates,
                             const uint8_t *nonpad, const uint8_t *left_mask, const uint8_t *right_mask,
                             const uint8_t *main_chain, const int *slot_of, const int *nodes, int M, int B, int L, int H,
                             int D, float *links, cudaStream_t st) {
    if (B == 0) return PCFGNAT_OK;
    if (H > kMaxHeads) return PCFGNAT_ERR_TOO_LARGE;
    const float scale = 1.f / sqrtf((float)D);
    const size_t smem = (size_t)(M + 16) / 16 * 16;
    if (smem > 40 * 1024) return PCFGNAT_ERR_TOO_LARGE;
    if (H == 8)
        links_from_scores_kernel<8><<<dim3(L, B), kLinkThreads, smem, st>>>(ac, bc, qm, klm, gates, nonpad, left_mask, right_mask,
                                                                          main_chain, slot_of, nodes, M, L, H, D, scale, links);
    else
        links_from_scores_kernel<0><<<dim3(L, B), kLinkThreads, smem, st>>>(ac, bc, qm, klm, gates, nonpad, left_mask, right_mask,
                                                                          main_chain, slot_of, nodes, M, L, H, D, scale, links);
    return cuda_rc(cudaGetLastError());
}

}  // namespace pcfgnat
