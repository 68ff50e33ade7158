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
//                              float32 products, one block per sentence, 128 x 64 tile and up to four heads).  Tiles
//                              without an admissible (node, right child) pair are left unwritten when the masks are
//                              given: ac and bc are defined at admissible pairs only;
//   links_from_scores_kernel   one block per (sentence, node) does the rest.
// Backward (training): links_grad [B][L][2][L] ->
//   links_scores_grad_kernel   one block per (sentence, node): the row's forward quantities once more, then the
//                              gradient of every logit (k, c, head) as X0, X1 [B][H][M][M] (left option 0 / 1,
//                              scaled), their row sums (gradient of ab) and the gradient of the gate logits;
//   links_features_grad_kernel the small products that turn X0, X1 into the gradients of q, kl, kr at the main-chain
//                              nodes and their left options, 64 x 64 tiles per (sentence, head).
#include <cuda_fp16.h>

#include <initializer_list>

#include "common.cuh"

namespace pcfgnat {

namespace {

constexpr int kMaxHeads = 32;
constexpr size_t kRowSmem = 40 * 1024;  // a row's exponentials are kept in shared memory up to here: five blocks per SM
inline int row_threads(int H) { return H <= 4 ? 128 : 256; }

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
// VEC: four features at a time (D a multiple of 4, everything on 16-byte boundaries).  Bound by the float32 writes.
template <bool VEC>
__global__ void __launch_bounds__(256)
    links_gather_kernel(const void *__restrict__ q, const void *__restrict__ kl, const void *__restrict__ kr, int is_half,
                        const int *__restrict__ nodes, int M, int L, int H, int D, float *qm, float *klm, float *krm) {
    constexpr int V = VEC ? 4 : 1;
    const int b = blockIdx.y, HD = H * D, per_row = HD / V;
    const int i = blockIdx.x * 256 + threadIdx.x;
    const int r = i / per_row, e = (i - r * per_row) * V;  // r = 0 .. M: row of klm; rows 1 .. M are also rows r - 1 of qm, krm
    if (r > M) return;
    const int h = e / D, d = e - h * D;
    const int node = r == 0 ? 0 : nodes[r - 1], left = node > 0 ? node - 1 : 0;
    auto copy = [&](const void *src, size_t from, float *dst, size_t to) {
        if constexpr (VEC) {
            float4 v;
            if (is_half) {
                const uint2 u = __ldg(reinterpret_cast<const uint2 *>(static_cast<const __half *>(src) + from));
                const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&u.x));
                const float2 hi = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
                v = make_float4(lo.x, lo.y, hi.x, hi.y);
            } else {
                v = __ldg(reinterpret_cast<const float4 *>(static_cast<const float *>(src) + from));
            }
            *reinterpret_cast<float4 *>(dst + to) = v;
        } else {
            dst[to] = feat(src, is_half, from);
        }
    };
    copy(kl, ((size_t)b * L + left) * HD + e, klm, (((size_t)b * H + h) * (M + 1) + r) * D + d);
    if (r > 0) {
        const size_t src = ((size_t)b * L + node) * HD + e, dst = (((size_t)b * H + h) * M + (r - 1)) * D + d;
        copy(q, src, qm, dst);
        copy(kr, src, krm, dst);
    }
}

// One (sentence, node) row of the transitions: what its forward and its gradient both start from.  The blocks of
// both kernels have a warp per head, up to eight.
struct RowArgs {
    const float *ac, *bc, *qm, *klm, *gates;
    const uint8_t *nonpad, *left_mask, *right_mask, *main_chain;
    const int *slot_of, *nodes;
    int M, L, H, D;
    float scale;
};

// Shared memory of a row: right_ok [M] (bytes), and with STAGED e [H][2][M] = exp(logit - top[head]), each head's
// logits relative to its largest one.  !STAGED (rows too long for that) forms e again from the scores when asked.
template <bool STAGED>
struct Row {
    const RowArgs &p;
    int a, b, sa, lo, hi;  // node, sentence, its slot; slots [lo, hi) hold every admissible right child
    const uint8_t *right_ok;
    float *e;
    const float (*ab)[kMaxHeads];
    const float *top;

    // logit of (left option k, right child slot s) for head h: (ab + bc) + ac
    __device__ __forceinline__ float logit(int h, int k, int s) const {
        const size_t bh = (size_t)b * p.H + h;
        const float vac = __ldg(p.ac + (bh * p.M + sa) * p.M + s) * p.scale;
        const float vbc = __ldg(p.bc + (bh * (p.M + 1) + (k ? 1 + sa : 0)) * p.M + s) * p.scale;
        return (ab[k][h] + vbc) + vac;
    }
    // -inf and NaN logits count nothing; nor does a head with a logit of +inf (its others would be -inf, itself NaN)
    __device__ __forceinline__ float rel(float v, float t) const { return v > neg_inf() && t < CUDART_INF_F ? expf(v - t) : 0.f; }
    __device__ __forceinline__ float exp_at(int h, int k, int s) const {
        if constexpr (STAGED) return e[((size_t)h * 2 + k) * p.M + s];
        else return rel(logit(h, k, s), top[h]);
    }
};

// A cell of the mixture is log sum_h e[h] c[h], c[h] = gate probability / sum of the head's e.  Below this sum the
// cell is formed from the log-probabilities instead: e of all heads may be about to flush to zero.
constexpr float kMixtureFloor = 1e-30f;

// Sets up a row: false when it has no admissible child on one of the sides (or the node is not on the main chain),
// uniformly over the block.  s_lse, s_lg: per head the log-sum-exp of the logits and the log gate probability;
// s_c, s_inv: gate probability / sum of e, and 1 / that sum, 0 where undefined.  Ends with the block in step.
template <bool STAGED>
__device__ __forceinline__ bool links_row(Row<STAGED> &row, uint8_t *right_ok, float (*s_ab)[kMaxHeads], float *s_top,
                                          float *s_lse, float *s_lg, float *s_c, float *s_inv) {
    const RowArgs &p = row.p;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = blockDim.x >> 5;
    const int a = row.a, sa = row.sa, M = p.M;
    const uint8_t *np = p.nonpad + (size_t)row.b * p.L;
    __shared__ int s_lo, s_hi;
    if (tid == 0) {
        s_lo = M;
        s_hi = 0;
    }
    // admissible children of a at all?  (the reference's link_left_nouse_mask / link_right_nouse_mask)
    bool any_left = false;
    for (int j = tid; j < p.L; j += blockDim.x) any_left |= np[j] && !p.left_mask[(size_t)a * p.L + j];
    int lo = M, hi = 0;
    for (int s = tid; s < M; s += blockDim.x) {
        const int c = p.nodes[s];
        const bool r_ok = np[c] && !p.right_mask[(size_t)a * p.L + c] && p.main_chain[c];
        right_ok[s] = r_ok;
        if (r_ok) {
            lo = min(lo, s);
            hi = s + 1;
        }
    }
    // ab[k][h]: one warp per head at a time, lanes over the chunk dimension
    const int left1 = a >= 1 ? a - 1 : 0;  // the reference's _max_left_index[a][1]
    const bool ok_left0 = np[0] && !p.left_mask[(size_t)a * p.L + 0];
    const bool ok_left1 = np[left1] && !p.left_mask[(size_t)a * p.L + left1];
    for (int h = warp; h < p.H; h += n_warps) {
        const size_t bh = (size_t)row.b * p.H + h;
        const float *qa = p.qm + (bh * M + sa) * p.D;
        const float *k0 = p.klm + bh * (M + 1) * p.D, *k1 = k0 + (size_t)(1 + sa) * p.D;
        float d0 = 0.f, d1 = 0.f;
        for (int d = lane; d < p.D; d += 32) {
            const float x = qa[d];
            d0 = fmaf(x, k0[d], d0);
            d1 = fmaf(x, k1[d], d1);
        }
        d0 = warp_sum_f(d0);
        d1 = warp_sum_f(d1);
        if (lane == 0) {
            s_ab[0][h] = ok_left0 ? d0 * p.scale : neg_inf();
            s_ab[1][h] = ok_left1 ? d1 * p.scale : neg_inf();
        }
    }
    if (warp == n_warps - 1) {  // log-softmax of the gate logits over the heads
        const float gt = lane < p.H ? p.gates[((size_t)row.b * p.L + a) * p.H + lane] : neg_inf();
        const float mx = warp_max_f(gt);
        const float sum = warp_sum_f(lane < p.H ? expf(gt - mx) : 0.f);
        if (lane < p.H) s_lg[lane] = gt - (mx + logf(sum));
    }
    if (!__syncthreads_or(any_left)) return false;
    if (hi > 0) {
        atomicMin(&s_lo, lo);
        atomicMax(&s_hi, hi);
    }
    __syncthreads();
    row.lo = s_lo;
    row.hi = s_hi;
    if (row.lo >= row.hi) return false;
    // per head: the largest logit, then the exponentials relative to it and their sum
    for (int h = warp; h < p.H; h += n_warps) {
        float mx = neg_inf();
        for (int s = row.lo + lane; s < row.hi; s += 32) {
            const bool ok = right_ok[s];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float v = ok ? row.logit(h, k, s) : neg_inf();
                if constexpr (STAGED) row.e[((size_t)h * 2 + k) * M + s] = v;
                mx = fmaxf(mx, v);  // drops NaN
            }
        }
        mx = warp_max_f(mx);
        float sum = 0.f;
        for (int s = row.lo + lane; s < row.hi; s += 32) {
#pragma unroll
            for (int k = 0; k < 2; k++) {
                if constexpr (STAGED) {
                    float &cell = row.e[((size_t)h * 2 + k) * M + s];
                    cell = row.rel(cell, mx);
                    sum += cell;
                } else {
                    sum += right_ok[s] ? row.rel(row.logit(h, k, s), mx) : 0.f;
                }
            }
        }
        sum = warp_sum_f(sum);
        if (lane == 0) {
            const float lg = s_lg[h], gate = lg > neg_inf() ? expf(lg) : 0.f;  // NaN: the head counts nothing
            s_top[h] = mx;
            s_lse[h] = isinf(mx) ? mx : mx + logf(sum);
            s_inv[h] = sum > 0.f ? 1.f / sum : 0.f;
            s_c[h] = gate * s_inv[h];
        }
    }
    __syncthreads();
    return true;
}

// The mixture of a cell from the log-probabilities of its heads: largest term, and sum of the others relative to it.
template <class LogProb>
__device__ __forceinline__ float mixture_terms(int H, LogProb term, float &sum) {
    float mx = neg_inf();
    for (int h = 0; h < H; h++) mx = fmaxf(mx, term(h));  // drops NaN
    sum = 0.f;
    if (!isinf(mx))
        for (int h = 0; h < H; h++) {
            const float t = term(h);
            if (t > neg_inf()) sum += expf(t - mx);
        }
    return mx;
}

// One block per (sentence, node).  A cell takes one exponential per head, one FMA per head and one logarithm.  Bound by
// its instructions (64 % of the issue slots) and the five barriers of a row of a few hundred cells: rows of nodes that are not on the main chain, and
// slots outside the admissible range, cost nothing but their -inf.  90 sentences, M = 161, eight heads: 136 us; 190 us
// with two exponentials per cell and head, each from scores read again.  Against float64 the transitions are off by
// 2.3e-7 (rms; 2.8e-7 before).
template <bool STAGED>
__global__ void __launch_bounds__(256)
    links_from_scores_kernel(const RowArgs p, float *__restrict__ links) {
    extern __shared__ __align__(16) float s_e[];  // STAGED: [H][2][M] exponentials; then [M] bytes
    __shared__ float s_ab[2][kMaxHeads], s_top[kMaxHeads], s_lse[kMaxHeads], s_lg[kMaxHeads], s_c[kMaxHeads], s_inv[kMaxHeads];
    const int a = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
    float *out = links + ((size_t)b * p.L + a) * 2 * p.L;
    for (int i = tid; i < 2 * p.L; i += blockDim.x) out[i] = neg_inf();  // admissible cells are overwritten below
    const int sa = p.slot_of[a];
    if (sa < 0) return;  // not on the main chain: no right child at max_left == 1
    uint8_t *right_ok = reinterpret_cast<uint8_t *>(s_e + (STAGED ? (size_t)p.H * 2 * p.M : 0));
    Row<STAGED> row{p, a, b, sa, 0, 0, right_ok, s_e, s_ab, s_top};
    if (!links_row(row, right_ok, s_ab, s_top, s_lse, s_lg, s_c, s_inv)) return;
    const int span = row.hi - row.lo;
    for (int i = tid; i < 2 * span; i += blockDim.x) {
        const int k = i >= span, s = row.lo + i - k * span;
        if (!right_ok[s]) continue;
        float sum = 0.f;
#pragma unroll 8
        for (int h = 0; h < p.H; h++) sum = fmaf(row.exp_at(h, k, s), s_c[h], sum);
        float res;
        if (sum > kMixtureFloor) {
            res = logf(sum);
        } else {
            float rest;
            res = mixture_terms(p.H, [&](int h) { return (row.logit(h, k, s) - s_lse[h]) + s_lg[h]; }, rest);
            if (!isinf(res)) res += logf(rest);
            else res = neg_inf();
        }
        out[(size_t)k * p.L + p.nodes[s]] = res;
    }
}

// Which score cells anybody reads: those of (node, right child) pairs that the masks admit.  All null: every cell.
struct ScoreMasks {
    const uint8_t *nonpad, *right_mask, *main_chain;
    const int *nodes;
    int L;
};

// Asynchronous copies into shared memory (16 or 4 bytes), zero-filled where there is nothing to copy.
__device__ __forceinline__ void copy_async16(float *dst, const float *src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dsm_smem_u32(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_async4(float *dst, const float *src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dsm_smem_u32(dst)), "l"(src), "r"(in ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// C[b][h] = A[b][h] krm[b][h]^T for the rows of A = qm (M rows -> ac) and A = klm (M + 1 rows -> bc): float32, 128 x 64
// output tiles of the 2 M + 1 stacked rows, the D axis walked in chunks of 32 through shared memory, 8 x 4 outputs per
// thread: twelve 16-byte shared-memory loads per 128 FMAs, conflict-free at a pitch of 36 floats when a thread's rows
// and columns lie 16 apart.  A block makes the same tile of `heads` heads, one after the other, the next chunk (or
// head) in flight while this one is multiplied.  A tile without a cell that anybody reads (children at or below the
// parents, padding: six tiles in ten of a ragged batch) is left alone; the test looks at a quarter of the tile's pairs
// at a time, so that a tile in use rarely pays for more than that.  90 sentences, M = 161, 8 x 64 features: 172 us; 296 us with a block per
// head and nothing in flight, 384 us as 64 x 64 tiles of 4 x 4 outputs, every tile formed.
// ROWS: 128, or 64 for chains of at most 31 nodes, whose rows fit one tile of either (128 sentences of 29 nodes, 8 x 64
// features: 27 us, 41 us with 128 rows; of 12 nodes 26 and 39 us), and where 128 would leave SMs without a block (2
// sentences of 65 nodes: 8.4 and 11.8 us).
constexpr int kScoreCols = 64, kScoreK = 32, kScorePitch = kScoreK + 4;
template <int ROWS>
constexpr int kScoreStage = (ROWS + kScoreCols) * kScorePitch;  // floats; two of them
template <int ROWS>
__global__ void __launch_bounds__(256, ROWS == 128 ? 2 : 3)
    links_scores_kernel(const float *__restrict__ qm, const float *__restrict__ klm, const float *__restrict__ krm, int M,
                        int H, int D, int heads, int vec, ScoreMasks masks, float *__restrict__ ac, float *__restrict__ bc) {
    extern __shared__ __align__(16) float s_tiles[];
    const int groups = (H + heads - 1) / heads, b = blockIdx.z / groups, h0 = (blockIdx.z - b * groups) * heads;
    const int r0 = blockIdx.y * ROWS, c0 = blockIdx.x * kScoreCols, tid = threadIdx.x;
    if (masks.nonpad != nullptr) {
        __shared__ int s_row[ROWS], s_col[kScoreCols];  // node of a row or column; -1: nobody's, -2: every node's
        const uint8_t *np = masks.nonpad + (size_t)b * masks.L;
        if (tid < ROWS) {
            const int row = r0 + tid;
            // row M is the left option "none", which every node shares
            s_row[tid] = row > 2 * M ? -1 : row == M ? -2 : masks.nodes[row < M ? row : row - M - 1];
        } else if (tid < ROWS + kScoreCols) {
            const int s = c0 + tid - ROWS, c = s < M ? masks.nodes[s] : -1;
            s_col[tid - ROWS] = c >= 0 && np[c] && masks.main_chain[c] ? c : -1;
        }
        __syncthreads();
        bool needed = false;
        for (int part = 0; part < 4 && !needed; part++) {  // rows part, part + 4, ... of the tile
            bool mine = false;
#pragma unroll
            for (int i = 0; i < ROWS / 4 * kScoreCols / 256; i++) {
                const int at = tid + 256 * i, a = s_row[part + at / kScoreCols * 4], c = s_col[at % kScoreCols];
                if (a != -1 && c >= 0) mine |= a == -2 || !__ldg(masks.right_mask + (size_t)a * masks.L + c);
            }
            needed = __syncthreads_or(mine);
        }
        if (!needed) return;
    }
    const int tx = tid & 15, ty = tid >> 4;
    const int chunks = (D + kScoreK - 1) / kScoreK, steps = chunks * min(heads, H - h0);
    auto stage = [&](int step) {
        const size_t bh = (size_t)b * H + h0 + step / chunks;
        const int k0 = step % chunks * kScoreK;
        float *tile = s_tiles + (step & 1) * kScoreStage<ROWS>;  // rows of A, then rows of krm
        auto source = [&](int r, bool &in) {
            in = r < ROWS ? r0 + r <= 2 * M : c0 + r - ROWS < M;
            if (!in) return krm;
            const int row = r0 + r;
            return r >= ROWS ? krm + (bh * M + c0 + r - ROWS) * D
                                   : row < M ? qm + (bh * M + row) * D : klm + (bh * (M + 1) + row - M) * D;
        };
        if (vec) {
#pragma unroll
            for (int i = tid; i < (ROWS + kScoreCols) * (kScoreK / 4); i += 256) {
                const int r = i / (kScoreK / 4), k = i % (kScoreK / 4) * 4;
                bool in;
                const float *src = source(r, in);
                in &= k0 + k < D;
                copy_async16(tile + r * kScorePitch + k, in ? src + k0 + k : krm, in);
            }
        } else {
            for (int i = tid; i < (ROWS + kScoreCols) * kScoreK; i += 256) {
                const int r = i / kScoreK, k = i % kScoreK;
                bool in;
                const float *src = source(r, in);
                in &= k0 + k < D;
                copy_async4(tile + r * kScorePitch + k, in ? src + k0 + k : krm, in);
            }
        }
        copy_commit();
    };
    float acc[ROWS / 16][4] = {};
    stage(0);
    for (int step = 0; step < steps; step++) {
        copy_wait();
        __syncthreads();  // this chunk is there, and nobody reads the other buffer any more
        if (step + 1 < steps) stage(step + 1);
        const float *sa = s_tiles + (step & 1) * kScoreStage<ROWS>, *sb = sa + ROWS * kScorePitch;
#pragma unroll 2
        for (int k = 0; k < kScoreK; k += 4) {
            float4 b4[4];
#pragma unroll
            for (int j = 0; j < 4; j++) b4[j] = *reinterpret_cast<const float4 *>(sb + (tx + 16 * j) * kScorePitch + k);
#pragma unroll
            for (int i = 0; i < ROWS / 16; i++) {
                const float4 a4 = *reinterpret_cast<const float4 *>(sa + (ty + 16 * i) * kScorePitch + k);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    acc[i][j] = fmaf(a4.x, b4[j].x, acc[i][j]);
                    acc[i][j] = fmaf(a4.y, b4[j].y, acc[i][j]);
                    acc[i][j] = fmaf(a4.z, b4[j].z, acc[i][j]);
                    acc[i][j] = fmaf(a4.w, b4[j].w, acc[i][j]);
                }
            }
        }
        if ((step + 1) % chunks == 0) {
            const size_t bh = (size_t)b * H + h0 + step / chunks;
#pragma unroll
            for (int i = 0; i < ROWS / 16; i++) {
                const int row = r0 + ty + 16 * i;
                float *out = row < M ? ac + (bh * M + row) * M : bc + (bh * (M + 1) + (row - M)) * M;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (row <= 2 * M && c0 + tx + 16 * j < M) out[c0 + tx + 16 * j] = acc[i][j];
                    acc[i][j] = 0.f;
                }
            }
        }
    }
}

// Gradient of the logits of one (sentence, node) row.  With G = links_grad[a][k][c], e and c as above, and
// w = G / sum_h e[h] c[h]:
//   d lp[k][c][h] = w e[h] c[h]                               (G times the share of head h in the mixture)
//   Gs[h] = sum_{k,c} d lp[k][c][h]                           (= d lg[h])
//   d logit[k][c][h] = d lp[k][c][h] - e[h] / sum e[h] Gs[h]
// written scaled by 1/sqrt(D) (the logits are scaled dot products) as X0 (k = 0) and X1 (k = 1) [B][H][M][M] at row
// slot(a); dab [B][H][M][2] = their row sums; dgates[a][h] = Gs[h] - softmax(gates)[h] sum_h' Gs[h'].  Rows of nodes
// that are not on the main chain, or have no admissible child, are zero (X rows) / zero (dgates).  A head with a
// logit of +inf gets NaN, as its gradient is undefined.  300 us at the size above, 562 us with the shares of a cell
// formed twice from log-probabilities; feature gradients off by 2.2e-7 of their norm (3.3e-7 before).
// KEEP: what stays in shared memory: 2 = e and w, 1 = w, 0 = neither (formed again when needed).
template <int KEEP>
__global__ void __launch_bounds__(256)
    links_scores_grad_kernel(const RowArgs p, const float *__restrict__ links_grad, float *__restrict__ X0,
                             float *__restrict__ X1, float *__restrict__ dab, float *__restrict__ dgates) {
    constexpr bool STAGED = KEEP == 2;
    extern __shared__ __align__(16) float s_e[];  // [H][2][M] exponentials; w [2][M]; bytes: [M], and [2][M] beside w
    __shared__ float s_ab[2][kMaxHeads], s_top[kMaxHeads], s_lse[kMaxHeads], s_lg[kMaxHeads], s_c[kMaxHeads], s_inv[kMaxHeads];
    __shared__ float s_gs[kMaxHeads];
    const int a = blockIdx.x, b = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = blockDim.x >> 5;
    const int M = p.M, H = p.H;
    float *dg = dgates + ((size_t)b * p.L + a) * H;
    const int sa = p.slot_of[a];
    float *s_w = s_e + (STAGED ? (size_t)H * 2 * M : 0);
    uint8_t *right_ok = reinterpret_cast<uint8_t *>(s_w + (KEEP ? 2 * M : 0)), *s_rare = right_ok + M;
    Row<STAGED> row{p, a, b, sa, 0, 0, right_ok, s_e, s_ab, s_top};
    if (sa < 0 || !links_row(row, right_ok, s_ab, s_top, s_lse, s_lg, s_c, s_inv)) {
        for (int h = tid; h < H; h += blockDim.x) dg[h] = 0.f;
        if (sa < 0) return;
        for (int i = tid; i < H * M; i += blockDim.x) {
            const size_t at = (((size_t)b * H + i / M) * M + sa) * M + i % M;
            X0[at] = 0.f;
            X1[at] = 0.f;
        }
        for (int i = tid; i < 2 * H; i += blockDim.x) dab[(((size_t)b * H + i / 2) * M + sa) * 2 + (i & 1)] = 0.f;
        return;
    }
    auto term = [&](int h, int k, int s) { return (row.logit(h, k, s) - s_lse[h]) + s_lg[h]; };
    const float *grow = links_grad + ((size_t)b * p.L + a) * 2 * p.L;
    // w of an admissible cell, or G itself (rare) below the floor of the mixture and where w leaves the floats
    auto weigh = [&](int k, int s, bool &rare) {
        rare = false;
        const float G = grow[(size_t)k * p.L + p.nodes[s]];
        if (G == 0.f) return 0.f;
        float sum = 0.f;
#pragma unroll 8
        for (int h = 0; h < H; h++) sum = fmaf(row.exp_at(h, k, s), s_c[h], sum);
        const float w = G / sum;
        rare = !(sum > kMixtureFloor && fabsf(w) < CUDART_INF_F);
        return rare ? G : w;
    };
    if constexpr (KEEP > 0) {
        const int span = row.hi - row.lo;
        for (int i = tid; i < 2 * span; i += blockDim.x) {
            const int k = i >= span, s = row.lo + i - k * span;
            bool rare = false;
            s_w[k * M + s] = right_ok[s] ? weigh(k, s, rare) : 0.f;
            s_rare[k * M + s] = rare;
        }
        __syncthreads();
    }
    // d lp of a cell: w e c, or formed from the log-probabilities where that is out of range (-inf cells: nothing)
    auto share = [&](int h, int k, int s, float e) {
        float w;
        bool rare;
        if constexpr (KEEP > 0) {
            w = s_w[k * M + s];
            rare = s_rare[k * M + s];
        } else {
            w = weigh(k, s, rare);
        }
        if (!rare) return w * (e * s_c[h]);
        float sum;
        const float mx = mixture_terms(H, [&](int i) { return term(i, k, s); }, sum), t = term(h, k, s);
        return !isinf(mx) && t > neg_inf() ? w * expf(t - mx) / sum : 0.f;
    };
    for (int h = warp; h < H; h += n_warps) {
        float gs = 0.f;
        for (int s = row.lo + lane; s < row.hi; s += 32) {
            if (!right_ok[s]) continue;
#pragma unroll
            for (int k = 0; k < 2; k++) gs += share(h, k, s, row.exp_at(h, k, s));
        }
        gs = warp_sum_f(gs);
        const float back = s_top[h] < CUDART_INF_F ? gs * s_inv[h] : CUDART_NAN_F;  // Gs / sum e
        float sums[2] = {0.f, 0.f};
        const size_t at = (((size_t)b * H + h) * M + sa) * M;
        for (int s = lane; s < M; s += 32) {
            const bool ok = s >= row.lo && s < row.hi && right_ok[s];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                float d = 0.f;
                if (ok) {
                    const float e = row.exp_at(h, k, s);
                    d = (share(h, k, s, e) - e * back) * p.scale;
                }
                (k ? X1 : X0)[at + s] = d;
                sums[k] += d;
            }
        }
        sums[0] = warp_sum_f(sums[0]);
        sums[1] = warp_sum_f(sums[1]);
        if (lane == 0) {
            s_gs[h] = gs;
            dab[(((size_t)b * H + h) * M + sa) * 2 + 0] = sums[0];
            dab[(((size_t)b * H + h) * M + sa) * 2 + 1] = sums[1];
        }
    }
    __syncthreads();
    if (warp == n_warps - 1) {  // gate logits: d lg - softmax(gates) sum d lg
        const float tot = warp_sum_f(lane < H ? s_gs[lane] : 0.f);
        if (lane < H) dg[lane] = s_gs[lane] - expf(s_lg[lane]) * tot;
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
// Four float32 matrix products, M x M x D each, per (sentence, head).  A block makes ROWS rows x 64 columns of d of the
// parents' two products (role 0) or of the children's two (role 1), 4 x 4 outputs of both per thread, the summed index
// walked in chunks of 32 through shared memory (the next chunk in flight while this one is multiplied): three 16-byte
// shared-memory loads per 32 FMAs, and no shape is too large for it.  The X matrices are zero wherever a child is not
// admissible (all children at or below the parent, padding): a chunk whose X are all zero is skipped, unless the
// features beside it are not finite (0 x inf stays NaN).  90 sentences, M = 161, 8 x 64 features: 284 us (366 us
// without the next chunk in flight); 3 095 us with one thread per output reading its operands from global memory, as
// it was.
// ROWS: rows of a tile, 64, or 32 or 16 where the chain has no more nodes (128 sentences of 29 nodes: 34 us, 54 us with 64
// rows; of 12 nodes: 20 and 51 us); four threads per row.
constexpr int kFgTile = 64, kFgChunk = 32, kFgPitch = kFgChunk + 4;
constexpr int fg_stage(int rows) { return 2 * kFgChunk * (rows + kFgTile); }  // floats of a chunk: role 1, the larger one
constexpr int fg_stages(int rows) { return rows > kFgChunk ? 2 : 1; }         // chains up to 32 nodes are one chunk
constexpr size_t fg_smem(int rows) { return (fg_stages(rows) * fg_stage(rows) + 4 * rows) * sizeof(float); }

__device__ __forceinline__ bool not_finite(float x) { return !(fabsf(x) < CUDART_INF_F); }

// rows r0 .. r0 + 31 (< rows), columns d0 .. d0 + 63 (< D) of src [rows][D] into dst [32][64], zero outside
template <int THREADS>
__device__ __forceinline__ void stage_features(const float *__restrict__ src, int r0, int rows, int d0, int D, bool vec,
                                               float *dst) {
    if (vec) {
#pragma unroll
        for (int i = threadIdx.x; i < kFgChunk * kFgTile / 4; i += THREADS) {
            const int r = r0 + i / (kFgTile / 4), d = d0 + i % (kFgTile / 4) * 4;
            const bool in = r < rows && d < D;
            copy_async16(dst + 4 * i, in ? src + (size_t)r * D + d : src, in);
        }
    } else {
        for (int i = threadIdx.x; i < kFgChunk * kFgTile; i += THREADS) {
            const int r = r0 + i / kFgTile, d = d0 + i % kFgTile;
            const bool in = r < rows && d < D;
            copy_async4(dst + i, in ? src + (size_t)r * D + d : src, in);
        }
    }
}
// whether what this thread staged there has an infinity or a NaN
template <int THREADS>
__device__ __forceinline__ bool staged_not_finite(const float *dst, bool vec) {
    bool odd = false;
#pragma unroll
    for (int j = 0; j < kFgChunk * kFgTile / THREADS; j++)
        odd |= not_finite(vec ? dst[4 * (threadIdx.x + j / 4 * THREADS) + j % 4] : dst[threadIdx.x + j * THREADS]);
    return odd;
}

__device__ __forceinline__ float part(const float4 &v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; }

// vec: D a multiple of 4 and the feature matrices on 16-byte boundaries
template <int ROWS>
__global__ void __launch_bounds__(4 * ROWS, 2 * (64 / ROWS))
    links_features_grad_kernel(const float *__restrict__ X0, const float *__restrict__ X1, const float *__restrict__ dab,
                               const float *__restrict__ qm, const float *__restrict__ klm, const float *__restrict__ krm,
                               const int *__restrict__ nodes, int M, int L, int H, int D, int vec, float *__restrict__ dq,
                               float *__restrict__ dkl, float *__restrict__ dkr) {
    extern __shared__ __align__(16) float s_tiles[];
    constexpr int THREADS = 4 * ROWS, STAGE = fg_stage(ROWS);
    // blocks by (sentence, head), tile of d, tile of rows, role: along x, which alone takes more than 65 535
    const unsigned per_d = 2 * ((M + ROWS - 1) / ROWS), d_tiles = (D + kFgTile - 1) / kFgTile;
    const unsigned at_d = blockIdx.x / per_d, at_r = blockIdx.x - at_d * per_d;
    const int role = at_r & 1, r0 = (at_r >> 1) * ROWS, d0 = at_d % d_tiles * kFgTile;
    const size_t bh = at_d / d_tiles;
    const int b = (int)bh / H, h = (int)bh - b * H;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const float *x0 = X0 + bh * M * M, *x1 = X1 + bh * M * M;
    const float *q = qm + bh * M * D, *kl = klm + bh * (M + 1) * D, *kr = krm + bh * M * D;
    const size_t pitch = (size_t)H * D, base = (size_t)b * L * pitch + (size_t)h * D;
    float acc0[4][4] = {}, acc1[4][4] = {};
    const int chunks = (M + kFgChunk - 1) / kFgChunk;
    if (role == 0) {  // rows are parents a; summed over the children s
        constexpr int kX1 = ROWS * kFgPitch, kK = 2 * kX1;  // X0, X1 [ROWS][36] and krm [32][64] in a stage
        auto stage = [&](int step) {
            const int s0 = step * kFgChunk;
            float *tile = s_tiles + (step & 1) * STAGE;
#pragma unroll
            for (int i = tid; i < ROWS * kFgChunk; i += THREADS) {
                const int r = i / kFgChunk, s = i % kFgChunk;
                const bool in = r0 + r < M && s0 + s < M;
                const size_t at = in ? (size_t)(r0 + r) * M + s0 + s : 0;
                copy_async4(tile + r * kFgPitch + s, x0 + at, in);
                copy_async4(tile + kX1 + r * kFgPitch + s, x1 + at, in);
            }
            stage_features<THREADS>(kr, s0, M, d0, D, vec, tile + kK);
            copy_commit();
        };
        stage(0);
        for (int step = 0; step < chunks; step++) {
            const float *sx0 = s_tiles + (step & 1) * STAGE, *sx1 = sx0 + kX1, *sk = sx0 + kK;
            copy_wait();
            bool work = staged_not_finite<THREADS>(sk, vec);  // a thread looks at what it copied itself: no barrier in between
#pragma unroll
            for (int i = tid; i < ROWS * kFgChunk; i += THREADS) {
                const int at = i / kFgChunk * kFgPitch + i % kFgChunk;
                work |= sx0[at] != 0.f || sx1[at] != 0.f;
            }
            work = __syncthreads_or(work);  // the chunk is there, and nobody reads the other buffer any more
            if (step + 1 < chunks) stage(step + 1);
            if (!work) continue;
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
        float *red = s_tiles;
#pragma unroll
        for (int c = 0; c < 4; c++) red[ty * kFgTile + 4 * tx + c] = kl0_part[c];
        __syncthreads();
        if (tid < kFgTile && d0 + tid < D) {
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < ROWS / 4; i++) sum += red[i * kFgTile + tid];
            atomicAdd(dkl + base + d0 + tid, sum);
        }
    } else {  // rows are children s; summed over the parents a
        constexpr int kX = kFgChunk * ROWS, kPart = kFgChunk * kFgTile;  // X0 (then X0 + X1), X1 [32][ROWS], qm, klm [32][64] in a stage
        float *sums = s_tiles + fg_stages(ROWS) * STAGE;  // [4][ROWS]
        const int own = tid % ROWS, a_own = tid / ROWS, s_own = r0 + own;  // the column whose X this thread stages
        float x0sum = 0.f;                                // its sum of X0 over a = a_own + 4 j
        auto stage = [&](int step) {
            const int a0 = step * kFgChunk;
            float *tile = s_tiles + (step & 1) * STAGE;
#pragma unroll
            for (int j = 0; j < kFgChunk / 4; j++) {
                const int a = a_own + 4 * j;
                const bool in = a0 + a < M && s_own < M;
                const size_t at = in ? (size_t)(a0 + a) * M + s_own : 0;
                copy_async4(tile + a * ROWS + own, x0 + at, in);
                copy_async4(tile + kX + a * ROWS + own, x1 + at, in);
            }
            stage_features<THREADS>(q, a0, M, d0, D, vec, tile + 2 * kX);
            stage_features<THREADS>(kl + D, a0, M, d0, D, vec, tile + 2 * kX + kPart);
            copy_commit();
        };
        stage(0);
        for (int step = 0; step < chunks; step++) {
            float *sxs = s_tiles + (step & 1) * STAGE;
            const float *sx1 = sxs + kX, *sq = sxs + 2 * kX, *sk = sq + kPart;
            copy_wait();
            bool work = staged_not_finite<THREADS>(sq, vec) || staged_not_finite<THREADS>(sk, vec);
#pragma unroll
            for (int j = 0; j < kFgChunk / 4; j++) {
                const int at = (a_own + 4 * j) * ROWS + own;
                const float v0 = sxs[at], v1 = sx1[at];
                work |= v0 != 0.f || v1 != 0.f;
                x0sum += v0;
                sxs[at] = v0 + v1;
            }
            work = __syncthreads_or(work);
            if (step + 1 < chunks) stage(step + 1);
            if (!work) continue;
#pragma unroll 4
            for (int a = 0; a < kFgChunk; a++) {
                const float4 xs = *reinterpret_cast<const float4 *>(sxs + a * ROWS + 4 * ty);
                const float4 xb = *reinterpret_cast<const float4 *>(sx1 + a * ROWS + 4 * ty);
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
        sums[a_own * ROWS + own] = x0sum;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = r0 + 4 * ty + i;
            if (r >= M) continue;
            const int t = 4 * ty + i;
            const float w = (sums[t] + sums[ROWS + t]) + (sums[2 * ROWS + t] + sums[3 * ROWS + t]);
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

static bool on_16_bytes(std::initializer_list<const void *> ptrs) {
    uintptr_t all = 0;
    for (const void *p : ptrs) all |= reinterpret_cast<uintptr_t>(p);
    return (all & 15) == 0;
}

// nonpad == nullptr: every cell is formed
int launch_links_scores(const float *qm, const float *klm, const float *krm, const uint8_t *nonpad, const uint8_t *right_mask,
                        const uint8_t *main_chain, const int *nodes, int L, int M, int B, int H, int D, float *ac, float *bc,
                        cudaStream_t st) {
    if (B == 0 || M == 0) return PCFGNAT_OK;
    const int vec = D % 4 == 0 && on_16_bytes({qm, klm, krm});
    const int cols = (M + kScoreCols - 1) / kScoreCols;
    const bool small = 2 * M + 1 <= 64 || (long long)cols * ((2 * M + 1 + 127) / 128) * B * H < sm_count();
    const int rows = small ? 64 : 128;
    const dim3 tiles(cols, (2 * M + 1 + rows - 1) / rows);
    // up to four heads per block (the test for tiles in use and the first chunk's latency are paid once), as long as
    // there are four blocks for every place on the GPU: tiles that are not in use leave at once
    int heads = 4;
    while (heads > 1 && (long long)tiles.x * tiles.y * B * ((H + heads - 1) / heads) < 4ll * 2 * sm_count()) heads /= 2;
    const auto launch = [&](auto kernel, size_t smem) {
        if (ensure_dynamic_smem(kernel, smem) != cudaSuccess) return PCFGNAT_ERR_CUDA;
        kernel<<<dim3(tiles.x, tiles.y, B * ((H + heads - 1) / heads)), 256, smem, st>>>(
            qm, klm, krm, M, H, D, heads, vec, ScoreMasks{nonpad, right_mask, main_chain, nodes, L}, ac, bc);
        return cuda_rc(cudaGetLastError());
    };
    return small ? launch(links_scores_kernel<64>, 2 * kScoreStage<64> * sizeof(float))
                 : launch(links_scores_kernel<128>, 2 * kScoreStage<128> * sizeof(float));
}

int launch_links_backward(const float *links_grad, const float *ac, const float *bc, const float *qm, const float *klm,
                          const float *krm, const float *gates, const uint8_t *nonpad, const uint8_t *left_mask,
                          const uint8_t *right_mask, const uint8_t *main_chain, const int *slot_of, const int *nodes, int M,
                          int B, int L, int H, int D, float *X0, float *X1, float *dab, float *dq, float *dkl, float *dkr,
                          float *dgates, cudaStream_t st) {
    if (B == 0) return PCFGNAT_OK;
    if (H > kMaxHeads) return PCFGNAT_ERR_TOO_LARGE;
    const RowArgs row{ac, bc, qm, klm, gates, nonpad, left_mask, right_mask, main_chain, slot_of, nodes, M, L, H, D,
                      1.f / sqrtf((float)D)};
    if ((size_t)M > 40 * 1024) return PCFGNAT_ERR_TOO_LARGE;
    const size_t staged = (size_t)H * 2 * M * sizeof(float), w = (size_t)2 * M * sizeof(float) + 3 * (size_t)M;
    if (staged + w <= kRowSmem)
        links_scores_grad_kernel<2><<<dim3(L, B), row_threads(H), staged + w, st>>>(row, links_grad, X0, X1, dab, dgates);
    else if (w <= kRowSmem)
        links_scores_grad_kernel<1><<<dim3(L, B), row_threads(H), w, st>>>(row, links_grad, X0, X1, dab, dgates);
    else
        links_scores_grad_kernel<0><<<dim3(L, B), row_threads(H), (size_t)M, st>>>(row, links_grad, X0, X1, dab, dgates);
    if (cudaGetLastError() != cudaSuccess) return PCFGNAT_ERR_CUDA;
    if (M == 0) return PCFGNAT_OK;
    const int vec = D % 4 == 0 && on_16_bytes({qm, klm, krm});
    const auto launch = [&](auto kernel, int rows) {
        const long long grid = 2ll * ((M + rows - 1) / rows) * ((D + kFgTile - 1) / kFgTile) * B * H;
        if (grid > INT32_MAX) return PCFGNAT_ERR_TOO_LARGE;
        if (ensure_dynamic_smem(kernel, fg_smem(rows)) != cudaSuccess) return PCFGNAT_ERR_CUDA;
        kernel<<<(unsigned)grid, 4 * rows, fg_smem(rows), st>>>(X0, X1, dab, qm, klm, krm, nodes, M, L, H, D, vec, dq, dkl, dkr);
        return cuda_rc(cudaGetLastError());
    };
    return M <= 16   ? launch(links_features_grad_kernel<16>, 16)
           : M <= 32 ? launch(links_features_grad_kernel<32>, 32)
                     : launch(links_features_grad_kernel<64>, 64);
}

int launch_links_gather(const void *q, const void *kl, const void *kr, int is_half, const int *nodes, int M, int B, int L,
                        int H, int D, float *qm, float *klm, float *krm, cudaStream_t st) {
    if (B == 0) return PCFGNAT_OK;
    const bool vec = D % 4 == 0 && on_16_bytes({q, kl, kr, qm, klm, krm});
    const long long items = (long long)(M + 1) * H * D / (vec ? 4 : 1);
    if (items > INT32_MAX - 256) return PCFGNAT_ERR_TOO_LARGE;
    const dim3 grid((unsigned)((items + 255) / 256), B);
    if (vec)
        links_gather_kernel<true><<<grid, 256, 0, st>>>(q, kl, kr, is_half, nodes, M, L, H, D, qm, klm, krm);
    else
        links_gather_kernel<false><<<grid, 256, 0, st>>>(q, kl, kr, is_half, nodes, M, L, H, D, qm, klm, krm);
    return cuda_rc(cudaGetLastError());
}

int launch_links_from_scores(const float *ac, const float *bc, const float *qm, const float *klm, const float *gates,
                             const uint8_t *nonpad, const uint8_t *left_mask, const uint8_t *right_mask,
                             const uint8_t *main_chain, const int *slot_of, const int *nodes, int M, int B, int L, int H,
                             int D, float *links, cudaStream_t st) {
    if (B == 0) return PCFGNAT_OK;
    if (H > kMaxHeads) return PCFGNAT_ERR_TOO_LARGE;
    if ((size_t)M > 40 * 1024) return PCFGNAT_ERR_TOO_LARGE;
    const RowArgs row{ac, bc, qm, klm, gates, nonpad, left_mask, right_mask, main_chain, slot_of, nodes, M, L, H, D,
                      1.f / sqrtf((float)D)};
    const size_t staged = (size_t)H * 2 * M * sizeof(float);
    if (staged + M <= kRowSmem)
        links_from_scores_kernel<true><<<dim3(L, B), row_threads(H), staged + M, st>>>(row, links);
    else
        links_from_scores_kernel<false><<<dim3(L, B), row_threads(H), M, st>>>(row, links);
    return cuda_rc(cudaGetLastError());
}

}  // namespace pcfgnat
