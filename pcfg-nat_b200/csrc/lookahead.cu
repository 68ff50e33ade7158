// Lookahead and greedy decoding (fs_plugins/models/glat_decomposed_with_link_two_hands_tri_pcfg.py:419-482) on the
// device, one launch: the reference forms links_lookahead [B, L, 2, L] with torch operators, takes its arg-max per
// node, copies the indices to the host (.cpu().tolist()) and walks the tree in a Python loop per sentence.
//
// Per node a the choice is the first maximum over (k, c), k-major (index k * L + c), of
//     lookahead:  (links[a][k][c] + ob[c] * beta) + ob[left(a, k)] * beta,   left(a, 0) = 0, left(a, k) = max(a - k, 0)
//     greedy:      links[a][k][c]
// in float32 with the reference's association (models/...pcfg.py:422-428, :431).  The walk is the reference's
// in-order traversal (:435-478): from node 1 descend to the chosen left child (k == 0: node 0; else a - k) unless
// left_tree_mask forbids it, emit the node's token unless it is padding (consecutive equal tokens are NOT merged
// here, unlike the Viterbi back-trace), continue with the chosen right child; node 0 or a node at or beyond the
// sentence's length ends a branch.
//
// The reference's lookahead term for the left child is gathered from unreduced_logits.unsqueeze(1).repeat(bsz,
// prelen, 1) with an index of batch extent 1 (:425), which for bsz > 1 hands every sentence the log-probabilities of
// sentence 0; its published lookahead decoding runs with batch size 1, where that is the sentence's own.  Here every
// sentence uses its own log-probabilities.
//
// A cluster of up to eight CTAs serves a sentence.  Its warps take the nodes in use (1 .. length - 1), read a node's
// 2 L transitions, eight loads in flight per lane, and leave in the first CTA's shared memory one word per node: the
// chosen child and left option, whether the walk may descend there (left_tree_mask), whether the token is emitted.
// One thread of the first CTA then walks on that table alone; what it visits it notes as node numbers in the output,
// which the block turns into tokens at the end.  The walk is a chain of shared-memory loads (the mask and token loads
// it used to wait for, one L2 round trip each per node, are made by the warps beforehand), and the scan of the
// transitions is spread over the GPU also when there are few sentences.  64 sentences, graph 240: 21 us, 220 us with a
// block per sentence whose walk read the mask and the tokens.
#include <cooperative_groups.h>

#include <climits>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace pcfgnat {

namespace {

constexpr int kLookThreads = 256, kLookWarps = kLookThreads / 32;
constexpr int kLookNodesPerCta = 16, kLookCluster = 8;

// word of a node: chosen child in the low bits, and
constexpr int kLookChild = (1 << 28) - 1;
constexpr int kLookLeft = 1 << 28;   // left option 1 (node a - 1), else 0 (node 0)
constexpr int kLookStop = 1 << 29;   // left_tree_mask forbids the descent
constexpr int kLookBad = 1 << 30;    // outside the mask
constexpr int kLookEmit = 1 << 31;   // the token is not padding

__global__ void __launch_bounds__(kLookThreads)
    lookahead_decode_kernel(const float *__restrict__ links, const float *__restrict__ ob, const int64_t *__restrict__ tokens,
                            const int64_t *__restrict__ ol, const int64_t *__restrict__ mask, int mask_dim, float beta,
                            int lookahead, int64_t pad, int L, int cap, int64_t *out, int64_t *cnt, int *status) {
    // first CTA: [L] words of the nodes, then [L] the walk's stack; node 0 has none, its word takes the number of tokens
    extern __shared__ int s_node[];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), nc = (int)cluster.num_blocks();
    const int b = blockIdx.x / nc;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float *lkb = links + (size_t)b * L * 2 * L;
    const float *obb = ob + (size_t)b * L;
    const int64_t given = ol[b];
    const bool fits = given >= 0 && given <= L;
    const int length = fits ? (int)given : 0;
    int *words = cluster.map_shared_rank(s_node, 0);
    // Another CTA's shared memory exists once that CTA has started: the cluster meets before the first store into it.
    // The barrier is split, so that a warp's first node is scanned meanwhile.
    cluster.barrier_arrive();
    bool met = false;  // uniform over the warp
    for (int a = 1 + rank * kLookWarps + warp; a < length; a += nc * kLookWarps) {
        const float *row = lkb + (size_t)a * 2 * L;
        // products and sums rounded one by one, as the reference's element-wise operators do it: fused, a near-tie may
        // go to another child
        const float left0 = lookahead ? __fmul_rn(obb[0], beta) : 0.f, left1 = lookahead ? __fmul_rn(obb[a - 1], beta) : 0.f;
        float best = neg_inf();
        int key = INT_MAX;
        for (int i0 = lane; i0 < 2 * L; i0 += 8 * 32) {  // a lane sees its candidates in increasing index order
            float v[8], o[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int i = i0 + 32 * j;
                v[j] = i < 2 * L ? __ldg(row + i) : CUDART_NAN_F;
                o[j] = lookahead && i < 2 * L ? __ldg(obb + (i >= L ? i - L : i)) : 0.f;
            }
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int i = i0 + 32 * j;
                const float x = lookahead ? __fadd_rn(__fadd_rn(v[j], __fmul_rn(o[j], beta)), i >= L ? left1 : left0) : v[j];
                if (x > best || (key == INT_MAX && !isnan(x))) {  // strict: the first maximum stays; -inf counts as a value
                    best = x;
                    key = i;
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int ok = __shfl_xor_sync(0xffffffffu, key, o);
            if (ok != INT_MAX && (key == INT_MAX || ov > best || (ov == best && ok < key))) {
                best = ov;
                key = ok;
            }
        }
        if (!met) cluster.barrier_wait();
        met = true;
        if (lane == 0) {
            if (key == INT_MAX) key = 0;
            const int k = key >= L, left = k ? a - 1 : 0;
            int word = (key - k * L) | (k ? kLookLeft : 0);
            if (a >= mask_dim) word |= kLookBad;  // left < a
            else if (mask[(size_t)a * mask_dim + left]) word |= kLookStop;
            if (tokens[(size_t)b * L + a] != pad) word |= kLookEmit;
            words[a] = word;
        }
    }
    if (!met) cluster.barrier_wait();  // a warp without a node
    cluster.sync();                    // the words are there
    if (rank != 0) return;
    int64_t *o = out + (size_t)b * cap;
    if (tid == 0) {
        int *stack = s_node + L;
        int sp = 0, count = 0, now = 1;
        bool bad = !fits;
        long guard = 0;
        while (!bad && ((now < length && now != 0) || sp > 0)) {
            while (now < length && now != 0) {
                if (sp >= L || ++guard > 4L * L + 16) {
                    bad = true;
                    break;
                }
                stack[sp++] = now;
                const int word = s_node[now];
                if (word & kLookBad) {
                    bad = true;
                    break;
                }
                if (word & kLookStop) break;
                now = word & kLookLeft ? now - 1 : 0;
            }
            if (bad || sp == 0) break;
            now = stack[--sp];
            const int word = s_node[now];
            if (word & kLookEmit) {
                if (count < cap) o[count] = now;
                count++;
            }
            now = word & kLookChild;
        }
        if (bad) flag(status, PCFGNAT_STATUS_BAD_TRACE);
        s_node[0] = count < cap ? count : cap;
        cnt[b] = s_node[0];
    }
    __syncthreads();
    const int kept = s_node[0];
    for (int i = tid; i < cap; i += kLookThreads) o[i] = i < kept ? tokens[(size_t)b * L + o[i]] : pad;
}

}  // namespace

int launch_lookahead_decode(const float *links, const float *ob, const int64_t *tokens, const int64_t *ol,
                            const int64_t *mask, int mask_dim, float beta, int lookahead, int64_t pad, int B, int L,
                            int cap, int64_t *out, int64_t *cnt, int *status, cudaStream_t st) {
    if (B == 0) return PCFGNAT_OK;
    if (L > kLookChild) return PCFGNAT_ERR_TOO_LARGE;
    const size_t smem = (size_t)2 * L * sizeof(int);
    if (smem > 48 * 1024 && ensure_dynamic_smem(lookahead_decode_kernel, smem) != cudaSuccess) return PCFGNAT_ERR_TOO_LARGE;
    const int want = (L + kLookNodesPerCta - 1) / kLookNodesPerCta, nc = want < kLookCluster ? want : kLookCluster;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)B * nc);
    cfg.blockDim = dim3(kLookThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = nc;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cuda_rc(cudaLaunchKernelEx(&cfg, lookahead_decode_kernel, links, ob, tokens, ol, mask, mask_dim, beta, lookahead,
                                      pad, L, cap, out, cnt, status));
}

}  // namespace pcfgnat
