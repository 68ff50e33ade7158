// Viterbi decode tables (max semiring over output lengths, with backpointers) and the
// back-trace, max_left == 1.
//
// viterbi_kernel replaces calculate_C_kernel / calculate_S_kernel of the reference
// (fs_plugins/custom_ops/pcfg_viterbi.cu:178-241, :23-140): one CTA per sentence loops over
// the output length inside the kernel (the reference spins on a global counter between
// lengths).  With max_left == 1 the two live expansions of node a at length len are
//     t0 = ((links[a][0][c] + 0) + S[c][len-1]) + ob[a]                (j = 0, no left child)
//     t1 = ((links[a][1][c] + ob[a-1]) + S[c][len-2]) + ob[a]          (j = 1, leaf a-1)
// The reference gives node id four threads x = 0..3; thread x scans c_id = id + x + 4k in increasing
// k, t0 before t1, under strict '>', and the four are merged with shfl_down 2 then 1 under strict
// '>'.  A maximum is order-free except for ties, so here G = 4 to 16 lanes own the node (lane q scans
// c_id = id + q + G i, which is reference thread x = q & 3) and the reference's choice among equal
// values is reproduced by an explicit tie key: thread priority 0 > 2 > 1 > 3, then the smaller c,
// then j = 0 before j = 1.  Values and backpointers are bit-exact.  Tables are indexed by node id;
// R, Lt hold node ids (Lt = 0 for "no left child"), Mt holds j.
//
// viterbi_cluster_kernel spreads the nodes of a sentence over the CTAs of a thread-block cluster
// (one cluster per sentence, sized so that the batch fills the GPU): every CTA keeps the rolling
// columns of the whole chain, and the lanes that finish a node send its value into every CTA's copy with
// st.async, counted on a barrier of the receiving CTA.
// viterbi_global_kernel (one CTA per sentence, links read from global memory) takes the shapes
// whose links do not fit the cluster's shared memory.
//
// backtrace_kernel replaces the host function viterbi_decoding
// (fs_plugins/custom_ops/pcfg_loss.cpp:12-73): one thread per sentence (a block each, so that the
// walks run on different SMs) does the in-order walk with an explicit stack, skipping pad tokens and
// collapsing repeats.  The three table entries of a node are fetched together when it is stacked.
#include <cooperative_groups.h>

#include <climits>
#include <cstdlib>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace pcfgnat {

namespace {

constexpr int kVitThreads = 512;

// Monotone map float -> unsigned (no NaN reaches it); -0 is mapped like +0 so that, as under the
// reference's '>', neither beats the other.
__device__ __forceinline__ unsigned ordered_bits(float v) {
    const unsigned u = __float_as_uint(v == 0.f ? 0.f : v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Warp arg-max of (best, key) pairs: the largest value, among equal values the smallest key.
// Every lane returns the winner's value and key (key INT_MAX: nothing finite was seen).
__device__ __forceinline__ void warp_argmax(float &best, int &key, int lane) {
    const unsigned ord = ordered_bits(best);
    const unsigned top = __reduce_max_sync(0xffffffffu, ord);
    const unsigned k = __reduce_min_sync(0xffffffffu, ord == top ? (unsigned)key : 0xffffffffu);
    const unsigned holders = __ballot_sync(0xffffffffu, ord == top && (unsigned)key == k);
    best = __shfl_sync(0xffffffffu, best, holders ? __ffs(holders) - 1 : lane);
    key = (int)k;
}

// One step of node `id` for the lanes of a warp: children ci = id + lane + 32 i.
//   t0 = ((links[a][0][c] + 0) + S[c][len-1]) + ob[a]      (k0[ci] holds links[a][0][c] + 0)
//   t1 = ((links[a][1][c] + ob[a-1]) + S[c][len-2]) + ob[a] (k1[ci] holds links[a][1][c] + ob[a-1];
//        -inf for the first node, which has no leaf, so that t1 never wins there)
// A NaN term never wins a '>' either, which is what the reference's NaN -> -inf cleaning achieves.
template <class K0, class K1>
__device__ __forceinline__ void viterbi_node(int id, int Mb, int lane, int prio, float oa, const float *S1,
                                             const float *S2, K0 k0, K1 k1, float &best, int &key) {
    best = neg_inf();
    key = INT_MAX;  // (prio << 24) | (c_slot << 1) | j of the current best; smaller wins ties
    for (int ci = id + lane; ci < Mb; ci += 32) {
        const int kk = (prio << 24) | (ci << 1);
        const float t0 = (k0(ci) + S1[ci]) + oa;
        if (t0 > best) {
            best = t0;
            key = kk;
        }
        const float t1 = (k1(ci) + S2[ci]) + oa;
        if (t1 > best) {
            best = t1;
            key = kk | 1;
        }
    }
    warp_argmax(best, key, lane);
}

__device__ __forceinline__ void viterbi_store(float best, int key, int a, int Q, int len, float *Sb, int64_t *Rb,
                                              int64_t *Lb, int64_t *Mtb) {
    if (isinf(best)) return;  // cell stays at its initial value (pcfg_viterbi.cu:113-121)
    const int bj = key & 1, bc = 2 * ((key >> 1) & 0x7FFFFF) + 1;
    const size_t o = (size_t)a * Q + len;
    Sb[o] = best;
    Lb[o] = bj ? a - 1 : 0;
    Rb[o] = bc;
    Mtb[o] = bj;
}

// Lanes per node: as few as let a block's warps take all of its nodes in one pass.  60 nodes on 16 warps: 76 / 69 / 94 us with
// 4 / 8 / 16 lanes (64 sentences of 120 nodes); 16 nodes: 141 / 103 / 93, and 101 with 32 (16 sentences of 128).
__host__ __device__ inline int viterbi_lanes(int rows, int warps) {
    int G = 16;
    while ((32 / G) * warps < rows && G > 4) G >>= 1;
    return G;
}
// How far past the chain's last child they read, 32 children at a time, when 32 / G nodes NC apart share a warp's trips.
__host__ __device__ constexpr int viterbi_overshoot(int G, int NC) { return 31 + NC * (32 / G - 1); }

// The lengths of a sentence, G lanes per node: lane q takes children id + q + G i, so that its reference thread
// (ci - id) & 3 = q & 3 is one per lane, blocks of 32 children without a test: the columns hold -inf past the chain, and
// whatever lies behind a node's row gives -inf or NaN with it, which never wins.  Both kinds of terms go as pairs: a child's
// links lie side by side and so do S[len - 1] and S[len - 2] in column len (a node stores its value into two columns).  Peers wait
// for the value alone: the maximum is sent, and which term it was, with the reference's order of ties, is looked up in the held
// terms while it is on its way (the terms of a node's first 128 children; of further ones value and term are carried together, or
// in LONG chains, of more than 256 nodes, the value alone and the first 32 children that have it, whose terms are formed again:
// 530 nodes on sixteen CTAs 632 -> 588 us, eight sentences of 320 on eight 242 -> 228.
//
// Bound by the latency of a length (loads, the chain of maxima, shuffles, exchange and barrier).  With value and key carried
// through every comparison, 1024 threads and one load and addition per term before: 64 sentences of up to 120 nodes 82 -> 68 us,
// 24 of 128 74 -> 57, 56 of up to 160 144 -> 119, one of 256 on eight CTAs 175 -> 141.
template <int G, bool LONG>
__device__ __forceinline__ bool viterbi_lengths(float2 *col, const float2 *lk, const float *s_oa, float *own_v, uint16_t *own_k,
                                                uint64_t *col_bar, int n_len, int Mb, int my_rows, int NC, int crank, int Q,
                                                int cs, int pitch) {
    constexpr int R = 32 / G, U = 32 / G, HELD = 128 / G;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
    const int q = lane % G, sub = lane / G;
    const int prio = ((q & 1) << 1) | ((q >> 1) & 1);
    const int half = q & 1;  // lane q sends to CTA q / 2: the left halves of the pairs if even, the right halves if odd
    const uint32_t bar0 = dsm_smem_u32(col_bar), cells = dsm_smem_u32(col) + 4u * half;
    bool arrived = true;
    for (int len = 2; len < n_len; len++) {
        const float2 *pairs = col + (len & 3) * cs;
        const uint32_t bar = bar0 + 8u * (len & 1);
        if (NC > 1 && tid == 0)  // this CTA expects the whole column of this length: two copies of a value per node of the chain
            asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(bar), "r"(8 * Mb)
                         : "memory");
        for (int first = warp * R; first < my_rows; first += warps * R) {  // warp-uniform
            const bool live = first + sub < my_rows;
            const int r = live ? first + sub : first, id = crank + NC * r;
            const int trips = (Mb - (crank + NC * first) + G - 1) / G;  // of the warp's first node, which has most children
            const float oa = s_oa[r];
            const Pair both(oa, oa);
            const float2 *lr = lk + r * pitch + id + q, *sr = pairs + id + q;
            // t0 = ((links[a][0][c] + 0) + S[c][len-1]) + ob[a], t1 = ((links[a][1][c] + ob[a-1]) + S[c][len-2]) + ob[a]
            auto terms = [&](int i) {
                const float2 l = lr[G * i], c = sr[G * i];
                return ((Pair(l.x, l.y) + Pair(c.x, c.y)) + both).get();
            };
            float2 held[HELD];
            float best = neg_inf();
#pragma unroll
            for (int k = 0; k < HELD / U; k++) {
                if (k * U >= trips) break;
#pragma unroll
                for (int j = 0; j < U; j++) held[k * U + j] = terms(k * U + j);
#pragma unroll
                for (int j = 0; j < U; j++) best = fmaxf(best, fmaxf(held[k * U + j].x, held[k * U + j].y));  // NaN never wins
            }
            float far = neg_inf();  // further children: the largest, and its trip or (LONG) that of the first 32 that have it
            int far_at = INT_MAX;
#pragma unroll 1
            for (int i = HELD; i < trips; i += U) {
                float2 t[U];
#pragma unroll
                for (int j = 0; j < U; j++) t[j] = terms(i + j);
                if (LONG) {
                    float most = neg_inf();
#pragma unroll
                    for (int j = 0; j < U; j++) most = fmaxf(most, fmaxf(t[j].x, t[j].y));
                    if (most > far) {
                        far = most;
                        far_at = i;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < U; j++) {
                        if (t[j].x > far) {
                            far = t[j].x;
                            far_at = 2 * (i + j);
                        }
                        if (t[j].y > far) {
                            far = t[j].y;
                            far_at = 2 * (i + j) + 1;
                        }
                    }
                }
            }
            best = fmaxf(best, far);
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
            int key = INT_MAX;
            const bool zero = __any_sync(0xffffffffu, best == 0.f);
            if (zero) {  // -0 and +0 compare equal: the value is the one that comes first
                best = neg_inf();
#pragma unroll 1
                for (int i = 0; i < trips; i++) {
                    const float2 t = terms(i);
                    const int kk = (prio << 24) | ((id + q + G * i) << 1);
                    if (t.x > best) {
                        best = t.x;
                        key = kk;
                    }
                    if (t.y > best) {
                        best = t.y;
                        key = kk | 1;
                    }
                }
                for (int o = G / 2; o > 0; o >>= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
                    const int ok = __shfl_xor_sync(0xffffffffu, key, o);
                    if (ov > best || (ov == best && ok < key)) {
                        best = ov;
                        key = ok;
                    }
                }
            }
            if (live) {  // the left half of column len + 1's pairs and the right half of column len + 2's
                const uint32_t to = cells + 8u * (((len + 1 + half) & 3) * cs + id);
                if (NC > 1) {
#pragma unroll 1
                    for (int i = q >> 1; i < NC; i += G / 2) dsm_store_async(dsm_map_to_cta(to, i), best, dsm_map_to_cta(bar, i));
                } else if (q < 2) {
                    asm volatile("st.shared.f32 [%0], %1;" ::"r"(to), "f"(best) : "memory");
                }
            }
            if (!zero) {  // which term it was, while the value is on its way
                int at = far == best ? far_at : INT_MAX;
                if (LONG && at != INT_MAX) {
                    at = INT_MAX;
#pragma unroll
                    for (int j = U - 1; j >= 0; j--) {
                        const float2 t = terms(far_at + j);
                        at = t.x == best ? 2 * (far_at + j) : t.y == best ? 2 * (far_at + j) + 1 : at;
                    }
                }
#pragma unroll
                for (int k = HELD / U - 1; k >= 0; k--) {
                    if (k * U < trips) {
#pragma unroll
                        for (int j = U - 1; j >= 0; j--) {
                            const int i = k * U + j;
                            at = held[i].x == best ? 2 * i : held[i].y == best ? 2 * i + 1 : at;
                        }
                    }
                }
                if (at != INT_MAX) key = (prio << 24) | ((id + q + G * (at >> 1)) << 1) | (at & 1);
#pragma unroll
                for (int o = G / 2; o > 0; o >>= 1) key = min(key, __shfl_xor_sync(0xffffffffu, key, o));
            }
            if (live && q == 0) {
                own_v[r * Q + len] = best;
                own_k[r * Q + len] = (uint16_t)key;
            }
        }
        // one warp waits for the column on the byte-counting barrier, the block barrier releases the others
        if (NC > 1 && warp == warps - 1) arrived = dsm_wait_column(bar, ((len - 2) >> 1) & 1) && arrived;
        __syncthreads();
    }
    return arrived;
}

template <bool LONG>
__global__ void __launch_bounds__(kVitThreads, 1)
    viterbi_cluster_kernel(const float *__restrict__ ob_lprob, const float *__restrict__ links,
                           const int64_t *__restrict__ ol, int L, float *S, int64_t *R, int64_t *Lt, int64_t *Mt,
                           int *status, int Mc, int cs, int rows_cap, int pitch, int B, int wide) {
    extern __shared__ float smem[];
    cg::cluster_group cluster = cg::this_cluster();
    int crank = (int)cluster.block_rank();  // below: the rank among the CTAs that work on this sentence
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = blockDim.x, warps = threads >> 5;
    // wide < 0: every sentence gets the whole cluster.  wide >= 0 (more sentences than half the SMs; clusters of
    // two): the sentences are taken in order of decreasing graph length, the `wide` longest get a cluster each and
    // the others share clusters, one CTA per sentence, so that the grid is one CTA per SM and every sentence
    // starts at once (a second CTA that merely left would not make room for clusters still waiting: a new cluster
    // needs both of its SMs free together).
    int NC = (int)cluster.num_blocks();
    int b = blockIdx.x / NC;
    if (wide >= 0) {
        __shared__ int s_b;
        const int want = b < wide ? b : wide + 2 * (b - wide) + crank;  // the length rank this CTA serves
        if (want >= B) return;  // the odd CTA of the last shared cluster
        if (b >= wide) {
            NC = 1;
            crank = 0;
        }
        for (int i = tid; i < B; i += threads) {
            const long long mi = ol[i], ci = (mi >= 2 && mi <= L) ? mi : 0;
            int before = 0;
            for (int j = 0; j < B; j++) {
                const long long mj = ol[j], cj = (mj >= 2 && mj <= L) ? mj : 0;
                before += cj > ci || (cj == ci && j < i);
            }
            if (before == want) s_b = i;
        }
        __syncthreads();
        b = s_b;
    }
    const int ctid = crank * threads + tid, cthreads = NC * threads;  // thread index inside the cluster
    const int Q = L / 4;
    const int m = (int)ol[b];
    const float *ob = ob_lprob + (size_t)b * L;
    const float *lkb = links + (size_t)b * L * 2 * L;
    float *Sb = S + (size_t)b * L * Q;
    int64_t *Rb = R + (size_t)b * L * Q, *Lb = Lt + (size_t)b * L * Q, *Mtb = Mt + (size_t)b * L * Q;
    for (int i = ctid; i < L * Q; i += cthreads) {
        Sb[i] = neg_inf();
        Rb[i] = 0;
        Lb[i] = 0;
        Mtb[i] = 0;
    }
    if (m < 2 || m > L) {  // uniform over the cluster: nobody reaches a cluster barrier
        if (ctid == 0) flag(status, PCFGNAT_STATUS_BAD_LENGTH);
        return;
    }
    const int Mb = main_nodes_below(m);
    const int my_rows = Mb > crank ? (Mb - crank + NC - 1) / NC : 0;  // nodes id = crank + NC * r
    // column len: (S[len - 1], S[len - 2]) of the whole chain, replicated per CTA
    float2 *col = reinterpret_cast<float2 *>(smem);  // [4][cs]
    float2 *lk = col + 4 * cs;  // [rows_cap][pitch] (links[a][0][c] + 0, links[a][1][c] + ob[a-1]) of this CTA's nodes, by child slot
    // results of this CTA's nodes, flushed to global memory after the last length: a global store inside
    // the loop would make every cluster barrier (a release) wait for it to reach L2
    float *own_v = reinterpret_cast<float *>(lk + (size_t)rows_cap * pitch + cs - Mc);  // [rows_cap][Q]
    float *s_oa = own_v + (size_t)rows_cap * Q;                        // [rows_cap] ob of this CTA's nodes
    uint16_t *own_k = reinterpret_cast<uint16_t *>(s_oa + rows_cap);  // [rows_cap][Q] child slot and kind, (c << 1) | j

    for (int r = warp; r < my_rows; r += warps) {
        const int id = crank + NC * r;
        const float *row = lkb + (size_t)(2 * id + 1) * 2 * L;
        const float olf = id >= 1 ? __ldg(ob + 2 * id) : neg_inf();  // C[a-1][1] = ob[a-1] (pcfg_viterbi.cu:203-205)
        if (lane == 0) s_oa[r] = __ldg(ob + 2 * id + 1);
#pragma unroll 4
        for (int ci = id + lane; ci < pitch; ci += 32)
            lk[r * pitch + ci] = make_float2(ci < Mb ? __ldg(row + 2 * ci + 1) + 0.f : neg_inf(),
                                             ci < Mb ? __ldg(row + L + 2 * ci + 1) + olf : neg_inf());
    }
    __shared__ __align__(8) uint64_t col_bar[2];
    for (int i = tid; i < 4 * cs; i += threads) col[i] = make_float2(neg_inf(), neg_inf());  // slots >= Mb for good
    if (tid == 0) {
        for (int i = 0; i < 2; i++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(dsm_smem_u32(&col_bar[i])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // S[m-1][1] = ob[m-1] (pcfg_viterbi.cu:58); it feeds the recurrence only if m-1 is a main-chain node
    if (tid == 0 && ((m - 1) & 1))  // every CTA fills its own copy
        col[2 * cs + (m - 2) / 2].x = col[3 * cs + (m - 2) / 2].y = __ldg(ob + (m - 1));
    // all copies initialised before anybody stores into a neighbour's; also orders the initial fill of the
    // global tables (done by threads of any CTA of the cluster) before the cells written below
    if (NC > 1) cluster.sync(); else __syncthreads();
    if (ctid == 0) Sb[(size_t)(m - 1) * Q + 1] = __ldg(ob + (m - 1));

    const int n_len = m / 4;
    const int G = viterbi_lanes(my_rows, warps);  // no fewer than the launch made room for
#define PCFGNAT_VITERBI_CASE(G_) \
    viterbi_lengths<G_, LONG>(col, lk, s_oa, own_v, own_k, col_bar, n_len, Mb, my_rows, NC, crank, Q, cs, pitch)
    const bool arrived = G == 4 ? PCFGNAT_VITERBI_CASE(4) : G == 8 ? PCFGNAT_VITERBI_CASE(8) : PCFGNAT_VITERBI_CASE(16);
#undef PCFGNAT_VITERBI_CASE
    if (!arrived && lane == 0) flag(status, PCFGNAT_STATUS_TIMEOUT);
    // no CTA leaves (its shared memory with it) while a peer may still send to it: the last column has arrived
    // everywhere once every CTA has passed its last wait
    if (NC > 1) cluster.sync();
    for (int i = tid; i < my_rows * (n_len - 2); i += threads) {  // computed cells: lengths 2 .. n_len-1
        const int r = i / (n_len - 2), len = 2 + i - r * (n_len - 2);
        viterbi_store(own_v[r * Q + len], own_k[r * Q + len], 2 * (crank + NC * r) + 1, Q, len, Sb, Rb, Lb, Mtb);
    }
}

__global__ void __launch_bounds__(1024)
    viterbi_global_kernel(const float *__restrict__ ob_lprob, const float *__restrict__ links,
                          const int64_t *__restrict__ ol, int L, float *S, int64_t *R, int64_t *Lt, int64_t *Mt,
                          int *status, int Mc, int cs) {
    extern __shared__ float smem[];
    const int b = blockIdx.x;
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31, n_warps = nthr >> 5;
    const int Q = L / 4;
    const int m = (int)ol[b];
    const float *ob = ob_lprob + (size_t)b * L;
    const float *lkb = links + (size_t)b * L * 2 * L;
    float *Sb = S + (size_t)b * L * Q;
    int64_t *Rb = R + (size_t)b * L * Q, *Lb = Lt + (size_t)b * L * Q, *Mtb = Mt + (size_t)b * L * Q;
    for (int i = tid; i < L * Q; i += nthr) {
        Sb[i] = neg_inf();
        Rb[i] = 0;
        Lb[i] = 0;
        Mtb[i] = 0;
    }
    if (m < 2 || m > L) {
        if (tid == 0) flag(status, PCFGNAT_STATUS_BAD_LENGTH);
        return;
    }
    const int Mb = main_nodes_below(m);
    float *col = smem;  // 3 rolling columns of S over main-chain slots
    for (int i = tid; i < 3 * cs; i += nthr) col[i] = neg_inf();
    __syncthreads();  // also orders the initial fill of the tables before the cells written below
    if (tid == 0) {
        const float v = __ldg(ob + (m - 1));
        Sb[(size_t)(m - 1) * Q + 1] = v;
        if ((m - 1) & 1) col[1 * cs + (m - 2) / 2] = v;
    }
    __syncthreads();
    const int x = lane & 3;
    const int prio = ((x & 1) << 1) | (x >> 1);
    for (int len = 2; len < m / 4; len++) {
        const float *S1 = col + ((len - 1) % 3) * cs;
        const float *S2 = col + ((len - 2) % 3) * cs;
        float *S0 = col + (len % 3) * cs;
        for (int id = warp; id < Mb; id += n_warps) {
            const int a = 2 * id + 1;
            const float *row = lkb + (size_t)a * 2 * L;
            const float olf = id >= 1 ? __ldg(ob + 2 * id) : neg_inf();
            float best;
            int key;
            viterbi_node(id, Mb, lane, prio, __ldg(ob + a), S1, S2, [&](int ci) { return __ldg(row + 2 * ci + 1) + 0.f; },
                         [&](int ci) { return __ldg(row + L + 2 * ci + 1) + olf; }, best, key);
            if (lane == 0) {
                S0[id] = best;
                viterbi_store(best, key, a, Q, len, Sb, Rb, Lb, Mtb);
            }
        }
        __syncthreads();
    }
}

// With S and penalty given, the output length is chosen here first, as the model does it
// (fs_plugins/models/glat_decomposed_with_link_two_hands_tri_pcfg.py:488-492): scores = S[b][1][len] /
// penalty[len] with NaN -> -inf, first maximum over len = 1 .. Q-1; it is written to pred_out.
//
// The walk is a chain of loads.  What does not depend on where it goes is read before it, by the whole block, into
// shared memory: a node's token, and whether left_tree_mask lets the walk descend to node 0 or to the node before it
// (STAGED; the tables of another program may name other left children, whose mask is read then).  A node's table
// entries are read when it is stacked, together with those of its right child where that is known by then: the walk waits
// for one L2 round trip per main-chain node, its leaf's overlaps with it.  64 sentences, graph 240: 15.6 us (18.8 us with
// the mask and the token read on the way), one sentence, graph 140: 10.7 us (12.9 us).
struct TraceCell {
    int left, right, mt;
};

template <bool STAGED>
__global__ void __launch_bounds__(128)
    backtrace_kernel(const float *__restrict__ S, const float *__restrict__ penalty, int64_t *pred_out,
                     const int64_t *__restrict__ pred, const int64_t *__restrict__ ol, const int64_t *__restrict__ Lt,
                     const int64_t *__restrict__ R, const int64_t *__restrict__ Mt, const int64_t *__restrict__ tokens,
                     const int64_t *__restrict__ mask, int mask_dim, int64_t pad, int B, int L, int Q, int cap, int64_t *out,
                     int64_t *cnt, int *status) {
    extern __shared__ int64_t s_token[];                           // STAGED: [L] tokens, then [L] bytes
    uint8_t *s_stop = reinterpret_cast<uint8_t *>(s_token + L);    // bit 0: not to node 0, bit 1: not to the node before
    __shared__ int s_kept;
    const int i = blockIdx.x, tid = threadIdx.x;
    const int max_h = (int)ol[i];
    int64_t *o = out + (size_t)i * cap;
    if (STAGED) {
        for (int a = tid; a < L && a < max_h; a += blockDim.x) {
            s_token[a] = tokens[(size_t)i * L + a];
            int stop = 0;
            if (a < mask_dim) {
                stop = mask[(size_t)a * mask_dim] != 0;
                if (a >= 1 && mask[(size_t)a * mask_dim + a - 1]) stop |= 2;
            }
            s_stop[a] = (uint8_t)stop;
        }
    }
    int chosen = 0;
    if (S && tid < 32) {
        const float *row = S + ((size_t)i * L + 1) * Q;
        float best = neg_inf();
        int key = INT_MAX;
        for (int len = 1 + tid; len < Q; len += 32) {
            float v = row[len] / penalty[len];
            if (isnan(v)) v = neg_inf();
            if (v > best || key == INT_MAX) {  // the first entry counts even at -inf: an all -inf row picks len = 1
                best = v;
                key = len;
            }
        }
        warp_argmax(best, key, tid);
        chosen = key == INT_MAX ? 1 : key;
        if (tid == 0) pred_out[i] = chosen;
    }
    __syncthreads();
    if (tid == 0) {
        constexpr int kStack = 32;  // the walk only stacks a node and its left spine: depth <= left_tree_layer + 2
        int stk_node[kStack], stk_len[kStack];
        TraceCell stk_next[kStack];  // the node's right child: its table entries (left < -1: not read yet)
        int stk_right[kStack], stk_right_len[kStack];
        int sp = 0, count = 0;
        int node = 1, len = S ? chosen : (int)pred[i];
        int64_t last = -1;
        bool bad = false;
        long guard = 0;
        const size_t base = (size_t)i * L * Q;
        constexpr int kUnread = INT_MIN;
        auto read = [&](int a, int n, TraceCell &cell) {
            const size_t at = base + (size_t)a * Q + n;
            cell.left = (int)Lt[at];
            cell.mt = (int)Mt[at];
            cell.right = (int)R[at];
        };
        auto inside = [&](int a, int n) { return a >= 0 && a < L && n >= 0 && n < Q; };
        TraceCell cell;
        cell.left = kUnread;
        cell.right = cell.mt = 0;
        while (!bad && ((node < max_h && node != 0) || sp > 0)) {
            while (node < max_h && node != 0) {
                if (!inside(node, len) || sp >= kStack || ++guard > 4L * L + 16) {
                    bad = true;
                    break;
                }
                if (cell.left == kUnread) read(node, len, cell);
                const int mt = cell.mt;
                int left = cell.left;
                stk_node[sp] = node;
                stk_len[sp] = len;
                stk_right[sp] = cell.right;
                stk_right_len[sp] = len - mt - 1;
                stk_next[sp].left = kUnread;
                if (cell.right != 0 && cell.right < max_h && inside(cell.right, len - mt - 1))
                    read(cell.right, len - mt - 1, stk_next[sp]);
                sp++;
                cell.left = kUnread;
                if (left == node) left = 0;
                if (left < 0 || left >= mask_dim || node >= mask_dim) {
                    bad = true;
                    break;
                }
                const bool stop = STAGED && left == 0          ? s_stop[node] & 1
                                  : STAGED && left == node - 1 ? s_stop[node] & 2
                                                               : mask[(size_t)node * mask_dim + left] != 0;
                if (stop) break;
                node = left;
                len = mt;
            }
            if (bad) break;
            sp--;
            node = stk_node[sp];
            const int64_t tok = STAGED ? s_token[node] : tokens[(size_t)i * L + node];
            if (tok != pad && tok != last) {
                last = tok;
                if (count < cap) o[count] = tok;
                count++;
            }
            len = stk_right_len[sp];
            node = stk_right[sp];
            cell = stk_next[sp];
        }
        if (bad) flag(status, PCFGNAT_STATUS_BAD_TRACE);
        cnt[i] = count;
        s_kept = count < cap ? count : cap;
    }
    __syncthreads();
    for (int k = s_kept + tid; k < cap; k += blockDim.x) o[k] = pad;
}

int launch_trace(const float *S, const float *penalty, int64_t *pred_out, const int64_t *pred, const int64_t *ol,
                 const int64_t *Lt, const int64_t *R, const int64_t *Mt, const int64_t *tokens, const int64_t *mask,
                 int mask_dim, int64_t pad, int B, int L, int Q, int cap, int64_t *out, int64_t *cnt, int *status,
                 cudaStream_t st) {
    const size_t smem = (size_t)L * (sizeof(int64_t) + 1);
    if (smem <= 40 * 1024)
        backtrace_kernel<true><<<B, 128, smem, st>>>(S, penalty, pred_out, pred, ol, Lt, R, Mt, tokens, mask, mask_dim, pad, B, L,
                                                     Q, cap, out, cnt, status);
    else  // graphs of more than 4 500 nodes
        backtrace_kernel<false><<<B, 128, 0, st>>>(S, penalty, pred_out, pred, ol, Lt, R, Mt, tokens, mask, mask_dim, pad, B, L, Q,
                                                   cap, out, cnt, status);
    return cuda_rc(cudaGetLastError());
}

}  // namespace

// How a CTA of n that share a sentence lays out its nodes' rows; smem 0: they do not fit.
struct VitRows {
    int cap, stride, cs, warps;
    size_t smem;
};

static VitRows viterbi_layout(int Mc, int Q, int n, int width, int warps) {
    VitRows r;
    r.cap = (Mc + n - 1) / n;  // also right for mixed widths: n is 1 there, every CTA may hold a chain
    r.warps = warps;
    const int G = viterbi_lanes(r.cap, warps);
    r.cs = Mc + viterbi_overshoot(G, width);
    for (int banks = 1; banks >= 0; banks--) {  // the rows that a half-warp reads in different banks where there is room for that
        r.stride = Mc;
        while (banks && G < 16 && (r.stride + n) % 16 != G) r.stride++;
        r.smem = ((size_t)4 * r.cs + (size_t)r.cap * r.stride + r.cs - Mc) * sizeof(float2) +
                 (size_t)r.cap * ((Q + 1) * sizeof(float) + Q * sizeof(uint16_t));
        if (r.smem <= (size_t)kSmemLimit - 1024) return r;
    }
    r.smem = 0;
    return r;
}

// With more CTAs than SMs no more warps than the nodes need, so that CTAs share SMs: 1000 sentences of 16 nodes 49 -> 24 us, 300 of
// 64 105 -> 78.  CTAs whose tables leave no room for a second one get all: 16 sentences of 430 nodes 1 798 -> 1 017 us, 32
// of 320 957 -> 698.
static VitRows viterbi_rows(int Mc, int Q, int n, int width, bool crowded) {
    constexpr int all = kVitThreads / 32;
    const int least = ((Mc + n - 1) / n + 31) / 32 * 4;
    if (crowded && least < all) {
        const VitRows r = viterbi_layout(Mc, Q, n, width, least);
        if (r.smem && 2 * (r.smem + 1024) <= (size_t)kSmemLimit) return r;
    }
    return viterbi_layout(Mc, Q, n, width, all);
}

int launch_viterbi(const float *ob, const float *links, const int64_t *ol, int B, int L, float *S, int64_t *R,
                   int64_t *Lt, int64_t *Mt, int *status, cudaStream_t st) {
    if (B == 0) return PCFGNAT_OK;
    if (L < 8) return PCFGNAT_ERR_INVALID_ARGUMENT;  // column 1 of an [L][L/4] table must exist
    const int Mc = main_slots(L, 1), Q = L / 4;
    const int cs = (Mc + 3) / 4 * 4;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // Cluster size: as many CTAs per sentence (up to 8) as still lets all sentences run at once; more when
    // a CTA's share of the links would not fit shared memory.  PCFGNAT_DP_KERNEL=rows forces the
    // single-CTA kernel (A/B runs and tests), PCFGNAT_DP_CLUSTER_SIZE a cluster size.
    int nc = 1;
    while (nc < 8 && (long long)B * nc * 2 <= sms && Mc > 8 * nc) nc *= 2;
    if (const char *v = getenv("PCFGNAT_DP_CLUSTER_SIZE")) {
        const int want = atoi(v);
        if (want == 1 || want == 2 || want == 4 || want == 8 || want == 16) nc = want;
    }
    // more sentences than half the SMs but fewer than SMs: clusters of two, which the longest sentences have to
    // themselves and the others share (see the kernel); `wide` = the SMs left over once every sentence has one
    int wide = -1;
    if (nc == 1 && B * 2 > sms && B < sms && B <= 256 && Mc > 16 && !getenv("PCFGNAT_DP_CLUSTER_SIZE")) wide = sms - B;
    if (dp_kernel_choice() == kDpRows) nc = 32;  // skips the loop below
    // mixed widths only while one CTA holds a chain; a grid larger than the GPU takes the sentences by
    // decreasing length (wide = B), so that the clusters that wait for a place get the shortest
    const auto mixed = [&](int n) { return wide >= 0 && n == 1; };
    const auto crowded = [&](int n) { return !mixed(n) && (long long)B * n > sms; };
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const auto kernel = Mc > 256 ? viterbi_cluster_kernel<true> : viterbi_cluster_kernel<false>;
    // the launch with n CTAs per sentence; returns the clusters that run at once, 0 where there is no such launch
    const auto configure = [&](int n, const VitRows &rows) {
        const int launch_nc = mixed(n) ? 2 : n;
        cfg.gridDim = dim3((unsigned)((mixed(n) ? wide + (B - wide + 1) / 2 : B) * launch_nc));
        cfg.dynamicSmemBytes = rows.smem;
        cfg.blockDim = dim3(32 * rows.warps);
        attr[0].val.clusterDim.x = (unsigned)launch_nc;
        int clusters = 0;
        if (ensure_dynamic_smem(kernel, rows.smem) != cudaSuccess ||
            (n > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
            cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return clusters;
    };
    // Sixteen CTAs where a chain is long and all sentences still run at once, every CTA on an SM of its own: one sentence of 257
    // nodes 175 -> 156 us, five of 380 348 -> 281, but nine of 300, for whose clusters there is no room, 226 -> 352, and 16 of 257,
    // whose CTAs would share SMs, 329 -> 390.
    if (nc == 8 && Mc > 256 && !crowded(16)) {
        const VitRows rows = viterbi_rows(Mc, Q, 16, 16, false);
        if (rows.smem && configure(16, rows) >= B) nc = 16;
    }
    for (; nc <= 16; nc *= 2) {
        const VitRows rows = viterbi_rows(Mc, Q, nc, mixed(nc) ? 2 : nc, crowded(nc));
        if (rows.smem == 0) continue;
        if (configure(nc, rows) < 1) continue;  // this cluster size cannot be scheduled here: try the next one
        const int order = mixed(nc) ? wide : (crowded(nc) && B <= 256 ? B : -1);
        return cuda_rc(cudaLaunchKernelEx(&cfg, kernel, ob, links, ol, L, S, R, Lt, Mt, status, Mc, rows.cs, rows.cap,
                                          rows.stride, B, order));
    }
    const size_t smem_cols = (size_t)3 * cs * sizeof(float);
    if (smem_cols > (size_t)kSmemLimit - 1024) return PCFGNAT_ERR_TOO_LARGE;
    if (ensure_dynamic_smem(viterbi_global_kernel, smem_cols) != cudaSuccess) return PCFGNAT_ERR_CUDA;
    const int warps = Mc < 4 ? 4 : (Mc > 32 ? 32 : Mc);
    viterbi_global_kernel<<<B, 32 * warps, smem_cols, st>>>(ob, links, ol, L, S, R, Lt, Mt, status, Mc, cs);
    return cuda_rc(cudaGetLastError());
}

int launch_backtrace(const int64_t *pred, const int64_t *ol, const int64_t *Lt, const int64_t *R, const int64_t *Mt,
                     const int64_t *tokens, const int64_t *mask, int mask_dim, int64_t pad, int B, int L, int Q,
                     int cap, int64_t *out, int64_t *cnt, int *status, cudaStream_t st) {
    if (B == 0) return PCFGNAT_OK;
    return launch_trace(nullptr, nullptr, nullptr, pred, ol, Lt, R, Mt, tokens, mask, mask_dim, pad, B, L, Q, cap, out, cnt,
                        status, st);
}

int launch_viterbi_decode(const float *S, const float *penalty, const int64_t *ol, const int64_t *Lt, const int64_t *R,
                          const int64_t *Mt, const int64_t *tokens, const int64_t *mask, int mask_dim, int64_t pad, int B,
                          int L, int Q, int cap, int64_t *pred_out, int64_t *out, int64_t *cnt, int *status,
                          cudaStream_t st) {
    if (B == 0) return PCFGNAT_OK;
    return launch_trace(S, penalty, pred_out, nullptr, ol, Lt, R, Mt, tokens, mask, mask_dim, pad, B, L, Q, cap, out, cnt, status,
                        st);
}

}  // namespace pcfgnat
