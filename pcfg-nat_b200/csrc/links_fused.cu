// Transition log-probabilities ("links") from half-precision link features, max_left == 1, without score matrices in global
// memory: what extract_links.cu forms over float32 operands, for features of any type and shape.  The same quantities
// (extract_links() of the reference model, fs_plugins/models/glat_decomposed_with_link_two_hands_tri_pcfg.py:163-199):
//
//     logit(a, k, c, h) = (q[a].kl[left(a,k)] + kl[left(a,k)].kr[c] + q[a].kr[c])[h] / sqrt(D),   left(a,0) = 0, left(a,1) = a - 1
//     links[a][k][c]    = log sum_h gate[a][h] softmax_(k,c)(logit(a, ., ., h))
//
//   links_prepare_kernel     a warp per main-chain node: what belongs to one node and head alone (q.kl of both options, the gate's
//                            log-softmax, kl[0].kr), the children that the masks admit, the features packed tile by tile;
//   links_fused_kernel       a block makes 16 main-chain nodes a, a warp a head, 16 children c at a step: m16n8k16 tensor-core
//                            products on the features as they are (half precision is exact there, sums in float32), whose results
//                            never leave the registers.  The softmax needs its sum before the heads can be mixed, so the
//                            products are formed twice: for the largest logit and the sum of each (node, head), the lanes'
//                            online, and for the mixture.
// Backward (training): links_grad [B][L][2][L] -> gradients of q, kl, kr and the gate logits, the logits formed again:
//   links_weights_kernel     w = links_grad / mixture of every cell;
//   links_parent_grad_kernel a warp per (16 nodes, head): the sum of the cells' d log-probabilities (which is what every logit of
//                            a row loses), then X = d logit in registers, times the children's features: d q, d kl;
//   links_child_grad_kernel  a warp per (16 children, head): the transposed tiles, times the parents' features: d kr; d gates.
//
// The scores are 0.5 GFLOP a pass on a training batch; what costs is what is done per cell (one exponential, a dozen instructions
// a pass), for which the registers of mma's accumulators are the right place: tcgen05 would put them into tensor memory, 128
// nodes a tile, more than most sentences have to give to an SM.  The tensor cores cut sums off where an FMA rounds them: chains
// of two or three instructions are started from zero and added up by the FMA pipe.  Logits are kept in units of log 2, so that an
// exponential is one ex2.  Against float64 (8 x 64 features, graphs of 162 to 514 nodes) the transitions are off by 2.0e-7 to
// 2.3e-7 (rms; 2.3e-7 to 2.5e-7 with the float32 kernels), the gradients by 1.5e-7 to 2.0e-7 of their norm (2.0e-7 to 2.7e-7) and
// every row of them (a node and head) by 1.9e-7 of its own norm in the median, also where the rows of links_grad are 1e12
// apart (2.3e-7).
// All five are bound by the issue of their instructions and the latency between them (38 to 56 % of the slots of an SM that has
// work, 12 to 20 warps; the tensor pipe 12 to 22 %).  90 sentences, M = 161, 8 x 64 features: 33 + 60 us forward, 357 us with
// extract_links.cu's three; 14 + 109 + 63 us backward, 643 us with its two, 33 of zero fills and 41 of conversions, which these
// need none of.
#include <cuda_fp16.h>

#include <initializer_list>
#include <type_traits>

#include "common.cuh"

namespace pcfgnat {

namespace {

constexpr int kTile = 16;       // nodes of a block, and children of a step
constexpr int kFusedWarps = 8;  // heads at a time
constexpr int kParentWarps = 4, kChildWarps = 4;  // of the gradients
constexpr int kPrepareWarps = 8;
constexpr int kMaxChain = 1024;     // main-chain nodes
constexpr int kMaxWidth = 1024;     // heads x head_dim
constexpr float kMixtureFloor = 1e-30f;  // below it a cell is formed from the log-probabilities, as in extract_links.cu
constexpr float kLog2E = 1.4426950408889634f, kLn2 = 0.6931471805599453f;

struct Chain {  // the masks, and the main-chain nodes
    const uint8_t *nonpad, *left_mask, *right_mask, *main_chain;
    const int *nodes;
    int M, L, tiles;  // tiles of 16 nodes
};

// What links_prepare_kernel leaves for the other kernels, in blocks of a tile of 16 nodes and a head that are copied as a whole.
// Nodes past the end of the last tile have features of zero.
template <int D>
constexpr int kChildBlock = kTile * D + 2 * kTile;   // halves: kr [16][D], then kl[0].kr (unscaled) [16] floats
template <int D>
constexpr int kParentBlock = 2 * kTile * D + 16 * kTile;  // halves: q [16][D], kl of left option 1 [16][D], Stat [16]
constexpr int kCells = 2 * kTile * kTile;            // of a tile of nodes and a tile of children: [16 nodes][2 options][16 children]

struct Stat {  // of a node and head, by links_fused_kernel; logits in units of log 2
    float4 par;   // q.kl of left option 0 and 1 (-inf: not admissible), largest logit, gate / sum
    float4 more;  // 1 / sum, log-sum-exp, log gate (natural), -
};

struct Prepared {
    float4 *node;       // [B][M][H] q.kl of left option 0 and 1, log gate, -
    __half *child;      // [B][tiles][H][kChildBlock]
    uint16_t *ok;       // [B][tiles][tiles][16] children that a node admits among 16, a bit each
    // training only (null otherwise):
    __half *parent;     // [B][tiles][H][kParentBlock]
    __half *kl0;        // [B][H D]
    uint8_t *odd;       // [B][H][16 tiles] features that are not finite: bit 0 q or kl, bit 1 kr
    float *mix;         // [B][tiles][tiles][kCells], by links_fused_kernel at admitted cells: the mixture, or where that is below the
                        // floor or no number its log-sum-exp in units of log 2, with the sign bit set
};

// ---- operands: a lane (row g = lane / 4, j = lane % 4) holds D / 4 consecutive features of its row.  Which of them is which
// k of an instruction is free as long as both operands agree, so a row is read in 16-byte pieces.
template <int KS>
struct Frag {  // 2 KS words: word 2 i and 2 i + 1 belong to instruction i
    uint32_t w[2 * KS];
    template <bool GLOBAL = false>
    __device__ __forceinline__ void load(const __half *row, int j) {
#pragma unroll
        for (int i = 0; i < KS / 2; i++) {
            const uint4 *p = reinterpret_cast<const uint4 *>(row + j * (4 * KS) + 8 * i);
            const uint4 v = GLOBAL ? __ldg(p) : *p;
            w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
        }
    }
};

// d[0], d[1]: row g, columns 2 j and 2 j + 1; d[2], d[3]: row g + 8
__device__ __forceinline__ void mma_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mma_add(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// c = (rows x0 over x1) . y, in two chains
template <int KS>
__device__ __forceinline__ void products(const Frag<KS> &x0, const Frag<KS> &x1, const Frag<KS> &y, float (&c)[4]) {
    float half[4];
#pragma unroll
    for (int i = 0; i < KS; i += KS / 2) {
        float(&d)[4] = i ? half : c;
        mma_zero(d, x0.w[2 * i], x1.w[2 * i], x0.w[2 * i + 1], x1.w[2 * i + 1], y.w[2 * i], y.w[2 * i + 1]);
#pragma unroll
        for (int at = 2 * i + 2; at < 2 * i + KS; at += 2) mma_add(d, x0.w[at], x1.w[at], x0.w[at + 1], x1.w[at + 1], y.w[at], y.w[at + 1]);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) c[i] += half[i];
}

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 2^(v - top), where -inf and NaN count nothing (fmaxf drops NaN; 2^-200 is 0), nor anything beside a +inf
__device__ __forceinline__ float rel_exp(float v, float top) { return ex2(fmaxf(v - top, -200.f)); }
// the log-probability of a head's logit, given less its head's largest one; all in units of log 2
__device__ __forceinline__ float log_probability(float less_top, float top, float lse, float lg) { return less_top + ((top - lse) + lg); }
// a head without a finite logit: any number will do
__device__ __forceinline__ float safe_top(float top) { return top > neg_inf() ? top : 0.f; }

// ---- a step is 16 nodes and 16 children, two tiles of eight children; a lane's cells of a tile: x = 4 * option + cell, cells 0 and 1
// of row g, 2 and 3 of row g + 8, of children 2 j and 2 j + 1 of the tile
// where a lane's are among the kCells of the step
__device__ __forceinline__ int cells_at(int g, int j) { return g * 2 * kTile + 2 * j; }
__device__ __forceinline__ constexpr int cell_at(int tile, int x) { return (x & 2) * 8 * kTile + (x >> 2) * kTile + 8 * tile + (x & 1); }
// whether a lane's cell is admitted; ok: of rows g and g + 8, shifted to the lane's children
__device__ __forceinline__ bool admitted(const uint32_t (&ok)[2], int tile, int x) { return ok[x >> 1 & 1] >> (8 * tile + (x & 1)) & 1; }
// all 256 cells of the warp are: most steps need no masks
__device__ __forceinline__ bool all_admitted(uint32_t ok0, uint32_t ok1) { return __all_sync(0xffffffffu, (ok0 & ok1) == 0xffffu); }

// 16 nodes' features of one head
template <int KS>
struct Parents {
    Frag<KS> q0, q1, k0, k1;
};

// Logits of a tile of eight children for one head, less `top` of the row, -inf where no child is admitted; qk[row][option]
template <int KS>
__device__ __forceinline__ void tile_logits(const Parents<KS> &rows, const Frag<KS> &children, const float2 &none,
                                            const float (&qk)[2][2], const float (&top)[2], float scale2, const uint32_t (&ok)[2], bool full,
                                            int tile, float (&v)[8]) {
    float sq[4], sk[4];
    products(rows.q0, rows.q1, children, sq);
    products(rows.k0, rows.k1, children, sk);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        v[i] = fmaf(sq[i] + (i & 1 ? none.y : none.x), scale2, qk[i >> 1][0]) - top[i >> 1];
        v[4 + i] = fmaf(sq[i] + sk[i], scale2, qk[i >> 1][1]) - top[i >> 1];
    }
    if (!full)
#pragma unroll
        for (int x = 0; x < 8; x++) v[x] = admitted(ok, tile, x) ? v[x] : neg_inf();
}

__device__ __forceinline__ float dot8(const uint4 &x, const uint4 &y) {
    const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
    float d = 0.f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(xs + i)), b = __half22float2(*reinterpret_cast<const __half2 *>(ys + i));
        d = fmaf(a.y, b.y, fmaf(a.x, b.x, d));
    }
    return d;
}
// whether one of eight halves is an infinity or a NaN
__device__ __forceinline__ bool not_finite(const uint4 &v) {
    const auto odd = [](uint32_t w) { return (w & 0x7c00u) == 0x7c00u || (w & 0x7c000000u) == 0x7c000000u; };
    return odd(v.x) | odd(v.y) | odd(v.z) | odd(v.w);
}

// Bound by the latency of its loads and by the copies (90 sentences, M = 161, 8 x 64 features: 65 MB read, 46 MB written).
template <int KS>
__global__ void __launch_bounds__(32 * kPrepareWarps)
    links_prepare_kernel(const __half *__restrict__ q, const __half *__restrict__ kl, const __half *__restrict__ kr,
                         const float *__restrict__ gates, const Chain c, int H, float scale2, const Prepared out) {
    constexpr int D = 16 * KS, PER_HEAD = D / 8;  // pieces of 16 bytes
    const int lane = threadIdx.x & 31, s = blockIdx.x * kPrepareWarps + (threadIdx.x >> 5), b = blockIdx.y;
    const int M = c.M, L = c.L, HD = H * D, P = c.tiles * kTile, tile = s / kTile, r = s % kTile;
    if (s >= P) return;
    __half *child = out.child + ((size_t)b * c.tiles + tile) * H * kChildBlock<D>;
    __half *parent = out.parent ? out.parent + ((size_t)b * c.tiles + tile) * H * kParentBlock<D> : nullptr;
    uint16_t *ok = out.ok + ((size_t)b * c.tiles + tile) * c.tiles * kTile + r;
    if (s >= M) {  // past the chain
        for (int t = lane; t < c.tiles; t += 32) ok[t * kTile] = 0;
        for (int i = lane; i < HD / 8; i += 32) {
            const int h = i / PER_HEAD, e = i % PER_HEAD * 8;
            const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4 *>(child + h * kChildBlock<D> + r * D + e) = zero;
            if (e == 0) reinterpret_cast<float *>(child + h * kChildBlock<D> + kTile * D)[r] = 0.f;
            if (parent) {
                *reinterpret_cast<uint4 *>(parent + h * kParentBlock<D> + r * D + e) = zero;
                *reinterpret_cast<uint4 *>(parent + h * kParentBlock<D> + (kTile + r) * D + e) = zero;
                if (e == 0) out.odd[((size_t)b * H + h) * P + s] = 0;
            }
        }
        return;
    }
    const uint8_t *np = c.nonpad + (size_t)b * L;
    const int a = c.nodes[s], left = a >= 1 ? a - 1 : 0;
    const size_t row = ((size_t)b * L + a) * HD, lrow = ((size_t)b * L + left) * HD, row0 = (size_t)b * L * HD;
    const float gate = lane < H ? gates[((size_t)b * L + a) * H + lane] : neg_inf();
    const uint8_t *lm = c.left_mask + (size_t)a * L, *rm = c.right_mask + (size_t)a * L;
    const bool ok0 = np[0] && !lm[0], ok1 = np[left] && !lm[left];
    float log_gate = 0.f;
#pragma unroll 2
    for (int i0 = 0; i0 < HD / 8; i0 += 32) {
        const int i = i0 + lane;
        const bool in = i < HD / 8;
        const int e = in ? 8 * i : 0, h = e / D, at = e % D;
        const uint4 x = __ldg(reinterpret_cast<const uint4 *>(q + row + e)), y = __ldg(reinterpret_cast<const uint4 *>(kl + lrow + e));
        const uint4 z = __ldg(reinterpret_cast<const uint4 *>(kl + row0 + e)), w = __ldg(reinterpret_cast<const uint4 *>(kr + row + e));
        if (i0 == 0) {  // log-softmax of the gate logits over the heads (at most 32)
            float top = gate;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            float sum = lane < H ? expf(gate - top) : 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            log_gate = gate - (top + logf(sum));
        }
        float d0 = dot8(x, z), d1 = dot8(x, y), dn = dot8(z, w);
#pragma unroll
        for (int o = 1; o < PER_HEAD; o *= 2) {
            d0 += __shfl_xor_sync(0xffffffffu, d0, o);
            d1 += __shfl_xor_sync(0xffffffffu, d1, o);
            dn += __shfl_xor_sync(0xffffffffu, dn, o);
        }
        const float lg = __shfl_sync(0xffffffffu, log_gate, h);
        const bool first = in && at == 0;
        if (in) *reinterpret_cast<uint4 *>(child + h * kChildBlock<D> + r * D + at) = w;
        if (first) {
            out.node[((size_t)b * M + s) * H + h] = make_float4(ok0 ? d0 * scale2 : neg_inf(), ok1 ? d1 * scale2 : neg_inf(), lg, 0.f);
            reinterpret_cast<float *>(child + h * kChildBlock<D> + kTile * D)[r] = dn;
        }
        if (parent) {
            const uint32_t mine = ((1u << PER_HEAD) - 1) << (lane & ~(PER_HEAD - 1));
            const bool odd_parent = __ballot_sync(0xffffffffu, not_finite(x) | not_finite(y)) & mine;
            const bool odd_child = __ballot_sync(0xffffffffu, not_finite(w)) & mine;
            if (in) {
                *reinterpret_cast<uint4 *>(parent + h * kParentBlock<D> + r * D + at) = x;
                *reinterpret_cast<uint4 *>(parent + h * kParentBlock<D> + (kTile + r) * D + at) = y;
                if (s == 0) *reinterpret_cast<uint4 *>(out.kl0 + (size_t)b * HD + e) = z;
            }
            if (first) out.odd[((size_t)b * H + h) * P + s] = (uint8_t)(odd_parent | odd_child << 1);
        }
    }
    bool any = ok0 || ok1;  // the two options that count, and as a rule the only ones; without a left child there is no transition
    for (int at = lane; !any && at - lane < L; at += 32) any = __any_sync(0xffffffffu, at < L && np[at] && !lm[at]);
#pragma unroll 4
    for (int c0 = 0; c0 < P; c0 += 32) {
        const int n = c.nodes[min(c0 + lane, M - 1)];
        const uint32_t bits = __ballot_sync(0xffffffffu, (c0 + lane < M) & any & (np[n] != 0) & (c.main_chain[n] != 0) & (rm[n] == 0));
        if (lane < 2 && c0 / kTile + lane < c.tiles) ok[(c0 / kTile + lane) * kTile] = (uint16_t)(bits >> (16 * lane));
    }
}

__device__ __forceinline__ void copy_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dsm_smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int D>
constexpr int kPitch = D + 8;  // halves between rows of a tile: a lane's pieces of two rows, and ldmatrix's rows, on different banks
// ROWS rows of D halves that lie one behind the other, by one warp
template <int D, int ROWS>
__device__ __forceinline__ void copy_rows(__half *dst, const __half *src, int lane) {
    constexpr int PER = D / 8;
    dst += lane / PER * kPitch<D> + lane % PER * 8;
    src += lane * 8;
#pragma unroll
    for (int i = 0; i < ROWS * PER / 32; i++) copy_async16(dst + i * (32 / PER) * kPitch<D>, src + i * 256);
}

// The tiles (at most 64) with an admitted child (ok: 32 bytes per tile, `ok_pitch` halfwords apart), or with a feature that zeros
// don't cancel, in order; by one warp.  Returns how many.
__device__ __forceinline__ int list_tiles(const uint16_t *ok, size_t ok_pitch, const uint8_t *odd, uint32_t odd_bits, int tiles, int lane,
                                          uint8_t *list) {
    int n = 0;
    for (int t0 = 0; t0 < tiles; t0 += 32) {
        const int t = t0 + lane;
        bool on = false;
        if (t < tiles) {
            const uint4 *o = reinterpret_cast<const uint4 *>(ok + t * ok_pitch);
            const uint4 x = __ldg(o), y = __ldg(o + 1);
            on = (x.x | x.y | x.z | x.w | y.x | y.y | y.z | y.w) != 0;
            if (odd) {
                const uint4 z = __ldg(reinterpret_cast<const uint4 *>(odd + t * kTile));
                on |= ((z.x | z.y | z.z | z.w) & odd_bits) != 0;
            }
        }
        const uint32_t set = __ballot_sync(0xffffffffu, on);
        if (on) list[n + __popc(set & ((1u << lane) - 1))] = (uint8_t)t;
        n += __popc(set);
    }
    __syncwarp();
    return n;
}

// ---- a warp's walk over (tile, head) pairs, the children's features of the next pairs on their way into its ring
template <int D>
constexpr int kChildTile = kTile * kPitch<D> + 2 * kTile;  // halves
struct Cursor {
    int i, h;  // place in the list of tiles, head
};
// Extra: how much more a pair takes in the ring (halves), and copy(to, t), which fetches it
struct NoExtra {
    static constexpr int kHalves = 0;
    __device__ __forceinline__ void copy(__half *, int, int) const {}
};
template <int KS, int STAGES, class Extra>
struct Children {
    static constexpr int D = 16 * KS, STAGE = kChildTile<D> + Extra::kHalves;
    __half *ring;         // [STAGES][STAGE]
    const __half *blocks; // of the sentence
    const uint8_t *list;
    int n, H, lane;
    Extra extra;

    __device__ __forceinline__ void ask(bool on, int stage, const Cursor &at) const {
        if (on) {
            const int t = list[at.i];
            __half *to = ring + stage * STAGE;
            const __half *from = blocks + (size_t)(t * H + at.h) * kChildBlock<D>;
            copy_rows<D, kTile>(to, from, lane);
            if (lane < 4) copy_async16(to + kTile * kPitch<D> + 8 * lane, from + kTile * D + 8 * lane);
            extra.copy(to + kChildTile<D>, t, lane);
        }
        copy_commit();
    }
    // next(cursor): to the pair after it, whether there is one
    template <class Next, class Work>
    __device__ __forceinline__ void walk(int h, Next next, Work work) const {
        Cursor now{0, h}, ahead = now;
        bool any = n > 0, more = any;
#pragma unroll
        for (int i = 0; i < STAGES - 1; i++) {
            ask(more, i, ahead);
            more = more && next(ahead);
        }
        int stage = 0;
        while (any) {
            copy_wait<STAGES - 2>();
            __syncwarp();  // this pair has arrived for every lane, and the tile before it has been read by every lane
            ask(more, stage ? stage - 1 : STAGES - 1, ahead);
            more = more && next(ahead);
            work(list[now.i], now.i, now.h, ring + stage * STAGE);
            stage = stage + 1 == STAGES ? 0 : stage + 1;
            any = next(now);
        }
        copy_wait<0>();
        __syncwarp();
    }
};
// the features and kl[0].kr of tile x of a step
template <int KS>
__device__ __forceinline__ void read_children(const __half *step, int x, int g, int j, Frag<KS> &f, float2 &none) {
    constexpr int D = 16 * KS;
    f.load(step + (8 * x + g) * kPitch<D>, j);
    none = *reinterpret_cast<const float2 *>(reinterpret_cast<const float *>(step + kTile * kPitch<D>) + 8 * x + 2 * j);
}

constexpr int kCellPitch = 24;                      // words between rows of 16 cells: float2 of half a warp on different banks
constexpr int kCellWords = 2 * kTile * kCellPitch;  // [row][option][16]
constexpr int kListBytes = 64;
static_assert(kMaxChain / kTile <= kListBytes, "tiles of a chain fit the list");

template <int D>
struct FusedSmem {
    static constexpr int kStages = 3;
    size_t ring, cells, sums, node, ok, total;
    int warps;  // that have a head; the others help to write
    __host__ __device__ FusedSmem(int M, int H) {
        const int tiles = M > 0 ? (M + kTile - 1) / kTile : 1;
        warps = H < kFusedWarps ? H : kFusedWarps;
        ring = (size_t)warps * kStages * kChildTile<D> * sizeof(__half);
        cells = (size_t)2 * warps * kCellWords * sizeof(float);
        sums = (size_t)H * kTile * (sizeof(float4) + sizeof(float2));
        node = (size_t)tiles * kTile * sizeof(int);
        ok = (size_t)tiles * kTile * sizeof(uint16_t);
        total = ring + cells + sums + node + ok + (kFusedWarps + 1) * kListBytes;
    }
};

// The block's rows of features where the caller has them
struct ParentRows {
    const __half *q, *kl;  // of the sentence
    const int *node;
    int r0, M, HD;
    template <int KS>
    __device__ __forceinline__ void load(Parents<KS> &rows, int h, int g, int j) const {
        const int a0 = node[min(r0 + g, M - 1)], a1 = node[min(r0 + g + 8, M - 1)], at = h * 16 * KS;
        rows.q0.template load<true>(q + (size_t)a0 * HD + at, j);
        rows.q1.template load<true>(q + (size_t)a1 * HD + at, j);
        rows.k0.template load<true>(kl + (size_t)max(a0 - 1, 0) * HD + at, j);
        rows.k1.template load<true>(kl + (size_t)max(a1 - 1, 0) * HD + at, j);
    }
};

// The cells of a step from the log-probabilities of a warp's heads: log-sum-exp, online, in units of log 2.  Largest term and sum
// into two buffers.
template <int KS>
__device__ __noinline__ void lay_down_terms(const __half *blocks, int t, int H, int h0, const float4 *par, const float2 *logs, float scale2,
                                            uint32_t ok0, uint32_t ok1, int g, int j, const ParentRows from, float *tops, float *rests) {
    constexpr int D = 16 * KS;
    const uint32_t ok[2] = {ok0, ok1};
#pragma unroll 1
    for (int tile = 0; tile < 2; tile++) {
        float z[8], rest[8];
#pragma unroll
        for (int x = 0; x < 8; x++) z[x] = neg_inf(), rest[x] = 0.f;
        for (int h = h0; h < H; h += kFusedWarps) {
            const __half *block = blocks + (size_t)(t * H + h) * kChildBlock<D>;
            Parents<KS> rows;
            from.load(rows, h, g, j);
            Frag<KS> f;
            f.template load<true>(block + (8 * tile + g) * D, j);
            const float2 none = __ldg(reinterpret_cast<const float2 *>(reinterpret_cast<const float *>(block + kTile * D) + 8 * tile + 2 * j));
            const float4 p0 = par[h * kTile + g], p1 = par[h * kTile + g + 8];
            const float top[2] = {safe_top(p0.z), safe_top(p1.z)};
            const float qk[2][2] = {{p0.x, p0.y}, {p1.x, p1.y}};
            const float2 l0 = logs[h * kTile + g], l1 = logs[h * kTile + g + 8];
            float v[8];
            tile_logits(rows, f, none, qk, top, scale2, ok, false, tile, v);
#pragma unroll
            for (int x = 0; x < 8; x++) {
                const float2 l = x & 2 ? l1 : l0;
                const float term = log_probability(v[x], top[x >> 1 & 1], l.x, l.y);
                if (term > z[x]) {  // drops NaN and -inf
                    rest[x] = fmaf(rest[x], rel_exp(z[x], term), 1.f);
                    z[x] = term;
                } else if (term > neg_inf() && z[x] < CUDART_INF_F) {
                    rest[x] += ex2(term - z[x]);
                }
            }
        }
#pragma unroll
        for (int x = 0; x < 8; x++) {
            const int at = ((g + (x & 2 ? 8 : 0)) * 2 + (x >> 2)) * kCellPitch + 8 * tile + 2 * j + (x & 1);
            tops[at] = z[x];
            rests[at] = rest[x];
        }
    }
}

// A block makes 16 nodes, a warp a head (or several: H > 8).  First the largest logit and the sum of exponentials of
// every (node, head), the lanes' online; then the mixture, tile by tile: the warps lay their heads' terms beside each other in
// shared memory, and all threads add them up and write the cells out.
// MANY: more heads than warps.
template <int KS, bool TRAINING, bool MANY>
__global__ void __launch_bounds__(32 * kFusedWarps, 2)
    links_fused_kernel(const __half *__restrict__ q, const __half *__restrict__ kl, const Chain c, int H, float scale2,
                       float *__restrict__ links, const Prepared in) {
    constexpr int D = 16 * KS;
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int threads = 32 * kFusedWarps;
    const int rt = blockIdx.y, r0 = rt * kTile, b = blockIdx.x;  // the first nodes have the most children: they go first
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, j = lane & 3, M = c.M, L = c.L, HD = H * D, P = c.tiles * kTile;
    const FusedSmem<D> shape(M, H);

    // -inf into the rows of this block's nodes and of the nodes between them; admissible cells are overwritten below
    const int first = r0 ? c.nodes[r0 - 1] + 1 : 0, last = r0 + kTile >= M ? L : c.nodes[r0 + kTile - 1] + 1;
    {
        float *from = links + ((size_t)b * L + first) * 2 * L;
        const size_t n = (size_t)(last - first) * 2 * L;
        const size_t head = min(n, ((16 - reinterpret_cast<uintptr_t>(from) % 16) / 4) % 4), body = (n - head) / 4;
        const float4 inf4 = make_float4(neg_inf(), neg_inf(), neg_inf(), neg_inf());
        if (tid < head) from[tid] = neg_inf();
        for (size_t i = tid; i < body; i += threads) reinterpret_cast<float4 *>(from + head)[i] = inf4;
        if (tid < n - head - 4 * body) from[head + 4 * body + tid] = neg_inf();
    }
    if (r0 >= M) return;
    float *cells = reinterpret_cast<float *>(smem + shape.ring);                // [2][warps][kCellWords]
    float4 *par = reinterpret_cast<float4 *>(smem + shape.ring + shape.cells);  // [H][16]
    float2 *logs = reinterpret_cast<float2 *>(par + H * kTile);                 // [H][16] log-sum-exp, log gate, units of log 2
    int *node = reinterpret_cast<int *>(smem + shape.ring + shape.cells + shape.sums);
    uint16_t *ok = reinterpret_cast<uint16_t *>(node + P);
    uint8_t *again = reinterpret_cast<uint8_t *>(ok + P), *list = again + (warp + 1) * kListBytes;
    const uint16_t *ok_rows = in.ok + ((size_t)b * c.tiles + rt) * c.tiles * kTile;
    const Children<KS, FusedSmem<D>::kStages, NoExtra> children{reinterpret_cast<__half *>(smem) + warp * FusedSmem<D>::kStages * kChildTile<D>,
                                in.child + (size_t)b * c.tiles * H * kChildBlock<D>, list,
                                list_tiles(ok_rows, kTile, nullptr, 0, c.tiles, lane, list), H, lane, {}};
    if (children.n == 0) return;
    for (int i = tid; i < P; i += threads) node[i] = c.nodes[min(i, M - 1)];
    for (int i = tid; i < kListBytes; i += threads) again[i] = 0;
    for (int i = tid; i < 2 * c.tiles; i += threads) reinterpret_cast<uint4 *>(ok)[i] = __ldg(reinterpret_cast<const uint4 *>(ok_rows) + i);
    __syncthreads();

    const ParentRows from{q + (size_t)b * L * HD, kl + (size_t)b * L * HD, node, r0, M, HD};
    const int n = children.n;
    Parents<KS> rows;
    int at_head = -1;

    // ---- largest logits and sums, head after head
    if (warp < H) {
        float m[2], sum[2], qk[2][2], log_gate[2];
        const float zero[2] = {0.f, 0.f};
        children.walk(
            warp,
            [&](Cursor &at) {
                if (++at.i < n) return true;
                at.i = 0, at.h += kFusedWarps;
                return MANY && at.h < H;
            },
            [&](int t, int i, int h, const __half *tile) {
                if (i == 0) {
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        const float4 p = __ldg(in.node + ((size_t)b * M + min(r0 + g + 8 * r, M - 1)) * H + h);
                        qk[r][0] = p.x, qk[r][1] = p.y, log_gate[r] = p.z;
                        m[r] = neg_inf(), sum[r] = 0.f;
                    }
                    from.load(rows, h, g, j);
                    at_head = h;
                }
                const uint32_t row_ok[2] = {ok[t * kTile + g], ok[t * kTile + g + 8]}, bits[2] = {row_ok[0] >> (2 * j), row_ok[1] >> (2 * j)};
                const bool full = all_admitted(row_ok[0], row_ok[1]);
#pragma unroll
                for (int half = 0; half < 2; half++) {
                    Frag<KS> f;
                    float2 none;
                    read_children<KS>(tile, half, g, j, f, none);
                    float v[8];
                    tile_logits(rows, f, none, qk, zero, scale2, bits, full, half, v);
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        const float x = fmaxf(fmaxf(m[r], fmaxf(v[2 * r], v[2 * r + 1])), fmaxf(v[4 + 2 * r], v[5 + 2 * r]));  // drops NaN
                        const float top = safe_top(x);
                        float all = (ex2(v[2 * r] - top) + ex2(v[2 * r + 1] - top)) + (ex2(v[4 + 2 * r] - top) + ex2(v[5 + 2 * r] - top));
                        if (isnan(all))
                            all = (rel_exp(v[2 * r], top) + rel_exp(v[2 * r + 1], top)) + (rel_exp(v[4 + 2 * r], top) + rel_exp(v[5 + 2 * r], top));
                        sum[r] = fmaf(sum[r], rel_exp(m[r], top), all);
                        m[r] = x;
                    }
                }
                if (i + 1 < n) return;
#pragma unroll
                for (int r = 0; r < 2; r++) {  // the quad's, and what follows from it
                    float top = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], 1));
                    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
                    float all = sum[r] * rel_exp(m[r], safe_top(top));
                    all += __shfl_xor_sync(0xffffffffu, all, 1);
                    all += __shfl_xor_sync(0xffffffffu, all, 2);
                    if (j == 0) {
                        const float lg = log_gate[r], gate = lg > neg_inf() ? expf(lg) : 0.f;  // NaN: the head counts nothing
                        const float inv = all > 0.f ? 1.f / all : 0.f, lse = isinf(top) ? top : top + log2f(all);
                        const Stat stat{make_float4(qk[r][0], qk[r][1], top, gate * inv), make_float4(inv, lse, lg, 0.f)};
                        par[h * kTile + g + 8 * r] = stat.par;
                        logs[h * kTile + g + 8 * r] = make_float2(lse, lg * kLog2E);
                        if (TRAINING)
                            reinterpret_cast<Stat *>(in.parent + (((size_t)b * c.tiles + rt) * H + h) * kParentBlock<D> + 2 * kTile * D)[g + 8 * r] = stat;
                    }
                }
            });
    }

    // ---- the mixture of the heads, tile after tile; a warp with several heads adds its own up first
    float mine[2][8];
    const int warps = shape.warps, warp_last = warp + (H - 1 - warp) / kFusedWarps * kFusedWarps;
    float *mix = TRAINING ? in.mix + ((size_t)b * c.tiles + rt) * c.tiles * kCells : nullptr;
    const auto write_out = [&](int t, int at) {  // all threads, when every head's terms lie there
        const float *buf = cells + (at & 1) * warps * kCellWords;
        __syncthreads();
        bool low = false;
        for (int i = tid; i < kCells / 2; i += threads) {  // two children of a (node, option)
            const int r = i / kTile, k = i / 8 & 1, col = 2 * (i & 7);
            const float *from = buf + (2 * r + k) * kCellPitch + col;
            float2 sum = make_float2(0.f, 0.f);
            for (int w = 0; w < warps; w++) {
                const float2 one = *reinterpret_cast<const float2 *>(from + w * kCellWords);
                sum.x += one.x, sum.y += one.y;
            }
            const uint32_t on = ok[t * kTile + r] >> col;
            if (!(on & 3)) continue;
            float *out = links + (((size_t)b * L + node[r0 + r]) * 2 + k) * L;
            const int *to = node + t * kTile + col;
            if (on & 1) out[to[0]] = logf(sum.x), low |= !(sum.x > kMixtureFloor);
            if (on & 2) out[to[1]] = logf(sum.y), low |= !(sum.y > kMixtureFloor);
            if (TRAINING) *reinterpret_cast<float2 *>(mix + (size_t)t * kCells + 2 * i) = sum;
        }
        if (low) again[at] = 1;
    };
    if (warp >= H)
        for (int at = 0; at < n; at++) write_out(list[at], at);
    else
    children.walk(
        warp,
        [&](Cursor &at) {
            if (MANY && at.h + kFusedWarps < H) at.h += kFusedWarps;
            else at.h = warp, at.i++;
            return at.i < n;
        },
        [&](int t, int at, int h, const __half *tile) {
            if (MANY && h != at_head) {
                from.load(rows, h, g, j);
                at_head = h;
            }
            const uint32_t row_ok[2] = {ok[t * kTile + g], ok[t * kTile + g + 8]}, bits[2] = {row_ok[0] >> (2 * j), row_ok[1] >> (2 * j)};
            const bool full = all_admitted(row_ok[0], row_ok[1]);
            const float4 p0 = par[h * kTile + g], p1 = par[h * kTile + g + 8];
            const float top[2] = {safe_top(p0.z), safe_top(p1.z)};
            const float qk[2][2] = {{p0.x, p0.y}, {p1.x, p1.y}};
            float *lay = cells + (at & 1) * warps * kCellWords + warp * kCellWords + 2 * g * kCellPitch + 2 * j;
#pragma unroll
            for (int half = 0; half < 2; half++) {
                Frag<KS> f;
                float2 none;
                read_children<KS>(tile, half, g, j, f, none);
                float v[8];
                tile_logits(rows, f, none, qk, top, scale2, bits, full, half, v);
#pragma unroll
                for (int x = 0; x < 8; x++) {
                    v[x] = ex2(v[x]) * (x & 2 ? p1.w : p0.w);
                    if (MANY) v[x] = mine[half][x] = h == warp ? v[x] : mine[half][x] + v[x];
                }
                if (MANY && h != warp_last) continue;
#pragma unroll
                for (int x = 0; x < 8; x += 2)
                    *reinterpret_cast<float2 *>(lay + ((x & 2) * 8 + (x >> 2)) * kCellPitch + 8 * half) = make_float2(v[x], v[x + 1]);
            }
            if (MANY && h != warp_last) return;
            write_out(t, at);
        });

    // ---- cells that are too small, or no number: log-sum-exp of the log-probabilities
    __syncthreads();
    float *tops = cells, *rests = cells + warps * kCellWords;
    for (int at = 0; at < n; at++) {
        if (!again[at]) continue;
        const int t = list[at];
        if (warp < H)
            lay_down_terms<KS>(children.blocks, t, H, warp, par, logs, scale2, ok[t * kTile + g] >> (2 * j), ok[t * kTile + g + 8] >> (2 * j), g, j,
                           from, tops + warp * kCellWords, rests + warp * kCellWords);
        __syncthreads();
        for (int i = tid; i < kCells; i += threads) {
            const int r = i / (2 * kTile), k = i / kTile & 1, col = i % kTile, cell = (2 * r + k) * kCellPitch + col;
            if (!(ok[t * kTile + r] >> col & 1)) continue;
            float *out = links + (((size_t)b * L + node[r0 + r]) * 2 + k) * L + node[t * kTile + col];
            if (*out > -69.f) continue;  // log(kMixtureFloor) is -69.08
            float z = neg_inf(), rest = 0.f;
            for (int w = 0; w < warps; w++) z = fmaxf(z, tops[w * kCellWords + cell]);
            for (int w = 0; w < warps; w++) rest += rests[w * kCellWords + cell] * rel_exp(tops[w * kCellWords + cell], safe_top(z));
            if (!isinf(z)) z += log2f(rest);
            *out = isinf(z) ? neg_inf() : z * kLn2;
            // the sign tells: its log-sum-exp, never above 0 but for rounding
            if (TRAINING) mix[(size_t)t * kCells + i] = isinf(z) ? neg_inf() : -fabsf(fminf(z, 0.f));
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// backward.  With G = links_grad[a][k][c], e[h] = exp(logit - top[h]) and c[h] = gate / sum as in the forward:
//   w = G / sum_h e[h] c[h],   d lp[h] = w e[h] c[h],   Gs[h] = sum_{k,c} d lp[h]   (= d log gate[h])
//   X[h] = d logit[h] = e[h] (w c[h] - Gs[h] / sum e[h])      (of the scaled logit: the 1 / sqrt(D) is in the results)
// A cell whose mixture is below the floor or no number, or whose w leaves the floats, takes its share from the log-probabilities
// instead: d lp[h] = G exp(log-probability[h] - z), z = the cell's log-sum-exp; it is marked in w and has (z, G) in `rare`.
// ---------------------------------------------------------------------------------------------------------------------
constexpr uint32_t kRareMark = 0x7fc0dea1u;  // a NaN that arithmetic does not make

struct Weights {        // of the cells: [B][tiles][tiles][kCells], written at admitted ones
    float *w;
    float2 *rare;       // written where w is marked
    float *gs, *back;   // [B][tiles][H][16] Gs, Gs / sum e
    float *none_part;   // [B][H][tiles][D]: d kl[0] (left option 0) of the tile's nodes
};

__device__ __forceinline__ bool marked(float w) { return __float_as_uint(w) == kRareMark; }
// d lp of a marked cell from its head's log-probability
__device__ __noinline__ float rare_share(const float2 *rare, float term) {
    const float2 zg = *rare;
    return !isinf(zg.x) && term > neg_inf() ? zg.y * ex2(term - zg.x) : 0.f;
}

// ---- X of a step as two operands of 16 rows and 16 columns: d[half][4 * operand + 2 * row + cell] is what a lane has of row g (0) or
// g + 8 (1), columns 8 * half + 2 j + cell.  Each row of an operand goes by a power of two of its own into the halves' range and is
// split in three: all 24 bits of whatever is above 2^-16 of the row's largest, 2^-40 of that below.  (One scale for 16 nodes or
// a whole chain, and two halves, before: 22 bits, and nothing below 2^-38 of the largest of all.)
struct Operands {
    uint32_t part[2][3][4];  // [operand][largest to smallest][register]
    float down[2][2];        // [operand][row]: undoes the scale
    __device__ __forceinline__ explicit Operands(const float (&d)[2][8]) {
        float up[2][2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            uint32_t top[2];  // of the lane, then of the quad: the upper halves of the floats suffice
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int x = 4 * k + 2 * r;
                top[k] = __float_as_uint(fmaxf(fmaxf(fabsf(d[0][x]), fabsf(d[0][x + 1])), fmaxf(fabsf(d[1][x]), fabsf(d[1][x + 1]))));
            }
            uint32_t both = __byte_perm(top[0], top[1], 0x7632);
            both = __vmaxu2(both, __shfl_xor_sync(0xffffffffu, both, 1));
            both = __vmaxu2(both, __shfl_xor_sync(0xffffffffu, both, 2));
#pragma unroll
            for (int k = 0; k < 2; k++) {  // the largest to 2^14 .. 2^15; both scales are normal floats
                const int exponent = (int)(both >> (k ? 23 : 7) & 0xff), shift = min(141 - exponent, 126);
                up[k][r] = __uint_as_float((uint32_t)(127 + shift) << 23);
                down[k][r] = __uint_as_float((uint32_t)(127 - shift) << 23);
            }
        }
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float x = d[i >> 1][4 * k + 2 * (i & 1)] * up[k][i & 1], y = d[i >> 1][4 * k + 2 * (i & 1) + 1] * up[k][i & 1];
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    const __half2 h = __floats2half2_rn(x, y);
                    part[k][p][i] = *reinterpret_cast<const uint32_t *>(&h);
                    const float2 back = __half22float2(h);
                    x -= back.x, y -= back.y;
                }
            }
    }
    // acc += operand k . f, the tensor cores' part from zero
    __device__ __forceinline__ void add_product(float (&acc)[4], int k, uint32_t f0, uint32_t f1) const {
        float sum[4];
        mma_zero(sum, part[k][2][0], part[k][2][1], part[k][2][2], part[k][2][3], f0, f1);
#pragma unroll
        for (int p = 1; p >= 0; p--) mma_add(sum, part[k][p][0], part[k][p][1], part[k][p][2], part[k][p][3], f0, f1);
#pragma unroll
        for (int i = 0; i < 4; i++) acc[i] = fmaf(sum[i], down[k][i >> 1], acc[i]);
    }
};
// 16 x 16 of a tile, transposed: the second operand of two neighbouring column tiles
__device__ __forceinline__ void load_transposed(uint32_t address, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(address)
                 : "memory");
}
template <int D>
__device__ __forceinline__ uint32_t transposed_base(const __half *tile, int lane) {
    return dsm_smem_u32(tile + (lane & 15) * kPitch<D> + (lane >> 4) * 8);
}
template <class T>
__device__ __forceinline__ void store2(T *p, float x, float y) {
    if constexpr (sizeof(T) == 2) *reinterpret_cast<__half2 *>(p) = __floats2half2_rn(x, y);
    else *reinterpret_cast<float2 *>(p) = make_float2(x, y);
}
__device__ __forceinline__ float2 half2_at(const __half *p) { return __half22float2(*reinterpret_cast<const __half2 *>(p)); }

// D values of one head of the rows [first, last) that `skip` does not claim, zero
template <int D, class T, class Skip>
__device__ __forceinline__ void zero_rows(T *dst, int first, int last, size_t pitch, int lane, Skip skip) {
    constexpr int V = 16 / sizeof(T), PER = D / V;
    for (int i = lane; i < (last - first) * PER; i += 32) {
        const int x = first + i / PER;
        if (!skip(x)) *reinterpret_cast<uint4 *>(dst + (size_t)x * pitch + i % PER * V) = make_uint4(0u, 0u, 0u, 0u);
    }
}

// w of every admitted cell, a block per step, four children a thread.  Bound by the latency of its loads (steps without an
// admitted child leave at once) and by reading every other word of the gradient.
__global__ void __launch_bounds__(kCells / 4)
    links_weights_kernel(const float *__restrict__ links_grad, const Prepared in, const Weights wt, const Chain c) {
    const int b = blockIdx.x, rt = blockIdx.y, t = blockIdx.z, tid = threadIdx.x, k = tid / 4 & 1, r = tid / 8, col = tid % 4 * 4;
    const size_t step = ((size_t)b * c.tiles + rt) * c.tiles + t, at = step * kCells + 4 * tid;
    const uint32_t on = __ldg(in.ok + step * kTile + r) >> col & 15;
    if (on == 0) return;
    const float *grad = links_grad + (((size_t)b * c.L + c.nodes[rt * kTile + r]) * 2 + k) * c.L;
    const float4 mix4 = __ldg(reinterpret_cast<const float4 *>(in.mix + at));
    const float mix[4] = {mix4.x, mix4.y, mix4.z, mix4.w};
    float w[4];
#pragma unroll
    for (int x = 0; x < 4; x++) w[x] = on >> x & 1 ? __ldg(grad + c.nodes[t * kTile + col + x]) : 0.f;
#pragma unroll
    for (int x = 0; x < 4; x++) {
        const float G = w[x];
        if (!(on >> x & 1)) continue;
        w[x] = G / mix[x];
        const bool low = signbit(mix[x]);
        if (low || (G != 0.f && !(fabsf(w[x]) < CUDART_INF_F))) {
            wt.rare[at + x] = make_float2(low ? mix[x] : log2f(mix[x]), G);
            w[x] = __uint_as_float(kRareMark);
        }
    }
    *reinterpret_cast<float4 *>(wt.w + at) = make_float4(w[0], w[1], w[2], w[3]);
}

// what a step of a gradient needs beside features: w of its cells [16 nodes][pitch], then its masks [16]
template <int PITCH>
struct CellWeights {
    static constexpr int kHalves = 2 * kTile * PITCH + kTile;
    const float *w;
    const uint16_t *ok;
    size_t w_pitch, ok_pitch;  // between tiles
    __device__ __forceinline__ void copy(__half *to, int t, int lane) const {
        const float *from = w + t * w_pitch + lane * 4;
        float *row = reinterpret_cast<float *>(to) + lane / 8 * PITCH + lane % 8 * 4;
#pragma unroll
        for (int i = 0; i < 4; i++) copy_async16(row + i * 4 * PITCH, from + i * 128);
        if (lane < 2) copy_async16(to + 2 * kTile * PITCH + 8 * lane, ok + t * ok_pitch + 8 * lane);
    }
};
using ParentWeights = CellWeights<40>;  // pitches that put a warp's reads on different banks
using ChildWeights = CellWeights<36>;

constexpr int kGradStages = 2;
template <int D>
constexpr int kParentRing = kGradStages * (kChildTile<D> + ParentWeights::kHalves);
template <int D>
constexpr int kParentWarpHalves = kParentRing<D> + 2 * kTile * kPitch<D> + kListBytes;  // and q and kl of the nodes, two lists
template <int D>
constexpr size_t kParentSmem = kParentWarps * kParentWarpHalves<D> * sizeof(__half);

// A warp makes 16 nodes of one head: first Gs, and with it
// d q[a] = dab0 kl[0] + dab1 kl[left] + sum_s (X0 + X1)[a][s] kr[s],  d kl[left(a)] = dab1 q[a] + sum_s X1[a][s] kr[s],
// d kl[0] += dab0 q[a] + sum_s X0[a][s] kr[s]  (and the gradient of left option 1 where that is node 0),  dab[k] = sum_s X_k.
template <int KS, class T>
__global__ void __launch_bounds__(32 * kParentWarps, 3)
    links_parent_grad_kernel(const Prepared in, const Weights wt, const Chain c, const int *__restrict__ slot_of, int H, float scale,
                             float scale2, T *__restrict__ dq, T *__restrict__ dkl) {
    constexpr int D = 16 * KS, PITCH = kPitch<D>, N = D / 8;
    extern __shared__ __align__(16) uint8_t smem[];
    const int rt = blockIdx.y, r0 = rt * kTile, b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int h = blockIdx.z * kParentWarps + warp, g = lane >> 2, j = lane & 3, M = c.M, L = c.L, HD = H * D, P = c.tiles * kTile;
    if (h >= H) return;
    const size_t pitch = HD, sentence = (size_t)b * L * HD, bh = (size_t)b * H + h;
    const int first = r0 ? c.nodes[r0 - 1] + 1 : 0, last = r0 + kTile >= M ? L : c.nodes[r0 + kTile - 1] + 1;
    zero_rows<D>(dq + sentence + h * D, first, last, pitch, lane, [&](int x) { return slot_of[x] >= 0; });
    zero_rows<D>(dkl + sentence + h * D, first, last, pitch, lane, [&](int x) { return x == 0 || (x + 1 < L && slot_of[x + 1] >= 0); });
    if (r0 >= M) {
        for (int d = lane; d < D; d += 32) wt.none_part[(bh * c.tiles + rt) * D + d] = 0.f;
        return;
    }
    __half *own = reinterpret_cast<__half *>(smem) + warp * kParentWarpHalves<D>;
    __half *ring = own + 2 * kTile * PITCH;
    uint8_t *lists = reinterpret_cast<uint8_t *>(ring + kParentRing<D>);
    const uint16_t *ok = in.ok + ((size_t)b * c.tiles + rt) * c.tiles * kTile;
    const size_t tile_cells = ((size_t)b * c.tiles + rt) * c.tiles * kCells;
    const __half *block = in.parent + (((size_t)b * c.tiles + rt) * H + h) * kParentBlock<D>;
    copy_rows<D, 2 * kTile>(own, block, lane);
    copy_commit();
    Children<KS, kGradStages, ParentWeights> children{ring, in.child + (size_t)b * c.tiles * H * kChildBlock<D>, lists,
                                                      list_tiles(ok, kTile, nullptr, 0, c.tiles, lane, lists), H, lane,
                                                      {wt.w + tile_cells, ok, kCells, kTile}};
    const int used = children.n;
    const auto step_weights = [&](const __half *step) { return reinterpret_cast<const float *>(step + kChildTile<D>) + g * 40 + 2 * j; };
    const auto step_masks = [&](const __half *step) { return reinterpret_cast<const uint16_t *>(step + kChildTile<D> + 2 * kTile * 40) + g; };
    const auto weight_at = [](int half, int x) { return (x & 2) * 4 * 40 + (x >> 2) * kTile + 8 * half + (x & 1); };
    const auto one_head = [&children](Cursor &at) { return ++at.i < children.n; };
    const Stat *stat = reinterpret_cast<const Stat *>(block + 2 * kTile * D) + g;  // of rows g and g + 8
    const float4 p0 = __ldg(&stat[0].par), p1 = __ldg(&stat[8].par);
    const float top[2] = {safe_top(p0.z), safe_top(p1.z)}, gate[2] = {p0.w, p1.w};
    const float qk[2][2] = {{p0.x, p0.y}, {p1.x, p1.y}};
    const auto logits = [&](const __half *step, int half, const uint32_t (&bits)[2], bool full, float (&v)[8]) {
        Parents<KS> rows;
        rows.q0.load(own + g * PITCH, j);
        rows.q1.load(own + (g + 8) * PITCH, j);
        rows.k0.load(own + (kTile + g) * PITCH, j);
        rows.k1.load(own + (kTile + g + 8) * PITCH, j);
        Frag<KS> f;
        float2 none;
        read_children<KS>(step, half, g, j, f, none);
        tile_logits(rows, f, none, qk, top, scale2, bits, full, half, v);
    };
    const auto rare_term = [&](float less_top, int r) {
        const float4 y = __ldg(&stat[8 * r].more);
        return log_probability(less_top, top[r], y.y, y.z * kLog2E);
    };
    // ---- Gs
    children.list = lists, children.n = used;
    float sum[2] = {0.f, 0.f};
    children.walk(h, one_head, [&](int t, int, int, const __half *step) {
        const uint32_t row_ok[2] = {step_masks(step)[0], step_masks(step)[8]}, bits[2] = {row_ok[0] >> (2 * j), row_ok[1] >> (2 * j)};
        const bool full = all_admitted(row_ok[0], row_ok[1]);
        const size_t at = tile_cells + (size_t)t * kCells + cells_at(g, j);
        float part[2] = {0.f, 0.f};  // short chains: a row has up to 2048 cells
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float w[8], v[8], share[8];
            bool rare = false;
#pragma unroll
            for (int x = 0; x < 8; x += 2) {
                const float2 two = *reinterpret_cast<const float2 *>(step_weights(step) + weight_at(half, x));
                w[x] = two.x, w[x + 1] = two.y;
            }
            logits(step, half, bits, full, v);
#pragma unroll
            for (int x = 0; x < 8; x++) {
                share[x] = w[x] * (ex2(v[x]) * gate[x >> 1 & 1]);
                rare |= marked(w[x]);
            }
            if (!full || __any_sync(0xffffffffu, rare))
#pragma unroll
                for (int x = 0; x < 8; x++)
                    if (!admitted(bits, half, x)) share[x] = 0.f;
                    else if (marked(w[x])) share[x] = rare_share(wt.rare + at + cell_at(half, x), rare_term(v[x], x >> 1 & 1));
#pragma unroll
            for (int r = 0; r < 2; r++) part[r] += (share[2 * r] + share[2 * r + 1]) + (share[4 + 2 * r] + share[5 + 2 * r]);
        }
#pragma unroll
        for (int r = 0; r < 2; r++) sum[r] += part[r];
    });
    float back[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
#pragma unroll
        for (int o = 1; o < 4; o *= 2) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o);
        // a block without an admitted child, and nodes past the chain, have no sums from the forward
        const bool on = used > 0 && r0 + g + 8 * r < M;
        back[r] = !on ? 0.f : (r ? p1.z : p0.z) < CUDART_INF_F ? sum[r] * __ldg(&stat[8 * r].more).x : CUDART_NAN_F;
        if (j == 0) {
            wt.gs[(((size_t)b * c.tiles + rt) * H + h) * kTile + g + 8 * r] = on ? sum[r] : 0.f;
            wt.back[(((size_t)b * c.tiles + rt) * H + h) * kTile + g + 8 * r] = back[r];
        }
    }

    // ---- X times the children's features; tiles with a feature that zeros don't cancel take part
    children.list = lists + kListBytes;
    children.n = list_tiles(ok, kTile, in.odd + bh * P, 0x02020202u, c.tiles, lane, lists + kListBytes);
    float acc[2][N][4] = {}, dab[2][2] = {};  // [option]; [row][option]
    children.walk(h, one_head, [&](int t, int, int, const __half *step) {
        const uint32_t row_ok[2] = {step_masks(step)[0], step_masks(step)[8]}, bits[2] = {row_ok[0] >> (2 * j), row_ok[1] >> (2 * j)};
        const bool full = all_admitted(row_ok[0], row_ok[1]);
        const size_t at = tile_cells + (size_t)t * kCells + cells_at(g, j);
        float X[2][8];  // [half of the children]: 4 * option + 2 * row + cell
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float w[8];
            float(&d)[8] = X[half];
            bool rare = false;
#pragma unroll
            for (int x = 0; x < 8; x += 2) {
                const float2 two = *reinterpret_cast<const float2 *>(step_weights(step) + weight_at(half, x));
                w[x] = two.x, w[x + 1] = two.y;
            }
            logits(step, half, bits, full, d);
#pragma unroll
            for (int x = 0; x < 8; x++) rare |= marked(w[x]);
            if (!full || __any_sync(0xffffffffu, rare))
#pragma unroll
                for (int x = 0; x < 8; x++) {
                    const int r = x >> 1 & 1;
                    if (!admitted(bits, half, x)) d[x] = 0.f;
                    else if (marked(w[x])) d[x] = rare_share(wt.rare + at + cell_at(half, x), rare_term(d[x], r)) - rel_exp(d[x], 0.f) * back[r];
                    else d[x] = ex2(d[x]) * fmaf(w[x], gate[r], -back[r]);
                }
            else
#pragma unroll
                for (int x = 0; x < 8; x++) d[x] = ex2(d[x]) * fmaf(w[x], gate[x >> 1 & 1], -back[x >> 1 & 1]);
#pragma unroll
            for (int x = 0; x < 8; x += 2) dab[x >> 1 & 1][x >> 2] += d[x] + d[x + 1];
        }
        const Operands operands(X);
        const uint32_t base = transposed_base<D>(step, lane);
#pragma unroll
        for (int m = 0; m < N; m += 2) {
            uint32_t f[4];
            load_transposed(base + 16 * m, f);
#pragma unroll
            for (int y = 0; y < 2; y++)
#pragma unroll
                for (int k = 0; k < 2; k++) operands.add_product(acc[k][m + y], k, f[2 * y], f[2 * y + 1]);
        }
    });
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
        for (int k = 0; k < 2; k++) {
            dab[r][k] *= scale;
            dab[r][k] += __shfl_xor_sync(0xffffffffu, dab[r][k], 1);
            dab[r][k] += __shfl_xor_sync(0xffffffffu, dab[r][k], 2);
        }
    T *q_out[2], *k_out[2];
    bool is_row[2], is_left[2];  // a node of the chain; with a left option 1 of its own
#pragma unroll
    for (int r = 0; r < 2; r++) {
        is_row[r] = r0 + g + 8 * r < M;
        const int node = c.nodes[min(r0 + g + 8 * r, M - 1)];
        is_left[r] = node > 1;
        q_out[r] = dq + sentence + node * pitch + h * D + 2 * j;
        k_out[r] = dkl + sentence + max(node - 1, 0) * pitch + h * D + 2 * j;
    }
#pragma unroll
    for (int m = 0; m < N; m++) {
        const float2 none0 = half2_at(in.kl0 + (size_t)b * HD + h * D + 8 * m + 2 * j);
        float part[2] = {0.f, 0.f};
#pragma unroll
        for (int r = 0; r < 2; r++) {
            if (!is_row[r]) continue;
            const float2 qv = half2_at(own + (g + 8 * r) * PITCH + 8 * m + 2 * j), kv = half2_at(own + (kTile + g + 8 * r) * PITCH + 8 * m + 2 * j);
            const float x0[2] = {acc[0][m][2 * r] * scale, acc[0][m][2 * r + 1] * scale};
            const float x1[2] = {acc[1][m][2 * r] * scale, acc[1][m][2 * r + 1] * scale};
            store2(q_out[r] + 8 * m, dab[r][0] * none0.x + dab[r][1] * kv.x + (x0[0] + x1[0]),
                   dab[r][0] * none0.y + dab[r][1] * kv.y + (x0[1] + x1[1]));
            const float l0 = dab[r][1] * qv.x + x1[0], l1 = dab[r][1] * qv.y + x1[1];
            if (is_left[r]) store2(k_out[r] + 8 * m, l0, l1);
            else part[0] += l0, part[1] += l1;
            part[0] += dab[r][0] * qv.x + x0[0];
            part[1] += dab[r][0] * qv.y + x0[1];
        }
#pragma unroll
        for (int o = 4; o < 32; o *= 2) {
            part[0] += __shfl_xor_sync(0xffffffffu, part[0], o);
            part[1] += __shfl_xor_sync(0xffffffffu, part[1], o);
        }
        if (g == 0) *reinterpret_cast<float2 *>(wt.none_part + (bh * c.tiles + rt) * D + 8 * m + 2 * j) = make_float2(part[0], part[1]);
    }
}

// A stage of the children's gradient: q and kl of 16 parents, their Stat, their Gs / sum e, the step's weights and masks
template <int D>
constexpr int kParentTile = 2 * kTile * kPitch<D> + 16 * kTile + 2 * kTile + ChildWeights::kHalves;  // halves
template <int D>
constexpr int kChildSmem = kChildWarps * (2 * kParentTile<D> * 2 + kListBytes);

// d kr[s] = sum_a ( (X0 + X1)[a][s] q[a] + X1[a][s] kl[left(a)] ) + kl[0] sum_a X0[a][s]; the first block of a sentence also
// adds up d kl[0]; and the gradient of the gate logits.  Launched behind links_parent_grad_kernel.
template <int KS, class T>
__global__ void __launch_bounds__(32 * kChildWarps)
    links_child_grad_kernel(const Prepared in, const Weights wt, const Chain c, const int *__restrict__ slot_of, int H, float scale,
                            float scale2, T *__restrict__ dkl, T *__restrict__ dkr, float *__restrict__ dgates) {
    constexpr int D = 16 * KS, PITCH = kPitch<D>, N = D / 8, STAGE = kParentTile<D>;
    extern __shared__ __align__(16) uint8_t smem[];
    const int ct = c.tiles - 1 - blockIdx.y, s0 = ct * kTile, b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int h = blockIdx.z * kChildWarps + warp, g = lane >> 2, j = lane & 3, HD = H * D, M = c.M, L = c.L, P = c.tiles * kTile;
    if (h >= H) return;
    const size_t pitch = HD, base = (size_t)b * L * HD + (size_t)h * D, bh = (size_t)b * H + h;
    const int first = s0 ? c.nodes[s0 - 1] + 1 : 0, last = s0 + kTile >= M ? L : c.nodes[s0 + kTile - 1] + 1;
    zero_rows<D>(dkr + base, first, last, pitch, lane, [&](int x) { return slot_of[x] >= 0; });
    // gate logits: d lg - softmax(gates) sum d lg, of this warp's nodes and head
    for (int x = first + lane; x < last; x += 32) {
        const int s = slot_of[x];
        float d = 0.f;
        if (s >= 0) {
            const float *gs = wt.gs + ((size_t)b * c.tiles + s / kTile) * H * kTile + s % kTile;
            float total = 0.f;
            for (int i = 0; i < H; i++) total += __ldg(gs + i * kTile);
            d = __ldg(gs + h * kTile) - (total != 0.f ? expf(__ldg(in.node + ((size_t)b * M + s) * H + h).z) * total : 0.f);
        }
        dgates[((size_t)b * L + x) * H + h] = d;
    }
    if (ct == 0)
        for (int d = 2 * lane; d < D; d += 64) {
            float x = 0.f, y = 0.f;
            for (int i = 0; i < c.tiles; i++) {
                const float2 v = *reinterpret_cast<const float2 *>(wt.none_part + (bh * c.tiles + i) * D + d);
                x += v.x, y += v.y;
            }
            store2(dkl + base + d, x, y);
        }
    if (s0 >= M) return;
    __half *ring = reinterpret_cast<__half *>(smem + warp * (2 * STAGE * 2 + kListBytes));
    uint8_t *list = reinterpret_cast<uint8_t *>(ring + 2 * STAGE);
    const uint16_t *ok = in.ok + ((size_t)b * c.tiles * c.tiles + ct) * kTile;
    const size_t ok_pitch = (size_t)c.tiles * kTile;  // per tile of parents
    const int n = list_tiles(ok, ok_pitch, in.odd + bh * P, 0x01010101u, c.tiles, lane, list);
    const __half *blocks = in.parent + ((size_t)b * c.tiles * H + h) * kParentBlock<D>;
    const float *backs = wt.back + ((size_t)b * c.tiles * H + h) * kTile;
    const size_t all_cells = ((size_t)b * c.tiles * c.tiles + ct) * kCells;
    const ChildWeights extra{wt.w + all_cells, ok, (size_t)c.tiles * kCells, ok_pitch};
    const auto load = [&](int stage, int at) {
        if (at < n) {
            const int t = list[at];
            __half *to = ring + stage * STAGE;
            const __half *from = blocks + (size_t)t * H * kParentBlock<D>;
            copy_rows<D, 2 * kTile>(to, from, lane);
            copy_async16(to + 2 * kTile * PITCH + 8 * lane, from + 2 * kTile * D + 8 * lane);
            if (lane < 4) copy_async16(to + 2 * kTile * PITCH + 16 * kTile + 8 * lane, backs + (size_t)t * H * kTile + 4 * lane);
            extra.copy(to + 2 * kTile * PITCH + 16 * kTile + 2 * kTile, t, lane);
        }
        copy_commit();
    };
    load(0, 0);
    const __half *mine = in.child + (((size_t)b * c.tiles + ct) * H + h) * kChildBlock<D>;
    Frag<KS> c0, c1;
    c0.template load<true>(mine + g * D, j);
    c1.template load<true>(mine + (g + 8) * D, j);
    const float none[2] = {__ldg(reinterpret_cast<const float *>(mine + kTile * D) + g), __ldg(reinterpret_cast<const float *>(mine + kTile * D) + g + 8)};
    // cell x = 8 * half of the parents + 4 * option + cell: child g or g + 8, parent 2 j or 2 j + 1; in rows of `row` words
    const auto place = [](int x, int g_, int j_, int row) { return (8 * (x >> 3) + 2 * j_ + (x & 1)) * row + (x >> 2 & 1) * kTile + g_ + (x & 2 ? 8 : 0); };
    float acc[N][4] = {}, x0sum[2] = {0.f, 0.f};
    for (int at = 0; at < n; at++) {
        const int t = list[at], stage = at & 1;
        load(stage ^ 1, at + 1);
        const size_t cells = all_cells + (size_t)t * c.tiles * kCells;
        copy_wait<1>();
        __syncwarp();
        const __half *sq = ring + stage * STAGE, *sk = sq + kTile * PITCH;
        const Stat *stat = reinterpret_cast<const Stat *>(sk + kTile * PITCH);
        const float *back = reinterpret_cast<const float *>(stat + kTile), *cell = back + kTile + place(0, g, j, 36);
        const uint16_t *masks = reinterpret_cast<const uint16_t *>(back + kTile + kTile * 36);
        uint32_t on[2];  // [half of the parents]: children that the parents 2 j and 2 j + 1 admit, 16 bits each
#pragma unroll
        for (int m = 0; m < 2; m++) on[m] = *reinterpret_cast<const uint32_t *>(masks + 8 * m + 2 * j);
        const auto admits = [&](int x) { return on[x >> 3] >> (16 * (x & 1) + g + (x & 2 ? 8 : 0)) & 1; };
        const bool full = __all_sync(0xffffffffu, (on[0] & on[1]) == 0xffffffffu);
        float X[2][8];  // [half of the parents]: X0 + X1 and X1 of 16 children
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float vq[4], vk[4];
            float(&d)[8] = X[half];
            Frag<KS> f;
            f.load(sq + (8 * half + g) * PITCH, j);
            products(c0, c1, f, vq);
            f.load(sk + (8 * half + g) * PITCH, j);
            products(c0, c1, f, vk);
            float w[8];
            bool rare = false;
#pragma unroll
            for (int x = 0; x < 8; x++) {
                w[x] = cell[place(8 * half + x, 0, 0, 36)];
                rare |= marked(w[x]);
            }
            const bool plain = full && !__any_sync(0xffffffffu, rare);
#pragma unroll
            for (int u = 0; u < 2; u++) {  // parent 2 j + u
                const float4 p = stat[8 * half + 2 * j + u].par;
                const float top = safe_top(p.z), less = back[8 * half + 2 * j + u];
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int i = 2 * r + u;
                    d[i] = fmaf(vq[i] + none[r], scale2, p.x) - top;
                    d[4 + i] = fmaf(vq[i] + vk[i], scale2, p.y) - top;
                }
                if (plain)
#pragma unroll
                    for (int x = u; x < 8; x += 2) d[x] = ex2(d[x]) * fmaf(w[x], p.w, -less);
                else
#pragma unroll
                    for (int x = u; x < 8; x += 2) {
                        if (!admits(8 * half + x)) {
                            d[x] = 0.f;
                        } else if (marked(w[x])) {
                            const float4 y = stat[8 * half + 2 * j + u].more;
                            d[x] = rare_share(wt.rare + cells + place(8 * half + x, g, j, 2 * kTile), log_probability(d[x], top, y.y, y.z * kLog2E)) - rel_exp(d[x], 0.f) * less;
                        } else {
                            d[x] = ex2(d[x]) * fmaf(w[x], p.w, -less);
                        }
                    }
            }
#pragma unroll
            for (int r = 0; r < 2; r++) x0sum[r] += d[2 * r] + d[2 * r + 1];
#pragma unroll
            for (int x = 0; x < 4; x++) d[x] += d[4 + x];
        }
        const Operands operands(X);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint32_t from = transposed_base<D>(k ? sk : sq, lane);
#pragma unroll
            for (int m = 0; m < N; m += 2) {
                uint32_t f[4];
                load_transposed(from + 16 * m, f);
#pragma unroll
                for (int y = 0; y < 2; y++) operands.add_product(acc[m + y], k, f[2 * y], f[2 * y + 1]);
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        x0sum[r] *= scale;
        x0sum[r] += __shfl_xor_sync(0xffffffffu, x0sum[r], 1);
        x0sum[r] += __shfl_xor_sync(0xffffffffu, x0sum[r], 2);
        if (s0 + g + 8 * r >= M) continue;
        T *to = dkr + base + c.nodes[s0 + g + 8 * r] * pitch + 2 * j;
#pragma unroll
        for (int m = 0; m < N; m++) {
            const float2 none0 = half2_at(in.kl0 + (size_t)b * HD + h * D + 8 * m + 2 * j);
            store2(to + 8 * m, fmaf(x0sum[r], none0.x, acc[m][2 * r] * scale), fmaf(x0sum[r], none0.y, acc[m][2 * r + 1] * scale));
        }
    }
}

inline int tiles_of(int M) { return M > 0 ? (M + kTile - 1) / kTile : 1; }
// A block walks its children one step after the other, which takes the longer the chain is, however few the sentences are;
// extract_links.cu's kernels spread a few long sentences over the GPU.  Forward and backward (us, these / those): one sentence of
// 257 nodes, eight heads 117 / 85, four 117 / 134, four with one head 101 / 85, 16 with one head 113 / 142; of 121 nodes, four
// heads: four sentences 66 / 60, 16 67 / 94; of 61: 47 / 47 and 48 / 53.  On the device alone, in a graph of calls, the line would lie elsewhere for few sentences: one of
// 41 nodes and eight heads 45 / 41, four of 256 and four heads 106 / 86, two of 513 213 / 141.  But these are five launches and seven
// allocations where the others are eight kernels, three conversions and twice the allocations: a training pass from Python over two
// sentences of 33 nodes 705 / 785 us, over four of 257 and four heads 690 / 775, over two of 513 2 134 / 2 116.
inline bool fused_shape_ok(int M, int B, int H, int D) {
    if ((D != 32 && D != 64) || (long long)H * D > kMaxWidth || M > kMaxChain) return false;
    return tiles_of(M) < 4 || (long long)B * tiles_of(M) * (H < 4 ? H : 4) >= 256;
}

// Pieces of one block of memory, 16 bytes each at least
struct Carver {
    char *base;
    size_t used = 0;
    template <class T>
    T *take(size_t n) {
        T *at = reinterpret_cast<T *>(base + used);
        used += (n * sizeof(T) + 15) / 16 * 16;
        return at;
    }
};
size_t carve_prepared(void *base, int M, int B, int H, int D, bool training, Prepared &p) {
    Carver c{static_cast<char *>(base)};
    const size_t tiles = tiles_of(M), blocks = B * tiles * H;
    p = {};
    p.node = c.take<float4>((size_t)B * M * H);
    p.child = c.take<__half>(blocks * (D == 64 ? kChildBlock<64> : kChildBlock<32>));
    p.ok = c.take<uint16_t>(B * tiles * tiles * kTile);
    if (training) {
        p.parent = c.take<__half>(blocks * (D == 64 ? kParentBlock<64> : kParentBlock<32>));
        p.kl0 = c.take<__half>((size_t)B * H * D);
        p.odd = c.take<uint8_t>(blocks * kTile);
        p.mix = c.take<float>(B * tiles * tiles * kCells);
    }
    return c.used;
}
size_t carve_weights(void *base, int M, int B, int H, int D, Weights &w) {
    Carver c{static_cast<char *>(base)};
    const size_t tiles = tiles_of(M), cells = B * tiles * tiles * kCells, blocks = B * tiles * H;
    w.w = c.take<float>(cells);
    w.rare = c.take<float2>(cells);
    w.gs = c.take<float>(blocks * kTile);
    w.back = c.take<float>(blocks * kTile);
    w.none_part = c.take<float>(blocks * D);
    return c.used;
}

}  // namespace

size_t links_fused_kept_bytes(int M, int B, int H, int D, int training) {
    Prepared p;
    return fused_shape_ok(M, B, H, D) ? carve_prepared(nullptr, M, B, H, D, training != 0, p) : 0;
}
size_t links_fused_scratch_bytes(int M, int B, int H, int D) {
    Weights w;
    return fused_shape_ok(M, B, H, D) ? carve_weights(nullptr, M, B, H, D, w) : 0;
}

int launch_links_fused(const void *q, const void *kl, const void *kr, const float *gates, const uint8_t *nonpad,
                       const uint8_t *left_mask, const uint8_t *right_mask, const uint8_t *main_chain, const int *nodes, int M,
                       int B, int L, int H, int D, float *links, void *kept, int training, cudaStream_t st) {
    if (B == 0) return PCFGNAT_OK;
    if (!fused_shape_ok(M, B, H, D)) return PCFGNAT_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kl) | reinterpret_cast<uintptr_t>(kr) | reinterpret_cast<uintptr_t>(kept)) & 15)
        return PCFGNAT_ERR_UNSUPPORTED;
    const Chain chain{nonpad, left_mask, right_mask, main_chain, nodes, M, L, tiles_of(M)};
    Prepared p;
    carve_prepared(kept, M, B, H, D, training != 0, p);
    const auto *fq = static_cast<const __half *>(q), *fkl = static_cast<const __half *>(kl), *fkr = static_cast<const __half *>(kr);
    const float scale2 = kLog2E / sqrtf((float)D);
    const auto run = [&](auto ks, auto train) {
        constexpr int KS = decltype(ks)::value;
        constexpr bool TRAINING = decltype(train)::value;
        const FusedSmem<16 * KS> shape(M, H);
        const auto kernel = H > kFusedWarps ? links_fused_kernel<KS, TRAINING, true> : links_fused_kernel<KS, TRAINING, false>;
        if (ensure_dynamic_smem(kernel, shape.total) != cudaSuccess) return PCFGNAT_ERR_CUDA;
        if (M > 0)
            links_prepare_kernel<KS><<<dim3(chain.tiles * kTile / kPrepareWarps, B), 32 * kPrepareWarps, 0, st>>>(fq, fkl, fkr, gates, chain, H, scale2, p);
        kernel<<<dim3(B, chain.tiles), 32 * kFusedWarps, shape.total, st>>>(fq, fkl, chain, H, scale2, links, p);
        return cuda_rc(cudaGetLastError());
    };
    using K4 = std::integral_constant<int, 4>;
    using K2 = std::integral_constant<int, 2>;
    if (training) return D == 64 ? run(K4{}, std::true_type{}) : run(K2{}, std::true_type{});
    return D == 64 ? run(K4{}, std::false_type{}) : run(K2{}, std::false_type{});
}

int launch_links_fused_backward(const float *links_grad, const void *kept, const int *slot_of, const int *nodes, int M, int B,
                                int L, int H, int D, void *scratch, int half_out, void *dq, void *dkl, void *dkr, float *dgates,
                                cudaStream_t st) {
    if (B == 0) return PCFGNAT_OK;
    if (!fused_shape_ok(M, B, H, D)) return PCFGNAT_ERR_UNSUPPORTED;
    uintptr_t all = reinterpret_cast<uintptr_t>(kept) | reinterpret_cast<uintptr_t>(scratch);
    for (const void *p : {dq, dkl, dkr}) all |= reinterpret_cast<uintptr_t>(p);
    if (all & 15) return PCFGNAT_ERR_INVALID_ARGUMENT;
    const Chain chain{nullptr, nullptr, nullptr, nullptr, nodes, M, L, tiles_of(M)};
    Prepared p;
    Weights w;
    carve_prepared(const_cast<void *>(kept), M, B, H, D, true, p);  // only read here
    carve_weights(scratch, M, B, H, D, w);
    const float scale = 1.f / sqrtf((float)D), scale2 = kLog2E / sqrtf((float)D);
    const auto run = [&](auto ks, auto type) {
        constexpr int KS = decltype(ks)::value, DIM = 16 * KS;
        using T = decltype(type);
        if (ensure_dynamic_smem(links_parent_grad_kernel<KS, T>, kParentSmem<DIM>) != cudaSuccess ||
            ensure_dynamic_smem(links_child_grad_kernel<KS, T>, kChildSmem<DIM>) != cudaSuccess)
            return PCFGNAT_ERR_CUDA;
        if (M > 0) links_weights_kernel<<<dim3(B, chain.tiles, chain.tiles), kCells / 4, 0, st>>>(links_grad, p, w, chain);
        links_parent_grad_kernel<KS, T><<<dim3(B, chain.tiles, (H + kParentWarps - 1) / kParentWarps), 32 * kParentWarps, kParentSmem<DIM>, st>>>(
            p, w, chain, slot_of, H, scale, scale2, static_cast<T *>(dq), static_cast<T *>(dkl));
        links_child_grad_kernel<KS, T><<<dim3(B, chain.tiles, (H + kChildWarps - 1) / kChildWarps), 32 * kChildWarps, kChildSmem<DIM>, st>>>(
            p, w, chain, slot_of, H, scale, scale2, static_cast<T *>(dkl), static_cast<T *>(dkr), dgates);
        return cuda_rc(cudaGetLastError());
    };
    using K4 = std::integral_constant<int, 4>;
    using K2 = std::integral_constant<int, 2>;
    if (half_out) return D == 64 ? run(K4{}, __half{}) : run(K2{}, __half{});
    return D == 64 ? run(K4{}, 0.f) : run(K2{}, 0.f);
}

}  // namespace pcfgnat
