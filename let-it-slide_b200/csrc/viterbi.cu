// The code-A trellis encoder (the offline half of the path): for every row, the symbol sequence q[0..n) in {0..3}
// whose shift-register walk  s = ((s << 2) | q) & (2^L - 1),  s_start = 0,  minimises
//   sum_i pos_weight[i] * (samples[i] - alphabet[s_i])^2           (rptc.py:13-71, diagonal corrections).
//
// Dynamic programme over the 2^L states (M = 2^L, P = M / 4, Q = M / 16).  The textbook step keeps the cost rho of every
// state; here only the quarter as many values best[p] = min over d of rho[d P + p] exist, because a cost is used nowhere
// else (rptc.py:27-30,52):
//   best'[p'] = min over d = 0..3 of  best[d Q + (p' >> 2)] + w * (x - alphabet[d P + p'])^2      (first minimum)
// A row's 2^14 values at L = 16 are 64 KiB: they stay in shared memory (two buffers) for the whole row, and the whole
// row is ONE piece of work of a persistent launch instead of one launch per position.  A thread owns G groups of four
// consecutive p', so a group needs four values of best and gives four, and its 16 alphabet entries, which no position
// changes, stay in registers.  At L = 16 the 65,536 entries are as large as a register file, so a cluster of two CTAs
// shares a row: each CTA makes half of the p' and sends the half of its results that its partner reads by bulk copies.  Two rows
// alternate in a CTA there, so that a row's values travel under the other's work.
// Bound: instruction issue (four unfused operations per state and the minima; pairs of fp32 values take half the issue
// slots for the former), then, at L = 16, the exchange.  1024 x 1024 samples, L = 16: 603 ms with one launch per position and batch of eight
// rows and the costs in L2; 23.1 ms with cluster barriers between positions (their release waits for the winners' stores); 30.8 ms
// with st.async into the partner; 16.5 ms with two groups a thread and 1024 threads, the last warp sending; 15.3 ms with four groups a
// thread, whose steps' fixed part (a fifth of 211 instructions per 32 states) counts half (13.4 ms without
// winners); 14.1 ms with every warp sending for itself.
// The winners d leave as two bits each, four to a byte; a second kernel walks them backwards (rptc.py:62-68).
// The arithmetic is spelled with round-to-nearest instructions so that no multiply-add is contracted: costs, and
// therefore ties and paths, are those of the fp32 reference.
#include "common.cuh"

namespace rptc {

struct ViterbiParams {
    const float *alphabets;        // [banks][M]
    const float *pos_weight;       // [n]
    const float *samples;          // [rows][ld_samples]
    int64_t ld_samples;
    uint8_t *back;                 // [rows][n][Q]: winners of position i (i >= 1), prefix 4b + j in bits 2j, 2j+1 of byte b
    int32_t *final_state;          // [rows]
    float *loss;                   // [rows]
    int32_t n, L;
    // The rows at hand: rows_per_bank of each bank, of the first bank the last `first_rows`, of the last one what is left of `rows`.  An
    // item is what a cluster takes at a time: R rows of a bank.
    int32_t rows, first_rows, rows_per_bank, first_items, items_per_bank, n_items;
    unsigned int *status;
};

// First minimum of four: returns the value and adds its index (the first of c0..c3 that equals it) to `bits`, a float
// that counts in units of 1 from 2^23, so that its low bits are the number added up.  The two additions go to the
// multiply-add pipe: the half-rate pipe of the minima, comparisons and logic is the busier one.
__device__ __forceinline__ float first_min(float c0, float c1, float c2, float c3, float &bits, int shift) {
    const float m01 = fminf(c0, c1), m = fminf(m01, fminf(c2, c3));
    asm("{\n\t.reg .pred hi, lo;\n\t.reg .f32 v;\n\t"
        "setp.neu.f32 hi, %1, %2;\n\t"
        "selp.f32 v, %3, %4, hi;\n\t"
        "setp.neu.f32 lo, v, %2;\n\t"
        "@hi add.rn.f32 %0, %0, %5;\n\t"
        "@lo add.rn.f32 %0, %0, %6;\n\t}"
        : "+f"(bits)
        : "f"(m01), "f"(m), "f"(c2), "f"(c0), "f"((float)(2 << shift)), "f"((float)(1 << shift)));
    return m;
}
// Shared memory of this CTA -> shared memory of a CTA of the cluster, counted in bytes on a barrier over there.
__device__ __forceinline__ void bulk_s2s(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src), "r"(bytes),
                 "r"(bar)
                 : "memory");
}

// Orders (cost, state) pairs: smaller cost first, then the smaller state (rptc.py:59, the first minimum).
__device__ __forceinline__ unsigned long long cost_key(float v, uint32_t state) {
    uint32_t u = __float_as_uint(v + 0.f);                      // -0 counts as +0
    u ^= (u >> 31) ? 0xFFFFFFFFu : 0x80000000u;
    return ((unsigned long long)u << 32) | state;
}

// CL CTAs share a row, a thread owns G groups of four prefixes, R rows alternate in a CTA.
template <int CL, int G, int R>
__global__ void __launch_bounds__(G == 4 ? 512 : 32, G == 4 ? 1 : 32) viterbi_forward_kernel(const ViterbiParams p) {
    static_assert(G == 4 || (CL == 1 && R == 1), "fewer groups a thread only where a warp is a row");
    extern __shared__ __align__(128) float best_sm[];           // per row and buffer: P / CL values, and with CL == 2 half as many to send
    __shared__ unsigned long long red[33];
    __shared__ __align__(8) unsigned long long full_bar[R][2];  // CL == 2
    __shared__ __align__(16) uint32_t word_sent[2][4];          // CL == 2: what a warp with nothing to send does send, and where that lands
    const int t = threadIdx.x;
    const int M = 1 << p.L, P = M >> 2, Q = M >> 4;
    const int QC = Q / CL, PC = P / CL;                         // this CTA's share of a quarter, of all prefixes
    const int slab = CL == 2 ? PC + PC / 2 : PC;                // floats per row and buffer
    uint32_t rank = 0;
    if (CL == 2) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const bool active = G * t < QC;                             // small L: fewer groups than a warp has lanes
    const int kk = active ? G * t : 0;                          // first group, within this CTA
    const int k = (int)rank * QC + kk;                          // and overall
    // Where this thread's 4 G results go: prefix i = 4 k is read as best[d Q + k'] with d = i / Q, k' = i % Q, by the CTA
    // that owns group k'.  4 G results never straddle two readers (CL == 2 has QC = 2048).  What the partner reads is
    // put down behind this CTA's own values, in the order in which the partner holds it (quarters 2 rank, 2 rank + 1).
    uint32_t out_off = 16u * (uint32_t)k;                       // 16-byte piece k
    if (CL == 2) {
        const int d = 4 * k / Q, o = 4 * k - d * Q, reader = o / QC;
        out_off = 4u * (uint32_t)((reader == (int)rank ? d * QC : PC + (d - 2 * (int)rank) * QC) + o - reader * QC);
    }
    // Pieces of 16 bytes change places within groups of G, piece c is at c ^ (c >> 3 & (G - 1)): a thread stores G of them side by side, and
    // eight lanes that store theirs at once meet all banks.  (Of 42 wavefronts per warp and step 8 were such conflicts with G = 2.)
    constexpr uint32_t kSwap = G - 1;                           // these bits of a piece are bits of kk: QC is 64 at least, with G == 4 128
    const uint32_t swap = ((uint32_t)k >> 3) & kSwap;           // of piece k
    const int load_at = kk ^ (int)(4u * (((uint32_t)kk >> 5) & kSwap));      // float kk is in piece kk / 4
    const uint32_t s0 = smem_addr(best_sm);
    // CL == 2, per row: `full` of a buffer completes when this CTA's warps have all put down their values of a position and every warp of
    // the partner has sent what it has: half of them 2 KiB that this CTA reads, the others sixteen bytes that nobody does.  So a
    // completed `full` also says that both CTAs have finished with the buffer that the next results go to, and that what was sent
    // from the other buffer has arrived.  Nothing here needs a fence at cluster scope, which would wait for the winners
    // on their way to global memory.  Once a wait has run
    // out no other is tried: the kernel goes on to its end with what it has.
    constexpr uint32_t kWarps = 16, kWarpBytes = 32 * G * 16;   // warps of a CTA, what one puts down per position
    const uint32_t full0 = smem_addr(full_bar);
    uint32_t peer_s0 = s0, peer_full0 = full0, peer_word = 0;
    const bool sends = out_off >= 4u * (uint32_t)PC;            // of a whole warp: 32 G pieces lie with one reader
    uint32_t full_phase = 0;                                    // bit 2 r + buffer
    bool ok = true;
    if (CL == 2) {
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer_full0) : "r"(full0), "r"(rank ^ 1u));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer_s0) : "r"(s0), "r"(rank ^ 1u));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer_word) : "r"(smem_addr(word_sent[1])), "r"(rank ^ 1u));
        if (t == 0) {
            for (int i = 0; i < 2 * R; ++i) mbar_init(full0 + 8 * i, kWarps);
            mbar_fence_init();
        }
    }

    auto arrive = [] { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); };
    auto wait = [] { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); };

    for (int item = blockIdx.x / CL; item < p.n_items; item += gridDim.x / CL) {
        // item number counted as if the first bank were whole
        const int it = item + p.items_per_bank - p.first_items;
        const int bank = item < p.first_items ? 0 : it / p.items_per_bank, j = item < p.first_items ? item : it - bank * p.items_per_bank;
        const int bank0 = bank == 0 ? 0 : p.first_rows + (bank - 1) * p.rows_per_bank;
        const int row0 = bank0 + j * R;
        const int n_rows = R == 1 ? 1 : min(R, min(p.rows, p.first_rows + bank * p.rows_per_bank) - row0);
        f32x2 na[G][4][2];                                      // alphabet entries, negated: x - e = x + (-e)
        {
            const float4 *alpha = reinterpret_cast<const float4 *>(p.alphabets + (int64_t)bank * M);
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    const float4 a = __ldg(alpha + d * Q + k + g);
                    na[g][d][0] = pack2(-a.x, -a.y);
                    na[g][d][1] = pack2(-a.z, -a.w);
                }
        }
        // before the first position only the state 0 is possible (rptc.py:57-58)
        for (int i = t; i < R * PC; i += blockDim.x) {
            const int r = i / PC, o = i - r * PC;
            best_sm[2 * r * slab + o] = (o == 0 && rank == 0) ? 0.f : INFINITY;
        }
        if (CL == 2) {
            arrive();
            wait();
        } else {
            __syncthreads();
        }
        const float *xp[R];
        uint8_t *bp[R];
        float xn[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = row0 + (r < n_rows ? r : 0);
            xp[r] = p.samples + (int64_t)row * p.ld_samples;
            bp[r] = p.back + (int64_t)row * p.n * Q + k;
            xn[r] = __ldg(xp[r]);
        }
        float wn = __ldg(p.pos_weight);

        // the four predecessors' values of this thread's groups
        auto load_best = [&](int r, int cur, float (&b)[4][G]) {
            const float *src = best_sm + (2 * r + cur) * slab + load_at;
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                if (G == 4) {
                    const float4 v = *reinterpret_cast<const float4 *>(src + d * QC);
                    b[d][0] = v.x, b[d][1 % G] = v.y, b[d][2 % G] = v.z, b[d][3 % G] = v.w;
                } else if (G == 2) {
                    const float2 v = *reinterpret_cast<const float2 *>(src + d * QC);
                    b[d][0] = v.x, b[d][G - 1] = v.y;
                } else {
                    b[d][0] = src[d * QC];
                }
            }
        };
        // costs of the states d P + 4 (k + g) + 2 h + {0, 1}
        auto costs = [&](const float (&b)[4][G], int g, int h, f32x2 x2, f32x2 w2, float (&lo)[4], float (&hi)[4]) {
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                const f32x2 diff = add2(x2, na[g][d][h]);
                unpack2(add2(pack2(b[d][g], b[d][g]), mul2(w2, mul2(diff, diff))), lo[d], hi[d]);
            }
        };
        auto step = [&](int r, int i, int cur, float x, float w) {
            const int nxt = cur ^ 1;
            if (CL == 2 && i > 0) {
                const uint32_t at = 2 * r + cur;
                if (ok) ok = mbar_wait(full0 + 8 * at, (full_phase >> at) & 1u, p.status);
                full_phase ^= 1u << at;
            }
            float b[4][G];
            load_best(r, cur, b);
            const f32x2 x2 = pack2(x, x), w2 = pack2(w, w);
            const uint32_t to = 4u * (uint32_t)((2 * r + nxt) * slab), dst = s0 + to + out_off;
            float bits[(G + 1) / 2];                            // sixteen bits each
#pragma unroll
            for (int i = 0; i < (G + 1) / 2; ++i) bits[i] = 8388608.f;      // 2^23
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float m[4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float lo[4], hi[4];
                    costs(b, g, h, x2, w2, lo, hi);
                    m[2 * h] = first_min(lo[0], lo[1], lo[2], lo[3], bits[g / 2], 8 * (g % 2) + 4 * h);
                    m[2 * h + 1] = first_min(hi[0], hi[1], hi[2], hi[3], bits[g / 2], 8 * (g % 2) + 4 * h + 2);
                }
                if (active)
                    asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(dst ^ (16u * ((uint32_t)g ^ swap))), "f"(m[0]), "f"(m[1]), "f"(m[2]), "f"(m[3]) : "memory");
            }
            if (CL == 2) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the copy engine reads what was put down
                __syncwarp();
                if ((t & 31) == 0) {
                    const uint32_t mine = full0 + 8 * (2 * r + nxt), theirs = peer_full0 + 8u * (uint32_t)(2 * r + nxt);
                    if (t == 0)
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mine), "r"(kWarps / 2 * (kWarpBytes + 16u)) : "memory");
                    else mbar_arrive(mine);
                    if (sends) bulk_s2s(peer_s0 + to + out_off - 4u * (uint32_t)PC + rank * 2u * (uint32_t)PC, s0 + to + out_off, kWarpBytes, theirs);
                    else bulk_s2s(peer_word, smem_addr(word_sent[0]), 16u, theirs);
                }
                __syncwarp();
            }
            bp[r] += Q;
            if (active) {
                if (G == 4) *reinterpret_cast<uint32_t *>(bp[r]) = __byte_perm(__float_as_uint(bits[0]), __float_as_uint(bits[(G - 1) / 2]), 0x5410);
                else if (G == 2) *reinterpret_cast<uint16_t *>(bp[r]) = (uint16_t)__float_as_uint(bits[0]);
                else *bp[r] = (uint8_t)__float_as_uint(bits[0]);
            }
        };
        int cur = 0;
#pragma unroll 1
        for (int i = 0; i + 1 < p.n; ++i) {
            const float w = wn;
            wn = __ldg(p.pos_weight + i + 1);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float x = xn[r];
                xn[r] = __ldg(xp[r] + i + 1);
                if (r < n_rows) step(r, i, cur, x, w);
            }
            if (CL == 1) __syncthreads();
            cur ^= 1;
        }
        // the last position: the cheapest of all states, first minimum
#pragma unroll
        for (int r = 0; r < R; ++r) {
            unsigned long long key = ~0ull;
            if (CL == 2 && r < n_rows && p.n > 1) {
                const uint32_t at = 2 * r + cur;
                if (ok) ok = mbar_wait(full0 + 8 * at, (full_phase >> at) & 1u, p.status);
                full_phase ^= 1u << at;
            }
            if (r < n_rows && active) {
                float b[4][G];
                load_best(r, cur, b);
                const f32x2 x2 = pack2(xn[r], xn[r]), w2 = pack2(wn, wn);
#pragma unroll
                for (int g = 0; g < G; ++g)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float lo[4], hi[4];
                        costs(b, g, h, x2, w2, lo, hi);
#pragma unroll
                        for (int d = 0; d < 4; ++d) {
                            const uint32_t s = (uint32_t)(d * P + 4 * (k + g) + 2 * h);
                            key = min(key, min(cost_key(lo[d], s), cost_key(hi[d], s + 1)));
                        }
                    }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) key = min(key, __shfl_xor_sync(0xFFFFFFFFu, key, o));
            __syncthreads();                                    // `red` is free
            if ((t & 31) == 0) red[t >> 5] = key;
            __syncthreads();
            if (t < 32) {
                key = t < (int)(blockDim.x + 31) / 32 ? red[t] : ~0ull;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) key = min(key, __shfl_xor_sync(0xFFFFFFFFu, key, o));
            }
            if (CL == 2) {
                if (t == 0 && rank == 1) {
                    uint32_t dst;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(dst) : "r"(smem_addr(&red[32])));
                    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(dst), "l"(key) : "memory");
                }
                __syncwarp();
                arrive();
                wait();
                if (t == 0 && rank == 0) key = min(key, red[32]);
            }
            if (t == 0 && rank == 0 && r < n_rows) {
                const uint32_t u = (uint32_t)(key >> 32);
                p.loss[row0 + r] = __uint_as_float(u ^ ((u >> 31) ? 0x80000000u : 0xFFFFFFFFu));
                p.final_state[row0 + r] = (int32_t)(key & 0xFFFFFFFFu);
            }
            __syncwarp();
            if (CL == 2) arrive(), wait();                      // red[32] has been read; at the end, nobody leaves early
        }
        if (CL == 1) __syncthreads();                           // the buffers are free for the next row
    }
}

// Walks a row's winners from position `hi` down to `lo`; returns the state at position lo - 1 (TO_START: lo is 0 and nothing is in front), and
// with WRITE sets the symbols on the way.  A position's winner is needed to know which winner of the position before it to read, but with two bits each there are only
// four (sixteen) candidates one (two) positions on: lanes 0, 1-4 and 5-20 fetch all of them at once, and the walk takes three
// positions per trip to memory.
struct TracedRow {
    const uint8_t *back;
    int32_t *symbols;
    int64_t Q;
    int L;
    template <bool WRITE, bool TO_START = false>
    __device__ __forceinline__ uint32_t walk(uint32_t state, int64_t hi, int64_t lo) const {
        const int lane = threadIdx.x & 31;
        const int level = lane == 0 ? 0 : lane < 5 ? 1 : 2;
        const uint32_t d1 = level == 0 ? 0u : level == 1 ? (uint32_t)lane - 1u : (uint32_t)(lane - 5) >> 2, d2 = (uint32_t)(lane - 5) & 3u;
        auto before = [&](uint32_t s, uint32_t d) { return (d << (L - 2)) | (s >> 2); };      // the state that reached s by winner d
        for (int64_t i = hi; i >= lo; i -= 3) {
            uint32_t s = state;
            if (level >= 1) s = before(s, d1);
            if (level >= 2) s = before(s, d2);
            const int64_t at = i - level;
            uint32_t d = 0;                                     // before position 1 there is only the start state
            if (lane < 21 && at >= 1) d = ((uint32_t)__ldg(back + at * Q + (s >> 4)) >> (2 * ((s >> 2) & 3u))) & 3u;
            const uint32_t w0 = __shfl_sync(0xFFFFFFFFu, d, 0);
            const uint32_t w1 = __shfl_sync(0xFFFFFFFFu, d, 1 + (int)w0);
            const uint32_t w2 = __shfl_sync(0xFFFFFFFFu, d, 5 + 4 * (int)w0 + (int)w1);
            const uint32_t s1 = before(state, w0), s2 = before(s1, w1);
            if (WRITE) {
                const uint32_t mine = lane == 0 ? state : lane == 1 ? s1 : s2;
                if (lane < 3 && i - lane >= lo) symbols[i - lane] = (int32_t)(mine & 3u);
            }
            state = TO_START || i - lo >= 2 ? before(s2, w2) : i == lo ? s1 : s2;
        }
        return state;
    }
};

// PIECES: a CTA per row, its positions in equal pieces, a warp each.  Without, four rows per CTA, a warp each.  The last piece starts from the row's final state.  Which state the path
// passes at the end of another piece is not known yet, but walks from different states meet after some times the L / 2 positions that a
// state remembers: such a warp starts kMeet * L positions further on from any state, and writes symbols from its own piece on.  Pieces whose
// state is not the one that the piece behind was left with are walked again from that one, all of them at once, until all fit (at
// L = 16 most of them once).
// Bound by the trips to memory one after the other: with a warp per row 256 rows of 1024 samples took 0.1 ms at L = 12.
constexpr int kTraceWarps = 16, kTraceRows = 4, kMeet = 4;
template <bool PIECES>
__global__ void __launch_bounds__(32 * (PIECES ? kTraceWarps : kTraceRows))
    viterbi_backtrack_kernel(const uint8_t *__restrict__ back, const int32_t *__restrict__ final_state, int64_t rows, int64_t n, int L,
                             int32_t *__restrict__ symbols, int64_t ld_sym, int64_t piece, int pieces) {
    __shared__ uint32_t left[kTraceWarps];                      // state in front of a piece's first position
    const int c = threadIdx.x >> 5;
    const int64_t row = PIECES ? (int64_t)blockIdx.x : (int64_t)blockIdx.x * kTraceRows + c;
    if (!PIECES && row >= rows) return;
    TracedRow r;
    r.Q = int64_t(1) << (L - 4);
    r.L = L;
    r.back = back + row * n * r.Q;
    r.symbols = symbols + row * ld_sym;
    if constexpr (!PIECES) {
        r.walk<true, true>((uint32_t)final_state[row], n - 1, 0);
        return;
    }
    const int64_t lo = c * piece, hi = c + 1 < pieces ? lo + piece - 1 : n - 1;
    const int64_t from = min(n - 1, hi + kMeet * L);
    uint32_t state = from == n - 1 ? (uint32_t)final_state[row] : 0u;
    state = r.walk<false>(state, from, hi + 1);
    uint32_t out = r.walk<true>(state, hi, lo);
    for (;;) {
        if ((threadIdx.x & 31) == 0) left[c] = out;
        __syncthreads();
        const uint32_t want = c + 1 < pieces ? left[c + 1] : state;
        // at the latest when the pieces have been set right one by one from the last on, all fit
        if (!__syncthreads_or(want != state)) break;
        if (want != state) state = want, out = r.walk<true>(state, hi, lo);
    }
}

// out[bank][i] = quantile (2 i + 1) / 2^(L+1) of the bank's sorted values, linear between the neighbours on their grid (2 j + 1) / (2 N)
// (quantize_hf.py:136-140), in double precision and unfused, as the tensor operations round that it stands for (fourteen launches).
__global__ void __launch_bounds__(256) quantiles_kernel(const float *__restrict__ sorted, int64_t n, int L, float *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= int64_t(1) << L) return;
    const double x = (double)(2 * i + 1) * 0.5 / (double)(int64_t(1) << L);
    const double pos = __dadd_rn(__dmul_rn(x, (double)n), -0.5);
    const double floor_pos = floor(pos);
    const int64_t lo = floor_pos < 0.0 ? 0 : floor_pos > (double)(n - 1) ? n - 1 : (int64_t)floor_pos, hi = lo + 1 < n ? lo + 1 : n - 1;
    const double frac = fmin(fmax(__dadd_rn(pos, -(double)lo), 0.0), 1.0);
    const float *row = sorted + blockIdx.y * n;
    const double a = row[lo], b = row[hi];
    out[((int64_t)blockIdx.y << L) + i] = (float)__dadd_rn(a, __dmul_rn(__dadd_rn(b, -a), frac));
}

template <int CL, int G, int R>
static int launch_forward(const ViterbiParams &p, int threads, int slots, cudaStream_t stream) {
    static SmemOptIn opted;
    auto kern = viterbi_forward_kernel<CL, G, R>;
    if (int e = allow_max_smem(kern, opted, 192 * 1024)) return e;
    const int64_t items = p.n_items;
    const int clusters = (int)(items < slots ? items : slots);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * CL));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)R * 2 * ((size_t(1) << p.L) / 4 / CL) * (CL == 2 ? 6 : 4);      // with CL == 2, half as much again to send
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    RPTC_CUDA(cudaLaunchKernelEx(&cfg, kern, p));
    return RPTC_OK;
}

}  // namespace rptc

using namespace rptc;

extern "C" int64_t rptc_viterbi_workspace_bytes(int64_t rows, int64_t n, int L) {
    if (rows <= 0 || n <= 0 || L < 4 || L > 16) return -1;
    const int64_t back = rows * n * (int64_t(1) << (L - 4));
    return (back + 255) / 256 * 256 + rows * 4;
}

extern "C" int rptc_quantiles(const float *sorted, int64_t banks, int64_t values, int L, float *out, rptc_stream_t stream) {
    if (!sorted || !out) return RPTC_ERR_ARG;
    if (L < 1 || L > 16) return RPTC_ERR_ARG;
    if (banks <= 0 || banks > 65535 || values <= 0) return RPTC_ERR_SHAPE;
    if (int e = rptc_check_device()) return e;
    quantiles_kernel<<<dim3(((1u << L) + 255) / 256, (unsigned)banks), 256, 0, static_cast<cudaStream_t>(stream)>>>(sorted, values, L, out);
    RPTC_CUDA(cudaGetLastError());
    return RPTC_OK;
}

extern "C" int rptc_viterbi_encode_rows(const float *alphabets, int64_t rows_per_bank, int64_t first_row, const float *pos_weight, const float *samples,
                                        int64_t ld_samples, int64_t rows, int64_t n, int L, int32_t *symbols, int64_t ld_sym, float *loss,
                                        void *workspace, int64_t workspace_bytes, rptc_stream_t stream) {
    if (!alphabets || !pos_weight || !samples || !symbols || !loss || !workspace) return RPTC_ERR_ARG;
    if (L < 4 || L > 16) return RPTC_ERR_UNSUPPORTED;
    if (rows <= 0 || rows > 65535 || n <= 0 || rows_per_bank <= 0 || first_row < 0 || first_row >= rows_per_bank || ld_samples < n || ld_sym < n)
        return RPTC_ERR_SHAPE;
    if (rows_per_bank > (int64_t(1) << 30)) return RPTC_ERR_TOO_LARGE;
    if (n > (int64_t(1) << 30)) return RPTC_ERR_TOO_LARGE;
    if (workspace_bytes < rptc_viterbi_workspace_bytes(rows, n, L)) return RPTC_ERR_TOO_LARGE;
    if ((reinterpret_cast<uintptr_t>(alphabets) & 15) || (reinterpret_cast<uintptr_t>(workspace) & 255)) return RPTC_ERR_ALIGN;
    if (int e = rptc_check_device()) return e;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    ViterbiParams p;
    p.alphabets = alphabets;
    p.pos_weight = pos_weight;
    p.samples = samples;
    p.ld_samples = ld_samples;
    p.back = static_cast<uint8_t *>(workspace);
    const int64_t back_bytes = (rows * n * (int64_t(1) << (L - 4)) + 255) / 256 * 256;
    p.final_state = reinterpret_cast<int32_t *>(p.back + back_bytes);
    p.loss = loss;
    p.n = (int32_t)n;
    p.L = L;
    p.rows = (int32_t)rows;
    p.rows_per_bank = (int32_t)rows_per_bank;
    p.first_rows = (int32_t)(rows < rows_per_bank - first_row ? rows : rows_per_bank - first_row);
    p.status = device_status_word();
    if (!p.status) return RPTC_ERR_CUDA;
    auto rows_at_once = [&](int r) {
        const int left = p.rows - p.first_rows;
        p.first_items = (p.first_rows + r - 1) / r;
        p.items_per_bank = (p.rows_per_bank + r - 1) / r;
        p.n_items = p.first_items + left / p.rows_per_bank * p.items_per_bank + (left % p.rows_per_bank + r - 1) / r;
    };
    // Threads per CTA: a quarter of 2^(L-2) prefixes in groups of four, four groups a thread from L = 11 on (512 x 512 samples, L = 14, with
    // two: 1250 us, with four 1026; 1024 x 512, L = 12: 630 and 566), two at L = 10, one below, where a warp has lanes to spare.  At
    // L = 15 and 16 one CTA of 512 threads fills an SM; two rows then alternate in it, unless every
    // row finds a place of its own: two at a time take less than one after the other (1024 samples, L = 16, 136 rows: 2.4
    // against 4.4 ms).  Smaller L run one row per CTA and as many CTAs as fit (128 registers a thread).
    const int groups = 1 << (L - 4), sms = num_sms(), places = L == 16 ? sms / 2 : sms;
    const bool pairs = L >= 15 && rows > places;
    rows_at_once(pairs ? 2 : 1);
    int e;
    if (L == 16) e = pairs ? launch_forward<2, 4, 2>(p, 512, places, s) : launch_forward<2, 4, 1>(p, 512, places, s);
    else if (pairs) e = launch_forward<1, 4, 2>(p, 512, places, s);
    else if (L >= 11) e = launch_forward<1, 4, 1>(p, groups / 4, sms * (2048 / groups), s);
    else if (L == 10) e = launch_forward<1, 2, 1>(p, 32, sms * 32, s);
    else e = launch_forward<1, 1, 1>(p, 32, sms * 32, s);
    if (e) return e;
    // In pieces, at least as long as the way to them, where there are five of them or more and rows too few to keep enough loads under way
    // by themselves: pieces walk up to twice the positions.  Whole encoder, a warp per row / in pieces (us): 512 x 1024 samples, L = 8 299 / 205,
    // L = 12 658 / 542; 128 x 1024, L = 16 2233 / 2126; 1024 x 256, L = 9 93 / 85; 2048 x 4096, L = 9 2397 / 2071.  On the other side of the line
    // 2048 x 256, L = 9 144 / 153; 4096 x 1024, L = 10 1550 / 1650; 1024 x 256, L = 15 1723 / 1763; 256 x 96, L = 11 49.6 / 53.7.
    const int64_t most = n / (kMeet * L) < kTraceWarps ? n / (kMeet * L) : kTraceWarps;
    if (most >= 5 && rows <= (L > 12 ? 256 : n >= 1024 ? 2048 : 1024)) {
        const int64_t piece = (n + most - 1) / most, pieces = (n + piece - 1) / piece;
        viterbi_backtrack_kernel<true><<<(unsigned)rows, (unsigned)(32 * pieces), 0, s>>>(p.back, p.final_state, rows, n, L, symbols, ld_sym, piece, (int)pieces);
    } else {
        viterbi_backtrack_kernel<false><<<(unsigned)((rows + kTraceRows - 1) / kTraceRows), 32 * kTraceRows, 0, s>>>(p.back, p.final_state, rows, n, L, symbols, ld_sym, n, 1);
    }
    RPTC_CUDA(cudaGetLastError());
    return RPTC_OK;
}

extern "C" int rptc_viterbi_encode_banked(const float *alphabets, int64_t banks, const float *pos_weight, const float *samples,
                                          int64_t ld_samples, int64_t rows, int64_t n, int L, int32_t *symbols, int64_t ld_sym, float *loss,
                                          void *workspace, int64_t workspace_bytes, rptc_stream_t stream) {
    if (rows <= 0 || banks <= 0 || rows % banks) return RPTC_ERR_SHAPE;
    return rptc_viterbi_encode_rows(alphabets, rows / banks, 0, pos_weight, samples, ld_samples, rows, n, L, symbols, ld_sym, loss, workspace,
                                    workspace_bytes, stream);
}

extern "C" int rptc_viterbi_encode(const float *alphabet, const float *pos_weight, const float *samples, int64_t ld_samples,
                                   int64_t rows, int64_t n, int L, int32_t *symbols, int64_t ld_sym, float *loss, void *workspace,
                                   int64_t workspace_bytes, rptc_stream_t stream) {
    return rptc_viterbi_encode_banked(alphabet, 1, pos_weight, samples, ld_samples, rows, n, L, symbols, ld_sym, loss, workspace,
                                      workspace_bytes, stream);
}
