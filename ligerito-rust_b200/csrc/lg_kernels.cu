// CUDA kernels of liblgpu (sm_100a).  All arithmetic is exact GF(2^32) /
// BLAKE3 integer work; there is no floating point and no tensor-core shape.
#include "lg_device.cuh"
#include "lg_fs.cuh"
#include "lg_kernels.h"

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <string>

using namespace lgd;

namespace lgk {

// ---------------------------------------------------------------- Launcher
cudaEvent_t Launcher::get_event() {
    if (!free_events.empty()) {
        cudaEvent_t e = free_events.back();
        free_events.pop_back();
        return e;
    }
    cudaEvent_t e;
    cudaEventCreate(&e);
    return e;
}
void Launcher::begin(const char *, cudaEvent_t *a) {
    ++launches;
    if (!timing) return;
    *a = get_event();
    cudaEventRecord(*a, stream);
}
void Launcher::end(const char *name, cudaEvent_t a) {
    const Work w = next_work;
    next_work = {};
    if (!timing) return;
    cudaEvent_t b = get_event();
    cudaEventRecord(b, stream);
    pending.push_back({name, a, b});
    Work &t = work[name];
    t.bytes += w.bytes;
    t.mults += w.mults;
    t.comps += w.comps;
    t.general += w.general;
}
void Launcher::resolve() {
    for (auto &p : pending) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, p.a, p.b) == cudaSuccess) {
            auto &s = stats[p.name];
            s.first += 1;
            s.second += ms;
        }
        free_events.push_back(p.a);
        free_events.push_back(p.b);
    }
    pending.clear();
}
void Launcher::release() {
    for (auto &p : pending) { cudaEventDestroy(p.a); cudaEventDestroy(p.b); }
    pending.clear();
    for (auto e : free_events) cudaEventDestroy(e);
    free_events.clear();
}


bool pdl_enabled() {
    static const bool on = [] {
        const char *e = std::getenv("LG_PDL");
        return !(e && e[0] == '0');
    }();
    return on;
}

static inline unsigned ilog2u(uint64_t x) { unsigned r = 0; while (x > 1) { x >>= 1; ++r; } return r; }

// ====================================================== RS scale + spread
__global__ void k_rs_scale_spread(const uint32_t *__restrict__ poly, const uint32_t *__restrict__ pis,
                                  uint32_t *__restrict__ E, uint32_t log_m, uint64_t total) {
    pdl_begin();
    const uint64_t m = 1ull << log_m;
    for (uint64_t idx = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t i = idx & (m - 1), j = idx >> log_m;
        uint32_t v = gf_mul(poly[idx], pis[i]);
        uint32_t *col = E + (j << (log_m + 2)) + i;
        col[0] = v;
        col[m] = v;
        col[2 * m] = v;
        col[3 * m] = v;
    }
}

cudaError_t rs_scale_spread(Launcher &L, const uint32_t *poly, const uint32_t *pis, uint32_t *E,
                            uint32_t log_m, uint32_t n) {
    uint64_t total = (uint64_t)n << log_m;
    unsigned blocks = (unsigned)std::min<uint64_t>((total + 255) / 256, 148ull * 16);
    L.note(20.0 * total, (double)total, 0, (double)total);
    LGK_LAUNCH(L, "rs_scale_spread", launch_k(k_rs_scale_spread, blocks, 256, 0, L.stream, poly, pis, E, log_m, total));
    return cudaGetLastError();
}

// ================================================================== FFT
// A launch runs K consecutive stages [d0, d0+K) of every vector.  Vector
// (j, q) starts at data + j*col_stride + q*q_stride and uses the twiddle
// subtree under heap node root_base + q; the node of stage d0+s with
// in-pass index t' is heap node ((root << d0) + P) << s | t'.
struct PassArgs {
    uint32_t *data;
    const uint32_t *tw;
    const uint4 *dtab;  // this pass's D tables (see build_pass_tables)
    uint64_t col_stride, q_stride;
    uint32_t L, d0, log_S, nvec, bpg, root_base;  // bpg: strided passes, units per (q, P)
    uint32_t bulk;                                // strided passes: rows come in by bulk copies
    uint32_t *fault, tries;                       // copies: set when a wait gives up, after so many looks
    uint32_t vchunk, nchunks;  // last pass: vectors per block, blocks per (q, P)
    uint64_t units;            // strided passes: (group, chunk) work units
    const uint32_t *src;       // strided passes: input, when not data (FftSrc)
    uint64_t src_col_stride;
    const uint32_t *pis;       // k_rs_first: the row scaling
};

// Slots f + 1 .. f + n - 1 of a stage whose first slot f holds C's table: C
// XOR D, a slot a warp, starting with warp `rot` (stages one after another
// keep every warp equally busy; a loop over all slots that finds its stage by
// counting leading zeros took 45 M more instructions in a 2^18 x 256 last
// pass of 247 M).  D's slot of the stage's slot t is df + (t << dsh).
__device__ __forceinline__ void fill_stage(uint4 *T, const uint4 *dtab, int f, int n, int df, int dsh, int rot) {
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, warp = ((threadIdx.x >> 5) - rot) & (nw - 1);
    if (1 + warp >= n) return;
    const uint4 c = T[f * 32 + lane];
    for (int t = 1 + warp; t < n; t += nw) {
        uint4 d = __ldg(dtab + (df + (t << dsh)) * 32 + lane);
        d.x ^= c.x; d.y ^= c.y; d.z ^= c.z; d.w ^= c.w;
        T[(f + t) * 32 + lane] = d;
    }
}

// The 2^K - 1 node tables of one (q, P), in 512-byte slots at the start of
// `sm` (slot 2^s - 1 + t for node t of in-pass stage s).
//
// A heap layer of twiddles is GF(2)-linear in the node's offset within
// the layer (compute_twiddles fills each layer by XOR from its basis,
// src/binary_fft.rs:30-58).  The node offsets of the group's stage-s nodes
// are (group offset << s) | t, so node t has twiddle C_s ^ D_{s,t}: C_s =
// the twiddle of the group's first node at that stage, D_{s,t} = the
// layer's value at offset t, the same for every group of the launch.  A
// multiplication table is linear in its constant too: the block builds the
// K tables of C_s (slot 2^s - 1, where t = 0 and D = 0) and XORs each other
// slot from D's table (k_fft_dtab, once per launch), 4 words per access.
// Ends with the block synchronised.
template <int K>
__device__ __forceinline__ void build_pass_tables(uint8_t *sm, const PassArgs &a, unsigned q, unsigned P) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint64_t hbase = ((uint64_t)(a.root_base + q) << a.d0) + P;
    for (int s = warp; s < K; s += nw)
        tab_build_warp(reinterpret_cast<uint32_t *>(sm + ((1 << s) - 1) * 512), __ldg(a.tw + (hbase << s) - 1), lane);
    __syncthreads();
#pragma unroll
    for (int s = 1; s < K; ++s)
        fill_stage(reinterpret_cast<uint4 *>(sm), a.dtab, (1 << s) - 1, 1 << s, (1 << s) - 1, 0, (1 << s) - s - 1);
    __syncthreads();
}

// D tables (see build_pass_tables) of every pass of one FFT: pass p's slot
// 2^s - 1 + t holds the table of the value at offset t of heap layer
// l0[p] + s, l0[p] = the layer of that pass's group roots.  One warp per
// slot; blockIdx.y = pass.
struct DtabArgs {
    uint32_t l0[kMaxFftPasses], K[kMaxFftPasses];
};
__global__ void k_fft_dtab(const uint32_t *__restrict__ tw, DtabArgs d, uint32_t *__restrict__ out) {
    pdl_begin();
    const int lane = threadIdx.x & 31, p = blockIdx.y, K = (int)d.K[p];
    const int slot = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (slot >= (1 << K) - 1) return;
    const int s = 31 - __clz(slot + 1);
    const uint64_t t = (uint64_t)(slot + 1 - (1 << s));
    tab_build_warp(out + ((size_t)p * 63 + slot) * kTabWords, __ldg(tw + ((1ull << (d.l0[p] + s)) - 1) + t), lane);
}

// The leaf layer's twiddles are unscaled: node u has the polynomial 2u.  The
// nodes t = 0..3 of a pencil's last stage so have those of the first one plus
// 0, x, x^2, x^2 + x: one table serves all four, and this is the rest of the
// product, (2t) v, by shifts as multiplies (the pipe the lookups leave idle).
static __constant__ uint32_t kLeafMul[4] = {2u, 4u, 0x8289u, 16u};
__device__ __forceinline__ uint32_t leaf_rest(int t, uint32_t v) {
    if (t == 0) return 0;
    const uint64_t a = t & 1 ? fma_mul_wide(v, kLeafMul[0]) : 0, b = t & 2 ? fma_mul_wide(v, kLeafMul[1]) : 0;
    const uint32_t hi = (uint32_t)(a >> 32) ^ (uint32_t)(b >> 32);  // at most 2 bits past x^31
    // times the tail 0x8299: {0, 3, 7, 9, 15} and 4 apart, so nothing overlaps
    return (uint32_t)a ^ (uint32_t)b ^ fma_mul(hi, kLeafMul[2]) ^ fma_mul(hi, kLeafMul[3]);
}

// K stages over the NV values of a register pencil, node index of value i at
// in-pass stage s = (i >> (K - s)) + node_off(s); tables at tb + 512 * slot.
// Forward: fft_twiddles / fft_mul (src/binary_fft.rs:143-159, 180-192),
// stages root-first.  Inverse: ifft_twiddles / ifft_mul (:161-178,
// 194-206), leaves-first.  One flat loop so every register index is a
// compile-time constant after unrolling.
// ZERO0: the twiddle of each stage's node 0 is zero (its products are left
// out).  LEAF: the last stage is the transform's; its table is that of the
// pencil's first node, slot 2^s - 1 + the prefix (see leaf_rest).
template <int KP, int S0, bool INV, bool ZERO0 = false, bool LEAF = false>
__device__ __forceinline__ void pencil_stages(uint32_t (&v)[1 << KP], const uint8_t *sm, uint32_t tb,
                                              uint32_t gshift_slot) {
#pragma unroll
    for (int it = 0; it < KP * (1 << (KP - 1)); ++it) {
        const int sl = INV ? KP - 1 - (it >> (KP - 1)) : (it >> (KP - 1));  // stage within the phase
        const int s = S0 + sl;                                                  // stage within the pass
        const int w = it & ((1 << (KP - 1)) - 1);
        const int lh = KP - sl - 1;
        const int tp = w >> lh, u = w & ((1 << lh) - 1);
        const int x = (tp << (lh + 1)) + u, y = x + (1 << lh);
        // gshift_slot: runtime prefix of the node index inside this stage,
        // folded into the (256-aligned) base; the rest is a constant offset
        const bool leaf = LEAF && sl == KP - 1;
        const uint32_t base = tb + 512u * (leaf ? gshift_slot : gshift_slot << sl);
        const uint32_t off = 512u * ((1u << s) - 1u + (leaf ? 0u : (uint32_t)tp));
        if (!INV) {
            if (!ZERO0 || tp != 0) v[x] ^= tab_mul_sa(sm, base, off, v[y]);
            if (leaf) v[x] ^= leaf_rest(tp, v[y]);
            v[y] ^= v[x];
        } else {
            v[y] ^= v[x];
            if (!ZERO0 || tp != 0) v[x] ^= tab_mul_sa(sm, base, off, v[y]);
            if (leaf) v[x] ^= leaf_rest(tp, v[y]);
        }
    }
}

// Strided passes: a thread owns one "pencil", the 2^K rows
// P*2^(L-d0) + t*S + o (t < 2^K) of one vector, S = 2^(L-d0-K) > 1, in
// registers.  Threads of a block share (q, P) and hence every twiddle of
// the pass; lanes run over o, so each row access is coalesced.
// Work units are (group (q, P), chunk of blockDim.x pencils) in group-major
// order; block b takes the contiguous range [b U / B, (b+1) U / B), so one
// wave of blocks gets equal shares, and builds the node tables again only
// where its range enters the next group.
// Bulk copies of a unit's 2^K rows into buf[2^K][B], issued by the whole block
// (a.bulk: rows of S >= 32 words, 16-byte aligned): `cnt` pencils from the
// one at `src` on, columns `cs` words apart.
template <int K>
__device__ __forceinline__ void issue_unit(const uint32_t *src, uint32_t cs, uint32_t log_S, uint32_t cnt, uint32_t *buf,
                                           uint64_t *bar) {
    constexpr uint32_t R = 1u << K;
    const uint32_t B = blockDim.x, tid = threadIdx.x, S4 = 4u << log_S;
    if (tid == 0) mbar_expect(bar, 4 * R * cnt);
    if ((1ull << log_S) >= B) {  // one column's run of B words per row
        for (uint32_t t = tid; t < R; t += B) bulk_load(buf + t * B, strided(src, t, S4), 4 * B, bar);
    } else {  // B / S whole columns
        const uint32_t n = R * (cnt >> log_S);
        for (uint32_t c = tid; c < n; c += B) {
            const uint32_t t = c & (R - 1), col = c >> K;
            bulk_load(buf + t * B + (col << log_S), strided(src + (uint64_t)col * cs, t, S4), S4, bar);
        }
    }
}

// K <= 4: a thread also holds the next unit's pencil, loaded before this
// one's stages run so that its HBM latency hides behind them (64 registers,
// 4 blocks per SM; at 2^18 x 256 columns 168 us against 176 us with the rows
// staged by bulk copies, whose hand-over is a block barrier per unit).
// Larger pencils leave no registers for that: with a.bulk, bulk copies bring
// a unit's rows into shared memory, the next unit's issued as soon as this
// one's values are in registers (K = 6 at 2^12 x 1472 columns x 4: 143 us
// without, 100 us with them).
// ZERO0: the pass at the root of a whole transform, whose single group is the
// leftmost of its layers: 1 + 1/2 + 1/4 .. stages' worth of its products are
// with twiddle zero and left out (4 stages at 2^20 x 64 columns 157 -> 112 us,
// of which 82 are its words' way from and to memory).
template <int K, bool INV, bool ZERO0>
__global__ void __launch_bounds__(256, K <= 4 ? 4 : (K == 5 ? 3 : 2)) k_fft_pass(PassArgs a) {
    pdl_begin();
    extern __shared__ __align__(16) uint8_t smraw[];
    constexpr uint32_t R = 1u << K;
    constexpr bool PF = K <= 4;
    const uint32_t B = blockDim.x, tid = threadIdx.x;
    uint32_t *buf = reinterpret_cast<uint32_t *>(smraw + (R - 1) * 512);  // a.bulk: [R][B]
    uint64_t *bar = reinterpret_cast<uint64_t *>(buf + R * B);
    const uint32_t U = (uint32_t)a.units, nb = gridDim.x;
    const uint32_t u0 = (uint32_t)((uint64_t)blockIdx.x * U / nb), u1 = (uint32_t)((uint64_t)(blockIdx.x + 1) * U / nb);
    const uint32_t G = a.nvec << a.log_S, smask = (1u << a.log_S) - 1;  // pencils of a group (< 2^32 - 256)
    const uint32_t S4 = 4u << a.log_S;  // bytes between pencil values (a vector is < 4 GiB)
    const uint32_t cs = (uint32_t)a.col_stride;
    // the group's first word, and where pencil g of it starts
    auto group = [&](uint32_t grp) {
        return a.data + (grp >> a.d0) * a.q_stride + ((uint64_t)(grp & ((1u << a.d0) - 1)) << (a.L - a.d0));
    };
    auto pencil = [&](uint32_t *gp, uint32_t g) { return gp + (uint64_t)(g >> a.log_S) * cs + (g & smask); };
    uint32_t grp = u0 / a.bpg, ch = u0 - grp * a.bpg, parity = 0;
    uint32_t *gp = group(grp);
    uint32_t nv[PF ? R : 1], *p = gp;
    bool mine = false;
    auto prefetch = [&]() {  // the pencil of chunk ch of the group at gp
        const uint32_t g = ch * B + tid;
        mine = g < G;
        p = pencil(gp, g);
        if (PF && mine) {
#pragma unroll
            for (uint32_t t = 0; PF && t < R; ++t) nv[t] = *strided(p, t, S4);
        }
    };
    auto issue = [&]() {
        const uint32_t g0 = ch * B;
        issue_unit<K>(pencil(gp, g0), cs, a.log_S, min(B, G - g0), buf, bar);
    };
    if (!PF && a.bulk) {
        if (tid == 0) {
            mbar_init(bar, 1);
            fence_async();
        }
        __syncthreads();
        issue();
    }
    prefetch();
    bool fresh = true;  // the group's tables are to be built
    for (uint32_t u = u0; u < u1; ++u) {
        if (fresh) {
            if (u != u0) __syncthreads();  // every thread is done with the old tables
            build_pass_tables<K>(smraw, a, grp >> a.d0, grp & ((1u << a.d0) - 1));  // ends with the block synchronised
        }
        uint32_t *const base = p;
        const bool here = mine;
        uint32_t v[R];
        fresh = ++ch == a.bpg;
        if (fresh) {
            ch = 0;
            gp = group(++grp);
        }
        if constexpr (PF) {
#pragma unroll
            for (uint32_t t = 0; t < R; ++t) v[t] = nv[t];
            if (u + 1 < u1) prefetch();
        } else {
            if (a.bulk) {
                const bool there = mbar_wait(bar, parity, a.tries);
                if (here) {
#pragma unroll
                    for (uint32_t t = 0; t < R; ++t) v[t] = buf[t * B + tid];
                }
                fence_async();  // these reads before the next copies' writes: a barrier alone does not order the two proxies
                // the values are in registers: the next unit's copies may land
                if (__syncthreads_or(!there)) {
                    mbar_gave_up(bar, parity, a.fault);
                    return;
                }
                parity ^= 1;
                if (u + 1 < u1) issue();
            } else if (here) {
#pragma unroll
                for (uint32_t t = 0; t < R; ++t) v[t] = *strided(base, t, S4);
            }
            prefetch();
        }
        if (!here) continue;
        pencil_stages<K, 0, INV, ZERO0>(v, smraw, 0, 0);
#pragma unroll
        for (uint32_t t = 0; t < R; ++t) *strided(base, t, S4) = v[t];
    }
}

// The first pass of a Reed-Solomon encoding (rate 1/4): quarters q < 4 of
// each output column are the transforms under heap nodes 4 + q of the same
// input column scaled row by row with pis.  A thread loads its pencil of the
// input once, scales it and runs the K stages of all four quarters:
//   * the scaling is a general product per value (a row's constant serves
//     one value of each column, too few for a table); it uses the multiply
//     and logic pipes, the stages the shared-memory one;
//   * the roots' twiddles are GF(2)-linear in q and zero for q = 0, so the
//     first stage takes the products with roots 1 and 2 only (2 instead of
//     4 per pair), and q = 3 adds both;
//   * quarter 0's first node of every stage has twiddle zero too.
// For K = 4 that is 105 table products and 16 scalings a pencil instead of
// 128, 64 row loads less, and no scaled copy of the input in memory.
template <int K>
__global__ void __launch_bounds__(256, K <= 4 ? 3 : 2) k_rs_first(PassArgs a) {
    pdl_begin();
    extern __shared__ __align__(16) uint8_t smraw[];
    constexpr uint32_t R = 1u << K, H = R / 2, QT = (R - 1) * 512;  // QT: bytes of a quarter's tables
    const uint32_t B = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = B >> 5;
    uint32_t *buf = reinterpret_cast<uint32_t *>(smraw + 4 * QT);  // a.bulk: [R][B]
    uint64_t *bar = reinterpret_cast<uint64_t *>(buf + R * B);
    volatile uint32_t *gave_up = reinterpret_cast<uint32_t *>(bar + 1);  // a thread's wait ran out
    // units blockIdx.x, + gridDim.x, ...: every SM's blocks get the same number
    // of units to one (contiguous shares of 9 or 10 units a block left SMs
    // with 27 to 30)
    const uint32_t U = (uint32_t)a.units, u0 = blockIdx.x, nb = gridDim.x;
    const uint32_t G = a.nvec << a.log_S, smask = (1u << a.log_S) - 1;  // pencils (< 2^32 - 256)
    const uint32_t S4 = 4u << a.log_S;  // bytes between pencil values
    const uint32_t cs = (uint32_t)a.col_stride, scs = (uint32_t)a.src_col_stride;
    auto issue = [&](uint32_t u) {
        const uint32_t g0 = u * B;
        issue_unit<K>(a.src + (uint64_t)(g0 >> a.log_S) * scs + (g0 & smask), scs, a.log_S, min(B, G - g0), buf, bar);
    };
    if (a.bulk) {
        if (tid == 0) {
            mbar_init(bar, 1);
            *gave_up = 0;
            fence_async();
        }
        __syncthreads();
        issue(u0);
    }
    // The node tables of all four quarters (see build_pass_tables): the
    // offset of a quarter's first node in its layer is linear in q too, so
    // its twiddles are 0, C_1, C_2 and C_1 ^ C_2, and only those of quarters
    // 1 and 2 are built.
    for (uint32_t i = warp; i < 2 * K; i += nw) {
        const uint32_t q = 1 + i / K, s = i % K;
        tab_build_warp(reinterpret_cast<uint32_t *>(smraw + q * QT + ((1u << s) - 1) * 512),
                       __ldg(a.tw + ((4u + q) << s) - 1), lane);
    }
    __syncthreads();
    const uint4 *T1 = reinterpret_cast<const uint4 *>(smraw + QT), *T2 = reinterpret_cast<const uint4 *>(smraw + 2 * QT);
    for (uint32_t e = 32 + tid; e < (R - 1) * 32; e += B) {  // (the roots' slot 0 is there)
        const uint32_t slot = e >> 5, first = (1u << (31 - __clz(slot + 1))) - 1, f = first * 32 + (e & 31);
        uint4 d = make_uint4(0, 0, 0, 0);
        if (slot != first) d = __ldg(a.dtab + e);
        const uint4 c1 = T1[f], c2 = T2[f];
        uint4 *T = reinterpret_cast<uint4 *>(smraw);
        if (slot != first) {
            T[e] = d;
            T[QT / 16 + e] = make_uint4(c1.x ^ d.x, c1.y ^ d.y, c1.z ^ d.z, c1.w ^ d.w);
            T[2 * (QT / 16) + e] = make_uint4(c2.x ^ d.x, c2.y ^ d.y, c2.z ^ d.z, c2.w ^ d.w);
        }
        T[3 * (QT / 16) + e] = make_uint4(c1.x ^ c2.x ^ d.x, c1.y ^ c2.y ^ d.y, c1.z ^ c2.z ^ d.z, c1.w ^ c2.w ^ d.w);
    }
    __syncthreads();
    uint32_t parity = 0, u = u0;
    for (; u < U; u += nb) {
        const uint32_t g = u * B + tid;
        const bool mine = g < G;
        const uint32_t col = g >> a.log_S, o = g & smask;
        uint32_t v[R];
        const uint32_t *pp = a.pis + o;
        if (a.bulk) {
            if (!mbar_wait(bar, parity, a.tries)) *gave_up = 1;
            if (mine) {
#pragma unroll
                for (uint32_t t = 0; t < R; ++t) v[t] = buf[t * B + tid];
            }
            fence_async();  // these reads before the next copies' writes: a barrier alone does not order the two proxies
            __syncthreads();  // the values are in registers: the next unit's copies may land
            parity ^= 1;
            if (*gave_up) u = U;  // this unit's words are worth nothing, and it is the last
            if (u + nb < U) issue(u + nb);
        } else if (mine) {
            const uint32_t *lb = a.src + (uint64_t)col * scs + o;
#pragma unroll
            for (uint32_t t = 0; t < R; ++t) v[t] = *strided(lb, t, S4);
        }
        if (!mine) continue;
#pragma unroll
        for (uint32_t t = 0; t < R; ++t) v[t] = gf_mul(v[t], __ldg(strided(pp, t, S4)));
        uint32_t p1[H], p2[H];  // the first stage's products with roots 1 and 2
#pragma unroll
        for (uint32_t i = 0; i < H; ++i) {
            p1[i] = tab_mul_sa(smraw, 0, QT, v[H + i]);
            p2[i] = tab_mul_sa(smraw, 0, 2 * QT, v[H + i]);
        }
        uint32_t *out = a.data + (uint64_t)col * cs + o;
        {
            uint32_t x[H], y[H];
#pragma unroll
            for (uint32_t i = 0; i < H; ++i) {
                x[i] = v[i];
                y[i] = v[H + i] ^ v[i];
            }
            if constexpr (K > 1) {
                pencil_stages<K - 1, 1, false, true>(x, smraw, 0, 0);
                pencil_stages<K - 1, 1, false>(y, smraw, 0, 1);
            }
#pragma unroll
            for (uint32_t i = 0; i < H; ++i) {
                *strided(out, i, S4) = x[i];
                *strided(out, H + i, S4) = y[i];
            }
        }
#pragma unroll 1
        for (uint32_t q = 1; q < 4; ++q) {
            out += a.q_stride;
            const uint32_t m1 = 0u - (q & 1), m2 = 0u - (q >> 1);
            uint32_t x[H], y[H];
#pragma unroll
            for (uint32_t i = 0; i < H; ++i) {
                x[i] = v[i] ^ (p1[i] & m1) ^ (p2[i] & m2);
                y[i] = v[H + i] ^ x[i];
            }
            if constexpr (K > 1) {
                pencil_stages<K - 1, 1, false>(x, smraw, q * QT, 0);
                pencil_stages<K - 1, 1, false>(y, smraw, q * QT, 1);
            }
#pragma unroll
            for (uint32_t i = 0; i < H; ++i) {
                *strided(out, i, S4) = x[i];
                *strided(out, H + i, S4) = y[i];
            }
        }
    }
    if (a.bulk && *gave_up) mbar_gave_up(bar, parity ^ 1, a.fault);
}

// The node tables of a last pass's tile (see build_pass_tables): slots of
// stages 0 .. K-2, then one slot per phase-B pencil for the leaf stage, that
// of the pencil's first node (leaf_rest).
template <int K>
struct TailTables {
    static constexpr int KA = K / 2, KB = K - KA;
    static constexpr int kInner = (1 << (K - 1)) - 1, kSlots = kInner + (1 << KA);
    static __device__ __forceinline__ void build(uint8_t *sm, const PassArgs &a, unsigned q, unsigned P) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
        const uint64_t hbase = ((uint64_t)(a.root_base + q) << a.d0) + P;
        for (int s = warp; s < K; s += nw)
            tab_build_warp(reinterpret_cast<uint32_t *>(sm + ((1 << s) - 1) * 512), __ldg(a.tw + (hbase << s) - 1), lane);
        __syncthreads();
        uint4 *T = reinterpret_cast<uint4 *>(sm);
#pragma unroll
        for (int s = 1; s < K - 1; ++s)
            fill_stage(T, a.dtab, (1 << s) - 1, 1 << s, (1 << s) - 1, 0, (1 << s) - s - 1);
        fill_stage(T, a.dtab, kInner, 1 << KA, kInner, KB - 1, kInner - (K - 1));
        __syncthreads();
    }
};

// BULK: tiles in and out by bulk copies (launch_tail); an instantiation of its
// own, because both forms in one cost the bulk one 0.6% (2^20 x 64).
template <int K, bool INV, bool BULK>
__global__ void __launch_bounds__(256, 4) k_fft_tail(PassArgs a) {
    pdl_begin();
    constexpr int KA = K / 2, KB = K - KA, RB = 1 << KB, R = 1 << K, STRIDE = R + 4;
    extern __shared__ __align__(16) uint8_t smraw[];
    const unsigned chunk = blockIdx.x % a.nchunks, rest = blockIdx.x / a.nchunks;
    const unsigned P = rest & ((1u << a.d0) - 1);
    const unsigned q = rest >> a.d0;
    const uint32_t nvec = min(a.vchunk, a.nvec - chunk * a.vchunk);
    uint32_t *tile = reinterpret_cast<uint32_t *>(smraw + TailTables<K>::kSlots * 512);
    uint64_t *bar = reinterpret_cast<uint64_t *>(tile + a.vchunk * STRIDE);
    uint32_t *gbase = a.data + (uint64_t)chunk * a.vchunk * a.col_stride + q * a.q_stride + ((uint64_t)P << K);
    [[maybe_unused]] bool there = true;
    if constexpr (BULK) {
        if (threadIdx.x == 0) {
            mbar_init(bar, 1);
            fence_async();
            mbar_expect(bar, 4 * R * nvec);
        }
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < nvec; j += blockDim.x)
            bulk_load(tile + j * STRIDE, gbase + j * a.col_stride, 4 * R, bar);
        TailTables<K>::build(smraw, a, q, P);
        there = mbar_wait(bar, 0, a.tries);
    } else {
        constexpr uint32_t D = R / 16;  // 16-byte pieces a thread: 64 vectors, 256 threads
        uint4 d[D];
#pragma unroll
        for (uint32_t k = 0; k < D; ++k) {
            const uint32_t i = threadIdx.x + k * blockDim.x, j = i / (R / 4);
            if (j < nvec) d[k] = *reinterpret_cast<const uint4 *>(gbase + j * a.col_stride + 4 * (i % (R / 4)));
        }
        TailTables<K>::build(smraw, a, q, P);
#pragma unroll
        for (uint32_t k = 0; k < D; ++k) {
            const uint32_t i = threadIdx.x + k * blockDim.x, j = i / (R / 4);
            if (j < nvec) *reinterpret_cast<uint4 *>(tile + j * STRIDE + 4 * (i % (R / 4))) = d[k];
        }
        __syncthreads();
    }

    // Two register phases: KA stages on pencils of 2^KA values at stride
    // 2^KB, then KB stages on contiguous pencils of 2^KB values.  Work items
    // run over (vector, pencil) with a power-of-two span of vectors, so the
    // split is masks and shifts.
    const uint32_t lnv = 32 - __clz(nvec - 1), cl = min(3u, lnv);
    auto phase_a = [&]() {
        // item bits: 8 vectors, pencil, the other vectors
        for (uint32_t item = threadIdx.x; item < ((uint32_t)RB << lnv); item += blockDim.x) {
            const uint32_t u = (item >> cl) & (RB - 1), j = (item >> (cl + KB) << cl) | (item & ((1u << cl) - 1));
            if (j >= nvec) continue;
            uint32_t v[1 << KA];
#pragma unroll
            for (int i = 0; i < (1 << KA); ++i) v[i] = tile[j * STRIDE + u + RB * i];
            pencil_stages<KA, 0, INV>(v, smraw, 0, 0);
#pragma unroll
            for (int i = 0; i < (1 << KA); ++i) tile[j * STRIDE + u + RB * i] = v[i];
        }
    };
    auto phase_b = [&]() {
        for (uint32_t item = threadIdx.x; item < ((1u << KA) << lnv); item += blockDim.x) {
            const uint32_t j = item & ((1u << lnv) - 1), gq = item >> lnv;
            if (j >= nvec) continue;
            uint4 *p = reinterpret_cast<uint4 *>(tile + j * STRIDE + RB * gq);
            uint32_t v[RB];
#pragma unroll
            for (int i = 0; i < RB / 4; ++i) {
                const uint4 x = p[i];
                v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
            }
            pencil_stages<KB, KA, INV, false, true>(v, smraw, 0, gq);
#pragma unroll
            for (int i = 0; i < RB / 4; ++i) p[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
    };
    if (!INV) phase_a();
    else phase_b();
    if constexpr (BULK) {
        if (__syncthreads_or(!there)) {
            mbar_gave_up(bar, 0, a.fault);
            return;
        }
    } else {
        __syncthreads();
    }
    if (!INV) phase_b();
    else phase_a();
    if constexpr (!BULK) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < nvec * (R / 4); i += blockDim.x)
            *reinterpret_cast<uint4 *>(gbase + (uint64_t)(i / (R / 4)) * a.col_stride + 4 * (i % (R / 4))) =
                *reinterpret_cast<const uint4 *>(tile + (i / (R / 4)) * STRIDE + 4 * (i % (R / 4)));
    } else {
        fence_async();  // this thread's tile words, before the copies out
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < nvec; j += blockDim.x)
            bulk_store(gbase + j * a.col_stride, tile + j * STRIDE, 4 * R);
        bulk_store_wait();
    }
}

constexpr uint32_t kMinPassThreads = 64;
constexpr uint32_t kTailChunk = 64;  // vectors per tile of the last pass
static size_t pass_smem(int K) { return (size_t)((1 << K) - 1) * 512; }
static size_t tail_smem(int K, uint32_t vchunk) {
    const int slots = K == 4 ? TailTables<4>::kSlots : K == 5 ? TailTables<5>::kSlots : TailTables<6>::kSlots;
    return (size_t)slots * 512 + (size_t)vchunk * ((1u << K) + 4) * 4 + 16;
}
// strided pass: tables, then (bulk copies) the unit's rows and the barrier
static size_t strided_smem(int K, unsigned threads, bool bulk, bool rs_first = false) {
    return pass_smem(K) * (rs_first ? 4 : 1) + (bulk ? ((size_t)threads << K) * 4 + 16 : 0);
}

// One wave of blocks of a kernel: as many as fit on the device at once
// (occupancy at this size, cached by the caller's array), at most one per unit.
static unsigned wave_grid(const void *kernel, std::atomic<int> *occ_c, uint64_t units, unsigned threads, size_t smem) {
    static std::atomic<int> sms_c{0};  // idempotent fills; contexts may run on several threads
    int sms = sms_c.load(std::memory_order_relaxed);
    if (!sms) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            sms = 148;
        sms_c.store(sms, std::memory_order_relaxed);
    }
    int o = occ_c->load(std::memory_order_relaxed);
    if (!o) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kernel, (int)threads, smem) != cudaSuccess || o < 1) o = 1;
        occ_c->store(o, std::memory_order_relaxed);
    }
    return (unsigned)std::min<uint64_t>(units, (uint64_t)sms * o);
}

template <bool INV, bool ZERO0>
static cudaError_t launch_pass(Launcher &L, int K, PassArgs a, unsigned threads) {
    char nmbuf[48];
    std::snprintf(nmbuf, sizeof nmbuf, "%s_L%u_K%d_n%u", INV ? "ifft_pass" : "fft_pass", a.L, K, a.nvec);
    if (K <= 4) a.bulk = 0;  // those hold the next unit's values in registers
    const size_t smem = strided_smem(K, threads, a.bulk);
    // the kernel's limit is always set to its largest unit: contexts on other
    // threads launch the same kernel with other sizes, and a smaller limit
    // set between another thread's set and launch would fail it
    const int smem_max = (int)strided_smem(K, 256, K > 4);
    switch (K) {
#define LGK_CASE(k)                                                                                  \
    case k: {                                                                                        \
        static std::atomic<int> occ[2][257];                                                         \
        const void *fn = reinterpret_cast<const void *>(k_fft_pass<k, INV, ZERO0>);                         \
        if (smem_max > 48 * 1024) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max); \
        const unsigned blocks = wave_grid(fn, &occ[a.bulk][threads], a.units, threads, smem);        \
        LGK_LAUNCH(L, nmbuf, launch_k(k_fft_pass<k, INV, ZERO0>, blocks, threads, smem, L.stream, a));      \
        break;                                                                                       \
    }
        LGK_CASE(1) LGK_CASE(2) LGK_CASE(3) LGK_CASE(4) LGK_CASE(5) LGK_CASE(6)
#undef LGK_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

static cudaError_t launch_rs_first(Launcher &L, int K, const PassArgs &a, unsigned threads) {
    char nmbuf[48];
    std::snprintf(nmbuf, sizeof nmbuf, "fft_pass_L%u_K%d_n%u_rs", a.L, K, a.nvec);
    const size_t smem = strided_smem(K, threads, a.bulk, true);
    const int smem_max = (int)strided_smem(K, 256, true, true);  // as in launch_pass
    switch (K) {
#define LGK_CASE(k)                                                                                  \
    case k: {                                                                                        \
        static std::atomic<int> occ[2][257];                                                         \
        const void *fn = reinterpret_cast<const void *>(k_rs_first<k>);                              \
        if (smem_max > 48 * 1024) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max); \
        const unsigned blocks = wave_grid(fn, &occ[a.bulk][threads], a.units, threads, smem);        \
        LGK_LAUNCH(L, nmbuf, launch_k(k_rs_first<k>, blocks, threads, smem, L.stream, a));           \
        break;                                                                                       \
    }
        LGK_CASE(1) LGK_CASE(2) LGK_CASE(3) LGK_CASE(4) LGK_CASE(5)
#undef LGK_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <bool INV>
static cudaError_t launch_tail(Launcher &L, int K, PassArgs a, unsigned blocks) {
    char nmbuf[48];
    std::snprintf(nmbuf, sizeof nmbuf, "%s_L%u_K%d_n%u", INV ? "ifft_tail" : "fft_tail", a.L, K, a.nvec);
    const size_t smem = tail_smem(K, a.vchunk);
    const int smem_max = (int)tail_smem(K, kTailChunk);
    uint32_t vp2 = 1;
    while (vp2 < a.vchunk) vp2 <<= 1;
    // Enough tiles for several blocks a SM: the tile in and out by bulk copies,
    // which leave the load/store unit to the lookups, a thread per pencil of a
    // phase (vectors x 2^(K - K/2), the larger one) and at most 128: two pencils
    // a thread and more tiles in flight hide a tile's table fill and barriers
    // better (2^18 points: 64 columns 279 -> 265 us, 32 columns 195 -> 168 us).
    // Fewer tiles wait for their own latency: plain 16-byte loads and stores
    // without the copies' hand-over, and 256 threads to fill the tables (2^6 x
    // 64: 11.5 -> 10.3 us, 2^6 x 3: 15.2 -> 9.8; 590 tiles of 64 18.5 -> 17.8).
    // Tiles of fewer than 8 vectors are all table fill: no copies either.
    const bool many = blocks >= 148 * 4, bulk = many && a.vchunk >= 8;
    const unsigned threads = many ? std::max<unsigned>(32, std::min<unsigned>(128, vp2 << (K - K / 2))) : 256;
    switch (2 * K + bulk) {
#define LGK_CASE(k, b)                                                                                         \
    case 2 * k + b:                                                                                            \
        cudaFuncSetAttribute(k_fft_tail<k, INV, b>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);    \
        LGK_LAUNCH(L, nmbuf, launch_k(k_fft_tail<k, INV, b>, blocks, threads, smem, L.stream, a));             \
        break;
        LGK_CASE(4, false) LGK_CASE(5, false) LGK_CASE(6, false) LGK_CASE(4, true) LGK_CASE(5, true) LGK_CASE(6, true)
#undef LGK_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Stage split of `words` words in all (rs: of a Reed-Solomon encoding, whose
// first pass runs all four quarters of a pencil; aligned: the last pass can run
// in tiles in shared memory).  The lines lie where the best splits of 2^5 ..
// 2^18 points x 1 .. 3000 vectors change; over them this rule is on average
// within 2% of each shape's best split.
//   * A tile of the last pass waits for its tables, which double with every
//     stage.  A few tiles' waits are the launch's latency anyway (below 2^14
//     words: 6 stages; but never a strided pass of fewer than 3).  With up to two
//     tiles an SM, 5 stages (2^14 x 8: 24.9 us as 3 + 3 + 3 + 5, 25.5 as 3 + 2 + 3
//     + 6; inverse 2^13 x 130: 30.3 us as 4 + 4 + 5, 30.8 as 4 + 3 + 6); past
//     that 6 again (2^10 x 3000: 35.9 us as 4 + 6, 37.3 as 5 + 5), unless a tile
//     holds few vectors (one of 2^22: 500 us with 6, 340 with 5).
//   * The strided passes before it hold a 2^K-value pencil a thread: at most 4
//     stages where more threads hide more latency, 5 in large transforms, whose
//     passes cost their products.  An encoding's first pass has four times the
//     work a thread, so passes of 3 serve it longer (2^15 x 40: 85 us as 3 + 3 +
//     3 + 6, 89 as 4 + 5 + 6).  In an encoding the shorter passes come first; a
//     plain transform's first pass leaves many products out, so there the longer
//     ones do (inverse 2^20 x 64: 790 -> 759 us).
//   * Without tiles a thread of the last pass reads 2^K words in a row: 4 stages
//     are the most whose warps' lines stay in L1 (2^12 x 500: 49 us as 4 + 4 + 4,
//     77 as 3 + 4 + 5; 2^18 x 8: 86 and 128).
// The autotuner may replace it per shape.
constexpr uint64_t kTwoTilesAnSm = 2 * 148 * 64ull * kTailChunk;  // of 6 stages
FftPlan default_fft_plan(uint32_t log_len, uint64_t words, uint32_t nvec, bool rs, bool aligned) {
    uint32_t kt, most;
    if (!aligned) {
        kt = 4;
        most = words < (1u << 18) ? 3 : 4;
    } else if (log_len <= 6) {
        kt = most = log_len;
    } else if (rs) {
        kt = words < (1u << 16) ? 6 : words <= kTwoTilesAnSm || nvec < 8 ? 5 : 6;
        most = words <= kTwoTilesAnSm ? 3 : words < (1u << 24) || nvec < 8 ? 4 : 5;
    } else if (words < (1u << 14)) {
        kt = std::max(4u, std::min(6u, log_len - 3));
        most = 4;
    } else {
        kt = words <= kTwoTilesAnSm || nvec < 8 ? 5 : 6;
        most = words < (1u << 23) || nvec < 8 ? 4 : 5;
    }
    kt = std::min(kt, log_len);
    while (kt + most * (kMaxFftPasses - 1) < log_len) ++most;
    const uint32_t rem = log_len - kt, first = rs ? std::min(most, kRsFirstStages) : most;
    uint32_t nps = 0;
    while (rem > 0 && (nps == 0 || first + most * (nps - 1) < rem)) ++nps;
    FftPlan pl;
    pl.np = nps + 1;
    for (uint32_t i = 0; i < nps && i < kMaxFftPasses; ++i) pl.ks[i] = rem / nps + (rs ? nps - i <= rem % nps : i < rem % nps);
    if (nps < kMaxFftPasses) pl.ks[nps] = kt;
    return pl;
}

static bool plan_valid(const FftPlan &pl, uint32_t log_len) {
    if (pl.np == 0 || pl.np > kMaxFftPasses) return false;
    uint32_t sum = 0;
    for (uint32_t i = 0; i < pl.np; ++i) {
        if (pl.ks[i] < 1 || pl.ks[i] > 6) return false;
        sum += pl.ks[i];
    }
    // the last pass runs in tiles when it has 4..6 stages; strided passes
    // before it need at least one level below them
    return sum == log_len;
}

constexpr uint64_t kMaxFftWords = 1ull << 32;  // of a call's vectors: pencils have at least two words
cudaError_t fft_vectors(Launcher &L, uint32_t *data, const uint32_t *tw, uint32_t log_len,
                        uint32_t nvec, uint64_t col_stride, uint32_t Q, uint64_t q_stride,
                        uint32_t root_base, bool inverse, FftPasses passes, const FftSrc *src) {
    if (log_len == 0 || nvec == 0) return cudaSuccess;
    if (inverse && passes != FFT_ALL) return cudaErrorInvalidValue;
    // a source is a Reed-Solomon encoding's: one input for the four quarters
    if (src && (inverse || log_len <= 6 || passes == FFT_LAST || Q != 4 || root_base != 4 || !src->pis))
        return cudaErrorInvalidValue;
    // the roots root_base + q (q < Q) must share one heap layer
    // the passes count pencils and stride columns in 32 bits: larger batches
    // run in parts
    if (col_stride >> 32 || (src && src->col_stride >> 32)) return cudaErrorInvalidValue;
    if (((uint64_t)nvec << log_len) > kMaxFftWords && nvec > 1) {
        const uint32_t half = nvec / 2;
        FftSrc s2;
        if (src) {
            s2 = *src;
            s2.p += half * src->col_stride;
        }
        cudaError_t e = fft_vectors(L, data, tw, log_len, half, col_stride, Q, q_stride, root_base, inverse, passes, src);
        if (e != cudaSuccess) return e;
        return fft_vectors(L, data + half * col_stride, tw, log_len, nvec - half, col_stride, Q, q_stride, root_base,
                           inverse, passes, src ? &s2 : nullptr);
    }
    const uint32_t lr = 31 - __builtin_clz(root_base);
    if (!L.dtab || root_base == 0 || ((root_base + Q - 1) >> lr) != 1) return cudaErrorInvalidValue;
    // head / last calls on column groups must agree on the split, so only
    // whole transforms take tuned plans
    // (nor does the size of one group change the default)
    const bool aligned = ((uintptr_t)data % 16 == 0) && (col_stride % 4 == 0) && (q_stride % 4 == 0);
    const uint64_t words = passes == FFT_ALL ? (uint64_t)Q * nvec << log_len : ~0ull;
    FftPlan plan = default_fft_plan(log_len, words, passes == FFT_ALL ? nvec : ~0u, src != nullptr || passes != FFT_ALL, aligned);
    if (L.split.np && plan_valid(L.split, log_len)) {
        plan = L.split;
    } else if (passes == FFT_ALL && !L.forced_plan) {
        const TuneKey tk{L.device, log_len, nvec, Q, src != nullptr, inverse, 0};
        if (!tuned_fft_plan(tk, &plan) && L.autotune) {
            cudaError_t e = tune_fft(L, tk, data, tw, col_stride, q_stride, root_base, src, &plan);
            if (e != cudaSuccess) return e;
        }
    }
    if (L.forced_plan) plan = *L.forced_plan;
    if (!plan_valid(plan, log_len) || (src && plan.ks[0] > kMaxRsFirst)) return cudaErrorInvalidValue;
    const uint32_t np = plan.np;
    std::vector<uint32_t> ks(plan.ks, plan.ks + np);
    std::vector<uint32_t> d0s(np);
    for (uint32_t i = 0, d = 0; i < np; ++i) { d0s[i] = d; d += ks[i]; }
    // D tables of every pass; kept while the same twiddle subtree is asked
    // for again with the same split (the twiddle arrays live, unchanged, as
    // long as the context)
    const Launcher::DtabKey key{tw, log_len, root_base, plan_code(plan)};
    uint32_t slot = 0;
    while (slot < kDtabSlots && !(L.dtab_key[slot] == key)) ++slot;
    if (slot == kDtabSlots) {
        slot = 0;
        for (uint32_t i = 1; i < kDtabSlots; ++i)
            if (L.dtab_used[i] < L.dtab_used[slot]) slot = i;
        DtabArgs d{};
        for (uint32_t p = 0; p < np; ++p) { d.l0[p] = lr + d0s[p]; d.K[p] = ks[p]; }
        LGK_LAUNCH(L, "fft_dtab",
                   launch_k(k_fft_dtab, dim3(8, np), 256, 0, L.stream, tw, d, L.dtab + slot * kDtabWords));
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) { L.dtab_key[slot] = {}; return e; }
        L.dtab_key[slot] = key;
    }
    L.dtab_used[slot] = ++L.dtab_clock;
    const uint32_t *dtab = L.dtab + slot * kDtabWords;
    uint32_t nvec_p2 = 1;
    while (nvec_p2 < nvec) nvec_p2 <<= 1;
    for (uint32_t pi = 0; pi < np; ++pi) {
        const uint32_t p = inverse ? np - 1 - pi : pi;
        if ((passes == FFT_HEAD && p == np - 1) || (passes == FFT_LAST && p != np - 1)) continue;
        const uint32_t K = ks[p], d0 = d0s[p];
        PassArgs a;
        a.data = data; a.tw = tw; a.col_stride = col_stride; a.q_stride = q_stride;
        a.dtab = reinterpret_cast<const uint4 *>(dtab + (size_t)p * 63 * kTabWords);
        a.src = (src && p == 0) ? src->p : nullptr;
        a.src_col_stride = src ? src->col_stride : 0;
        a.pis = a.src ? src->pis : nullptr;
        a.L = log_len; a.d0 = d0; a.log_S = log_len - d0 - K;
        a.nvec = nvec; a.root_base = root_base; a.fault = L.fault; a.tries = L.copy_tries;
        const bool tail = a.log_S == 0 && K >= 4 && aligned;
        // the root of a whole transform: each stage's first node is the first of
        // its layer, whose twiddle is zero
        const bool zero0 = !tail && !a.src && d0 == 0 && Q == 1 && (root_base & (root_base - 1)) == 0;
        {
            // every vector read (the source once for all quarters) and written
            // once; a product a butterfly and stage, but those with twiddle zero
            // that the pass leaves out (see k_fft_pass and k_rs_first)
            const double words = (double)Q * nvec * (1ull << log_len), R = 1u << K;
            if (a.src) {
                const double in = words / Q, table = R + 2 * (K - 1) * R - (R / 2 - 1);  // a pencil's
                L.note(4.0 * (in + words), in / R * (R + table), 0, in);
            } else {
                L.note(8.0 * words, words / 2 * K - (zero0 ? words * (1 - 1 / R) : 0));
            }
        }
        if (tail) {
            a.vchunk = std::min<uint32_t>(nvec, kTailChunk);
            a.nchunks = (nvec + a.vchunk - 1) / a.vchunk;
            const uint64_t blocks = ((uint64_t)Q << d0) * a.nchunks;
            if (blocks > 0x7FFFFFFFull) return cudaErrorInvalidValue;
            cudaError_t e = inverse ? launch_tail<true>(L, (int)K, a, (unsigned)blocks)
                                    : launch_tail<false>(L, (int)K, a, (unsigned)blocks);
            if (e != cudaSuccess) return e;
            continue;
        }
        const uint64_t G = (uint64_t)nvec << a.log_S;  // pencils per (q, P)
        uint32_t B = (uint32_t)std::max<uint64_t>(32, std::min<uint64_t>((uint64_t)nvec_p2 << a.log_S, 256));
        // small transforms: smaller blocks until every SM has one
        while (B > kMinPassThreads && (a.src ? 1 : ((uint64_t)Q << d0)) * ((G + B - 1) / B) < 148) B /= 2;
        a.bpg = (uint32_t)((G + B - 1) / B);
        a.units = a.src ? a.bpg : ((uint64_t)Q << d0) * a.bpg;  // k_rs_first: all quarters in a unit
        a.nchunks = 0;
        const bool src_aligned = !a.src || ((uintptr_t)a.src % 16 == 0 && a.src_col_stride % 4 == 0);
        // rows of at least 32 words: below that a bulk copy moves too little
        a.bulk = aligned && src_aligned && a.log_S >= 5;
        cudaError_t e = a.src     ? launch_rs_first(L, (int)K, a, B)
                        : zero0   ? (inverse ? launch_pass<true, true>(L, (int)K, a, B)
                                             : launch_pass<false, true>(L, (int)K, a, B))
                        : inverse ? launch_pass<true, false>(L, (int)K, a, B)
                                  : launch_pass<false, false>(L, (int)K, a, B);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// =============================================================== Merkle
// a tree node (or chaining value): 8 words, two 16-byte accesses
__device__ __forceinline__ void load_node(const uint32_t *p, uint32_t (&h)[8]) {
    const uint4 x = reinterpret_cast<const uint4 *>(p)[0], y = reinterpret_cast<const uint4 *>(p)[1];
    h[0] = x.x; h[1] = x.y; h[2] = x.z; h[3] = x.w; h[4] = y.x; h[5] = y.y; h[6] = y.z; h[7] = y.w;
}
__device__ __forceinline__ void store_node(uint32_t *p, const uint32_t (&h)[8]) {
    reinterpret_cast<uint4 *>(p)[0] = make_uint4(h[0], h[1], h[2], h[3]);
    reinterpret_cast<uint4 *>(p)[1] = make_uint4(h[4], h[5], h[6], h[7]);
}

constexpr uint64_t kHashBound = 1ull << 13;

// Leaf = the row's n words as LE bytes, one BLAKE3 chunk (n <= 256):
// blocks of 16 words, CHUNK_START on the first, CHUNK_END|ROOT on the last.
// A thread hashes blocks b0 .. b0 + nb_run - 1 of one row's leaf, from the IV
// or from the chaining value an earlier call left in out.  Bound by the
// compression (lg_device.cuh); a whole block's 16 loads take one
// multiply-add each for their address and no predicate.  MA: see b3_add.
template <bool MA>
__global__ void __launch_bounds__(128) k_leaf_hash(const uint32_t *__restrict__ E, uint64_t rows, uint32_t ncols,
                                                   uint32_t b0, uint32_t nb_run, uint32_t *__restrict__ out,
                                                   uint64_t e_stride, uint64_t out_stride) {
    pdl_begin();
    E += blockIdx.y * e_stride;  // lockstep batch: proof blockIdx.y
    out += blockIdx.y * out_stride;
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= rows) return;
    const uint32_t nb = (ncols + 15) / 16, rows4 = (uint32_t)(4 * rows);  // a column is < 4 GiB
    uint32_t cv[8];
    if (b0 == 0) b3_iv(cv);
    else load_node(out + 8 * i, cv);
    // a block's words are loaded while the one before it is compressed
    const uint32_t *p = E + 16ull * b0 * rows + i;
    uint32_t nx[16];
    auto load = [&](uint32_t b) {
        if (16 * (b + 1) <= ncols) {
#pragma unroll
            for (uint32_t w = 0; w < 16; ++w) nx[w] = __ldg(strided(p, w, rows4));
        } else {
#pragma unroll
            for (uint32_t w = 0; w < 16; ++w) nx[w] = b * 16 + w < ncols ? __ldg(strided(p, w, rows4)) : 0u;
        }
        p += 16 * rows;
    };
    load(b0);
    for (uint32_t b = b0; b < b0 + nb_run; ++b) {
        uint32_t m[16];
#pragma unroll
        for (uint32_t w = 0; w < 16; ++w) m[w] = nx[w];
        if (b + 1 < b0 + nb_run) load(b + 1);
        const bool last = b + 1 == nb;
        const uint32_t blen = last ? 4 * ncols - 64 * (nb - 1) : 64;
        const uint32_t flags = (b == 0 ? B3_CHUNK_START : 0u) | (last ? (B3_CHUNK_END | B3_ROOT) : 0u);
        b3_compress<MA>(cv, m, blen, flags);
    }
    store_node(out + 8 * i, cv);
}

// Few hashes wait for their compressions' latency, which plain additions
// shorten (a 2^12-leaf tree: 13.2 us against 14.0); more are bound by the
// logic pipe's rate (2^16 leaves of 64 words: 22.8 us with plain additions,
// 19.4 with multiply-adds; their tree 21.4 and 17.5).
static bool hash_bound(uint64_t hashes) { return hashes > kHashBound; }
static auto hash_kernel(uint64_t rows, uint32_t B) { return hash_bound(rows * B) ? k_leaf_hash<true> : k_leaf_hash<false>; }

cudaError_t leaf_hash_block(Launcher &L, const uint32_t *E, uint64_t rows, uint32_t ncols, uint32_t b0,
                            uint32_t nb, uint32_t *out) {
    if (ncols == 0 || ncols > 256 || nb == 0 || b0 + nb > (ncols + 15) / 16 || rows >= (1ull << 30))
        return cudaErrorInvalidValue;
    const unsigned blocks = (unsigned)((rows + 127) / 128);
    const uint32_t cols = std::min<uint32_t>(16 * nb, ncols - 16 * b0);
    L.note((double)rows * (4.0 * cols + (b0 ? 64.0 : 32.0)), 0, (double)rows * nb);
    LGK_LAUNCH(L, "leaf_hash_block", launch_k(hash_kernel(rows, 1), blocks, 128, 0, L.stream, E, rows, ncols, b0, nb, out, 0, 0));
    return cudaGetLastError();
}

cudaError_t leaf_hashes(Launcher &L, const uint32_t *E, uint64_t rows, uint32_t ncols, uint32_t *out, uint32_t B,
                        uint64_t e_stride, uint64_t out_stride) {
    if (B == 0 || B > 65535 || ncols == 0 || rows >= (1ull << 30)) return cudaErrorInvalidValue;
    const uint32_t nb = (ncols + 15) / 16;
    const dim3 blocks((unsigned)((rows + 127) / 128), B);
    L.note((double)B * rows * (4.0 * ncols + 32.0), 0, (double)B * rows * nb);
    LGK_LAUNCH(L, "leaf_hash", launch_k(hash_kernel(rows, B), blocks, 128, 0, L.stream, E, rows, ncols, 0, nb, out, e_stride,
                                        out_stride));
    return cudaGetLastError();
}

// Node = blake3(left || right): one 64-byte block, CHUNK_START|CHUNK_END|ROOT
// (src/merkle_tree.rs:42-51).  A block reduces 2^c consecutive nodes of one
// layer through c layers in shared memory and writes every layer it makes.
template <bool MA = true>
__device__ __forceinline__ void hash_node(const uint32_t *l, const uint32_t *r, uint32_t *o) {
    uint32_t m[16];
#pragma unroll
    for (int w = 0; w < 8; ++w) { m[w] = l[w]; m[8 + w] = r[w]; }
    uint32_t cv[8];
    b3_iv(cv);
    b3_compress<MA>(cv, m, 64, B3_CHUNK_START | B3_CHUNK_END | B3_ROOT);
#pragma unroll
    for (int w = 0; w < 8; ++w) o[w] = cv[w];
}

// The tree is stored leaves first, layer after layer, 8 words per node.
// Wide layers: a thread takes 8 consecutive nodes (256 contiguous bytes)
// and hashes the 7 nodes of the three layers above them, keeping at most
// three pending hashes; every lane does full work, so these launches run
// at hashing throughput.
__global__ void __launch_bounds__(128) k_merkle_thread3(uint32_t *__restrict__ tree, uint64_t in_off, uint64_t n_in,
                                                        uint64_t tree_stride) {
    pdl_begin();
    tree += blockIdx.y * tree_stride;  // lockstep batch: proof blockIdx.y
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (8 * t >= n_in) return;
    const uint64_t off1 = in_off + n_in, off2 = off1 + n_in / 2, off3 = off2 + n_in / 4;
    const uint32_t *src = tree + 8 * (in_off + 8 * t);
    // The 7 nodes in post order, one compression per iteration (a single
    // copy of it in the code: seven inlined copies stalled on instruction
    // fetch): i = 0, 1 hash leaf pairs 0, 1 into layer-1 nodes A0, A1; i = 2
    // hashes (A0, A1) into B0; i = 3, 4 leaf pairs 2, 3 into A2, A3; i = 5
    // (A2, A3) into B1; i = 6 (B0, B1) into the layer-3 node.
    uint32_t l[8], r[8], h[8], a[8], b[8];
    load_node(src, l);
    load_node(src + 8, r);
#pragma unroll 1
    for (uint32_t i = 0; i < 7; ++i) {
        hash_node(l, r, h);
        const uint64_t at = (i == 6)                ? off3 + t
                            : (i == 2 || i == 5)    ? off2 + 2 * t + (i == 5)
                                                    : off1 + 4 * t + (i < 2 ? i : i - 1);
        store_node(tree + 8 * at, h);
        if (i == 0 || i == 2 || i == 3) {
            // the next compression hashes leaf pair 1 (after i = 0), 2 or 3
            if (i != 2) {
#pragma unroll
                for (int w = 0; w < 8; ++w) a[w] = h[w];
            } else {
#pragma unroll
                for (int w = 0; w < 8; ++w) b[w] = h[w];
            }
            const uint32_t *s = src + 16 * (i == 0 ? 1 : i);
            load_node(s, l);
            load_node(s + 8, r);
        } else {
            // i = 1, 4: (a, h) are the two layer-1 children; i = 5: (b, h)
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                l[w] = i == 5 ? b[w] : a[w];
                r[w] = h[w];
            }
        }
    }
}

// Narrow layers (a layer of at most 2^18 nodes up to the root) in one
// launch: a block of 256 threads takes 512 consecutive nodes (or the whole
// layer when it is smaller) and climbs 9 layers, one per barrier -- the
// first layer up reads the tree, the later ones a shared-memory copy of the
// layer below -- writing every node to the tree.  Each block then takes a
// ticket; the last block to finish climbs from the blocks' roots (at most
// 512 nodes, read back from the tree) to the root.  No block waits for
// another.
constexpr uint32_t kNarrowNodes = 512, kNarrowMax = kNarrowNodes * kNarrowNodes;

// Climbs from m nodes (m a power of two, <= 512) of the layer at `off`
// (nodes first .. first + m - 1 of a layer of n) to their common ancestor;
// src_tree: the first layer is read from the tree with loads that bypass
// L1 (nodes other blocks wrote).  Ends with the block synchronised.
template <bool MA>
__device__ __forceinline__ void narrow_climb(uint32_t *__restrict__ tree, uint64_t off, uint64_t n, uint64_t first,
                                             uint32_t m, uint32_t *buf_a, uint32_t *buf_b) {
    const uint32_t t = threadIdx.x;
    if (t < m / 2) {
        uint32_t l[8], r[8], h[8];
        const uint4 *pl = reinterpret_cast<const uint4 *>(tree + 8 * (off + first + 2 * t));
        const uint4 a0 = __ldcg(pl), a1 = __ldcg(pl + 1), b0 = __ldcg(pl + 2), b1 = __ldcg(pl + 3);
        l[0] = a0.x; l[1] = a0.y; l[2] = a0.z; l[3] = a0.w; l[4] = a1.x; l[5] = a1.y; l[6] = a1.z; l[7] = a1.w;
        r[0] = b0.x; r[1] = b0.y; r[2] = b0.z; r[3] = b0.w; r[4] = b1.x; r[5] = b1.y; r[6] = b1.z; r[7] = b1.w;
        hash_node<MA>(l, r, h);
        store_node(tree + 8 * (off + n + first / 2 + t), h);
#pragma unroll
        for (int j = 0; j < 8; ++j) buf_a[j * (kNarrowNodes / 2) + t] = h[j];
    }
    off += n;
    n >>= 1;
    first >>= 1;
    m >>= 1;
    __syncthreads();
    uint32_t *src = buf_a, *dst = buf_b;
    uint32_t ss = kNarrowNodes / 2, ds = kNarrowNodes / 4;
    while (m > 1) {
        if (t < m / 2) {
            uint32_t l[8], r[8], h[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint2 x = *reinterpret_cast<const uint2 *>(src + j * ss + 2 * t);
                l[j] = x.x;
                r[j] = x.y;
            }
            hash_node<MA>(l, r, h);
            store_node(tree + 8 * (off + n + first / 2 + t), h);
#pragma unroll
            for (int j = 0; j < 8; ++j) dst[j * ds + t] = h[j];
        }
        off += n;
        n >>= 1;
        first >>= 1;
        m >>= 1;
        __syncthreads();
        uint32_t *tp = src;
        src = dst;
        dst = tp;
        const uint32_t ts = ss;
        ss = ds;
        ds = ts;
    }
}

template <bool MA>
__global__ void __launch_bounds__(256) k_merkle_narrow(uint32_t *__restrict__ tree, uint64_t in_off, uint64_t n_in,
                                                       uint32_t *ticket, uint64_t tree_stride, uint32_t *root) {
    pdl_begin();
    tree += blockIdx.y * tree_stride;  // lockstep batch: proof blockIdx.y, its own ticket
    ticket += blockIdx.y;
    // layers in shared memory word-major (word j of node i at [j * stride +
    // i]): a thread reads its two children's word j as one 8-byte load
    __shared__ __align__(16) uint32_t buf_a[8 * (kNarrowNodes / 2)];
    __shared__ __align__(16) uint32_t buf_b[8 * (kNarrowNodes / 4)];
    __shared__ uint32_t last;
    const uint32_t per = (uint32_t)(n_in < kNarrowNodes ? n_in : kNarrowNodes), nb = gridDim.x;
    narrow_climb<MA>(tree, in_off, n_in, (uint64_t)blockIdx.x * per, per, buf_a, buf_b);
    // the root once more where the caller asks for it
    auto copy_root = [&](uint64_t off) {
        if (root && threadIdx.x < 8) root[threadIdx.x] = __ldcg(tree + 8 * off + threadIdx.x);
    };
    if (nb == 1) {
        copy_root(in_off + 2 * n_in - 2);
        return;
    }
    // the layer of the blocks' roots
    uint64_t off = in_off, n = n_in;
    for (uint32_t m = per; m > 1; m >>= 1) { off += n; n >>= 1; }
    __threadfence();  // this block's nodes are visible before its ticket
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == nb - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x == 0) *ticket = 0;  // ready for the next launch on the stream
    narrow_climb<MA>(tree, off, n, 0, nb, buf_a, buf_b);
    copy_root(in_off + 2 * n_in - 2);
}

cudaError_t merkle_upper(Launcher &L, uint32_t *tree, uint64_t num_leaves, uint32_t B, uint64_t tree_stride,
                         uint32_t *root) {
    if ((root && (B != 1 || num_leaves < 2)) || num_leaves == 0 || (num_leaves & (num_leaves - 1)) || !L.tickets || B == 0 || B > kMaxTickets)
        return cudaErrorInvalidValue;
    uint64_t off = 0, n = num_leaves;
    // Three layers per launch with a thread per 8 nodes while a layer has
    // more than 2^18 nodes (every lane does full work); from a layer of
    // 2^18 or fewer, one launch climbs to the root.
    while (n > 1) {
        cudaError_t e;
        if (n > kNarrowMax) {
            const uint64_t threads = n / 8;
            L.note(32.0 * B * (n + n / 2 + n / 4 + n / 8), (double)0, (double)B * (n / 2 + n / 4 + n / 8));
            LGK_LAUNCH(L, "merkle_thread3", launch_k(k_merkle_thread3, dim3((unsigned)((threads + 127) / 128), B), 128,
                                                     0, L.stream, tree, off, n, tree_stride));
            e = cudaGetLastError();
            for (int l = 0; l < 3; ++l) { off += n; n /= 2; }
        } else {
            const uint64_t per = std::min<uint64_t>(n, kNarrowNodes);
            L.note(32.0 * B * (2 * n - 1), 0, (double)B * (n - 1));
            LGK_LAUNCH(L, "merkle_narrow", launch_k(hash_bound(n * B) ? k_merkle_narrow<true> : k_merkle_narrow<false>, dim3((unsigned)(n / per), B), 256, 0, L.stream,
                                                    tree, off, n, L.tickets, tree_stride, root));
            e = cudaGetLastError();
            n = 1;
        }
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// ============================================================== gathers
// An opening in one launch: threads below nq*ncols copy the opened rows
// (row q[k] of every column), the rest the 8 words of each Merkle node
// (the node count on the device when d_count is given, at most count).
__global__ void k_gather_opening(const uint32_t *__restrict__ E, uint64_t rows, uint32_t ncols,
                                 const uint64_t *__restrict__ q, uint32_t nq, const uint32_t *__restrict__ tree,
                                 const uint64_t *__restrict__ node_idx, uint32_t count, const uint32_t *d_count,
                                 uint32_t *__restrict__ out, GatherStrides st) {
    pdl_begin();
    const uint32_t b = blockIdx.y;  // lockstep batch: proof b
    E += b * st.E;
    q += b * st.q;
    tree += b * st.tree;
    node_idx += b * st.nodes;
    if (d_count) d_count += b * st.count;
    out += b * st.out;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, nrow = nq * ncols;
    if (t < nrow) {
        const uint32_t k = t / ncols, j = t % ncols;
        out[t] = E[(uint64_t)j * rows + q[k]];
        return;
    }
    const uint32_t u = t - nrow;
    if (d_count) count = min(count, *d_count);
    if (u >= count * 8) return;
    out[t] = tree[8 * node_idx[u / 8] + (u % 8)];
}
cudaError_t gather_opening(Launcher &L, const uint32_t *E, uint64_t rows, uint32_t ncols, const uint64_t *d_queries,
                           uint32_t nq, const uint32_t *tree, const uint64_t *d_node_index, uint32_t count,
                           const uint32_t *d_count, uint32_t *out, uint32_t B, const GatherStrides &st) {
    const uint64_t total = (uint64_t)nq * ncols + 8ull * count;
    if (total == 0) return cudaSuccess;
    if (total > 0xFFFFFFFFull || B == 0 || B > 65535) return cudaErrorInvalidValue;
    L.note(8.0 * B * total, 0);
    LGK_LAUNCH(L, "gather_opening", launch_k(k_gather_opening, dim3((unsigned)((total + 255) / 256), B), 256, 0,
                                             L.stream, E, rows, ncols, d_queries, nq, tree, d_node_index, count,
                                             d_count, out, st));
    return cudaGetLastError();
}

// evaluate_lagrange_basis (src/utils.rs:4-27) entry j of k challenges:
// rs[0] selects the index MSB, factor rs[i] where the bit is set, 1 + rs[i]
// where not (field products commute, so the order is immaterial).
__device__ __forceinline__ uint32_t lagrange_at(const uint32_t *rs, uint32_t k, uint32_t j) {
    uint32_t p = 1;
    for (uint32_t i = 0; i < k; ++i) p = gf_mul(p, ((j >> (k - 1 - i)) & 1) ? rs[i] : 1u ^ rs[i]);
    return p;
}

// ============================================================== clusters
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_load(const uint32_t *p, uint32_t rank) {
    uint32_t v;
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.u32 %0, [a];\n\t}"
                 : "=r"(v)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank)
                 : "memory");
    return v;
}
__device__ __forceinline__ void cluster_store(const uint32_t *p, uint32_t rank, uint32_t v) {
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.shared::cluster.u32 [a], %2;\n\t}" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(p)),
                 "r"(rank), "r"(v)
                 : "memory");
}

// ================================================================= folds
// partial_eval over the top k variables (src/multilinear_poly.rs:66-87):
// out[i] = sum_j eq(rs, j) in[j*M + i], j's top bit with rs[0] -- the
// reference's sequence of folds (1 + r) a + r b, each exact, collapsed into
// one sum of products (the same field element).  The eq weights split over
// j = (jh, jl): eq(rs, j) = eq(rs[..kh], jh) * eq(rs[kh..], jl), so
// out[i] = sum_jh EH[jh] * (sum_jl EL[jl] * in[(jh 2^kl + jl) M + i]): the
// inner sums take 2^k products over 2^kl tables shared by every lane, the
// outer 2^kh more over 2^kh tables.  A block builds its 2^kl + 2^kh tables
// once and then loops over outputs, four consecutive ones per thread (one
// 16-byte load per term); every product in an inner sum is independent of
// the others, so loads and lookups overlap.
struct Rs6 { uint32_t v[kMaxFold]; };

template <int KH, int KL, int V>
__global__ void __launch_bounds__(256) k_fold_eq(const uint32_t *__restrict__ in, uint32_t *__restrict__ out,
                                                 uint64_t M, Rs6 rs, const uint32_t *d_rs, FoldStrides st) {
    pdl_begin();
    in += blockIdx.y * st.in;  // lockstep batch: proof blockIdx.y
    out += blockIdx.y * st.out;
    if (d_rs) d_rs += blockIdx.y * st.rs;
    constexpr int NH = 1 << KH, NL = 1 << KL;
    __shared__ __align__(512) uint32_t tabs[NH + NL][kTabWords];  // EL tables, then EH
    __shared__ uint32_t r[KH + KL];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    // V consecutive outputs per thread (16-byte loads for V = 4)
    const uint64_t groups = M / V, gstride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    // V = 1: all 2^k inputs of an output are loaded at once, the first
    // output's before the tables are built and the next one's right after
    // the current one's products, so that the loads' HBM latency overlaps
    // the table builds and the products
    constexpr int NV = V == 1 ? NH * NL : 1;
    uint32_t pre[NV];
    auto load_all = [&](uint64_t gg) {
#pragma unroll
        for (int j = 0; j < NV; ++j) pre[j] = __ldg(in + gg + (uint64_t)j * M);
    };
    if (V == 1 && g < groups) load_all(g);
    if (threadIdx.x < KH + KL) r[threadIdx.x] = d_rs ? d_rs[threadIdx.x] : rs.v[threadIdx.x];
    __syncthreads();
    // evaluate_lagrange_basis (src/utils.rs:4-27) of each half: entry j has
    // r where j's bit is set and 1 + r where not, the half's first challenge
    // on j's top bit
    for (int t = warp; t < NL + NH; t += nw) {
        const bool lo = t < NL;
        const int j = lo ? t : t - NL, nb = lo ? KL : KH, off = lo ? KH : 0;
        uint32_t e = 1;
        for (int b = 0; b < nb; ++b) e = gf_mul(e, ((j >> (nb - 1 - b)) & 1) ? r[off + b] : 1u ^ r[off + b]);
        tab_build_warp(tabs[t], e, lane);
    }
    __syncthreads();
    const uint8_t *t8 = reinterpret_cast<const uint8_t *>(&tabs[0][0]);
    if constexpr (V == 1) {
        for (; g < groups; g += gstride) {
            uint32_t acc = 0;
#pragma unroll
            for (int jh = 0; jh < NH; ++jh) {
                uint32_t part = 0;
#pragma unroll
                for (int jl = 0; jl < NL; ++jl) part ^= tab_mul_sa(t8, 512u * jl, 0, pre[jh * NL + jl]);
                acc ^= KH ? tab_mul_sa(t8, 512u * (NL + jh), 0, part) : part;
            }
            if (g + gstride < groups) load_all(g + gstride);
            out[g] = acc;
        }
    } else {
        for (; g < groups; g += gstride) {
            const uint32_t *src = in + g * V;
            uint32_t acc[V];
#pragma unroll
            for (int x = 0; x < V; ++x) acc[x] = 0;
#pragma unroll
            for (int jh = 0; jh < NH; ++jh) {
                uint32_t v[NL][V];
#pragma unroll
                for (int jl = 0; jl < NL; ++jl) {
                    const uint32_t *p = src + (uint64_t)(jh * NL + jl) * M;
                    const uint4 t = __ldg(reinterpret_cast<const uint4 *>(p));
                    v[jl][0] = t.x; v[jl][1] = t.y; v[jl][2] = t.z; v[jl][3] = t.w;
                }
#pragma unroll
                for (int x = 0; x < V; ++x) {
                    uint32_t part = 0;
#pragma unroll
                    for (int jl = 0; jl < NL; ++jl) part ^= tab_mul_sa(t8, 512u * jl, 0, v[jl][x]);
                    acc[x] ^= KH ? tab_mul_sa(t8, 512u * (NL + jh), 0, part) : part;
                }
            }
            *reinterpret_cast<uint4 *>(out + g * 4) = make_uint4(acc[0], acc[1], acc[2], acc[3]);
        }
    }
}

// The same sum when there are few outputs: a cluster of 8 blocks takes 256
// of them, block c the terms of its NH / 8 high indexes jh, and the blocks'
// partial sums meet in shared memory (block c adds up outputs 32 c .. 32 c +
// 31).  Bound by latency: a term's load, product and sum are 8 times fewer a
// thread, and up to 9 variables fold at once.
template <int KH, int KL>
__global__ void __launch_bounds__(256) k_fold_split(const uint32_t *__restrict__ in, uint32_t *__restrict__ out,
                                                    uint64_t M, Rs6 rs, const uint32_t *d_rs, FoldStrides st) {
    pdl_begin();
    in += blockIdx.y * st.in;  // lockstep batch: proof blockIdx.y
    out += blockIdx.y * st.out;
    if (d_rs) d_rs += blockIdx.y * st.rs;
    constexpr int NH = 1 << KH, NL = 1 << KL, H = NH / 8;
    __shared__ __align__(512) uint32_t tabs[NL + H][kTabWords];  // EL tables, then this block's EH
    __shared__ uint32_t r[KH + KL], ec[NL + H], part[256], red[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t c = cluster_rank();
    const uint64_t o0 = (uint64_t)(blockIdx.x / 8) * 256, o = o0 + threadIdx.x;
    const bool mine = o < M;
    uint32_t v[H * NL];
    if (mine) {
#pragma unroll
        for (int j = 0; j < H * NL; ++j) v[j] = __ldg(in + o + (uint64_t)(c * H * NL + j) * M);
    }
    if (threadIdx.x < KH + KL) r[threadIdx.x] = d_rs ? d_rs[threadIdx.x] : rs.v[threadIdx.x];
    __syncthreads();
    if (threadIdx.x < NL + H) {  // the constants as in k_fold_eq
        const int t = threadIdx.x;
        const bool lo = t < NL;
        const int j = lo ? t : (int)c * H + t - NL, nb = lo ? KL : KH, off = lo ? KH : 0;
        uint32_t e = 1;
        for (int b = 0; b < nb; ++b) e = gf_mul(e, ((j >> (nb - 1 - b)) & 1) ? r[off + b] : 1u ^ r[off + b]);
        ec[t] = e;
    }
    __syncthreads();
    for (int t = warp; t < NL + H; t += 8) tab_build_warp(tabs[t], ec[t], lane);
    __syncthreads();
    const uint8_t *t8 = reinterpret_cast<const uint8_t *>(&tabs[0][0]);
    uint32_t acc = 0;
    if (mine) {
#pragma unroll
        for (int h = 0; h < H; ++h) {
            uint32_t sum = 0;
#pragma unroll
            for (int j = 0; j < NL; ++j) sum ^= tab_mul_sa(t8, 512u * j, 0, v[h * NL + j]);
            acc ^= tab_mul_sa(t8, 512u * (NL + h), 0, sum);
        }
    }
    part[threadIdx.x] = acc;
    cluster_sync();
    red[warp][lane] = cluster_load(&part[32 * c + lane], warp);
    __syncthreads();
    if (warp == 0) {
        uint32_t x = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) x ^= red[w][lane];
        if (o0 + 32 * c + lane < M) out[o0 + 32 * c + lane] = x;
    }
    cluster_sync();  // no block leaves while its sums may still be read
}

// Few outputs: the split form, where one thread an output would leave most of
// the device idle (2^10 outputs of 64 terms on 4 blocks: 5.8 us, split 3.6).
// Sixteen terms leave a cluster's blocks two each, less than their exchange
// costs (2^14 words by 4, a call: 17.8 us, split 19.1).
// More than 6 variables at once only for very few outputs: 2^22 words by 9
// take 22 us so, 13 us as 6 and then 3.
bool fold_splits(uint32_t log_len, uint32_t k, uint32_t B) {
    if (k < 5 || k > kMaxFold || log_len < k) return false;
    const uint64_t chunks = (((1ull << (log_len - k)) + 255) / 256) * B;
    return chunks <= (k <= 6 ? 64 : 8);
}

static bool tuned_fold(const TuneKey &k, int *bps);
static void tune_fold(Launcher &L, const TuneKey &k, bool few);
constexpr int kFoldVec4 = 0x100, kFoldSplit = 0x200;

cudaError_t fold_eq(Launcher &L, const uint32_t *in, uint32_t *out, uint32_t log_len, uint32_t k,
                    const uint32_t *rs, const uint32_t *d_rs, uint32_t B, const FoldStrides &st) {
    const bool few = fold_splits(log_len, k, B);
    if (k < 1 || (k > 6 && !few) || k > log_len || (!rs && !d_rs) || B == 0 || B > 65535) return cudaErrorInvalidValue;
    Rs6 c{};
    if (!d_rs)
        for (uint32_t j = 0; j < k; ++j) c.v[j] = rs[j];
    const uint64_t M = 1ull << (log_len - k);
    const uint32_t kh = k / 2;
    // choice: blocks per SM in the low byte, kFoldVec4 for four outputs per
    // thread, or kFoldSplit; tuned per shape (by default split with few
    // outputs, else one output per thread and 4 blocks per SM)
    int choice = few ? kFoldSplit : 4;
    if (k > 6) {
        // only split
    } else if (L.forced_fold) {
        choice = L.forced_fold;
    } else {
        const TuneKey tk{L.device, log_len, k, 1, false, false, 1};
        if (!tuned_fold(tk, &choice) && L.autotune) {
            tune_fold(L, tk, few);
            tuned_fold(tk, &choice);
        }
    }
    if (choice == kFoldSplit && few) {
        const dim3 grid((unsigned)((M + 255) / 256) * 8, B);
        L.note(B * (4.0 * (M << k) + 4.0 * M), (double)B * M * ((1u << k) + (k >= 8 ? 16 : 8)));
        switch (k) {
#define LGK_CASE(kk, kh)                                                                                   \
    case kk:                                                                                               \
        LGK_LAUNCH(L, "fold_eq", launch_kc(k_fold_split<kh, kk - kh>, grid, 256, 8, 0, L.stream, in, out, M, c, d_rs, st)); \
        break;
            LGK_CASE(5, 3) LGK_CASE(6, 3) LGK_CASE(7, 3) LGK_CASE(8, 4) LGK_CASE(9, 4)
#undef LGK_CASE
        }
        return cudaGetLastError();
    }
    if (choice == kFoldSplit) choice = 4;  // tuned for fewer proofs at a time
    const int bps = choice & 0xFF;
    const bool vec4 = (choice & kFoldVec4) && M % 4 == 0 && (uintptr_t)in % 16 == 0 && (uintptr_t)out % 16 == 0;
    const uint64_t groups = vec4 ? M / 4 : M;
    const dim3 blocks(
        (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((groups + 255) / 256, 148ull * (uint64_t)bps)), B);
    L.note(B * (4.0 * (M << k) + 4.0 * M), (double)B * M * ((1u << k) + (kh ? (1u << kh) : 0)));
    switch (2 * k + (vec4 ? 1 : 0)) {
#define LGK_CASE(kk)                                                                                          \
    case 2 * kk:                                                                                              \
        LGK_LAUNCH(L, "fold_eq", launch_k(k_fold_eq<kk / 2, kk - kk / 2, 1>, blocks, 256, 0, L.stream, in, out, M, c, d_rs, st)); \
        break;                                                                                                \
    case 2 * kk + 1:                                                                                          \
        LGK_LAUNCH(L, "fold_eq", launch_k(k_fold_eq<kk / 2, kk - kk / 2, 4>, blocks, 256, 0, L.stream, in, out, M, c, d_rs, st)); \
        break;
        LGK_CASE(1) LGK_CASE(2) LGK_CASE(3) LGK_CASE(4) LGK_CASE(5) LGK_CASE(6)
#undef LGK_CASE
    }
    return cudaGetLastError();
}

// =============================================================== sumcheck
__device__ __forceinline__ uint32_t warp_xor(uint32_t v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v ^= __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void block_xor3(uint32_t s0, uint32_t s1, uint32_t s2, uint32_t *acc3) {
    __shared__ uint32_t red[3];
    if (threadIdx.x < 3) red[threadIdx.x] = 0;
    __syncthreads();
    s0 = warp_xor(s0); s1 = warp_xor(s1); s2 = warp_xor(s2);
    if ((threadIdx.x & 31) == 0) { atomicXor(&red[0], s0); atomicXor(&red[1], s1); atomicXor(&red[2], s2); }
    __syncthreads();
    if (threadIdx.x < 3) atomicXor(acc3 + threadIdx.x, red[threadIdx.x]);
}

// evals_at_x with x = 3 (src/ligerito.rs:130-141): 3*hi + (1+3)*lo = x*(hi+lo) + hi
__device__ __forceinline__ uint32_t at3(uint32_t lo, uint32_t hi) { return gf_mulx(hi ^ lo) ^ hi; }

// eval_013_product (src/multilinear_poly.rs:90-131)
// the FS tail of proof b of a lockstep batch
__device__ __forceinline__ FsTail tail_for(FsTail t, const RoundStrides &st, uint32_t b) {
    if (t.fs) {
        t.fs += b * st.fs;
        t.ticket += b * st.ticket;
        if (t.out) t.out += b * st.out;
    }
    return t;
}

__global__ void k_eval013(const uint32_t *__restrict__ f, const uint32_t *__restrict__ g, uint64_t half,
                          uint32_t *acc3, FsTail tail, RoundStrides st) {
    pdl_begin();
    const uint32_t b = blockIdx.y;  // lockstep batch: proof b
    f += b * st.f;
    g += b * st.g;
    acc3 += b * st.acc;
    tail = tail_for(tail, st, b);
    const uint32_t fs_pre = fsd::fs_tail_prefetch(tail);
    uint32_t s0 = 0, s1 = 0, s2 = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < half; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t f0 = f[i], f1 = f[half + i], g0 = g[i], g1 = g[half + i];
        s0 ^= gf_mul(f0, g0);
        s1 ^= gf_mul(f1, g1);
        s2 ^= gf_mul(at3(f0, f1), at3(g0, g1));
    }
    block_xor3(s0, s1, s2, acc3);
    if (tail.fs) fsd::fs_tail_block(tail, acc3, fs_pre);
}
cudaError_t eval013(Launcher &L, const uint32_t *f, const uint32_t *g, uint32_t log_len, uint32_t *acc3,
                    const FsTail *tail, uint32_t B, const RoundStrides &st) {
    if (B == 0 || B > 65535) return cudaErrorInvalidValue;
    const uint64_t half = 1ull << (log_len - 1);
    const dim3 blocks((unsigned)std::max<uint64_t>(1, std::min<uint64_t>((half + 255) / 256, 148ull * 4)), B);
    const FsTail t = tail ? *tail : FsTail{};
    L.note(16.0 * B * half, 3.0 * B * half, 0, 3.0 * B * half);
    LGK_LAUNCH(L, "eval013", launch_k(k_eval013, blocks, 256, 0, L.stream, f, g, half, acc3, t, st));
    return cudaGetLastError();
}

// SumcheckProverInstance::fold (src/ligerito.rs:119-127): partial_eval of f
// and of the (summed) basis by r, (1+r)a + r b = a + r(a+b), then
// eval_01x_product on the folded pair.
__global__ void __launch_bounds__(256) k_fold_round(const uint32_t *__restrict__ f, const uint32_t *__restrict__ B,
                                                    uint64_t quarter, uint32_t r, const uint32_t *d_r,
                                                    uint32_t *__restrict__ fo, uint32_t *__restrict__ Bo,
                                                    uint32_t *acc3, FsTail tail, RoundStrides st) {
    pdl_begin();
    {
        const uint32_t b = blockIdx.y;  // lockstep batch: proof b
        f += b * st.f;
        B += b * st.g;
        fo += b * st.fo;
        Bo += b * st.go;
        acc3 += b * st.acc;
        if (d_r) d_r += b * st.r;
        tail = tail_for(tail, st, b);
    }
    __shared__ __align__(128) uint32_t T[kTabWords];
    // the thread's first words are loaded before the challenge's table is
    // built, so the two memory latencies overlap; each later iteration's
    // words load while the current one is multiplied
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    uint32_t v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    auto load = [&](uint64_t j) {
        v[0] = f[j]; v[1] = f[quarter + j]; v[2] = f[2 * quarter + j]; v[3] = f[3 * quarter + j];
        v[4] = B[j]; v[5] = B[quarter + j]; v[6] = B[2 * quarter + j]; v[7] = B[3 * quarter + j];
    };
    if (i < quarter) load(i);
    const uint32_t fs_pre = fsd::fs_tail_prefetch(tail);
    if (threadIdx.x < 32) tab_build_warp(T, d_r ? *d_r : r, threadIdx.x);
    __syncthreads();
    const uint8_t *t8 = reinterpret_cast<const uint8_t *>(T);
    uint32_t s0 = 0, s1 = 0, s2 = 0;
    for (; i < quarter; i += stride) {
        const uint32_t a0 = v[0], a1 = v[1], a2 = v[2], a3 = v[3], c0 = v[4], c1 = v[5], c2 = v[6], c3 = v[7];
        if (i + stride < quarter) load(i + stride);
        const uint32_t flo = a0 ^ tab_mul_sa(t8, 0, 0, a0 ^ a2), fhi = a1 ^ tab_mul_sa(t8, 0, 0, a1 ^ a3);
        const uint32_t blo = c0 ^ tab_mul_sa(t8, 0, 0, c0 ^ c2), bhi = c1 ^ tab_mul_sa(t8, 0, 0, c1 ^ c3);
        fo[i] = flo; fo[quarter + i] = fhi;
        Bo[i] = blo; Bo[quarter + i] = bhi;
        s0 ^= gf_mul(flo, blo);
        s1 ^= gf_mul(fhi, bhi);
        s2 ^= gf_mul(at3(flo, fhi), at3(blo, bhi));
    }
    block_xor3(s0, s1, s2, acc3);
    if (tail.fs) fsd::fs_tail_block(tail, acc3, fs_pre);
}
cudaError_t fold_round(Launcher &L, const uint32_t *f, const uint32_t *B, uint32_t log_len, uint32_t r,
                       uint32_t *fo, uint32_t *Bo, uint32_t *acc3, const uint32_t *d_r, const FsTail *tail,
                       uint32_t NB, const RoundStrides &st) {
    if (log_len < 2 || NB == 0 || NB > 65535) return cudaErrorInvalidValue;
    const uint64_t quarter = 1ull << (log_len - 2);
    const dim3 blocks((unsigned)std::max<uint64_t>(1, std::min<uint64_t>((quarter + 255) / 256, 148ull * 4)), NB);
    L.note(48.0 * NB * quarter, 7.0 * NB * quarter, 0, 3.0 * NB * quarter);
    LGK_LAUNCH(L, "fold_round_grid", launch_k(k_fold_round, blocks, 256, 0, L.stream, f, B, quarter, r, d_r, fo, Bo, acc3,
                                         tail ? *tail : FsTail{}, st));
    return cudaGetLastError();
}

// glue (src/ligerito.rs:59-67) folded into the running basis sum
__global__ void k_axpy(uint32_t *__restrict__ B, const uint32_t *__restrict__ bi, uint64_t n, uint32_t beta,
                       const uint32_t *d_beta, RoundStrides st) {
    pdl_begin();
    B += blockIdx.y * st.f;  // lockstep batch: proof blockIdx.y
    bi += blockIdx.y * st.g;
    if (d_beta) d_beta += blockIdx.y * st.r;
    __shared__ __align__(128) uint32_t T[kTabWords];
    // the first words load before the table is built (their latencies overlap)
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    uint32_t b0 = 0, x0 = 0;
    if (i < n) { b0 = B[i]; x0 = bi[i]; }
    if (threadIdx.x < 32) tab_build_warp(T, d_beta ? *d_beta : beta, threadIdx.x);
    __syncthreads();
    for (; i < n; i += stride) {
        const uint32_t b = b0, x = x0;
        if (i + stride < n) { b0 = B[i + stride]; x0 = bi[i + stride]; }
        B[i] = b ^ tab_mul_sa(reinterpret_cast<const uint8_t *>(T), 0, 0, x);
    }
}
cudaError_t axpy(Launcher &L, uint32_t *B, const uint32_t *bi, uint32_t log_len, uint32_t beta,
                 const uint32_t *d_beta, uint32_t NB, const RoundStrides &st) {
    if (NB == 0 || NB > 65535) return cudaErrorInvalidValue;
    const uint64_t n = 1ull << log_len;
    const dim3 blocks((unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, 148ull * 4)), NB);
    L.note(12.0 * NB * n, (double)NB * n);
    LGK_LAUNCH(L, "axpy", launch_k(k_axpy, blocks, 256, 0, L.stream, B, bi, n, beta, d_beta, st));
    return cudaGetLastError();
}

// A whole sumcheck step, or its last rounds, in one launch: a cluster of C
// blocks keeps f and the basis in its shared memory, evaluates the step's
// opening triple and folds round after round, and warp 0 of its first block
// runs the transcript between them.
//   * Block c holds the words whose index modulo M = 2^(log_len - rounds - 1)
//     lies in [c M / C, (c+1) M / C): every fold and every triple pairs words
//     that differ in a higher bit, so no round moves data between blocks.
//   * A round is one product table, the folds and products, an XOR reduction,
//     two cluster barriers (the blocks' partial triples to the first block,
//     its challenge back) and the transcript's one or two SHA-256
//     compressions.
// Bound by that chain's latency: a step of 2^10 words (opening triple and four
// rounds) takes 29 us in one launch, 54 us as five (event-timed), one of 2^14
// with its glue 33 against 70 us as six.
struct SumStepArgs {
    const uint32_t *f, *B, *bi;  // bi: the basis to glue into B (after the opening triple), or null
    uint32_t log_len, rounds;
    uint32_t eval, nsq;          // eval: opening triple over (f, bi or B), checked against tri[3], then nsq challenges
    uint32_t *tri;               // 4 words a triple: the opening one's, then one a round
    uint32_t *chal;              // the opening's challenges and the rounds' after them; !eval: the first round's is there
    uint32_t *fo, *Bo;           // 2^(log_len - rounds) words
    FsState *fs;
    const uint32_t *end;  // mirror: end_words words from here go to pinned memory at the end
    uint32_t end_words, *mirror;
};
// in shared memory, without its words
struct SumStepShared {
    FsState S;
    fsd::FsWork work;
    uint32_t tri[2][4];   // the triple, a copy for each transcript warp
    uint32_t part[8][4];  // the blocks' partial triples (first block)
    uint32_t red[8][4];   // the warps'
    uint32_t r[4];        // the challenges the first block hands out
};
static_assert(offsetof(SumStepShared, work) % 16 == 0, "the schedules' rows are read 16 bytes at a time");
constexpr uint32_t kSumThreads = 256;
__global__ void __launch_bounds__(kSumThreads) k_sum_step(SumStepArgs a, RoundStrides st, uint32_t C) {
    pdl_begin();
    extern __shared__ __align__(512) uint8_t ssraw[];
    {
        const uint32_t b = blockIdx.y;  // lockstep batch: proof b
        a.f += b * st.f;
        a.B += b * st.g;
        if (a.bi) a.bi += b * st.f;
        a.tri += b * st.acc;
        a.chal += b * st.out;
        a.fo += b * st.fo;
        a.Bo += b * st.go;
        a.fs += b * st.fs;
    }
    uint32_t *T = reinterpret_cast<uint32_t *>(ssraw);  // the table of the challenge
    SumStepShared &sh = *reinterpret_cast<SumStepShared *>(ssraw + 4 * kTabWords);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c = cluster_rank();
    const uint32_t lw = a.log_len - a.rounds - 1 - (31 - __clz(C)), w = 1u << lw;  // 2^lw words a run of this block
    uint32_t len = w << (a.rounds + 1);                                            // its words
    uint32_t *F = reinterpret_cast<uint32_t *>(ssraw + 4 * kTabWords + ((sizeof(SumStepShared) + 15) & ~15u)), *G = F + len;
    uint32_t *I = G + len;  // bi's words
    // global index of local word x: run x >> lw, offset x & (w - 1)
    auto at = [&](uint32_t x) { return (x >> lw << (lw + 31 - __clz(C))) + c * w + (x & (w - 1)); };
    for (uint32_t x = tid; x < len; x += kSumThreads) {
        F[x] = a.f[at(x)];
        G[x] = a.B[at(x)];
        if (a.bi) I[x] = a.bi[at(x)];
    }
    if (c == 0)
        for (uint32_t i = tid; i < fsd::kFsStateWords; i += kSumThreads)
            reinterpret_cast<uint32_t *>(&sh.S)[i] = reinterpret_cast<const uint32_t *>(a.fs)[i];
    cluster_sync();  // the block's words are there, and every block of the cluster has started
    const uint8_t *t8 = reinterpret_cast<const uint8_t *>(T);
    // the triple s0, s1, s2 over the whole cluster, absorbed by the first
    // block (checked against tri[3] if `check`), then nsq challenges; the
    // last one, and the one before it in beta's place, in sh.r everywhere
    uint32_t *tri = a.tri, *chal = a.eval ? a.chal : a.chal + 1;
    auto transcript = [&](uint32_t s0, uint32_t s1, uint32_t s2, bool check, uint32_t nsq) {
        s0 = __reduce_xor_sync(0xffffffffu, s0);
        s1 = __reduce_xor_sync(0xffffffffu, s1);
        s2 = __reduce_xor_sync(0xffffffffu, s2);
        if (lane == 0) { sh.red[warp][0] = s0; sh.red[warp][1] = s1; sh.red[warp][2] = s2; }
        __syncthreads();
        if (tid < 3) {
            uint32_t x = 0;
#pragma unroll
            for (uint32_t i = 0; i < kSumThreads / 32; ++i) x ^= sh.red[i][tid];
            cluster_store(&sh.part[c][tid], 0, x);
        }
        cluster_sync();
        if (c == 0 && warp < 2) {
            if (lane < 3) {
                uint32_t x = 0;
                for (uint32_t i = 0; i < C; ++i) x ^= sh.part[i][lane];
                sh.tri[warp][lane] = x;
                if (warp == 0) tri[lane] = x;
            }
            __syncwarp();
            fsd::fs_step_warps(sh.S, sh.work, sh.tri[warp], 3, nsq);
            if (warp == 0) {
                if (lane == 0 && check && (sh.tri[0][0] ^ sh.tri[0][1]) != tri[3]) sh.S.err |= FS_ERR_SUMCHECK;
                if (lane < nsq) chal[lane] = sh.work.sq[lane];
                for (uint32_t i = 0; i < nsq; ++i)
                    if (lane < C) cluster_store(&sh.r[i], lane, sh.work.sq[i]);
            }
        }
        tri += 4;
        chal += nsq;
        if (nsq) cluster_sync();
    };
    auto table = [&](uint32_t x) {  // T = the table of x; the block's words are settled too
        if (warp == 0) tab_build_warp(T, x, lane);
        __syncthreads();
    };
    uint32_t nsq = 1;
    if (a.eval) {
        const uint32_t *g = a.bi ? I : G;
        uint32_t s0 = 0, s1 = 0, s2 = 0;
        for (uint32_t x = tid; x < len / 2; x += kSumThreads) {
            const uint32_t f0 = F[x], f1 = F[len / 2 + x], g0 = g[x], g1 = g[len / 2 + x];
            s0 ^= gf_mul(f0, g0);
            s1 ^= gf_mul(f1, g1);
            s2 ^= gf_mul(at3(f0, f1), at3(g0, g1));
        }
        nsq = a.nsq;
        transcript(s0, s1, s2, true, nsq);
        if (a.bi) {  // glue: B += beta bi
            table(sh.r[0]);
            for (uint32_t x = tid; x < len; x += kSumThreads) G[x] ^= tab_mul_sa(t8, 0, 0, I[x]);
            __syncthreads();
        }
    } else {
        if (tid == 0) sh.r[0] = *a.chal;
        __syncthreads();
    }
    for (uint32_t k = 0; k < a.rounds; ++k) {
        table(sh.r[k == 0 ? nsq - 1 : 0]);
        const uint32_t q = len / 4;
        uint32_t s0 = 0, s1 = 0, s2 = 0;
        for (uint32_t i = tid; i < q; i += kSumThreads) {
            const uint32_t a0 = F[i], a1 = F[q + i], a2 = F[2 * q + i], a3 = F[3 * q + i];
            const uint32_t c0 = G[i], c1 = G[q + i], c2 = G[2 * q + i], c3 = G[3 * q + i];
            const uint32_t flo = a0 ^ tab_mul_sa(t8, 0, 0, a0 ^ a2), fhi = a1 ^ tab_mul_sa(t8, 0, 0, a1 ^ a3);
            const uint32_t blo = c0 ^ tab_mul_sa(t8, 0, 0, c0 ^ c2), bhi = c1 ^ tab_mul_sa(t8, 0, 0, c1 ^ c3);
            F[i] = flo; F[q + i] = fhi;
            G[i] = blo; G[q + i] = bhi;
            s0 ^= gf_mul(flo, blo);
            s1 ^= gf_mul(fhi, bhi);
            s2 ^= gf_mul(at3(flo, fhi), at3(blo, bhi));
        }
        len /= 2;
        transcript(s0, s1, s2, false, k + 1 < a.rounds ? 1 : 0);
    }
    __syncthreads();
    for (uint32_t x = tid; x < len; x += kSumThreads) {
        a.fo[at(x)] = F[x];
        a.Bo[at(x)] = G[x];
    }
    if (c == 0)
        for (uint32_t i = tid; i < fsd::kFsStateWords; i += kSumThreads)
            reinterpret_cast<uint32_t *>(a.fs)[i] = reinterpret_cast<const uint32_t *>(&sh.S)[i];
    // The last step of a proof hands the host its results itself: a copy after
    // the kernel cost 7 us of a 2^16 proof's 186.
    if (a.mirror) {
        cluster_sync();  // the other blocks' words of `end` are written
        for (uint32_t i = c * kSumThreads + tid; i < a.end_words; i += C * kSumThreads) a.mirror[i] = __ldcg(a.end + i);
    }
}
static size_t sum_step_smem(uint32_t log_len, uint32_t C, bool bi) {
    return 4 * kTabWords + ((sizeof(SumStepShared) + 15) & ~size_t(15)) + ((bi ? 12ull : 8ull) << log_len) / C;
}
// Blocks of a step's cluster: enough that a round gives a thread one or two
// items, at most 8 (the portable size) and no more than the device's SMs for
// the whole batch; 0 when the step does not fit.
static uint32_t sum_step_cluster(uint32_t log_len, uint32_t rounds, uint32_t NB, bool bi) {
    if (rounds == 0 || log_len < rounds + 1 || log_len > kSumStepMaxLog) return 0;
    uint32_t C = 1;
    while (C < 8 && (1ull << (log_len - 2)) / C > kSumThreads && 2 * C * NB <= 148 && (2 * C >> (log_len - rounds - 1)) == 0)
        C *= 2;
    return sum_step_smem(log_len, C, bi) <= 200 * 1024 ? C : 0;
}
bool sum_step_fits(uint32_t log_len, uint32_t rounds, uint32_t NB, bool glue) {
    return sum_step_cluster(log_len, rounds, NB, glue) != 0;
}
cudaError_t sum_step(Launcher &L, const SumStep &s, uint32_t NB, const RoundStrides &st) {
    const uint32_t C = sum_step_cluster(s.log_len, s.rounds, NB, s.bi != nullptr);
    if (C == 0 || NB == 0 || NB > 65535 || s.nsq > 2 || (s.eval && s.nsq == 0) || (s.mirror && NB != 1))
        return cudaErrorInvalidValue;
    SumStepArgs a;
    a.f = s.f; a.B = s.B; a.bi = s.bi; a.log_len = s.log_len; a.rounds = s.rounds; a.eval = s.eval; a.nsq = s.nsq;
    a.tri = s.tri; a.chal = s.chal; a.fo = s.fo; a.Bo = s.Bo; a.fs = s.fs;
    a.end = s.end; a.end_words = s.end_words; a.mirror = s.mirror;
    const size_t smem = sum_step_smem(s.log_len, C, s.bi != nullptr);
    if (smem > 48 * 1024) cudaFuncSetAttribute(k_sum_step, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    // the opening triple takes 3 general products a pair of words, the glue one
    // table product a word, a round 4 and 3 for four words; the rounds' words
    // halve
    const double n = (double)NB * (1ull << s.log_len), out = n / (1u << s.rounds), folded = 2 * (n - out) / 4;
    const double opening = s.eval ? 1.5 * n : 0, glue = s.bi ? n : 0;
    L.note(8.0 * n + 4.0 * glue + 8.0 * out, opening + glue + 7.0 * folded, 0, opening + 3.0 * folded);
    // (the name of the rounds in a cluster; a round over the whole device, bound
    // otherwise, is a fold_round_grid)
    LGK_LAUNCH(L, "fold_round", launch_kc(k_sum_step, dim3(C, NB), kSumThreads, C, smem, L.stream, a, st, C));
    return cudaGetLastError();
}

// ================================================================ induce
// basis[t] = sum_k apow[k] prod_{bit i of t} S_k[i]   (t < 2^n)
//          = sum_k Hi_k[t >> b] * Lo_k[t & (2^b-1)]
// Lo_k[u] = prod_{i<b, bit i of u} S_k[i];  Hi_k[c] = apow[k] prod_{i<n-b} S_k[b+i]^bit
// (field products are associative/commutative, so this grouping equals the
// reference's doubling order exactly).  The main kernel gives each warp one
// query at a time: the warp builds the table of Hi_k[block] and multiplies
// the whole Lo_k vector by it.
InducePlan induce_plan(uint32_t n) {
    InducePlan p;
    p.b = std::min<uint32_t>(n, 9);
    return p;
}

// Per-query setup of induce_sumcheck_poly_parallel, one warp per query:
//   dot_k = <row_k, gr> (rows gathered on the device; lanes split the row),
//   apow_k = alpha^k (precompute_alpha_powers, src/sumcheck_polys.rs:6-20;
//   lane i holds alpha^(2^i) and the set bits of k are multiplied together),
//   S_k[0] = q_k, S_k[i] = next_s(S_k[i-1], sks[i-1]) (sks_at_x,
//   src/binary_fft.rs:289-292), and contrib_k = apow_k * dot_k, stored at
//   apow[nq + k]; induce_prep folds the contributions into the enforced sum.
struct InduceSetupArgs {
    uint32_t gr[256];
    uint32_t sks[32];
};
__global__ void __launch_bounds__(128) k_induce_setup(const uint32_t *__restrict__ rows, uint32_t glen,
                                                      const uint64_t *__restrict__ q, uint32_t nq, uint32_t alpha,
                                                      uint32_t n, InduceSetupArgs args, uint32_t *__restrict__ S,
                                                      uint32_t *__restrict__ apow, const uint32_t *d_rs, uint32_t nch,
                                                      const uint32_t *d_alpha, InduceStrides st) {
    pdl_begin();
    {
        const uint32_t b = blockIdx.y;  // lockstep batch: proof b
        rows += b * st.rows;
        q += b * st.q;
        S += b * st.S;
        apow += b * st.apow;
        if (d_rs) d_rs += b * st.rs;
        if (d_alpha) d_alpha += b * st.alpha;
    }
    // gr: the Lagrange basis of the challenges (from the device when given)
    __shared__ uint32_t gr[256];
    for (uint32_t j = threadIdx.x; j < glen; j += blockDim.x) gr[j] = d_rs ? lagrange_at(d_rs, nch, j) : args.gr[j];
    if (d_alpha) alpha = *d_alpha;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (k >= nq) return;
    uint32_t dot = 0;
    for (uint32_t j = lane; j < glen; j += 32) dot ^= gf_mul(rows[(uint64_t)k * glen + j], gr[j]);
    dot = warp_xor(dot);
    // alpha^k for k < 2^16
    uint32_t a2 = alpha;
    for (uint32_t i = 0; i < lane && i < 16; ++i) a2 = gf_mul(a2, a2);
    uint32_t p = (lane < 16 && ((k >> lane) & 1)) ? a2 : 1u;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) p = gf_mul(p, __shfl_xor_sync(0xffffffffu, p, o));
    p = __shfl_sync(0xffffffffu, p, 0);
    if (lane == 0) {
        apow[k] = p;
        apow[nq + k] = gf_mul(dot, p);
        if (n) {
            uint32_t sx = (uint32_t)q[k];
            S[(uint64_t)k * n] = sx;
            for (uint32_t i = 1; i < n; ++i) {
                sx = gf_mul(sx, sx) ^ gf_mul(args.sks[i - 1], sx);
                S[(uint64_t)k * n + i] = sx;
            }
        }
    }
}

cudaError_t induce_setup(Launcher &L, const uint32_t *d_rows, uint32_t glen, const uint32_t *gr,
                         const uint64_t *d_q, uint32_t nq, uint32_t alpha, uint32_t n, const uint32_t *sks,
                         uint32_t *d_S, uint32_t *d_apow, const uint32_t *d_rs, const uint32_t *d_alpha, uint32_t B,
                         const InduceStrides &st) {
    if (glen > 256 || n > 32 || nq == 0 || nq > 65536 || (glen & (glen - 1)) || (!gr && !d_rs) || B == 0 ||
        B > 65535)
        return cudaErrorInvalidValue;
    InduceSetupArgs args{};
    if (!d_rs)
        for (uint32_t j = 0; j < glen; ++j) args.gr[j] = gr[j];
    for (uint32_t i = 0; i + 1 < n && i < 32; ++i) args.sks[i] = sks[i];
    const double products = (double)B * nq * (glen + 2 * n + 20);
    L.note(4.0 * B * nq * (glen + n + 2), products, 0, products);
    LGK_LAUNCH(L, "induce_setup", launch_k(k_induce_setup, dim3((nq + 3) / 4, B), 128, 0, L.stream, d_rows, glen, d_q,
                                           nq, alpha, n, args, d_S, d_apow, d_rs, ilog2u(glen), d_alpha, st));
    return cudaGetLastError();
}

// Lo_k and Hi_k of one query per block, by doubling: entry u with top bit h
// is entry u - 2^h times S_k[h] (Lo; Hi from apow_k and S_k[b + h]), one
// product per entry and a block barrier per bit.  Block 0 also XORs the
// queries' contributions into the enforced sum.
// The doubling runs in shared memory when Lo and Hi fit (in_smem), one
// barrier per level, and the finished vectors are written out coalesced;
// larger ones double in place in global memory.
__global__ void k_induce_prep(const uint32_t *__restrict__ S, const uint32_t *__restrict__ apow, uint32_t n,
                              uint32_t b, uint32_t nq, uint32_t *__restrict__ lo, uint32_t *__restrict__ hi,
                              uint32_t *sum_out, int in_smem, uint32_t *__restrict__ out, InduceStrides st) {
    pdl_begin();
    {
        const uint32_t pb = blockIdx.y;  // lockstep batch: proof pb
        S += pb * st.S;
        apow += pb * st.apow;
        lo += pb * st.lo;
        hi += pb * st.hi;
        sum_out += pb * st.sum;
        out += pb * st.out;
    }
    // induce_main XORs its partial sums into the basis: zero it first
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < (1ull << n);
         i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = 0;
    extern __shared__ uint32_t sbuf[];  // Lo then Hi, when in_smem
    __shared__ uint32_t Ss[32];          // the query's subspace values, read once
    const uint32_t k = blockIdx.x, nlo = 1u << b, nhi = 1u << (n - b);
    const uint32_t *Sk = S + (uint64_t)k * n;
    uint32_t *glk = lo + ((uint64_t)k << b), *ghk = hi + ((uint64_t)k << (n - b));
    uint32_t *lk = in_smem ? sbuf : glk, *hk = in_smem ? sbuf + nlo : ghk;
    if (threadIdx.x < n && threadIdx.x < 32) Ss[threadIdx.x] = Sk[threadIdx.x];
    if (threadIdx.x == 0) {
        lk[0] = 1;
        hk[0] = apow[k];
    }
    __syncthreads();
    for (uint32_t h = 0; h < b; ++h) {
        const uint32_t s = Ss[h];
        for (uint32_t u = threadIdx.x; u < (1u << h); u += blockDim.x) lk[(1u << h) + u] = gf_mul(lk[u], s);
        __syncthreads();
    }
    for (uint32_t h = 0; h < n - b; ++h) {
        const uint32_t s = Ss[b + h];
        for (uint32_t c = threadIdx.x; c < (1u << h); c += blockDim.x) hk[(1u << h) + c] = gf_mul(hk[c], s);
        __syncthreads();
    }
    if (in_smem) {
        for (uint32_t u = threadIdx.x; u < nlo; u += blockDim.x) glk[u] = lk[u];
        for (uint32_t c = threadIdx.x; c < nhi; c += blockDim.x) ghk[c] = hk[c];
    }
    if (k == 0 && threadIdx.x < 32) {
        uint32_t x = 0;
        for (uint32_t j = threadIdx.x; j < nq; j += 32) x ^= apow[nq + j];
        x = warp_xor(x);
        if (threadIdx.x == 0) *sum_out = x;
    }
}

// basis[(t_hi << b) | t_lo] = sum_k Hi_k[t_hi] * Lo_k[t_lo].  Work items are
// the (proof, t_hi, query) triples in that order; block i takes the
// contiguous range [i P / G, (i+1) P / G) of the P triples, so one wave of
// blocks gets equal shares (no partial last wave).  A range splits into
// segments of one (proof, t_hi): each warp takes every 8th query of the
// segment, builds the table of Hi_k[t_hi] and multiplies it into its
// lane's share of Lo_k; at the segment's end the warps' sums meet in
// shared memory and go to out (zeroed by induce_prep) by store when the
// segment covers all queries, else by XOR.
template <int ACC>  // ACC = max(1, 2^b / 32) words per lane (b <= 9)
__global__ void __launch_bounds__(256, 3) k_induce_main(const uint32_t *__restrict__ lo, const uint32_t *__restrict__ hi,
                                                     uint32_t n, uint32_t b, uint32_t nq, uint32_t B,
                                                     uint32_t *__restrict__ out, InduceStrides st) {
    pdl_begin();
    __shared__ __align__(128) uint32_t tabs[8][kTabWords];
    __shared__ uint32_t red[512];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t nlo = 1u << b, nhi = 1u << (n - b);
    const uint64_t P = (uint64_t)B * nhi * nq;
    uint64_t p = blockIdx.x * P / gridDim.x;
    const uint64_t pend = (blockIdx.x + 1) * P / gridDim.x;
    while (p < pend) {
        const uint64_t seg = p / nq;
        const uint32_t k0 = (uint32_t)(p - seg * nq);
        const uint64_t left = pend - p;
        const uint32_t k1 = left < (uint64_t)(nq - k0) ? k0 + (uint32_t)left : nq;
        const uint32_t pb = (uint32_t)(seg / nhi), tb = (uint32_t)(seg - (uint64_t)pb * nhi);
        const uint32_t *lop = lo + pb * st.lo, *hip = hi + pb * st.hi;
        uint32_t acc[ACC], va[ACC], vb[ACC];
#pragma unroll
        for (int c = 0; c < ACC; ++c) acc[c] = va[c] = vb[c] = 0;
        // (ACC > 1 means nlo = 32 ACC: every lane word is in range)
        auto in_range = [&](int c) { return ACC > 1 || lane + 32u * c < nlo; };
        // the next query's Hi value and Lo vector are loaded while the
        // current one is multiplied (the loads come from L2); the two
        // register sets swap roles by unrolling the query loop twice
        auto load = [&](uint32_t k, uint32_t (&v)[ACC]) {
            const uint32_t *lk = lop + (uint64_t)k * nlo + lane;
#pragma unroll
            for (int c = 0; c < ACC; ++c)
                if (in_range(c)) v[c] = __ldg(lk + 32 * c);
            return __ldg(hip + (uint64_t)k * nhi + tb);
        };
        auto step = [&](uint32_t k, uint32_t h, const uint32_t (&v)[ACC], uint32_t (&nv)[ACC], uint32_t &hn) {
            if (k + nw < k1) hn = load(k + nw, nv);
            tab_build_warp(tabs[warp], h, lane);
            __syncwarp();
#pragma unroll
            for (int c = 0; c < ACC; ++c)
                if (in_range(c)) acc[c] ^= tab_mul_sa(reinterpret_cast<const uint8_t *>(tabs), 512u * warp, 0, v[c]);
            __syncwarp();
        };
        uint32_t k = k0 + warp, ha = 0, hb = 0;
        if (k < k1) ha = load(k, va);
        for (; k < k1; k += 2 * nw) {
            step(k, ha, va, vb, hb);
            if (k + nw >= k1) break;
            step(k + nw, hb, vb, va, ha);
        }
        for (uint32_t w = threadIdx.x; w < nlo; w += blockDim.x) red[w] = 0;
        __syncthreads();
#pragma unroll
        for (int c = 0; c < ACC; ++c)
            if (in_range(c)) atomicXor(&red[lane + 32 * c], acc[c]);
        __syncthreads();
        uint32_t *dst = out + pb * st.out + (uint64_t)tb * nlo;
        const bool whole = k0 == 0 && k1 == nq;
        for (uint32_t w = threadIdx.x; w < nlo; w += blockDim.x) {
            if (whole) dst[w] = red[w];
            else atomicXor(dst + w, red[w]);
        }
        __syncthreads();  // red is reused by the next segment
        p += k1 - k0;
    }
}

// The same basis when 2^(n-b) >= 2 (n > 9, so 2^b = 512 and ACC = 16):
// work items are (proof, pair of t_hi, query) triples, and each warp builds
// the interleaved table of (Hi_k[2 t], Hi_k[2 t + 1]) and multiplies each
// Lo_k word by both with one lookup per window (tab2_mul_sa), so the two
// output rows 2t and 2t + 1 share every nibble spread, permute and load
// instruction.
__global__ void __launch_bounds__(256, 2) k_induce_main2(const uint32_t *__restrict__ lo, const uint32_t *__restrict__ hi,
                                                      uint32_t n, uint32_t nq, uint32_t B, uint32_t *__restrict__ out,
                                                      InduceStrides st) {
    pdl_begin();
    constexpr int ACC = 16;
    constexpr uint32_t nlo = 32 * ACC;  // b = 9
    __shared__ __align__(256) uint2 tabs[8][kTabWords];
    __shared__ uint32_t red[2 * nlo];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t nhi = 1u << (n - 9), npair = nhi / 2;
    const uint64_t P = (uint64_t)B * npair * nq;
    uint64_t p = blockIdx.x * P / gridDim.x;
    const uint64_t pend = (blockIdx.x + 1) * P / gridDim.x;
    const uint8_t *tab8 = reinterpret_cast<const uint8_t *>(tabs);
    while (p < pend) {
        const uint64_t seg = p / nq;
        const uint32_t k0 = (uint32_t)(p - seg * nq);
        const uint64_t left = pend - p;
        const uint32_t k1 = left < (uint64_t)(nq - k0) ? k0 + (uint32_t)left : nq;
        const uint32_t pb = (uint32_t)(seg / npair), tp = (uint32_t)(seg - (uint64_t)pb * npair);
        const uint32_t *lop = lo + pb * st.lo, *hip = hi + pb * st.hi;
        uint32_t acc0[ACC], acc1[ACC];
#pragma unroll
        for (int c = 0; c < ACC; ++c) acc0[c] = acc1[c] = 0;
        // the next query's Hi pair and Lo words are loaded (from L2) while the
        // current one's are multiplied: each Lo word right after the product
        // that frees its register
        uint32_t v[ACC];
        uint2 h = make_uint2(0, 0);
        if (k0 + warp < k1) {
            const uint32_t *lk = lop + (uint64_t)(k0 + warp) * nlo + lane;
#pragma unroll
            for (int c = 0; c < ACC; ++c) v[c] = __ldg(lk + 32 * c);
            h = __ldg(reinterpret_cast<const uint2 *>(hip + (uint64_t)(k0 + warp) * nhi) + tp);
        }
        for (uint32_t k = k0 + warp; k < k1; k += nw) {
            tab2_build_warp(tabs[warp], h.x, h.y, lane);
            __syncwarp();
            const uint32_t kn = k + nw < k1 ? k + nw : k;
            const uint32_t *lk = lop + (uint64_t)kn * nlo + lane;
            h = __ldg(reinterpret_cast<const uint2 *>(hip + (uint64_t)kn * nhi) + tp);
#pragma unroll
            for (int c = 0; c < ACC; ++c) {
                const uint2 r = tab2_mul_sa(tab8, 1024u * warp, v[c]);
                v[c] = __ldg(lk + 32 * c);
                acc0[c] ^= r.x;
                acc1[c] ^= r.y;
            }
            __syncwarp();
        }
        for (uint32_t w = threadIdx.x; w < 2 * nlo; w += blockDim.x) red[w] = 0;
        __syncthreads();
#pragma unroll
        for (int c = 0; c < ACC; ++c) {
            atomicXor(&red[lane + 32 * c], acc0[c]);
            atomicXor(&red[nlo + lane + 32 * c], acc1[c]);
        }
        __syncthreads();
        uint32_t *dst = out + pb * st.out + (uint64_t)(2 * tp) * nlo;  // rows 2tp and 2tp + 1
        const bool whole = k0 == 0 && k1 == nq;
        for (uint32_t w = threadIdx.x; w < 2 * nlo; w += blockDim.x) {
            if (whole) dst[w] = red[w];
            else atomicXor(dst + w, red[w]);
        }
        __syncthreads();  // red is reused by the next segment
        p += k1 - k0;
    }
}

// One wave of induce_main blocks (occupancy of the instantiation, cached).
template <int ACC>
static unsigned induce_grid(uint64_t work) {
    static std::atomic<int> occ_c{0}, sms_c{0};
    int sms = sms_c.load(std::memory_order_relaxed), o = occ_c.load(std::memory_order_relaxed);
    if (!sms) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            sms = 148;
        sms_c.store(sms, std::memory_order_relaxed);
    }
    if (!o) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_induce_main<ACC>, 256, 0) != cudaSuccess || o < 1) o = 1;
        occ_c.store(o, std::memory_order_relaxed);
    }
    // at least 32 (proof, t_hi, query) triples a block, so its 8 warps all work
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((work + 31) / 32, (uint64_t)sms * o));
}

static cudaError_t launch_induce_main(Launcher &L, const InducePlan &p, uint32_t n, uint32_t nq, const uint32_t *d_lo,
                                      const uint32_t *d_hi, uint32_t *out, uint32_t B, const InduceStrides &st);
cudaError_t induce_basis(Launcher &L, const InducePlan &p, const uint32_t *d_S, const uint32_t *d_apow,
                         uint32_t n, uint32_t nq, uint32_t *d_lo, uint32_t *d_hi, uint32_t *out, uint32_t *d_sum,
                         uint32_t B, const InduceStrides &st) {
    if (B == 0 || B > 65535) return cudaErrorInvalidValue;
    const double vec = (double)nq * ((1ull << p.b) + (1ull << (n - p.b)));  // Lo and Hi words
    L.note(4.0 * B * vec, B * vec, 0, B * vec);
    const size_t words = (1ull << p.b) + (1ull << (n - p.b));
    const int in_smem = words <= 12288;  // 48 KB: no opt-in needed
    LGK_LAUNCH(L, "induce_prep", launch_k(k_induce_prep, dim3(nq, B), 256, in_smem ? 4 * words : 0, L.stream, d_S,
                                          d_apow, n, p.b, nq, d_lo, d_hi, d_sum, in_smem, out, st));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_induce_main(L, p, n, nq, d_lo, d_hi, out, B, st);
}

// induce_main (pair tables when 2^(n-b) >= 2) over Lo / Hi from the prep
static cudaError_t launch_induce_main(Launcher &L, const InducePlan &p, uint32_t n, uint32_t nq, const uint32_t *d_lo,
                                      const uint32_t *d_hi, uint32_t *out, uint32_t B, const InduceStrides &st) {
    const double vec = (double)nq * ((1ull << p.b) + (1ull << (n - p.b)));
    const uint64_t work = (uint64_t)B * (1ull << (n - p.b)) * nq;
    L.note(4.0 * B * (vec + (1ull << n)), (double)B * nq * (1ull << n));
    if (p.b == 9 && n > 9) {
        static std::atomic<int> occ2{0};
        int o = occ2.load(std::memory_order_relaxed);
        if (!o) {
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_induce_main2, 256, 0) != cudaSuccess || o < 1) o = 1;
            occ2.store(o, std::memory_order_relaxed);
        }
        int dev = 0, sms = 148;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            sms = 148;
        // at least 8 (proof, t_hi pair, query) triples a block: one a warp
        const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((work / 2 + 7) / 8, (uint64_t)sms * o));
        LGK_LAUNCH(L, "induce_main", launch_k(k_induce_main2, grid, 256, 0, L.stream, d_lo, d_hi, n, nq, B, out, st));
        return cudaGetLastError();
    }
    switch (std::max<uint32_t>(1, (1u << p.b) / 32)) {
#define LGK_CASE(a) \
    case a: LGK_LAUNCH(L, "induce_main", launch_k(k_induce_main<a>, induce_grid<a>(work), 256, 0, L.stream, d_lo, d_hi, n, p.b, nq, B, out, st)); break;
        LGK_CASE(1) LGK_CASE(2) LGK_CASE(4) LGK_CASE(8) LGK_CASE(16)
#undef LGK_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// induce_setup and induce_prep in one launch: block k (query k) first
// runs the setup of its query (the row's dot product with the Lagrange
// basis, alpha^k, the subspace values) into shared memory, then the block
// doubles out Lo_k and Hi_k from them.  Bound by the latency of those serial
// products, so independent ones run side by side.  Each block leaves its
// contribution alpha^k * dot_k in contrib[k]; the last block to finish (a
// ticket, reset by it) XORs them into the enforced sum.
__global__ void __launch_bounds__(256) k_induce_sp(const uint32_t *__restrict__ rows, uint32_t glen,
                                                   const uint64_t *__restrict__ q, uint32_t nq, uint32_t alpha,
                                                   uint32_t n, uint32_t b, InduceSetupArgs args,
                                                   const uint32_t *d_rs, uint32_t nch, const uint32_t *d_alpha,
                                                   uint32_t *__restrict__ contrib, uint32_t *__restrict__ lo,
                                                   uint32_t *__restrict__ hi, uint32_t *sum_out, int in_smem,
                                                   uint32_t *__restrict__ out, uint32_t *ticket, InduceStrides st) {
    pdl_begin();
    {
        const uint32_t pb = blockIdx.y;  // lockstep batch: proof pb
        rows += pb * st.rows;
        q += pb * st.q;
        contrib += pb * st.apow;
        lo += pb * st.lo;
        hi += pb * st.hi;
        sum_out += pb * st.sum;
        out += pb * st.out;
        if (d_rs) d_rs += pb * st.rs;
        if (d_alpha) d_alpha += pb * st.alpha;
        ticket += pb;
    }
    // induce_main XORs its partial sums into the basis: zero it first
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < (1ull << n);
         i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = 0;
    extern __shared__ uint32_t sbuf[];  // Lo then Hi, when in_smem
    __shared__ uint32_t Ss[32], apk;
    __shared__ bool last;
    // The setup of query k (as k_induce_setup), its three parts on warps of
    // their own: the subspace values on warp 0, alpha^k on warp 1, the row's
    // dot product with the Lagrange basis on the rest.
    const uint32_t k = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ uint32_t dots[8];
    if (warp == 0) {
        if (lane == 0) {
            uint32_t sx = (uint32_t)q[k];
            Ss[0] = sx;
            for (uint32_t i = 1; i < n; ++i) {
                sx = gf_mul(sx, sx) ^ gf_mul(args.sks[i - 1], sx);
                Ss[i] = sx;
            }
        }
    } else if (warp == 1) {
        uint32_t a2 = d_alpha ? *d_alpha : alpha;
        for (uint32_t i = 0; i < lane && i < 16 && (k >> i) != 0; ++i) a2 = gf_mul(a2, a2);
        uint32_t pw = (lane < 16 && ((k >> lane) & 1)) ? a2 : 1u;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) pw = gf_mul(pw, __shfl_xor_sync(0xffffffffu, pw, o));
        if (lane == 0) apk = pw;
    } else {
        uint32_t dot = 0;
        for (uint32_t j = threadIdx.x - 64; j < glen; j += blockDim.x - 64)
            dot ^= gf_mul(rows[(uint64_t)k * glen + j], d_rs ? lagrange_at(d_rs, nch, j) : args.gr[j]);
        dot = __reduce_xor_sync(0xffffffffu, dot);
        if (lane == 0) dots[warp] = dot;
    }
    __syncthreads();
    // the prep of query k (as k_induce_prep), a level of Lo and one of Hi at a
    // time
    const uint32_t nlo = 1u << b, nhi = 1u << (n - b);
    uint32_t *glk = lo + ((uint64_t)k << b), *ghk = hi + ((uint64_t)k << (n - b));
    uint32_t *lk = in_smem ? sbuf : glk, *hk = in_smem ? sbuf + nlo : ghk;
    if (threadIdx.x == 0) {
        lk[0] = 1;
        hk[0] = apk;
        uint32_t dot = 0;
        for (uint32_t w = 2; w < blockDim.x >> 5; ++w) dot ^= dots[w];
        contrib[k] = gf_mul(dot, apk);
    }
    __syncthreads();
    for (uint32_t h = 0; h < max(b, n - b); ++h) {
        const uint32_t m = 1u << h, cl = h < b ? m : 0, ch = h < n - b ? m : 0;
        for (uint32_t u = threadIdx.x; u < cl + ch; u += blockDim.x) {
            if (u < cl) lk[m + u] = gf_mul(lk[u], Ss[h]);
            else hk[m + u - cl] = gf_mul(hk[u - cl], Ss[b + h]);
        }
        __syncthreads();
    }
    if (in_smem) {
        for (uint32_t u = threadIdx.x; u < nlo; u += blockDim.x) glk[u] = lk[u];
        for (uint32_t c = threadIdx.x; c < nhi; c += blockDim.x) ghk[c] = hk[c];
    }
    // the enforced sum, by the last block to finish
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last || threadIdx.x >= 32) return;
    __threadfence();
    uint32_t x = 0;
    for (uint32_t j = lane; j < nq; j += 32) x ^= __ldcg(contrib + j);
    x = warp_xor(x);
    if (lane == 0) {
        *sum_out = x;
        *ticket = 0;
    }
}

cudaError_t induce_fused(Launcher &L, const InducePlan &p, const uint32_t *d_rows, uint32_t glen, const uint32_t *gr,
                         const uint64_t *d_q, uint32_t nq, uint32_t alpha, uint32_t n, const uint32_t *sks,
                         uint32_t *d_S, uint32_t *d_apow, const uint32_t *d_rs, const uint32_t *d_alpha,
                         uint32_t *d_lo, uint32_t *d_hi, uint32_t *out, uint32_t *d_sum, uint32_t B,
                         const InduceStrides &st) {
    if (!L.tickets || B > kMaxTickets || n > 32 || n == 0) {
        cudaError_t e = induce_setup(L, d_rows, glen, gr, d_q, nq, alpha, n, sks, d_S, d_apow, d_rs, d_alpha, B, st);
        if (e != cudaSuccess) return e;
        return induce_basis(L, p, d_S, d_apow, n, nq, d_lo, d_hi, out, d_sum, B, st);
    }
    if (glen > 256 || nq == 0 || nq > 65536 || (glen & (glen - 1)) || (!gr && !d_rs) || B == 0 || B > 65535)
        return cudaErrorInvalidValue;
    InduceSetupArgs args{};
    if (!d_rs)
        for (uint32_t j = 0; j < glen; ++j) args.gr[j] = gr[j];
    for (uint32_t i = 0; i + 1 < n && i < 32; ++i) args.sks[i] = sks[i];
    const double vec = (double)nq * ((1ull << p.b) + (1ull << (n - p.b)));
    const double products = B * (vec + nq * (glen + 2.0 * n + 20));
    L.note(4.0 * B * (vec + nq * (glen + 2)), products, 0, products);
    const size_t words = (1ull << p.b) + (1ull << (n - p.b));
    const int in_smem = words <= 10240;  // with the static arrays, under the 48 KB that needs no opt-in
    // one block a query: more than the device holds at 256 threads go out with
    // 128, twice as many at a time (23 x 148 queries of 2^12: 55 -> 48 us)
    const unsigned threads = (uint64_t)nq * B > 148 * 8 ? 128 : 256;
    LGK_LAUNCH(L, "induce_sp", launch_k(k_induce_sp, dim3(nq, B), threads, in_smem ? 4 * words : 0, L.stream, d_rows, glen,
                                        d_q, nq, alpha, n, p.b, args, d_rs, ilog2u(glen), d_alpha, d_apow, d_lo, d_hi,
                                        d_sum, in_smem, out, L.tickets, st));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_induce_main(L, p, n, nq, d_lo, d_hi, out, B, st);
}

// ====================================================== opening check
// merkle_tree::verify (src/merkle_tree.rs:120-188) of well-formed openings,
// one block each: nq <= 256 sorted distinct queries below 2^depth, their rows
// of ncols words (1..256) hashed as the leaves, and at least as many 32-byte
// proof nodes as the opening consumes.
// Thread i climbs from query i and keeps the hash of the node it stands on in
// registers.  It and query i-1 meet where their indices' highest differing
// bit is: there it leaves its hash to the first query under its left sibling
// and stops.  Everything else about the climb follows from the queries too
// (which layers have a partner, the place of each proof node: layers in
// order, nodes in query order), so it is worked out before it, and a layer is
// one barrier and one compression.  Bound by that chain's latency: the three
// openings of a 2^24 proof (2^20, 2^16 and 2^12 leaves) take 42 us in one
// launch (event-timed); a launch each, with the layers compacted in shared
// memory, took 57 us apiece.
__global__ void __launch_bounds__(256) k_opening_check(OpeningChecks list) {
    pdl_begin();
    const OpeningCheck o = list.c[blockIdx.x];
    __shared__ uint32_t qs[256], pmask[256];
    __shared__ uint32_t slot[2][8][256];
    __shared__ uint32_t wmask[32][8], wbase[32][8];
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const bool have = t < o.nq;
    qs[t] = have ? (uint32_t)o.q[t] : 0u;
    pmask[t] = 0;
    __syncthreads();
    // hp: the layer in which this thread's node meets its left sibling (thread
    // 0 climbs to the root); owner: the first query under that sibling
    uint32_t hp = have ? o.depth : 0, owner = 0;
    const uint32_t qt = qs[t];
    if (have && t > 0) {
        hp = 31 - __clz(qt ^ qs[t - 1]);
        const uint32_t lo = ((qt >> hp) - 1) << hp;
        uint32_t l = 0, r = t - 1;
        while (l < r) {
            const uint32_t m = (l + r) / 2;
            if (qs[m] < lo) l = m + 1;
            else r = m;
        }
        owner = l;
        atomicOr(&pmask[owner], 1u << hp);
    }
    __syncthreads();
    const uint32_t partner = pmask[t], act = have ? (hp >= 32 ? ~0u : (1u << hp) - 1) : 0u, uses = act & ~partner;
    for (uint32_t d = 0; d < o.depth; ++d) {
        const uint32_t m = __ballot_sync(0xffffffffu, (uses >> d) & 1);
        if (lane == 0) wmask[d][warp] = m;
    }
    // the leaf
    uint32_t cv[8];
    b3_iv(cv);
    if (have) {
        const uint32_t nb = (o.ncols + 15) / 16;
        const uint32_t *row = o.rows + (uint64_t)t * o.ncols;
        for (uint32_t b = 0; b < nb; ++b) {
            uint32_t m[16];
#pragma unroll
            for (uint32_t w = 0; w < 16; ++w) m[w] = 16 * b + w < o.ncols ? row[16 * b + w] : 0u;
            const bool last = b + 1 == nb;
            const uint32_t blen = last ? 4 * o.ncols - 64 * (nb - 1) : 64;
            const uint32_t flags = (b == 0 ? B3_CHUNK_START : 0u) | (last ? (B3_CHUNK_END | B3_ROOT) : 0u);
            b3_compress<false>(cv, m, blen, flags);
        }
    }
    __syncthreads();
    if (warp == 0) {  // lane l: layer l's proof nodes before each warp's
        uint32_t tot = 0;
        if (lane < o.depth)
            for (uint32_t w = 0; w < 8; ++w) {
                wbase[lane][w] = tot;
                tot += __popc(wmask[lane][w]);
            }
        uint32_t inc = tot;
        for (uint32_t s = 1; s < 32; s <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, s);
            if (lane >= s) inc += y;
        }
        if (lane < o.depth)
            for (uint32_t w = 0; w < 8; ++w) wbase[lane][w] += inc - tot;
    }
    __syncthreads();
    uint32_t nxt[8];
    auto fetch = [&](uint32_t d) {  // this thread's proof node of layer d
        if (d >= o.depth || !((uses >> d) & 1)) return;
        const uint32_t pos = wbase[d][warp] + __popc(wmask[d][warp] & ((1u << lane) - 1));
        load_node(o.proof + 8ull * pos, nxt);
    };
    fetch(0);
    for (uint32_t d = 0; d < o.depth; ++d) {
        if (have && t > 0 && hp == d) {
#pragma unroll
            for (int w = 0; w < 8; ++w) slot[d & 1][w][owner] = cv[w];
        }
        __syncthreads();
        if ((act >> d) & 1) {
            // even nodes have the other one on the right
            uint32_t m[16];
            const bool right = (qt >> d) & 1;
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                const uint32_t x = (partner >> d) & 1 ? slot[d & 1][w][t] : nxt[w];
                m[w] = right ? x : cv[w];
                m[8 + w] = right ? cv[w] : x;
            }
            fetch(d + 1);
            b3_iv(cv);
            b3_compress<false>(cv, m, 64, B3_CHUNK_START | B3_CHUNK_END | B3_ROOT);
        }
    }
    if (t == 0) store_node(o.out, cv);
}
cudaError_t opening_check(Launcher &L, const OpeningChecks &list, uint32_t count) {
    if (count == 0) return cudaSuccess;
    if (count > kMaxOpenings) return cudaErrorInvalidValue;
    for (uint32_t i = 0; i < count; ++i) {
        const OpeningCheck &o = list.c[i];
        if (o.nq == 0 || o.nq > 256 || o.ncols == 0 || o.ncols > 256 || o.depth > 31) return cudaErrorInvalidValue;
    }
    LGK_LAUNCH(L, "opening_check", launch_k(k_opening_check, count, 256, 0, L.stream, list));
    return cudaGetLastError();
}

// ======================================================= ligero_verify
// One block per opened row k: dot = <row_k, gr> over the first min(row
// length, glen) entries (zip truncation), e = sum_j yr[j] * basis_k[j]
// with basis_k[j] the product of sx[t] over the set bits t of j, sx[0] =
// q_k and sx[t] = sx[t-1]^2 + sks[t-1] sx[t-1]; a mismatch sets *bad.
// The product form gives the same field elements as the reference's
// doubling (src/ligero.rs:97-131, evaluate_scaled_basis_inplace).
__global__ void __launch_bounds__(256) k_ligero_check(const uint32_t *__restrict__ rows,
                                                      const uint64_t *__restrict__ row_off, uint32_t nrows,
                                                      const uint32_t *__restrict__ gr, uint32_t glen,
                                                      const uint32_t *__restrict__ yr, uint32_t nv,
                                                      const uint64_t *__restrict__ q, ligero_sks sks,
                                                      uint32_t *bad) {
    pdl_begin();
    __shared__ uint32_t sx[32];
    __shared__ uint32_t part[2][8];
    const uint32_t k = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (k >= nrows) return;
    if (threadIdx.x == 0) {
        uint32_t s = (uint32_t)q[k];
        sx[0] = s;
        for (uint32_t t = 1; t < nv; ++t) {
            s = gf_mul(s, s) ^ gf_mul(sks.v[t - 1], s);
            sx[t] = s;
        }
    }
    __syncthreads();
    const uint64_t r0 = row_off[k], rlen = row_off[k + 1] - r0, zl = rlen < glen ? rlen : (uint64_t)glen;
    uint32_t dot = 0, e = 0;
    for (uint64_t j = threadIdx.x; j < zl; j += blockDim.x) dot ^= gf_mul(rows[r0 + j], gr[j]);
    const uint32_t ylen = 1u << nv;
    for (uint32_t j = threadIdx.x; j < ylen; j += blockDim.x) {
        uint32_t b = 1;
        for (uint32_t t = 0; t < nv; ++t)
            if ((j >> t) & 1) b = gf_mul(b, sx[t]);
        e ^= gf_mul(yr[j], b);
    }
    dot = warp_xor(dot);
    e = warp_xor(e);
    if (lane == 0) { part[0][warp] = dot; part[1][warp] = e; }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t d = 0, s = 0;
        for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) { d ^= part[0][w]; s ^= part[1][w]; }
        if (d != s) *bad = 1u;
    }
}
cudaError_t ligero_check(Launcher &L, const uint32_t *rows, const uint64_t *row_off, uint32_t nrows,
                         const uint32_t *gr, uint32_t glen, const uint32_t *yr, uint32_t nv, const uint64_t *q,
                         const uint32_t *sks, uint32_t *bad) {
    if (nrows == 0) return cudaSuccess;
    if (nv > 31) return cudaErrorInvalidValue;
    ligero_sks s{};
    for (uint32_t t = 0; t + 1 < nv; ++t) s.v[t] = sks[t];
    LGK_LAUNCH(L, "ligero_check", launch_k(k_ligero_check, nrows, 256, 0, L.stream, rows, row_off, nrows, gr, glen,
                                           yr, nv, q, s, bad));
    return cudaGetLastError();
}

// ============================================================ GF(2^128)
// out[i] = a[i] * b[i] in BinaryElem128, elements as two u64 limbs (low
// first), 16-byte loads and stores.
__global__ void k_gf128_mul(const ulonglong2 *__restrict__ a, const ulonglong2 *__restrict__ b,
                            ulonglong2 *__restrict__ out, uint64_t n) {
    pdl_begin();
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const ulonglong2 x = a[i], y = b[i];
        const U128 r = lgd::gf128_mul({x.x, x.y}, {y.x, y.y});
        out[i] = make_ulonglong2(r.lo, r.hi);
    }
}
cudaError_t gf128_mul(Launcher &L, const uint64_t *a, const uint64_t *b, uint64_t *out, uint64_t n) {
    if (n == 0) return cudaSuccess;
    if ((uintptr_t)a % 16 || (uintptr_t)b % 16 || (uintptr_t)out % 16) return cudaErrorInvalidValue;
    const unsigned blocks = (unsigned)std::min<uint64_t>((n + 255) / 256, 148ull * 8);
    L.note(48.0 * n, 0);
    LGK_LAUNCH(L, "gf128_mul", launch_k(k_gf128_mul, blocks, 256, 0, L.stream, reinterpret_cast<const ulonglong2 *>(a),
                                        reinterpret_cast<const ulonglong2 *>(b), reinterpret_cast<ulonglong2 *>(out), n));
    return cudaGetLastError();
}

// ============================================================== splitmix
__global__ void k_splitmix(uint64_t seed, uint32_t *out, uint64_t n) {
    pdl_begin();
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t z = seed + (i + 1) * 0x9E3779B97F4A7C15ull;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        out[i] = (uint32_t)(z ^ (z >> 31));
    }
}
cudaError_t splitmix(Launcher &L, uint64_t seed, uint32_t *out, uint64_t n) {
    const unsigned blocks = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, 148ull * 16));
    L.note(4.0 * n, 0);
    LGK_LAUNCH(L, "splitmix", launch_k(k_splitmix, blocks, 256, 0, L.stream, seed, out, n));
    return cudaGetLastError();
}

// ============================================================= autotuner
bool TuneKey::operator<(const TuneKey &o) const {
    auto t = [](const TuneKey &k) { return std::make_tuple(k.device, k.kind, k.log_len, k.nvec, k.Q, k.src, k.inverse); };
    return t(*this) < t(o);
}

namespace {
std::mutex g_tune_mu;
std::map<TuneKey, FftPlan> g_fft_plans;
std::map<TuneKey, int> g_fold_bps;

// Candidate splits: the last pass 4-6 stages, the strided passes before it
// 3-6 each (at most kMaxFftPasses passes), the default first.
std::vector<FftPlan> fft_candidates(uint32_t log_len, uint64_t words, uint32_t nvec, bool rs) {
    std::vector<FftPlan> out{default_fft_plan(log_len, words, nvec, rs, true)};
    if (log_len <= 6) return out;
    auto add = [&](const FftPlan &p) {
        for (auto &q : out)
            if (plan_code(q) == plan_code(p)) return;
        out.push_back(p);
    };
    for (uint32_t kt = 6; kt >= 4; --kt) {
        const uint32_t rem = log_len - kt;
        for (uint32_t nps = 1; nps < kMaxFftPasses && nps <= rem; ++nps) {
            if (rem > 6 * nps || rem < 3 * nps) continue;
            // even split (larger first) and with the larger passes last
            FftPlan a, b;
            a.np = b.np = nps + 1;
            for (uint32_t i = 0; i < nps; ++i) {
                a.ks[i] = rem / nps + (i < rem % nps ? 1 : 0);
                b.ks[nps - 1 - i] = a.ks[i];
            }
            a.ks[nps] = b.ks[nps] = kt;
            add(a);
            add(b);
        }
    }
    if (out.size() > 10) out.resize(10);
    return out;
}
}  // namespace

bool tuned_fft_plan(const TuneKey &k, FftPlan *out) {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_fft_plans.find(k);
    if (it == g_fft_plans.end()) return false;
    *out = it->second;
    return true;
}

// Times every candidate split of this transform shape on scratch buffers
// of the same extent (the values do not change the work), keeps the
// fastest for the process and returns it.  Buffers that cannot be
// allocated leave the default split, untuned.
cudaError_t tune_fft(Launcher &L, const TuneKey &k, uint32_t *data, const uint32_t *tw, uint64_t col_stride,
                     uint64_t q_stride, uint32_t root_base, const FftSrc *src, FftPlan *out) {
    (void)data;
    const uint64_t n = 1ull << k.log_len, words = (uint64_t)k.Q * k.nvec * n;
    const uint64_t extent = (uint64_t)(k.nvec - 1) * col_stride + (uint64_t)(k.Q - 1) * q_stride + n;
    const uint64_t src_extent = src ? (uint64_t)(k.nvec - 1) * src->col_stride + n : 0;
    uint32_t *sd = nullptr, *ss = nullptr;
    if (cudaMallocAsync(&sd, 4 * extent, L.stream) != cudaSuccess ||
        (src && cudaMallocAsync(&ss, 4 * src_extent, L.stream) != cudaSuccess)) {
        cudaGetLastError();
        if (sd) cudaFreeAsync(sd, L.stream);
        *out = default_fft_plan(k.log_len, words, k.nvec, src != nullptr, true);
        return cudaSuccess;
    }
    FftSrc s2;
    if (src) { s2 = *src; s2.p = ss; }
    // every timed run starts with L2 holding none of the data, as in a proof
    // (its inputs were written long before): a write over more than L2
    uint8_t *flush = nullptr;
    const size_t kFlush = 192u << 20;
    if (cudaMallocAsync(&flush, kFlush, L.stream) != cudaSuccess) { cudaGetLastError(); flush = nullptr; }
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    const bool timing = L.timing;
    L.timing = false;
    FftPlan best = default_fft_plan(k.log_len, words, k.nvec, src != nullptr, true);
    float best_ms = 1e30f;
    cudaError_t err = cudaSuccess;
    for (const FftPlan &c : fft_candidates(k.log_len, words, k.nvec, src != nullptr)) {
        if (src && c.ks[0] > kMaxRsFirst) continue;
        L.forced_plan = &c;
        float ms = 1e30f;
        for (int rep = 0; rep < 3 && err == cudaSuccess; ++rep) {
            if (flush) cudaMemsetAsync(flush, rep, kFlush, L.stream);
            cudaEventRecord(a, L.stream);
            err = fft_vectors(L, sd, tw, k.log_len, k.nvec, col_stride, k.Q, q_stride, root_base, k.inverse, FFT_ALL,
                              src ? &s2 : nullptr);
            cudaEventRecord(b, L.stream);
            cudaEventSynchronize(b);
            float t = 0.f;
            cudaEventElapsedTime(&t, a, b);
            if (rep > 0) ms = std::min(ms, t);  // the first run builds the split's tables
        }
        L.forced_plan = nullptr;
        if (err != cudaSuccess) break;
        if (ms < best_ms) { best_ms = ms; best = c; }
    }
    L.forced_plan = nullptr;
    L.timing = timing;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFreeAsync(sd, L.stream);
    if (ss) cudaFreeAsync(ss, L.stream);
    if (flush) cudaFreeAsync(flush, L.stream);
    if (err != cudaSuccess) return err;
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_fft_plans[k] = best;
    }
    *out = best;
    return cudaSuccess;
}

static bool tuned_fold(const TuneKey &k, int *bps) {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_fold_bps.find(k);
    if (it == g_fold_bps.end()) return false;
    *bps = it->second;
    return true;
}

// Times the fold grid at 1, 2, 3 and 4 blocks per SM, one or four outputs
// per thread, and split where there are few outputs, on scratch buffers and keeps the fastest (nothing is recorded
// if they cannot be allocated).
static void tune_fold(Launcher &L, const TuneKey &k, bool few) {
    const uint64_t n = 1ull << k.log_len;
    uint32_t *in = nullptr, *out = nullptr, *drs = nullptr;
    if (cudaMallocAsync(&in, 4 * n, L.stream) != cudaSuccess ||
        cudaMallocAsync(&out, 4 * (n >> k.nvec) + 16, L.stream) != cudaSuccess ||
        cudaMallocAsync(&drs, 64, L.stream) != cudaSuccess) {
        cudaGetLastError();
        if (in) cudaFreeAsync(in, L.stream);
        if (out) cudaFreeAsync(out, L.stream);
        return;
    }
    // the challenges' values do not change the work
    cudaMemsetAsync(drs, 0x5A, 64, L.stream);
    uint8_t *flush = nullptr;  // as in tune_fft: runs start with a cold L2
    const size_t kFlush = 192u << 20;
    if (cudaMallocAsync(&flush, kFlush, L.stream) != cudaSuccess) { cudaGetLastError(); flush = nullptr; }
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    const bool timing = L.timing;
    L.timing = false;
    int best = few ? kFoldSplit : 4;
    float best_ms = 1e30f;
    for (int cand = 0; cand < (few ? 9 : 8); ++cand) {
        const int choice = cand == 8 ? kFoldSplit : (1 + (cand & 3)) | (cand >= 4 ? kFoldVec4 : 0);
        L.forced_fold = choice;
        float ms = 1e30f;
        for (int rep = 0; rep < 3; ++rep) {
            if (flush) cudaMemsetAsync(flush, rep, kFlush, L.stream);
            cudaEventRecord(a, L.stream);
            fold_eq(L, in, out, k.log_len, k.nvec, nullptr, drs);
            cudaEventRecord(b, L.stream);
            cudaEventSynchronize(b);
            float t = 0.f;
            cudaEventElapsedTime(&t, a, b);
            if (rep > 0) ms = std::min(ms, t);
        }
        if (ms < best_ms) { best_ms = ms; best = choice; }
    }
    L.forced_fold = 0;
    L.timing = timing;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFreeAsync(in, L.stream);
    cudaFreeAsync(out, L.stream);
    cudaFreeAsync(drs, L.stream);
    if (flush) cudaFreeAsync(flush, L.stream);
    if (cudaGetLastError() != cudaSuccess) return;
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_fold_bps[k] = best;
}

std::string tuned_choices() {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    std::string s;
    char buf[160];
    for (auto &kv : g_fft_plans) {
        std::snprintf(buf, sizeof buf, "fft device %d log_len %u vectors %u subtrees %u src %d inverse %d : passes",
                      kv.first.device, kv.first.log_len, kv.first.nvec, kv.first.Q, (int)kv.first.src,
                      (int)kv.first.inverse);
        s += buf;
        for (uint32_t i = 0; i < kv.second.np; ++i) s += " " + std::to_string(kv.second.ks[i]);
        s += "\n";
    }
    for (auto &kv : g_fold_bps) {
        if (kv.second == kFoldSplit)
            std::snprintf(buf, sizeof buf, "fold device %d log_len %u k %u : split over clusters\n", kv.first.device,
                          kv.first.log_len, kv.first.nvec);
        else
            std::snprintf(buf, sizeof buf, "fold device %d log_len %u k %u : blocks/SM %d outputs/thread %d\n",
                          kv.first.device, kv.first.log_len, kv.first.nvec, kv.second & 0xFF,
                          (kv.second & kFoldVec4) ? 4 : 1);
        s += buf;
    }
    return s;
}

}  // namespace lgk
