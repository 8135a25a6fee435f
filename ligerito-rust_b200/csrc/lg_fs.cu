// Fiat-Shamir transcript on the device: the prover's challenges, queries
// and Merkle opening lists come from here, so a proof runs as one stream
// of kernels without host round trips.
//
// The transcript (src/emulated_fs.rs:6-76) is a running SHA-256 (sha2
// 0.10.9, FIPS 180-4): absorb appends bytes; squeeze appends the LE u32
// counter, increments it and finalises a clone of the state; a field
// element is the low 32 bits of the digest's first 16 bytes read as a LE
// u128, a query the low 64 bits mod n.  get_distinct_queries rejects
// repeats and sorts.  Everything absorbed is whole u32s, so the pending
// message is kept as big-endian words.
//
// Squeeze i of a batch finalises the state after i+1 more counters, so one
// warp compresses the full blocks that the absorbed words and the counters
// complete (the only serial part; their schedules come from other warps), then
// every thread finalises its own clone.
#include <cstdint>

#include "lg_device.cuh"
#include "lg_fs.cuh"

namespace lgk {

namespace {

using namespace fsd;
using lgd::pdl_begin;

__global__ void k_fs_step(FsState *g, FsStep a, FsStrides st) {
    pdl_begin();
    {
        const uint32_t b = blockIdx.x;  // lockstep batch: one block per proof
        g += b;
        a.src += b * st.src;
        if (a.out) a.out += b * st.out;
        if (a.mirror) a.mirror += b * st.mirror;
        if (a.zero) a.zero += b * st.zero;
    }
    __shared__ FsState S;
    __shared__ Batch B;
    __shared__ uint32_t stage[64];
    __shared__ FsWork W;
    static_assert(kKwBlocks <= 32, "the long runs' schedules share the step's rows");
    for (uint32_t i = threadIdx.x; i < a.nzero; i += blockDim.x) a.zero[i] = 0;
    if (a.init) {  // FS::new(seed): the seed's LE bytes absorbed
        for (uint32_t i = threadIdx.x; i < sizeof(FsState) / 4; i += blockDim.x) reinterpret_cast<uint32_t *>(&S)[i] = 0;
        __syncthreads();
        if (threadIdx.x == 0) {
            const uint32_t iv[8] = {0x6a09e667, 0xbb67ae85, 0x3c6ef372, 0xa54ff53a,
                                    0x510e527f, 0x9b05688c, 0x1f83d9ab, 0x5be0cd19};
            for (int k = 0; k < 8; ++k) S.h[k] = iv[k];
            fs_absorb(S, &a.seed, 1);
        }
        __syncthreads();
    } else {
        load_state(S, g);
    }
    const bool bad = threadIdx.x == 0 && a.check && (a.src[0] ^ a.src[1]) != a.src[3];
    if (a.nwords <= kStepMax && a.nsq <= kStepMax) {
        if (threadIdx.x < a.nwords) {
            stage[threadIdx.x] = a.src[threadIdx.x];
            if (a.mirror) a.mirror[threadIdx.x] = stage[threadIdx.x];
        }
        __syncthreads();
        fs_step_warps(S, W, stage, a.nwords, a.nsq);
        __syncthreads();
        if (threadIdx.x == 0 && bad) S.err |= FS_ERR_SUMCHECK;
        if (threadIdx.x < a.nsq) a.out[threadIdx.x] = W.sq[threadIdx.x];
        store_state(S, g);
        return;
    }
    // long runs (yr) with the message schedules in parallel
    if (a.nwords >= 64) fs_absorb_sched(S, a.src, a.nwords, W.kw, a.mirror);
    else fs_absorb_block(S, a.src, a.nwords, stage, 64, a.mirror);
    if (bad) S.err |= FS_ERR_SUMCHECK;
    __syncthreads();
    fs_fields(S, B, a.nsq, a.out);
    store_state(S, g);
}

// Exclusive prefix count of `flag` over the block (kQBlock threads) and
// the total; `scratch` holds kQBlock / 32 words.
__device__ uint32_t block_rank(bool flag, uint32_t *scratch, uint32_t *total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t m = __ballot_sync(0xffffffffu, flag);
    if (lane == 0) scratch[warp] = __popc(m);
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (uint32_t w = 0; w < kQBlock / 32; ++w) {
        const uint32_t c = scratch[w];
        before += w < warp ? c : 0;
        all += c;
    }
    __syncthreads();
    *total = all;
    return before + __popc(m & ((1u << lane) - 1));
}

// At most 2 kQBlock values (the queries taken and a batch) go into a set
// of kHash slots, so probing always ends within the table.
constexpr uint32_t kHash = 4 * kQBlock;
static_assert(kHash == 1024, "hash_insert takes 10 bits of the hash");
__device__ uint32_t hash_insert(unsigned long long *key, uint32_t *rank, uint64_t v, uint32_t r) {
    uint32_t h = ((uint32_t)(v ^ (v >> 31)) * 0x9E3779B1u) >> 22;  // 10 bits: kHash = 1024 slots
    for (uint32_t probe = 0; probe < kHash; ++probe) {
        const unsigned long long prev = atomicCAS(key + h, ~0ull, (unsigned long long)v);
        if (prev == ~0ull || prev == v) {
            atomicMin(rank + h, r);
            return h;
        }
        h = (h + 1) & (kHash - 1);
    }
    return kHash - 1;  // unreachable: the table is never more than half full
}

// Squeezes of a batch, and the blocks hashed in it: the full blocks of the
// chain, one final block a squeeze and a second one for the squeezes whose
// last data leaves no room for the padding (two words of each 16).
constexpr uint32_t kBatch = 176;
constexpr uint32_t kChainRows = (15 + kStepMax + kBatch) / 16 + 1;
constexpr uint32_t kFinalRows = kBatch + 2 * (kBatch / 16 + 2);
constexpr size_t kQuerySmem = (size_t)(kChainRows + kFinalRows) * kKwStride * 4;
// p' < p with p' % 16 >= 14
__device__ __forceinline__ uint32_t two_below(uint32_t p) { return 2 * (p >> 4) + ((p & 15) > 14 ? 1u : 0u); }

// Warp 0 runs the chain of full blocks the batch's counters complete (about
// ten), warp 1 ahead of it their schedules and the other warps meanwhile the
// schedules of every squeeze's final blocks, which depend on the counters
// only; then all squeezes finish side by side.  Bound by the chain: rounds of
// one warp, about 1 us a block.
__global__ void __launch_bounds__(kQBlock) k_fs_queries(FsState *g, FsQueries a, FsStrides st) {
    pdl_begin();
    {
        const uint32_t b = blockIdx.x;  // lockstep batch: one block per proof
        g += b;
        if (a.src) a.src += b * st.src;
        if (a.out) a.out += b * st.out;
        if (a.mirror) a.mirror += b * st.mirror;
        a.q += b * st.q;
        a.nodes += b * st.nodes;
        a.nnodes += b * st.nnodes;
    }
    extern __shared__ __align__(16) uint32_t kw_rows[];
    auto chain_kw = [&](uint32_t f) { return kw_rows + f * kKwStride; };
    auto final_kw = [&](uint32_t f) { return kw_rows + (kChainRows + f) * kKwStride; };
    __shared__ FsState S;
    __shared__ Batch B;
    __shared__ uint32_t root[kStepMax];
    __shared__ __align__(16) uint32_t acc[kQBlock];  // the queries taken
    __shared__ uint32_t sorted[kQBlock];
    __shared__ unsigned long long hkey[kHash];
    __shared__ uint32_t hrank[kHash];
    __shared__ uint32_t lo32[kQBlock];  // a batch's squeezes, by index
    __shared__ uint32_t scratch[kQBlock / 32];
    __shared__ uint32_t wcnt[32][kQBlock / 32], wmask[32][kQBlock / 32];
    __shared__ uint32_t take_sh, batch_sh;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    load_state(S, g);
    uint32_t na = a.nwords;  // words absorbed with the first batch
    if (tid < na) {
        root[tid] = a.src[tid];
        if (a.mirror) a.mirror[tid] = root[tid];
    }
    __syncthreads();
    const bool ok = a.n >= a.s && a.s >= 1 && a.s <= kQBlock;
    const uint32_t mask = (uint32_t)(a.n - 1);  // n is a power of two: % n is a mask
    uint32_t count = 0, batch = 0, take = 0;
    // get_distinct_queries in batches of squeezes; the round bound only
    // guards a state that cannot progress (n >= s always can)
    for (uint32_t round = 0; ok && count < a.s && round < 1024; ++round) {
        // the queries still needed, about twice the repeats expected among
        // them (need (need/2 + count) / n) plus 2 more, and the challenges
        // squeezed after them: the chain of full blocks a batch completes is
        // its serial part, so the batch is kept tight; a short batch just
        // takes another round
        const uint32_t need = a.s - count;
        const uint64_t margin = ((uint64_t)need * (need + 2ull * count)) / a.n + 2;
        const uint64_t want = need + margin + a.nsq;
        batch = want < kBatch ? (uint32_t)want : kBatch;
        const FsStream str(S, root, na);
        const uint32_t s0 = str.nw + na + 1;  // squeeze i ends after s0 + i words
        const uint32_t full = (s0 - 1 + batch) / 16, t0 = two_below(s0);
        for (uint32_t i = tid; i < kHash; i += blockDim.x) {
            hkey[i] = ~0ull;  // never a value: values are < n <= 2^31
            hrank[i] = ~0u;
        }
        if (warp == 0) {
            uint32_t h[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) h[k] = S.h[k];
            if (lane == 0)
#pragma unroll
                for (int k = 0; k < 8; ++k) B.chain[0][k] = h[k];
            for (uint32_t f = 0; f < full; ++f) {
                sha_rounds_kw(h, chain_kw(f), [&](int c) {
                    if (f == 0) asm volatile("bar.sync %0, 64;" ::"r"(1 + c) : "memory");
                });
                if (lane == 0)
#pragma unroll
                    for (int k = 0; k < 8; ++k) B.chain[f + 1][k] = h[k];
            }
        } else if (warp == 1) {
            uint32_t blk[16];
            const uint32_t f = min(lane, kChainRows - 1);
#pragma unroll
            for (int k = 0; k < 16; ++k) blk[k] = str.word(16 * f + k);
            if (full)
                sha_schedule_kw(blk, chain_kw(f), [](int c) {
                    __syncwarp();
                    asm volatile("bar.arrive %0, 64;" ::"r"(1 + c) : "memory");
                });
        } else {
            // row i: squeeze i's first final block; row batch + r: the r-th
            // two-block squeeze's second
            const uint32_t n2 = two_below(s0 + batch) - t0;
            for (uint32_t t = tid - 64; t < batch + n2; t += kQBlock - 64) {
                uint32_t i = t;
                if (t >= batch) {
                    const uint32_t r = t - batch + t0;
                    i = 16 * (r >> 1) + 14 + (r & 1) - s0;
                }
                uint32_t blk[16];
                str.final_block(i, t >= batch, blk);
                sha_schedule_kw(blk, final_kw(t));
            }
        }
        __syncthreads();
        {
            // the two-block squeezes on the first threads, so that only their
            // warps run two compressions
            const uint32_t n2 = two_below(s0 + batch) - t0;
            if (tid < batch) {
                uint32_t p;
                if (tid < n2) {
                    const uint32_t r = tid + t0;
                    p = 16 * (r >> 1) + 14 + (r & 1);
                } else {
                    const uint32_t r = tid - n2 + (s0 - t0);
                    p = 16 * (r / 14) + r % 14;
                }
                const uint32_t i = p - s0, fb = p / 16;
                uint32_t h[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) h[k] = B.chain[fb][k];
                sha_rounds_kw(h, final_kw(i));
                if (tid < n2) sha_rounds_kw(h, final_kw(batch + tid));
                lo32[i] = bswap32(h[0]);
            }
        }
        __syncthreads();
        const uint32_t qv = tid < batch ? lo32[tid] & mask : 0;
        // Repeats: the queries taken so far (rank 0) and this batch's
        // squeezes (rank i + 1) go into a shared hash set that keeps each
        // value's smallest rank; a squeeze is new iff it holds its value's.
        if (tid < count) hash_insert(hkey, hrank, acc[tid], 0);
        const uint32_t slot = tid < batch ? hash_insert(hkey, hrank, qv, tid + 1) : 0;
        __syncthreads();
        const bool dup = tid >= batch || hrank[slot] != tid + 1;
        uint32_t fresh;
        const uint32_t rank = block_rank(!dup, scratch, &fresh);
        if (!dup && rank < need) acc[count + rank] = qv;
        // squeezes consumed: the whole batch, or up to the one that
        // completes the set
        if (tid == 0) take_sh = batch;
        __syncthreads();
        if (fresh >= need && !dup && rank == need - 1) take_sh = tid + 1;
        __syncthreads();
        take = take_sh;
        count += min(fresh, need);
        // the challenges after the last query are the next squeezes of this
        // batch when it has them; commit past those too
        const uint32_t extra = count == a.s && take + a.nsq <= batch ? a.nsq : 0;
        if (tid < extra) a.out[tid] = lo32[take + tid];
        if (warp == 0) {  // the state past them
            const uint32_t len = str.nw + na + take + extra, rem = len & 15;
            const uint32_t w = lane < rem ? str.word((len & ~15u) + lane) : 0u;
            __syncwarp();
            if (lane < 16) S.w[lane] = w;
            if (lane < 8) S.h[lane] = B.chain[len / 16][lane];
            if (lane == 0) {
                S.nw = rem;
                S.total += 4ull * (na + take + extra);
                S.counter += take + extra;
                batch_sh = extra;
            }
        }
        na = 0;
        __syncthreads();
    }
    const uint32_t done_extra = ok && count == a.s ? batch_sh : 0;
    if (!ok || count < a.s) {
        if (tid == 0) {
            S.err |= FS_ERR_QUERIES;
            *a.nnodes = 0;
        }
        for (uint32_t i = tid; i < a.s && i < kQBlock; i += blockDim.x) a.q[i] = 0;
    } else {
        // sorted by rank: the queries are distinct, so a query's place is the
        // number of smaller ones (four compared a load)
        if (tid >= count) acc[tid] = ~0u;
        __syncthreads();
        const bool have = tid < count;
        {
            const uint32_t v = acc[tid];
            uint32_t below = 0;
            for (uint32_t j = 0; j < (count + 3) / 4; ++j) {
                const uint4 x = reinterpret_cast<const uint4 *>(acc)[j];
                below += (x.x < v) + (x.y < v) + (x.z < v) + (x.w < v);
            }
            if (have) sorted[below] = v;
        }
        __syncthreads();
        if (have) a.q[tid] = sorted[tid];
        // Multi-proof siblings (merkle_tree::prove, src/merkle_tree.rs:62-111):
        // at layer d the present nodes are x = q >> d; the sibling x ^ 1 is
        // emitted, in order of x, unless it is present too.  Queries are
        // sorted, so the nodes equal to x form a run and x's sibling can only
        // be the run's neighbour: an odd x is settled at its run's first
        // query by the previous query, an even x at its run's last query by
        // the next one.  Either emits iff the neighbour is not under x's
        // parent, i.e. iff it differs from q in a bit above d: so query i
        // emits in layer d if bit d is set and the previous query's highest
        // differing bit is above d, or bit d is clear and the next one's is.
        const uint32_t qi = have ? sorted[tid] : 0;
        const uint32_t dp = have && tid > 0 ? qi ^ sorted[tid - 1] : ~0u;
        const uint32_t dn = have && tid + 1 < count ? qi ^ sorted[tid + 1] : ~0u;
        uint32_t nl = 0;
        while ((1ull << nl) < a.n) ++nl;
        // bits below the highest set bit of d (all of them when there is no neighbour)
        auto under = [](uint32_t d) { return d == ~0u ? ~0u : (1u << (31 - __clz(d))) - 1; };
        const uint32_t emask =
            have ? ((qi & under(dp)) | (~qi & under(dn))) & (nl >= 32 ? ~0u : (1u << nl) - 1) : 0u;
        // Per-warp counts of every layer, then one scan gives each warp its
        // start in each layer (layers in order, threads in query order).
        for (uint32_t d = 0; d < nl; ++d) {
            const uint32_t m = __ballot_sync(0xffffffffu, (emask >> d) & 1);
            if (lane == 0) {
                wcnt[d][warp] = __popc(m);
                wmask[d][warp] = m;
            }
        }
        __syncthreads();
        if (warp == 0) {  // lane l scans layer l
            uint32_t tot = 0;
            if (lane < nl)
                for (uint32_t w = 0; w < kQBlock / 32; ++w) {
                    const uint32_t c = wcnt[lane][w];
                    wcnt[lane][w] = tot;
                    tot += c;
                }
            uint32_t inc = tot;
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane < nl)
                for (uint32_t w = 0; w < kQBlock / 32; ++w) wcnt[lane][w] += inc - tot;
            if (lane == 31) take_sh = inc;
        }
        __syncthreads();
        uint32_t left = emask;
        while (left) {
            const uint32_t d = __ffs(left) - 1;
            left &= left - 1;
            const uint32_t pos = wcnt[d][warp] + __popc(wmask[d][warp] & ((1u << lane) - 1));
            // layer d starts after n + n/2 + ... = 2n - 2n/2^d nodes
            if (pos < a.nodes_cap) a.nodes[pos] = 2 * a.n - (2 * a.n >> d) + ((qi >> d) ^ 1);
        }
        const uint32_t nout = take_sh;
        if (tid == 0) {
            *a.nnodes = nout;
            if (nout > a.nodes_cap) S.err |= FS_ERR_QUERIES;
        }
    }
    __syncthreads();
    if (done_extra < a.nsq) fs_fields(S, B, a.nsq - done_extra, a.out + done_extra);
    store_state(S, g);
}

}  // namespace

cudaError_t fs_step(Launcher &L, FsState *d, const FsStep &a, uint32_t B, const FsStrides &st) {
    if (a.nwords > 1024 || (a.nwords && !a.src) || a.nsq > 256 || (a.nsq && !a.out) ||
        (a.check && (!a.src || a.nwords < 3)) || (a.nzero && !a.zero) || B == 0 || B > 65535)
        return cudaErrorInvalidValue;
    LGK_LAUNCH(L, "fs_step", launch_k(k_fs_step, B, 64, 0, L.stream, d, a, st));
    return cudaGetLastError();
}

cudaError_t fs_queries(Launcher &L, FsState *d, const FsQueries &a, uint32_t B, const FsStrides &st) {
    if (a.s == 0 || a.s > kQBlock || a.n == 0 || (a.n & (a.n - 1)) || a.n > (1ull << 31) || a.nwords > kStepMax ||
        (a.nwords && !a.src) ||
        a.nsq > kQBlock || (a.nsq && !a.out) || !a.q || !a.nodes || !a.nnodes || B == 0 || B > 65535)
        return cudaErrorInvalidValue;
    cudaFuncSetAttribute(k_fs_queries, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kQuerySmem);
    LGK_LAUNCH(L, "fs_queries", launch_k(k_fs_queries, B, kQBlock, kQuerySmem, L.stream, d, a, st));
    return cudaGetLastError();
}

}  // namespace lgk
