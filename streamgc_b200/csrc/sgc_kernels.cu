// sgc_kernels.cu -- kernels of the handle API (sm_100a).
//
//   seq_apply_kernel      one warp applies a batch (or each graph's part of it)
//                         in stream order: the reference's local_update_kernel
//                         run as a single warp (local_update.cu:61-147),
//                         bit-exact; the block's other warps prepare ahead.
//   conc_*                a batch applied by one warp per edge. A hash pre-pass
//                         links each update to the previous and the next update
//                         of the same edge in the batch; the persistent apply
//                         kernel hands out update tickets and the first update
//                         of each edge applies that edge's updates in stream
//                         order, so the edge set after a batch equals the
//                         sequential one; updates of different edges overlap.
//   dirty list + compact  stable per-row compaction (epoch_maintenance.cu:20-61)
//                         of only the rows edited since their last compaction
//                         (every other row is already compact, so compacting it
//                         is the identity); reads each row up to its high-water.
//   drain                 streamgc.cu:967-995 + epoch_maintenance.cu:66-87.
//   sweep                 degree-balanced pass over every live adjacency entry:
//                         rebuild_bitmaps (epoch_maintenance.cu:113-128) and the
//                         Tier-1 decision (conflict_repair.cu:10-114) fused, as a
//                         Jacobi sweep (every decision reads start-of-sweep
//                         colors; new words are committed after the sweep).
#include <cuda_runtime.h>
#include <cuda/atomic>

#include <algorithm>

#include "sgc_kernels.cuh"

namespace sgc {

// ---------------------------------------------------------------------------
// warp helpers
// ---------------------------------------------------------------------------

// One atomicAdd per warp; returns this lane's slot when pred, else NONE32.
__device__ __forceinline__ uint32_t warp_append(uint32_t* count, bool pred) {
    const uint32_t m = __ballot_sync(FULL, pred);
    if (!m) return NONE32;
    const uint32_t lane = lane_id();
    const int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if ((int)lane == leader) base = atomicAdd(count, (uint32_t)__popc(m));
    base = __shfl_sync(FULL, base, leader);
    return pred ? base + __popc(m & ((1u << lane) - 1)) : NONE32;
}

// Exclusive warp prefix sum.
__device__ __forceinline__ uint32_t warp_excl_scan(uint32_t v, uint32_t& total) {
    const uint32_t lane = lane_id();
    uint32_t x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, x, off);
        if (lane >= (uint32_t)off) x += y;
    }
    total = __shfl_sync(FULL, x, 31);
    return x - v;
}

// One warp's words of a bitmask as list entries, appended at *count.
__device__ __forceinline__ void list_bits(uint32_t w, uint32_t bits, uint32_t* list, uint32_t* count) {
    if (!__any_sync(FULL, bits)) return;
    uint32_t total = 0;
    const uint32_t off = warp_excl_scan(__popc(bits), total);
    uint32_t base = 0;
    if (lane_id() == 0 && total) base = atomicAdd(count, total);
    base = __shfl_sync(FULL, base, 0);
    uint32_t k = base + off;
    while (bits) {
        const int i = __ffs(bits) - 1;
        bits &= bits - 1;
        list[k++] = w * 32 + i;
    }
}

// ---------------------------------------------------------------------------
// update kernels
// ---------------------------------------------------------------------------

// Stream order: block per segment [segs[k], segs[k+1]) of the batch (one
// graph's updates; without `segs` the whole batch is one). Warp 0 applies the
// segment's updates one after another while the others prepare the next chunk's,
// a warp each; chunks meet at a block barrier. The time is one warp's chain of
// dependent loads and instructions. One warp alone, its words in L2, took 4.1 us
// per update (8,192 updates of an R-MAT graph of 16,384 vertices, 34 ms); with
// the searches prepared and the words in L1 0.84 us. Reading ahead without
// handing over the slots gave 2.4 us: the search's instructions, not only its
// loads, are on the chain.
__global__ void __launch_bounds__(32 * kSeqWarps, 1) seq_apply_kernel(Dev g, const EdgeUpdate* __restrict__ ups,
                                                                   const uint32_t* __restrict__ segs,
                                                                   const uint32_t* dyn, uint32_t n) {
    __shared__ SeqShared sh;
    const uint32_t nseg = segs ? ld_cg(dyn + 2) : 1u;
    const uint32_t warp = threadIdx.x >> 5;
    for (uint32_t i = threadIdx.x; i < kSeqMarks; i += blockDim.x) sh.mark[i] = 0;
    for (uint32_t i = threadIdx.x; i < 4 * kSeqChunk; i += blockDim.x) (&sh.log[0][0])[i] = make_uint2(NOSLOT, 0);
    uint32_t chunk = 2;  // a mark of 0 reads as not edited
    for (uint32_t k = blockIdx.x; k < nseg; k += gridDim.x) {
        const uint32_t a = segs ? segs[k] : 0u, e = segs ? segs[k + 1] : n;
        if (a >= e) continue;
        auto prepare = [&](uint32_t c, uint32_t to) {  // warp w takes update c + w - 1
            const uint32_t j = warp - 1;
            if (warp != 0 && j < e - c)
                seq_prepare(g, sh, to & 1u, j, ld_w4<true>(reinterpret_cast<const uint32_t*>(ups + c + j)));
        };
        prepare(a, chunk);
        __syncthreads();
        for (uint32_t c = a;; c += kSeqChunk, chunk++) {
            const uint32_t m = e - c < kSeqChunk ? e - c : kSeqChunk;
            if (warp == 0) {
                for (uint32_t j = 0; j < m; j++) seq_apply(g, sh, chunk, j);
                if (lane_id() < 2 * (kSeqChunk - m)) sh.log[chunk & 1u][2 * m + lane_id()] = make_uint2(NOSLOT, 0);
            } else if (e - c > kSeqChunk) {
                prepare(c + kSeqChunk, chunk + 1);
            }
            __syncthreads();
            if (e - c <= kSeqChunk) break;
        }
        chunk++;
    }
}
void launch_det_apply(const Dev& g, const EdgeUpdate* ups, uint32_t n, cudaStream_t s) {
    if (n) seq_apply_kernel<<<1, 32 * kSeqWarps, 0, s>>>(g, ups, nullptr, nullptr, n);
}
// A block per segment, but not one on every SM (spare_sms): the kernel is as long
// as its longest segments.
void launch_seg_apply(const Dev& g, const EdgeUpdate* ups, const uint32_t* segs, const uint32_t* dyn, uint32_t max_segs,
                      int num_sms, cudaStream_t s) {
    const uint32_t blocks = std::min(std::max(max_segs, 1u), spare_sms(num_sms));
    seq_apply_kernel<<<blocks, 32 * kSeqWarps, 0, s>>>(g, ups, segs, dyn, 0);
}

__device__ __forceinline__ unsigned long long edge_key(uint32_t u, uint32_t v) {
    const uint32_t a = u < v ? u : v, b = u < v ? v : u;
    return ((unsigned long long)a << 32) | b;
}
__device__ __forceinline__ unsigned long long key_hash(unsigned long long k) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return k;
}

// `dyn` (device words, optional): [0] the batch size; it replaces the `n`
// argument so that a captured CUDA graph can replay the launches on every
// tick. Grid-stride loops.
__device__ __forceinline__ uint32_t batch_n(uint32_t n, const uint32_t* dyn) { return dyn ? ld_cg(dyn) : n; }

__global__ void conc_prep_insert(Dev g, const EdgeUpdate* __restrict__ ups, uint32_t n_arg, EdgeOrder eo,
                                 const uint32_t* dyn) {
    const uint32_t n = batch_n(n_arg, dyn);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *eo.ticket = 0;
        if (g.hub_count) *g.hub_count = 0;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint4 r = ld_cg4(reinterpret_cast<const uint32_t*>(ups + i));
        const uint32_t u = r.x, v = r.y;
        const uint8_t type = (uint8_t)(r.z & 0xFFu);
        if ((type != SGC_UPDATE_ADD && type != SGC_UPDATE_DEL) || u >= g.n || v >= g.n) {
            eo.tslot[i] = NONE32;
            continue;
        }
        const unsigned long long key = edge_key(u, v);
        // Double hashing (an odd step visits every slot of the power-of-two table):
        // the kernel's time is its longest chain of probes, which at half load is
        // near log2(n) this way but over fifty slots' cluster in a row with step 1
        // (an epoch of 65,536 updates, this kernel 16 us of it, became 7 us shorter).
        const unsigned long long mix = key_hash(key);
        const uint32_t step = (uint32_t)(mix >> 32) | 1u;
        uint32_t h = (uint32_t)mix & eo.tmask;
        for (uint32_t probe = 0; probe <= eo.tmask; probe++) {
            const unsigned long long k = atomicCAS(eo.tkey + h, EMPTY64, key);
            if (k == EMPTY64 || k == key) break;
            h = (h + step) & eo.tmask;
        }
        eo.tslot[i] = h;
        eo.tnext[i] = atomicExch(eo.thead + h, i);
    }
}

// Per update: the previous and the next update of the same edge in stream
// order (NONE32 at the ends), from the slot's push list.
__global__ void conc_prep_prev(uint32_t n_arg, EdgeOrder eo, const uint32_t* dyn, uint32_t* err) {
    const uint32_t n = batch_n(n_arg, dyn);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t h = ld_cg(eo.tslot + i);
        uint32_t prev = NONE32, next = NONE32;
        if (h != NONE32) {
            // a list holds distinct positions of this batch: at most n links
            uint32_t links = 0;
            for (uint32_t j = ld_cg(eo.thead + h); j != NONE32; j = ld_cg(eo.tnext + j)) {
                if (j >= n || ++links > n) {
                    atomicOr(err, ERR_CHAIN);
                    break;
                }
                if (j < i && (prev == NONE32 || j > prev)) prev = j;
                if (j > i && (next == NONE32 || j < next)) next = j;
            }
        }
        eo.tprev[i] = prev;
        eo.tsucc[i] = next;
    }
}

// Warp per edge: a warp takes tickets (update positions) and, when the update
// is the first of its edge in the batch, applies every update of that edge in
// stream order; the later ones are skipped at their own tickets. So the
// updates of one edge never run concurrently and no warp waits for another.
// The batch and the ordering words were written by the copy and the prep
// kernels before this launch: L2-coherent loads. A warp takes its next ticket
// while it applies the current update, and reads a position's ordering words
// and record in one round (the next update of an edge's chain with them).
// Three blocks per SM: 80 registers (the budget the one-warp-per-update
// version ran fastest with; 64 registers spill the update path).
__global__ void __launch_bounds__(256, 3) conc_apply_kernel(Dev g, const EdgeUpdate* __restrict__ ups, uint32_t n_arg,
                                                            EdgeOrder eo, const uint32_t* dyn) {
    const uint32_t n = batch_n(n_arg, dyn);
    uint32_t i = 0;
    if (lane_id() == 0) i = atomicAdd(eo.ticket, 1u);
    i = __shfl_sync(FULL, i, 0);
    while (i < n) {
        uint32_t next = 0;
        if (lane_id() == 0) next = atomicAdd(eo.ticket, 1u);  // used after this update
        const uint32_t h = ld_cg(eo.tslot + i);
        const uint32_t prev = ld_cg(eo.tprev + i);
        uint32_t succ = ld_cg(eo.tsucc + i);
        uint4 r = ld_cg4(reinterpret_cast<const uint32_t*>(ups + i));
        if (h == NONE32) {
            if ((r.x >= g.n || r.y >= g.n) && lane_id() == 0) atomicAdd(g.nskip, 1ull);
        } else if (prev == NONE32) {  // the first update of its edge applies the whole chain
            uint32_t steps = 1;
            for (;;) {
                if (r.x >= g.n || r.y >= g.n) {
                    if (lane_id() == 0) atomicOr(g.err, ERR_CHAIN);
                    break;
                }
                warp_apply(g, r.x, r.y, (uint8_t)(r.z & 0xFFu));
                const uint32_t j = succ;
                if (j == NONE32) break;
                if (j >= n || j < i || ++steps > n) {  // ordering words inconsistent with the batch
                    if (lane_id() == 0) atomicOr(g.err, ERR_CHAIN);
                    break;
                }
                succ = ld_cg(eo.tsucc + j);
                r = ld_cg4(reinterpret_cast<const uint32_t*>(ups + j));
            }
            if (lane_id() == 0 && h <= eo.tmask) {  // no kernel reads the table during apply: reset it for the next batch
                eo.tkey[h] = EMPTY64;
                eo.thead[h] = NONE32;
            }
            __syncwarp();
        }
        i = __shfl_sync(FULL, next, 0);
    }
}

// ---------------------------------------------------------------------------
// The pass after a concurrent batch: row-scale operations the apply left
// (HubOp), one block of kHubThreads per operation. Each re-reads x's state
// word; the scans and the neighbor walk after a move take 8192 slots per
// round over the whole block. Decisions are made on words thread 0 read and
// shared, so every branch is block-uniform.
// ---------------------------------------------------------------------------
constexpr uint32_t kHubThreads = 1024;

// The ids of one round's slots: thread t loads the 16-byte chunks at
// c + 4t and c + 4t + 4096 (INV outside [s, e) and for ids >= n).
__device__ __forceinline__ void hub_round(const Dev& g, uint64_t c, uint64_t s, uint64_t e, uint32_t (&y)[8]) {
    const uint64_t i0 = c + 4ull * threadIdx.x, i1 = i0 + 4ull * kHubThreads;
    uint4 q0 = make_uint4(INV, INV, INV, INV), q1 = q0;
    if (i0 < e) q0 = ld_cg4(g.col + i0);
    if (i1 < e) q1 = ld_cg4(g.col + i1);
    const uint32_t v[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
    for (int t = 0; t < 8; t++) {
        const uint64_t p = (t < 4 ? i0 : i1) + (t & 3);
        y[t] = (p >= s && p < e && v[t] < g.n) ? v[t] : INV;
    }
}

// Does a live neighbor in [s, e) hold color c? Stops after the first round that finds one.
__device__ __forceinline__ bool block_color_held(const Dev& g, uint64_t s, uint64_t e, uint16_t c) {
    for (uint64_t r = s & ~3ull; r < e; r += 8ull * kHubThreads) {
        uint32_t y[8];
        hub_round(g, r, s, e, y);
        uint32_t w[8];
#pragma unroll
        for (int t = 0; t < 8; t++) w[t] = y[t] != INV ? ld_cg(g.st + y[t]) : 0u;
        bool hit = false;
#pragma unroll
        for (int t = 0; t < 8; t++) hit |= y[t] != INV && color_of(w[t]) == c;
        if (__syncthreads_or(hit)) return true;
    }
    return false;
}

// Exact selection: the first color no live neighbor in [s, e) holds (colors
// 1..2047, else 2048), as warp_fac_exact. `used`: 64 words of shared memory.
__device__ __forceinline__ uint16_t block_fac_exact(const Dev& g, uint64_t s, uint64_t e, uint32_t* used,
                                                    uint32_t* pick) {
    if (threadIdx.x < 64) used[threadIdx.x] = 0;
    __syncthreads();
    uint32_t lo = 0, hi = 0;  // colors 1..64 (bits 0..63 of a 64-bit mask)
    for (uint64_t r = s & ~3ull; r < e; r += 8ull * kHubThreads) {
        uint32_t y[8];
        hub_round(g, r, s, e, y);
        uint32_t w[8];
#pragma unroll
        for (int t = 0; t < 8; t++) w[t] = y[t] != INV ? ld_cg(g.st + y[t]) : 0u;
#pragma unroll
        for (int t = 0; t < 8; t++) {
            if (y[t] == INV) continue;
            const uint16_t c = color_of(w[t]);
            add_color_bit(c, lo, hi);
            if (c > 64 && c < 2048) atomicOr(&used[c >> 5], 1u << (c & 31));
        }
    }
    lo = __reduce_or_sync(FULL, lo);
    hi = __reduce_or_sync(FULL, hi);
    if (lane_id() == 0) {  // fold colors 1..64 into the same set (color c: word c >> 5, bit c & 31)
        if (lo) atomicOr(&used[0], lo << 1);
        if (lo >> 31) atomicOr(&used[1], 1u);
        if (hi) atomicOr(&used[1], hi << 1);
        if (hi >> 31) atomicOr(&used[2], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t l = threadIdx.x;
        uint32_t w0 = ~used[l], w1 = ~used[l + 32];
        if (l == 0) w0 &= ~1u;  // color 0 is never a candidate
        const uint32_t b0 = __ballot_sync(FULL, w0 != 0), b1 = __ballot_sync(FULL, w1 != 0);
        if (l == 0) {
            uint32_t c = 2048;
            if (b0) {
                const int src = __ffs(b0) - 1;
                c = src * 32 + __ffs(~used[src] & (src == 0 ? ~1u : FULL)) - 1;
            } else if (b1) {
                const int src = __ffs(b1) - 1;
                c = 1024 + src * 32 + __ffs(~used[src + 32]) - 1;
            }
            *pick = c;
        }
    }
    __syncthreads();
    const uint16_t c = (uint16_t)*pick;
    __syncthreads();
    return c;
}

__global__ void __launch_bounds__(kHubThreads) hub_ops_kernel(Dev g) {
    __shared__ uint32_t used[64];
    __shared__ uint32_t word[2];
    const uint32_t total = ld_cg(g.hub_count);
    const uint32_t cnt = total < g.hub_cap ? total : g.hub_cap;
    if (blockIdx.x == 0 && threadIdx.x == 0 && cnt) atomicAdd(g.hub_total, (unsigned long long)cnt);
    for (uint32_t k = blockIdx.x; k < cnt; k += gridDim.x) {
        const HubOp op = g.hub_ops[k];
        const uint32_t x = op.x;
        if (x >= g.n) continue;  // block-uniform: every thread read the same record
        const uint32_t kind = op.op >> 16;
        const uint16_t freed = (uint16_t)(op.op & 0xFFFFu);
        const uint64_t s = g.rp[x], e = live_end(g, x, s);
        if (threadIdx.x == 0) word[0] = ld_cg(g.st + x);
        __syncthreads();
        uint32_t cur = word[0];
        __syncthreads();
        uint16_t newc;
        if (kind == HUB_REDUCE) {
            if (freed == 0 || freed >= color_of(cur) || block_color_held(g, s, e, freed)) continue;
            newc = freed;
        } else {
            newc = block_fac_exact(g, s, e, used, &word[1]);
        }
        // recolor_vertex: compare-and-swap (newc, version + 1) in; a changed word
        // re-selects from the live neighbors, as the warp's recolor does
        bool moved = false;
        for (uint32_t tries = 0;; tries++) {
            if (newc == color_of(cur)) break;
            if (threadIdx.x == 0) word[0] = atomicCAS(g.st + x, cur, pack(newc, (uint16_t)(version_of(cur) + 1)));
            __syncthreads();
            const uint32_t got = word[0];
            __syncthreads();
            if (got == cur) {
                moved = true;
                break;
            }
            if (tries >= 1024u) {  // the repair after the batch settles x
                if (threadIdx.x == 0) atomicOr(g.err, ERR_RETRY);
                break;
            }
            cur = got;
            newc = block_fac_exact(g, s, e, used, &word[1]);
        }
        if (!moved) continue;
        if (threadIdx.x == 0) {
            mark_touched(g, x);
            note_color(g, x);
        }
        const uint16_t oldc = color_of(cur);
        for (uint64_t r = s & ~3ull; r < e; r += 8ull * kHubThreads) {
            uint32_t y[8];
            hub_round(g, r, s, e, y);
#pragma unroll
            for (int t = 0; t < 8; t++)
                if (y[t] != INV) nbr_color_change(g, y[t], oldc, newc);
        }
    }
}

// After a batch (exact selection): both endpoints of every ADD whose colors
// are equal are marked for the next repair. Together with the marks of every
// color change, this makes every conflict of the rows have a marked endpoint
// once the last repair ended proper.
__global__ void add_check_kernel(Dev g, const EdgeUpdate* __restrict__ ups, uint32_t n, const uint32_t* dyn) {
    const uint32_t cnt = dyn ? ld_cg(dyn) : n;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
        const uint4 r = ld_cg4(reinterpret_cast<const uint32_t*>(ups + i));
        if ((r.z & 0xFFu) != SGC_UPDATE_ADD || r.x >= g.n || r.y >= g.n || r.x == r.y) continue;
        const uint16_t a = color_of(ld_cg(g.st + r.x)), b = color_of(ld_cg(g.st + r.y));
        if (a == b && a != 0) {
            mark_touched(g, r.x);
            mark_touched(g, r.y);
        }
    }
}
void launch_add_check(const Dev& g, const EdgeUpdate* ups, uint32_t n, const uint32_t* dyn, int num_sms,
                      cudaStream_t s) {
    if (!g.touched || (!dyn && !n)) return;
    uint32_t blk = dyn ? (uint32_t)num_sms * 4 : (n + 255) / 256;
    if (blk > (uint32_t)num_sms * 4) blk = num_sms * 4;
    add_check_kernel<<<blk, 256, 0, s>>>(g, ups, n, dyn);
}

// The ingest ring's drain: positions [head, head + n) of a host ring of
// mask + 1 slots, read straight from pinned, device-mapped host memory (16
// bytes per thread, consecutive slots) into the batch buffer.
__global__ void ring_gather_kernel(const uint4* __restrict__ ring, unsigned long long mask, unsigned long long head,
                                   uint32_t n, uint4* __restrict__ out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = ring[(head + i) & mask];
}
void launch_ring_gather(const EdgeUpdate* ring, uint64_t mask, uint64_t head, uint32_t n, EdgeUpdate* out,
                        int num_sms, cudaStream_t s) {
    if (!n) return;
    uint32_t blk = (n + 255) / 256;
    if (blk > (uint32_t)num_sms * 4) blk = num_sms * 4;
    ring_gather_kernel<<<blk, 256, 0, s>>>(reinterpret_cast<const uint4*>(ring), mask, head, n,
                                           reinterpret_cast<uint4*>(out));
}

int conc_apply_occupancy() {
    static int occ = 0;
    if (!occ) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, conc_apply_kernel, 256, 0);
        if (occ < 1) occ = 1;
    }
    return occ;
}

void launch_conc_apply(const Dev& g, const EdgeUpdate* ups, uint32_t n, const EdgeOrder& eo, int num_sms,
                       cudaStream_t s) {
    if (!n) return;
    uint32_t blk = (n + 255) / 256;
    if (blk > (uint32_t)num_sms * 16) blk = num_sms * 16;
    conc_prep_insert<<<blk, 256, 0, s>>>(g, ups, n, eo, nullptr);
    conc_prep_prev<<<blk, 256, 0, s>>>(n, eo, nullptr, g.err);
    uint32_t grid = (uint32_t)(num_sms * conc_apply_occupancy());
    const uint32_t need = (n + 7) / 8;  // 8 warps per block
    if (grid > need) grid = need;
    conc_apply_kernel<<<grid, 256, 0, s>>>(g, ups, n, eo, nullptr);
    if (g.hub_ops) hub_ops_kernel<<<num_sms, kHubThreads, 0, s>>>(g);
}

void launch_conc_apply_dyn(const Dev& g, const EdgeUpdate* ups, const uint32_t* dyn, const EdgeOrder& eo,
                           int num_sms, int blocks_per_sm, cudaStream_t s) {
    conc_prep_insert<<<num_sms * 16, 256, 0, s>>>(g, ups, 0, eo, dyn);
    conc_prep_prev<<<num_sms * 16, 256, 0, s>>>(0, eo, dyn, g.err);
    const int occ = conc_apply_occupancy();
    const int bps = (blocks_per_sm > 0 && blocks_per_sm < occ) ? blocks_per_sm : occ;
    conc_apply_kernel<<<num_sms * bps, 256, 0, s>>>(g, ups, 0, eo, dyn);
    if (g.hub_ops) hub_ops_kernel<<<num_sms, kHubThreads, 0, s>>>(g);
}

// ---------------------------------------------------------------------------
// compaction of edited rows
// ---------------------------------------------------------------------------

__global__ void dirty_list_kernel(Dev g, uint32_t* list, uint32_t* count) {
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nw = (g.n + 31) / 32;
    uint32_t bits = 0;
    if (w < nw) {
        bits = g.dirty[w];
        if (bits) g.dirty[w] = 0;
    }
    list_bits(w, bits, list, count);
}

void launch_dirty_list(const Dev& g, uint32_t* list, uint32_t* count, cudaStream_t s) {
    const uint32_t nw = (g.n + 31) / 32;
    dirty_list_kernel<<<(nw + 255) / 256, 256, 0, s>>>(g, list, count);
}

// Warp per edited row: stable in-place compaction of [rp, rp + hw), INV tail,
// hw = live count.
// Under exact selection a tombstone (id | TOMB) is a hole too, and the live
// entries of the base run, which stay in front and in order, form the new run.
// With `merge` (exact selection), a compacted row of at most kMergeMax live
// entries is also sorted into one base run (warp-wide bitonic sort in shared
// memory), so its later searches stay 32-ary instead of scanning a growing
// unsorted tail; and a row whose tail outgrows an eighth of it is compacted
// even with few holes.
constexpr uint32_t kMergeMax = 1024;

// Ascending bitonic sort of buf[0, m), m a power of two: only as many slots as
// the row fills. (Sorting kMergeMax slots for every row made 55 rounds over 32
// slots per lane of a row of twenty entries, most of the 114 us that an epoch's
// compaction took on a Chung-Lu graph of 300,007 vertices.)
__device__ __forceinline__ void warp_sort_row(uint32_t* buf, uint32_t m, uint32_t lane) {
    for (uint32_t k = 2; k <= m; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = lane; i < m; i += 32) {
                const uint32_t p = i ^ j;
                if (p > i) {
                    const uint32_t a = buf[i], b = buf[p];
                    if ((a > b) == ((i & k) == 0)) {
                        buf[i] = b;
                        buf[p] = a;
                    }
                }
            }
            __syncwarp();
        }
}

// A lane decides about a row of its own, so the words of 32 rows arrive in one
// round; the warp then compacts, one after another, those that need it. (A warp
// per row spent two round trips on each row it left alone: 16 us for the 50,000
// rows of an epoch of 32,768 updates on a mesh, 67 us for 262,144 on a power-law
// graph. With it the epochs became 8 and 60 us shorter.) One thread takes the
// overflow count for the drain that follows; nothing appends to the buffer meanwhile.
__global__ void __launch_bounds__(256) compact_kernel(Dev g, const uint32_t* __restrict__ list,
                                                      const uint32_t* __restrict__ count, int force, int merge,
                                                      uint32_t* drain_n) {
    extern __shared__ uint32_t sort_buf[];  // kMergeMax words per warp, only with `merge`
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t lane = lane_id();
    const uint32_t cnt = *count;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const uint32_t c = *g.ovf_count;
        if (c) *g.ovf_count = 0;
        *drain_n = c < OVF_CAP ? c : OVF_CAP;
    }
    merge = merge && g.blen;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    // Where every row is compacted, lane i of warp w takes entry w + i * warps: the
    // list ascends, and where low ids are the hubs a warp with consecutive entries
    // compacted several of the longest rows, one after another (R-MAT, 262,144
    // vertices: 328 us, 160 this way). Else few rows are, the words decided on are
    // most of the time, and consecutive entries share their sectors (power-law
    // epochs of 262,144 updates: 14 us against 18); as many per warp as leave every
    // warp something to do.
    const bool every = force || !g.live;
    const uint32_t each = every || cnt >= 32 * warps ? 32u : (cnt + warps - 1) / warps;
    const uint64_t apart = every ? warps : 1u;
    for (uint64_t k0 = every ? warp : warp * each; k0 < cnt; k0 += (uint64_t)warps * each) {
        uint32_t row = 0, row_hw = 0, row_run = 0;
        uint64_t row_s = 0;
        bool todo = false;
        const uint64_t k = k0 + lane * apart;
        if (lane < each && k < cnt) {
            row = list[k];
            row_s = g.rp[row];
            row_hw = row_len(g, row);
            row_run = g.blen ? g.blen[row] : 0u;
            // Lazy mode: a row whose holes fill at most a quarter of its extent stays
            // as it is (every reader skips INV slots and tombstones); it is compacted later.
            const uint32_t run = merge ? min(row_run, row_hw) : 0u;
            const bool long_tail = merge && row_hw - run > max(32u, row_hw >> 3);
            const uint32_t holes = g.live ? row_holes(g, row, g.hw[row]) : 0u;
            todo = every || 4u * holes > row_hw || long_tail;
            if (!todo && (holes || (merge && run < row_hw)))  // still a candidate (holes, or a tail to merge)
                atomicOr(g.dirty + (row >> 5), 1u << (row & 31));
        }
        for (uint32_t left = __ballot_sync(FULL, todo); left; left &= left - 1) {
            const int src = __ffs(left) - 1;
            const uint32_t x = __shfl_sync(FULL, row, src), hwx = __shfl_sync(FULL, row_hw, src);
            const uint64_t s = __shfl_sync(FULL, (unsigned long long)row_s, src);
            const uint64_t e = s + hwx;
            const uint64_t run_end = s + __shfl_sync(FULL, row_run, src);
            uint64_t w = s, run_live = 0;
            for (uint64_t c = s & ~3ull; c < e; c += 128) {
                const uint64_t i = c + 4ull * lane;
                uint4 q = make_uint4(INV, INV, INV, INV);
                if (i < e) q = ld_cg4(g.col + i);
                uint32_t vals[4] = {q.x, q.y, q.z, q.w};
                uint32_t m = 0, mr = 0;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const bool live = g.blen ? (vals[j] & TOMB) == 0 : vals[j] != INV;
                    if (i + j >= s && i + j < e && live) {
                        m |= 1u << j;
                        if (i + j < run_end) mr |= 1u << j;
                    }
                }
                run_live += __reduce_add_sync(FULL, (uint32_t)__popc(mr));
                uint32_t total = 0;
                const uint32_t pre = warp_excl_scan(__popc(m), total);
                __syncwarp();
                uint64_t dst = w + pre;
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (m & (1u << j)) {
                        if (dst != i + j) g.col[dst] = vals[j];
                        dst++;
                    }
                w += total;
                __syncwarp();
            }
            for (uint64_t j = w + lane; j < e; j += 32) g.col[j] = INV;
            const uint32_t live = (uint32_t)(w - s);
            if (merge && live > run_live && live <= kMergeMax) {  // tail entries behind the run: one sorted run
                __syncwarp();
                uint32_t* buf = sort_buf + ((threadIdx.x >> 5) & 7) * kMergeMax;
                const uint32_t m = live < 2 ? live : 1u << (32 - __clz(live - 1));
                for (uint32_t i = lane; i < m; i += 32) buf[i] = i < live ? g.col[s + i] : INV;
                __syncwarp();
                warp_sort_row(buf, m, lane);
                for (uint32_t i = lane; i < live; i += 32) g.col[s + i] = buf[i];
                run_live = live;
            }
            if (lane == 0) {
                g.hw[x] = live;
                if (g.live) g.live[x] = live;
                if (g.blen) g.blen[x] = (uint32_t)run_live;
            }
            __syncwarp();
        }
    }
}

void launch_compact(const Dev& g, const uint32_t* list, const uint32_t* count, uint32_t max_rows, bool force,
                    cudaStream_t s, bool merge, uint32_t* drain_n) {
    uint32_t blocks = (max_rows + 7) / 8;
    if (blocks > 148 * 16) blocks = 148 * 16;
    const size_t smem = merge && g.blen ? 8 * kMergeMax * sizeof(uint32_t) : 0;  // 32 KiB: under the 48 KiB default
    compact_kernel<<<blocks, 256, smem, s>>>(g, list, count, force ? 1 : 0, (merge && g.blen) ? 1 : 0,
                                         drain_n);
}

// ---------------------------------------------------------------------------
// overflow drain (streamgc.cu:967-995, epoch_maintenance.cu:66-87)
// ---------------------------------------------------------------------------

// Re-insert without re-appending: first INV or equal slot; none -> failure.
// Unordered drains under exact selection look in the sorted base run first.
__device__ __forceinline__ bool warp_drain_insert(const Dev& g, uint32_t x, uint32_t nbr, bool ordered) {
    const uint64_t s = g.rp[x], e = g.rp[x + 1];
    uint64_t from = s;
    if (!ordered && g.blen) {
        const uint32_t bl = ld_cg(g.blen + x);
        if (bl && warp_run_add(g, x, nbr, s, bl) >= 0) return true;
        from = s + bl;
    }
    for (;;) {
        uint64_t p = 0;
        uint32_t v = 0;
        if (!warp_find(g.col, from, e, [nbr](uint32_t t) { return t == INV || t == nbr; }, p, v)) return false;
        if (v == nbr) return true;
        uint32_t old = 0;
        if (lane_id() == 0) {
            old = atomicCAS(g.col + p, INV, nbr);
            if (old == INV) {
                extend_row(g, x, (uint32_t)(p - s));
                mark_dirty(g, x);
            }
        }
        old = __shfl_sync(FULL, old, 0);
        if (old == INV || old == nbr) return true;
        from = p + 1;
    }
}

__global__ void drain_kernel(Dev g, const uint32_t* __restrict__ drain_n, int ordered, unsigned long long* failed) {
    const uint32_t cnt = *drain_n;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t step = ordered ? 1 : warps;
    if (ordered && w0 != 0) return;
    for (uint32_t k = w0; k < cnt; k += step) {
        const OverflowEdge oe = g.ovf[k];
        const bool ok = warp_drain_insert(g, oe.local_vertex_idx, oe.neighbor_global, ordered != 0);
        if (!ok && lane_id() == 0) {
            if (failed) atomicAdd(failed, 1ull);
            flag_asym(g, oe.local_vertex_idx);
            g.gctl[graph_of(g, oe.local_vertex_idx)].dropped = 1u;
        }
    }
}
void launch_drain(const Dev& g, const uint32_t* drain_n, bool ordered, unsigned long long* failed, cudaStream_t s) {
    if (ordered) drain_kernel<<<1, 32, 0, s>>>(g, drain_n, 1, failed);
    else drain_kernel<<<148 * 4, 256, 0, s>>>(g, drain_n, 0, failed);
}

// ---------------------------------------------------------------------------
// snapshot / query / colors
// ---------------------------------------------------------------------------

__global__ void snapshot_kernel(Dev g, uint16_t* snap) {
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < g.n; x += gridDim.x * blockDim.x)
        snap[x] = color_of(g.st[x]);
}
// Incremental snapshot into the back half, which was last written two
// snapshots ago: the colors of the vertices noted since then (`chg`, this
// epoch's, and `prev`, the epoch before) are copied from the state words;
// then this epoch's marks become `prev` and `chg` starts empty.
__global__ void snapshot_changes_kernel(Dev g, uint32_t* __restrict__ prev, uint16_t* __restrict__ snap) {
    const uint32_t nw = (g.n + 31) / 32;
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += gridDim.x * blockDim.x) {
        const uint32_t cur = g.chg[w], old = prev[w];
        if (cur | old) {
            prev[w] = cur;
            if (cur) g.chg[w] = 0;
        }
        uint32_t bits = cur | old;
        while (bits) {
            const uint32_t x = w * 32 + (__ffs(bits) - 1);
            bits &= bits - 1;
            snap[x] = color_of(g.st[x]);
        }
    }
}
void launch_snapshot_changes(const Dev& g, uint32_t* prev, uint16_t* snap, cudaStream_t s) {
    const uint32_t nw = (g.n + 31) / 32;
    uint32_t blk = (nw + 255) / 256;
    if (blk > 148 * 8) blk = 148 * 8;
    snapshot_changes_kernel<<<blk, 256, 0, s>>>(g, prev, snap);
}

void launch_snapshot(const Dev& g, uint16_t* snap, cudaStream_t s) {
    snapshot_kernel<<<(g.n + 255) / 256 < 148 * 16 ? (g.n + 255) / 256 : 148 * 16, 256, 0, s>>>(g, snap);
}
void launch_colors(const Dev& g, uint16_t* out, cudaStream_t s) { launch_snapshot(g, out, s); }

__global__ void query_kernel(const uint16_t* __restrict__ snap, uint32_t n, const uint32_t* __restrict__ v,
                             uint16_t* __restrict__ out, uint32_t k) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < k) {
        const uint32_t x = v[i];
        out[i] = x < n ? snap[x] : 0;
    }
}
void launch_query(const uint16_t* snap, uint32_t n, const uint32_t* v, uint16_t* out, uint32_t k, cudaStream_t s) {
    if (k) query_kernel<<<(k + 255) / 256, 256, 0, s>>>(snap, n, v, out, k);
}

// ---------------------------------------------------------------------------
// degree-balanced sweeps and the device-driven repair loop
// ---------------------------------------------------------------------------
//
// A repair is a loop of sweeps whose state lives in the RepairCtl block on the
// device: repair_begin starts it, each sweep reads its index and its vertex set
// (every vertex, or the worklist b.wl) from there, and repair_step decides
// whether another sweep runs. One kernel runs the loop (repair_fused_kernel);
// sweeps over many vertices, and timed ones, run pass by pass as kernels of their
// own, between which the host or a CUDA-graph while-node reads the decision.

// Worklists short enough for a few blocks (see the one-kernel repair).
constexpr uint32_t kTailBlocks = 16, kTailList = 2048, kTailItems = 768;

// A warp's place in a pass over a list by the first `nb` blocks: neighboring warps
// of the list sit on different SMs. A list shorter than the grid then occupies
// every SM a little instead of the first few fully: loading a Chung-Lu graph of
// 300,007 vertices took 4.73 ms with consecutive warps in one block and 4.14 this
// way, epochs on a mesh of 131,072 vertices became 5 us shorter. (The reference
// rules' first sweep, which visits every vertex in order, lost 1 % with it.)
__device__ __forceinline__ uint32_t spread_warp(uint32_t nb) { return (threadIdx.x >> 5) * nb + blockIdx.x; }

// list_mode of the per-vertex passes: 0 every vertex, 1 b.wl, 2 as RepairCtl says.
__device__ __forceinline__ bool use_list(const SweepBufs& b, int list_mode) {
    return list_mode == 2 ? ld_cg(&b.rc->list) != 0 : list_mode == 1;
}

// Warp-collective: vertex x's k work items (k = 0: none).
__device__ __forceinline__ void append_items(const Dev& g, const SweepBufs& b, uint32_t x, uint32_t k) {
    uint32_t total = 0;
    const uint32_t off = warp_excl_scan(k, total);
    uint32_t wbase = 0;
    if (lane_id() == 0 && total) wbase = atomicAdd(b.item_count, total);
    wbase = __shfl_sync(FULL, wbase, 0);
    if (wbase + off + k > b.item_cap) {
        if (k) atomicOr(g.err, ERR_LIST_OVERFLOW);
        return;
    }
    for (uint32_t j = 0; j < k; j++) b.items[wbase + off + j] = (unsigned long long)x | ((unsigned long long)j << 32);
}

__device__ __forceinline__ void build_items(const Dev& g, const SweepBufs& b, int list_mode) {
    const bool list = use_list(b, list_mode);
    const uint32_t lim = list ? *b.wl_count : g.n;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < lim; base += stride) {  // warp-uniform trip count
        const uint32_t t = base + threadIdx.x;
        uint32_t k = 0, x = 0;
        if (t < lim) {
            x = list ? b.wl[t] : t;
            const uint32_t len = row_len(g, x);
            if (len > SWEEP_TINY) k = (len + b.tile - 1) / b.tile;
        }
        append_items(g, b, x, k);
    }
}
__global__ void build_items_kernel(Dev g, SweepBufs b, int list_mode) { build_items(g, b, list_mode); }
void launch_build_items(const Dev& g, const SweepBufs& b, int list_mode, int num_sms, cudaStream_t s) {
    cudaMemsetAsync(b.item_count, 0, sizeof(uint32_t), s);
    uint32_t blocks = (g.n + 255) / 256;
    if (list_mode != 0 && blocks > (uint32_t)num_sms * 8) blocks = num_sms * 8;
    build_items_kernel<<<blocks ? blocks : 1, 256, 0, s>>>(g, b, list_mode);
}

// Ordered-pair hash for the symmetry checksum: the sum over all entries x->y
// of H(x,y) - H(y,x) is 0 when every entry has its mirror (and otherwise is 0
// only with probability ~2^-64).
__device__ __forceinline__ unsigned long long pair_hash(uint32_t x, uint32_t y) {
    const unsigned long long z = (((unsigned long long)x << 32) | y) * 0x9E3779B97F4A7C15ull;
    return z ^ (z >> 29);
}
__device__ __forceinline__ unsigned long long sym_term(uint32_t x, uint32_t y) {
    return pair_hash(x, y) - pair_hash(y, x);
}

// The bounds of item `it` (row x, chunk j) in slot space.
__device__ __forceinline__ void item_bounds(const Dev& g, const SweepBufs& b, unsigned long long it, uint32_t& x,
                                            uint64_t& s, uint64_t& e) {
    x = (uint32_t)it;
    const uint32_t j = (uint32_t)(it >> 32);
    const uint64_t rs = g.rp[x];
    s = rs + (uint64_t)j * b.tile;
    const uint64_t re = rs + row_len(g, x);
    e = s + b.tile < re ? s + b.tile : re;
}

// Warp per item: up to b.tile live slots of one row. State words and conflict
// flags are read with plain loads throughout the sweep's passes: in the
// one-kernel repair they change between passes. Each lane keeps two
// 16-byte slot loads and their eight state gathers in flight per round.
// SYM: accumulate the mirror checksum of rows whose graph wants it. PUSH
// (independent-set rule): a same-colored neighbor that loses to x (lower
// priority) is marked for the next sweep, which decides it from its own row.
template <bool SYM, bool PUSH>
__device__ __forceinline__ void sweep_items_body(const Dev& g, const SweepBufs& b, uint32_t nb) {
    const uint32_t warps = (nb * blockDim.x) >> 5;
    const uint32_t lane = lane_id();
    const uint32_t cnt = *b.item_count;
    for (uint32_t k = spread_warp(nb); k < cnt; k += warps) {
        uint32_t x;
        uint64_t s, e;
        item_bounds(g, b, b.items[k], x, s, e);
        GraphCtl* gc = SYM ? &g.gctl[graph_of(g, x)] : nullptr;
        const bool symx = SYM && gc->full && ld_cg(&gc->asym);
        const uint32_t myc = color_of(g.st[x]);
        const uint32_t mydeg = (g.abl & ABL_LIVE_DEG) ? row_len(g, x) : __ldg(g.deg + x);
        uint32_t lo = 0, hi = 0;
        unsigned long long sym = 0;
        bool conf = false;
        for (uint64_t c = s & ~3ull; c < e; c += 256) {
            const uint64_t i0 = c + 4ull * lane, i1 = i0 + 128;
            uint4 q0 = make_uint4(INV, INV, INV, INV), q1 = q0;
            if (i0 < e) q0 = __ldg(reinterpret_cast<const uint4*>(g.col + i0));
            if (i1 < e) q1 = __ldg(reinterpret_cast<const uint4*>(g.col + i1));
            uint32_t v[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
            uint32_t nc[8];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                const uint64_t p = (t < 4 ? i0 : i1) + (t & 3);
                const bool in = p >= s && p < e && v[t] < g.n;
                v[t] = in ? v[t] : INV;
                nc[t] = in ? color_of(g.st[v[t]]) : 0u;
            }
#pragma unroll
            for (int t = 0; t < 8; t++) {
                add_color_bit(nc[t], lo, hi);
                if (nc[t] == myc && myc != 0) {
                    if (PUSH) {
                        if (prio_less(mydeg, x, __ldg(g.deg + v[t]), v[t])) conf = true;
                        else if (v[t] != x) atomicOr(b.wmark + (v[t] >> 5), 1u << (v[t] & 31));
                    } else if (!conf) {
                        conf = prio_less(mydeg, x, __ldg(g.deg + v[t]), v[t]);
                    }
                }
                if (SYM && symx && v[t] != INV && v[t] != x) sym += sym_term(x, v[t]);
            }
        }
        lo = __reduce_or_sync(FULL, lo);
        hi = __reduce_or_sync(FULL, hi);
        const bool anyc = __any_sync(FULL, conf);
        if (SYM)
            for (int off = 16; off > 0; off >>= 1) sym += __shfl_xor_sync(FULL, sym, off);
        if (lane == 0) {
            const unsigned long long m = ((unsigned long long)hi << 32) | lo;
            if (m) atomicOr(b.acc_bm + x, m);
            if (anyc) atomicOr(b.acc_fl + x, 1u);
            if (SYM && sym) atomicAdd(&gc->sym, sym);
        }
    }
}

// sym_mode 0: no checksum; 2: the first sweep of a repair accumulates it for
// the graphs of this repair that visit every vertex with asym set (RepairCtl).
__device__ __forceinline__ bool want_sym(const SweepBufs& b, int sym_mode) {
    return sym_mode == 2 && ld_cg(&b.rc->it) == 0 && ld_cg(&b.rc->any_sym) != 0;
}

__device__ __forceinline__ void sweep_items(const Dev& g, const SweepBufs& b, int mode, int sym_mode, uint32_t nb) {
    const bool sym = want_sym(b, sym_mode);
    const bool push = mode == SWEEP_INDEP;
    if (push) {
        if (sym) sweep_items_body<true, true>(g, b, nb);
        else sweep_items_body<false, true>(g, b, nb);
    } else {
        if (sym) sweep_items_body<true, false>(g, b, nb);
        else sweep_items_body<false, false>(g, b, nb);
    }
}

__global__ void __launch_bounds__(256, 5) sweep_items_kernel(Dev g, SweepBufs b, int mode, int sym_mode) {
    sweep_items(g, b, mode, sym_mode, gridDim.x);
}

// One vertex of the finalize pass (warp-collective: every lane calls it; `valid`
// lanes own a vertex). Short rows are swept here directly; long rows read the
// accumulators. REBUILD writes bitmaps; TIER1 and INDEP also decide.
// A thread sweeps a row of at most SWEEP_TINY live slots in pieces of
// kPiece slots: the vertex ids of slots [s, e) (any alignment; INV where no
// vertex) come from the covering 16-byte chunks, all loaded in one round
// (aligned, inside the slab: chunks past e are not loaded); the caller then
// gathers what it needs for all of them in a second round. One row of up to
// 64 entries costs a thread at most eight dependent round trips, instead of
// two per slot, and 32 rows share a warp.
constexpr uint32_t kPiece = 16;
constexpr int kPieceIds = 4 * ((kPiece + 3) / 4 + 1);
template <bool READONLY>
__device__ __forceinline__ void piece_ids(const Dev& g, uint64_t s, uint64_t e, uint32_t (&y)[kPieceIds]) {
    const uint64_t base = s & ~3ull;
#pragma unroll
    for (int c = 0; c < kPieceIds / 4; c++) {
        const uint64_t i = base + 4ull * c;
        uint4 q = make_uint4(INV, INV, INV, INV);
        if (i < e) q = READONLY ? __ldg(reinterpret_cast<const uint4*>(g.col + i)) : ld_cg4(g.col + i);
        const uint32_t v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const uint64_t p = i + t;
            y[4 * c + t] = (p >= s && p < e && v[t] < g.n) ? v[t] : INV;
        }
    }
}

__device__ __forceinline__ void finalize_one(const Dev& g, const SweepBufs& b, int mode, bool valid, uint32_t x,
                                             bool with_sym, bool push, unsigned long long& live_sum) {
    bool fac_needed = false, pend = false, need = false;
    uint32_t pend_word = 0;
    unsigned long long sym = 0;
    if (valid) {
        if (with_sym) {
            const GraphCtl& gc = g.gctl[graph_of(g, x)];
            with_sym = gc.full && ld_cg(&gc.asym);
        }
        const uint32_t len = row_len(g, x);
        const uint32_t hd = __ldg(g.hdmap + x);
        const uint32_t w = g.st[x];
        const uint16_t myc = color_of(w);
        unsigned long long bits = 0;
        bool conf = false;
        live_sum += len;
        if (len <= SWEEP_TINY) {
            const uint32_t mydeg = (g.abl & ABL_LIVE_DEG) ? len : __ldg(g.deg + x);
            uint32_t lo = 0, hi = 0;
            const uint64_t s0 = g.rp[x], e0 = s0 + len;
            for (uint64_t s = s0; s < e0; s += kPiece) {
                uint32_t y[kPieceIds], sw[kPieceIds];
                piece_ids<true>(g, s, s + kPiece < e0 ? s + kPiece : e0, y);
#pragma unroll
                for (int t = 0; t < kPieceIds; t++) sw[t] = y[t] != INV ? g.st[y[t]] : 0u;
#pragma unroll
                for (int t = 0; t < kPieceIds; t++) {
                    const uint32_t ng = y[t];
                    if (ng == INV) continue;
                    if (with_sym && ng != x) sym += sym_term(x, ng);
                    const uint32_t nc = color_of(sw[t]);
                    add_color_bit(nc, lo, hi);
                    if (nc == myc && nc != 0) {
                        if (prio_less(mydeg, x, __ldg(g.deg + ng), ng)) conf = true;
                        else if (push && ng != x) atomicOr(b.wmark + (ng >> 5), 1u << (ng & 31));
                    }
                }
            }
            bits = ((unsigned long long)hi << 32) | lo;
        } else {
            bits = b.acc_bm[x];
            conf = b.acc_fl[x] != 0;
            if (bits) b.acc_bm[x] = 0;
            if (conf) b.acc_fl[x] = 0;
        }
        if (mode == SWEEP_REBUILD) {
            if (hd == EMPTY) g.bm[x] = bits;
        } else {
            bool decide = false;
            const bool indep = mode == SWEEP_INDEP;
            if (myc == 0) {
                decide = len > (g.live ? row_holes(g, x, g.hw[x]) : 0u);  // has_neighbors: any non-INV slot
            } else if (conf) {
                decide = true;
                if (myc <= 64) bits |= 1ull << (myc - 1);
            }
            if (indep) {
                if (hd == EMPTY) g.bm[x] = bits;
                else if (decide && myc != 0 && myc <= 64) g.bm[x] |= 1ull << (myc - 1);
                if (decide) b.acc_bm[x] = bits;  // the selection step reads and clears it
                b.needf[x] = decide ? 1 : 0;
                need = decide;
            } else if (hd == EMPTY) {
                g.bm[x] = bits;
                if (decide) {
                    if (~bits) {
                        pend = true;
                        pend_word = pack((uint16_t)__ffsll((long long)~bits), (uint16_t)(version_of(w) + 1));
                    } else {
                        fac_needed = true;
                    }
                }
            } else if (decide) {
                if (myc != 0 && myc <= 64) g.bm[x] |= 1ull << (myc - 1);  // own bit on the (unused) bitmap
                fac_needed = true;
            }
        }
    }
    if (sym) atomicAdd(&g.gctl[graph_of(g, x)].sym, sym);  // per lane: the lanes' rows may sit in different graphs
    if (mode == SWEEP_INDEP) {
        const uint32_t ni = warp_append(b.need_count, need);
        if (need) b.need_v[ni] = x;
    }
    if (mode == SWEEP_TIER1) {
        const uint32_t pi = warp_append(b.pend_count, pend);
        if (pend) {
            b.pend_v[pi] = x;
            b.pend_w[pi] = pend_word;
        }
        const uint32_t fi = warp_append(b.fac_count, fac_needed);
        if (fac_needed) b.fac_v[fi] = x;
    }
}

// The live entries and vertices a pass visited, summed per warp over the whole
// pass: one atomic per warp and counter.
__device__ __forceinline__ void count_visits(const SweepBufs& b, unsigned long long live, uint32_t seen) {
    for (int off = 16; off > 0; off >>= 1) live += __shfl_xor_sync(FULL, live, off);
    seen = __reduce_add_sync(FULL, seen);
    if (lane_id() != 0 || !seen) return;
    if (live) {
        atomicAdd(b.live, live);
        atomicAdd(b.swept, live);
    }
    atomicAdd(b.swept + 1, (unsigned long long)seen);
}

// Thread per vertex (every vertex, or the worklist).
__device__ __forceinline__ void sweep_finalize(const Dev& g, const SweepBufs& b, int mode, int list_mode, int sym_mode, uint32_t nb) {
    const bool list = use_list(b, list_mode);
    const uint32_t lim = list ? *b.wl_count : g.n;
    const uint32_t stride = nb * blockDim.x;
    const bool sym = want_sym(b, sym_mode);
    const bool push = mode == SWEEP_INDEP;
    unsigned long long live = 0;
    uint32_t seen = 0;
    for (uint32_t base = spread_warp(nb) * 32; base < lim; base += stride) {  // warp-uniform trip count
        const uint32_t t = base + lane_id();
        const bool valid = t < lim;
        seen += valid;
        finalize_one(g, b, mode, valid, valid ? (list ? b.wl[t] : t) : 0, sym, push, live);
    }
    count_visits(b, live, seen);
}
__global__ void __launch_bounds__(256, 3) sweep_finalize_kernel(Dev g, SweepBufs b, int mode, int list_mode,
                                                             int sym_mode) {
    sweep_finalize(g, b, mode, list_mode, sym_mode, gridDim.x);
}

// Warp per vertex whose new color needs the histogram row or the >64 scan;
// colors read are the start-of-sweep ones (nothing is committed yet).
// (The scratch of the exact selection serves eight warps of a block.)
__device__ __forceinline__ void sweep_fac(const Dev& g, const SweepBufs& b, uint32_t nb) {
    if (threadIdx.x >= 256) return;
    const uint32_t warps = nb * 8;
    const uint32_t cnt = *b.fac_count;
    for (uint32_t k = spread_warp(nb); k < cnt; k += warps) {
        const uint32_t x = b.fac_v[k];
        const uint32_t w = ld_cg(g.st + x);
        const uint16_t c = warp_fac(g, x, g.st);
        if (lane_id() == 0) {
            const uint32_t pi = atomicAdd(b.pend_count, 1u);
            b.pend_v[pi] = x;
            b.pend_w[pi] = pack(c, (uint16_t)(version_of(w) + 1));
        }
        __syncwarp();
    }
}
__global__ void __launch_bounds__(256) sweep_fac_kernel(Dev g, SweepBufs b) { sweep_fac(g, b, gridDim.x); }

// Independent-set selection, step 1: warp per item (chunk) of a conflicted
// row. Sets the row's blocked flag (acc_fl) when a conflicted neighbor in the
// chunk ranks above it; for a histogram-class row whose neighbors take every
// color 1..64 (acc_bm, from the sweep) it also gathers the taken colors 65..2047
// into the row's words of b.hiused. Colors are the start-of-sweep ones.
template <int WARPS>
__device__ __forceinline__ void indep_items(const Dev& g, const SweepBufs& b, uint32_t nb) {
    __shared__ uint32_t s_used[WARPS][64];
    uint32_t* used = s_used[threadIdx.x >> 5];
    const uint32_t warps = (nb * blockDim.x) >> 5;
    const uint32_t lane = lane_id();
    const uint32_t cnt = *b.item_count;
    const uint32_t salt = sweep_salt(ld_cg(&b.rc->it));
    used[lane] = 0;
    used[lane + 32] = 0;
    __syncwarp();
    for (uint32_t k = spread_warp(nb); k < cnt; k += warps) {
        const unsigned long long it = b.items[k];
        uint32_t x;
        uint64_t s, e;
        item_bounds(g, b, it, x, s, e);
        // the row's words in one round trip, before the first is tested
        const uint32_t hd = __ldg(g.hdmap + x), met = ld_cg(b.acc_fl + x);
        const unsigned long long mask = b.acc_bm[x];
        const bool full = hd != EMPTY && g.exact && ~mask == 0ull;
        if (!b.needf[x] || met) continue;  // not conflicted, or another chunk already found it blocked
        const uint32_t base = g.gctl[graph_of(g, x)].base;  // ranks use the graph's own ids
        const unsigned long long rx = sel_rank(x - base, salt);
        bool blocked = false;
        for (uint64_t c = s & ~3ull; c < e; c += 256) {
            const uint64_t i0 = c + 4ull * lane, i1 = i0 + 128;
            uint4 q0 = make_uint4(INV, INV, INV, INV), q1 = q0;
            if (i0 < e) q0 = __ldg(reinterpret_cast<const uint4*>(g.col + i0));
            if (i1 < e) q1 = __ldg(reinterpret_cast<const uint4*>(g.col + i1));
            uint32_t v[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
            uint8_t nf[8];
            uint32_t nc[8];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                const uint64_t p = (t < 4 ? i0 : i1) + (t & 3);
                const bool in = p >= s && p < e && v[t] < g.n && v[t] != x;
                v[t] = in ? v[t] : INV;
                nf[t] = in ? b.needf[v[t]] : (uint8_t)0;
                nc[t] = (in && full) ? color_of(g.st[v[t]]) : 0u;
            }
#pragma unroll
            for (int t = 0; t < 8; t++) {
                if (nf[t] && sel_rank(v[t] - base, salt) > rx) blocked = true;
                if (full && nc[t] > 64 && nc[t] < 2048) atomicOr(&used[nc[t] >> 5], 1u << (nc[t] & 31));
            }
            if (__any_sync(FULL, blocked)) break;  // a blocked row needs nothing more
        }
        blocked = __any_sync(FULL, blocked);
        if (lane == 0 && blocked) atomicOr(b.acc_fl + x, 1u);
        if (full) {
            __syncwarp();
            uint32_t* dst = b.hiused + (uint64_t)hd * 64;
            const uint32_t w0 = used[lane], w1 = used[lane + 32];
            if (w0) atomicOr(dst + lane, w0);
            if (w1) atomicOr(dst + lane + 32, w1);
            used[lane] = 0;
            used[lane + 32] = 0;
            __syncwarp();
        }
    }
}

__global__ void __launch_bounds__(256, 5) indep_items_kernel(Dev g, SweepBufs b) { indep_items<8>(g, b, gridDim.x); }

// Independent-set selection, step 2: thread per conflicted vertex. A row of at
// most SWEEP_TINY slots checks its neighbors here; longer rows read step 1's
// flag. An unblocked vertex takes the first color its neighbors leave free:
// from the sweep's 64-bit mask, else from the gathered 65..2047 set
// (histogram-class rows), else through the warp scan of sweep_fac_kernel
// (bitmap rows whose 64 low colors are all taken). Blocked vertices are marked
// for the next sweep.
__device__ __forceinline__ void indep_decide(const Dev& g, const SweepBufs& b, uint32_t nb) {
    const uint32_t cnt = *b.need_count;
    const uint32_t salt = sweep_salt(ld_cg(&b.rc->it));
    for (uint32_t t = spread_warp(nb) * 32 + lane_id(); t < cnt; t += nb * blockDim.x) {
        const uint32_t x = b.need_v[t];
        const uint32_t len = row_len(g, x);
        bool blocked = false;
        if (len <= SWEEP_TINY) {
            const uint32_t base = g.gctl[graph_of(g, x)].base;  // ranks use the graph's own ids
            const unsigned long long rx = sel_rank(x - base, salt);
            const uint64_t s0 = g.rp[x], e0 = s0 + len;
            for (uint64_t s = s0; s < e0 && !blocked; s += kPiece) {
                uint32_t y[kPieceIds];
                uint8_t nf[kPieceIds];
                piece_ids<true>(g, s, s + kPiece < e0 ? s + kPiece : e0, y);
#pragma unroll
                for (int t = 0; t < kPieceIds; t++) nf[t] = (y[t] != INV && y[t] != x) ? b.needf[y[t]] : 0;
#pragma unroll
                for (int t = 0; t < kPieceIds; t++)
                    if (nf[t] && sel_rank(y[t] - base, salt) > rx) blocked = true;
            }
        } else if (b.acc_fl[x]) {
            blocked = true;
            b.acc_fl[x] = 0;
        }
        if (blocked) atomicOr(b.wmark + (x >> 5), 1u << (x & 31));
        const unsigned long long mask = b.acc_bm[x];
        if (mask) b.acc_bm[x] = 0;
        const uint32_t hd = __ldg(g.hdmap + x);
        const bool full = ~mask == 0ull;
        uint32_t c = 0;
        if (full && hd != EMPTY && g.exact && len > SWEEP_TINY) {
            uint32_t* w = b.hiused + (uint64_t)hd * 64;
            c = 2048;
            for (uint32_t k = 2; k < 64; k++) {
                const uint32_t word = w[k];
                if (word) w[k] = 0;
                const uint32_t freew = ~word & (k == 2 ? ~1u : FULL);  // color 64 is taken (full mask)
                if (c == 2048 && freew) c = k * 32 + __ffs(freew) - 1;
            }
        }
        if (blocked) continue;
        if (!full) {
            c = __ffsll((long long)~mask);
        } else if (c == 0) {  // the scan over colors above 64 needs a warp
            b.fac_v[atomicAdd(b.fac_count, 1u)] = x;
            continue;
        }
        const uint32_t w = g.st[x];
        const uint32_t pi = atomicAdd(b.pend_count, 1u);
        b.pend_v[pi] = x;
        b.pend_w[pi] = pack((uint16_t)c, (uint16_t)(version_of(w) + 1));
    }
}

__global__ void __launch_bounds__(256) indep_decide_kernel(Dev g, SweepBufs b) { indep_decide(g, b, gridDim.x); }

// Writes the chosen colors and clears the recolored vertices' conflict flags.
// Reference rule (TIER1): marks each recolored vertex and, for rows of at most
// SWEEP_TINY slots, its neighbors for the next worklist (longer rows: per item
// in mark_items_kernel). Independent-set rule: ORs the new color into the
// neighbors' bitmaps instead (the next sweep needs no neighbor of a recolored
// vertex: under that rule a recolor creates no conflict).
__device__ __forceinline__ void sweep_commit(const Dev& g, const SweepBufs& b, int mode, uint32_t nb) {
    const uint32_t cnt = *b.pend_count;
    const bool incr = mode == SWEEP_INDEP;
    for (uint32_t k = spread_warp(nb) * 32 + lane_id(); k < cnt; k += nb * blockDim.x) {
        const uint32_t x = b.pend_v[k];
        const uint32_t nw = b.pend_w[k];
        g.st[x] = nw;
        note_color(g, x);
        b.needf[x] = 0;
        atomicOr(b.rbits + (x >> 5), 1u << (x & 31));
        if (!incr) atomicOr(b.wmark + (x >> 5), 1u << (x & 31));
        const uint32_t len = row_len(g, x);
        if (len <= SWEEP_TINY) {
            const uint32_t c = color_of(nw);
            const uint64_t s0 = g.rp[x], e0 = s0 + len;
            for (uint64_t s = s0; s < e0; s += kPiece) {
                uint32_t y[kPieceIds];
                piece_ids<false>(g, s, s + kPiece < e0 ? s + kPiece : e0, y);
#pragma unroll
                for (int t = 0; t < kPieceIds; t++) {
                    if (y[t] == INV) continue;
                    if (!incr) atomicOr(b.wmark + (y[t] >> 5), 1u << (y[t] & 31));
                    else if (c != 0 && c <= 64) atomicOr((unsigned long long*)(g.bm + y[t]), 1ull << (c - 1));
                }
            }
        }
    }
}

__global__ void sweep_commit_kernel(Dev g, SweepBufs b, int mode) { sweep_commit(g, b, mode, gridDim.x); }

// Warp per item of the last sweep whose row was recolored: marks the
// neighbors in the item's slots (reference rule) or ORs the row's new color
// into their bitmaps (independent-set rule).
__device__ __forceinline__ void mark_items(const Dev& g, const SweepBufs& b, uint32_t nb) {
    const uint32_t warps = (nb * blockDim.x) >> 5;
    const uint32_t lane = lane_id();
    const uint32_t cnt = *b.item_count;
    const bool incr = ld_cg(&b.rc->mode) == SWEEP_INDEP;
    for (uint32_t k = spread_warp(nb); k < cnt; k += warps) {
        const unsigned long long it = b.items[k];
        const uint32_t x0 = (uint32_t)it;
        if (!(b.rbits[x0 >> 5] & (1u << (x0 & 31)))) continue;
        uint32_t x;
        uint64_t s, e;
        item_bounds(g, b, it, x, s, e);
        const uint32_t c = color_of(g.st[x]);
        const unsigned long long bit = (c != 0 && c <= 64) ? 1ull << (c - 1) : 0ull;
        if (incr && !bit) continue;
        for (uint64_t p = s + lane; p < e; p += 32) {
            const uint32_t y = g.col[p];
            if (y >= g.n) continue;
            if (incr) atomicOr((unsigned long long*)(g.bm + y), bit);
            else atomicOr(b.wmark + (y >> 5), 1u << (y & 31));
        }
    }
}

__global__ void __launch_bounds__(256) mark_items_kernel(Dev g, SweepBufs b) { mark_items(g, b, gridDim.x); }

// A pass over the `nw` words of a bitmask by the first `nb` blocks: f(w, bits), a
// word per lane and warp-collective, with the words cleared. With many words per
// thread they are read sixteen bytes per lane, and 128 that are all zero skipped
// together: a mask of 65.6 M vertices has 2 M words, most of them zero, which were
// thirty-seven rounds of 55,296 threads. (Epochs of 32,768 updates on a Chung-Lu
// graph of that size: 474 us, 422 with these passes, sixteen-byte clearing and the
// short sweeps left to the whole grid, kTailWords.)
template <class F>
__device__ __forceinline__ void take_words(uint32_t* words, uint32_t nw, uint32_t nb, F f) {
    const uint32_t threads = nb * blockDim.x;
    if (nw <= 4 * threads) {
        for (uint32_t base = spread_warp(nb) * 32; base < nw; base += threads) {
            const uint32_t w = base + lane_id();
            uint32_t bits = 0;
            if (w < nw) {
                bits = words[w];
                if (bits) words[w] = 0;
            }
            f(w, bits);
        }
        return;
    }
    for (uint32_t base = spread_warp(nb) * 128; base < nw; base += 4 * threads) {
        const uint32_t w = base + 4 * lane_id();
        uint4 q = make_uint4(0, 0, 0, 0);
        if (w < nw) q = *reinterpret_cast<const uint4*>(words + w);  // there is room for the last three
        if (!__any_sync(FULL, q.x | q.y | q.z | q.w)) continue;
        if (q.x | q.y | q.z | q.w) *reinterpret_cast<uint4*>(words + w) = make_uint4(0, 0, 0, 0);
        f(w, q.x);
        f(w + 1, q.y);
        f(w + 2, q.z);
        f(w + 3, q.w);
    }
}

// The next worklist: the marked vertices; clears the marks.
__device__ __forceinline__ void collect_marks(const Dev& g, const SweepBufs& b, uint32_t nb) {
    take_words(b.wmark, (g.n + 31) / 32, nb, [&](uint32_t w, uint32_t bits) {
        if (!__any_sync(FULL, bits)) return;
        list_bits(w, bits, b.wl, b.wl_count);
        // the work items they will make (asked for only of a short list: many marks
        // in one word count as too many, and cost no walk over their rows)
        uint32_t k = __popc(bits) > 4 ? 4 * kTailItems + 1 : 0u;
        for (uint32_t r = k ? 0u : bits; r; r &= r - 1) {
            const uint32_t len = row_len(g, w * 32 + (__ffs(r) - 1));
            if (len > SWEEP_TINY) k += (len + b.tile - 1) / b.tile;
        }
        k = __reduce_add_sync(FULL, k);
        if (k && lane_id() == 0) atomicAdd(b.next_items, k);
    });
}
// (and the recolored bits, which nothing reads any more)
__global__ void collect_marks_kernel(Dev g, SweepBufs b) {
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w < (g.n + 31) / 32 && b.rbits[w]) b.rbits[w] = 0;
    collect_marks(g, b, gridDim.x);
}

void launch_next_worklist(const Dev& g, const SweepBufs& b, int num_sms, cudaStream_t s) {
    mark_items_kernel<<<num_sms * 8, 256, 0, s>>>(g, b);
    cudaMemsetAsync(b.wl_count, 0, sizeof(uint32_t), s);
    const uint32_t nw = (g.n + 31) / 32;
    collect_marks_kernel<<<(nw + 255) / 256, 256, 0, s>>>(g, b);
}

void launch_sweep(const Dev& g, const SweepBufs& b, SweepMode mode, int list_mode, int sym_mode, int num_sms,
                  cudaStream_t s, cudaEvent_t* phase) {
    if (mode != SWEEP_REBUILD) {
        cudaMemsetAsync(b.pend_count, 0, sizeof(uint32_t), s);
        cudaMemsetAsync(b.fac_count, 0, sizeof(uint32_t), s);
        cudaMemsetAsync(b.need_count, 0, sizeof(uint32_t), s);
    }
    sweep_items_kernel<<<num_sms * 5, 256, 0, s>>>(g, b, (int)mode, sym_mode);  // one wave: 5 blocks per SM
    if (phase) cudaEventRecord(phase[0], s);
    uint32_t fblocks = (g.n + 255) / 256;
    if (list_mode != 0 && fblocks > (uint32_t)num_sms * 3) fblocks = num_sms * 3;  // one wave: 3 blocks per SM
    sweep_finalize_kernel<<<fblocks ? fblocks : 1, 256, 0, s>>>(g, b, (int)mode, list_mode, sym_mode);
    if (phase) cudaEventRecord(phase[1], s);
    if (mode == SWEEP_INDEP) {
        indep_items_kernel<<<num_sms * 5, 256, 0, s>>>(g, b);
        indep_decide_kernel<<<num_sms * 2, 256, 0, s>>>(g, b);
    }
    if (mode != SWEEP_REBUILD) {
        sweep_fac_kernel<<<num_sms * 2, 256, 0, s>>>(g, b);
        sweep_commit_kernel<<<num_sms * 2, 256, 0, s>>>(g, b, (int)mode);
    }
}

// Starts a repair. Reference rule (TIER1, one graph): the first sweep visits
// every vertex. Independent-set rule: per graph, the first worklist is every
// vertex of the graph when it must be repaired in full (its last repair did
// not end proper, its rows may miss mirror entries, or the host forces it),
// else the vertices its updates touched since the last repair: every new
// conflict then has a touched endpoint. One block.
__device__ __forceinline__ void repair_begin(const Dev& g, const SweepBufs& b) {
    RepairCtl& rc = *b.rc;
    const bool indep = rc.mode == SWEEP_INDEP;
    uint32_t any_sym = 0, any_incr = 0;
    for (uint32_t k = threadIdx.x; k < b.G; k += blockDim.x) {
        GraphCtl& c = g.gctl[k];
        const bool full = !indep || !c.clean || c.asym || c.force || rc.force_all || !g.touched;
        c.full = full ? 1u : 0u;
        c.force = 0;
        c.sym = 0;
        if (full && c.asym) any_sym = 1;
        if (!full) any_incr = 1;
    }
    any_sym = __syncthreads_or(any_sym);
    any_incr = __syncthreads_or(any_incr);
    if (threadIdx.x == 0) {
        rc.any_sym = any_sym;
        rc.incr = any_incr;
        rc.list = indep ? 1u : 0u;
        rc.it = 0;
        rc.cont = 1;
        rc.done = 0;
        rc.fault = 0;
        rc.need = 0;
        rc.next = 0;
        rc.prev = 0xFFFFFFFFu;
        rc.plateau = 0;
        rc.sym = 0;
        rc.live = 0;
        *b.live = 0;
        *b.wl_count = 0;
        b.swept[0] = 0;
        b.swept[1] = 0;
    }
}

__global__ void repair_begin_kernel(Dev g, SweepBufs b) { repair_begin(g, b); }

// First worklist of an independent-set repair: every vertex of the graphs
// repaired in full, the touched vertices of the others; clears the touched
// marks; the list's length goes to *count. Thread per 32-vertex word.
__device__ __forceinline__ void seed_worklist(const Dev& g, const SweepBufs& b, uint32_t nb, uint32_t* count) {
    const uint32_t nw = (g.n + 31) / 32;
    if (!g.gidw && !g.gctl[0].full) {  // one graph, its touched vertices
        take_words(g.touched, nw, nb, [&](uint32_t w, uint32_t bits) { list_bits(w, bits, b.wl, count); });
        return;
    }
    for (uint32_t base = spread_warp(nb) * 32; base < nw; base += nb * blockDim.x) {
        const uint32_t w = base + lane_id();
        uint32_t bits = 0;
        if (w < nw) {
            const uint32_t t = g.touched[w];
            if (t) g.touched[w] = 0;
            if (g.gctl[g.gidw ? g.gidw[w] : 0u].full) {
                const uint32_t left = g.n - w * 32;
                bits = left >= 32 ? FULL : (1u << left) - 1u;
            } else {
                bits = t;
            }
        }
        list_bits(w, bits, b.wl, count);
    }
}
__global__ void seed_worklist_kernel(Dev g, SweepBufs b) { seed_worklist(g, b, gridDim.x, b.wl_count); }

// After each sweep: reads the counts, decides whether another sweep runs,
// advances the index. Reference rule (TIER1): stop at 0 conflicts, after 3
// equal counts, or at max_sweeps (streamgc.cu:1317-1393); later sweeps visit
// the worklist only when the first found the rows mirror-complete.
// Independent-set rule: stop when the next worklist is empty. After the first
// sweep a graph whose checksum came out 0 is known mirror-complete; when the
// loop ends every graph records whether it ended proper. `cond` (graph mode):
// the while-node's handle receives the decision. One block.
__device__ __forceinline__ void repair_step(const Dev& g, const SweepBufs& b) {
    RepairCtl& rc = *b.rc;
    __shared__ uint32_t s_stop;
    const bool indep = rc.mode == SWEEP_INDEP;
    uint32_t sym_any = 0;
    if (rc.it == 0) {
        for (uint32_t k = threadIdx.x; k < b.G; k += blockDim.x) {
            GraphCtl& c = g.gctl[k];
            if (c.full && c.asym) {
                if (c.sym == 0) c.asym = 0;  // found mirror-complete
                else sym_any = 1;
            }
        }
    }
    sym_any = __syncthreads_or(sym_any);
    if (threadIdx.x == 0) {
        const uint32_t count = indep ? *b.need_count : *b.pend_count;
        const uint32_t next = *b.wl_count;
        if (rc.it == 0) {
            rc.sym = sym_any ? (g.gctl[0].sym ? g.gctl[0].sym : 1ull) : 0ull;
            rc.live = *b.live;
        }
        rc.need = count;
        rc.next = next;
        bool done, stop;
        if (indep) {
            done = next == 0;
            stop = done;
        } else {
            done = count == 0;
            stop = done;
            if (!done) {
                if (count == rc.prev) stop = ++rc.plateau >= 3;
                else rc.plateau = 0;
            }
            rc.prev = count;
        }
        rc.done = done ? 1u : 0u;
        rc.list = (indep || rc.sym == 0) ? 1u : 0u;
        rc.swept[0] = b.swept[0];
        rc.swept[1] = b.swept[1];
        rc.it += 1;
        rc.cont = (!stop && rc.it < rc.max_sweeps) ? 1u : 0u;
        s_stop = rc.cont ? 0u : 1u;
    }
    __syncthreads();
    if (s_stop) {
        const bool done = rc.done != 0;
        for (uint32_t k = threadIdx.x; k < b.G; k += blockDim.x) {
            GraphCtl& c = g.gctl[k];
            c.clean = (done && c.sym == 0) ? 1u : 0u;
            c.t2 = c.sym != 0 ? 1u : 0u;
        }
        __syncthreads();
        if (!done) {  // the graphs of the vertices still to visit hold the unresolved conflicts
            const uint32_t nx = *b.wl_count;
            for (uint32_t i = threadIdx.x; i < nx; i += blockDim.x) g.gctl[graph_of(g, b.wl[i])].t2 = 1;
        }
    }
}

__global__ void repair_step_kernel(Dev g, SweepBufs b, cudaGraphConditionalHandle cond, int has_cond) {
    repair_step(g, b);
    if (has_cond && threadIdx.x == 0) cudaGraphSetConditional(cond, b.rc->cont);
}

void launch_repair_begin(const Dev& g, const SweepBufs& b, SweepMode mode, int num_sms, cudaStream_t s) {
    repair_begin_kernel<<<1, 256, 0, s>>>(g, b);
    if (mode == SWEEP_INDEP && g.touched) {
        const uint32_t nw = (g.n + 31) / 32;
        seed_worklist_kernel<<<(nw + 255) / 256, 256, 0, s>>>(g, b);
    }
    (void)num_sms;
}

// ---------------------------------------------------------------------------
// the repair as one kernel
// ---------------------------------------------------------------------------
//
// Most repairs are short: an epoch's worklist of some ten thousand vertices, two
// to ten sweeps of a few microseconds of work each. As fourteen launches per
// sweep, and a host or while-node round trip, a sweep took 55 us (epochs of 4,096
// updates on a mesh of 24,001 vertices: 245 us, now 142). One cooperative launch
// runs the same passes with a barrier across the grid (2 us) between them and
// leaves out the passes that have nothing to do; a short worklist is left to
// kTailBlocks blocks, whose barrier costs less.
//   kTailList, kTailItems: what sixteen blocks finish in a few rounds of their
// warps. Sweeps of a power-law graph of 2 M vertices there: 40 us against 49 on
// the whole grid.
//   kTailWords: the marks that sixteen blocks read in four rounds (3.1 M vertices).
// They read all of them every sweep; for 65.6 M vertices that were eighty rounds.
//   kFusedMax: a sweep over many vertices, where the item passes' 40 warps per SM
// pay and a launch costs little, is left to the kernels above.
//   kFusedThreads: a cooperative launch starts only when all its blocks have room,
// so a block takes no more than half of an SM's registers (384 threads of 80) and
// two handles' repairs, or one and another handle's stream-order apply, run side
// by side. With 768 threads a publish of 157 us waited up to 7.7 ms for such an
// apply, and two loads of a Chung-Lu graph of 300,007 vertices at once took 6.3 ms
// each, now 4.7. Alone, sweeps of that load pay 2 % for the halved blocks.
constexpr uint32_t kFusedThreads = 384;
constexpr uint32_t kTailWords = 4 * 4 * kTailBlocks * kFusedThreads;

// A thread per vertex and a warp per work item of the rows when full is as much as
// a sweep can use; never a block on every SM (spare_sms), and a few at least.
uint32_t repair_blocks(uint64_t vertices, uint64_t items, int num_sms) {
    const uint64_t want = std::max<uint64_t>((vertices + kFusedThreads - 1) / kFusedThreads,
                                             (items + kFusedThreads / 32 - 1) / (kFusedThreads / 32));
    return (uint32_t)std::min<uint64_t>(std::max<uint64_t>(want, kTailBlocks), spare_sms(num_sms));
}

// The first `nb` blocks of the grid meet. A thread's writes before the barrier
// are seen after it by plain loads in all of them. Round by round the arrivals
// only grow by nb, so a round is over when they reach the next multiple. The
// wait is bounded (seconds): false means a block is missing, and the caller
// returns.
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
struct GridSync {
    GridBar* bar;
    uint32_t* err;
    uint32_t nb;
    unsigned long long due = 0, serials = 0;  // thread 0: arrivals and serial sections awaited so far

    __device__ __forceinline__ GridSync(GridBar* p, uint32_t* e) : bar(p), err(e), nb(gridDim.x) {}
    __device__ __forceinline__ bool wait(const unsigned long long* word, unsigned long long target) {
        for (uint32_t polls = 0; ld_acquire(word) < target; polls++) {
            if (polls > 2000u) __nanosleep(200);
            if (polls >= (1u << 25) || *(volatile uint32_t*)&bar->failed) {
                *(volatile uint32_t*)&bar->failed = 1;
                atomicOr(err, ERR_BARRIER);
                return false;
            }
        }
        return true;
    }
    __device__ __forceinline__ void arrive() {
        fence_gpu();
        atomicAdd(&bar->count, 1ull);
        due += nb;
    }
    __device__ __forceinline__ bool operator()() {
        bool ok = true;
        __syncthreads();
        if (threadIdx.x == 0) {
            arrive();
            ok = wait(&bar->count, due);
        }
        return __syncthreads_and(ok);
    }
    // The grid goes on with its first `k` blocks: the others call part() and return.
    // Their last arrivals are awaited at the next barrier of those that stay, so
    // what they still read or write comes before anything after that barrier.
    __device__ __forceinline__ void part() {
        __syncthreads();
        if (threadIdx.x == 0) arrive();
    }
    __device__ __forceinline__ void shrink(uint32_t k) {
        due += nb - k;
        nb = k;
    }
    // The same, where block 0 runs `last` when all have arrived, before any goes on.
    template <class F>
    __device__ __forceinline__ bool serial(F last) {
        bool ok = true;
        __syncthreads();
        if (threadIdx.x == 0) {
            arrive();
            ok = blockIdx.x == 0 ? wait(&bar->count, due) : wait(&bar->gen, ++serials);
        }
        if (!__syncthreads_and(ok)) return false;
        if (blockIdx.x == 0) {
            last();
            __syncthreads();
            if (threadIdx.x == 0) {
                fence_gpu();
                atomicAdd(&bar->gen, 1ull);
            }
        }
        return true;
    }
    // Every block ends here, `ok` false where a barrier gave up on it. The last one
    // makes the words zero for the next launch and, on its thread 0 alone, returns
    // true; `ok` then says whether all blocks met at every barrier.
    __device__ __forceinline__ bool leave(bool& ok) {
        __syncthreads();
        if (threadIdx.x != 0) return false;
        fence_gpu();
        const uint32_t before = atomicAdd(&bar->left, ok ? 1u : 0x10001u);  // blocks, and those given up on above
        if ((before & 0xFFFFu) != gridDim.x - 1) return false;
        fence_gpu();
        ok = ok && before < 0x10000u;
        bar->count = 0;
        bar->gen = 0;
        bar->left = 0;
        bar->failed = 0;
        return true;
    }
};

// First pass of a sweep: work items for the long rows, the short rows whole.
__device__ __forceinline__ void sweep_short(const Dev& g, const SweepBufs& b, int mode, bool list, uint32_t lim,
                                            bool sym, uint32_t nb) {
    unsigned long long live = 0;
    uint32_t seen = 0;
    for (uint32_t base = spread_warp(nb) * 32; base < lim; base += nb * blockDim.x) {
        const uint32_t t = base + lane_id();
        uint32_t k = 0, x = 0;
        if (t < lim) {
            x = list ? b.wl[t] : t;
            const uint32_t len = row_len(g, x);
            if (len > SWEEP_TINY) k = (len + b.tile - 1) / b.tile;
        }
        append_items(g, b, x, k);
        const bool valid = t < lim && k == 0;
        seen += valid;
        finalize_one(g, b, mode, valid, x, sym, mode == SWEEP_INDEP, live);
    }
    count_visits(b, live, seen);
}
// After the items: the long rows (each at its first item).
__device__ __forceinline__ void sweep_long(const Dev& g, const SweepBufs& b, int mode, uint32_t items, bool sym,
                                           uint32_t nb) {
    unsigned long long live = 0;
    uint32_t seen = 0;
    for (uint32_t base = spread_warp(nb) * 32; base < items; base += nb * blockDim.x) {
        const uint32_t t = base + lane_id();
        const unsigned long long it = t < items ? b.items[t] : ~0ull;
        const bool valid = (it >> 32) == 0;
        seen += valid;
        finalize_one(g, b, mode, valid, (uint32_t)it, sym, mode == SWEEP_INDEP, live);
    }
    count_visits(b, live, seen);
}

// ---------------------------------------------------------------------------
// first-fit coloring of a list, in its order
// ---------------------------------------------------------------------------
//
// A vertex takes the first color in 1..2047 that no neighbor in its row holds
// (2048 when all are held), version 1; colors given earlier in the list count,
// vertices already colored are passed over. One vertex after another, a block on
// each row, was a dependent chain of loads per vertex: 2.2 ms for the core of a
// Chung-Lu graph of 300,007 vertices, 0.77 ms this way. The
// list is taken a window at a time: a block per vertex gathers the colors its
// neighbors hold and which earlier vertices of the window are among them, and
// then one warp colors the window in order from those sets in shared memory.

// place[v]: 1 + v's place in the list (0: not in it).
__global__ void list_places_kernel(const uint32_t* __restrict__ list, uint32_t m, uint32_t* place) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x) place[list[k]] = k + 1;
}

constexpr uint32_t kColorThreads = 512;
__global__ void __launch_bounds__(kColorThreads, 1) color_list_kernel(Dev g, const uint32_t* __restrict__ list,
                                                                      uint32_t m, const uint32_t* __restrict__ place,
                                                                      uint32_t* rows, GridBar* bar, uint32_t* colored) {
    constexpr uint32_t AW = kColorWindow / 32;
    __shared__ uint32_t used[kColorWindow][64];  // blocks gather into used[0], near[0]
    __shared__ uint32_t near[kColorWindow][AW];  // earlier vertices of the window in the row
    GridSync sync(bar, g.err);
    const uint32_t tid = threadIdx.x, lane = lane_id();
    uint32_t done = 0;
    bool ok = true;
    for (uint32_t w0 = 0; ok && w0 < m; w0 += kColorWindow) {
        const uint32_t cnt = m - w0 < kColorWindow ? m - w0 : kColorWindow;
        for (uint32_t i = blockIdx.x; i < cnt; i += gridDim.x) {
            if (tid < 64) used[0][tid] = 0;
            if (tid < AW) near[0][tid] = 0;
            __syncthreads();
            const uint32_t v = list[w0 + i];
            const uint64_t s = g.rp[v], e = s + row_len(g, v);
            for (uint64_t c = s & ~3ull; c < e; c += 4ull * kColorThreads) {
                const uint64_t at = c + 4ull * tid;
                uint4 q = make_uint4(INV, INV, INV, INV);
                if (at < e) q = ld_cg4(g.col + at);
                uint32_t y[4] = {q.x, q.y, q.z, q.w}, w[4];
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    if (!(at + t >= s && at + t < e && y[t] < g.n)) y[t] = INV;
                    w[t] = y[t] != INV ? color_of(g.st[y[t]]) : 2048u;
                }
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    if (w[t] >= 2048) continue;
                    if (w[t]) {
                        atomicOr(&used[0][w[t] >> 5], 1u << (w[t] & 31));
                    } else {
                        const uint32_t p = place[y[t]] - 1 - w0;  // not in the list, or before the window: wraps
                        if (p < i) atomicOr(&near[0][p >> 5], 1u << (p & 31));
                    }
                }
            }
            __syncthreads();
            if (tid == 0 && color_of(g.st[v]) != 0) used[0][0] |= 1u;  // color 0 is no candidate: passed over
            __syncthreads();
            if (tid < 64) rows[i * 64 + tid] = used[0][tid];
            if (tid < AW) rows[kColorWindow * 64 + i * AW + tid] = near[0][tid];
        }
        if (!(ok = sync())) break;
        if (blockIdx.x == 0) {
            for (uint32_t k = tid; k < cnt * 64; k += kColorThreads) used[k >> 6][k & 63] = rows[k];
            for (uint32_t k = tid; k < cnt * AW; k += kColorThreads) near[k / AW][k % AW] = rows[kColorWindow * 64 + k];
            __syncthreads();
            for (uint32_t i = 0; tid < 32 && i < cnt; i++) {
                const uint32_t f0 = ~used[i][lane], f1 = ~used[i][lane + 32];
                const uint32_t skip = used[i][0] & 1u;
                const uint32_t b0 = __ballot_sync(FULL, (lane ? f0 : f0 & ~1u) != 0), b1 = __ballot_sync(FULL, f1 != 0);
                uint32_t c = 2048;
                if (b0) {
                    const uint32_t src = __ffs(b0) - 1;
                    c = 32 * src + __ffs(~used[i][src] & (src ? FULL : ~1u)) - 1;
                } else if (b1) {
                    const uint32_t src = __ffs(b1) - 1;
                    c = 1024 + 32 * src + __ffs(~used[i][32 + src]) - 1;
                }
                if (skip) continue;  // warp-uniform
                if (lane == 0) {
                    const uint32_t v = list[w0 + i];
                    g.st[v] = pack((uint16_t)c, 1);
                    note_color(g, v);
                    done++;
                }
                if (c < 2048)
                    for (uint32_t j = i + 1 + lane; j < cnt; j += 32)  // later vertices of the window next to it
                        if (near[j][i >> 5] >> (i & 31) & 1u) used[j][c >> 5] |= 1u << (c & 31);
                __syncwarp();
            }
        }
        ok = sync();
    }
    if (blockIdx.x == 0 && tid == 0) *colored = done;
    if (sync.leave(ok) && !ok) *colored = NONE32;
}
void launch_color_list(const Dev& g, const uint32_t* list, uint32_t m, uint32_t* place, uint32_t* rows, GridBar* bar,
                       uint32_t* colored, int num_sms, cudaStream_t s) {
    cudaMemsetAsync(place, 0, (size_t)g.n * 4, s);
    list_places_kernel<<<num_sms, 256, 0, s>>>(list, m, place);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::min(kColorWindow, spare_sms(num_sms)));  // a block per vertex of a window
    cfg.blockDim = dim3(kColorThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, color_list_kernel, g, list, m, (const uint32_t*)place, rows, bar, colored);
}

// The first `threads` threads of the grid: words [0, nw) of an array on a 16-byte
// boundary with room for three more become zero.
__device__ __forceinline__ void zero_words(uint32_t* words, uint32_t nw, uint32_t tid, uint32_t threads) {
    for (uint64_t i = 4ull * tid; i < nw; i += 4ull * threads)
        *reinterpret_cast<uint4*>(words + i) = make_uint4(0, 0, 0, 0);
}

// False: a barrier gave up.
__device__ __forceinline__ bool repair_fused(const Dev& g, const SweepBufs& b, GridSync& sync, int start,
                                             const RepairIn& in, uint32_t most) {
    RepairCtl& rc = *b.rc;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nw = (g.n + 31) / 32;
    if (start) {  // no marks, no vertex conflicted
        const uint32_t threads = gridDim.x * blockDim.x;
        zero_words(b.wmark, nw, tid, threads);
        zero_words(b.rbits, nw, tid, threads);
        zero_words(reinterpret_cast<uint32_t*>(b.needf), (g.n + 3) / 4, tid, threads);
    }
    auto reset = [&] {
        if (threadIdx.x == 0) {
            *b.item_count = 0;
            *b.pend_count = 0;
            *b.fac_count = 0;
            *b.need_count = 0;
        }
    };
    // Block 0 between two sweeps: what the next one visits and who runs it. The
    // count of the list it visits is kept in the control block and its words are
    // made zero here, where no other block runs: the collection at the sweep's end
    // adds to them, and a sweep that finds no conflict has no barrier before it.
    auto plan = [&](bool counted) {
        if (threadIdx.x != 0) return;
        const uint32_t lim = rc.list ? *b.wl_count : g.n;
        const uint32_t next = counted ? *b.next_items : NONE32;
        uint32_t go = SWEEP_ELSEWHERE;
        if (rc.cont && lim <= most) {
            const bool tail = gridDim.x > kTailBlocks && nw <= kTailWords && lim <= kTailList && next <= kTailItems;
            if (sync.nb == gridDim.x) go = tail ? SWEEP_TAIL : SWEEP_GRID;
            else if (lim <= 4 * kTailList && next <= 4 * kTailItems) go = SWEEP_TAIL;  // else another launch goes on
        }
        rc.go = go;
        rc.lim = lim;
        if (go == SWEEP_ELSEWHERE) return;  // the kernels that go on read the list's length there
        *b.wl_count = 0;
        *b.next_items = 0;
    };
    if (!sync.serial([&] {
            reset();
            if (threadIdx.x == 0) *b.seed_count = 0;
            if (start) {
                if (threadIdx.x == 0) {
                    rc.mode = in.mode;
                    rc.max_sweeps = in.max_sweeps;
                    rc.force_all = in.force_all;
                }
                __syncthreads();
                repair_begin(g, b);
                __syncthreads();
            }
            plan(false);
        }))
        return false;
    const int mode = (int)rc.mode;
    const bool indep = mode == SWEEP_INDEP;
    uint32_t go = rc.go, lim = rc.lim;
    if (start && indep) {  // the first list, which has a counter of its own
        seed_worklist(g, b, sync.nb, b.seed_count);
        if (!sync()) return false;
        lim = *b.seed_count;
        go = lim <= most ? SWEEP_GRID : SWEEP_ELSEWHERE;
        if (go == SWEEP_ELSEWHERE && tid == 0) *b.wl_count = lim;
    }
    bool recolored = false;  // bits set in b.rbits
    for (;;) {
        if (recolored)
            zero_words(b.rbits, nw, tid, sync.nb * blockDim.x);
        if (go == SWEEP_ELSEWHERE) return true;
        const bool list = rc.list != 0;
        if (go == SWEEP_TAIL && sync.nb > kTailBlocks) {
            if (blockIdx.x >= kTailBlocks) {  // the decision is read, its share of the recolored bits cleared
                sync.part();
                return true;
            }
            sync.shrink(kTailBlocks);
        }
        const uint32_t nb = sync.nb;
        const bool sym = want_sym(b, 2);
        sweep_short(g, b, mode, list, lim, sym, nb);
        if (!sync()) return false;
        const uint32_t items = *b.item_count < b.item_cap ? *b.item_count : b.item_cap;
        if (items) {
            sweep_items(g, b, mode, 2, nb);
            if (!sync()) return false;
            sweep_long(g, b, mode, items, sym, nb);
            if (!sync()) return false;
        }
        if (indep && *b.need_count) {
            if (items) {
                indep_items<kFusedThreads / 32>(g, b, nb);
                if (!sync()) return false;
            }
            indep_decide(g, b, nb);
            if (!sync()) return false;
        }
        if (*b.fac_count) {
            sweep_fac(g, b, nb);
            if (!sync()) return false;
        }
        recolored = *b.pend_count != 0;
        if (recolored) {
            sweep_commit(g, b, mode, nb);
            if ((items || !indep) && !sync()) return false;  // else the commit marks nothing and sets no bit that is read
            if (items) {
                mark_items(g, b, nb);
                if (!indep && !sync()) return false;
            }
        }
        collect_marks(g, b, nb);
        if (!sync.serial([&] {
                repair_step(g, b);
                __syncthreads();
                reset();
                plan(true);
            }))
            return false;
        go = rc.go;
        lim = rc.lim;
    }
}
__global__ void __launch_bounds__(kFusedThreads, 2) repair_fused_kernel(Dev g, SweepBufs b, int start, RepairIn in,
                                                                        uint32_t most,
                                                                        cudaGraphConditionalHandle cond,
                                                                        int has_cond) {
    GridSync sync(b.bar, g.err);
    bool ok = repair_fused(g, b, sync, start, in, most);
    if (!sync.leave(ok)) return;
    RepairCtl& rc = *b.rc;
    if (!ok) {  // nothing in the block may be taken for a result; the next repair visits every vertex
        rc.fault = 1;
        rc.cont = 0;
        for (uint32_t k = 0; k < b.G; k++) g.gctl[k].clean = 0;
    }
    if (has_cond) cudaGraphSetConditional(cond, rc.cont);
}

void launch_repair_fused(const Dev& g, const SweepBufs& b, const RepairIn* start, cudaStream_t s,
                         const cudaGraphConditionalHandle* cond) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(b.blocks);
    cfg.blockDim = dim3(kFusedThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, repair_fused_kernel, g, b, start ? 1 : 0, start ? *start : RepairIn{}, kFusedMax,
                       cond ? *cond : (cudaGraphConditionalHandle)0, cond ? 1 : 0);
}

void launch_repair_sweep(const Dev& g, const SweepBufs& b, SweepMode mode, int num_sms, cudaStream_t s,
                         cudaEvent_t* phase) {
    launch_build_items(g, b, 2, num_sms, s);
    if (phase) cudaEventRecord(phase[0], s);
    launch_sweep(g, b, mode, 2, 2, num_sms, s, phase ? phase + 1 : nullptr);
}

void launch_repair_step(const Dev& g, const SweepBufs& b, int num_sms, cudaStream_t s,
                        const cudaGraphConditionalHandle* cond) {
    launch_next_worklist(g, b, num_sms, s);
    repair_step_kernel<<<1, 256, 0, s>>>(g, b, cond ? *cond : (cudaGraphConditionalHandle)0, cond ? 1 : 0);
}

}  // namespace sgc
