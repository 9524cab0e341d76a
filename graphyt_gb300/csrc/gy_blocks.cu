// gy_blocks.cu -- the step's sort: particles kept in cell-key order by merging cell blocks.
//
// After a sorted step the slab holds each 4x4x4 cell block's particles side by side, so a block's
// particles of the next order are those of its old range that stayed in it and the few that came
// in from other blocks ("movers").  G2P, which knows every particle's old and new key, keeps the
// particle count per block current, marks the blocks in which any particle changed cell and lists
// the movers, each with its arrival number at its new block.  The stable order of the new keys
// then takes two launches:
//   k_blocks_scan   one cluster: the blocks' first positions (a prefix sum of the counts), the
//                   non-empty blocks, the place of each one's segments among those the particle
//                   kernels take (a block's particles in pieces), and the movers grouped by their
//                   new block;
//   k_blocks_place  a CTA per non-empty block: its segments, the permutation and the sorted keys.
//                   A block that nothing entered, left or changed cell in is copied; the others
//                   are sorted by (cell, old slot), a stable counting sort over their 64 cells of
//                   the movers from lower slots, the old range and the movers from higher slots,
//                   in this order.
// The result is the permutation of a stable sort of all keys.  It replaced ten launches (a merge
// of all movers with all stayers through particle-wide prefix sums: gy_resort.cu, which still
// serves sorts that several steps of movement precede), whose launch latencies were most of the
// step on small problems and whose sparse passes over per-particle masks were on large ones.
#include <algorithm>
#include <cooperative_groups.h>

#include "gy_kernels.cuh"

namespace gy {

namespace cg = cooperative_groups;

constexpr int BS_CTAS = 8;         // one portable cluster
constexpr int BS_ONE = 8192;       // blocks up to which one CTA scans them
constexpr int BS_THREADS = 1024;
constexpr int BS_WARPS = BS_THREADS / 32;
constexpr int BS_TILE = 4 * BS_THREADS;
constexpr int BP_THREADS = 128;
constexpr int BP_WARPS = BP_THREADS / 32;

// particles, entering movers, segments, non-empty blocks
struct Sums {
    int n, in, seg, ne;
};
__device__ __forceinline__ Sums operator+(Sums a, Sums b) { return {a.n + b.n, a.in + b.in, a.seg + b.seg, a.ne + b.ne}; }
// the segments a block's n particles are taken in
__device__ __forceinline__ int block_pieces(int n, Pieces piece)
{
    return n <= piece.len() ? (n > 0 ? 1 : 0) : (n - piece.merge + piece.len() - 1) >> piece.shift;
}

__device__ __forceinline__ Sums block_sums(int n, int in, Pieces piece)
{
    return {n, in, block_pieces(n, piece), n > 0 ? 1 : 0};
}
__device__ __forceinline__ Sums shfl_up(Sums a, int d)
{
    return {__shfl_up_sync(0xffffffffu, a.n, d), __shfl_up_sync(0xffffffffu, a.in, d),
            __shfl_up_sync(0xffffffffu, a.seg, d), __shfl_up_sync(0xffffffffu, a.ne, d)};
}
// inclusive scan over the CTA; *total receives the CTA's sum
__device__ __forceinline__ Sums cta_scan(Sums v, Sums *wsum, Sums *total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const Sums u = shfl_up(v, d);
        if (lane >= d) v = v + u;
    }
    __syncthreads();  // the previous use of wsum is over
    if (lane == 31) wsum[warp] = v;
    __syncthreads();
    if (warp == 0) {
        Sums w = wsum[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const Sums u = shfl_up(w, d);
            if (lane >= d) w = w + u;
        }
        wsum[lane] = w;
    }
    __syncthreads();
    if (warp > 0) v = v + wsum[warp - 1];
    *total = wsum[BS_WARPS - 1];
    return v;
}

// CTAS > 1: each CTA of the cluster takes a contiguous share of the blocks; it sums the share,
// learns the shares before its own through distributed shared memory, and scans it.  first_new is
// written, the entering counts are cleared for the next G2P and the movers
// grouped by their new block; the step's
// scalars are taken.  clear0 to clear3 (may be null): counters of the caller zeroed on
// the way.
// It is all latency: a grid of 125 blocks took 10 us in eight CTAs, of which the three cluster
// barriers and the exchange were half; one CTA takes 3.4 us, and is the faster one up to BS_ONE
// blocks (two tiles of BS_TILE).  54,000 blocks take 16 us in the cluster.
template <int CTAS>
__device__ __forceinline__ void blocks_scan(const BlockSort &b, const ScalarRing &ring, int *first_new, Pieces piece, int *nseg, int *clear0,
                                            int *clear1, int *clear2, int *clear3)
{
    __shared__ Sums wsum[BS_WARPS];
    __shared__ Sums share;
    pdl_prologue();
    const int tid = threadIdx.x, rank = CTAS > 1 ? (int)blockIdx.x : 0;
    const int nmov = *b.mov_n;
    if (rank == 0 && tid >= BS_THREADS - 32) take_scalars(ring);
    if (rank == 0 && tid == 0) {
        if (clear0) *clear0 = 0;
        if (clear1) *clear1 = 0;
        if (clear2) *clear2 = 0;
        if (clear3) *clear3 = 0;
    }
    const int per = ((b.nblk + CTAS - 1) / CTAS + 3) & ~3;  // the arrays are padded to four blocks
    const int lo = min(rank * per, b.nblk), hi = min(lo + per, b.nblk);
    Sums total, base{0, 0, 0, 0}, all{0, 0, 0, 0};
    if (CTAS > 1) {
        Sums mine{0, 0, 0, 0};
        for (int i = lo + 4 * tid; i < hi; i += BS_TILE) {
            const int4 c = *reinterpret_cast<const int4 *>(b.cnt + i), m = *reinterpret_cast<const int4 *>(b.in_cnt + i);
            mine = mine + block_sums(c.x, m.x, piece) + block_sums(c.y, m.y, piece) + block_sums(c.z, m.z, piece) +
                   block_sums(c.w, m.w, piece);
        }
        cta_scan(mine, wsum, &total);
        if (tid == 0) share = total;
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
#pragma unroll
        for (int r = 0; r < CTAS; r++) {
            const Sums q = *cl.map_shared_rank(&share, r);
            if (r < rank) base = base + q;
            all = all + q;
        }
    }
    for (int i0 = lo; i0 < hi; i0 += BS_TILE) {
        const int i = i0 + 4 * tid;
        int4 c = make_int4(0, 0, 0, 0), m = c;
        if (i < hi) {
            c = *reinterpret_cast<const int4 *>(b.cnt + i);
            m = *reinterpret_cast<const int4 *>(b.in_cnt + i);
        }
        const int cv[4] = {c.x, c.y, c.z, c.w}, mv[4] = {m.x, m.y, m.z, m.w};
        Sums s{0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 4; q++) s = s + block_sums(cv[q], mv[q], piece);
        const Sums inc = cta_scan(s, wsum, &total);
        if (i < hi) {
            Sums at{base.n + inc.n - s.n, base.in + inc.in - s.in, base.seg + inc.seg - s.seg, base.ne + inc.ne - s.ne};
            int f[4], o[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                f[q] = at.n;
                o[q] = at.in;
                if (cv[q] > 0) {
                    b.list[at.ne] = i + q;
                    b.seg_at[at.ne] = at.seg;
                }
                at = at + block_sums(cv[q], mv[q], piece);
            }
            *reinterpret_cast<int4 *>(first_new + i) = make_int4(f[0], f[1], f[2], f[3]);
            *reinterpret_cast<int4 *>(b.in_off + i) = make_int4(o[0], o[1], o[2], o[3]);
            *reinterpret_cast<int4 *>(b.in_cnt + i) = make_int4(0, 0, 0, 0);
        }
        base = base + total;
    }
    // every block's offsets are written, every share and the mover count have been read
    if (CTAS > 1) {
        __threadfence();
        cg::this_cluster().sync();
    } else {
        __syncthreads();
        all = base;
    }
    for (int m = rank * BS_THREADS + tid; m < nmov; m += CTAS * BS_THREADS) {
        const int4 q = b.mov[m];  // key, slot, arrival number
        b.in_list[__ldcg(b.in_off + (q.x >> CB_SHIFT)) + q.z] = make_int2(q.x, q.y);
    }
    if (rank == 0 && tid == 0) {
        // the ends of the last block, after the padding's writes
        first_new[b.nblk] = all.n;
        b.in_off[b.nblk] = all.in;
        *b.list_n = all.ne;
        *nseg = all.seg;
        *b.mov_n = 0;
    }
}
__global__ void __cluster_dims__(BS_CTAS, 1, 1) __launch_bounds__(BS_THREADS)
    k_blocks_scan(BlockSort b, ScalarRing ring, int *first_new, Pieces piece, int *nseg, int *clear0, int *clear1, int *clear2,
                  int *clear3)
{
    blocks_scan<BS_CTAS>(b, ring, first_new, piece, nseg, clear0, clear1, clear2, clear3);
}
__global__ void __launch_bounds__(BS_THREADS)
    k_blocks_scan_one(BlockSort b, ScalarRing ring, int *first_new, Pieces piece, int *nseg, int *clear0, int *clear1, int *clear2,
                  int *clear3)
{
    blocks_scan<1>(b, ring, first_new, piece, nseg, clear0, clear1, clear2, clear3);
}

// key: the particles' keys in the old order.  A block's members are numbered movers from lower
// slots, old range, movers from higher slots; a member of the old range that left has no cell.
// Members go through in rounds of BP_ROUND (a full block of eight particles per cell), BP_PER
// consecutive warps' worth per warp, so that ranks within a warp need no barrier: a warp matches
// its lanes' cells, and the warps' counts per cell are added up once per round.  Bound by the
// latency of its loads: 24 us (cold caches) on 2.4 million particles in nearly all of whose 4750
// blocks a particle had changed cell; with a barrier-separated count per 128 members it took 28,
// with a warp per block 38.
constexpr int BP_PER = 4;
constexpr int BP_ROUND = BP_THREADS * BP_PER;
// the segments of the block at `s` in the list (a few: written by the CTA's first threads)
__device__ __forceinline__ void put_segments(const BlockSort &b, int s, int nf, int nc, Pieces piece, int *seg_start,
                                             int *seg_len)
{
    const int at = b.seg_at[s];
    const int np = block_pieces(nc, piece);
    for (int k = threadIdx.x; k < np; k += blockDim.x) {
        seg_start[at + k] = nf + (k << piece.shift);
        seg_len[at + k] = k < np - 1 ? piece.len() : nc - (k << piece.shift);
    }
}

// the segments alone, of an order that another sort made
__global__ void __launch_bounds__(BP_THREADS) k_blocks_segments(BlockSort b, const int *first_new, Pieces piece,
                                                                int *seg_start, int *seg_len)
{
    for (int s = blockIdx.x; s < *b.list_n; s += gridDim.x) {
        const int nf = first_new[b.list[s]];
        put_segments(b, s, nf, first_new[b.list[s] + 1] - nf, piece, seg_start, seg_len);
    }
}

// The n movers entering a block, `a`, into slot order in `b` (no two have the same slot; a is
// overwritten): a stable counting sort by six bits of the slot at a time, in an odd number of passes,
// BP_THREADS movers at a time ranked by warp.  wcnt and base are the CTA's, in shared memory.
// For blocks that more than BP_RANK movers enter, where a rank by comparing each mover with all others
// loses: placement and scan with 200 / 400 / 1600 / 3200 entering at once took 14.4 / 24.6 / 180 / 610 us
// by ranks and 14.0 / 16.4 / 30.7 / 51.0 sorted (25.0 / 41 / 195 / 655 and 24.4 / 34 / 51 / 86 among a million
// particles); a pile of 64,000 crossing into a block in one step took 470 ms, and takes 1.2.
constexpr int BP_RANK = 256;
__device__ __forceinline__ void sort_by_slot(int2 *a, int2 *b, int n, int slots, int (*wcnt)[64], int *base)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    int passes = 1;
    while (6 * passes < 31 && (slots - 1) >> (6 * passes)) passes++;
    passes |= 1;
    for (int p = 0; p < passes; p++) {
        const int shift = min(6 * p, 31);  // (slots are below 2^31: a pass past them only copies)
        const int2 *src = p & 1 ? b : a;
        int2 *dst = p & 1 ? a : b;
        __syncthreads();  // the previous pass is done, and what the arrays held before
        if (tid < 64) base[tid] = 0;
        __syncthreads();
        for (int m = tid; m < n; m += BP_THREADS) atomicAdd(&base[(src[m].y >> shift) & 63], 1);
        __syncthreads();
        if (warp == 0) {
            const int u = base[2 * lane], v = base[2 * lane + 1];
            int sum = u + v;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int w = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += w;
            }
            base[2 * lane] = sum - u - v;
            base[2 * lane + 1] = sum - v;
        }
        for (int m0 = 0; m0 < n; m0 += BP_THREADS) {
            for (int q = tid; q < BP_WARPS * 64; q += BP_THREADS) wcnt[q >> 6][q & 63] = 0;
            __syncthreads();
            const int2 e = m0 + tid < n ? src[m0 + tid] : make_int2(0, 0);
            const int digit = m0 + tid < n ? (e.y >> shift) & 63 : -1;
            const unsigned same = __match_any_sync(0xffffffffu, digit);
            const int below = __popc(same & lt);
            if (digit >= 0 && below == 0) wcnt[warp][digit] = __popc(same);
            __syncthreads();
            if (tid < 64) {
                int at = base[tid];
#pragma unroll
                for (int q = 0; q < BP_WARPS; q++) {
                    const int c = wcnt[q][tid];
                    wcnt[q][tid] = at;
                    at += c;
                }
                base[tid] = at;
            }
            __syncthreads();
            if (digit >= 0) dst[wcnt[warp][digit] + below] = e;
            __syncthreads();
        }
    }
    for (int q = tid; q < BP_WARPS * 64; q += BP_THREADS) wcnt[q >> 6][q & 63] = 0;
    __syncthreads();
}

__global__ void __launch_bounds__(BP_THREADS, 12) k_blocks_place(BlockSort b, const int *key, const int *first_old,
                                                             const int *first_new, Pieces piece, int *seg_start, int *seg_len,
                                                             int *skey_out, int *perm_out)
{
    __shared__ int next[64];            // next position of each cell, in the rounds after the first
    __shared__ int tot[64];             // members per cell, of blocks of more than one round
    __shared__ int wcnt[BP_WARPS][64];  // members per cell of each warp of the round, then its first position
    __shared__ int n_lo;
    pdl_prologue();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int nb = *b.list_n;
    for (int s = blockIdx.x; s < nb; s += gridDim.x) {
        const int blk = b.list[s];
        const int nf = first_new[blk], nc = first_new[blk + 1] - nf;
        const int of = first_old[blk], oc = first_old[blk + 1] - of;
        const int io = b.in_off[blk], ic = b.in_off[blk + 1] - io;
        put_segments(b, s, nf, nc, piece, seg_start, seg_len);
        if (!b.dirty[blk] && ic == 0) {
            for (int q = tid; q < nc; q += BP_THREADS) {
                skey_out[nf + q] = key[of + q];
                perm_out[nf + q] = of + q;
            }
            continue;
        }
        // the movers in slot order: each one's rank among the block's few, or a sort of many
        __syncthreads();  // the previous block is done with the shared arrays; dirty has been read
        if (tid == 0) {
            n_lo = 0;
            b.dirty[blk] = 0;
        }
        if (tid < 64) tot[tid] = 0;
        for (int q = tid; q < BP_WARPS * 64; q += BP_THREADS) wcnt[q >> 6][q & 63] = 0;
        __syncthreads();
        if (ic <= BP_RANK) {
            for (int q = tid; q < ic; q += BP_THREADS) {
                const int2 v = b.in_list[io + q];
                int r = 0;
                for (int u = 0; u < ic; u++) r += b.in_list[io + u].y < v.y;
                b.in_sorted[io + r] = v;
                if (v.y < of) atomicAdd(&n_lo, 1);
            }
            if (ic) __syncthreads();
        } else {
            for (int q = tid; q < ic; q += BP_THREADS)
                if (b.in_list[io + q].y < of) atomicAdd(&n_lo, 1);
            sort_by_slot(b.in_list + io, b.in_sorted + io, ic, first_new[b.nblk], wcnt, next);
        }
        const int lo = n_lo, members = oc + ic;
        auto cell_of = [&](int m) {  // the member's cell, -1 if it left (or none)
            if (m >= members) return -1;
            if (m >= lo && m < lo + oc) {
                const int k = key[of + m - lo];
                return (k >> CB_SHIFT) == blk ? (k & 63) : -1;
            }
            return b.in_sorted[io + (m < lo ? m : m - oc)].x & 63;
        };
        auto slot_of = [&](int m) {  // its old slot
            return m >= lo && m < lo + oc ? of + m - lo : b.in_sorted[io + (m < lo ? m : m - oc)].y;
        };
        const bool rounds = members > BP_ROUND;
        if (rounds) {
            for (int m = tid; m < members; m += BP_THREADS) {
                const int c = cell_of(m);
                if (c >= 0) atomicAdd(&tot[c], 1);
            }
            __syncthreads();
        }
        for (int m0 = 0; m0 < members; m0 += BP_ROUND) {
            int c[BP_PER], r[BP_PER];
#pragma unroll
            for (int u = 0; u < BP_PER; u++) c[u] = cell_of(m0 + (warp * BP_PER + u) * 32 + lane);
#pragma unroll
            for (int u = 0; u < BP_PER; u++) {
                const unsigned same = __match_any_sync(0xffffffffu, c[u]);
                const int below = __popc(same & lt), first = __ffs(same) - 1;
                int before = 0;
                if (c[u] >= 0 && below == 0) {  // one lane per cell: the warp's earlier members of it
                    before = wcnt[warp][c[u]];
                    wcnt[warp][c[u]] = before + __popc(same);
                }
                r[u] = __shfl_sync(0xffffffffu, before, first) + below;
                __syncwarp();
            }
            __syncthreads();
            if (warp == 0) {
                // counts per cell -> positions: cells in order, within a cell the warps in order
                int half = 0;  // members of the first 32 cells
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int cell = 32 * h + lane;
                    int w[BP_WARPS], t = 0;
#pragma unroll
                    for (int q = 0; q < BP_WARPS; q++) {
                        w[q] = wcnt[q][cell];
                        t += w[q];
                    }
                    int at;
                    if (m0 == 0) {
                        const int mine = rounds ? tot[cell] : t;
                        int sc = mine;
#pragma unroll
                        for (int d = 1; d < 32; d <<= 1) {
                            const int u = __shfl_up_sync(0xffffffffu, sc, d);
                            if (lane >= d) sc += u;
                        }
                        at = nf + half + sc - mine;
                        half = __shfl_sync(0xffffffffu, sc, 31);
                    } else {
                        at = next[cell];
                    }
                    next[cell] = at + t;
#pragma unroll
                    for (int q = 0; q < BP_WARPS; q++) {
                        wcnt[q][cell] = at;
                        at += w[q];
                    }
                }
            }
            __syncthreads();
#pragma unroll
            for (int u = 0; u < BP_PER; u++)
                if (c[u] >= 0) {
                    const int p = wcnt[warp][c[u]] + r[u];
                    skey_out[p] = (blk << CB_SHIFT) | c[u];
                    perm_out[p] = slot_of(m0 + (warp * BP_PER + u) * 32 + lane);
                }
            if (m0 + BP_ROUND < members) {
                __syncthreads();
                for (int q = tid; q < BP_WARPS * 64; q += BP_THREADS) wcnt[q >> 6][q & 63] = 0;
                __syncthreads();
            }
        }
    }
}

// particles per block of a sorted key array: the block's last position + 1 less its first
// (cnt zero on entry)
__global__ void __launch_bounds__(256) k_blocks_count(const int *skey, int n, int *cnt)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int blk = skey[i] >> CB_SHIFT;
        if (i == 0 || (skey[i - 1] >> CB_SHIFT) != blk) atomicSub(&cnt[blk], i);
        if (i == n - 1 || (skey[i + 1] >> CB_SHIFT) != blk) atomicAdd(&cnt[blk], i + 1);
    }
}

size_t block_sort_ints(long long nblk, long long cap)
{
    const size_t pad = ((size_t)nblk + 8) & ~(size_t)3;
    return 6 * pad + 16 + 4 * (size_t)cap + 2 * 2 * (size_t)cap + 2 * (size_t)std::min(nblk, cap) + 64;
}

void block_sort_bind(BlockSort &b, int *mem, long long nblk, long long cap)
{
    const size_t pad = ((size_t)nblk + 8) & ~(size_t)3;  // four-block loads, one entry past the end
    int *p = mem;
    b.mov = reinterpret_cast<int4 *>(p); p += 4 * cap;
    b.in_list = reinterpret_cast<int2 *>(p); p += 2 * cap;
    b.in_sorted = reinterpret_cast<int2 *>(p); p += 2 * cap;
    b.cnt = p; p += pad;
    b.in_cnt = p; p += pad;
    b.dirty = p; p += pad;
    b.first[0] = p; p += pad;
    b.first[1] = p; p += pad;
    b.in_off = p; p += pad;
    b.mov_n = p;
    b.list_n = p + 1;
    p += 16;
    b.list = p; p += std::min(nblk, cap);
    b.seg_at = p;
    b.nblk = (int)nblk;
}

void launch_blocks_count(const BlockSort &b, const int *skey, long long n, cudaStream_t s)
{
    // and no movers: what a G2P before the sort from scratch noted is void
    cudaMemsetAsync(b.cnt, 0, (size_t)(b.in_cnt - b.cnt) * 2 * sizeof(int), s);
    cudaMemsetAsync(b.mov_n, 0, sizeof(int), s);
    if (n <= 0) return;
    k_blocks_count<<<(unsigned)std::min<long long>((n + 255) / 256, 4096), 256, 0, s>>>(skey, (int)n, b.cnt);
    note_launch(1);
}

__global__ void k_take_scalars(ScalarRing ring) { take_scalars(ring); }

void launch_take_scalars(const ScalarRing &ring, cudaStream_t s)
{
    k_take_scalars<<<1, 32, 0, s>>>(ring);
    note_launch(1);
}

void launch_blocks_scan(const BlockSort &b, const ScalarRing &ring, int which, Pieces piece, int *nseg, cudaStream_t s,
                        int *clear0, int *clear1, int *clear2, int *clear3)
{
    if (b.nblk <= BS_ONE)
        launch_pdl(k_blocks_scan_one, 1, BS_THREADS, s, b, ring, b.first[which], piece, nseg, clear0, clear1, clear2,
                   clear3);
    else
        launch_pdl(k_blocks_scan, BS_CTAS, BS_THREADS, s, b, ring, b.first[which], piece, nseg, clear0, clear1, clear2,
                   clear3);
    note_launch(1);
}

void launch_blocks_place(const BlockSort &b, const int *key, int which, Pieces piece, int *seg_start, int *seg_len,
                         int *skey_out, int *perm_out, long long n, cudaStream_t s)
{
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    const long long blocks = std::min<long long>(b.nblk, n);
    const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>(blocks, (long long)sms * 16));
    if (key)
        launch_pdl(k_blocks_place, grid, BP_THREADS, s, b, key, (const int *)b.first[which ^ 1],
                   (const int *)b.first[which], piece, seg_start, seg_len, skey_out, perm_out);
    else
        k_blocks_segments<<<grid, BP_THREADS, 0, s>>>(b, b.first[which], piece, seg_start, seg_len);
    note_launch(1);
}

}  // namespace gy
