// table_kernels.cuh -- histogram -> 12-bit frequency table on the device.
//
// normalize_tables_kernel is ANSCompressor::normalize_histogram
// (src/ANSCompressor.cpp:416-503 in the Checkers tree) for a whole batch of
// tables, one CTA of 256 threads (one per symbol) per table, followed by what
// build_enc_entries (tables.hpp) derives from the result.  With it the
// histograms never leave the device and the compress pipeline needs no host
// step between counting and encoding.
//
// The reference hands out (or takes back) rounding slots in the order
// std::sort leaves the symbols in when sorted by the fractional part of their
// ideal share, and std::sort is not stable: where fractions are equal the order
// is whatever the library's algorithm leaves behind.  sort_replica.hpp restates
// that algorithm move for move; here the same moves are made by the 256 threads
// of the table's CTA together (block_sort_order).
#pragma once
#include "sort_replica.hpp"

namespace chk {

enum : uint32_t {
    kTableFullAlphabet = 1u,  // every symbol gets at least one slot (tables shared by a cluster)
    kTableRepair = 2u,        // repeat the take-back pass until the sum is 4096 (opt-in deviation)
};

// Which work item owns table t and how it is built.
struct TableJob {
    uint32_t owner;  // index of the owning tensor in the batch (histogram row)
    uint32_t flags;  // kTable*
};

struct NormSmem {
    FracKey keys[256];
    uint32_t mask_a[8], mask_b[8];
    uint16_t pos_a[256], pos_b[256], cut[256];
    uint16_t place[256];  // by symbol: its position in the sorted order
    uint32_t warp_a[8], warp_b[8];
    unsigned long long warp_c[8];
};

// Sums over the 256 threads of a CTA (all threads get the result).
__device__ __forceinline__ uint32_t block_sum256(uint32_t v, uint32_t* warp_part) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();  // warp_part may still be read from a previous use
    if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t s = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += warp_part[w];
    return s;
}
__device__ __forceinline__ unsigned long long block_sum256_u64(unsigned long long v, unsigned long long* warp_part) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = v;
    __syncthreads();
    unsigned long long s = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += warp_part[w];
    return s;
}
// Exclusive prefix sum over the 256 threads; *total_out receives the sum.
__device__ __forceinline__ uint32_t block_scan256(uint32_t v, uint32_t* warp_part, uint32_t* total_out) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t n = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += n;
    }
    __syncthreads();
    if (lane == 31) warp_part[warp] = inc;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if ((uint32_t)w < warp) before += warp_part[w];
        total += warp_part[w];
    }
    *total_out = total;
    return before + inc - v;
}

// Set bits of a 256-bit mask in [lo, hi).
__device__ __forceinline__ uint32_t mask_count(const uint32_t* mask, uint32_t lo, uint32_t hi) {
    uint32_t c = 0;
    for (uint32_t w = lo >> 5; w * 32 < hi; ++w) {
        uint32_t m = mask[w];
        if (w * 32 < lo) m &= 0xFFFFFFFFu << (lo & 31);
        if (hi < w * 32 + 32) m &= ~(0xFFFFFFFFu << (hi & 31));
        c += (uint32_t)__popc(m);
    }
    return c;
}

// keys[0..n) sorted as sort_replica sorts them; sm.place[symbol] receives the positions.
// One thread walking the introsort took about 100 us a table; almost all of it is the Hoare partitions, and those
// can be done at once.  A partition of [F + 1, L) about p swaps the k-th element from the left that does not stand
// before p with the k-th from the right that p does not stand before, for as long as the first lies left of the
// second: thread i finds the rank of its element among either kind by counting bits, and the pairs are disjoint.
// With K swaps made, the next left stop (or, if that is further right, the last element swapped to the right, which
// now stops the scan) is the cut.  Ranges of one recursion level are independent and run side by side, all at
// the same depth; the final insertion sort never moves an element past an equal one, so it is a stable sort of
// what the partitions leave, and an element only moves inside its range of 16 or fewer.
__device__ __forceinline__ void block_sort_order(NormSmem& sm, uint32_t n) {
    const uint32_t i = threadIdx.x, warp = i >> 5, lane = i & 31;
    uint32_t F = 0, L = n, depth = 0;  // this position's range
    while ((2u << depth) <= n) ++depth;
    depth *= 2;  // 2 * floor(log2 n)
    for (;; --depth) {
        const bool active = i < n && L - F > 16;
        if (block_sum256(active ? 1u : 0u, sm.warp_a) == 0) break;
        if (depth == 0) {
            if (active && i == F) sr_heap_sort(sm.keys + F, sm.keys + L);
            __syncthreads();
            break;
        }
        if (active && i == F) sr_median_to_first(sm.keys + F, sm.keys + F + 1, sm.keys + F + (L - F) / 2, sm.keys + L - 1);
        __syncthreads();
        const double p = active ? sm.keys[F].frac : 0.0, v = active ? sm.keys[i].frac : 0.0;
        const bool a = active && i > F && !(v > p), b = active && i > F && !(p > v);
        const uint32_t ma = __ballot_sync(0xffffffffu, a), mb = __ballot_sync(0xffffffffu, b);
        if (lane == 0) {
            sm.mask_a[warp] = ma;
            sm.mask_b[warp] = mb;
        }
        __syncthreads();
        const uint32_t ra = a ? mask_count(sm.mask_a, F + 1, i) : 0u;
        if (a) sm.pos_a[F + ra] = (uint16_t)i;
        if (b) sm.pos_b[F + mask_count(sm.mask_b, i + 1, L)] = (uint16_t)i;
        __syncthreads();
        if (a) {
            const uint32_t na = mask_count(sm.mask_a, F + 1, L), nb = mask_count(sm.mask_b, F + 1, L);
            const uint32_t mate = ra < nb ? sm.pos_b[F + ra] : 0u;  // 0: none (a position right of F is never below it)
            if (i < mate) {
                const uint32_t next = ra + 1 < na ? sm.pos_a[F + ra + 1] : 0xFFFFu;
                if (!(ra + 1 < nb && next < sm.pos_b[F + ra + 1])) sm.cut[F] = (uint16_t)(next < mate ? next : mate);
                sr_swap(sm.keys[i], sm.keys[mate]);
            } else if (ra == 0) {
                sm.cut[F] = (uint16_t)i;
            }
        }
        __syncthreads();
        if (active) {
            const uint32_t c = sm.cut[F];
            if (i < c) L = c; else F = c;
        }
    }
    if (i < n) {
        const double v = sm.keys[i].frac;
        uint32_t at = F;
        for (uint32_t k = F; k < L; ++k) {
            const double o = sm.keys[k].frac;
            at += o > v || (o == v && k < i);
        }
        sm.place[sm.keys[i].sym] = (uint16_t)at;
    }
    __syncthreads();
}

// The encode entry of one symbol (same arithmetic as build_enc_entries in tables.hpp).
__device__ __forceinline__ EncEntry make_enc_entry(uint32_t f, uint32_t c) {
    EncEntry e;
    e.rcp = e.freq_shift = e.bias = e.cmpl = 0;
    if (f == 1) {
        e.rcp = 0xFFFFFFFFu;
        e.freq_shift = 1u;
        e.bias = c + (kM - 1);
        e.cmpl = kM - 1;
    } else if (f > 1) {
        uint32_t sh = 0;
        while ((1u << sh) < f) ++sh;
        const unsigned long long num = 1ull << (31 + sh);
        e.rcp = (uint32_t)((num + f - 1) / f);
        e.freq_shift = f | ((sh - 1) << 16);
        e.bias = c;
        e.cmpl = kM - f;
    }
    return e;
}

// hist: [batch tensors][256] counts of the codec-input bytes EXCEPT the zeroed low bytes
// (split_hist_kernel's output); the kernel adds those to bin 0 from the descriptor.
// Outputs for table t (t counts from the first table of this launch): freq[t][256],
// cum[t][257], enc[t][256], sums[t] (4096 for a decodable table).
__global__ void __launch_bounds__(256) normalize_tables_kernel(const TableJob* __restrict__ jobs,
                                                               const TensorDesc* __restrict__ descs,
                                                               const uint32_t* __restrict__ hist,
                                                               EncEntry* __restrict__ enc, uint32_t* __restrict__ freq,
                                                               uint32_t* __restrict__ cum, uint32_t* __restrict__ sums,
                                                               uint32_t n_tables) {
    CHK_SHARED NormSmem sm;
    const uint32_t s = threadIdx.x;
    for (uint32_t t = blockIdx.x; t < n_tables; t += gridDim.x) {
        const TableJob job = jobs[t];
        const TensorDesc d = descs[job.owner];
        const bool full = (job.flags & kTableFullAlphabet) != 0;
        uint32_t h = hist[(size_t)job.owner * 256 + s];
        if (s == 0 && d.es) h += (uint32_t)(d.n_bytes / d.es * d.spe);  // the zeroed low bytes are codec input too
        const unsigned long long total = block_sum256_u64(h, sm.warp_c);
        const uint32_t distinct = block_sum256(h ? 1u : 0u, sm.warp_a);
        uint32_t slot = 0;
        if ((full ? 256u : distinct) == 0) {
            slot = s == 0 ? kM : 0u;  // empty input: all mass on symbol 0 (:432-441)
        } else {
            const bool present = full || h != 0;
            const uint32_t hc = h > 1u ? h : 1u;
            if (present) {
                const uint32_t v = total ? (uint32_t)(((unsigned long long)hc * kM) / total) : 0u;
                slot = v ? v : 1u;
            }
            const double exact = total ? ((double)hc * (double)kM / (double)total) : 1.0;
            const double fr = exact - (double)(int)exact;
            const uint32_t assigned = block_sum256(slot, sm.warp_a);
            const uint32_t n_keys = block_sum256(present ? 1u : 0u, sm.warp_b);
            if (assigned < kM && kM - assigned >= n_keys) {
                slot += present ? 1u : 0u;
            } else if (assigned != kM) {
                // keys in symbol order, exactly the vector the reference sorts
                uint32_t n_tot;
                const uint32_t pos = block_scan256(present ? 1u : 0u, sm.warp_a, &n_tot);
                if (present) {
                    FracKey key;
                    key.frac = fr;
                    key.sym = (int32_t)s;
                    key.pad_ = 0;
                    sm.keys[pos] = key;
                }
                __syncthreads();
                block_sort_order(sm, n_tot);
                const uint32_t at = present ? sm.place[s] : 0u;
                if (assigned < kM) {
                    slot += present && at < kM - assigned ? 1u : 0u;
                } else {
                    // slots are taken back from the end of the order, one per symbol that has more than one
                    uint32_t rem = assigned - kM;
                    for (;;) {
                        if (s < 8) sm.mask_a[s] = 0;
                        __syncthreads();
                        const bool can = present && slot > 1;
                        if (can) atomicOr(&sm.mask_a[at >> 5], 1u << (at & 31));
                        __syncthreads();
                        if (can && mask_count(sm.mask_a, at + 1, n_tot) < rem) --slot;
                        const uint32_t before = rem, able = mask_count(sm.mask_a, 0, n_tot);
                        rem -= able < rem ? able : rem;
                        __syncthreads();
                        if (!(job.flags & kTableRepair) || rem == 0 || rem == before) break;
                    }
                }
            }
        }
        uint32_t sum;
        const uint32_t c = block_scan256(slot, sm.warp_b, &sum);
        freq[(size_t)t * 256 + s] = slot;
        cum[(size_t)t * 257 + s] = c;
        if (s == 255) {
            cum[(size_t)t * 257 + 256] = c + slot;
            sums[t] = sum;
        }
        enc[(size_t)t * 256 + s] = make_enc_entry(slot, c);
        __syncthreads();
    }
}

}  // namespace chk
