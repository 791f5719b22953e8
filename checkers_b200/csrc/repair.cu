// repair.cu -- host side of the prefix-mask Re-Pair estimator (C ABI: chk_repair_*).
//
// Drives the kernels of repair_kernels.cuh the way build_shared_grammar /
// apply_existing_grammar drive their loops in the reference
// (src/tensor_group_prefix_mask_repair.cpp:423-463 in the Checkers tree).
//
// Tie order.  The reference picks the most frequent pair by iterating a
// std::unordered_map and keeping the first entry whose count is strictly larger
// (:389-395), so among pairs with equal counts the winner is whichever the map
// yields first.  The map's order depends only on the bucket count
// (reserve(tokens.size())), the hash, and the order in which distinct keys were
// first inserted.  When the device finds more than one pair at the maximum, the
// distinct pairs are brought to the host with their first positions, inserted
// in that order into a map built exactly like the reference's, and the map is
// walked the same way; otherwise the host is not involved.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/checkers_b200.h"
#include "repair_kernels.cuh"

namespace chkrp {

struct Error {
    int code;
    std::string msg;
};
static thread_local std::string g_err;

#define RP_CUDA(call)                                                                        \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess) throw Error{CHK_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)}; \
    } while (0)

struct Dev {
    void* p = nullptr;
    ~Dev() {
        if (p) cudaFree(p);
    }
    template <typename T>
    T* as() const {
        return static_cast<T*>(p);
    }
    void alloc(size_t bytes) { RP_CUDA(cudaMalloc(&p, bytes ? bytes : 16)); }
};

// symbol value the reference would hold for a token id
static inline uint64_t symbol_of(uint32_t id, uint32_t masked_bits) {
    return id < kRuleBase ? ((uint64_t)id << masked_bits) : ((1ull << 63) + (uint64_t)(id - kRuleBase));
}

struct PairKey {
    uint64_t lhs, rhs;
    bool operator==(const PairKey& o) const { return lhs == o.lhs && rhs == o.rhs; }
};
struct PairKeyHash {  // same mixing as the reference's PairKeyHash (:363-371)
    size_t operator()(const PairKey& k) const {
        const size_t a = std::hash<uint64_t>{}(k.lhs), b = std::hash<uint64_t>{}(k.rhs);
        return a ^ (b + 0x9e3779b97f4a7c15ull + (a << 6u) + (a >> 2u));
    }
};

// Device working set of one call.  One instance per device is kept for the life of the process and
// only grows, so a run over many tensors does not pay an allocation per tensor.
struct Workspace {
    uint32_t n_cap = 0, contiguous_cap = 0, capacity = 0;
    size_t raw_cap = 0;
    Dev tok_a, tok_b, mark, run_start, keep, pos, blocks, keys, counts, first, small, tie_keys, tie_first, dump_keys,
        dump_counts, dump_first, raw, tile_tok, tile_ends, tile_table, rules;
    uint32_t rules_cap = 0;
    bool smem_set = false;
    cudaStream_t s = nullptr;
    std::mutex mu;          // one call at a time works on a device's workspace
    ~Workspace() {
        if (s) cudaStreamDestroy(s);
    }
    static void drop(std::initializer_list<Dev*> all) {
        for (Dev* d : all) {
            if (d->p) cudaFree(d->p);
            d->p = nullptr;
        }
    }
    // the tensor itself, its tiles and what goes with them
    void init(uint32_t n, size_t raw_bytes) {
        if (!s) RP_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        if (raw_bytes > raw_cap || !raw.p) {
            drop({&raw});
            raw_cap = 0;
            raw.alloc(raw_bytes);
            raw_cap = raw_bytes;
        }
        if (n > n_cap || !tile_tok.p) {
            drop({&tile_tok, &tile_ends});
            n_cap = 0;
            const size_t tiles = ((size_t)n + kTile - 1) / kTile + 1;
            tile_tok.alloc(2 * tiles * kTile * 2);
            tile_ends.alloc(2 * tiles * sizeof(TileEnds));
            n_cap = n;
        }
        if (!tile_table.p) tile_table.alloc(kTileTableBytes);
    }
    // what the kernels on contiguous sequences need
    void init_contiguous(uint32_t n) {
        capacity = 1024;  // table sized for THIS tensor: the hash mask must match what is cleared
        while (capacity < 2ull * n) capacity <<= 1;
        if (n <= contiguous_cap && tok_a.p) return;
        drop({&tok_a, &tok_b, &mark, &run_start, &keep, &pos, &blocks, &keys, &counts, &first, &small, &tie_keys, &tie_first,
              &dump_keys, &dump_counts, &dump_first});
        contiguous_cap = 0;
        const size_t nb = (size_t)(n ? n : 1) * 4;
        tok_a.alloc(nb);
        tok_b.alloc(nb);
        mark.alloc(nb);
        run_start.alloc(nb);
        keep.alloc(nb);
        pos.alloc(nb);
        blocks.alloc(((size_t)n / kScanBlock + 8) * 4);
        keys.alloc((size_t)capacity * 8);
        counts.alloc((size_t)capacity * 4);
        first.alloc((size_t)capacity * 4);
        small.alloc(64);
        tie_keys.alloc(64);
        tie_first.alloc(32);
        contiguous_cap = n;
    }
    void ensure_rules(uint32_t n) {
        if (n <= rules_cap) return;
        drop({&rules});
        rules_cap = 0;
        rules.alloc((size_t)(n + 64) * 12);
        rules_cap = n + 64;
    }
    // state, words that occur, numbers, words by number, matrix, two dumps
    static constexpr size_t kMatrixBytes = (size_t)kDense * kDense * 4;
    static constexpr size_t kTileTableBytes = 128 + 2 * (1u << kTileBits) + 512 + 3 * kMatrixBytes;
};
static_assert(sizeof(RoundState) <= 128 && kDense * 2 <= 512, "layout of the tile table");

template <int OP>
static void scan(Workspace& w, const uint32_t* in, uint32_t n, uint32_t* out) {
    const uint32_t nb = (n + kScanBlock - 1) / kScanBlock;
    scan_reduce_kernel<OP><<<nb, 256, 0, w.s>>>(in, n, w.blocks.as<uint32_t>());
    scan_blocks_kernel<OP><<<1, 256, 0, w.s>>>(w.blocks.as<uint32_t>(), nb);
    scan_apply_kernel<OP><<<nb, 256, 0, w.s>>>(in, n, w.blocks.as<uint32_t>(), out);
    RP_CUDA(cudaGetLastError());
}

static uint32_t grid_for(uint32_t n) {
    const uint32_t g = (n + 255) / 256;
    return g < 1 ? 1 : (g > 148 * 16 ? 148 * 16 : g);
}

// Rewrites `in` (n tokens) under rule (lhs, rhs) -> new_sym into `out`; returns the new length.
static uint32_t apply_rule(Workspace& w, const uint32_t* in, uint32_t n, uint32_t lhs, uint32_t rhs, uint32_t new_sym,
                           uint32_t* out) {
    if (n == 0) return 0;
    const uint32_t g = grid_for(n);
    if (lhs == rhs) {
        run_mark_kernel<<<g, 256, 0, w.s>>>(in, n, lhs, w.mark.as<uint32_t>());
        scan<1>(w, w.mark.as<uint32_t>(), n, w.run_start.as<uint32_t>());
    }
    rule_flags_kernel<<<g, 256, 0, w.s>>>(in, n, lhs, rhs, w.run_start.as<uint32_t>(), w.keep.as<uint32_t>());
    scan<0>(w, w.keep.as<uint32_t>(), n, w.pos.as<uint32_t>());
    rule_scatter_kernel<<<g, 256, 0, w.s>>>(in, n, lhs, rhs, new_sym, w.run_start.as<uint32_t>(),
                                            w.keep.as<uint32_t>(), w.pos.as<uint32_t>(), out);
    RP_CUDA(cudaGetLastError());
    uint32_t total = 0;  // scan_blocks leaves the grand total after the last block value
    const uint32_t nb = (n + kScanBlock - 1) / kScanBlock;
    RP_CUDA(cudaMemcpyAsync(&total, w.blocks.as<uint32_t>() + nb, 4, cudaMemcpyDeviceToHost, w.s));
    RP_CUDA(cudaStreamSynchronize(w.s));
    return total;
}

// The tensor to the device.  (Filling a pinned buffer with several threads instead: 203 against 253 us for 4 MB, slower
// below 2 MB, the same from 16 MB on.)
static void upload_raw(Workspace& w, const void* h_raw, size_t bytes) {
    if (bytes) RP_CUDA(cudaMemcpyAsync(w.raw.p, h_raw, bytes, cudaMemcpyHostToDevice, w.s));
}

static void mask_tokens(Workspace& w, uint64_t numel, uint32_t storage_bytes, uint32_t masked_bits) {
    if (numel == 0) return;
    mask_words_kernel<<<grid_for((uint32_t)numel), 256, 0, w.s>>>(w.raw.as<uint8_t>(), numel, storage_bytes, masked_bits,
                                                                  w.tok_a.as<uint32_t>());
    RP_CUDA(cudaGetLastError());
}

// ---- the tile path
static TileParams tile_params(Workspace& w, uint32_t n, uint32_t max_rules) {
    w.ensure_rules(max_rules + 1);
    TileParams P{};
    P.n_tiles = (n + kTile - 1) / kTile;
    P.max_rules = max_rules;
    P.tokens[0] = w.tile_tok.as<uint16_t>();
    P.tokens[1] = P.tokens[0] + (size_t)P.n_tiles * kTile;
    P.ends[0] = w.tile_ends.as<TileEnds>();
    P.ends[1] = P.ends[0] + P.n_tiles;
    P.rules = w.rules.as<uint2>();
    P.rule_freq = reinterpret_cast<uint32_t*>(P.rules + w.rules_cap);
    uint8_t* t = w.tile_table.as<uint8_t>();
    P.state = reinterpret_cast<RoundState*>(t);
    P.present = t + 128;
    P.pairs = reinterpret_cast<uint32_t*>(P.present + (1u << kTileBits));
    P.dump_counts = P.pairs + kDense * kDense;
    P.dump_first = P.dump_counts + kDense * kDense;
    P.number = reinterpret_cast<uint8_t*>(P.dump_first + kDense * kDense);
    P.word_of = reinterpret_cast<uint16_t*>(P.number + (1u << kTileBits));
    if (!w.smem_set) {  // per device
        const int most = (int)tile_count_smem(kDense);
        RP_CUDA(cudaFuncSetAttribute(tile_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        RP_CUDA(cudaFuncSetAttribute(tile_rule_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        RP_CUDA(cudaFuncSetAttribute(tile_dump_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most + (int)Workspace::kMatrixBytes));
        w.smem_set = true;
    }
    return P;
}

// A launch that may begin while the one before it is still running (its kernel waits for that one itself).
template <typename K, typename... A>
static void launch_overlapping(cudaStream_t s, K kernel, uint32_t grid, size_t smem, A... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kTileThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    RP_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
}

// token of the tiles <-> token id of the interface
static uint32_t id_of_token(uint32_t t) { return t < kRuleToken ? t : kRuleBase + (t - kRuleToken); }
static bool token_of_id(uint32_t id, uint32_t* t) {
    if (id < kRuleToken) {
        *t = id;
        return true;
    }
    *t = kRuleToken + (id - kRuleBase);
    return id >= kRuleBase && id - kRuleBase < kRuleToken;
}

// Which of several pairs with the largest count the reference's map yields first: the distinct pairs inserted in order of
// their first position into a map built exactly like the reference's, and the map walked the same way.
static unsigned long long first_in_map_order(const std::vector<unsigned long long>& hk, const std::vector<uint32_t>& hc,
                                             const std::vector<uint32_t>& hf, uint32_t n_tokens, uint32_t masked_bits) {
    const uint32_t d = (uint32_t)hk.size();
    std::vector<uint32_t> order(d);
    for (uint32_t i = 0; i < d; ++i) order[i] = i;
    std::sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return hf[a] < hf[b]; });
    std::unordered_map<PairKey, size_t, PairKeyHash> counts;
    counts.reserve(n_tokens);
    std::unordered_map<PairKey, unsigned long long, PairKeyHash> back;  // symbol pair -> id key
    back.reserve(d);
    for (uint32_t i : order) {
        const PairKey pk{symbol_of((uint32_t)(hk[i] >> 32), masked_bits), symbol_of((uint32_t)hk[i], masked_bits)};
        counts[pk] = hc[i];
        back[pk] = hk[i];
    }
    size_t best_count = 0;
    PairKey best_pair{};
    for (const auto& kv : counts)
        if (kv.second > best_count) {
            best_count = kv.second;
            best_pair = kv.first;
        }
    return back[best_pair];
}

// The grammar of the tensor in w.raw on tiles.  False: too many symbols, nothing has been decided.
static bool build_on_tiles(Workspace& w, uint32_t numel, uint32_t storage_bytes, uint32_t masked_bits, uint32_t max_rules,
                           uint32_t* rule_lhs, uint32_t* rule_rhs, uint64_t* rule_freq, uint32_t* n_rules_out,
                           uint64_t* tokens_out, uint64_t* max_freq_out, uint64_t* tie_rounds_out) {
    const TileParams P = tile_params(w, numel, max_rules);
    RP_CUDA(cudaMemsetAsync(P.state, 0, 128 + (1u << kTileBits) + Workspace::kMatrixBytes, w.s));  // state, words, matrix
    tile_words_kernel<true><<<P.n_tiles, kTileThreads, sizeof(TileCountSmem), w.s>>>(w.raw.as<uint8_t>(), numel, storage_bytes,
                                                                                     masked_bits, P);
    tile_pairs_kernel<<<P.n_tiles, kTileThreads, tile_count_smem(kDense), w.s>>>(P);
    RP_CUDA(cudaGetLastError());
    RoundState st{};
    auto read_state = [&] {
        RP_CUDA(cudaMemcpyAsync(&st, P.state, sizeof(st), cudaMemcpyDeviceToHost, w.s));
        RP_CUDA(cudaStreamSynchronize(w.s));
    };
    read_state();
    if (st.stop == kTooMany) return false;
    uint64_t ties = 0;
    uint32_t applied = 0;  // rules whose launch is queued
    for (;;) {
        if (st.stop == kNoMore) break;
        if (st.stop == kTie) {
            ++ties;
            const uint32_t cells = st.side * st.side, current = st.n_rules - 1;
            RP_CUDA(cudaMemsetAsync(P.dump_counts, 0, (size_t)cells * 4, w.s));
            RP_CUDA(cudaMemsetAsync(P.dump_first, 0xFF, (size_t)cells * 4, w.s));
            tile_dump_kernel<<<P.n_tiles, kTileThreads, tile_count_smem(st.side) + cells * 4, w.s>>>(P, current & 1u);
            RP_CUDA(cudaGetLastError());
            std::vector<uint32_t> counts(cells), first(cells);
            std::vector<uint16_t> words(st.n_symbols);
            RP_CUDA(cudaMemcpyAsync(counts.data(), P.dump_counts, (size_t)cells * 4, cudaMemcpyDeviceToHost, w.s));
            RP_CUDA(cudaMemcpyAsync(first.data(), P.dump_first, (size_t)cells * 4, cudaMemcpyDeviceToHost, w.s));
            RP_CUDA(cudaMemcpyAsync(words.data(), P.word_of, words.size() * 2, cudaMemcpyDeviceToHost, w.s));
            RP_CUDA(cudaStreamSynchronize(w.s));
            auto id = [&](uint32_t k) { return k < st.n_symbols ? (uint32_t)words[k] : kRuleBase + (k - st.n_symbols); };
            std::vector<unsigned long long> hk;
            std::vector<uint32_t> hc, hf;
            for (uint32_t i = 0; i < cells; ++i)
                if (counts[i]) {
                    hk.push_back(((unsigned long long)id(i / st.side) << 32) | id(i % st.side));
                    hc.push_back(counts[i]);
                    hf.push_back(first[i]);
                }
            const unsigned long long key = first_in_map_order(hk, hc, hf, st.n_tokens, masked_bits);
            uint2 rule;
            token_of_id((uint32_t)(key >> 32), &rule.x);
            token_of_id((uint32_t)key, &rule.y);
            RP_CUDA(cudaMemcpyAsync(P.rules + current, &rule, sizeof(rule), cudaMemcpyHostToDevice, w.s));
            const uint32_t go_on = kGoOn;
            RP_CUDA(cudaMemcpyAsync(&P.state->stop, &go_on, 4, cudaMemcpyHostToDevice, w.s));
            RP_CUDA(cudaStreamSynchronize(w.s));  // rule and go_on are on this stack frame
            applied = current;
        } else if (applied == max_rules) {
            break;
        }
        // everything that may follow is queued at once; launches behind a stop do nothing.  Where one tie has come more
        // are likely, so then a few at a time.
        for (const uint32_t until = ties ? std::min(max_rules, applied + 8) : max_rules; applied < until; ++applied)
            if (applied + 1 < max_rules)
                launch_overlapping(w.s, tile_rule_kernel<true>, P.n_tiles, tile_count_smem(st.side), P, applied);
            else
                launch_overlapping(w.s, tile_rule_kernel<false>, P.n_tiles, sizeof(TileCountSmem), P, applied);
        if (applied == max_rules) launch_overlapping(w.s, tile_total_kernel, 1, 0, P, max_rules & 1u);
        read_state();
    }
    const uint32_t n_rules = st.n_rules;
    std::vector<uint2> rules(n_rules);
    std::vector<uint32_t> freq(n_rules);
    if (n_rules) {
        RP_CUDA(cudaMemcpyAsync(rules.data(), P.rules, (size_t)n_rules * 8, cudaMemcpyDeviceToHost, w.s));
        RP_CUDA(cudaMemcpyAsync(freq.data(), P.rule_freq, (size_t)n_rules * 4, cudaMemcpyDeviceToHost, w.s));
        RP_CUDA(cudaStreamSynchronize(w.s));
    }
    for (uint32_t r = 0; r < n_rules; ++r) {
        if (rule_lhs) rule_lhs[r] = id_of_token(rules[r].x);
        if (rule_rhs) rule_rhs[r] = id_of_token(rules[r].y);
        if (rule_freq) rule_freq[r] = freq[r];
    }
    *n_rules_out = n_rules;
    *tokens_out = st.n_tokens;
    if (max_freq_out) *max_freq_out = st.max_freq;
    if (tie_rounds_out) *tie_rounds_out = ties;
    return true;
}

static Workspace& workspace_for(int device) {
    static Workspace* per_device[64] = {};
    static std::mutex mu;
    if (device < 0 || device >= 64) throw Error{CHK_ERR_INVALID, "device ordinal out of range"};
    std::lock_guard<std::mutex> lock(mu);
    if (!per_device[device]) per_device[device] = new Workspace();
    return *per_device[device];
}

static void check_args(uint64_t numel, uint32_t storage_bytes, uint32_t masked_bits) {
    if (storage_bytes != 2 && storage_bytes != 4) throw Error{CHK_ERR_INVALID, "storage_bytes must be 2 or 4"};
    if (masked_bits > storage_bytes * 8) throw Error{CHK_ERR_INVALID, "masked_bits exceeds the word width"};
    if (storage_bytes * 8 - masked_bits > 31)
        throw Error{CHK_ERR_CAPACITY, "at least one bit of a 32-bit word must be masked (token ids are 31-bit)"};
    if (numel >= (1ull << 31)) throw Error{CHK_ERR_CAPACITY, "tensor too long for 32-bit token positions"};
}

}  // namespace chkrp

using namespace chkrp;

#define RP_BEGIN try {
#define RP_END                       \
    }                                \
    catch (const chkrp::Error& e) {  \
        chkrp::g_err = e.msg;        \
        return e.code;               \
    }                                \
    catch (const std::exception& e) {\
        chkrp::g_err = e.what();     \
        return CHK_ERR_INVALID;      \
    }                                \
    return CHK_OK;

extern "C" {

const char* chk_repair_last_error(void) { return chkrp::g_err.c_str(); }

int chk_repair_build(int device, const void* h_raw, uint64_t numel, uint32_t storage_bytes, uint32_t masked_bits,
                     uint32_t max_rules, uint32_t* rule_lhs, uint32_t* rule_rhs, uint64_t* rule_freq,
                     uint32_t* n_rules_out, uint64_t* tokens_out, uint64_t* max_pair_frequency_out,
                     uint64_t* tie_rounds_out) {
    RP_BEGIN
    if (!h_raw && numel) throw Error{CHK_ERR_INVALID, "NULL tensor"};
    if (!n_rules_out || !tokens_out) throw Error{CHK_ERR_INVALID, "NULL output"};
    check_args(numel, storage_bytes, masked_bits);
    RP_CUDA(cudaSetDevice(device));
    Workspace& w = workspace_for(device);
    std::lock_guard<std::mutex> lock(w.mu);
    w.init((uint32_t)numel, numel * storage_bytes);
    upload_raw(w, h_raw, numel * storage_bytes);
    if (numel && max_rules && max_rules < kDense && storage_bytes * 8 - masked_bits <= kTileBits &&
        build_on_tiles(w, (uint32_t)numel, storage_bytes, masked_bits, max_rules, rule_lhs, rule_rhs, rule_freq, n_rules_out,
                       tokens_out, max_pair_frequency_out, tie_rounds_out))
        return CHK_OK;
    w.init_contiguous((uint32_t)numel);
    mask_tokens(w, numel, storage_bytes, masked_bits);
    uint32_t* cur = w.tok_a.as<uint32_t>();
    uint32_t* nxt = w.tok_b.as<uint32_t>();
    uint32_t n = (uint32_t)numel, n_rules = 0;
    uint64_t max_freq = 0, tie_rounds = 0;
    for (uint32_t r = 0; r < max_rules; ++r) {
        if (n < 2) break;
        RP_CUDA(cudaMemsetAsync(w.keys.p, 0xFF, (size_t)w.capacity * 8, w.s));
        RP_CUDA(cudaMemsetAsync(w.counts.p, 0, (size_t)w.capacity * 4, w.s));
        RP_CUDA(cudaMemsetAsync(w.first.p, 0xFF, (size_t)w.capacity * 4, w.s));
        RP_CUDA(cudaMemsetAsync(w.small.p, 0, 64, w.s));
        uint32_t* small = w.small.as<uint32_t>();  // [0] best, [1] ties, [2] overflow, [3] dump count
        pair_count_kernel<<<grid_for(n), 256, 0, w.s>>>(cur, n, w.keys.as<unsigned long long>(), w.counts.as<uint32_t>(),
                                                        w.first.as<uint32_t>(), w.capacity - 1, small + 2);
        pair_max_kernel<<<grid_for(w.capacity), 256, 0, w.s>>>(w.counts.as<uint32_t>(), w.capacity, small);
        pair_ties_kernel<<<grid_for(w.capacity), 256, 0, w.s>>>(w.keys.as<unsigned long long>(), w.counts.as<uint32_t>(),
                                                                w.first.as<uint32_t>(), w.capacity, small,
                                                                w.tie_keys.as<unsigned long long>(),
                                                                w.tie_first.as<uint32_t>());
        RP_CUDA(cudaGetLastError());
        uint32_t h_small[4];
        unsigned long long h_tie_keys[8];
        RP_CUDA(cudaMemcpyAsync(h_small, small, 16, cudaMemcpyDeviceToHost, w.s));
        RP_CUDA(cudaMemcpyAsync(h_tie_keys, w.tie_keys.p, 64, cudaMemcpyDeviceToHost, w.s));
        RP_CUDA(cudaStreamSynchronize(w.s));
        if (h_small[2]) throw Error{CHK_ERR_CAPACITY, "pair table overflow"};
        const uint32_t best = h_small[0];
        if (best > max_freq) max_freq = best;
        if (best < 2) break;  // k_min_rule_frequency
        unsigned long long key = h_tie_keys[0];
        if (h_small[1] > 1) {
            // several pairs share the maximum: replay the reference's map to see which it meets first
            ++tie_rounds;
            if (!w.dump_keys.p) {
                w.dump_keys.alloc((size_t)w.contiguous_cap * 8 + 8);
                w.dump_counts.alloc((size_t)w.contiguous_cap * 4 + 4);
                w.dump_first.alloc((size_t)w.contiguous_cap * 4 + 4);
            }
            pair_dump_kernel<<<grid_for(w.capacity), 256, 0, w.s>>>(
                w.keys.as<unsigned long long>(), w.counts.as<uint32_t>(), w.first.as<uint32_t>(), w.capacity, small + 3,
                w.dump_keys.as<unsigned long long>(), w.dump_counts.as<uint32_t>(), w.dump_first.as<uint32_t>());
            RP_CUDA(cudaGetLastError());
            uint32_t d = 0;
            RP_CUDA(cudaMemcpyAsync(&d, small + 3, 4, cudaMemcpyDeviceToHost, w.s));
            RP_CUDA(cudaStreamSynchronize(w.s));
            std::vector<unsigned long long> hk(d);
            std::vector<uint32_t> hc(d), hf(d);
            RP_CUDA(cudaMemcpy(hk.data(), w.dump_keys.p, (size_t)d * 8, cudaMemcpyDeviceToHost));
            RP_CUDA(cudaMemcpy(hc.data(), w.dump_counts.p, (size_t)d * 4, cudaMemcpyDeviceToHost));
            RP_CUDA(cudaMemcpy(hf.data(), w.dump_first.p, (size_t)d * 4, cudaMemcpyDeviceToHost));
            key = first_in_map_order(hk, hc, hf, n, masked_bits);
        }
        const uint32_t lhs = (uint32_t)(key >> 32), rhs = (uint32_t)key, sym = kRuleBase + n_rules;
        const uint32_t m = apply_rule(w, cur, n, lhs, rhs, sym, nxt);
        if (m >= n) break;  // no shrink: the rule is not kept (:440-443)
        std::swap(cur, nxt);
        n = m;
        if (rule_lhs) rule_lhs[n_rules] = lhs;
        if (rule_rhs) rule_rhs[n_rules] = rhs;
        if (rule_freq) rule_freq[n_rules] = best;
        ++n_rules;
    }
    *n_rules_out = n_rules;
    *tokens_out = n;
    if (max_pair_frequency_out) *max_pair_frequency_out = max_freq;
    if (tie_rounds_out) *tie_rounds_out = tie_rounds;
    RP_END
}

int chk_repair_apply(int device, const void* h_raw, uint64_t numel, uint32_t storage_bytes, uint32_t masked_bits,
                     const uint32_t* rule_lhs, const uint32_t* rule_rhs, uint32_t n_rules, uint64_t* tokens_out) {
    RP_BEGIN
    if ((!h_raw && numel) || !tokens_out) throw Error{CHK_ERR_INVALID, "NULL argument"};
    if (n_rules && (!rule_lhs || !rule_rhs)) throw Error{CHK_ERR_INVALID, "NULL rules"};
    check_args(numel, storage_bytes, masked_bits);
    RP_CUDA(cudaSetDevice(device));
    Workspace& w = workspace_for(device);
    std::lock_guard<std::mutex> lock(w.mu);
    uint32_t n = (uint32_t)numel;
    if (!n || !n_rules) {
        *tokens_out = n;
        return CHK_OK;
    }
    w.init(n, numel * storage_bytes);
    upload_raw(w, h_raw, numel * storage_bytes);
    std::vector<uint2> rules(n_rules);
    bool on_tiles = storage_bytes * 8 - masked_bits <= 15 && n_rules < kRuleToken;  // 16-bit tokens
    for (uint32_t r = 0; r < n_rules && on_tiles; ++r)
        on_tiles = token_of_id(rule_lhs[r], &rules[r].x) && token_of_id(rule_rhs[r], &rules[r].y);
    if (on_tiles) {
        const TileParams P = tile_params(w, n, n_rules);
        RP_CUDA(cudaMemcpyAsync(P.rules, rules.data(), (size_t)n_rules * 8, cudaMemcpyHostToDevice, w.s));
        RP_CUDA(cudaMemsetAsync(P.state, 0, sizeof(RoundState), w.s));
        tile_words_kernel<false><<<P.n_tiles, kTileThreads, sizeof(TileCountSmem), w.s>>>(w.raw.as<uint8_t>(), numel, storage_bytes,
                                                                                          masked_bits, P);
        for (uint32_t r = 0; r < n_rules; ++r)
            launch_overlapping(w.s, tile_rule_kernel<false>, P.n_tiles, sizeof(TileCountSmem), P, r);
        launch_overlapping(w.s, tile_total_kernel, 1, 0, P, n_rules & 1u);
        RoundState st{};
        RP_CUDA(cudaMemcpyAsync(&st, P.state, sizeof(st), cudaMemcpyDeviceToHost, w.s));
        RP_CUDA(cudaStreamSynchronize(w.s));
        n = st.n_tokens;
    } else {
        w.init_contiguous(n);
        mask_tokens(w, numel, storage_bytes, masked_bits);
        uint32_t* cur = w.tok_a.as<uint32_t>();
        uint32_t* nxt = w.tok_b.as<uint32_t>();
        for (uint32_t r = 0; r < n_rules; ++r) {
            n = apply_rule(w, cur, n, rule_lhs[r], rule_rhs[r], kRuleBase + r, nxt);
            std::swap(cur, nxt);
        }
    }
    *tokens_out = n;
    RP_END
}

}  // extern "C"
