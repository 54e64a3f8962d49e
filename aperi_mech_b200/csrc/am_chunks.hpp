// am_chunks.hpp -- warp-chunk plans of one-thread-per-element blocks, and where the blocks'
// logical slots begin (host code).
//
// The force kernels of such blocks sum, per warp, the nodal forces of the warp's 32 units
// (elements, or split-hex half patches) on each node they share, and write one slot per
// distinct node. The plan built here tells each lane which staged entries it sums, in an
// order fixed by the connectivity's unit order and corner order alone.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

namespace am {

// Warp chunks of a Gauss block of nn-node elements run one thread per element: chunk c
// holds elements [32c, 32c + 32) in the processing order. Its distinct nodes, ranked by first
// appearance over the entry codes q = 32 a + lane (connectivity node a of the chunk's element
// lane), take logical slots ptr[c] + rank. The chunk's entries sorted by (rank, code) go nn to
// a lane, a byte each: words (32 c + l) nn/4 .. (32 c + l + 1) nn/4 - 1 of code / rank hold
// lane l's, rank 0xFF past the chunk's last element. All of it follows from the element order
// and the corner order, not from the node numbers. Fails (false) when a chunk has more than
// 254 distinct nodes, which the rank bytes cannot hold.
struct WarpChunks {
    std::vector<int32_t> ptr, nodes;
    std::vector<uint32_t> code, rank;
};
namespace chunk_detail {

// Chunks [c0, c1) of the plan: their code and rank bytes, their node counts in ptr[c + 1] and
// their nodes, chunk after chunk. The bytes of chunk c begin at 32 nn c, the sorted entry j's at
// byte j there (on a little-endian host the words' bytes in order).
inline bool build_range(const int32_t* conn, int64_t E, int nn, int64_t c0, int64_t c1, uint8_t* code, uint8_t* rank,
                        int32_t* ptr, std::vector<int32_t>& nodes) {
    const int Q = 32 * nn;
    int32_t node[256];
    int count[257];
    uint8_t which[256];
    // rank of the chunk's nodes seen so far by a hash of the node id (linear probing; at most 256
    // of the 1024 places fill up); a place counts when it carries this chunk's stamp
    int64_t stamp[1024];
    uint8_t seen[1024];
    std::fill(stamp, stamp + 1024, int64_t{-1});
    for (int64_t c = c0; c < c1; ++c) {
        const int64_t e0 = 32 * c;
        const int n = static_cast<int>(std::min<int64_t>(32, E - e0));
        int nd = 0;
        for (int a = 0; a < nn; ++a)
            for (int l = 0; l < n; ++l) {
                const int32_t v = conn[nn * (e0 + l) + a];
                uint32_t h = (static_cast<uint32_t>(v) * 2654435761u) >> 22;
                while (stamp[h] == c && node[seen[h]] != v) h = (h + 1) & 1023u;
                if (stamp[h] != c) {
                    if (nd == 254) return false;
                    stamp[h] = c;
                    seen[h] = static_cast<uint8_t>(nd);
                    count[nd + 1] = 0;
                    node[nd++] = v;
                }
                which[32 * a + l] = seen[h];
                ++count[seen[h] + 1];
            }
        // sorted positions by rank: count[k] becomes the first of rank k, then its next
        count[0] = 0;
        for (int k = 0; k < nd; ++k) count[k + 1] += count[k];
        uint8_t* const cb = code + static_cast<int64_t>(Q) * c;
        uint8_t* const rb = rank + static_cast<int64_t>(Q) * c;
        for (int a = 0; a < nn; ++a)
            for (int l = 0; l < n; ++l) {
                const int q = 32 * a + l, j = count[which[q]]++;
                cb[j] = static_cast<uint8_t>(q);
                rb[j] = which[q];
            }
        nodes.insert(nodes.end(), node, node + nd);
        ptr[c + 1] = nd;
    }
    return true;
}

}  // namespace chunk_detail

// The chunks do not depend on one another: ranges of at least kChunkRange of them run on the
// host's threads (at most sixteen). 741,150 tets, eight cores: 45 ms one by one with the words
// shifted together, 25 ms one by one, 6 to 10 ms on eight threads.
constexpr int64_t kChunkRange = 1024;
inline bool build_warp_chunks(const int32_t* conn, int64_t E, int nn, WarpChunks& t) {
    const int64_t C = (E + 31) / 32;
    const size_t words = static_cast<size_t>(32 * (nn / 4) * C);
    t.ptr.assign(C + 1, 0);
    t.nodes.clear();
    t.code.assign(words, 0xFFFFFFFFu);
    t.rank.assign(words, 0xFFFFFFFFu);
    const int64_t hw = std::min<int64_t>(16, std::max(1u, std::thread::hardware_concurrency()));
    const int64_t R = std::min(hw, std::max<int64_t>(1, C / kChunkRange));
    std::vector<std::vector<int32_t>> nodes(R);
    std::vector<char> ok(R, 0);  // 1: built, 0: a chunk beyond the rank bytes, 2: out of memory
    const auto range = [&](int64_t r) noexcept {
        try {
            ok[r] = chunk_detail::build_range(conn, E, nn, C * r / R, C * (r + 1) / R, reinterpret_cast<uint8_t*>(t.code.data()),
                                              reinterpret_cast<uint8_t*>(t.rank.data()), t.ptr.data(), nodes[r]);
        } catch (const std::bad_alloc&) {
            ok[r] = 2;
        }
    };
    std::vector<std::thread> threads;
    threads.reserve(R - 1);
    int64_t r = 1;
    try {
        for (; r < R; ++r) threads.emplace_back(range, r);
    } catch (const std::system_error&) {
        // no more threads: the ranges left run here
    }
    range(0);
    for (; r < R; ++r) range(r);
    for (auto& th : threads) th.join();
    for (char x : ok) {
        if (x == 2) throw std::bad_alloc();
        if (x == 0) return false;
    }
    for (int64_t c = 0; c < C; ++c) t.ptr[c + 1] += t.ptr[c];
    t.nodes.reserve(static_cast<size_t>(t.ptr[C]));
    for (const auto& part : nodes) t.nodes.insert(t.nodes.end(), part.begin(), part.end());
    return true;
}

// First logical slot of each block from the blocks' logical slot counts, and behind them the
// size of the slot-position array. Kernels read a block's positions two and four at a time, so
// every block begins at a multiple of four whatever the blocks before it hold (a warp-chunked,
// per-entry or cell-stress block may hold an odd number); positions in the gaps stay unused.
inline std::vector<int64_t> slot_bases(const std::vector<int64_t>& counts) {
    std::vector<int64_t> base(counts.size() + 1, 0);
    for (size_t k = 0; k < counts.size(); ++k) base[k + 1] = (base[k] + counts[k] + 3) / 4 * 4;
    return base;
}

}  // namespace am
