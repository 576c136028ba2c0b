// tree_plan.h -- the chunks of samples that a frame's ray trees are grown in (host code).
//
// The trees of a chunk share a node pool, or half of it where two lanes run.  Chunks are cut from runs of samples
// still to do.  One that fills the pool goes again in halves.  The chunk after one that did not holds as many samples
// as that one's nodes a sample let expect, at most twice as many as it.  After a frame of as many samples the
// chunks are planned by where its nodes were: a frame with more nodes than the pool holds would otherwise
// fill it in vain each time (all-glass scenes at 8 recursions, 18 to 39 rays a sample, 1.2 to 2 times as long).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <utility>
#include <vector>

namespace rg {

// what a frame learned of its chunks: whether one filled a pool of its size, and where its nodes were
struct TreeLoad {
    bool full = false;
    bool again = false;  // the only chunk did, and the frame was left to a larger pool
    std::vector<std::pair<uint32_t, double>> upTo;  // by sample: one past a chunk's last, nodes of all samples before that
    uint32_t samples() const { return upTo.empty() ? 0u : upTo.back().first; }
    double nodes_before(uint32_t sample) const {  // linear within a chunk
        const auto it = std::lower_bound(upTo.begin(), upTo.end(), sample, [](const auto& e, uint32_t s) { return e.first < s; });
        const uint32_t b = it == upTo.begin() ? 0u : (it - 1)->first;
        const double n = it == upTo.begin() ? 0.0 : (it - 1)->second;
        return it == upTo.end() ? n : n + (it->second - n) * ((double)(sample - b) / (it->first - b));
    }
};

class ChunkPlan {
  public:
    // `pool`: nodes of a lane; `nominal`: samples it is meant for
    ChunkPlan(uint32_t work, uint32_t lanes, uint32_t pool, uint32_t nominal, TreeLoad last)
        : pool_(pool), part_(((work + lanes - 1) / lanes + 31) / 32 * 32), nominal_(std::max(1u, nominal)), size_(std::max(1u, std::min(part_, nominal))),
          planned_(last.samples() == work), last_(std::move(last)) {
        if (work) todo_.emplace_back(0u, work);
    }
    // the next chunk; false: none is left to start
    bool next(uint32_t& base, uint32_t& samples) {
        if (todo_.empty()) return false;
        auto& [at, n] = todo_.back();
        base = at;
        samples = std::min(planned_ ? planned(at, n) : even(n), pool_);  // (a root is a node)
        at += samples;
        n -= samples;
        if (!n) todo_.pop_back();
        return true;
    }
    // a chunk of more than one sample filled the pool
    void filled(uint32_t base, uint32_t samples) {
        full_ = full_ || samples <= nominal_;
        planned_ = false;
        todo_.emplace_back(base, samples);
        size_ = (samples + 1) / 2;
    }
    void done(uint32_t base, uint32_t samples, uint32_t nodes) {
        chunks_.push_back({base, samples, nodes});
        const double fit = (pool_ - pool_ / 8u) * ((double)samples / std::max(nodes, 1u));
        size_ = std::max(1u, std::min(part_, (uint32_t)std::min(fit, 2.0 * samples)));
    }
    TreeLoad load() {
        TreeLoad l;
        l.full = full_;
        std::sort(chunks_.begin(), chunks_.end(), [](const Chunk& a, const Chunk& b) { return a.base < b.base; });
        double sum = 0.0;
        for (const Chunk& k : chunks_) l.upTo.emplace_back(k.base + k.samples, sum += k.nodes);
        if (l.samples() == last_.samples()) refine(l);
        return l;
    }

  private:
    struct Chunk {
        uint32_t base, samples, nodes;
    };
    // within its chunks l takes the distribution that the frame before had (its points, 64 over the frame at most)
    void refine(TreeLoad& l) const {
        std::vector<std::pair<uint32_t, double>> more;
        const uint32_t apart = l.samples() / 64u + 1u;
        uint32_t from = 0, at = 0;  // the chunk's first sample, the point before
        auto p = last_.upTo.begin();
        for (const auto& [to, nodes] : l.upTo) {
            const double n0 = l.nodes_before(from), o0 = last_.nodes_before(from), o1 = last_.nodes_before(to);
            for (; p != last_.upTo.end() && p->first < to; ++p)
                if (p->first > from && p->first - at >= apart && to - p->first >= apart && o1 > o0) {
                    more.emplace_back(p->first, n0 + (nodes - n0) * ((p->second - o0) / (o1 - o0)));
                    at = p->first;
                }
            more.emplace_back(to, nodes);
            from = at = to;
        }
        l.upTo = std::move(more);
    }
    // pieces of whole tiles, as equal as `size_` allows
    uint32_t even(uint32_t n) const {
        const uint32_t pieces = (n - 1) / size_ + 1, piece = ((n - 1) / pieces + 1 + 31) / 32 * 32;
        return std::min(std::min(n, size_), piece);
    }
    // the samples from `at` on, all of a lane's where they had no more nodes than 63/64 of the pool, else parts with an equal
    // share of the nodes, at most 7/8 of the pool
    uint32_t planned(uint32_t at, uint32_t n) const {
        n = std::min(n, part_);
        const double before = last_.nodes_before(at), nodes = last_.nodes_before(at + n) - before;
        if (nodes <= pool_ - pool_ / 64u) return n;
        const double want = before + nodes / std::ceil(nodes / (pool_ - pool_ / 8u));
        uint32_t lo = 1, hi = n;
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo + 1) / 2;
            if (last_.nodes_before(at + mid) <= want) lo = mid;
            else hi = mid - 1;
        }
        return lo;
    }

    uint32_t pool_, part_, nominal_, size_;
    bool planned_, full_ = false;
    TreeLoad last_;
    std::vector<std::pair<uint32_t, uint32_t>> todo_;  // runs still to do (first work item, samples)
    std::vector<Chunk> chunks_;                        // done
};

}  // namespace rg
