// How the prompt portions of a step are dealt to the blocks of the tcgen05 prompt attention (csrc/attention_tc5.cu).
//
// A stream of the kernel takes up to `tokens` tokens.  A block of two streams reads keys and values once for both and costs less a
// row; a block of a single stream is done sooner and leaves fewer multiprocessors idle at the end.  So the longest blocks are pairs
// and the rest are not; how many are is what ends first by the costs given, of none, all, and as many as fill the device evenly.
#include <algorithm>
#include <cmath>
#include <functional>
#include <queue>
#include <vector>

#define HOST_API extern "C" __attribute__((visibility("default")))

namespace {

constexpr int KEYS = 128;                 // of a tile of the kernel

struct Wide {                             // tokens of one portion, up to two streams
    int keys, end, first, count;          // tiles of keys they see, position behind the last, first row
};
struct Block {
    double cost;
    int first, count;
};

// Tiles of keys that `count` tokens see whose last one is at position end - 1.
int keys_of(int end, int count, int window) {
    const int from = end - count;
    const int low = window == 0 ? 0 : window > 0 ? std::max(0, from - window + 1) : from / -window * -window;
    return (end - 1) / KEYS - low / KEYS + 1;
}

// When the last of `machines` is done, each taking the next block as it gets free.
double makespan(const std::vector<Block>& blocks, int machines) {
    if ((int)blocks.size() <= machines) return blocks.empty() ? 0.0 : blocks.front().cost;      // sorted, the longest first
    std::priority_queue<double, std::vector<double>, std::greater<double>> free;
    for (int i = 0; i < machines; ++i) free.push(0.0);
    double last = 0.0;
    for (const Block& block : blocks) {
        const double end = free.top() + block.cost;
        free.pop();
        free.push(end);
        last = std::max(last, end);
    }
    return last;
}

void sort_blocks(std::vector<Block>& blocks) {
    std::stable_sort(blocks.begin(), blocks.end(), [](const Block& a, const Block& b) { return a.cost > b.cost; });
}

}  // namespace

// portions: {first row, tokens, position of the first} each; those of up to `longer_than` tokens are left out.  window as in
// first_visible() of the kernels.  blocks_at_once: a kv head's on the device.  Costs in us: of a block whatever its keys, of a tile of keys
// for a pair, for a single stream.  out gets the blocks' first rows, then their tokens, the longest block first; room: the
// blocks it has place for.  Returns the number of blocks, or -1 where they do not fit.
HOST_API int mrun_prompt_blocks(int n, const int* portions, int tokens, int longer_than, int streams, int window, double blocks_at_once,
                                double block_cost, double pair_tile, double single_tile, int* out, int room) {
    std::vector<Wide> wide;
    bool pairs_possible = false;
    for (int i = 0; i < n; ++i) {
        const int row = portions[3 * i], len = portions[3 * i + 1], pos = portions[3 * i + 2];
        if (len <= longer_than) continue;
        for (int t = 0; t < len; t += streams * tokens) {
            const int count = std::min(streams * tokens, len - t), end = pos + t + count;
            wide.push_back({keys_of(end, count, window), end, row + t, count});
            pairs_possible |= count > tokens;
        }
    }
    std::stable_sort(wide.begin(), wide.end(), [](const Wide& a, const Wide& b) { return a.keys != b.keys ? a.keys > b.keys : a.end > b.end; });
    auto deal = [&](int pairs) {
        std::vector<Block> blocks;
        blocks.reserve(2 * wide.size());
        for (int i = 0; i < (int)wide.size(); ++i) {
            const Wide& w = wide[i];
            if (w.count <= tokens) {
                blocks.push_back({single_tile * w.keys + block_cost, w.first, w.count});
            } else if (i < pairs) {
                blocks.push_back({pair_tile * w.keys + block_cost, w.first, w.count});
            } else {
                const int rest = w.count - tokens;
                blocks.push_back({single_tile * keys_of(w.end, rest, window) + block_cost, w.first + tokens, rest});
                blocks.push_back({single_tile * keys_of(w.end - rest, tokens, window) + block_cost, w.first, tokens});
            }
        }
        sort_blocks(blocks);
        return blocks;
    };
    std::vector<Block> best = deal((int)wide.size());
    if (streams == 2 && pairs_possible) {
        const int machines = std::max(1, (int)blocks_at_once);
        const int even = (int)(std::floor(wide.size() / blocks_at_once) * blocks_at_once);
        double ends = makespan(best, machines);
        int before = (int)wide.size();
        for (int pairs : {even, 0}) {
            if (pairs >= before) continue;
            before = pairs;
            std::vector<Block> blocks = deal(pairs);
            const double now = makespan(blocks, machines);
            if (now < ends) {
                ends = now;
                best.swap(blocks);
            }
        }
    }
    const int found = (int)best.size();
    if (found > room) return -1;
    for (int i = 0; i < found; ++i) {
        out[i] = best[i].first;
        out[found + i] = best[i].count;
    }
    return found;
}
