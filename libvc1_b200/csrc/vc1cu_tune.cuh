// vc1cu_tune.cuh - which launch a tuned shape belongs to, and which of the tried shapes a launch keeps
// (host code; vc1cu_autotune and launch_group in vc1cu_api.cu).
#pragma once

#include <map>
#include <utility>
#include <vector>

namespace vc1cu {

// One pass of a launch, as far as the launch's best shape depends on it.
struct TunePass {
    int W, H, mode, allow_intra;
};

// The launches that share a tuned shape: same search configuration, instantiation and MV modes, and as
// many passes of each raster. The passes' number decides how many macroblocks a wavefront step holds,
// and with it the best shape (one 1080p picture wants one block per SM, 24 of them two).
inline std::vector<int> tune_key(int range, int local_range, int me_algorithm, int kind, const std::vector<TunePass>& passes) {
    int modes = 0;
    std::map<std::pair<int, int>, int> rasters;
    for (const TunePass& p : passes) {
        modes |= 1 << (2 * p.mode + (p.allow_intra ? 1 : 0));
        ++rasters[{p.W, p.H}];
    }
    std::vector<int> key{range, local_range, me_algorithm, kind, modes};
    for (const auto& r : rasters) key.insert(key.end(), {r.first.first, r.first.second, r.second});
    return key;
}

// The times of one launch under the tried shapes; below zero: the shape does not fit it.
struct TuneTrial {
    std::vector<int> key;
    std::vector<double> ms;
};

// Each key's best shape (its index; -1 where none fits): launches of one call may share a key (two steps
// of a seed chain), and then take the shape that is fastest for them together.
inline std::map<std::vector<int>, int> tune_choice(const std::vector<TuneTrial>& trials) {
    std::map<std::vector<int>, std::vector<double>> sum;
    for (const TuneTrial& t : trials) {
        auto it = sum.find(t.key);
        if (it == sum.end()) {
            sum[t.key] = t.ms;
            continue;
        }
        for (size_t s = 0; s < t.ms.size(); ++s) it->second[s] = it->second[s] < 0 || t.ms[s] < 0 ? -1.0 : it->second[s] + t.ms[s];
    }
    std::map<std::vector<int>, int> best;
    for (const auto& k : sum) {
        int b = -1;
        for (size_t s = 0; s < k.second.size(); ++s)
            if (k.second[s] >= 0 && (b < 0 || k.second[s] < k.second[b])) b = (int)s;
        best[k.first] = b;
    }
    return best;
}

}  // namespace vc1cu
