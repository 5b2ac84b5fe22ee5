// Which way a call of the stand-alone frontend goes: one launch of clusters or two launches. Plain host code, the CUDA calls behind `Api`.
#pragma once
#include <atomic>

namespace mm {

constexpr int kFcCluster = 16;               // CTAs of a cluster (of 8, 8 tokens over 384 experts: 9.4 us, of 16 9.1)

// Tokens of a cluster where one launch is the faster way, 0 where two launches are. `clusters`: what the GPU holds at a time, `grid`: the caller's CTAs.
// A cluster per token wherever the clusters fit (seven on a B200: us in a graph, two launches against one, 7 tokens: 48 experts of 3072 7.1 and 4.7, NVFP4
// 9.1 and 4.8, 384 of 3072 10.0 and 7.7, of 4096 11.1 and 9.0; only one or two tokens of hidden 512 over 128 to 256 experts lose, 0.1 to 0.3).
// Two tokens to a cluster where two launches take longer than a cluster's second token: from hidden 2048 on (8 tokens: 48 experts 5.9 and
// 5.3, 128 6.8 and 6.8, 256 7.5 and 7.3; of 1536 6.5 and 6.8 with 128) and beyond 256 experts (of 512 7.6 and 7.1; 256 6.0 and 6.3), and with two more tokens
// than clusters also from hidden 1536 on (9 tokens: 128 experts 0.4 less) and beyond 192 experts (224 of 512 0.7 less; 192 of 512 level, 128 of 1024
// 0.1 more). A call from Python takes 1.5 us less of the host too.
inline int frontend_cluster_tokens(int tokens, int hidden, int experts, int clusters, int grid) {
    const bool two = hidden >= 2048 || experts > 256 || (tokens > clusters + 1 && (hidden >= 1536 || experts > 192));
    if (tokens > 2 * clusters || (tokens > clusters && !two)) return 0;
    const int per = tokens > clusters ? 2 : 1;
    return kFcCluster * ((tokens + per - 1) / per) <= grid ? per : 0;
}

// How many clusters a device holds at a time. Kept once a query has succeeded (asking takes 0.25 us of a call's 9), by threads in any order; a failed one is
// asked again. The answer is that of the context that asked first: in a later one with fewer SMs it may be too high, which costs time, or the launch
// is refused, which the caller sees. `keep` false (a captured launch is refused only when the graph is made): asked anew.
class KnownClusters {
 public:
    template <typename Ask>
    bool get(bool keep, int* clusters, Ask ask) {
        const int known = keep ? known_.load(std::memory_order_acquire) : 0;
        if (known != 0) { *clusters = known - 1; return true; }
        if (!ask(clusters)) return false;
        if (keep) known_.store(*clusters + 1, std::memory_order_release);
        return true;
    }

 private:
    std::atomic<int> known_{0};              // + 1 (0: not known)
};

// A query that fails or a launch that is refused leaves the two launches, and no error that was not there before.
template <typename Api>
int launch_frontend_by_size(Api& api, int tokens, int hidden, int experts, int grid) {
    if (tokens <= 32 && hidden <= 4096 && experts <= 384) {
        const bool pending = api.error_pending();
        int clusters = 0;
        bool ok = api.clusters(&clusters);
        const int per = ok ? frontend_cluster_tokens(tokens, hidden, experts, clusters, grid) : 0;
        if (per != 0) {
            ok = api.one_launch(per);
            if (ok) return 0;
        }
        if (!ok && !pending) api.clear_error();
    }
    return api.two_launches();
}

}  // namespace mm
