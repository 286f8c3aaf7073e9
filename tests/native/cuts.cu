// Deals the edges of random graphs, some with nodes of very many, out to the blocks of the kernels by node and
// checks that every edge half is in one block's stretch, that a cut node's stretches are those its first and last
// cut say, and that no stretch is longer than two steps.  Arguments: seed, trials.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <vector>

#include "zp_rotate.cuh"

int main(int argc, char **argv) {
  std::mt19937 rng(std::atoi(argv[1]));
  auto pick = [&](int lo, int hi) { return std::uniform_int_distribution<int>(lo, hi)(rng); };
  int cut_nodes = 0;
  for (int trial = 0; trial < std::atoi(argv[2]); ++trial) {
    const int N = pick(0, 2) ? pick(1, 400) : pick(1, 4), E = pick(0, 4) ? pick(0, 6000) : pick(0, 40);
    const int hub = pick(0, N - 1), hubs = pick(0, 3), outside = pick(0, 2) ? 0 : pick(0, 3);
    std::vector<std::vector<int>> in(N), out(N);
    std::vector<int> src, dst, left;
    for (int e = 0; e < E; ++e) {
      if (outside && pick(0, 9) < outside) { left.push_back(e); continue; }
      in[hubs & 1 && pick(0, 2) ? hub : pick(0, N - 1)].push_back(e);
    }
    std::vector<int32_t> row_ptr(1, 0), row_ptr_src(1, 0), view;
    int slot = 0;
    for (int n = 0; n < N; ++n) {
      for (size_t i = 0; i < in[n].size(); ++i) out[hubs & 2 && pick(0, 2) ? hub : pick(0, N - 1)].push_back(slot++);
      row_ptr.push_back(slot);
    }
    for (; slot < E; ++slot) out[0].push_back(slot);        // left out: count for source 0
    for (int n = 0; n < N; ++n) {
      view.insert(view.end(), out[n].begin(), out[n].end());
      row_ptr_src.push_back((int)view.size());
    }
    for (int both = 0; both < 2; ++both) {
      const int parts = 1 << pick(0, 2);
      const NodeCut cut = zp_node_cut(N, E, both, parts);
      if (cut.cuts >= kZpNodeCuts || (int64_t)cut.cuts > zp_node_cut(1, E, true, 1).cuts) return std::puts("cuts"), 1;
      std::vector<int> into(E, 0), from(E, 0);
      std::map<int, int> stretches;
      std::map<int, std::pair<uint32_t, uint32_t>> said;
      for (int b = 0; b < (int)cut.blocks(); ++b) {
        const NodeEdges s(b, cut, E, row_ptr.data(), both ? view.data() : nullptr, row_ptr_src.data());
        const bool tail = b >= cut.ends();
        if (s.first > s.last || s.first < 0 || s.last > s.total || s.last - s.first > 2 * (int)cut.step) return std::puts("stretch"), 1;
        if (s.n < 0 || s.n > N || s.row(cut) >= N || (!tail && s.n != b / parts)) return std::puts("node"), 1;
        if (s.edge(s.last) != -1) return std::puts("end"), 1;
        for (int i = s.first; i < s.last; ++i) {
          const int e = s.edge(i);
          if (e < 0 || e >= E) return std::puts("edge"), 1;
          if (i < s.own ? into[e]++ || (s.n < N ? e < row_ptr[s.n] || e >= row_ptr[s.n + 1] : e < row_ptr[N])
                        : from[e]++ != 0)
            return std::puts("twice"), 1;
        }
        if (s.cut0 > s.cut1) continue;
        said[s.n] = {s.cut0, s.cut1};
        // as the kernel numbers what follows a cut
        const uint32_t k = (uint32_t)(b - cut.ends() + 1);
        if (tail && s.last > s.first && (k < s.cut0 || k > s.cut1)) return std::puts("number"), 1;
        if (tail ? s.last > s.first : b % parts == 0) ++stretches[s.n];
      }
      for (int e = 0; e < E; ++e)
        if (into[e] != 1 || from[e] != (both ? 1 : 0)) return std::puts("left out"), 1;
      for (auto &[n, cuts] : said) {
        ++cut_nodes;
        if (cuts.first < 1 || cuts.second > cut.cuts || stretches[n] != (int)(cuts.second - cuts.first) + 2) return std::puts("count"), 1;
      }
    }
  }
  std::puts(cut_nodes > 100 ? "ok" : "none cut");
}
