// Host model of the hand-overs in the prompt attention kernels: every order in which the tensor pipe, the arrivals on the barriers, the
// issuing warp and a softmax warp can proceed, for the waits of nfai_b200/csrc/attn_phases.h, the header that the kernels compile.
//
//   attn_phases_model <kind> <tiles> [skip]
//
// kind 0: scores one tile ahead in two places, two barriers for the products with the values (gqa_prefill_umma.cu)
//      1: scores behind the product before (attn_prefill_umma.cu, heads of 128)
//      2: scores one tile ahead in one place that is handed back (attn_prefill_umma.cu, heads of 64)
// skip (kinds 0, 1): a planted mistake: phases that follow from other barriers are not waited for.
//
// An mbarrier is the number of its phases that have ended; a wait for parity p passes where that number's parity is not p. The pipe
// works in order; an arrival lands at any time after the work before it. Checked in every reachable state: a row's sums are rescaled, and
// read at the end, only when no product with the values is waiting or running, none is left out, nobody waits for good, and all arrivals
// have landed when the softmax warp is through. Exit code 0: all hold; 1: one does not (said on stdout).
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>
#include <string>
#include <vector>

#include "attn_phases.h"

namespace {

enum { S_READY = 0, P_READY = 2, S_FREE = 4, PV_DONE = 5, kBars = 7 };
struct Op {
  enum Kind { WAIT, ARRIVE, WORK, COMMIT, RESCALE, MAYBE } kind;
  int a = 0, b = 0;  // barrier and parity; WORK: 1 + tile for a product with the values; RESCALE: tile; MAYBE: operations to pass over
};
struct State {
  int soft = 0, issue = 0, done = 0;  // operations begun by either warp; work and commits that have left the pipe
  int ended[kBars] = {};
  std::vector<int> landing;           // barriers whose arrivals are on their way
  std::string key() const {
    std::string k;
    for (int v : {soft, issue, done}) k += std::to_string(v) + ",";
    for (int v : ended) k += std::to_string(v) + ",";
    for (int v : std::multiset<int>(landing.begin(), landing.end())) k += "l" + std::to_string(v);
    return k;
  }
};

template <uint32_t BARRIERS>
struct Model {
  using V = nfai::ValuePhases<BARRIERS>;
  std::vector<Op> soft, issue;
  int places;
  Model(int kind, int n, bool skip) : places(kind == 0 ? 2 : 1) {
    auto s_ready = [&](int it) { return Op{Op::WAIT, S_READY + it % places, it / places & 1}; };
    auto value = [&](uint32_t it) { soft.push_back({Op::WAIT, PV_DONE + (int)V::barrier(it), (int)V::parity(it)}); };
    for (int it = 0; it < n; ++it) {
      soft.push_back(s_ready(it));
      if (kind != 2 && !skip) V::at_tile(it, value);
      const size_t maybe = soft.size();
      soft.push_back({Op::MAYBE});
      if (!(skip && kind == 1)) V::at_rescaling(it, value);
      if (it) soft.push_back({Op::RESCALE, it});
      soft[maybe].a = (int)(soft.size() - maybe - 1);
      if (kind == 2) {
        soft.push_back({Op::ARRIVE, S_FREE});
        V::at_tile(it, value);
      }
      soft.push_back({Op::ARRIVE, P_READY + it % places});
    }
    if (skip) value(n - 1);
    else V::at_end(n, value);
    soft.push_back({Op::RESCALE, n});
    auto scores = [&](int it) {
      issue.push_back({Op::WORK, 0});
      issue.push_back({Op::COMMIT, S_READY + it % places});
    };
    scores(0);
    for (int it = 0; it < n; ++it) {
      if (kind != 1 && it + 1 < n) {
        if (kind == 2) issue.push_back({Op::WAIT, S_FREE, it & 1});
        scores(it + 1);
      }
      issue.push_back({Op::WAIT, P_READY + it % places, it / places & 1});
      issue.push_back({Op::WORK, 1 + it});
      issue.push_back({Op::COMMIT, PV_DONE + (int)V::barrier(it)});
      if (kind == 1 && it + 1 < n) scores(it + 1);
    }
  }
  int wrong(const char* what, const State& s) const {
    printf("%s (softmax at %d of %d, issue at %d of %d, pipe at %d)\n", what, s.soft, (int)soft.size(), s.issue, (int)issue.size(), s.done);
    return 1;
  }
  int run() const {
    std::set<std::string> seen;
    std::vector<State> todo(1);
    while (!todo.empty()) {
      State s = todo.back();
      todo.pop_back();
      if (!seen.insert(s.key()).second) continue;
      std::vector<State> next;
      auto passes = [&](const Op& o) { return (s.ended[o.a] & 1) != o.b; };
      if (s.soft < (int)soft.size()) {
        const Op& o = soft[s.soft];
        State t = s;
        ++t.soft;
        if (o.kind == Op::WAIT) {
          if (passes(o)) next.push_back(t);
        } else if (o.kind == Op::RESCALE) {
          int begun = 0, left = 0;  // products with the values that the pipe was given, and that have left it
          for (int i = 0; i < s.issue; ++i)
            if (issue[i].kind == Op::WORK && issue[i].a > 0) ++begun, left += i < s.done;
          if (begun != left || left != o.a) return wrong("sums touched while a product is on its way", s);
          next.push_back(t);
        } else {
          if (o.kind == Op::ARRIVE) ++t.ended[o.a];
          next.push_back(t);
          if (o.kind == Op::MAYBE) {
            t.soft += o.a;
            next.push_back(t);
          }
        }
      }
      if (s.issue < (int)issue.size() && (issue[s.issue].kind != Op::WAIT || passes(issue[s.issue]))) {
        State t = s;
        ++t.issue;
        next.push_back(t);
      }
      if (s.done < s.issue) {  // the pipe: in order; a commit's arrival sets out
        State t = s;
        if (issue[t.done].kind == Op::COMMIT) t.landing.push_back(issue[t.done].a);
        ++t.done;
        next.push_back(t);
      }
      for (size_t i = 0; i < s.landing.size(); ++i) {
        State t = s;
        ++t.ended[t.landing[i]];
        t.landing.erase(t.landing.begin() + i);
        next.push_back(t);
      }
      if (s.soft == (int)soft.size())
        for (int b : s.landing)
          if (b >= PV_DONE) return wrong("an arrival is on its way at the end", s);
      if (next.empty() && (s.soft < (int)soft.size() || s.issue < (int)issue.size())) return wrong("a wait that does not end", s);
      todo.insert(todo.end(), next.begin(), next.end());
    }
    printf("%zu states\n", seen.size());
    return 0;
  }
};

}  // namespace

int main(int argc, char** argv) {
  if (argc < 3) return 2;
  const int kind = atoi(argv[1]), n = atoi(argv[2]);
  const bool skip = argc > 3 && !strcmp(argv[3], "skip");
  if (kind < 0 || kind > 2 || n < 1 || n > 64 || (skip && kind == 2)) return 2;
  if (kind == 0 && !skip) return Model<2>(kind, n, false).run();
  return Model<1>(kind, n, skip).run();
}
