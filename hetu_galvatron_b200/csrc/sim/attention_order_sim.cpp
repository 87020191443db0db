// Host-side check of the order of events in the attention forward kernel (attention_sm100.cu): every interleaving of the issuing
// thread, the tensor core (products in order) and two softmax warps is walked for a tile of n key blocks. Reported:
//   stuck : somebody waits for a phase that has passed or will never come;
//   early : O is read or rescaled before the products it needs, or a score buffer is written over what is still needed.
// The phases waited for are the kernel's (include/gv_attn_order.h); `--schedule single` puts one barrier in their place, with the
// last wait by way of the product before, and `--schedule direct` without, to show that the check sees both hazards.
//
//   g++ -std=c++17 -O1 attention_order_sim.cpp -o attention_order_sim && ./attention_order_sim --blocks 5 [--schedule single|direct]
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>
#include <string>
#include <vector>

#include "../include/gv_attn_order.h"

namespace {

constexpr int WARPS = 2;
enum Schedule { KERNEL, SINGLE, DIRECT };

struct Barrier {                      // an mbarrier: completed phases, arrivals of the current one
  int done = 0, arrived = 0;
  void arrive(int expected) {
    if (++arrived == expected) { arrived = 0; ++done; }
  }
  bool passes(unsigned parity) const { return (done & 1u) != parity; }
};

struct State {
  int issuer = 0;                     // step of the issuing thread
  int warp[WARPS] = {};               // step of each softmax warp
  bool rescale[WARPS] = {};           // the warp has decided to rescale O in its current block
  std::vector<int> queue;             // issued, not finished: j = S of block j, -1 - j = P V of block j
  int s_issued = 0, s_done = 0, pv_done = 0;
  int p_given[WARPS] = {};            // blocks whose P the warp has handed over
  Barrier s_full[2], p_full[2], pv[2];
  std::string key() const {
    std::string k;
    auto put = [&](int v) { k += static_cast<char>(v + 64); };
    put(issuer); put(s_issued); put(s_done); put(pv_done);
    for (int w = 0; w < WARPS; ++w) { put(warp[w]); put(rescale[w]); put(p_given[w]); }
    for (int b = 0; b < 2; ++b)
      for (const Barrier* x : {&s_full[b], &p_full[b], &pv[b]}) { put(x->done); put(x->arrived); }
    for (int q : queue) put(q);
    return k;
  }
};

struct Checker {
  int n;
  Schedule sched;
  std::set<std::string> seen;
  long stuck = 0, early = 0;

  gv::PvPhase phase(int block) const { return sched == KERNEL ? gv::pv_phase(block) : gv::PvPhase{0, block & 1u}; }
  bool pv_passes(const State& s, int block) const { return s.pv[phase(block).barrier].passes(phase(block).parity); }

  // Issuer: step 0 is S of block 0; then per block j (steps 1 + 2 j, 2 + 2 j): S of j + 1, P V of j.
  bool issuer_step(const State& s, State& t) {
    if (s.issuer > 2 * n) return false;
    t = s;
    if (s.issuer == 0) {
      t.queue.push_back(t.s_issued++);
    } else if (s.issuer % 2 == 1) {
      const int j = (s.issuer - 1) / 2;
      if (j + 1 < n) {
        if (j > 0) {
          if (!pv_passes(s, j - 1)) return false;
          if (s.pv_done < j) ++early;                        // the buffer still holds P of block j - 1
        }
        t.queue.push_back(t.s_issued++);
      }
    } else {
      const int j = (s.issuer - 2) / 2;
      if (!s.p_full[j & 1].passes((j >> 1) & 1)) return false;
      for (int w = 0; w < WARPS; ++w)
        if (s.p_given[w] <= j) ++early;                      // a warp's P is not there yet
      t.queue.push_back(-1 - j);
    }
    ++t.issuer;
    return true;
  }

  bool tensor_step(const State& s, State& t) {
    if (s.queue.empty()) return false;
    t = s;
    const int op = t.queue.front();
    t.queue.erase(t.queue.begin());
    if (op >= 0) { ++t.s_done; t.s_full[op & 1].arrive(1); }
    else { ++t.pv_done; t.pv[phase(-1 - op).barrier].arrive(1); }
    return true;
  }

  // Softmax warp, per block j: step 3 j waits for S and decides, 3 j + 1 rescales, 3 j + 2 hands over P; then the waits of the end.
  // `want` is the decision where there is one (block 0 never rescales).
  bool warp_step(const State& s, int w, bool want, State& t) {
    t = s;
    const int step = s.warp[w];
    if (step < 3 * n) {
      const int j = step / 3;
      if (step % 3 == 0) {
        if (!s.s_full[j & 1].passes((j >> 1) & 1)) return false;
        if (s.s_done <= j) ++early;
        if (s.s_issued > j + 2) ++early;                     // somebody writes over the scores
        t.rescale[w] = want && j > 0;
      } else if (step % 3 == 1) {
        if (s.rescale[w]) {
          if (!pv_passes(s, j - 1)) return false;
          if (s.pv_done < j) ++early;
        }
        t.rescale[w] = false;
      } else {
        ++t.p_given[w];
        t.p_full[j & 1].arrive(WARPS);
      }
    } else if (step == 3 * n) {
      if (sched == SINGLE && n > 1 && !pv_passes(s, n - 2)) return false;
    } else if (step == 3 * n + 1) {
      if (!pv_passes(s, n - 1)) return false;
      if (s.pv_done < n) ++early;                            // O is read
    } else {
      return false;
    }
    ++t.warp[w];
    return true;
  }

  void walk(const State& start) {
    std::vector<State> todo{start};
    seen.insert(start.key());
    while (!todo.empty()) {
      const State s = todo.back();
      todo.pop_back();
      bool moved = false;
      auto go = [&](bool ok, const State& t) {
        if (!ok) return;
        moved = true;
        if (seen.insert(t.key()).second) todo.push_back(t);
      };
      State t;
      bool ok = issuer_step(s, t);
      go(ok, t);
      ok = tensor_step(s, t);
      go(ok, t);
      for (int w = 0; w < WARPS; ++w)
        for (int want = 0; want < 2; ++want) {
          ok = warp_step(s, w, want != 0, t);
          go(ok, t);
        }
      if (moved) continue;
      bool finished = s.issuer > 2 * n;
      for (int w = 0; w < WARPS; ++w) finished = finished && s.warp[w] == 3 * n + 2;
      if (!finished) ++stuck;
    }
  }
};

}  // namespace

int main(int argc, char** argv) {
  Checker c{1, KERNEL, {}, 0, 0};
  for (int i = 1; i + 1 < argc; i += 2) {
    if (!strcmp(argv[i], "--blocks")) c.n = atoi(argv[i + 1]);
    if (!strcmp(argv[i], "--schedule")) c.sched = !strcmp(argv[i + 1], "single") ? SINGLE : !strcmp(argv[i + 1], "direct") ? DIRECT : KERNEL;
  }
  c.walk(State());
  printf("{\"blocks\": %d, \"states\": %zu, \"stuck\": %ld, \"early\": %ld}\n", c.n, c.seen.size(), c.stuck, c.early);
  return c.stuck || c.early ? 1 : 0;
}
