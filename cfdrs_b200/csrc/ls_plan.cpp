// Host construction of the elimination plans (ls_plan.h).
#include "ls_plan.h"

#include <algorithm>

namespace cfd {
namespace {

constexpr int kNone = -1;

// A neighbour j of node i: the slots of entries (i, j) and (j, i).
struct Nb {
  int node, out, in;
};

Nb* find(std::vector<Nb>& a, int node) {
  for (Nb& q : a)
    if (q.node == node) return &q;
  return nullptr;
}

struct Update {
  int target, i, j;
};

}  // namespace

void ls_plan_build(int n, const int* rp, const int* col, LsPlanOne& out) {
  out = LsPlanOne{};
  const int k0 = rp[0], nnz = rp[n] - k0;
  std::vector<std::vector<Nb>> adj(n);
  std::vector<int> diag(n, kNone);
  int slots = 0;
  out.init.resize(nnz);
  // A pattern this wide has no sparse order worth writing out.
  if (nnz > 8 * n + 64) return;
  for (int i = 0; i < n; ++i)
    for (int e = rp[i]; e < rp[i + 1]; ++e) {
      const int j = col[e];
      int* s;
      if (j == i) {
        s = &diag[i];
      } else {
        if (!find(adj[i], j)) {
          adj[i].push_back({j, kNone, kNone});
          adj[j].push_back({i, kNone, kNone});
        }
        s = &find(adj[i], j)->out;
      }
      if (*s == kNone) {  // a repeated entry adds into the first one's slot
        *s = slots++;
        if (j != i) find(adj[j], i)->in = *s;
      }
      out.init[e - k0] = (uint16_t)*s;
    }
  auto fill = [&](int i, int j) -> Nb& {  // the pair's slots, made where the pattern lacks them
    Nb* q = find(adj[i], j);
    if (!q) {
      adj[i].push_back({j, kNone, kNone});
      adj[j].push_back({i, kNone, kNone});
      q = find(adj[i], j);
    }
    Nb* r = find(adj[j], i);
    if (q->out == kNone) q->out = r->in = slots++;
    if (q->in == kNone) q->in = r->out = slots++;
    return *q;
  };
  for (int i = 0; i < n; ++i) {
    if (diag[i] == kNone) diag[i] = slots++;
    for (size_t q = 0; q < adj[i].size(); ++q) fill(i, adj[i][q].node);
  }
  // Right-hand-side slots are numbered after the fill: bslot(i) = ~i until then.
  auto bslot = [](int i) { return ~i; };
  struct Round {
    std::vector<std::pair<int, int>> div;
    std::vector<Update> upd;
    std::vector<int> nodes;
    std::vector<std::vector<Nb>> nbs;
  };
  std::vector<Round> rounds;
  std::vector<char> alive(n, 1);
  std::vector<int> blocked(n, -1);
  int left = n;
  for (int r = 0; left > 0; ++r) {
    size_t lo = SIZE_MAX;
    for (int i = 0; i < n; ++i)
      if (alive[i]) lo = std::min(lo, adj[i].size());
    if (lo > (size_t)kLsPlanDegree) break;
    const size_t cap = std::max<size_t>(2, lo);
    Round R;
    for (size_t deg = 0; deg <= cap; ++deg)
      for (int v = 0; v < n; ++v) {
        if (!alive[v] || adj[v].size() != deg || blocked[v] == r) continue;
        R.nodes.push_back(v);
        blocked[v] = r;
        for (const Nb& q : adj[v]) blocked[q.node] = r;
      }
    for (int v : R.nodes) {
      const std::vector<Nb> nb = adj[v];
      for (const Nb& u : nb) {
        R.div.push_back({u.in, diag[v]});
        R.upd.push_back({bslot(u.node), u.in, bslot(v)});
        for (const Nb& w : nb)
          R.upd.push_back({u.node == w.node ? diag[u.node] : fill(u.node, w.node).out, u.in, w.out});
      }
      R.nbs.push_back(nb);
    }
    for (size_t q = 0; q < R.nodes.size(); ++q) {
      const int v = R.nodes[q];
      for (const Nb& u : R.nbs[q]) {
        auto& a = adj[u.node];
        a.erase(std::find_if(a.begin(), a.end(), [&](const Nb& w) { return w.node == v; }));
      }
      alive[v] = 0;
      --left;
    }
    rounds.push_back(std::move(R));
    if (slots + n > kLsPlanMaxSlots) return;
  }
  const int b0 = slots;
  slots += n;
  if (slots > kLsPlanMaxSlots || 2 * left > n) return;
  auto slot = [&](int s) { return (uint16_t)(s < 0 ? b0 + ~s : s); };
  auto& w = out.words;
  for (Round& R : rounds) {
    LsRound d{};
    d.at_l = (int32_t)w.size();
    d.nl = (int32_t)R.div.size();
    for (auto& q : R.div) {
      w.push_back(slot(q.first));
      w.push_back(slot(q.second));
    }
    std::stable_sort(R.upd.begin(), R.upd.end(), [&](const Update& a, const Update& b) {
      return slot(a.target) < slot(b.target);
    });
    std::vector<uint16_t> pairs;
    d.at_t = (int32_t)w.size();
    for (size_t q = 0; q < R.upd.size();) {
      const size_t first = q;
      while (q < R.upd.size() && R.upd[q].target == R.upd[first].target) {
        pairs.push_back(slot(R.upd[q].i));
        pairs.push_back(slot(R.upd[q].j));
        ++q;
      }
      w.push_back(slot(R.upd[first].target));
      w.push_back((uint16_t)first);
      w.push_back((uint16_t)(q - first));
      d.nt++;
    }
    if (R.upd.size() > 65535) return;
    d.pairs = (int32_t)w.size();
    w.insert(w.end(), pairs.begin(), pairs.end());
    pairs.clear();
    d.at_x = (int32_t)w.size();
    d.nx = (int32_t)R.nodes.size();
    for (size_t q = 0; q < R.nodes.size(); ++q) {
      w.push_back(slot(bslot(R.nodes[q])));
      w.push_back(slot(diag[R.nodes[q]]));
      w.push_back((uint16_t)(pairs.size() / 2));
      w.push_back((uint16_t)R.nbs[q].size());
      for (const Nb& u : R.nbs[q]) {
        pairs.push_back(slot(u.out));
        pairs.push_back(slot(bslot(u.node)));
      }
    }
    d.xpairs = (int32_t)w.size();
    w.insert(w.end(), pairs.begin(), pairs.end());
    out.rounds.push_back(d);
  }
  std::vector<int> place(n, kNone);
  int core = 0;
  out.head.at_core = (int32_t)w.size();
  for (int i = 0; i < n; ++i)
    if (alive[i]) {
      place[i] = core++;
      w.push_back((uint16_t)i);
    }
  out.head.at_entries = (int32_t)w.size();
  for (int i = 0; i < n; ++i) {
    if (!alive[i]) continue;
    w.push_back(slot(diag[i]));
    w.push_back((uint16_t)place[i]);
    w.push_back((uint16_t)place[i]);
    for (const Nb& u : adj[i]) {
      w.push_back(slot(u.out));
      w.push_back((uint16_t)place[i]);
      w.push_back((uint16_t)place[u.node]);
    }
  }
  out.head.entries = (int32_t)(w.size() - out.head.at_entries) / 3;
  out.head.core = core;
  out.head.slots = slots;
  out.head.b0 = b0;
  out.head.rounds = (int32_t)out.rounds.size();
  out.head.ok = 1;
}

}  // namespace cfd
