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

// Neighbour lists in one array: a list that outgrows its place moves to the end.
class Lists {
 public:
  Lists(int n, int total) : at_(n, 0), len_(n, 0), room_(n, 0) { pool_.reserve((size_t)4 * total + 64); }
  int size(int i) const { return len_[i]; }
  Nb* begin(int i) { return pool_.data() + at_[i]; }
  Nb* end(int i) { return begin(i) + len_[i]; }
  Nb* find(int i, int node) {
    for (Nb* q = begin(i); q != end(i); ++q)
      if (q->node == node) return q;
    return nullptr;
  }
  void push(int i, const Nb& b) {
    if (len_[i] == room_[i]) {
      const int room = room_[i] ? 2 * room_[i] : 4;
      const size_t to = pool_.size();
      pool_.resize(to + room);
      std::copy(pool_.begin() + at_[i], pool_.begin() + at_[i] + len_[i], pool_.begin() + to);
      at_[i] = to;
      room_[i] = room;
    }
    begin(i)[len_[i]++] = b;
  }
  void drop(int i, int node) {  // keeps the order of the others
    Nb* q = find(i, node);
    std::copy(q + 1, end(i), q);
    --len_[i];
  }

 private:
  std::vector<Nb> pool_;
  std::vector<size_t> at_;
  std::vector<int> len_, room_;
};

struct Update {
  int target, i, j;
};

}  // namespace

void ls_plan_build(int n, const int* rp, const int* col, LsPlanOne& out) {
  out = LsPlanOne{};
  const int k0 = rp[0], nnz = rp[n] - k0;
  std::vector<int> diag(n, kNone);
  int slots = 0;
  out.init.resize(nnz);
  // A pattern this wide has no sparse order worth writing out.
  if (nnz > 8 * n + 64) return;
  Lists adj(n, nnz);
  for (int i = 0; i < n; ++i)
    for (int e = rp[i]; e < rp[i + 1]; ++e) {
      const int j = col[e];
      int* s;
      if (j == i) {
        s = &diag[i];
      } else {
        if (!adj.find(i, j)) {
          adj.push(i, {j, kNone, kNone});
          adj.push(j, {i, kNone, kNone});
        }
        s = &adj.find(i, j)->out;
      }
      if (*s == kNone) {  // a repeated entry adds into the first one's slot
        *s = slots++;
        if (j != i) adj.find(j, i)->in = *s;
      }
      out.init[e - k0] = (uint16_t)*s;
    }
  auto fill = [&](int i, int j) -> int {  // slot (i, j), the pair made where the pattern lacks it
    Nb* q = adj.find(i, j);
    if (q && q->out != kNone && q->in != kNone) return q->out;
    if (!q) {
      adj.push(i, {j, kNone, kNone});
      adj.push(j, {i, kNone, kNone});
      q = adj.find(i, j);
    }
    Nb* r = adj.find(j, i);
    if (q->out == kNone) q->out = r->in = slots++;
    if (q->in == kNone) q->in = r->out = slots++;
    return q->out;
  };
  for (int i = 0; i < n; ++i) {
    if (diag[i] == kNone) diag[i] = slots++;
    for (int q = 0; q < adj.size(i); ++q) fill(i, adj.begin(i)[q].node);
  }
  // Right-hand-side slots are numbered after the fill: bslot(i) = ~i until then.
  auto bslot = [](int i) { return ~i; };
  struct Round {
    std::vector<std::pair<int, int>> div;
    std::vector<Update> upd;
    std::vector<int> nodes;
    std::vector<Nb> nbs;       // the nodes' neighbours when they go
    std::vector<int> nb_end;
  };
  std::vector<Round> rounds;
  std::vector<char> alive(n, 1);
  std::vector<int> blocked(n, -1);
  int left = n;
  for (int r = 0; left > 0; ++r) {
    int lo = n;
    for (int i = 0; i < n; ++i)
      if (alive[i]) lo = std::min(lo, adj.size(i));
    if (lo > kLsPlanDegree) break;
    const int cap = std::max(2, lo);
    Round R;
    for (int deg = 0; deg <= cap; ++deg)
      for (int v = 0; v < n; ++v) {
        if (!alive[v] || adj.size(v) != deg || blocked[v] == r) continue;
        R.nodes.push_back(v);
        blocked[v] = r;
        for (Nb* q = adj.begin(v); q != adj.end(v); ++q) blocked[q->node] = r;
      }
    for (int v : R.nodes) {
      const size_t b = R.nbs.size();
      R.nbs.insert(R.nbs.end(), adj.begin(v), adj.end(v));
      R.nb_end.push_back((int)R.nbs.size());
      for (size_t a = b; a < R.nbs.size(); ++a) {
        const Nb u = R.nbs[a];
        R.div.push_back({u.in, diag[v]});
        R.upd.push_back({bslot(u.node), u.in, bslot(v)});
        for (size_t c = b; c < R.nbs.size(); ++c)
          R.upd.push_back({a == c ? diag[u.node] : fill(u.node, R.nbs[c].node), u.in, R.nbs[c].out});
      }
    }
    for (size_t q = 0, a = 0; q < R.nodes.size(); ++q) {
      for (; a < (size_t)R.nb_end[q]; ++a) adj.drop(R.nbs[a].node, R.nodes[q]);
      alive[R.nodes[q]] = 0;
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
  std::vector<int> count(slots + 1);
  std::vector<Update> sorted;
  for (Round& R : rounds) {
    LsRound d{};
    d.at_l = (int32_t)w.size();
    d.nl = (int32_t)R.div.size();
    for (auto& q : R.div) {
      w.push_back(slot(q.first));
      w.push_back(slot(q.second));
    }
    // by target, the order within a target kept
    std::fill(count.begin(), count.end(), 0);
    for (Update& q : R.upd) {
      q.target = slot(q.target);
      count[q.target + 1]++;
    }
    for (int k = 0; k < slots; ++k) count[k + 1] += count[k];
    sorted.resize(R.upd.size());
    for (const Update& q : R.upd) sorted[count[q.target]++] = q;
    R.upd.swap(sorted);
    std::vector<uint16_t> pairs;
    d.at_t = (int32_t)w.size();
    for (size_t q = 0; q < R.upd.size();) {
      const size_t first = q;
      while (q < R.upd.size() && R.upd[q].target == R.upd[first].target) {
        pairs.push_back(slot(R.upd[q].i));
        pairs.push_back(slot(R.upd[q].j));
        ++q;
      }
      w.push_back((uint16_t)R.upd[first].target);
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
      const int b = q ? R.nb_end[q - 1] : 0;
      w.push_back((uint16_t)(R.nb_end[q] - b));
      for (int a = b; a < R.nb_end[q]; ++a) {
        pairs.push_back(slot(R.nbs[a].out));
        pairs.push_back(slot(bslot(R.nbs[a].node)));
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
    for (Nb* u = adj.begin(i); u != adj.end(i); ++u) {
      w.push_back(slot(u->out));
      w.push_back((uint16_t)place[i]);
      w.push_back((uint16_t)place[u->node]);
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
