// Host construction of the elimination plans (ls_plan.h).
#include "ls_plan.h"

#include <algorithm>

namespace cfd {
namespace {

constexpr int kNone = -1;

using Nb = LsPlanWork::Nb;

// The neighbour lists: a list that outgrows its place moves to the end.
class Lists {
 public:
  Lists(LsPlanWork& w, int n, int total) : w_(w) {
    w_.at.assign(n, 0);
    w_.len.assign(n, 0);
    w_.room.assign(n, 0);
    w_.pool.clear();
    w_.pool.reserve((size_t)4 * total + 64);
  }
  int size(int i) const { return w_.len[i]; }
  Nb* begin(int i) { return w_.pool.data() + w_.at[i]; }
  Nb* end(int i) { return begin(i) + w_.len[i]; }
  Nb* find(int i, int node) {
    for (Nb* q = begin(i); q != end(i); ++q)
      if (q->node == node) return q;
    return nullptr;
  }
  // i and j neighbours of each other, no slots yet.
  void join(int i, int j) {
    const int a = w_.len[i], b = w_.len[j];
    push(i, {j, kNone, kNone, b});
    push(j, {i, kNone, kNone, a});
  }
  // Drops the dead nodes of list i, the order of the others kept.
  void compact(int i) {
    Nb* e = std::remove_if(begin(i), end(i), [&](const Nb& q) { return !w_.alive[q.node]; });
    w_.len[i] = (int)(e - begin(i));
  }

 private:
  void push(int i, const Nb& b) {
    if (w_.len[i] == w_.room[i]) {
      const int room = w_.room[i] ? 2 * w_.room[i] : 4;
      const size_t to = w_.pool.size();
      w_.pool.resize(to + room);
      std::copy(w_.pool.begin() + w_.at[i], w_.pool.begin() + w_.at[i] + w_.len[i], w_.pool.begin() + to);
      w_.at[i] = to;
      w_.room[i] = room;
    }
    begin(i)[w_.len[i]++] = b;
  }
  LsPlanWork& w_;
};

}  // namespace

bool ls_plan_build(int n, const int* rp, const int* col, LsPlanWork& work, LsPlanSet& set, uint16_t* init,
                   LsPlanHead& head) {
  head = LsPlanHead{};
  const int k0 = rp[0], nnz = rp[n] - k0;
  // A pattern this wide has no sparse order worth writing out.
  if (nnz > 8 * n + 64) return false;
  int slots = 0;
  auto& diag = work.diag;
  diag.assign(n, kNone);
  Lists adj(work, n, nnz);
  // place[j]: where j stands in the list of the row at hand
  auto& place = work.place;
  place.assign(n, kNone);
  for (int i = 0; i < n; ++i) {
    for (int k = 0; k < adj.size(i); ++k) place[adj.begin(i)[k].node] = k;
    for (int e = rp[i]; e < rp[i + 1]; ++e) {
      const int j = col[e];
      int* s = &diag[i];
      if (j != i) {
        if (place[j] == kNone) {
          place[j] = adj.size(i);
          adj.join(i, j);
        }
        s = &adj.begin(i)[place[j]].out;
      }
      if (*s == kNone) {  // a repeated entry adds into the first one's slot
        *s = slots++;
        if (j != i) adj.begin(j)[adj.begin(i)[place[j]].rev].in = *s;
      }
      init[e - k0] = (uint16_t)*s;
    }
    for (Nb* q = adj.begin(i); q != adj.end(i); ++q) place[q->node] = kNone;
  }
  // the pattern closed under transposition, every diagonal entry there
  for (int i = 0; i < n; ++i) {
    if (diag[i] == kNone) diag[i] = slots++;
    for (Nb* q = adj.begin(i); q != adj.end(i); ++q) {
      Nb& r = adj.begin(q->node)[q->rev];
      if (q->out == kNone) q->out = r.in = slots++;
      if (q->in == kNone) q->in = r.out = slots++;
    }
  }
  // Slot (i, j), the pair made where it is missing; looked for in the shorter list.
  auto fill = [&](int i, int j) -> int {
    const bool swap = adj.size(j) < adj.size(i);
    if (const Nb* q = swap ? adj.find(j, i) : adj.find(i, j)) return swap ? q->in : q->out;
    adj.join(i, j);
    Nb &q = adj.end(i)[-1], &r = adj.end(j)[-1];
    q.out = r.in = slots++;
    q.in = r.out = slots++;
    return q.out;
  };
  // Right-hand-side slots are numbered after the fill: bslot(i) = ~i until then.
  auto bslot = [](int i) { return ~i; };
  auto& div = work.div;
  auto& upd = work.upd;
  auto &nodes = work.nodes, &live = work.live, &blocked = work.blocked;
  auto& nbs = work.nbs;  // the nodes' neighbours when they go
  auto& nb_end = work.nb_end;
  auto& rounds = work.rounds;
  auto& alive = work.alive;
  auto& thin = work.thin;
  div.clear();
  upd.clear();
  nodes.clear();
  nbs.clear();
  nb_end.clear();
  rounds.clear();
  live.resize(n);
  for (int i = 0; i < n; ++i) live[i] = i;
  constexpr int kSeen = -2;
  blocked.assign(n, -1);
  alive.assign(n, 1);
  for (int r = 0; !live.empty(); ++r) {
    int lo = n;
    for (auto& q : work.by_degree) q.clear();
    for (int v : live) {
      const int d = adj.size(v);
      lo = std::min(lo, d);
      if (d <= kLsPlanDegree) work.by_degree[d].push_back(v);
    }
    if (lo > kLsPlanDegree) break;
    const LsPlanWork::Round R{div.size(), upd.size(), nodes.size(), nbs.size()};
    for (int deg = 0; deg <= std::max(2, lo); ++deg)
      for (int v : work.by_degree[deg]) {
        if (blocked[v] == r) continue;
        nodes.push_back(v);
        blocked[v] = r;
        for (Nb* q = adj.begin(v); q != adj.end(v); ++q) blocked[q->node] = r;
      }
    for (size_t q = R.node; q < nodes.size(); ++q) {
      const int v = nodes[q];
      const size_t b = nbs.size();
      nbs.insert(nbs.end(), adj.begin(v), adj.end(v));
      nb_end.push_back(nbs.size());
      for (size_t a = b; a < nbs.size(); ++a) {
        const Nb u = nbs[a];
        div.push_back({u.in, diag[v]});
        upd.push_back({bslot(u.node), u.in, bslot(v), kNone});
        for (size_t c = b; c < nbs.size(); ++c)
          upd.push_back({a == c ? diag[u.node] : fill(u.node, nbs[c].node), u.in, nbs[c].out, kNone});
      }
    }
    for (size_t q = R.node; q < nodes.size(); ++q) alive[nodes[q]] = 0;
    thin.clear();
    for (size_t a = R.nb; a < nbs.size(); ++a)
      if (blocked[nbs[a].node] == r) {  // a neighbour, not yet looked at
        blocked[nbs[a].node] = kSeen;
        thin.push_back(nbs[a].node);
      }
    for (int v : thin) adj.compact(v);
    live.erase(std::remove_if(live.begin(), live.end(), [&](int v) { return !alive[v]; }), live.end());
    rounds.push_back(R);
    if (slots + n > kLsPlanMaxSlots) return false;
  }
  const int b0 = slots;
  slots += n;
  if (slots > kLsPlanMaxSlots || 2 * (int)live.size() > n) return false;
  auto slot = [&](int s) { return s < 0 ? b0 + ~s : s; };
  for (size_t q = 0; q < rounds.size(); ++q)
    if ((q + 1 == rounds.size() ? upd.size() : rounds[q + 1].upd) - rounds[q].upd > 65535) return false;
  auto& w = set.words;  // offsets are from this system's first word
  head.words = (int64_t)w.size();
  head.round0 = (int32_t)set.rounds.size();
  const size_t w0 = w.size();
  auto &first = work.first, &last = work.last, &order = work.order;
  first.assign(slots, kNone);
  last.resize(slots);
  for (size_t q = 0; q < rounds.size(); ++q) {
    const LsPlanWork::Round& R = rounds[q];
    const bool end = q + 1 == rounds.size();
    const size_t div_e = end ? div.size() : rounds[q + 1].div, upd_e = end ? upd.size() : rounds[q + 1].upd;
    const size_t node_e = end ? nodes.size() : rounds[q + 1].node, nb_e = end ? nbs.size() : rounds[q + 1].nb;
    // by target, the order within a target kept
    order.clear();
    for (size_t u = R.upd; u < upd_e; ++u) {
      const int t = slot(upd[u].target);
      if (first[t] == kNone) {
        first[t] = (int)u;
        order.push_back(t);
      } else {
        upd[last[t]].next = (int)u;
      }
      last[t] = (int)u;
    }
    LsRound d{};
    d.nl = (int32_t)(div_e - R.div);
    d.nt = (int32_t)order.size();
    d.nx = (int32_t)(node_e - R.node);
    d.at_l = (int32_t)(w.size() - w0);
    d.at_t = d.at_l + 2 * d.nl;
    d.pairs = d.at_t + 3 * d.nt;
    d.at_x = d.pairs + 2 * (int32_t)(upd_e - R.upd);
    d.xpairs = d.at_x + 4 * d.nx;
    w.resize(w0 + (size_t)d.xpairs + 2 * (nb_e - R.nb));
    uint16_t* const words = w.data() + w0;
    uint16_t* o = words + d.at_l;
    for (size_t k = R.div; k < div_e; ++k) {
      *o++ = (uint16_t)div[k].first;
      *o++ = (uint16_t)div[k].second;
    }
    uint16_t* p = words + d.pairs;
    int at = 0;
    for (int t : order) {
      int count = 0;
      for (int u = first[t]; u != kNone; u = upd[u].next, ++count) {
        *p++ = (uint16_t)slot(upd[u].i);
        *p++ = (uint16_t)slot(upd[u].j);
      }
      first[t] = kNone;
      *o++ = (uint16_t)t;
      *o++ = (uint16_t)at;
      *o++ = (uint16_t)count;
      at += count;
    }
    o = words + d.at_x;
    p = words + d.xpairs;
    size_t a = R.nb;
    at = 0;
    for (size_t k = R.node; k < node_e; ++k) {
      *o++ = (uint16_t)slot(bslot(nodes[k]));
      *o++ = (uint16_t)diag[nodes[k]];
      *o++ = (uint16_t)at;
      *o++ = (uint16_t)(nb_end[k] - a);
      at += (int)(nb_end[k] - a);
      for (; a < nb_end[k]; ++a) {
        *p++ = (uint16_t)nbs[a].out;
        *p++ = (uint16_t)slot(bslot(nbs[a].node));
      }
    }
    set.rounds.push_back(d);
  }
  int core = 0;  // place: the core's numbering from here on
  head.at_core = (int32_t)(w.size() - w0);
  for (int i : live) {
    place[i] = core++;
    w.push_back((uint16_t)i);
  }
  head.at_entries = (int32_t)(w.size() - w0);
  for (int i : live) {
    w.push_back((uint16_t)diag[i]);
    w.push_back((uint16_t)place[i]);
    w.push_back((uint16_t)place[i]);
    for (Nb* u = adj.begin(i); u != adj.end(i); ++u) {
      w.push_back((uint16_t)u->out);
      w.push_back((uint16_t)place[i]);
      w.push_back((uint16_t)place[u->node]);
    }
  }
  head.entries = (int32_t)((w.size() - w0 - head.at_entries) / 3);
  head.core = core;
  head.slots = slots;
  head.b0 = b0;
  head.rounds = (int32_t)rounds.size();
  head.ok = 1;
  return true;
}

}  // namespace cfd
