// Elimination plans of the 1-D cascade's direct solves (batch_ls.cu).
//
// A pipe network is a tree with a few loops, so Gaussian elimination in an order
// that takes nodes of low degree first creates almost no fill: nodes of degree
// one and two leave a core of at most twice the loops, and eliminating up to
// degree kLsPlanDegree shrinks it further. The plan is that order written out
// for one sparsity pattern: rounds of independent nodes (no two adjacent), each a
// list of divisions and a list of updates whose targets differ, and the core that
// is left, which is solved densely. Diagonal pivots throughout; the kernel checks
// every multiplier and hands a system that needs row exchanges to the dense path.
//
// Values live in numbered slots: the pattern's entries (closed under transposition,
// the added ones zero), the fill, then one slot per row for the right-hand side,
// which the solution replaces.
#pragma once

#include <cstdint>
#include <utility>
#include <vector>

namespace cfd {

constexpr int kLsPlanDegree = 4;
constexpr int kLsPlanMaxSlots = 20000;

// Words (uint16) of a round, from `at`:
//   divisions: nl pairs (l, d): v[l] /= v[d]
//   targets:   nt triples (t, first, count): v[t] -= sum of count products,
//              products being pairs (i, j) from word pairs + 2 first
//   solutions: nx quadruples (b, d, first, count): v[b] = (v[b] - sum of count
//              products) / v[d], products from word xpairs + 2 first
struct LsRound {
  int32_t at_l, nl, at_t, nt, pairs, at_x, nx, xpairs;
};

struct LsPlanHead {
  int32_t ok;             // 0: no plan (the dense path)
  int32_t slots, b0;      // slots in all, first right-hand-side slot
  int32_t round0, rounds; // this system's rounds
  int32_t core, at_core;  // core nodes: word at_core + k
  int32_t entries, at_entries;  // core entries: triples (slot, row, col)
  int32_t pad;
  int64_t words;          // this system's first word
};

// Plans one after another.
struct LsPlanSet {
  std::vector<uint16_t> words;
  std::vector<LsRound> rounds;
};

// Scratch of ls_plan_build, kept from one system to the next: with arrays of their
// own for every system the builder spent half its time in the allocator.
struct LsPlanWork {
  struct Nb {  // a neighbour: its node, the slots of the entries to and from it, and, while
    int node, out, in, rev;  // lists only grow, this node's place in the neighbour's list
  };
  struct Update {  // v[target] -= v[i] v[j]; next: the target's next update of its round, -1 the last
    int target, i, j, next;
  };
  struct Round {  // where a round's part of the arrays below begins
    size_t div, upd, node, nb;
  };
  std::vector<Nb> pool;  // neighbour lists in one array
  std::vector<size_t> at;
  std::vector<int> len, room;
  std::vector<int> diag, live, blocked, by_degree[kLsPlanDegree + 1], nodes, first, last, order, place, thin;
  std::vector<char> alive;
  std::vector<std::pair<int, int>> div;
  std::vector<Update> upd;
  std::vector<Nb> nbs;
  std::vector<size_t> nb_end;
  std::vector<Round> rounds;
};

// The plan of one square pattern (rows rp[0..n], local columns), appended to the
// set; init takes the slot of every stored entry. False where the pattern has none
// (the set is as it was).
bool ls_plan_build(int n, const int* rp, const int* col, LsPlanWork& work, LsPlanSet& set, uint16_t* init,
                   LsPlanHead& head);

}  // namespace cfd
