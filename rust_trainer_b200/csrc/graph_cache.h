// Which batch shapes are kept as captured graphs.
#pragma once
#include <algorithm>
#include <optional>
#include <utility>
#include <vector>

namespace rt {

// Up to MAX graphs, least recently used first.  A shape is worth capturing (a whole step's capture, instantiation and, with
// all places taken, the destruction of another graph) when it comes again among the last MAX distinct shapes: only then
// will its graph still be there the next time.  Whoever cycles through more shapes than that launches them
// eagerly and keeps the graphs there are.  (Captured whenever a shape had ever been met before, a cycle of more than
// MAX shapes paid all of that on every pass for a single replay: 28 layers of the 0.6B shape, one sequence of 200 to 264
// tokens, MAX = 32: a cycle of 64 lengths 11.2 ms a pass, 6.5 eagerly; of 32, all replayed, 6.1.)
template <class Shape, class Graph, size_t MAX>
class GraphCache {
 public:
  // the shape's graph, now the most recently used, or null
  Graph* find(const Shape& s) {
    for (size_t i = 0; i < graphs_.size(); ++i)
      if (graphs_[i].first == s) {
        std::rotate(graphs_.begin() + i, graphs_.begin() + i + 1, graphs_.end());
        touch(s);
        return &graphs_.back().second;
      }
    return nullptr;
  }
  bool worth_capturing(const Shape& s) const { return std::find(recent_.begin(), recent_.end(), s) != recent_.end(); }
  // the shape has been met; the oldest of more than MAX is forgotten
  void touch(const Shape& s) {
    auto it = std::find(recent_.begin(), recent_.end(), s);
    if (it != recent_.end()) recent_.erase(it);
    else if (recent_.size() >= MAX) recent_.erase(recent_.begin());
    recent_.push_back(s);
  }
  // keeps a graph and gives back the one that had to go
  std::optional<Graph> put(const Shape& s, const Graph& g) {
    std::optional<Graph> out;
    if (graphs_.size() >= MAX) {
      out = graphs_.front().second;
      graphs_.erase(graphs_.begin());
    }
    graphs_.emplace_back(s, g);
    touch(s);
    return out;
  }
  template <class F>
  void for_each(F f) {
    for (auto& e : graphs_) f(e.second);
  }

 private:
  std::vector<std::pair<Shape, Graph>> graphs_;
  std::vector<Shape> recent_;  // distinct, most recent last, with a graph or without
};

}  // namespace rt
