// Device constants of geometries (correction factors, twiddles), shared between
// calls and plans.
//
// Unplanned calls: the first KEPT geometries are kept for the life of the process
// (a captured graph of a call may use them at any time); beyond that a call makes
// its own.  Plans: an entry is shared with the calls' and the other plans' of the
// same geometry; the last RECENT ones of a device are kept for plans to come (about
// 16 bytes per cell of the oversampled axes each; a batch of 64 different plans that
// is made again and again finds all of its own) and the
// oldest is given up first, freed when no plan holds it any more.  Plans take no
// place of the calls': a program that makes many different plans does not make its
// unplanned calls upload every time.
#pragma once

#include <cstddef>
#include <list>
#include <map>
#include <memory>
#include <mutex>
#include <utility>

namespace dnufft {

// make(): a new V, complete before it returns (other host threads and streams may
// use it at once).  drop(V &): called before the last reference to an entry goes.
template <typename Key, typename V> class ConstTable {
 public:
  static constexpr size_t KEPT = 32, RECENT = 128;
  using Ptr = std::shared_ptr<V>;

  // for an unplanned call; null: no place left
  template <typename Make> const V *for_call(const Key &k, int dev, Make make) {
    std::lock_guard<std::mutex> lk(mu_);
    const auto it = kept_.find(k);
    if (it != kept_.end()) return it->second.get();
    if (kept_.size() >= KEPT) return nullptr;
    const Ptr *p = find_recent(k, dev);
    return (kept_[k] = p ? *p : Ptr(make())).get();
  }

  // for a plan, which gives the pointer back to release()
  template <typename Make, typename Drop> Ptr for_plan(const Key &k, int dev, Make make, Drop drop) {
    std::lock_guard<std::mutex> lk(mu_);
    const auto it = kept_.find(k);
    if (it != kept_.end()) return it->second;
    if (const Ptr *p = find_recent(k, dev)) return *p;
    auto &l = recent_[dev];
    l.emplace_front(k, Ptr(make()));
    Ptr p = l.front().second;
    if (l.size() > RECENT) {
      if (l.back().second.use_count() == 1) drop(*l.back().second);
      l.pop_back();
    }
    return p;
  }

  template <typename Drop> void release(Ptr &p, Drop drop) {
    std::lock_guard<std::mutex> lk(mu_);
    if (p && p.use_count() == 1) drop(*p);
    p.reset();
  }

 private:
  using List = std::list<std::pair<Key, Ptr>>;

  const Ptr *find_recent(const Key &k, int dev) {   // and move it to the front
    List &l = recent_[dev];
    for (auto it = l.begin(); it != l.end(); ++it)
      if (!(it->first < k) && !(k < it->first)) {
        l.splice(l.begin(), l, it);
        return &l.front().second;
      }
    return nullptr;
  }

  std::mutex mu_;
  std::map<Key, Ptr> kept_;
  std::map<int, List> recent_;   // by device, the last used first
};

}  // namespace dnufft
