// isp_tails.hpp - which frame is the last work of each stream: a host-side
// register without CUDA calls of its own.
//
// A frame that follows on its stream waits for the event of the frame that was
// queued last there instead of its own pipeline's last one. Both come earlier in
// the stream, so either order is right; but when nothing was queued since, the
// wait is for the stream's last operation, which costs nothing and leaves the
// frame's kernels free to start under that frame's end (frame_overlap),
// whichever camera it belongs to. With the cameras of a rig in turn on one
// stream, each waiting for its own last frame, no two frames overlapped. If the
// caller queued other work since, the wait keeps the frame behind all of it,
// unless that work lets its dependents start early; this library's own kernels
// that do (launch_dependent) take the stream's entry away, and a frame that finds
// none does not overlap: it may read what they write.
#pragma once

#include <atomic>
#include <cstddef>
#include <cstdint>
#include <map>
#include <mutex>
#include <tuple>

namespace isp_b200 {

// A place in the order of queued work. Outside captures the stream, by its id,
// which unlike a handle is never used again. In a capture the graph node that
// the stream's next work will depend on: an entry then stands for as long as
// nothing else is captured behind its frame.
struct StreamKey {
  int device = -1;                 // -1: unknown (or, capturing, not behind exactly one node)
  unsigned long long capture = 0;  // the capture's id
  unsigned long long at = 0;       // the stream's id, or the node
  bool capturing = false;          // or possibly so
  bool known() const { return device >= 0; }
  friend bool operator<(const StreamKey& a, const StreamKey& b) {
    return std::tie(a.device, a.capture, a.at) < std::tie(b.device, b.capture, b.at);
  }
};

// At most one entry per frame owner (a live pipeline), removed when its next
// frame goes elsewhere or it is destroyed.
template <class Owner>
class StreamTails {
 public:
  struct Tail {
    Owner* owner;
    uintptr_t out_begin, out_end;  // the frame's image
  };

  // Calls f(tail) with the register locked, so that the owner stays alive;
  // false when there is no entry.
  template <class F>
  bool find(const StreamKey& key, F f) {
    std::lock_guard<std::mutex> lock(mutex_);
    const auto it = tails_.find(key);
    if (!key.known() || it == tails_.end()) return false;
    f(it->second);
    return true;
  }

  void set(const StreamKey& key, const Tail& tail) {
    std::lock_guard<std::mutex> lock(mutex_);
    remove(tail.owner);
    if (key.known()) {
      const auto it = tails_.find(key);
      if (it != tails_.end()) places_.erase(it->second.owner);
      tails_[key] = tail;
      places_[tail.owner] = key;
    }
    count_ = tails_.size();
  }

  void drop(Owner* owner) {
    std::lock_guard<std::mutex> lock(mutex_);
    remove(owner);
    count_ = tails_.size();
  }

  // Takes the entry at `key` away, or every entry when the place is unknown.
  void forget(const StreamKey& key) {
    std::lock_guard<std::mutex> lock(mutex_);
    if (key.known()) {
      const auto it = tails_.find(key);
      if (it != tails_.end()) remove(it->second.owner);
    } else {
      tails_.clear();
      places_.clear();
    }
    count_ = tails_.size();
  }

  // Without the lock: whether there is anything to forget.
  bool empty() const { return count_ == 0; }

 private:
  void remove(Owner* owner) {
    const auto it = places_.find(owner);
    if (it == places_.end()) return;
    tails_.erase(it->second);
    places_.erase(it);
  }

  std::mutex mutex_;
  std::map<StreamKey, Tail> tails_;
  std::map<Owner*, StreamKey> places_;
  std::atomic<size_t> count_{0};
};

}  // namespace isp_b200
