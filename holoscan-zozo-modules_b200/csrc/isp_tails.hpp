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
// that do (launch_dependent, and the frames of isp_noalloc.cu) end the entry, and a frame that finds
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
//
// Several threads may queue work on one stream, and an entry must not outlive
// work queued behind its frame by another thread. So a frame is queued within a
// Call, other work is announced after its launch (forget), and a frame in whose
// Call anything else was announced at the same place gets no entry: which of the
// two came last on the stream is not known.
template <class Owner>
class StreamTails {
 public:
  struct Tail {
    Owner* owner;
    uintptr_t out_begin, out_end;  // the frame's image
  };

  // From before a frame's first operation until its event is recorded. A Call
  // that ends without that may have queued a part of the frame: no entry stays.
  class Call {
   public:
    Call(StreamTails& tails, const StreamKey& key) : tails_(tails), key_(key) {
      std::lock_guard<std::mutex> lock(tails_.mutex_);
      next_ = tails_.calls_;
      tails_.calls_ = this;
      tails_.recount();
    }
    ~Call() {
      if (finished_) return;
      std::lock_guard<std::mutex> lock(tails_.mutex_);
      leave();
      tails_.announce(key_);
      tails_.recount();
    }
    Call(const Call&) = delete;
    Call& operator=(const Call&) = delete;

    // The frame is queued, and the next work will come at `place` (the Call's
    // own outside captures); `before`: the place after the owner's last frame.
    // Frames in turn on one stream cost no allocation.
    void finish(const Tail& tail, const StreamKey& place, const StreamKey& before) {
      std::lock_guard<std::mutex> lock(tails_.mutex_);
      leave();
      finished_ = true;
      tails_.announce(key_);
      if (disturbed_ || !place.known() || !same(place, before)) tails_.remove(tail.owner, before);
      if (!disturbed_ && place.known()) tails_.put(place, tail);
      tails_.recount();
    }

   private:
    friend class StreamTails;
    void leave() {
      for (Call** c = &tails_.calls_; *c != nullptr; c = &(*c)->next_) {
        if (*c == this) {
          *c = next_;
          break;
        }
      }
    }
    StreamTails& tails_;
    const StreamKey key_;
    Call* next_ = nullptr;
    bool disturbed_ = false;
    bool finished_ = false;
  };

  // Calls f(tail) with the register locked, so that the owner stays alive;
  // false when there is no entry.
  template <class F>
  bool find(const StreamKey& key, F f) {
    std::lock_guard<std::mutex> lock(mutex_);
    const auto it = tails_.find(key);
    if (!key.known() || it == tails_.end() || !it->second.last) return false;
    f(it->second.tail);
    return true;
  }

  // `place`: the place after the owner's last frame.
  void drop(Owner* owner, const StreamKey& place) {
    std::lock_guard<std::mutex> lock(mutex_);
    remove(owner, place);
    recount();
  }

  // Without the lock: whether there is nothing to forget. Asked after the launch
  // of other work, since a frame's Call that begins later queues behind it.
  bool idle() const { return count_ == 0; }

  // Work other than a frame was queued at `key`, by a call that returns after
  // this. Neither allocates nor frees memory.
  void forget(const StreamKey& key) {
    std::lock_guard<std::mutex> lock(mutex_);
    announce(key);
    recount();
  }

 private:
  struct Entry {
    Tail tail{};
    bool last = false;  // nothing was announced behind it
  };

  void put(const StreamKey& key, const Tail& tail) {
    Entry& e = tails_[key];
    if (!e.last) ++last_;
    e = {tail, true};
  }

  void remove(Owner* owner, const StreamKey& place) {
    const auto it = tails_.find(place);
    if (it == tails_.end() || it->second.tail.owner != owner) return;
    bury(it->second);
    tails_.erase(it);
  }

  void bury(Entry& e) {
    if (e.last) --last_;
    e.last = false;
  }

  // Work was queued at `key`, or, when that is unknown, anywhere. (At an unknown
  // place of a capture there is no entry.)
  void announce(const StreamKey& key) {
    if (!key.known() && key.capturing) return;
    for (Call* c = calls_; c != nullptr; c = c->next_) {
      if (!key.known() || !c->key_.known() || same(c->key_, key)) c->disturbed_ = true;
    }
    if (key.known()) {
      const auto it = tails_.find(key);
      if (it != tails_.end()) bury(it->second);
    } else {
      for (auto& t : tails_) bury(t.second);
    }
  }

  static bool same(const StreamKey& a, const StreamKey& b) { return !(a < b) && !(b < a); }
  void recount() { count_ = last_ + (calls_ != nullptr ? 1 : 0); }

  std::mutex mutex_;
  std::map<StreamKey, Entry> tails_;
  Call* calls_ = nullptr;
  size_t last_ = 0;               // entries that are still last
  std::atomic<size_t> count_{0};  // these, and one more while there are Calls
};

}  // namespace isp_b200
