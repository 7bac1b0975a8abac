// Checks of the register of each stream's last frame (csrc/isp_tails.hpp):
// sequences of calls as one or two threads make them, each step's effect exact.
// Prints the name of every failed check; exits 0 when there is none.
#include <cstdio>

#include "isp_tails.hpp"

namespace {

struct Camera {
  isp_b200::StreamKey last;
};
using Tails = isp_b200::StreamTails<Camera>;
using isp_b200::StreamKey;

int failures = 0;

StreamKey stream(unsigned long long id) {
  StreamKey k;
  k.device = 0;
  k.at = id;
  return k;
}

StreamKey node(unsigned long long capture, unsigned long long at) {
  StreamKey k = stream(at);
  k.capture = capture;
  k.capturing = true;
  return k;
}

Camera* last(Tails& t, const StreamKey& k) {
  Camera* found = nullptr;
  t.find(k, [&](const Tails::Tail& tail) { found = tail.owner; });
  return found;
}

void expect(const char* name, Camera* got, Camera* want) {
  if (got == want) return;
  std::printf("%s\n", name);
  ++failures;
}

void frame(Tails& t, Camera& c, const StreamKey& k) {
  Tails::Call call(t, k);
  call.finish({&c, 0, 1}, k, c.last);
  c.last = k;
}

}  // namespace

int main() {
  Camera a, b;
  const StreamKey s = stream(7), other = stream(8), nowhere;
  {
    Tails t;
    frame(t, a, s);
    expect("a frame is its stream's last", last(t, s), &a);
    frame(t, b, s);
    expect("the next camera's frame follows", last(t, s), &b);
    frame(t, b, other);
    expect("a camera is the last of one stream", last(t, s), nullptr);
    expect("the other stream", last(t, other), &b);
    t.forget(s);
    expect("work on another stream leaves it", last(t, other), &b);
    t.forget(other);
    expect("a conversion takes the entry", last(t, other), nullptr);
    frame(t, a, s);
    t.drop(&a, a.last);
    expect("a dropped camera", last(t, s), nullptr);
    frame(t, a, s);
    frame(t, b, nowhere);
    expect("work at an unknown place", last(t, s), nullptr);
    Tails u;
    if (!u.idle()) ++failures, std::printf("idle without a frame\n");
    frame(u, a, s);
    frame(u, b, other);
    u.forget(s);
    if (u.idle()) ++failures, std::printf("idle with a frame\n");
    frame(u, b, s);
    expect("a camera in the place of an ended entry", last(u, s), &b);
    frame(u, a, other);
    expect("the camera of the ended entry", last(u, other), &a);
    u.drop(&a, a.last);
    u.drop(&b, b.last);
    if (!u.idle()) ++failures, std::printf("idle again\n");
  }
  {
    // A frame's call on one thread; the other thread's conversion is launched
    // and announced within it: before or after the frame's kernels, unknown.
    Tails t;
    {
      Tails::Call call(t, s);
      t.forget(s);
      call.finish({&a, 0, 1}, s, a.last);
    }
    expect("a conversion within a frame's call", last(t, s), nullptr);
    // Launched within the call, announced after it.
    frame(t, a, s);
    t.forget(s);
    expect("a conversion announced after the call", last(t, s), nullptr);
    // On another stream.
    {
      Tails::Call call(t, s);
      t.forget(other);
      call.finish({&a, 0, 1}, s, a.last);
    }
    expect("a conversion on another stream", last(t, s), &a);
  }
  {
    // Two frames' calls that overlap: the order of their kernels is unknown.
    Tails t;
    Tails::Call first(t, s);
    Tails::Call second(t, s);
    second.finish({&b, 0, 1}, s, b.last);
    first.finish({&a, 0, 1}, s, a.last);
    expect("two frames at once", last(t, s), nullptr);
  }
  {
    // A call that ends early may have queued its statistics pass.
    Tails t;
    frame(t, a, s);
    { Tails::Call call(t, s); }
    expect("a frame that failed", last(t, s), nullptr);
  }
  {
    // In a capture an entry is good for work captured right behind its frame.
    Tails t;
    frame(t, a, s);
    {
      Tails::Call call(t, node(1, 100));
      call.finish({&b, 0, 1}, node(1, 101), b.last);
    }
    expect("the captured frame", last(t, node(1, 101)), &b);
    expect("another node", last(t, node(1, 102)), nullptr);
    expect("another capture", last(t, node(2, 101)), nullptr);
    expect("outside the capture", last(t, s), &a);
    StreamKey begin;  // of a capture: behind no node
    begin.capturing = true;
    {
      Tails::Call call(t, begin);
      call.finish({&b, 0, 1}, node(3, 100), node(1, 101));
    }
    expect("the first frame of a capture", last(t, node(3, 100)), &b);
    expect("outside that capture", last(t, s), &a);
  }
  return failures == 0 ? 0 : 1;
}
