// Order among the calls that use one buffer of the library (a grouped plan's scratch, a kept pointer
// array), whatever streams they run on. Free of CUDA -- Api supplies streams and events -- so that it is
// unit-tested on the CPU.
//
//   struct Api {
//     using Stream, Event, Error;                 // Error{} is success
//     static Error create(Event&), wait(Stream, Event), record(Event, Stream), sync(Event);
//     static void sync_stream(Stream), destroy(Event);
//     static uint64_t id(Stream);                 // no other stream ever has it; 0 where that is not known
//   };
#pragma once

#include <stdint.h>

namespace ssb {

template <class Api>
struct UseOrder {
  using Stream = typename Api::Stream;
  using Error = typename Api::Error;
  typename Api::Event used{};
  bool made = false;       // `used` exists
  bool in_use = false;     // `used` marks the end of a use

  uint64_t last = 0;       // id of the stream of that use, and from begin() on of the next

  // Before the first use by a call on `st`, which then runs after the use before it. A stream is known by its
  // id, not by its handle: one handle can stand for a stream per host thread (cudaStreamPerThread), and a
  // destroyed stream's handle can come back while its work still runs.
  Error begin(Stream st) {
    if (!made) {
      const Error e = Api::create(used);
      if (e != Error{}) return e;
      made = true;
    }
    const uint64_t id = Api::id(st);
    const Error e = in_use && (id == 0 || id != last) ? Api::wait(st, used) : Error{};
    last = e == Error{} ? id : 0;
    return e;
  }
  // After the last use by that call, on the same stream.
  void end(Stream st) {
    if (Api::record(used, st) == Error{}) {
      in_use = true;
      return;
    }
    Api::sync_stream(st);   // nothing to wait for later, so wait now
  }
  // The host waits until nothing uses the buffer.
  Error idle() {
    if (!in_use) return Error{};
    const Error e = Api::sync(used);
    if (e == Error{}) in_use = false;
    return e;
  }
  void destroy() {
    if (made) Api::destroy(used);
    made = in_use = false;
  }
};

// One call's use of a buffer: ended on every way out of the scope, also where a launch failed after others
// were queued.
template <class Api>
class Use {
 public:
  Use(UseOrder<Api>& order, typename Api::Stream st) : order_(&order), st_(st), error_(order.begin(st)) {}
  ~Use() {
    if (error_ == typename Api::Error{}) order_->end(st_);
  }
  Use(const Use&) = delete;
  Use& operator=(const Use&) = delete;
  typename Api::Error error() const { return error_; }   // of the wait; nothing may be queued then

 private:
  UseOrder<Api>* order_;
  typename Api::Stream st_;
  typename Api::Error error_;
};

}  // namespace ssb
