// A second, high-priority stream beside the caller's, for the dependent chain of
// a factorisation while the caller's stream carries the bulk of its updates.
#pragma once
#include "common.cuh"

namespace mnpb {

struct Fork {
    cudaStream_t p;            // non-blocking, highest priority
    cudaEvent_t ep, es;        // recorded on p, on the caller's stream
    int dev;
};

// Takes a Fork of the current device from a pool for the time of one call.  None
// (get() is null, the caller runs everything on its own stream) while `s` is being
// captured, which would outlive the lease, or when kForks of the device are in
// use.  A Fork goes back with its last user's work still queued: the next user's
// follows it in stream order.
class ForkLease {
  public:
    explicit ForkLease(cudaStream_t s);
    ~ForkLease();
    ForkLease(const ForkLease &) = delete;
    ForkLease &operator=(const ForkLease &) = delete;
    Fork *get() const { return f_; }

  private:
    Fork *f_;
};

// Work queued on `to` from here on follows all that `from` holds now.
inline int stream_after(cudaStream_t to, cudaStream_t from, cudaEvent_t ev) {
    if (cudaEventRecord(ev, from) != cudaSuccess || cudaStreamWaitEvent(to, ev, 0) != cudaSuccess) {
        set_error("stream ordering failed: %s", cudaGetErrorString(cudaGetLastError()));
        return MNPB_ECUDA;
    }
    return MNPB_OK;
}

// The right-hand sides [0, m) in two halves (`cut`), the first on a second stream:
// part(stream, first, end) does [first, end).  The halves meet at a multiple of 64;
// up to 64 right-hand sides are one part.  Without a second stream the halves follow
// each other: a product may be summed in another order when its size is another, and
// the result must not depend on whether the pool had a stream left.
template <typename F>
inline int in_halves(cudaStream_t s, int m, bool cut, F part) {
    const int h = ceil_div(m, 128) * 64;
    if (!cut || h >= m) return part(s, 0, m);
    ForkLease lease(s);
    const Fork *f = lease.get();
    if (f) MNPB_TRY(stream_after(f->p, s, f->es));
    int rc = part(f ? f->p : s, 0, h);
    if (rc == MNPB_OK) rc = part(s, h, m);
    const int rj = f ? stream_after(s, f->p, f->ep) : MNPB_OK;   // also after an error
    return rc != MNPB_OK ? rc : rj;
}

}  // namespace mnpb
