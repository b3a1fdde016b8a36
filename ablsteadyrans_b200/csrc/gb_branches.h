// Side streams between a fork and a join (host only).
#pragma once

#include <cuda_runtime.h>

namespace gb {

//! The side streams and events of one owner, made on first use.
struct SideStreams {
    static constexpr int kSides = 4;
    cudaStream_t side[kSides]{};
    cudaEvent_t fork_ev{nullptr};
    cudaEvent_t join_ev[kSides]{};
    int made{-1};        // -1: not yet; 0: could not be made
    bool forked{false};  // between a fork and its join
    SideStreams() = default;
    SideStreams(const SideStreams&) = delete;
    SideStreams& operator=(const SideStreams&) = delete;
    ~SideStreams()
    {
        for (int n = 0; n < kSides; ++n) {
            if (side[n]) { cudaStreamDestroy(side[n]); }
            if (join_ev[n]) { cudaEventDestroy(join_ev[n]); }
        }
        if (fork_ev) { cudaEventDestroy(fork_ev); }
    }
    bool ready()
    {
        if (made >= 0) { return made > 0; }
        bool ok = cudaEventCreateWithFlags(&fork_ev, cudaEventDisableTiming) == cudaSuccess;
        for (int n = 0; n < kSides && ok; ++n) {
            ok = cudaStreamCreateWithFlags(&side[n], cudaStreamNonBlocking) == cudaSuccess
                 && cudaEventCreateWithFlags(&join_ev[n], cudaEventDisableTiming) == cudaSuccess;
        }
        if (!ok) { cudaGetLastError(); }
        made = ok ? kSides : 0;
        return ok;
    }
};

//! Launch sequences that do not depend on one another, each on a stream of its
//! own between a fork and a join: on(b) makes `stream` (the variable launches
//! read theirs from) branch b's, 0 the main one's; join() makes the main stream
//! wait for all of them. Every side stream starts after the work queued before
//! the fork and the main stream goes on after the join, so callers see one
//! stream. Under capture the branches become parallel paths of the graph.
//! A step that cannot be queued costs the overlap and never the order: without
//! the fork's event there is one stream, a branch that cannot wait for it stays
//! on the main stream, and one that the main stream cannot wait for is waited
//! for by the host.
class SideBranches {
public:
    SideBranches(SideStreams& s, cudaStream_t& stream, bool wanted) : s_(s), stream_(stream), main_(stream)
    {
        if (!wanted || s.forked || !s.ready()) { return; }
        open_ = s.forked = queued(cudaEventRecord(s.fork_ev, main_));
    }
    SideBranches(const SideBranches&) = delete;
    SideBranches& operator=(const SideBranches&) = delete;
    ~SideBranches() { join(); }
    void on(int b)
    {
        if (!open_) { return; }
        stream_ = main_;
        if (b == 0 || (refused_ & (1u << b))) { return; }
        if (!(used_ & (1u << b))) {
            if (!queued(cudaStreamWaitEvent(s_.side[b - 1], s_.fork_ev, 0))) {
                refused_ |= 1u << b;
                return;
            }
            used_ |= 1u << b;
        }
        stream_ = s_.side[b - 1];
    }
    //! Branch b alone: the main stream goes on after what it was sent so far.
    void join(int b)
    {
        if (!open_) { return; }
        stream_ = main_;
        if (!(used_ & (1u << b))) { return; }
        if (!queued(cudaEventRecord(s_.join_ev[b - 1], s_.side[b - 1]))
            || !queued(cudaStreamWaitEvent(main_, s_.join_ev[b - 1], 0))) {
            cudaStreamSynchronize(s_.side[b - 1]);  // (its error, if any, is the call's)
        }
    }
    void join()
    {
        if (!open_) { return; }
        for (int b = 1; b <= SideStreams::kSides; ++b) { join(b); }
        open_ = s_.forked = false;
    }

private:
    static bool queued(cudaError_t e)
    {
        if (e != cudaSuccess) { cudaGetLastError(); }
        return e == cudaSuccess;
    }
    SideStreams& s_;
    cudaStream_t& stream_;
    cudaStream_t main_;
    unsigned used_{0};
    unsigned refused_{0};
    bool open_{false};
};

}  // namespace gb
