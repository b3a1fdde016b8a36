// A stand-in for the stream and event calls, for host-only tests: every call
// is written to `calls`; the one numbered `fail_at` (from 0) fails.
#pragma once

#include <string>
#include <vector>

enum cudaError_t { cudaSuccess = 0, cudaErrorUnknown = 999 };
constexpr unsigned cudaEventDisableTiming = 2, cudaStreamNonBlocking = 1;

struct Handle {
    std::string name;
};
using cudaStream_t = Handle*;
using cudaEvent_t = Handle*;

inline std::vector<std::string> calls;
inline int fail_at = -1, n_calls = 0, n_made = 0, n_destroyed = 0;
inline cudaError_t last_error = cudaSuccess;

inline cudaError_t call(const std::string& what)
{
    const bool bad = n_calls++ == fail_at;
    calls.push_back(what + (bad ? " fails" : ""));
    if (bad) { last_error = cudaErrorUnknown; }
    return bad ? cudaErrorUnknown : cudaSuccess;
}
inline cudaError_t make(const char* kind, Handle** out)
{
    const std::string name = kind + std::to_string(n_made);
    const cudaError_t e = call("create " + name);
    if (e == cudaSuccess) {
        *out = new Handle{name};
        ++n_made;
    }
    return e;
}
inline cudaError_t drop(Handle* h)
{
    ++n_destroyed;
    delete h;
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return make("event", e); }
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return make("stream", s); }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { return drop(e); }
inline cudaError_t cudaStreamDestroy(cudaStream_t s) { return drop(s); }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return call("record " + e->name + " on " + s->name); }
inline cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
{
    return call(s->name + " waits for " + e->name);
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) { return call("host waits for " + s->name); }
inline cudaError_t cudaGetLastError()
{
    const cudaError_t e = last_error;
    last_error = cudaSuccess;
    return e;
}
