// batch_lanes.hpp — side streams for the small launches of one batch.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace tgp {

// The lanes of one batch's small launches (fewer tiles than SMs: 15-20 us each
// of mostly latency, most SMs idle): next() gives the stream of the following
// one in turn (the context's own among them), by pointing ctx->stream at it;
// join() puts the context's stream back, behind every lane. Launches that fill
// the SMs stay one after another: their CTAs split the rows evenly and expect
// to start together, and side by side (three queries over 22M-30M rows) took
// 0.39 ms instead of 0.34. Off while launches are profiled (their events
// bracket one stream).
template <class Ctx>
class BatchLanes {
  public:
    explicit BatchLanes(Ctx* c, size_t launches) : ctx(c), main(c->stream) {
        if (launches < 3 || c->profile) return;
        bool ok = c->fork || cudaEventCreateWithFlags(&c->fork, cudaEventDisableTiming) == cudaSuccess;
        for (int i = 0; ok && i < Ctx::kLanes; ++i)
            ok = (c->lane[i] || cudaStreamCreateWithFlags(&c->lane[i], cudaStreamNonBlocking) == cudaSuccess) &&
                 (c->join[i] || cudaEventCreateWithFlags(&c->join[i], cudaEventDisableTiming) == cudaSuccess);
        if (!ok || cudaEventRecord(c->fork, main) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        on = true;
    }
    ~BatchLanes() { join(); }
    void next() {
        if (!on) return;
        at = (at + 1) % (Ctx::kLanes + 1);
        ctx->stream = main;
        if (at == 0) return;
        // A lane's first launch runs behind the fork (the batch's upload); a
        // lane that cannot be made to wait for it is not used.
        if (!used[at - 1] && cudaStreamWaitEvent(ctx->lane[at - 1], ctx->fork, 0) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        used[at - 1] = true;
        ctx->stream = ctx->lane[at - 1];
    }
    // False when a lane could not be joined (its work may still run).
    bool join() {
        ctx->stream = main;
        bool ok = true;
        for (int i = 0; i < Ctx::kLanes; ++i) {
            if (!used[i]) continue;
            used[i] = false;
            if (cudaEventRecord(ctx->join[i], ctx->lane[i]) != cudaSuccess ||
                cudaStreamWaitEvent(main, ctx->join[i], 0) != cudaSuccess)
                ok = cudaStreamSynchronize(ctx->lane[i]) == cudaSuccess && ok;
        }
        return ok;
    }

  private:
    Ctx* ctx;
    cudaStream_t main;
    bool on = false;
    bool used[Ctx::kLanes] = {};
    int at = -1;
};

}  // namespace tgp
