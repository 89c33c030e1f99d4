// The fibers of tests/emu/warp/cuda_runtime.h: run_cta runs one CTA, its threads taken in ascending or in descending order
// between barriers (what depends on the order is a race). Test infrastructure only.
#pragma once
#include <cstdio>
#include <functional>
#include <vector>

#include <ucontext.h>

#include "cuda_runtime.h"

dim3e threadIdx{0}, blockIdx{0}, blockDim{32};
unsigned char* emu_smem;
uint64_t emu_slot[1024];

namespace {
constexpr size_t kStack = 256 * 1024;
struct Fiber {
    ucontext_t ctx;
    std::vector<char> stack;
    int state = 0;  // 0 runs, 1 at a warp barrier, 2 at the CTA's, 3 done
};
std::vector<Fiber> fibers;
ucontext_t scheduler;
const std::function<void()>* body;
void entry() {
    (*body)();
    fibers[threadIdx.x].state = 3;
    swapcontext(&fibers[threadIdx.x].ctx, &scheduler);
}
void wait_at(int state) {
    const unsigned me = threadIdx.x;
    fibers[me].state = state;
    swapcontext(&fibers[me].ctx, &scheduler);
    threadIdx.x = me;
}
// one CTA of `threads` fibers running f, with `bytes` of dynamic shared memory
void run_cta(int threads, size_t bytes, const std::function<void()>& f, bool descending = false) {
    std::vector<double> smem((bytes + 7) / 8);
    emu_smem = reinterpret_cast<unsigned char*>(smem.data());
    fibers.resize(threads);
    body = &f;
    blockDim.x = threads;
    for (int k = 0; k < threads; ++k) {
        Fiber& b = fibers[k];
        b.stack.resize(kStack);
        getcontext(&b.ctx);
        b.ctx.uc_stack.ss_sp = b.stack.data();
        b.ctx.uc_stack.ss_size = kStack;
        b.ctx.uc_link = nullptr;
        makecontext(&b.ctx, entry, 0);
        b.state = 0;
    }
    for (;;) {
        bool any = false;
        for (int q = 0; q < threads; ++q) {
            const int k = descending ? threads - 1 - q : q;
            if (fibers[k].state == 0) {
                any = true;
                threadIdx.x = k;
                swapcontext(&scheduler, &fibers[k].ctx);
            }
        }
        int done = 0, at_block = 0;
        for (int w = 0; w < threads; w += 32) {
            int at = 0, gone = 0;
            for (int k = w; k < w + 32; ++k) {
                at += fibers[k].state == 1;
                gone += fibers[k].state == 3;
                at_block += fibers[k].state == 2;
            }
            done += gone;
            if (at && at + gone == 32)
                for (int k = w; k < w + 32; ++k)
                    if (fibers[k].state == 1) fibers[k].state = 0, any = true;
        }
        if (done == threads) return;
        if (at_block && at_block + done == threads)
            for (int k = 0; k < threads; ++k)
                if (fibers[k].state == 2) fibers[k].state = 0, any = true;
        if (!any) {
            std::printf("FAIL: the emulated threads wait for one another\n");
            std::exit(1);
        }
    }
}
}  // namespace
void emu_block_sync() { wait_at(2); }
void emu_warp_sync() { wait_at(1); }
