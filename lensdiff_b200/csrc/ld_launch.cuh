// ld_launch.cuh — kernels launched ahead of the stream (programmatic dependent
// launch): a kernel launched by launch_after() is set up as soon as the CTAs of
// the kernel before it on the stream have exited; its first statement,
// stream_order(), waits until that kernel has completed and its writes are
// visible.  Each wait follows the previous kernel's, so a kernel runs its body
// after everything that was before it on the stream, as with a plain launch.
//
// What it saved when it came is the launch between the short kernels of a pass:
// 1024x576 with 3 wavelengths, cold (14 kernels), 77 -> 70 us; 3 x 3 zones at
// 1917x803 (80 kernels) 935 -> 917 us; UHD with 31 wavelengths, cold, 706 -> 696
// us.
// No kernel lets its successor start earlier (launch_dependents): the waiting
// CTAs then hold shared memory and registers that the other stream's kernels
// could use, and the successor's CTAs crowd the SMs that drain first.  With
// that, UHD warm took 335 us instead of 304 and the zones 968 (allowed in every
// kernel) or 1017 us (allowed in grids of up to four CTAs per SM).
#pragma once

#include <cuda_runtime.h>

namespace ld {

// First statement of every kernel launched by launch_after().  (Nothing to
// wait for in a plain launch.)
__device__ __forceinline__ void stream_order() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A call's launches (per thread).  The first launch on a stream, and the first
// after another stream's, is a plain one: the kernel before it is the caller's,
// which need not itself have waited for the one before.  So are launches into a
// caller's capture, whose graph then holds only plain edges (the edge queries
// of the older API refuse others); the library's own captures are `own`.
class LaunchScope {
public:
    explicit LaunchScope(bool own) : outer_(current()) { current() = {true, own, false, nullptr}; }
    ~LaunchScope() { current() = outer_; }
    LaunchScope(const LaunchScope&) = delete;
    LaunchScope& operator=(const LaunchScope&) = delete;

    static bool ahead(cudaStream_t s) {
        State& c = current();
        if (!c.on) return false;
        if (!c.any || c.last != s) {
            c.any = true;
            c.last = s;
            return false;
        }
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (!c.own) cudaStreamIsCapturing(s, &cap);
        return cap == cudaStreamCaptureStatusNone;
    }

private:
    struct State {
        bool on, own, any;
        cudaStream_t last;
    };
    static State& current() {
        static thread_local State c{false, false, false, nullptr};
        return c;
    }
    State outer_;
};

template <class... P, class... A>
void launch_after(void (*f)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = LaunchScope::ahead(s) ? 1 : 0;
    cudaLaunchKernelEx(&cfg, f, P(args)...);
}

}  // namespace ld
