"""A kernel that fails late, for tests of what its successors do: it lets the next launch of the stream start, waits a
millisecond and only then sets the device's error word, as a kernel whose own wait runs out does."""
import ctypes as C

SRC = r"""
extern "C" __global__ void late_failure(int* word, int code, long long cycles) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long t0 = clock64();
    for (int i = 0; i < (1 << 20) && clock64() - t0 < cycles; ++i) {}
    if (threadIdx.x == 0) atomicExch(word, code);
}
"""
_fn = None


def _ok(r):
    assert int(r[0]) == 0, r[0]
    return r[1] if len(r) == 2 else r[1:]


def late_failure(pkg, code, cycles=2000000):
    """Enqueues the kernel on torch's current stream."""
    global _fn
    import torch
    from cuda.bindings import driver, nvrtc
    if _fn is None:
        prog = _ok(nvrtc.nvrtcCreateProgram(SRC.encode(), b"late.cu", 0, [], []))
        _ok(nvrtc.nvrtcCompileProgram(prog, 1, [b"--gpu-architecture=sm_100a"]) + (None,))
        image = b" " * _ok(nvrtc.nvrtcGetCUBINSize(prog))
        _ok(nvrtc.nvrtcGetCUBIN(prog, image) + (None,))
        _fn = _ok(driver.cuModuleGetFunction(_ok(driver.cuModuleLoadData(image)), b"late_failure"))
    word = pkg.lib["_ZN2o117device_error_wordEv"]        # o1::device_error_word()
    word.restype, word.argtypes = C.c_void_p, []
    args = ((word(), int(code), int(cycles)), (C.c_void_p, C.c_int, C.c_longlong))
    _ok(driver.cuLaunchKernel(_fn, 1, 1, 1, 32, 1, 1, 0, torch.cuda.current_stream().cuda_stream, args, 0) + (None,))
