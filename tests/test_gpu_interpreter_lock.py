"""The compiled host path does not hold Python's interpreter lock in its calls of the library.  A stand-in for the library
takes every call, and returns from it only when another Python thread has said so; it gives up after some seconds, which is
what happens if that thread cannot run."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

STAND_IN = textwrap.dedent("""
    #include <atomic>
    #include <chrono>
    #include <thread>
    #include "rm_b200.h"
    static std::atomic<int> entered{0}, go{0};
    static int wait_for_go() {
      entered = 1;
      for (int i = 0; i < 5000 && !go; ++i) std::this_thread::sleep_for(std::chrono::milliseconds(1));
      return go ? RM_OK : RM_ERR_INVALID_ARG;
    }
    extern "C" {
    int stand_in_entered() { return entered; }
    void stand_in_set(int value) { go = value; if (!value) entered = 0; }
    const char* rm_strerror(int) { return "nobody came"; }
    int rm_debug_bounds_checked(void) { return 0; }
    void rm_debug_set_extent(int, int64_t) {}
    size_t rm_bin_workspace_bytes(int64_t, int64_t) { return 256; }
    size_t rm_list_scratch_bytes(int64_t, int, int) { return 256; }
    int rm_project_and_bin_visible(const int32_t*, int64_t, const float*, int64_t, const RmCamera*, int32_t*, int32_t*, float*,
                                   float*, int32_t*, RmBinInfo*, void*, size_t, uint8_t*, RmBinInfo*, void*) { return wait_for_go(); }
    int rm_build_tile_lists(const int32_t*, const int32_t*, int64_t, const RmCamera*, int64_t, int64_t, void*, void*, size_t,
                            int32_t*, void*) { return wait_for_go(); }
    int rm_pack_records_and_clear(const int32_t*, const float*, const float*, int64_t, int64_t, const RmCamera*, const int32_t*,
                                  float*, uint8_t*, uint8_t*, void*) { return wait_for_go(); }
    int rm_forward_sized(const int32_t*, const int32_t*, const float*, const RmCamera*, const float*, float*, float*, int32_t*,
                         const RmHitList*, int64_t, void*) { return wait_for_go(); }
    int rm_backward(const int32_t*, const int32_t*, const float*, const RmCamera*, const float*, const float*, const float*,
                    const int32_t*, const RmHitList*, const float*, const float*, const int32_t*, const float*, const float*,
                    int64_t, int64_t, float*, float*, float*, void*) { return wait_for_go(); }
    int rm_vertex_backward(const int32_t*, const float*, int64_t, int64_t, const RmCamera*, const int32_t*, const float*,
                           const float*, float*, void*) { return wait_for_go(); }
    int rm_tet_err(const int32_t*, const int32_t*, const float*, const RmCamera*, const float*, const float*, int64_t, float*,
                   int32_t*, void*) { return wait_for_go(); }
    int rm_activate_output(const float*, const float*, const float*, const float*, const void*, int, const int32_t*, const float*,
                           const float*, int64_t, int, int, float*, void*) { return wait_for_go(); }
    int rm_distortion_loss(const float*, int64_t, float*, float*, void*) { return wait_for_go(); }
    int rm_distortion_loss_backward(const float*, int64_t, const float*, float*, void*) { return wait_for_go(); }
    }
""")

CHILD = textwrap.dedent("""
    import ctypes, sys, threading, time
    import torch
    sys.path.insert(0, {root!r})
    from radiance_meshes_b200 import _rm_torch as native, scenes
    native.bind({lib!r})
    stand_in = ctypes.PyDLL({lib!r})  # calls that keep the lock, so that they say nothing about it
    dev = torch.device("cuda:0")
    cam = native.Camera(scenes.make_tcam(scenes.look_at((0, 0, 3.0)), 8, 8, 60.0, tile=4), dev, None)
    idx, v = torch.zeros((4, 4), dtype=torch.int32, device=dev), torch.zeros((4, 3), device=dev)
    cell, img, dist = torch.zeros((4, 7), device=dev), torch.zeros((8, 8, 4), device=dev), torch.zeros((8, 8, 5), device=dev)
    i4, rec = torch.zeros((4, 4), dtype=torch.int32, device=dev), torch.zeros((4, 36), device=dev)
    calls = dict(
        project_and_bin=lambda: native.project_and_bin(idx, v, cam.address, True),
        build_tile_lists=lambda: native.build_tile_lists(i4, i4, i4, cam.address, 4, 4),
        pack_records=lambda: native.pack_records(idx, v, cell, cam.address, None, None, None),
        forward=lambda: native.forward(i4, i4, rec, cam.address, False, None, None),
        blend_forward=lambda: native.blend_forward(i4, i4, idx, v, cell, cam.address, False, None, None, True),
        backward=lambda: native.backward(i4, i4, rec, cam.address, None, img, dist, i4, i4, i4, i4, i4, img, dist, idx, v, cell),
        distortion_loss=lambda: native.distortion_loss(dist),
        distortion_loss_backward=lambda: native.distortion_loss_backward(dist, torch.zeros((), device=dev)))
    torch.cuda.synchronize()
    for name, call in calls.items():
        stand_in.stand_in_set(0)
        failed = []
        def run():
            try:
                call()
            except Exception as e:
                failed.append(repr(e))
        t = threading.Thread(target=run)
        t.start()
        while t.is_alive() and not stand_in.stand_in_entered():
            time.sleep(0.001)
        stand_in.stand_in_set(1)
        t.join()
        print("CALL", name, "locked out: " + failed[0] if failed else "free")
""")


def test_other_threads_run_during_library_calls(cuda_lib, tmp_path):
    from radiance_meshes_b200.csrc import build
    build.build_torch_module()
    source, lib = tmp_path / "stand_in.cpp", tmp_path / "stand_in.so"
    source.write_text(STAND_IN)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", build.INCLUDE, str(source), "-o", str(lib), "-lpthread"])
    out = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, lib=str(lib))], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    lines = [ln for ln in out.stdout.splitlines() if ln.startswith("CALL")]
    assert len(lines) == 8 and all(ln.endswith(" free") for ln in lines), out.stdout
