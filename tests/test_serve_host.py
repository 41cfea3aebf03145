"""CPU test of the serve loop's set-up against a fake CUDA runtime and a fake
engine: the built object of gb_serve.cu, linked with stand-ins whose pinned
allocation (or event) fails when told to."""
import ctypes
import os
import subprocess

import pytest

FAKE = r"""
#include <cstdlib>
#include <cstring>
struct gb_context; struct gb_layer; struct DStatus;
extern "C" {
int fail_pinned = 0, fail_event = 0, contexts = 0, pinned = 0, events = 0;
static int pinned_calls = 0, event_calls = 0;
void fake_reset(int p, int e) { fail_pinned = p; fail_event = e; pinned_calls = event_calls = 0; }
int cudaHostAlloc(void** p, size_t n, unsigned) {
  if (++pinned_calls == fail_pinned) return 2;
  ++pinned;
  *p = calloc(1, n);
  return 0;
}
int cudaFreeHost(void* p) { --pinned; free(p); return 0; }
int cudaEventCreateWithFlags(void** e, unsigned) {
  if (++event_calls == fail_event) return 2;
  ++events;
  *e = malloc(1);
  return 0;
}
int cudaEventDestroy(void* e) { --events; free(e); return 0; }
int cudaEventQuery(void*) { return 0; }
int cudaEventRecord(void*, void*) { return 0; }
int cudaGetLastError() { return 0; }
int gb_context_create(int, unsigned long long, gb_context** out) {
  ++contexts;
  *out = (gb_context*)calloc(1, 1 << 16);
  return 0;
}
int gb_context_destroy(gb_context* c) { --contexts; free(c); return 0; }
int gb_set_tile_scratch(gb_context*, unsigned long long) { return 0; }
unsigned long long gb_arena_mark(gb_context*) { return 0; }
int gb_sync(gb_context*, long long*) { return 0; }
void gb_clear_status(gb_context*) {}
void gb_layer_free(gb_context*, gb_layer*) {}
int gb_layer_from_host(...) { return 5; }
int gb_layer_to_host(...) { return 5; }
int gb_op_bool(...) { return 5; }
int gb_op_grow(...) { return 5; }
int gb_op_size(...) { return 5; }
int __cudaGetKernel(...) { return 0; }
int __cudaLaunchKernel(...) { return 0; }
int __cudaPopCallConfiguration(...) { return 0; }
int __cudaPushCallConfiguration(...) { return 0; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaRegisterFunction(...) {}
void __cudaUnregisterFatBinary(void**) {}
}
namespace gbi {
void arena_rewind(gb_context*, unsigned long long, bool) {}
gb_layer* binned_of(gb_context*, gb_layer*, int) { return nullptr; }
const unsigned long long* mark_word(gb_context*, unsigned long long) { return nullptr; }
}
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    from vlsi_layout_gb300 import build as B
    B.build()
    d = tmp_path_factory.mktemp("serve")
    (d / "fake.cpp").write_text(FAKE)
    so = str(d / "libserve.so")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-o", so, str(d / "fake.cpp"), os.path.join(B.BUILD, "gb_serve.o"),
                    "-Wl,--no-undefined"], check=True, capture_output=True)
    L = ctypes.CDLL(so, mode=os.RTLD_LOCAL | os.RTLD_NOW | getattr(os, "RTLD_DEEPBIND", 0))
    L.gb_serve_create.argtypes = [ctypes.c_int, ctypes.c_uint64, ctypes.c_int, ctypes.c_uint64, ctypes.c_void_p]
    L.gb_serve_destroy.argtypes = [ctypes.c_void_p]
    return L


def _live(L):
    return [ctypes.c_int.in_dll(L, k).value for k in ("contexts", "pinned", "events")]


@pytest.mark.parametrize("pinned,event", [(1, 0), (3, 0), (0, 1), (0, 2)])
def test_failed_allocation_is_out_of_memory(fake, pinned, event):
    fake.fake_reset(pinned, event)
    S = ctypes.c_void_p()
    assert fake.gb_serve_create(0, 1 << 30, 3, 1 << 20, ctypes.byref(S)) == 3  # GB_ERR_OOM
    assert not S.value and _live(fake) == [0, 0, 0]


def test_create_and_destroy(fake):
    fake.fake_reset(0, 0)
    S = ctypes.c_void_p()
    assert fake.gb_serve_create(0, 1 << 30, 3, 1 << 20, ctypes.byref(S)) == 0
    assert _live(fake) == [4, 3, 3]
    fake.gb_serve_destroy(S)
    assert _live(fake) == [0, 0, 0]
