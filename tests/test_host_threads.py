"""First calls of several threads at once, on the CPU: a copy of the library
linked with fake_cuda.cpp, loaded anew (the fake's allocator and log take one
thread at a time, so the threads share nothing but what is looked up)."""
import ctypes as C
import shutil
import threading

from tests.fakecuda import _build


def test_tensor_map_encoder_is_ready_for_every_thread(tmp_path):
    lib = C.CDLL(shutil.copy(_build(), tmp_path / "fresh.so"))
    fn = getattr(lib, "_ZN5swave18tensor_map_encoderEv")
    fn.restype, fn.argtypes = C.c_void_p, []
    got = []
    threads = [threading.Thread(target=lambda: got.append(fn())) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 4 and None not in got
