"""The benchmark's end-to-end host over the C API, against a stand-in for the library: buffers go when they are dropped."""
import gc
import threading
import weakref

import bench


class FakeCapi:
    """Counts the handles that are alive and completes transfers from another thread, as the driver does."""

    def __init__(self):
        self.alive, self.threads, owner = [], [], self

        class Handle:
            def __init__(self, *_keep):
                self._h, self._client = len(owner.alive) + 1, _keep
                owner.alive.append(weakref.ref(self))

        class Executable(Handle):
            def execute(self, args):
                assert all(isinstance(a, Handle) for a in args)
                return [Handle(self)]

        class Client(Handle):
            def buffer(self, array):
                return Handle(self)

            def compile(self, text, opt_level):
                return Executable(self)

        class ToHostAsync:
            def __call__(self, handle, ptr, nbytes, done, user):
                owner.threads.append(threading.Thread(target=done, args=(user,)))
                owner.threads[-1].start()
                return 0

        class Lib:
            mhlo_b200_buffer_to_host_async = ToHostAsync()
            mhlo_buffer_to_host = staticmethod(lambda handle, ptr, nbytes: 0)

        self.Client, self.lib = Client, Lib

    @staticmethod
    def _check(status):
        assert status == 0

    def count(self):
        return sum(r() is not None for r in self.alive)


def test_dropped_buffers_are_freed_without_the_cycle_collector():
    capi = FakeCapi()
    gc.collect()
    gc.disable()
    try:
        host = bench.CApiHost(capi)
        exe, params = host.compile("module"), [host.buffer(None)]
        resident = capi.count()
        pending = None
        for _ in range(20):
            ids = host.buffer(None)
            out = exe.execute([ids] + params)[0]
            out.to_host_pointer(0, 0)
            if pending is not None:
                assert pending[0]()
            pending = (out.to_host_pointer_start(0, 0), out, ids)
            assert capi.count() <= resident + 4  # this step's and the one whose transfer is awaited next
        assert pending[0]()
        del out, ids, pending
        assert capi.count() == resident
        del exe, params, host
        assert capi.count() == 0
    finally:
        gc.enable()
    for t in capi.threads:
        t.join()
    assert not bench.CApiHost._landed


def test_completion_callback_outlives_the_transfer():
    capi = FakeCapi()
    host = bench.CApiHost(capi)
    waits = [host.buffer(None).to_host_pointer_start(0, 0) for _ in range(50)]
    assert all(w() for w in waits)
    done = weakref.ref(bench.CApiHost._done)
    del host, waits
    gc.collect()
    assert done() is not None
    for t in capi.threads:
        t.join()
