"""Step calls of small boxes in one launch, beside the results themselves
(test_gpu_fixed_point.py): what happens when a wait between the stages runs out,
and boxes that step at the same time."""
import numpy as np
import pytest

from helpers import Case

pytestmark = pytest.mark.gpu

both = pytest.mark.parametrize("opt", ["OPT_EVENODD", "OPT_OPT1"])


def _fields(c):
    return [a[: c.nown].copy() for a in (c.q, c.u, c.v, c.w)]


def _solver(c, opt, **kw):
    import sdg
    return sdg.Solver(c.NeX, c.NeY, c.NeZ, c.p, c.D, c.Lift, opt=getattr(sdg, opt), **kw)


CALLS = {
    "step_timed": lambda s, c: s.step_timed(c.dt, 0),
    "minmax": lambda s, c: s.minmax(),
    "run": lambda s, c: s.run(c.dt, 2, 1),
    "tendency": lambda s, c: s.tendency(),
    "download": lambda s, c: s.download(),
    "solve_host_pipelined": lambda s, c: _pipelined(s, c),
}


def _pipelined(s, c):
    f = _fields(c)
    out = np.zeros(c.nown)
    s.solve_host_pipelined(*[[a.ctypes.data] for a in f], [out.ctypes.data], c.dt, 1)


@both
@pytest.mark.parametrize("call", sorted(CALLS))
def test_a_wait_that_runs_out_is_reported_once_by_the_next_waiting_call(opt, call):
    """The wait gives up at once (no block waits for another); the kernel returns,
    the next call that waits says so, step calls in between advance nothing, and
    after an upload the solver steps as a new one."""
    import sdg
    c = Case(4, 3, 5, 3)
    s, fresh = _solver(c, opt), _solver(c, opt)
    s.upload(*_fields(c))
    s.set_wait_limit(0)
    s.step(c.dt, 3)
    s.set_wait_limit(-1)
    s.step(c.dt, 2)
    with pytest.raises(sdg.SdgError) as e:
        CALLS[call](s, c)
    assert e.value.status == sdg.ERR_TIMEOUT
    for x in (s, fresh):
        x.upload(*_fields(c))
        x.step(c.dt, 4)
    assert np.array_equal(s.download(), fresh.download())
    assert np.array_equal(s.tendency(), fresh.tendency())


@both
def test_steps_after_a_wait_ran_out_leave_an_uploaded_state_alone(opt):
    """A new state uploaded before anyone has asked stays as it is: its steps find
    the flag and do nothing."""
    import sdg
    c = Case(4, 3, 5, 3)
    s = _solver(c, opt)
    q, u, v, w = _fields(c)
    s.upload(q, u, v, w)
    s.set_wait_limit(0)
    s.step(c.dt, 1)
    s.set_wait_limit(-1)
    s.upload(q + 1.0, u, v, w)
    s.step(c.dt, 3)  # the current buffer is the uploaded one again
    out = np.zeros(c.nown)
    with pytest.raises(sdg.SdgError):
        s.download(out=out)
    assert np.array_equal(out, q + 1.0)


@both
def test_two_boxes_on_two_streams_at_once(opt):
    """Whole-grid launches of two solvers in flight together: the bits of each
    alone."""
    import torch
    cases = [Case(9, 8, 9, 3), Case(5, 6, 4, 7)]
    streams = [torch.cuda.Stream() for _ in cases]
    alone, both_ = [], []
    for c in cases:
        s = _solver(c, opt)
        s.upload(*_fields(c))
        s.step(c.dt, 60)
        alone.append(s.download())
    for c, st in zip(cases, streams):
        s = _solver(c, opt, stream=st.cuda_stream)
        s.upload(*_fields(c))
        both_.append(s)
    for _ in range(20):
        for c, s in zip(cases, both_):
            s.step(c.dt, 3)
    for s, want in zip(both_, alone):
        assert np.array_equal(s.download(), want)


class _GreenStream:
    """A stream confined to some of the device's SMs (a green context)."""

    def __init__(self, sms):
        import ctypes as C

        import sdg
        sdg.DeviceArray(n=1)  # the primary context
        self.cu = C.CDLL("libcuda.so.1")
        dev, n = C.c_int(), C.c_uint(1)
        resource = lambda: C.create_string_buffer(256)
        whole, part, rest = resource(), resource(), resource()
        desc, self.ctx, self.stream = C.c_void_p(), C.c_void_p(), C.c_void_p()
        self._ok(self.cu.cuDeviceGet(C.byref(dev), 0))
        self._ok(self.cu.cuDeviceGetDevResource(dev, whole, 1))
        self._ok(self.cu.cuDevSmResourceSplitByCount(part, C.byref(n), whole, rest, 0, sms))
        self._ok(self.cu.cuDevResourceGenerateDesc(C.byref(desc), part, 1))
        self._ok(self.cu.cuGreenCtxCreate(C.byref(self.ctx), desc, dev, 1))
        self._ok(self.cu.cuGreenCtxStreamCreate(C.byref(self.stream), self.ctx, 1, 0))

    @staticmethod
    def _ok(status):
        if status != 0:
            pytest.skip("no green context here: CUresult %d" % status)

    def close(self):
        self.cu.cuStreamSynchronize(self.stream)
        self.cu.cuStreamDestroy_v2(self.stream)
        self.cu.cuGreenCtxDestroy(self.ctx)


@both
def test_a_stream_of_few_sms_takes_a_launch_a_stage(opt):
    """A box whose one-launch grid the device holds and the stream's SMs do not:
    the step call succeeds with the same bits."""
    c = Case(13, 12, 13, 3)
    s = _solver(c, opt)
    green = _GreenStream(16)
    g = _solver(c, opt, stream=green.stream.value)
    for x in (s, g):
        x.upload(*_fields(c))
        x.step(c.dt, 3)
        x.step(c.dt, 2)
    assert np.array_equal(s.download(), g.download())
    g.close()
    green.close()
