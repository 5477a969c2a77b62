"""Order groups of the batched forms on one stream and on several."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_serial_and_parallel_servers_give_the_same_states():
    """The server's three settings (one stream, several, the library's choice) on a
    burst of five orders."""
    import sdg
    import workloads as W
    ops = {p: W.reference_operators(p) for p in (2, 3, 5, 7, 9)}
    states = []
    for setting in (False, True, None):
        srv = sdg.Server(ops, parallel_groups=setting)
        t = [srv.submit(3 + p % 3, 2, 4, p, 9, 1e-3 / p, (0.4, 0.5, 0.6), 0.2, (1.0, 0.5, 0.25),
                        want_state=True) for p in ops]
        states.append([srv.wait(x)[1] for x in t])
        srv.close()
    for other in states[1:]:
        for a, b in zip(states[0], other):
            assert np.array_equal(a, b)


def test_the_binding_passes_each_setting(monkeypatch):
    """What reaches the library's configuration for each setting."""
    import sdg
    import workloads as W
    seen = []
    create = sdg.lib.sdg_server_create

    class Spy:
        def __getattr__(self, name):
            if name != "sdg_server_create":
                return getattr(lib, name)

            def f(h, cfg, *rest):
                seen.append(cfg._obj.parallel_groups)
                return create(h, cfg, *rest)
            return f

    lib = sdg.lib
    monkeypatch.setattr(sdg, "lib", Spy())
    ops = {2: W.reference_operators(2)}
    for setting in (False, True, None):
        sdg.Server(ops, parallel_groups=setting).close()
    assert seen == [-1, 1, 0]
