"""A handle belongs to one host thread; several threads build with handles of their own."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch
    assert torch.cuda.is_available()
    import scp3_b200
    return scp3_b200


def build(api, name, precision, estimator, nm, n2, n3, pes="qtip4pf"):
    from scp3_b200 import inputs
    nw, x0, MUa, omega = inputs.load(name)
    return api.HBuild(nw, x0, MUa, omega, modes=np.arange(omega.size)[-nm:], n2=n2, n3=n3, pes=pes,
                      precision=precision, estimator=estimator)


# small and large tables and operands beside one another
@pytest.mark.parametrize("estimator,precision", [("direct", "fp64"), ("gradient", "fp64"), ("gradient", "bf16x3"),
                                                 ("direct", "bf16x3")])
def test_two_handles_in_two_threads(api, estimator, precision):
    sizes = [("cluster_2_800", 3, 3, 0), ("cluster_6_100", 40, 12, 2)]
    rounds, out, errors = 300, [None, None], []
    want = []
    for s in sizes:
        h = build(api, s[0], precision, estimator, *s[1:])
        h.accumulate(100, 500)
        want.append(h.read(0))
        h.close()
    gate = threading.Barrier(2)

    def work(k):
        try:
            h = build(api, sizes[k][0], precision, estimator, *sizes[k][1:])
            gate.wait()
            for _ in range(rounds):
                h.reset()
                h.accumulate(100, 500)
            out[k] = h.read(0)
            h.close()
        except Exception as e:
            errors.append(e)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    for k in range(2):
        assert np.array_equal(out[k], want[k])


def test_smaller_handle_leaves_the_larger_one(api):
    """A second, smaller handle does not take shared memory from the first one's kernels."""
    first = build(api, "cluster_8_0", "bf16x3", "gradient", 66, 66, 0)
    first.accumulate(100, 300)
    want = first.read(0)
    second = build(api, "cluster_7_500", "bf16x3", "gradient", 57, 57, 0)
    second.accumulate(100, 300)
    first.reset()
    first.accumulate(100, 300)
    assert np.array_equal(first.read(0), want)


def test_new_handle_beside_default_stream_work(api):
    """A new handle's buffers are cleared before its first pass, also while another thread
    keeps the default stream busy: the same matrix, bit for bit."""
    import torch
    h = build(api, "cluster_6_100", "fp64", "direct", 48, 10, 0)
    h.accumulate(100, 1 << 17)
    want = h.read(0)
    h.close()
    stop = threading.Event()

    def busy():
        a = torch.randn(2048, 2048, device="cuda")
        while not stop.is_set():
            for _ in range(20):
                torch.mm(a, a)
            torch.cuda.current_stream().synchronize()

    t = threading.Thread(target=busy)
    t.start()
    try:
        for _ in range(8):
            h = build(api, "cluster_6_100", "fp64", "direct", 48, 10, 0)
            h.accumulate(100, 1 << 17)
            got = h.read(0)
            h.close()
            assert np.array_equal(got, want)
    finally:
        stop.set()
        t.join()


@pytest.mark.parametrize("kind", ["bf16x3", "gradient_bf16x3", "gradient_fp64", "batch", "network", "scp1"])
def test_new_handles_of_every_form_beside_default_stream_work(api, kind):
    """As above for the handles whose tables or operands are cleared or copied to on the
    default stream: their first result is an old handle's, bit for bit."""
    import torch
    from scp3_b200 import inputs, surrogate
    rng = np.random.default_rng(0)
    q, t = rng.normal(size=(512, 48)).astype(np.float32), rng.normal(size=512).astype(np.float32)
    nw, x0, MUa, omega = inputs.load("cluster_6_100")

    def first():
        if kind == "batch":
            b = api.Batch([dict(nw=nw, x0=x0, MUa=MUa, omega=omega)] * 2)
            b.accumulate(100, 5000)
            out = b.read(1)
        elif kind == "network":
            b = surrogate.MLP(48, 256, 512)
            b.set_params(b.get_params()[::-1].copy())
            out = np.append(b(q), b.loss_and_grad(q, t)[1])
        elif kind == "scp1":
            b = api.SCP1Average("qtip4pf", nw)
            out = b.sums(x0, np.full(54, 0.5), np.eye(54) * 0.03, 5, 0, 500)[2]
        else:
            b = build(api, "cluster_6_100", kind.split("_")[-1], "gradient" if "_" in kind else "direct", 48, 10, 0)
            b.accumulate(100, 5000)
            out = b.read(1)
        b.close()
        return out

    want = first()
    stop = threading.Event()

    def busy():
        a = torch.randn(4096, 4096, device="cuda")
        while not stop.is_set():
            for _ in range(20):
                torch.mm(a, a)
            torch.cuda.current_stream().synchronize()

    th = threading.Thread(target=busy)
    th.start()
    try:
        for _ in range(6):
            assert np.array_equal(first(), want)
    finally:
        stop.set()
        th.join()
