"""What the pair network hands to its kernels: tensors of its own device only.  Shapes, types and devices follow torch's rules
for (feats - mean) / std, targets * target_scale and an assignment of the weights."""
import pytest
import torch

from dftbaby_b200 import learned, native, tcgemm

N = 5


@pytest.fixture
def calls(monkeypatch):
    """The native calls of a network on the CPU, recorded instead of made; addresses by tensor."""
    made, known = [], {}

    def ptr(t):
        if t is None:
            return None
        known[t.data_ptr()] = t
        assert t.device.type == "cpu"  # the network's device
        return t.data_ptr()

    monkeypatch.setattr(native, "ptr", ptr)
    monkeypatch.setattr(native, "stream", lambda: None)
    monkeypatch.setattr(native, "call", lambda name, *a: made.append((name, [known.get(x, x) if isinstance(x, int) else x
                                                                            for x in a])))
    monkeypatch.setattr(tcgemm, "_errword", lambda dev: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(learned, "_mm", lambda *a, **k: None)
    return made


def _standardised(made):
    """(F - mean) / std as dftb_mlp_inputs would form it from its arguments."""
    name, a = made[0]
    assert name == "dftb_mlp_inputs"
    n, F, ld, mean, std = a[0], a[4], a[5], a[6], a[7]
    F = F.as_strided((n, learned.NFEAT), (ld, 1))
    assert F.dtype == mean.dtype == std.dtype == torch.float32 and mean.is_contiguous() and std.is_contiguous()
    return (F - mean) / std


def _head(made):
    a = [x for name, x in made if name == "dftb_mlp_head"][0]
    T, tscale, m = a[8], a[9], a[10]
    assert T.shape == (N, 2) and T.is_contiguous() and m.shape == (N,) and m.is_contiguous()
    assert T.dtype == m.dtype == tscale.dtype == torch.float32
    return T * tscale, m


def _net():
    net = learned.GuessNet(device="cpu")
    net.mean, net.std = torch.arange(8.0), 1.0 + torch.arange(8.0) / 3
    return net


def test_other_devices_are_refused(calls):
    net, f, t, w = _net(), torch.rand(N, 8), torch.rand(N, 2), torch.rand(N)
    far = torch.device("meta")
    with pytest.raises((RuntimeError, NotImplementedError)):
        net.predict(f.to(far))
    net.mean = net.mean.to(far)
    with pytest.raises((RuntimeError, NotImplementedError)):
        net.predict(f)
    with pytest.raises((RuntimeError, NotImplementedError)):
        net.loss_and_gradients(f, t, w)
    assert not calls


def test_targets_on_another_device_are_refused(calls):
    net, f, t, w = _net(), torch.rand(N, 8), torch.rand(N, 2), torch.rand(N)
    with pytest.raises((RuntimeError, NotImplementedError)):
        net.loss_and_gradients(f, t.to("meta"), w)
    assert not [1 for name, _ in calls if name == "dftb_mlp_head"]


@pytest.mark.parametrize("form", ["plain", "strided", "transposed", "double", "one column", "one row", "leading one",
                                  "statistics in FP64", "scalar statistics", "broadcast rows"])
def test_features(calls, form):
    net, f = _net(), torch.rand(N, 8)
    if form == "strided":
        f = torch.rand(N, 20)[:, 3:19:2]
    elif form == "transposed":
        f = torch.rand(8, N).T
    elif form == "double":
        f = f.double()
    elif form == "one column":
        f = f[:, :1]
    elif form == "one row":
        f = torch.rand(8)  # eight samples, the same row each
    elif form == "leading one":
        f = torch.rand(1, 1, 8)
    elif form == "statistics in FP64":
        net.mean, net.std = net.mean.double(), net.std.double()
    elif form == "scalar statistics":
        net.mean, net.std = torch.tensor(0.5), torch.tensor(2.0)
    elif form == "broadcast rows":
        f = torch.rand(1, 8).expand(N, 8)
    n = f.shape[0]
    want = torch.zeros(n, 8)
    want[:] = (f.float() - net.mean) / net.std
    net.predict(f)
    assert torch.equal(_standardised(calls), want)


@pytest.mark.parametrize("form", ["plain", "strided", "double", "one number", "one row", "column", "leading one"])
def test_targets_and_weights(calls, form):
    net, f, t, w = _net(), torch.rand(N, 8), torch.rand(N, 2), torch.rand(N)
    if form == "strided":
        t, w = torch.rand(N, 7)[:, ::4], torch.rand(N, 3)[:, 1]
    elif form == "double":
        t, w = t.double(), w.double()
    elif form == "one number":
        t, w = torch.tensor(0.25), torch.tensor(2.0)
    elif form == "one row":
        t, w = torch.rand(2), torch.rand(1)
    elif form == "column":
        t = torch.rand(N, 1)
    elif form == "leading one":
        t, w = t[None], w[None]
    T, m = torch.zeros(N, 2), torch.zeros(N)
    T[:] = t.float() * net.target_scale
    m[:] = w.float()
    net.loss_and_gradients(f, t, w)
    got_T, got_m = _head(calls)
    assert torch.equal(got_T, T) and torch.equal(got_m, m)


@pytest.mark.gpu
def test_host_samples_with_host_statistics():
    """Features and statistics on the host: standardised there, then moved."""
    net = learned.GuessNet(device="cuda")
    f = torch.randn(300, 8)
    net.fit_statistics(f)
    got = net.predict(f)
    net.mean, net.std = net.mean.cuda(), net.std.cuda()
    want = net.predict(f.cuda())
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    with pytest.raises(RuntimeError):
        net.predict(f)
    with pytest.raises(RuntimeError):
        net.loss_and_gradients(f.cuda(), torch.zeros(300, 2), torch.ones(300))
    loss, grads = net.loss_and_gradients(f.cuda(), torch.zeros(300, 2).cuda(), torch.ones(300))  # weights may be anywhere
    ref, want = net.loss_and_gradients(f.cuda(), torch.zeros(300, 2).cuda(), torch.ones(300).cuda())
    assert abs(loss - ref) <= 1e-12 * abs(ref)
