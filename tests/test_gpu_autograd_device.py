"""autograd.substep on tensors that live on the scene's GPU against the same
call on host tensors: the same kernels on the same values, so results and
gradients are equal bit for bit."""
import numpy as np
import pytest

from libwetcloth_b200 import _capi, scenes
from libwetcloth_b200.solver import FluidScene, make_params

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _run(sc, where, precision, mu, fixed_x, dtype=torch.float64):
    from libwetcloth_b200 import autograd
    g = FluidScene(sc, precision=precision)
    g.set_adjoint_positions(not fixed_x)
    rng = np.random.default_rng(5)
    n = sc.x.shape[0]
    t = [torch.tensor(a, dtype=dtype, device=where, requires_grad=True)
         for a in (sc.x, sc.v, rng.normal(0, 1, (n, 9)))]
    m = torch.tensor(1e-3, dtype=torch.float64, device=where, requires_grad=True) if mu else None
    cot = [torch.tensor(rng.normal(0, 1, (n, k)), device=where) for k in (3, 3, 9)]
    out = autograd.substep(g, *t, 1e-3, viscosity=m, correction_call=2)
    # the third output's cotangent is left out in one setting
    used = 2 if fixed_x else 3
    grads = torch.autograd.grad(out[:used], t + ([m] if mu else []), cot[:used])
    res = [o.detach().cpu().numpy() for o in out] + [q.cpu().numpy() for q in grads]
    assert all(o.device.type == where for o in out)
    g.close()
    return res


@pytest.mark.parametrize("precision", [_capi.WCG_FP64, _capi.WCG_FP32_REFINE])
@pytest.mark.parametrize("mu,fixed_x", [(False, False), (True, False), (False, True)])
def test_device_tensors_equal_host_tensors(precision, mu, fixed_x, wcg):
    sc = scenes.dam_break(16, 8, 0)
    sc.v = np.random.default_rng(1).normal(0.0, 0.2, sc.x.shape)
    a = _run(sc, "cpu", precision, mu, fixed_x)
    b = _run(sc, "cuda", precision, mu, fixed_x)
    assert len(a) == len(b)
    for p, q in zip(a, b):
        assert p.shape == q.shape and p.dtype == q.dtype and np.array_equal(p, q)


@pytest.mark.parametrize("fixed_x", [False, True])
def test_on_a_side_stream(fixed_x, wcg):
    """The same under a stream of the caller's, which nothing orders with the
    default stream: what the call returns is finished when it returns."""
    sc = scenes.dam_break(32, 8, 0)
    a = _run(sc, "cuda", _capi.WCG_FP64, False, fixed_x)
    for _ in range(3):
        with torch.cuda.stream(torch.cuda.Stream()):
            b = _run(sc, "cuda", _capi.WCG_FP64, False, fixed_x)
        assert all(np.array_equal(p, q) for p, q in zip(a, b))


def test_device_tensors_of_other_kinds(wcg):
    """float32 leaves convert as on the host; non-finite input is refused with
    the host path's error."""
    from libwetcloth_b200 import autograd
    sc = scenes.dam_break(16, 8, 0)
    a = _run(sc, "cpu", _capi.WCG_FP64, False, False, torch.float32)
    b = _run(sc, "cuda", _capi.WCG_FP64, False, False, torch.float32)
    for p, q in zip(a, b):
        assert np.array_equal(p, q)
    g = FluidScene(sc)
    x = torch.tensor(sc.x, device="cuda")
    x[3, 1] = float("nan")
    C = torch.zeros((x.shape[0], 9), device="cuda", dtype=torch.float64)
    with pytest.raises(_capi.WcgError) as e:
        autograd.substep(g, x, torch.zeros_like(x), C, 1e-3)
    assert e.value.code == _capi.WCG_ERR_ARG
    g.close()


@pytest.mark.parametrize("change", ["split", "merge", "terminator", "empty"])
def test_particle_count_of_the_results(change, wcg):
    """A sub-step that changes the number of particles returns as many rows as
    the scene holds after it, on the device as on the host."""
    from libwetcloth_b200 import autograd

    def run(where):
        sc = scenes.dam_break(16, 8, 0)
        if change in ("split", "merge"):
            scenes.mixed_volumes(sc, 3, mrel=(0.3, 0.7, 1.0, 2.5, 5.0))
            sc.params.particle_split = change == "split"
            sc.params.particle_merge = change == "merge"
        if change == "empty":
            sc.vol[5:50] = 0.0
        g = FluidScene(sc)
        if change == "terminator":
            g.set_terminators([{"type": "sphere", "inside": True, "center": sc.x.mean(0),
                                "param": (0.1,)}])
        n = g.num_particles
        if change == "merge":  # it works on the grid of a sub-step before
            g.substep(1e-3)
            g.set_state(sc.x, sc.v, np.zeros((n, 9)))
        t = [torch.tensor(a, dtype=torch.float64, device=where)
             for a in (sc.x, sc.v, np.zeros((n, 9)))]
        out = [o.cpu().numpy() for o in autograd.substep(g, *t, 1e-3, correction_call=1)]
        assert all(o.shape[0] == g.num_particles != n for o in out) and g.num_particles > 0
        now = g.download()
        g.close()
        assert all(np.array_equal(o, a) for o, a in zip(out, now))
        return out

    for p, q in zip(run("cpu"), run("cuda")):
        assert p.shape == q.shape and np.array_equal(p, q)


def test_widths_and_masses_are_checked(wcg):
    """Tensors of another width, and a scene whose masses are of another
    particle set, do not reach the device route: what the host arrays can take
    gives the same as on the host, the rest is refused."""
    from libwetcloth_b200 import autograd
    sc = scenes.dam_break(16, 8, 0)
    n = sc.x.shape[0]
    wide = np.concatenate([sc.x, sc.v], 1)  # (n, 6): the first 3 n values are taken
    wide.reshape(-1)[:3 * n] = sc.x.reshape(-1)
    res = []
    for where in ("cpu", "cuda"):
        g = FluidScene(sc)
        x, v, C = (torch.tensor(a, device=where) for a in (sc.x, sc.v, np.zeros((n, 9))))
        res.append([o.cpu().numpy() for o in autograd.substep(
            g, torch.tensor(wide, device=where), v, C, 1e-3, correction_call=0)])
        for bad in ((x, v, C[:, :3]), (x, v[:, :1], C), (x[:-1], v, C)):
            with pytest.raises(ValueError):
                autograd.substep(g, *bad, 1e-3)
        g.close()
    assert all(p.shape == q.shape and np.array_equal(p, q) for p, q in zip(*res))
    # more particles than masses, uploaded from the device
    g = FluidScene(scenes.dam_break(12, 8, 0))
    dev = [torch.tensor(a, device="cuda") for a in (sc.x, sc.v, np.zeros((n, 9)), sc.mass, sc.vol,
                                                   sc.radius)]
    g.upload_device(n, *[t.data_ptr() for t in dev])
    m = g._attrs[0].size
    assert m < n == g.num_particles
    out = autograd.substep(g, *dev[:3], 1e-3, correction_call=0)
    assert all(o.shape[0] == m for o in out)  # the host route: the particles with masses
    g.close()
    # masses never uploaded from the host
    g = FluidScene(None, params=make_params(sc.params))
    g.upload_device(n, *[t.data_ptr() for t in dev])
    with pytest.raises(ValueError):
        autograd.substep(g, *dev[:3], 1e-3)
    g.close()


def test_checkpoint_leaves_half_of_the_memory(wcg, monkeypatch):
    """A node's checkpoint is on the device while half of its memory stays free,
    else on the host; results and gradients are the same bits."""
    from libwetcloth_b200 import autograd
    sc = scenes.dam_break(16, 8, 0)
    n = sc.x.shape[0]
    total = torch.cuda.mem_get_info()[1]
    res = []
    for room in (True, False):
        free = total // 2 + 120 * n - (0 if room else 1)
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda d=None: (free, total))
        monkeypatch.setattr(torch.cuda, "memory_reserved", lambda d=None: 0)
        monkeypatch.setattr(torch.cuda, "memory_allocated", lambda d=None: 0)
        g = FluidScene(sc)
        t = [torch.tensor(a, device="cuda", requires_grad=True)
             for a in (sc.x, sc.v, np.zeros((n, 9)))]
        out = autograd.substep(g, *t, 1e-3, correction_call=0)
        assert isinstance(out[0].grad_fn.state[0], torch.Tensor) == room
        grads = torch.autograd.grad(out[1].square().sum(), t)
        assert all(o.is_cuda for o in (*out, *grads))
        res.append([o.detach().cpu().numpy() for o in (*out, *grads)])
        g.close()
    assert all(np.array_equal(p, q) for p, q in zip(*res))


def test_cotangents_with_the_negative_bit(wcg):
    """A cotangent that torch holds as a lazily negated view arrives negated, and
    bfloat16 tensors, which have no host array, stay refused."""
    from libwetcloth_b200 import autograd
    sc = scenes.dam_break(16, 8, 0)
    n = sc.x.shape[0]
    g = FluidScene(sc)
    t = [torch.tensor(a, device="cuda", requires_grad=True)
         for a in (sc.x, sc.v, np.zeros((n, 9)))]
    c = torch.randn((n, 3), device="cuda", dtype=torch.float64)
    res = []
    for cot in (-c, torch._neg_view(c)):
        out = autograd.substep(g, *t, 1e-3, correction_call=0)
        res.append([q.cpu().numpy() for q in torch.autograd.grad(out[1], t, cot)])
    assert all(np.array_equal(p, q) for p, q in zip(*res))
    with pytest.raises(TypeError):
        autograd.substep(g, t[0].detach().bfloat16(), t[1], t[2], 1e-3)
    g.close()


def test_masses_are_those_uploaded(wcg):
    """The masses, volumes and radii are those of the upload on either route, also
    after the caller has changed its arrays in place."""
    from libwetcloth_b200 import autograd
    res = []
    for where in ("cpu", "cuda"):
        sc = scenes.dam_break(16, 8, 0)
        g = FluidScene(sc)
        t = [torch.tensor(a, device=where)
             for a in (sc.x, sc.v, np.zeros((sc.x.shape[0], 9)))]
        a = autograd.substep(g, *t, 1e-3, correction_call=0)
        sc.mass *= 2.0
        sc.radius *= 0.5
        b = autograd.substep(g, *t, 1e-3, correction_call=0)
        res += [[o.cpu().numpy() for o in q] for q in (a, b)]
        g.close()
    for r in res[1:]:
        assert all(np.array_equal(p, q) for p, q in zip(res[0], r))
