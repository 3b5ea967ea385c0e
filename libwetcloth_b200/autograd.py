"""torch.autograd binding of the liquid sub-step (the C-ABI's wcg_substep and
wcg_substep_vjp); the arithmetic is all in libwcgpu.so.

``substep(scene, x, v, C, dt, viscosity)`` returns (x', v', C') as float64
tensors and records a node whose backward restores the checkpoint (x, v, C)
in the scene, recomputes the forward grid there and runs the reverse-mode
kernels; an optional 0-d ``viscosity`` tensor gets its gradient too.  The
gradient in x follows the positions through the transfer weights (P2G, G2P
and the advection), the liquid phi behind the ghost-fluid fractions and the
solid projection of the particle correction; the grid's discrete structure
(activation, DOFs, valid faces) is held at the checkpoint's values.  The
scene's particle state after backward is the checkpoint of the last node
differentiated.  Tensors on the scene's device stay there, and so does their
checkpoint while half of the device's memory is free; every other
checkpoint is held on the host.

``rollout(scene, x, v, C, dt, steps, viscosity, checkpoint_every)`` runs
``steps`` sub-steps as one node that keeps only every ``checkpoint_every``-th
state (on the host); its backward recomputes each segment of sub-steps from
its checkpoint and runs the sub-steps' reverse modes in reverse order, so the
memory held is one segment of states, not the whole trajectory.

The particle correction of a sub-step (run in every sub-step; at strength 0
it only projects its subset out of the solid) takes the subset of one call of
the scene's seeded stream: ``correction_call`` fixes that call (the default,
None, takes the scene's next call); sub-step k of a rollout takes call
``correction_call + k``, and the backward replays the same calls.
"""
from __future__ import annotations

import ctypes

import numpy as np
import torch

from . import _capi


def _host(t):
    return t.detach().cpu().numpy().astype(np.float64)


_DTYPES = (torch.float64, torch.float32, torch.float16)  # those that numpy has too
_ASK = 256 << 20  # bytes of checkpoints that a scene makes between two looks at the memory


def _room(scene, device, nbytes):
    """Whether a checkpoint of nbytes may stay on the device: half of its memory
    is left to everything else, so a chain of any length still fits (its later
    nodes keep their checkpoints on the host).  The driver is asked once for
    every _ASK bytes of a scene's checkpoints (asking takes 70 us and up to
    1 ms, a sub-step and its reverse of 110 000 particles 11 ms)."""
    scene._checkpoint_bytes += nbytes
    if scene._checkpoint_bytes < _ASK:
        return True
    free, total = torch.cuda.mem_get_info(device)
    if free - nbytes < total // 2:  # blocks that the allocator holds unused are room too
        free += torch.cuda.memory_reserved(device) - torch.cuda.memory_allocated(device)
    if free - nbytes < total // 2:
        scene._checkpoint_bytes = _ASK  # the next one asks again
        return False
    scene._checkpoint_bytes = nbytes
    return True


def _on_scene(scene, x, v, C):
    """Whether a sub-step can take these tensors where they are: on the scene's
    device, 3, 3 and 9 finite values for every particle that the scene holds
    and that has a mass, volume and radius from the last upload, and room for
    the checkpoint (anything else goes through the host arrays and their
    checks)."""
    n = scene.num_particles
    dev = int(scene.L.wcg_device(scene.h))
    attrs = scene._attrs
    if n <= 0 or attrs is None or any(a is None or a.size != n for a in attrs):
        return False
    if not all(t.is_cuda and t.device.index == dev and t.shape[:1] == (n,) and
               t.numel() == n * w and t.dtype in _DTYPES
               for t, w in ((x, 3), (v, 3), (C, 9))):
        return False
    if not _room(scene, x.device, 15 * 8 * n):
        return False
    return bool(torch.stack([torch.isfinite(t).all() for t in (x, v, C)]).all())


def _snapshot(t, k):
    """A float64 copy of t's values, k per particle, on t's device."""
    return t.detach().to(torch.float64).reshape(-1, k).contiguous().clone()


def _ptr(t):
    return ctypes.cast(t.data_ptr(), _capi._D)


def _load(scene, x, v, C):
    """set_state from device tensors (masses, volumes and radii as uploaded)."""
    n = x.shape[0]
    if scene._attrs is None or any(a.size != n for a in scene._attrs):
        raise ValueError(f"the scene's masses, volumes and radii are not those of {n} particles")
    if scene._attrs_dev is None or scene._attrs_dev[0].device != x.device:
        scene._attrs_dev = tuple(torch.from_numpy(a).to(x.device) for a in scene._attrs)
    # the library runs on the scene's own stream
    torch.cuda.current_stream(x.device).synchronize()
    scene.upload_device(n, *[t.data_ptr() for t in (x, v, C, *scene._attrs_dev)])


def _read(scene, device):
    """The scene's particle state as new tensors on its device.  The count is
    the scene's after the sub-step: the split, the merge, a terminator and the
    removal of particles without volume change it."""
    n = scene.num_particles
    out = tuple(torch.empty((n, w), dtype=torch.float64, device=device) for w in (3, 3, 9))
    # memory that the allocator hands out again may have work pending on this
    # stream; the library writes on its own
    torch.cuda.current_stream(device).synchronize()
    _capi.check(scene.L.wcg_download_liquid_device(scene.h, *[t.data_ptr() for t in out]))
    return out


class _Substep(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, v, C, mu, scene, dt, substeps, call):
        m = float(mu.detach().cpu().item()) if mu is not None else None
        if m is not None:
            scene.set_viscosity(m, substeps)
        k = scene.correction_count if call is None else int(call)
        ctx.call = k
        ctx.scene = scene
        ctx.dt = dt
        ctx.mu = (m, substeps)
        dev = v.device
        if _on_scene(scene, x, v, C):
            # state already on the scene's device: the checkpoint and the results
            # stay there (through the host, the copies were most of the call)
            ctx.state = tuple(_snapshot(t, w) for t, w in ((x, 3), (v, 3), (C, 9)))
            _load(scene, *ctx.state)
            scene.set_correction_count(k)
            scene.substep(dt)
            return _read(scene, x.device)
        xs, vs, Cs = (_host(t) for t in (x, v, C))
        scene.set_state(xs, vs, Cs)
        scene.set_correction_count(k)
        scene.substep(dt)
        x1, v1, C1 = scene.download()
        ctx.state = (xs, vs, Cs)
        return (torch.from_numpy(x1).to(dev), torch.from_numpy(v1).to(dev),
                torch.from_numpy(C1).to(dev))

    @staticmethod
    def backward(ctx, gx1, gv1, gC1):
        n = ctx.state[0].shape[0]
        dev = gv1.device if gv1 is not None else gx1.device

        def host(g, k):
            return np.zeros((n, k)) if g is None else _host(g)

        scene = ctx.scene
        m, substeps = ctx.mu
        if m is not None:
            scene.set_viscosity(m, substeps)
        if isinstance(ctx.state[0], torch.Tensor):
            where = ctx.state[0].device
            cot = [torch.zeros((n, w), dtype=torch.float64, device=where) if g is None else
                   g.detach().resolve_neg().to(where, torch.float64).reshape(n, w).contiguous()
                   for g, w in ((gv1, 3), (gC1, 9), (gx1, 3))]
            bar = [torch.empty_like(t) for t in cot]
            mub = ctypes.c_double(0.0)
            _load(scene, *ctx.state)
            scene.set_correction_count(ctx.call)
            _capi.check(scene.L.wcg_substep_vjp(scene.h, ctx.dt, *[_ptr(t) for t in cot + bar],
                                                ctypes.byref(mub)))
            vb, Cb, xb = bar
            gmu = None if m is None else torch.tensor(mub.value, dtype=torch.float64, device=dev)
            return xb, vb, Cb, gmu, None, None, None, None
        scene.set_state(*ctx.state)
        scene.set_correction_count(ctx.call)
        vb, Cb, xb, mub = scene.substep_vjp(ctx.dt, host(gv1, 3), host(gC1, 9), host(gx1, 3),
                                            with_viscosity=True)
        gmu = None if m is None else torch.tensor(mub, dtype=torch.float64, device=dev)
        return (torch.from_numpy(xb).to(dev), torch.from_numpy(vb).to(dev),
                torch.from_numpy(Cb).to(dev), gmu, None, None, None, None)


def substep(scene, x, v, C, dt: float, viscosity=None, viscosity_substeps: int = 1,
            correction_call=None):
    """One differentiable sub-step of a FluidScene (liquid).  viscosity: an
    optional 0-d tensor (LiquidInfo::viscosity) that receives a gradient;
    correction_call: the call of the seeded correction stream the sub-step
    takes (None: the scene's next)."""
    return _Substep.apply(x, v, C, viscosity, scene, dt, viscosity_substeps, correction_call)


class _Rollout(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, v, C, mu, scene, dt, steps, every, substeps, call):
        m = float(mu.detach().cpu().item()) if mu is not None else None
        if m is not None:
            scene.set_viscosity(m, substeps)
        k0 = scene.correction_count if call is None else int(call)
        state = (_host(x), _host(v), _host(C))
        ckpts = []
        scene.set_state(*state)
        for k in range(steps):
            if k % every == 0:
                ckpts.append(state if k == 0 else scene.download())
            scene.set_correction_count(k0 + k)
            scene.substep(dt)
        x1, v1, C1 = scene.download()
        ctx.scene, ctx.dt, ctx.steps, ctx.every = scene, dt, steps, every
        ctx.mu = (m, substeps)
        ctx.k0 = k0
        ctx.ckpts = ckpts
        dev = v.device
        return (torch.from_numpy(x1).to(dev), torch.from_numpy(v1).to(dev),
                torch.from_numpy(C1).to(dev))

    @staticmethod
    def backward(ctx, gx1, gv1, gC1):
        scene, dt, steps, every = ctx.scene, ctx.dt, ctx.steps, ctx.every
        m, substeps = ctx.mu
        n = ctx.ckpts[0][0].shape[0]
        dev = gv1.device if gv1 is not None else gx1.device

        def host(g, k):
            return np.zeros((n, k)) if g is None else _host(g)

        xb, vb, Cb = host(gx1, 3), host(gv1, 3), host(gC1, 9)
        mub = 0.0
        if m is not None:
            scene.set_viscosity(m, substeps)
        for seg in range(len(ctx.ckpts) - 1, -1, -1):
            k_lo = seg * every
            k_hi = min(steps, k_lo + every)
            # recompute the segment's sub-step inputs from its checkpoint
            states = [ctx.ckpts[seg]]
            scene.set_state(*states[0])
            for k in range(k_lo, k_hi - 1):
                scene.set_correction_count(ctx.k0 + k)
                scene.substep(dt)
                states.append(scene.download())
            for k in range(k_hi - 1, k_lo - 1, -1):
                scene.set_state(*states[k - k_lo])
                scene.set_correction_count(ctx.k0 + k)
                vb, Cb, xb, mk = scene.substep_vjp(dt, vb, Cb, xb, with_viscosity=True)
                mub += mk
        gmu = None if m is None else torch.tensor(mub, dtype=torch.float64, device=dev)
        return (torch.from_numpy(xb).to(dev), torch.from_numpy(vb).to(dev),
                torch.from_numpy(Cb).to(dev), gmu, None, None, None, None, None, None)


def rollout(scene, x, v, C, dt: float, steps: int, viscosity=None, viscosity_substeps: int = 1,
            checkpoint_every: int = 10, correction_call=None):
    """`steps` differentiable sub-steps of a FluidScene (liquid) as one node
    with a checkpoint every `checkpoint_every` sub-steps (recomputed in the
    backward).  Arguments as substep's; returns the final (x, v, C)."""
    if steps < 1 or checkpoint_every < 1:
        raise ValueError("steps and checkpoint_every must be positive")
    return _Rollout.apply(x, v, C, viscosity, scene, dt, int(steps), int(checkpoint_every),
                          viscosity_substeps, correction_call)
