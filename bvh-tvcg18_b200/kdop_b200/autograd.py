"""torch.autograd wrapper of contact generation and its hand-written adjoint.

ContactGeometry.apply(xyz, scene, pairs) runs refit + tandem traversal +
MOST_OPPOSING contact generation on the world vertex positions `xyz` (a CUDA
float32 tensor, all meshes of the scene concatenated) and returns per-contact
depth (n,) and normal (n, 3) tensors.  Its backward calls the adjoint kernel
(kdop_contacts_adjoint), which carries dL/d(depth) and dL/d(normal) back to the
vertex positions with the candidate pair set and every discrete choice of the
forward pass (contact face, extreme candidates) held fixed.
"""
from __future__ import annotations

import numpy as np
import torch

from . import lib as kd


def _scene_stream(scene, device):
    """The scene's stream and torch's current one on `device`."""
    handle = scene.ctx.stream
    # cudaStreamLegacy (1) is the stream torch calls the default one, and no ExternalStream's
    work = torch.cuda.default_stream(device) if handle == 1 else torch.cuda.ExternalStream(handle, device=device)
    return work, torch.cuda.current_stream(device)


class ContactGeometry(torch.autograd.Function):
    """The contact rows stay on the device: forward copies them into a tensor
    of its own, and the two streams wait for each other by events (reading the
    rows through host memory and uploading depths and normals again took 10 of
    the 11 ms of a step of 64 touching pairs, 0.9 M contacts)."""

    @staticmethod
    def forward(ctx, xyz: torch.Tensor, scene: "kd.DeviceScene", pairs, opts=None):
        if not xyz.is_cuda or xyz.dtype != torch.float32:
            raise TypeError("xyz must be a float32 CUDA tensor")
        work, current = _scene_stream(scene, xyz.device)
        # conversions run on the current stream: before the scene's waits for it
        x = xyz.detach().contiguous()
        pairs = kd._arg(pairs, np.uint32)
        work.wait_stream(current)
        scene.set_vertices(x)
        scene.refit(kd.REFIT_VERTICES)
        st = scene.traverse_sync(pairs, opts, contacts=True)  # synchronises: x is read
        n = int(st.n_contacts)
        rows = torch.empty((n, 8), dtype=torch.float32, device=xyz.device)
        work.wait_stream(current)  # the block behind rows may have pending work there
        scene.read_contacts_into(rows)  # synchronises
        ctx.scene = scene
        ctx.n_verts, ctx.n_contacts = xyz.shape[0], n
        # copies for any n: of at most one row a slice is contiguous as it is, and
        # an output that is a view may not be written in place by the caller
        return (rows[:, 6].clone(memory_format=torch.contiguous_format),
                rows[:, 3:6].clone(memory_format=torch.contiguous_format))

    @staticmethod
    def backward(ctx, g_depth, g_normal):
        scene = ctx.scene
        dev = g_depth.device if g_depth is not None else g_normal.device
        n = ctx.n_contacts
        gd = (g_depth if g_depth is not None else torch.zeros(n, device=dev)).float().contiguous()
        gn = (g_normal if g_normal is not None else torch.zeros((n, 3), device=dev)).float().contiguous()
        grad = torch.zeros((ctx.n_verts, 3), dtype=torch.float32, device=dev)
        if n == 0:  # nothing to carry back, and no addresses for the adjoint
            return grad, None, None, None
        work, current = _scene_stream(scene, dev)
        work.wait_stream(current)
        scene.adjoint(gd, gn, grad)
        # later work of the current stream, the reuse of gd's and gn's memory
        # included, comes after the adjoint
        current.wait_stream(work)
        return grad, None, None, None


def contact_geometry(xyz: torch.Tensor, scene: "kd.DeviceScene", pairs, opts=None):
    """(depth, normal) of every contact, differentiable in xyz."""
    return ContactGeometry.apply(xyz, scene, pairs, opts)
