"""Per-process inferer implementation: the ``dist_render`` seam for a model forward.

Mirrors ``AbstractDDPInfererImpl`` / ``TorchNerfDDPInfererImpl``
(dist_render/ddp_infer/inferer_impl.py:27-145): ``load_model(H, W)`` builds the model from a
checkpoint's ``kwargs`` and installs its forward with ``set_forward_func``; ``renderer_fn``
walks the rays in chunks of ``render_batch_size`` and concatenates ``rgb_map``.  The forward
installed here is ``B200GridNeRF``, i.e. the CUDA library.
"""

from __future__ import annotations

from typing import Callable, Optional

import torch

from .gridnerf import B200GridNeRF


def _rgb_of(result) -> torch.Tensor:
    """``rgb_map`` of a forward's result: the models return ``({"rgb_map": ...}, extra)``, some
    forwards return the dict alone (both shapes are accepted by inferer_impl.py:112-118)."""
    maps = result[0] if isinstance(result, tuple) else result
    try:
        return maps["rgb_map"]
    except (KeyError, TypeError, IndexError):
        raise Exception("cannot find correct key for ret") from None


def renderer_fn(forward: Callable, rays: torch.Tensor, chunk_size: int, **kwargs) -> torch.Tensor:
    """The chunk loop of inferer_impl.py:95-120: ``forward`` on consecutive slices of
    ``chunk_size`` rays, colours concatenated; a result without ``rgb_map`` is an error."""
    if rays.shape[0] == 0:
        return rays.new_zeros((0, 3))
    with torch.inference_mode():
        parts = [_rgb_of(forward(piece, **kwargs)) for piece in torch.split(rays, chunk_size)]
    return parts[0] if len(parts) == 1 else torch.cat(parts, 0)


# Precision presets of the drop-in inferer.  "exact": fp32 everywhere, no termination (what the
# reference's torch path computes; about 4x slower than "fast" on a city frame).  "fast": the
# configuration the benchmark measures: tcgen05 MLP with fp16 operands, fp16 appearance planes,
# rays stop at transmittance 2e-5, density from the pre-summed lattice; rgb stays within 1e-4 of
# "exact" on the tested scenes.
PRESETS = {
    "exact": {"mlp_mode": 0, "ert_transmittance": 0.0, "app_plane_fp16": False, "density_lattice": False},
    "fast": {"mlp_mode": 2, "ert_transmittance": 2e-5, "app_plane_fp16": True, "density_lattice": True},
}


class B200NerfDDPInfererImpl:
    """Drop-in for ``TorchNerfDDPInfererImpl``: same constructor argument (a context with
    ``args_nerf`` and ``model_path``), same methods and properties."""

    RENDER_CHUNK = 65536      # rays of a device chunk, unless render_batch_size is larger (0: always render_batch_size)
    RENDER_SAMPLES = 1 << 25  # and at most that many samples of them: the ids and lists of a chunk grow with both
    RENDER_MEMORY = 0.125     # and as long as the workspaces take no more than that share of the free device memory ...
    RENDER_UNASKED = 1 << 28  # ... which is asked for (70 us) when they need more than this

    def __init__(self, context, profile_stages: bool = False, mlp_mode: Optional[int] = None, preset: str = "exact",
                 **model_options) -> None:
        """``preset`` picks a row of ``PRESETS`` ("exact" is the default so that a drop-in run first
        reproduces the reference's numbers; "fast" is the benchmarked configuration);
        ``mlp_mode`` and any further ``B200GridNeRF`` option (``ert_transmittance``,
        ``app_plane_fp16``, ``density_plane_fp16``, ...) override single entries of it."""
        if preset not in PRESETS:
            raise ValueError(f"preset {preset!r} (one of {sorted(PRESETS)})")
        self._model_options = dict(PRESETS[preset])
        if mlp_mode is not None:
            self._model_options["mlp_mode"] = int(mlp_mode)
        self._model_options.update(model_options)
        self._chunk_size = context.args_nerf.render_batch_size
        self._args = context.args_nerf
        self._tensor_parallel = False
        self._forward: Optional[Callable] = None
        self._profile_stages = profile_stages
        self._model = None
        self._model_path = getattr(context, "model_path", None)
        self._ckpt = getattr(context, "checkpoint", None)  # an already loaded checkpoint dict
        self._out_of_memory = False  # larger device chunks did not fit once: render_batch_size from then on

    @property
    def args(self):
        return self._args

    @property
    def tensor_parallel(self):
        return self._tensor_parallel

    @property
    def model(self):
        return self._model

    def set_pose(self, pose):
        pass

    def edit_model(self, edit_mode):
        pass

    def set_forward_func(self, func):
        self._forward = func

    def remove_old_kwargs(self, kwargs):
        kwargs.pop("shadingMode", None)
        return kwargs

    def set_distributed_args(self, data_parallel_local_rank, rank, data_parallel_group_world_size):
        self._args.local_rank = data_parallel_local_rank
        self._args.rank = rank
        self._args.world_size = data_parallel_group_world_size
        self._args.distributed = data_parallel_group_world_size > 1

    def load_model(self, H, W):
        if self._model is not None:
            return
        ckpt = self._ckpt if self._ckpt is not None else torch.load(self._model_path, map_location="cpu", weights_only=False)
        device = getattr(self._args, "device", "cuda")
        if device == "cuda":
            device = f"cuda:{torch.cuda.current_device()}"
        kwargs = dict(ckpt["kwargs"])
        kwargs.update({"device": device, "args": self._args, "is_train": False})
        kwargs = self.remove_old_kwargs(kwargs)
        self._model = B200GridNeRF(**kwargs, **self._model_options)
        self._model.load(ckpt)
        self.set_forward_func(self._model)

    def _plain_forward(self) -> bool:
        """The installed forward is the model's own, with nothing hooked to it or put in its place: the chunk loop can then
        go past it."""
        m = self._model
        hooks = torch.nn.modules.module
        return (self._forward is m and isinstance(m, B200GridNeRF) and type(m).forward is B200GridNeRF.forward
                and type(m).__call__ is torch.nn.Module.__call__ and "forward" not in vars(m)
                and not (m._forward_hooks or m._forward_pre_hooks or hooks._global_forward_hooks or hooks._global_forward_pre_hooks))

    def _device_chunk(self, n_rays: int, n_samples: int):
        """(rays of a device chunk, lanes) of a call: RENDER_CHUNK rays on two lanes, halved while their workspaces would take
        too much of the memory; at the least what ``render_batch_size`` says, in one workspace."""
        m, least = self._model, self._chunk_size
        chunk = least if self._out_of_memory else max(least, min(self.RENDER_CHUNK, self.RENDER_SAMPLES // n_samples))
        while not self._out_of_memory:
            need = m.workspace_bytes(min(chunk, n_rays), n_samples) + 256
            lanes = 2 if n_rays > chunk else 1
            missing = 0
            for slot in range(lanes):
                held = m._ws.get(slot)
                if held is None or held.numel() < need:
                    missing += need
            if missing <= self.RENDER_UNASKED or missing <= self.RENDER_MEMORY * torch.cuda.mem_get_info(m.device)[0]:
                return chunk, lanes
            if chunk <= least:
                break
            chunk = max(least, chunk // 2)
        return least, 1

    def renderer_fn(self, rays, N_samples=-1, white_bg=True, is_train=False, app_code=None):
        if self._forward is None:
            raise RuntimeError("load_model() has not been called")
        kw = {"N_samples": N_samples, "white_bg": white_bg, "is_train": is_train}
        if getattr(self._model, "encode_app", False):
            # the reference's single-block inferer drops app_code (inferer_impl.py:144-145), which fails
            # for an encode_app checkpoint; here it reaches the model
            kw["app_code"] = app_code
        if self._plain_forward() and not is_train and rays.shape[0] > 0:
            # The same chunks as one library call: pixels do not depend on how rays are cut into chunks, so larger chunks
            # rotate over two lanes and the status blocks are read once at the end, instead of a wait per chunk of
            # render_batch_size rays (960x540 in chunks of 8192: 64 waits).
            with torch.inference_mode():
                model = self._model
                model.set_app_code(kw.get("app_code"))
                chunk, lanes = self._device_chunk(rays.shape[0], model._samples(N_samples))
                try:
                    rgb, _ = model.render_rays(rays, N_samples, white_bg, chunk=chunk, overlap=lanes)
                except torch.cuda.OutOfMemoryError:
                    if (chunk, lanes) == (self._chunk_size, 1):
                        raise
                    self._out_of_memory = True
                    model.release_workspaces()
                    rgb, _ = model.render_rays(rays, N_samples, white_bg, chunk=self._chunk_size)
                if model.check_status_every_call:
                    model.check_pending_status()
            return rgb
        return renderer_fn(self._forward, rays, self._chunk_size, **kw)
