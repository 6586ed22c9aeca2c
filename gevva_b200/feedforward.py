"""Feed-forward steps around the expert path and the dense FP8 GeGLU MLP (ctypes mirror of
the gevva_ff_* / gevva_dense_* entry points), plus the layer wiring of the reference's
layer loop (src/cuda/runtime/prefill.cuh:1200-1250) with attention left out."""
import ctypes
from dataclasses import dataclass

import torch

from .runtime import (EXPERTS, HIDDEN, GevvaMoeError, Nvfp4ExpertRunner, _address, _check, _enqueue, _ptr, _stream_handle,
                      _view, library)

DENSE = 2112


class _DenseWeights(ctypes.Structure):
    _fields_ = [("gate_up", ctypes.c_void_p), ("down", ctypes.c_void_p), ("gate_scale", ctypes.c_float),
                ("up_scale", ctypes.c_float), ("down_scale", ctypes.c_float)]


class _Layer(ctypes.Structure):
    _fields_ = [(n, ctypes.c_void_p) for n in
                ("dense_pre", "expert_pre", "router_scale", "router_weight", "expert_scale", "dense_post",
                 "expert_post", "combined_post", "layer_scalar", "experts", "dense")]


def _lib():
    lib = library()
    if getattr(lib, "_gv_ff_ready", False):
        return lib
    vp, i32, f32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    lib.gevva_ff_prepare.argtypes = [vp] * 7 + [i32, vp]
    lib.gevva_ff_finalize.argtypes = [vp] * 10 + [i32, vp, vp, vp]
    lib.gevva_dense_create.argtypes = [ctypes.POINTER(vp), ctypes.POINTER(_DenseWeights), i32]
    lib.gevva_dense_destroy.argtypes = [vp]
    lib.gevva_dense_destroy.restype = None
    lib.gevva_dense_launch.argtypes = [vp, vp, vp, i32, vp]
    lib.gevva_dense_last_status.argtypes = [vp]
    lib.gevva_dense_status_word.argtypes = [vp]
    lib.gevva_dense_status_word.restype = vp
    lib.gevva_dense_output_scales.argtypes = [vp]
    lib.gevva_dense_output_scales.restype = vp
    lib.gevva_dense_projection_scale.argtypes = [vp]
    lib.gevva_dense_projection_scale.restype = vp
    lib.gevva_dense_buffer.argtypes = [vp, i32, ctypes.POINTER(vp), ctypes.POINTER(ctypes.c_size_t)]
    lib.gevva_pack_fp8.argtypes = [vp, ctypes.c_size_t, vp, vp, vp]
    lib.gevva_ff_layer_workspace_bytes.argtypes = [i32]
    lib.gevva_ff_layer_workspace_bytes.restype = ctypes.c_size_t
    lib.gevva_ff_layer_launch.argtypes = [ctypes.POINTER(_Layer), vp, vp, vp, i32, vp, vp]
    lib._gv_ff_ready = True
    return lib


def _status(status, where):
    if status != 0:
        raise GevvaMoeError(status, where)


def pack_fp8(weight_fp32):
    """Per-tensor E4M3 quantisation: returns (uint8 tensor of the same shape, float scale)."""
    w = weight_fp32.contiguous()
    out = torch.empty(w.shape, dtype=torch.uint8, device=w.device)
    scale = torch.empty(1, dtype=torch.float32, device=w.device)
    with torch.cuda.device(w.device):
        _status(_lib().gevva_pack_fp8(_ptr(w), w.numel(), _ptr(out), _ptr(scale), _stream_handle(None)),
                "pack_fp8")
    return out, float(scale.item())


def ff_prepare(x, dense_weight, expert_weight, router_scale):
    rows = x.shape[0]
    _check(x, torch.bfloat16, (rows, HIDDEN), "input")
    outs = [torch.empty_like(x) for _ in range(3)]
    _status(_enqueue(_lib().gevva_ff_prepare, x.device, None, x.data_ptr(), _address(dense_weight),
                     _address(expert_weight), _address(router_scale), outs[0].data_ptr(), outs[1].data_ptr(),
                     outs[2].data_ptr(), rows), "ff_prepare")
    return outs  # dense_pre, expert_pre, router_input


def ff_finalize(dense, dense_weight, expert_routes, route_weights, inverse_routes, expert_weight,
                combined_weight, residual, layer_scalar, dense_activation_scales=None,
                dense_projection_scale=None):
    """dense_activation_scales f32 [rows] and dense_projection_scale f32 [1] are CUDA tensors (or both
    None), as the reference kernel takes them."""
    rows = dense.shape[0]
    out = torch.empty_like(residual)
    _status(_enqueue(
        _lib().gevva_ff_finalize, dense.device, None, _address(dense), _address(dense_weight), _address(expert_routes),
        _address(route_weights), _address(inverse_routes), _address(expert_weight), _address(combined_weight),
        _address(residual), _address(layer_scalar), _address(out), rows, _address(dense_activation_scales),
        _address(dense_projection_scale)), "ff_finalize")
    return out


class DenseMlp:
    """Dense FP8 GeGLU MLP; launch() returns the unscaled bf16 output and its row scales."""

    def __init__(self, gate_up_fp8, down_fp8, gate_scale, up_scale, down_scale, max_tokens):
        _check(gate_up_fp8, torch.uint8, (2 * DENSE, HIDDEN), "gate_up")
        _check(down_fp8, torch.uint8, (HIDDEN, DENSE), "down")
        self._keep = (gate_up_fp8, down_fp8)
        self.device = gate_up_fp8.device
        self.down_scale = float(down_scale)
        self.max_tokens = max_tokens
        w = _DenseWeights(gate_up_fp8.data_ptr(), down_fp8.data_ptr(), gate_scale, up_scale, down_scale)
        handle = ctypes.c_void_p()
        with torch.cuda.device(self.device):
            _status(_lib().gevva_dense_create(ctypes.byref(handle), ctypes.byref(w), max_tokens), "DenseMlp")
        self._handle = handle
        # f32 [1] on the device, owned by the runner: what ff_finalize takes beside the row scales
        self.projection_scale = _view(_lib().gevva_dense_projection_scale(self._handle), (1,), torch.int32,
                                      self.device).view(torch.float32)

    def __del__(self):
        if getattr(self, "_handle", None):
            _lib().gevva_dense_destroy(self._handle)
            self._handle = None

    def launch(self, x, out=None, stream=None):
        tokens = x.shape[0]
        _check(x, torch.bfloat16, (tokens, HIDDEN), "input")
        if out is None:
            out = torch.empty_like(x)
        _status(_enqueue(_lib().gevva_dense_launch, self.device, stream, self._handle, x.data_ptr(), _address(out),
                         tokens), "dense launch")
        scales = _view(_lib().gevva_dense_output_scales(self._handle), (tokens,), torch.int32,
                       self.device).view(torch.float32)
        return out, scales

    def last_status(self):
        """Synchronises, then returns and clears the status of launch() (0 = ok); a layer's is its experts'."""
        with torch.cuda.device(self.device):
            return _lib().gevva_dense_last_status(self._handle)

    def check(self):
        _status(self.last_status(), "device status")

    def buffer(self, which, dtype):
        ptr, size = ctypes.c_void_p(), ctypes.c_size_t()
        _status(_lib().gevva_dense_buffer(self._handle, which, ctypes.byref(ptr), ctypes.byref(size)), "buffer")
        item = {torch.uint8: 1, torch.int32: 4, torch.bfloat16: 2, torch.float32: 4}[dtype]
        base = torch.int32 if dtype == torch.float32 else dtype
        t = _view(ptr.value, (size.value // item,), base, self.device)
        return t.view(torch.float32) if dtype == torch.float32 else t


@dataclass
class FeedForwardLayer:
    """One layer of the FFN stack: pre-norms + router, experts and dense MLP side by side,
    fused finalize (the wiring of src/cuda/runtime/prefill.cuh:1200-1250)."""
    dense_pre: torch.Tensor        # bf16 [2816] norm weights
    expert_pre: torch.Tensor
    router_scale: torch.Tensor
    router_w: torch.Tensor         # bf16 [128, 2816]
    expert_scale: torch.Tensor     # bf16 [128]
    dense_post: torch.Tensor
    expert_post: torch.Tensor
    combined_post: torch.Tensor
    layer_scalar: torch.Tensor     # bf16 [1]
    experts: Nvfp4ExpertRunner
    dense: DenseMlp

    def forward(self, hidden, aux_stream=None):
        """The layer's output, a new tensor; with `aux_stream` the dense MLP runs there, beside the
        experts.  One native call (gevva_ff_layer_launch) does all launches: called one by one from
        Python they took 137 us of host time a layer, four times what the GPU needs for one token."""
        tokens = hidden.shape[0]
        _check(hidden, torch.bfloat16, (tokens, HIDDEN), "input")
        _check(self.router_w, torch.bfloat16, (EXPERTS, HIDDEN), "router_weight")
        _check(self.expert_scale, torch.bfloat16, (EXPERTS,), "expert_scale")
        lib = _lib()
        out = torch.empty_like(hidden)
        workspace = torch.empty(lib.gevva_ff_layer_workspace_bytes(tokens), dtype=torch.uint8, device=hidden.device)
        layer = _Layer(self.dense_pre.data_ptr(), self.expert_pre.data_ptr(), self.router_scale.data_ptr(),
                       self.router_w.data_ptr(), self.expert_scale.data_ptr(), self.dense_post.data_ptr(),
                       self.expert_post.data_ptr(), self.combined_post.data_ptr(), self.layer_scalar.data_ptr(),
                       self.experts._handle, self.dense._handle)

        def launch(main):
            return lib.gevva_ff_layer_launch(ctypes.byref(layer), hidden.data_ptr(), out.data_ptr(),
                                             workspace.data_ptr(), tokens, main,
                                             main if aux_stream is None else aux_stream.cuda_stream)

        _status(_enqueue(launch, hidden.device, None), "feed-forward layer")
        self.experts._tokens = tokens
        return out
