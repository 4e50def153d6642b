"""The convolution block Conv3d(1, f) - ReLU - Conv3d(f, f) - ReLU - Conv3d(f, 1) in
BF16 through the library's kernels (csrc/conv.cu)."""
from __future__ import annotations

import ctypes
import math
import threading

import torch
import torch.nn as nn
import torch.nn.functional as F

from . import _lib
from .geometry import _ptr, _stream

_CONVS = (0, 2, 4)  # of the block's modules
_HOOKS = ("_forward_hooks", "_forward_pre_hooks", "_backward_hooks", "_backward_pre_hooks")


def _plain(m: nn.Module, kind) -> bool:
    """A module of exactly this class whose call runs its class's forward alone."""
    return (type(m) is kind and "forward" not in m.__dict__
            and not any(getattr(m, h, None) for h in _HOOKS))


def _watchers():
    """Tests for whatever watches or transforms the calls made here: tracing, functorch,
    forward-mode differentiation, dispatch and function modes, global module hooks. Some
    have no public name; a torch that lacks one of these keeps the general path."""
    try:
        peek, level = torch._C._functorch.peek_interpreter_stack, torch.autograd.forward_ad
        dispatch, function = torch._C._len_torch_dispatch_stack, torch._C._len_torch_function_stack
        level._current_level
        return (torch.compiler.is_compiling, torch.jit.is_tracing, lambda: peek() is not None,
                lambda: level._current_level >= 0, lambda: dispatch() > 0, lambda: function() > 0,
                torch.nn.modules.module._has_any_global_hook)
    except AttributeError:
        return (lambda: True,)


_WATCHERS = _watchers()


def _special_modes() -> bool:
    return any(w() for w in _WATCHERS)


_UNKNOWN = object()


def _checkpoint_hook():
    """What marks the non-reentrant torch.utils.checkpoint that saves, or recomputes, the
    tensors saved here: its pack hook, None outside one (_UNKNOWN where torch does not
    tell)."""
    try:
        top = torch._C._autograd._top_saved_tensors_default_hooks(True)
    except (AttributeError, TypeError):
        return _UNKNOWN
    if top is None or getattr(top[0], "__module__", None) != "torch.utils.checkpoint":
        return None
    return top[0]


_local = threading.local()  # .run: the call of a SamePath that this thread is in


class SamePath:
    """``fn``, to be checkpointed: the blocks called in it take the paths of its first call
    at every later one. What watches the calls (_watchers, module hooks) may be there in
    the forward pass and not when a checkpoint repeats it, or the other way round, and
    the two paths save different tensors, which a checkpoint refuses."""

    def __init__(self, fn):
        self.fn = fn
        self.paths = None  # of the first call, in order
        # one of the caller's own checkpoints may repeat the first call itself
        self.general = _checkpoint_hook() is not None

    def __call__(self, *args):
        outer = getattr(_local, "run", None)
        replay = None if self.paths is None else iter(self.paths)
        if replay is None:
            self.paths = []
        _local.run = (self, replay, _checkpoint_hook())
        try:
            return self.fn(*args)
        finally:
            _local.run = outer


def fused(body: nn.Sequential, x: torch.Tensor) -> bool:
    """Whether this call of the block goes to the kernels. In a checkpoint that is not a
    SamePath's it does not: nothing tells its repetition what was chosen."""
    run, replay, hook = getattr(_local, "run", None) or (None, None, None)
    if _checkpoint_hook() not in (None, hook):
        return False
    if replay is not None:
        return next(replay, False) and _computable(body, x)
    path = supported(body, x) and not (run is not None and run.general)
    if run is not None:
        run.paths.append(path)
    return path


def supported(body: nn.Sequential, x: torch.Tensor) -> bool:
    """Whether the block's call is one that the kernels compute and nothing watches."""
    return (_computable(body, x) and not _special_modes() and _plain(body, nn.Sequential)
            and all(_plain(m, nn.ReLU if i % 2 else nn.Conv3d) for i, m in enumerate(body)))


def _fits(shape) -> bool:
    """Whether the kernels index a volume of this shape, [batch, 1, z, y, x]: a plane in 32
    bits, an axis in FP32."""
    return (max(shape) < 1 << 24 and math.prod(shape) < 1 << 32
            and shape[-1] * shape[-2] < 1 << 31)


def _computable(body: nn.Sequential, x: torch.Tensor) -> bool:
    """Whether the kernels compute it: FP32 input and weights on a GPU under BF16 autocast,
    16 or 32 features (the weights of all taps stay in shared memory), the block as it
    was built."""
    if not (type(x) is torch.Tensor and x.is_cuda and x.dtype == torch.float32 and x.dim() == 5
            and x.shape[1] == 1 and x.numel() > 0 and torch.is_autocast_enabled("cuda")
            and torch.get_autocast_dtype("cuda") == torch.bfloat16):
        return False
    if type(body) is not nn.Sequential or len(body) != 5:
        return False
    f = body[0].out_channels if type(body[0]) is nn.Conv3d else 0
    if f not in (16, 32) or type(body[1]) is not nn.ReLU or type(body[3]) is not nn.ReLU:
        return False
    if not _fits(x.shape):
        return False
    for i, (ci, co) in zip(_CONVS, ((1, f), (f, f), (f, 1))):
        m = body[i]
        if not (type(m) is nn.Conv3d and m.kernel_size == (3, 3, 3) and m.stride == (1, 1, 1)
                and m.padding == (1, 1, 1) and m.dilation == (1, 1, 1) and m.groups == 1
                and m.padding_mode == "zeros" and m.bias is not None):
            return False
        for p, shape in ((m.weight, (co, ci, 3, 3, 3)), (m.bias, (co,))):
            if not (type(p) in (torch.Tensor, nn.Parameter) and p.dtype == torch.float32
                    and p.device == x.device and p.shape == shape):
                return False
    return True


def _reference(x, w1, b1, w2, b2, w3, b3):
    h = F.relu(F.conv3d(x, w1, b1, padding=1))
    h = F.relu(F.conv3d(h, w2, b2, padding=1))
    return F.conv3d(h, w3, b3, padding=1)


def _pointers(ts):
    return (ctypes.c_void_p * 3)(*[None if t is None else t.data_ptr() for t in ts])


def _strides(ts):
    return (ctypes.c_int64 * 15)(*[s for t in ts for s in t.stride()])


class _Block(torch.autograd.Function):
    """x, weights and biases in BF16."""

    @staticmethod
    def forward(ctx, x, *params):
        x_ = x.contiguous()
        w = [p.detach() for p in params[0::2]]
        b = [p.detach().contiguous() for p in params[1::2]]
        B, _, Z, Y, X = x.shape
        f = w[0].shape[0]
        new = dict(dtype=torch.bfloat16, device=x.device, memory_format=torch.channels_last_3d)
        h1, h2 = torch.empty((B, f, Z, Y, X), **new), torch.empty((B, f, Z, Y, X), **new)
        y = torch.empty((B, 1, Z, Y, X), **new)
        ws = torch.empty(_lib.load().dtv_conv_block_workspace_bytes(f), dtype=torch.uint8,
                         device=x.device)
        with torch.cuda.device(x.device):
            _lib.call("dtv_conv_block", _ptr(x_), _pointers(w), _strides(w), _pointers(b), _ptr(h1),
                      _ptr(h2), _ptr(y), _lib.ivec((X, Y, Z)), B, f, _ptr(ws), _stream(x.device))
        ctx.save_for_backward(x, *params, h1, h2)
        return y

    @staticmethod
    def backward(ctx, gy):
        x, w1, b1, w2, b2, w3, b3, h1, h2 = ctx.saved_tensors
        need = ctx.needs_input_grad
        if torch.is_grad_enabled():  # a differentiable gradient was asked for
            with torch.autocast("cuda", enabled=False):
                args = [x, w1, b1, w2, b2, w3, b3]
                y = _reference(*args)
                wanted = [a for a, n in zip(args, need) if n]
                got = iter(torch.autograd.grad(y, wanted, gy, create_graph=True, allow_unused=True))
            return tuple(next(got) if n else None for n in need)
        B, _, Z, Y, X = x.shape
        f = w1.shape[0]
        last = dict(memory_format=torch.channels_last_3d)
        h1, h2 = h1.contiguous(**last), h2.contiguous(**last)
        gy, x_ = gy.contiguous(), x.contiguous()
        w = [w1, w2, w3]
        gw = [torch.empty_like(t) if n else None for t, n in zip(w, need[1::2])]
        gb = [torch.empty_like(t) if n else None for t, n in zip((b1, b2), need[2:5:2])]
        gx = torch.empty_like(x_) if need[0] else None
        g2 = torch.empty_like(h2) if any(need[:5]) else None
        g1 = torch.empty_like(h1) if any(need[:3]) else None
        size = _lib.ivec((X, Y, Z))
        with torch.cuda.device(x.device):
            ws = torch.empty(_lib.load().dtv_conv_block_backward_workspace_bytes(size, B, f),
                             dtype=torch.uint8, device=x.device)
            _lib.call("dtv_conv_block_backward", _ptr(gy), _ptr(x_), _pointers(w), _strides(w), _ptr(h1),
                      _ptr(h2), None if g1 is None else _ptr(g1), None if g2 is None else _ptr(g2),
                      None if gx is None else _ptr(gx), _pointers(gw),
                      _strides([t if g is None else g for t, g in zip(w, gw)]), _pointers(gb + [None]),
                      size, B, f, _ptr(ws), _stream(x.device))
        gb3 = gy.sum((0, 2, 3, 4)) if need[6] else None
        return gx, gw[0], gb[0], gw[1], gb[1], gw[2], gb3


def conv_block(body: nn.Sequential, x: torch.Tensor) -> torch.Tensor:
    params = [p.to(torch.bfloat16) for i in _CONVS for p in (body[i].weight, body[i].bias)]
    return _Block.apply(x.to(torch.bfloat16), *params)
