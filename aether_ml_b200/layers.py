"""Layer, loss and optimizer classes with the names, constructor arguments, methods and attributes of
Aether-ML's ``CNN/models/CNN_classes_cupy.py``, computing on a B200 through libaether_b200.so.

Every ``forward`` / ``backward`` below is a thin host-side wrapper: it validates shapes, owns the
output / workspace buffers (torch CUDA tensors are used purely as device memory) and makes one or
two C-ABI calls.  No arithmetic on activations happens in Python and there is no CPU fallback.

Arrays: fp32, C-contiguous, NHWC activations, (fH, fW, Cin, Cout) filters -- the reference's layouts.
Inputs may be torch CUDA tensors, objects exposing ``__cuda_array_interface__`` (CuPy arrays) or
NumPy arrays (copied to the device).  Outputs are torch CUDA tensors.
"""
import ctypes as C
import functools
import math
import os
import weakref

import numpy as np
import torch

from . import _lib
from ._lib import AetherConvDesc, host, lib

DEFAULT_MATH_MODE = os.environ.get("AETHER_MATH_MODE", "bf16")


def _device():
    if not torch.cuda.is_available():
        raise _lib.AetherError("aether_ml_b200 needs a CUDA device (no CPU fallback exists)")
    return torch.device("cuda", torch.cuda.current_device())


def to_device(a, dtype=torch.float32):
    """Return `a` as a contiguous CUDA tensor of `dtype` (no copy when it already is one)."""
    if dtype is torch.float32:
        t = host().ready(a)
        if t is not None:
            return t
    if isinstance(a, torch.Tensor):
        t = a
    elif hasattr(a, "__cuda_array_interface__"):
        t = torch.as_tensor(a, device=_device())
    else:
        t = torch.as_tensor(np.asarray(a))
    if t.device.type != "cuda":
        t = t.to(_device(), non_blocking=True)
    if t.dtype != dtype:
        t = t.to(dtype)
    return t if t.is_contiguous() else t.contiguous()


class _Neighbour:
    """An attribute that refers to another layer: owned when it is assigned, like any attribute, and not when a model links its
    layers (`_link`).  The layer list of a model owns its layers; with owning links between neighbours a dropped model, its
    workspaces and its activations stayed in device memory until Python's cycle collector happened to run, and the next
    model paid for fresh allocations."""

    def __set_name__(self, owner, name):
        self.name, self.slot = name, "_link_" + name

    def __get__(self, obj, owner=None):
        if obj is None:
            return self
        try:
            held = obj.__dict__[self.slot]
        except KeyError:
            raise AttributeError(self.name) from None
        return held() if type(held) is weakref.ref else held

    def __set__(self, obj, value):
        obj.__dict__[self.slot] = value


def _link(layer, name, other):
    """Sets ``layer.name`` to another layer of the same model without owning it."""
    if isinstance(getattr(type(layer), name, None), _Neighbour):
        try:
            layer.__dict__["_link_" + name] = weakref.ref(other) if other is not None else None
            return
        except TypeError:                       # an object that takes no weak references (a caller's own class)
            pass
    setattr(layer, name, other)


class _Saved:
    """Pickling of a layer / loss / optimizer for ``Model.save`` (the reference pickles the whole model after
    stripping the per-step arrays, CNN_model_cupy.py:291-309): device arrays travel as NumPy arrays, everything that
    belongs to one forward/backward pass (activations, gradients, workspaces, operand-copy bookkeeping, links to the
    neighbouring layers) is left out and rebuilt empty on loading."""

    prev = _Neighbour()
    next = _Neighbour()

    _TRANSIENT = ("inputs", "output", "dinputs", "dweights", "dbiases", "prev", "next", "bn_partials", "binary_mask",
                  "channel_mask", "batch_mean", "batch_var", "running_mean", "running_var", "inputs_shape",
                  "trainable_layers", "accumulated_sum", "accumulated_count", "step_dev", "stats_from", "fused_dropout",
                  "fused_pool", "fused_bn", "copy_consumer", "copy_dy_consumer", "fixed_mask", "fused_into_prev")

    def __getstate__(self):
        state = {}
        for k, v in self.__dict__.items():
            if k in self._TRANSIENT or (k.startswith("_") and k not in ("_rm", "_rv", "_calls")):
                continue
            state[k] = ("__device_array__", v.detach().cpu().numpy()) if isinstance(v, torch.Tensor) else v
        return state

    def __setstate__(self, state):
        for k, v in state.items():
            if isinstance(v, tuple) and len(v) == 2 and isinstance(v[0], str) and v[0] == "__device_array__":
                v = to_device(v[1], torch.from_numpy(v[1]).dtype)
            self.__dict__[k] = v
        self._restore_transient()

    def _restore_transient(self):
        pass


def _copied(x):
    y = host().empty_like(x)
    if x.numel():
        host().aether_copy(x, y, x.numel())
    return y


class _Workspace:
    """Grow-only byte buffer owned by a layer and handed to the library as scratch."""

    def __init__(self):
        self.buf = None
        self.size = 0
        self.refused = math.inf     # bytes that there was no memory for: from there on the least has to do

    def get(self, nbytes, plan=None):
        """The buffer, of at least ``nbytes`` or, where there is no memory for that, of what the plan's calls can do with."""
        if self.size < nbytes or self.buf is None:
            if plan is None or nbytes < self.refused:
                try:
                    return self._grow(nbytes)
                except torch.OutOfMemoryError:
                    if plan is None or plan.least_ws_bytes() >= nbytes:
                        raise
                    self.refused = nbytes
            return self.get(plan.least_ws_bytes())
        return self.buf

    def _grow(self, nbytes):
        nbytes = max(int(nbytes), 256)
        self.buf = host().empty_u8((nbytes,))
        self.size = nbytes
        return self.buf


class _OperandCopies:
    """Remembers which arrays the forward pass left bf16 operand copies of in a layer's workspace, so that the
    backward pass reuses a copy only while it still describes the array: same workspace buffer, same array, and
    no in-place change since (torch's per-tensor version counter).  Anything else -- a regrown workspace, an input
    modified between the passes, weights replaced -- makes the backward pass rebuild the copy."""

    def __init__(self):
        self.ws_ptr = None
        self.x = None
        self.w = None

    def record(self, ws, x, w):
        self.ws_ptr = ws.data_ptr()
        tag = host().tag
        self.x = tag(x)
        self.w = tag(w)

    def weights_valid(self, ws, w):
        """Whether the copies of the weights that the last forward pass left describe `w` still."""
        return self.ws_ptr is not None and ws.data_ptr() == self.ws_ptr and host().same(w, self.w)

    def flags(self, ws, x, w):
        """Bit 0: the copy of x is valid; bit 1: the copies of the weights are (aether_conv2d_bwd's x_shadow_valid)."""
        if self.ws_ptr is None or ws.data_ptr() != self.ws_ptr:
            return 0
        same = host().same
        return (1 if same(x, self.x) else 0) | (2 if same(w, self.w) else 0)


_unwritten_exist = False        # whether any array has ever been marked (the check below is on every layer's path)


def _mark_unwritten(t):
    """Marks a device array whose fp32 contents were deliberately not written (lean mode: only its bf16 operand copy
    exists, inside the consuming layer's workspace).  A layer that would have to READ such an array raises."""
    global _unwritten_exist
    _unwritten_exist = True
    t._aether_unwritten = True
    return t


def _require_written(t, who):
    if _unwritten_exist and getattr(t, "_aether_unwritten", False):
        raise _lib.AetherError("%s: the input array was not materialised (Model.finalize(lean=True)) and its operand copy is "
                               "no longer current; run the producing layer again" % who)


def _array_tag(t):
    """Identity of a device array's contents as far as the host can tell: address, element count, version counter
    (a reshaped view of the same memory has the same tag)."""
    return host().tag(t)[:3]


class _Branch:
    """A second stream inside the capture of a train step: work that nothing on the main one waits for until its end.  Arrays that
    the branch uses must outlive the capture or be held here: memory that the main stream's arrays give back is handed out
    to its next ones whatever the branch still does."""

    def __init__(self):
        self.stream = torch.cuda.Stream()
        self.open = False
        self.held = []

    def fork(self, *arrays):
        """What is put on the branch from here on starts behind what the current stream has been given so far."""
        self.stream.wait_stream(torch.cuda.current_stream())
        self.open = True
        self.held.extend(arrays)

    def join(self):
        if self.open:
            torch.cuda.current_stream().wait_stream(self.stream)
            self.open = False


class _TakesCopies:
    """What the layers with bf16 operand copies in their workspace share."""
    _weights_fixed = False      # Model: the weights do not change between the batches of a predict / evaluate call, or have been copied ahead of a captured step
    _branch = None              # a _Branch while Model captures a step

    def _copy_weights(self):
        """The operand copies of the weights alone, on the branch, for a forward pass like the last one; False: it makes its own."""
        p, w = self._last_plan()
        ws = self._ws
        if p is None or p.layout is None or p.layout.x_copy_ld == 0 or ws.buf is None or ws.size < p.ws_bytes:
            return False
        self._branch.fork(w, ws.buf)
        with torch.cuda.stream(self._branch.stream):
            host().aether_conv2d_filter_copies(p.raw, w, ws.buf, ws.size)
        self._copies.record(ws.buf, w, w)       # (of an x there is none)
        return True

    def _products(self, p, x, dy, w, dx, db, ws, flags, rows, behind=None):
        """The backward pass's library call while a step is captured, then `behind` (of the parameters' gradients): dW goes to the branch, beside
        the kernels of the layers in front, which wait for dX only."""
        H, b = host(), self._branch
        if dx is None or not flags & _lib.CONV_DY_COPY_READY:
            H.aether_conv2d_bwd_ex(p.raw, x, dy, w, dx, self.dweights, db, ws, self._ws.size, flags, rows)
            if behind is not None:
                behind()
            return
        b.fork(x, dy, w, ws, self.dweights, self.dbiases)
        H.aether_conv2d_bwd_ex(p.raw, x, dy, w, dx, None, None, ws, self._ws.size, flags, rows)
        with torch.cuda.stream(b.stream):
            H.aether_conv2d_bwd_ex(p.raw, x, dy, w, None, self.dweights, db, ws, self._ws.size, flags, rows)
            if behind is not None:
                behind()

    def _forget_copies(self):
        """The workspace's contents are no longer what the last passes left there."""
        self._copies.ws_ptr = self._handed.x = self._handed.dy = None


class _HandedIn:
    """Operand copies that a neighbouring layer's kernel wrote into this layer's workspace (see
    aether_conv2d_operand_layout): which array each describes, so the layer skips its own cast pass only for
    exactly that array in exactly that workspace buffer."""

    def __init__(self):
        self.x = None        # (workspace address, tag of x)
        self.dy = None       # (workspace address, tag of dy, rows of column sums)

    def x_ready(self, ws, x):
        return self.x is not None and self.x[0] == ws.data_ptr() and host().same(x, self.x[1])

    def dy_rows(self, ws, dy):
        if self.dy is not None and self.dy[0] == ws.data_ptr() and host().same(dy, self.dy[1]):
            return self.dy[2]
        return 0


def _operand_layout(d):
    """AetherOperandLayout of a convolution descriptor, or None when the shape reads no bf16 operand copies."""
    lay = _lib.AetherOperandLayout()
    return lay if lib().aether_conv2d_operand_layout(C.byref(d), C.byref(lay)) else None


class _ConvPlan:
    """Sizes and queries of one convolution shape: the descriptor's bytes, the output shape (None when the filter does
    not fit the padded input), the workspaces, the operand layout and the blocks of epilogue statistics."""

    def __init__(self, desc, Ho, Wo):
        d = C.byref(desc)
        self.raw = bytes(desc)
        self.x_shape = (desc.S, desc.H, desc.W, desc.Cin)
        self.y_shape = (desc.S, Ho, Wo, desc.Cout) if Ho >= 1 and Wo >= 1 else None
        self.b_shape = (desc.Cout,)
        self.layout, self.ws_bytes, self.stats_blocks, self.head = None, 0, 0, False
        if self.y_shape is not None:
            self.ws_bytes = int(lib().aether_conv2d_workspace_bytes(d))
            self.stats_blocks = int(lib().aether_conv2d_bnstats_blocks(d))
            self.layout = _operand_layout(desc)
            self.head = bool(lib().aether_head_supported(d))
        self.fwd_ws_bytes = self.ws_bytes              # of the workspace, what inference uses
        # (less than all of it only where neither the kernels on operand copies nor those of first layers and heads serve the shape)
        if self.layout is None and self.y_shape is not None and self.stats_blocks == 0 and not self.head:
            self.fwd_ws_bytes = int(lib().aether_conv2d_fwd_workspace_bytes(d))

    @functools.cached_property
    def pools(self):
        """Whether a forward call that goes on to the pooled output (aether_conv2d_pool_fwd) is the faster way there."""
        return bool(lib().aether_conv2d_pool_faster(AetherConvDesc.from_buffer_copy(self.raw)))

    def least_ws_bytes(self):
        """The workspace that every call can do with."""
        return int(lib().aether_conv2d_least_workspace_bytes(AetherConvDesc.from_buffer_copy(self.raw)))


# ------------------------------------------------------------------------------------- Conv_Layer
class Conv_Layer(_TakesCopies, _Saved):
    """Drop-in for ``Conv_Layer`` (CNN_classes_cupy.py:37-161).

    Same constructor arguments and attributes (``filter_weights``/``weights`` alias, ``biases``, the
    four regularizer attributes; after ``forward``: ``output``, ``inputs``; after ``backward``:
    ``dweights``, ``dbiases``, ``dinputs``).  ``dinputs`` is the scatter-ADD gradient that the
    reference's CUDA scatter kernel produces (:4-35), returned contiguous instead of as a sliced view.
    One extra keyword, ``math_mode`` in {"bf16", "tf32", "fp32"}, selects the operand precision of
    the tensor-core kernels (default from $AETHER_MATH_MODE, else bf16)."""

    def __init__(self, input_shape, num_filters=1, filter_size=(3, 3), strides=(1, 1), padding="same",
                 math_mode=None):
        self.input_shape = input_shape
        self.num_filters = num_filters
        self.filter_size = filter_size
        self.strides = strides
        self.padding = padding
        self.math_mode = math_mode or DEFAULT_MATH_MODE
        if self.math_mode not in _lib.MATH_MODES:
            raise ValueError("math_mode must be one of %s" % sorted(_lib.MATH_MODES))
        self.weight_regularizer_l1 = 0
        self.weight_regularizer_l2 = 0
        self.bias_regularizer_l1 = 0
        self.bias_regularizer_l2 = 0
        input_depth = input_shape[-1]
        n = filter_size[0] * filter_size[1] * input_depth
        std = np.float32(np.sqrt(np.float32(2.0 / n)))
        # He-normal initialisation (:54-66), drawn on the host from NumPy's global generator
        w = np.random.randn(filter_size[0], filter_size[1], input_depth, num_filters).astype(np.float32) * std
        self.filter_weights = to_device(w)
        self.biases = torch.zeros(num_filters, dtype=torch.float32, device=_device())
        self._ws = _Workspace()
        self._stats_ws = _Workspace()
        self.emit_bn_stats = False      # set when a Batch_Norm consumes this layer's output (Model.finalize does it)
        self.bn_partials = None         # (buffer, blocks, data_ptr of the output they describe) after a training forward
        self._desc = None               # the plan of the last forward pass
        self._plans = {}
        self._copies = _OperandCopies()
        self._handed = _HandedIn()
        self.first_in_model = False     # Model.finalize: this layer's dinputs are never needed

    def _restore_transient(self):
        self._ws = _Workspace()
        self._stats_ws = _Workspace()
        self.bn_partials = None
        self._desc = None
        self._plans = {}
        self._copies = _OperandCopies()
        self._handed = _HandedIn()
        self.emit_bn_stats = False
        self.first_in_model = False

    # `weights` is the same array object as `filter_weights` (:68); in-place optimizer updates on
    # either name are visible through both.
    @property
    def weights(self):
        return self.filter_weights

    @weights.setter
    def weights(self, value):
        self.filter_weights = value

    def _last_plan(self):
        return self._desc, self.filter_weights

    def _plan(self, shape):
        """What follows from an input shape and this layer's settings, worked out once per combination."""
        key = (shape, *self.filter_size, *self.strides, self.padding, self.math_mode, self.num_filters, host().device())
        p = self._plans.get(key)
        if p is None:
            if len(self._plans) >= 64:          # a caller with ever new batch sizes: start over
                self._plans.clear()
            p = self._plans[key] = self._make_plan(*shape)
        return p

    def _extent(self, H, W):
        """(padding, output rows, output columns) for images of that size."""
        fH, fW = self.filter_size
        sH, sW = self.strides
        P = (fH - 1) // 2 if self.padding == "same" else 0      # :78-81, same amount on both axes
        return P, int((H + 2 * P - fH) / sH + 1), int((W + 2 * P - fW) / sW + 1)

    def _make_plan(self, S, H, W, Cin):
        fH, fW = self.filter_size
        sH, sW = self.strides
        P, Ho, Wo = self._extent(H, W)
        return _ConvPlan(AetherConvDesc(S, H, W, Cin, self.num_filters, fH, fW, sH, sW, P, P, _lib.MATH_MODES[self.math_mode]), Ho, Wo)

    # -- operand-copy hand-off: the kernel that produces this layer's x (going forward) or dy (going back) may write
    # the bf16 copy the tensor-core kernels read straight into this layer's workspace
    def x_copy_target(self, shape):
        """(address, row length) where the bf16 copy of an input of `shape` goes, or None."""
        if len(shape) != 4 or shape[3] != self.filter_weights.shape[2]:
            return None
        p = self._plan(tuple(shape))
        lay = p.layout
        if lay is None or lay.x_copy_ld == 0:          # (first layers gather x themselves: no copy of x is read)
            return None
        ws = self._ws.get(p.ws_bytes)
        return ws.data_ptr() + lay.x_copy_offset, lay.x_copy_ld

    def x_copy_written(self, x):
        self._handed.x = (self._ws.buf.data_ptr(), _array_tag(x))

    def dy_copy_target(self):
        """(address, row length, column-sum address, rows available) for the bf16 copy of the coming dvalues, or None."""
        if self._desc is None:
            return None
        lay = self._desc.layout
        if lay is None:
            return None
        # A first layer's filter-gradient kernel takes the copy, but its dX runs on the CUDA cores from the fp32 array:
        # the hand-off is only for a layer whose dinputs nobody asks for (the first layer of a Model).
        if lay.x_copy_ld == 0 and not self.first_in_model:
            return None
        ws = self._ws.get(self._desc.ws_bytes)
        return ws.data_ptr() + lay.dy_copy_offset, lay.dy_copy_ld, ws.data_ptr() + lay.dy_colsum_offset, lay.dy_colsum_rows_max

    def dy_copy_written(self, dy, rows):
        self._handed.dy = (self._ws.buf.data_ptr(), _array_tag(dy), int(rows))

    def forward(self, inputs, training):
        x = to_device(inputs)
        if x.ndim != 4:
            raise ValueError(f"Expected a 4D tensor, got {x.ndim} instead.")
        shape = x.shape
        if shape[3] != self.filter_weights.shape[2]:
            raise ValueError(f"input has {shape[3]} channels, filters expect {self.filter_weights.shape[2]}")
        p = self._plan(shape)
        if p.y_shape is None:
            raise ValueError("filter larger than the padded input")
        H = host()
        y = H.empty(p.y_shape)                  # (before the workspace, which can do with less)
        ws = self._ws.get(p.ws_bytes if training else p.fwd_ws_bytes, p)
        w = self.filter_weights
        flags = 0
        if self._handed.x is not None:
            flags = _lib.CONV_X_COPY_READY if self._handed.x_ready(ws, x) else 0
            self._handed.x = None
        if not flags:
            _require_written(x, "Conv_Layer.forward")
        if self._weights_fixed and p.layout is not None and self._copies.weights_valid(ws, w):
            flags |= _lib.CONV_W_COPY_READY
            if self._branch is not None:
                self._branch.join()
        # With emit_bn_stats the kernel's epilogue also writes the per-channel partial statistics that the
        # Batch_Norm behind this layer would otherwise compute in a pass of its own over y (:467-470).
        nblk = p.stats_blocks if (training and self.emit_bn_stats) else 0
        self.bn_partials = None
        if nblk > 0:
            stats = self._stats_ws.get(nblk * 3 * self.num_filters * 4)
            H.aether_conv2d_fwd_ex(p.raw, x, w, self.biases, y, stats, self._stats_ws.size, ws, self._ws.size, flags)
            self.bn_partials = (stats, nblk, y.data_ptr())
        else:
            H.aether_conv2d_fwd_ex(p.raw, x, w, self.biases, y, None, 0, ws, self._ws.size, flags)
        self.inputs = x
        self.output = y
        self._desc = p
        self._copies.record(ws, x, w)
        return y

    def forward_pooled(self, x, p, bn, alpha, pooled, target):
        """Inference over `x` by plan `p` up to the pooled output of the Batch_Norm, activation and 2x2 max Pooling behind this layer
        (Model), with its operand copy at `target`; the layers' attributes stay as they are."""
        H = host()
        ws = self._ws.get(p.fwd_ws_bytes, p)
        w = self.filter_weights
        flags = 0
        if self._handed.x is not None:
            flags = _lib.CONV_X_COPY_READY if self._handed.x_ready(ws, x) else 0
            self._handed.x = None
        if not flags:
            _require_written(x, "Conv_Layer.forward")
        if self._weights_fixed and p.layout is not None and self._copies.weights_valid(ws, w):
            flags |= _lib.CONV_W_COPY_READY
        H.aether_conv2d_pool_fwd(p.raw, x, w, self.biases, bn.gamma, bn.beta, bn._rm, bn._rv, bn.epsilon, alpha, pooled, target[0] if target else None,
                                 target[1] if target else 0, ws, self._ws.size, flags)
        self._copies.record(ws, x, w)

    def backward(self, dvalues, need_dinputs=True):
        p = self._desc
        if p is None:
            raise RuntimeError("Conv_Layer.backward called before forward")
        dy = to_device(dvalues)
        x = self.inputs
        if dy.shape != p.y_shape:
            raise ValueError(f"dvalues has shape {tuple(dy.shape)}, expected {p.y_shape}")
        H = host()
        w = self.filter_weights
        if getattr(self, "_grad_views", None) is not None:
            self.dweights, self.dbiases = self._grad_views
        else:
            self.dweights = H.empty(w.shape)
            self.dbiases = H.empty(p.b_shape)
        dx = H.empty(p.x_shape) if need_dinputs else None
        ws = self._ws.get(p.ws_bytes, p)
        shadow_ok = self._copies.flags(ws, x, w)
        rows = 0
        if self._handed.dy is not None:
            rows = self._handed.dy_rows(ws, dy)
            self._handed.dy = None
        if rows and self.first_in_model and need_dinputs:
            rows = 0                        # a first layer asked for dinputs after all: that path reads the fp32 array
        if rows:
            shadow_ok |= _lib.CONV_DY_COPY_READY
        else:
            _require_written(dy, "Conv_Layer.backward")
        if not (shadow_ok & _lib.CONV_X_COPY_READY):
            _require_written(x, "Conv_Layer.backward")
        if self._branch is None:
            H.aether_conv2d_bwd_ex(p.raw, x, dy, w, dx, self.dweights, self.dbiases, ws, self._ws.size, shadow_ok, rows)
        else:
            self._products(p, x, dy, w, dx, self.dbiases, ws, shadow_ok, rows)
        self.dinputs = dx
        return dx

    def get_parameters(self):
        return self.filter_weights, self.biases

    def set_parameters(self, weights, biases):
        # copy into the existing arrays so `weights` stays the same object as `filter_weights`
        w = to_device(weights)
        b = to_device(biases).reshape(-1)
        if tuple(w.shape) != tuple(self.filter_weights.shape) or b.numel() != self.biases.numel():
            raise ValueError("parameter shapes do not match this layer")
        self.filter_weights.copy_(w)
        self.biases.copy_(b)


# ------------------------------------------------------------------------------------- Pooling
class Pooling(_Saved):
    """Drop-in for ``Pooling`` (CNN_classes_cupy.py:204-312), 'valid' padding, max or average.
    The argmax is kept as one byte per output (window-local index of the first maximum);
    ``max_indicies`` reconstructs the reference's (rows, cols) pair on demand."""
    fused_bn = _Neighbour()

    def __init__(self, filter_size=(2, 2), strides=(2, 2), padding="valid", pooling_type="max"):
        self.filter_size = filter_size
        self.strides = strides
        self.padding = padding
        self.pooling_type = pooling_type
        self.fused_bn = None            # (a weak link) a Batch_Norm that pools inside its own kernels (Model.finalize(fuse=True))

    def _restore_transient(self):
        self.fused_bn = None

    def _kind(self):
        if self.pooling_type == "max":
            return _lib.POOL_MAX
        if self.pooling_type == "average":
            return _lib.POOL_AVG
        raise ValueError(f"Expected pooling_type == max or average, recieved {self.pooling_type} instead")

    def forward(self, inputs, training):
        x = to_device(inputs)
        if self.fused_bn is not None and self.fused_bn.pooled_now:
            # the fused Batch_Norm already produced the pooled tensor (and keeps the argmax codes)
            self.inputs = self.output = x
            self._argmax = self.fused_bn._pool_arg
            return self.output
        if x.ndim != 4:
            raise ValueError(f"Expected a 4D tensor, got {x.ndim} instead.")
        if self.padding != "valid":
            # the reference's "same" branch reads H_out before assigning it (:226-233) and cannot run
            raise ValueError(f"Expected padding == valid, recieved {self.padding} instead")
        S, H, W, Cc = x.shape
        fH, fW = self.filter_size
        sH, sW = self.strides
        Ho = (H - fH) // sH + 1
        Wo = (W - fW) // sW + 1
        kind = self._kind()
        h = host()
        y = h.empty((S, Ho, Wo, Cc))
        self._argmax = h.empty_u8((S, Ho, Wo, Cc)) if kind == _lib.POOL_MAX else None
        h.aether_pool_fwd(x, y, self._argmax, S, H, W, Cc, fH, fW, sH, sW, kind)
        self.inputs = x
        self.output = y
        return self.output

    @property
    def max_indicies(self):
        fW = self.filter_size[1]
        code = self._argmax.to(torch.int64)
        return code // fW, code % fW

    def backward(self, dvalues):
        dy = to_device(dvalues)
        if self.fused_bn is not None and self.fused_bn.pooled_now:
            self.dinputs = dy
            return self.dinputs
        S, H, W, Cc = self.inputs.shape
        fH, fW = self.filter_size
        sH, sW = self.strides
        dx = host().empty_like(self.inputs)
        host().aether_pool_bwd(dy, self._argmax, dx, S, H, W, Cc, fH, fW, sH, sW, self._kind())
        self.dinputs = dx
        return self.dinputs


# ------------------------------------------------------------------------------------- activations
class ReLU(_Saved):
    """Drop-in for ``ReLU`` (CNN_classes_cupy.py:406-415).  With ``fused_into_prev`` (set by
    ``Model.finalize(fuse=True)`` when the layer follows a Batch_Norm) the activation is applied by that
    Batch_Norm's kernels and this layer only hands tensors through."""
    _alpha = 0.0
    fused_into_prev = False
    # From this many values on a training pass keeps a bit of each for the way back, which then need not read the inputs again: arrays of 16 MB,
    # several of which L2 does not hold.  The seven layers' passes around it, us: 16 MB 67.4 -> 65.7, 32 MB 102.4 -> 99.8, 64 MB 190.3 -> 184.5,
    # 175 MB 567 -> 544; the layer alone 16 MB 17.0 -> 15.3, 64 MB 57.5 -> 48.1.
    MASK_FROM = 1 << 22
    _mask = None                # (bits, the inputs they are of, their version)

    def forward(self, inputs, training):
        x = to_device(inputs)
        if self.fused_into_prev:
            self.inputs = self.output = x
            return self.output
        h = host()
        y = h.empty_like(x)
        n = x.numel()
        version = h.counted(x) if training and n >= self.MASK_FROM and n % 4 == 0 else -1
        if version >= 0:                        # (a change between the passes would be noticed)
            bits = h.empty_u8(((n + 127) // 128 * 16,))
            h.aether_leaky_relu_fwd_mask(x, y, bits, n, self._alpha)
            self._mask = (bits, weakref.ref(x), version)
        else:
            self._mask = None
            h.aether_leaky_relu_fwd(x, y, n, self._alpha)
        self.inputs = x
        self.output = y
        return self.output

    def backward(self, dvalues):
        dy = to_device(dvalues)
        if self.fused_into_prev:
            self.dinputs = dy
            return self.dinputs
        h = host()
        dx = h.empty_like(dy)
        x, mask = self.inputs, self._mask
        if mask is not None and mask[1]() is x and mask[2] == x._version and dy.numel() == x.numel():
            h.aether_leaky_relu_bwd_mask(mask[0], dy, dx, dy.numel(), self._alpha)
        else:
            h.aether_leaky_relu_bwd(x, dy, dx, dy.numel(), self._alpha)
        self.dinputs = dx
        return self.dinputs


class Leaky_ReLU(ReLU):
    """Drop-in for ``Leaky_ReLU`` (CNN_classes_cupy.py:417-428)."""

    def __init__(self, alpha=0.01):
        self.alpha = alpha

    @property
    def _alpha(self):
        return self.alpha


# ------------------------------------------------------------------------------------- dropout
class Layer_Dropout_Spatial(_Saved):
    """Drop-in for ``Layer_Dropout_Spatial`` (CNN_classes_cupy.py:384-404): one Bernoulli(keep) draw per
    channel, shared by the whole batch, scaled by 1/keep.  The draw uses NumPy's global generator like
    the reference's NumPy twin; ``channel_mask`` (1,1,1,C) may be overwritten before ``forward`` by
    setting ``fixed_mask``.  Output stays fp32 (the reference promotes to fp64 through its mask)."""

    _next_seed = 0xC4A7

    def __init__(self, rate):
        self.rate = rate
        self.keep_prob = 1 - rate
        self.fixed_mask = None
        self.seed = Layer_Dropout_Spatial._next_seed
        Layer_Dropout_Spatial._next_seed += 1
        self.step_dev = None            # int64 device counter: draw the mask on the device (CUDA-graph train step)
        self.fused_into_prev = False    # the Batch_Norm in front applies the mask (Model.finalize(fuse=True))

    def _restore_transient(self):
        self.fixed_mask = None
        self.step_dev = None
        self.fused_into_prev = False

    def draw_mask(self, Cc):
        """Draws this step's channel mask (Bernoulli(keep)/keep per channel) into ``channel_mask``."""
        if self.fixed_mask is None and self.step_dev is not None:
            self.channel_mask = host().empty((1, 1, 1, Cc))
            host().aether_channel_mask_dev(self.channel_mask, Cc, self.keep_prob, self.seed, self.step_dev)
        else:
            if self.fixed_mask is not None:
                mask = np.ascontiguousarray(self.fixed_mask, dtype=np.float32).reshape(1, 1, 1, Cc)
            else:
                mask = (np.random.binomial(1, self.keep_prob, size=(1, 1, 1, Cc)) / self.keep_prob).astype(np.float32)
            self.channel_mask = host().upload(mask, (1, 1, 1, Cc))
        return self.channel_mask

    def forward(self, inputs, training):
        x = to_device(inputs)
        self.inputs = x
        if self.fused_into_prev:        # already masked by the fused Batch_Norm (training) / identity (inference)
            self.output = x
            return self.output
        if not training:
            self.output = _copied(x)
            return self.output
        Cc = x.shape[-1]
        self.draw_mask(Cc)
        h = host()
        y = h.empty_like(x)
        h.aether_channel_scale(x, self.channel_mask, y, x.numel(), Cc)
        self.output = y
        return self.output

    def backward(self, dvalues):
        dy = to_device(dvalues)
        if self.fused_into_prev:
            self.dinputs = dy
            return self.dinputs
        h = host()
        dx = h.empty_like(dy)
        h.aether_channel_scale(dy, self.channel_mask, dx, dy.numel(), dy.shape[-1])
        self.dinputs = dx
        return self.dinputs


class Layer_Dropout(_Saved):
    """Drop-in for ``Layer_Dropout`` (CNN_classes_cupy.py:364-382).  ``rate`` is the drop rate; the
    element mask Bernoulli(1-rate)/(1-rate) is drawn on the device from a Philox stream keyed by
    ``seed`` and a per-call offset (``rank_offset`` separates data-parallel ranks)."""
    _next_seed = 0x5EED

    def __init__(self, rate, seed=None, rank_offset=0):
        self.rate = 1 - rate          # the reference stores the KEEP probability under this name (:367)
        if seed is None:
            seed = Layer_Dropout._next_seed
            Layer_Dropout._next_seed += 1
        self.seed = int(seed)
        self.rank_offset = int(rank_offset)
        self._calls = 0
        self.step_dev = None

    def _restore_transient(self):
        self.step_dev = None

    def forward(self, inputs, training):
        x = to_device(inputs)
        self.inputs = x
        if not training:
            self.output = _copied(x)
            return self.output
        h = host()
        y = h.empty_like(x)
        self.binary_mask = h.empty_like(x)
        if self.step_dev is not None:   # the call counter lives on the device (CUDA-graph train step)
            h.aether_dropout_fwd_dev(x, y, self.binary_mask, x.numel(), self.rate, self.seed, self.rank_offset << 32, self.step_dev)
        else:
            offset = (self._calls << 40) + (self.rank_offset << 32)
            self._calls += 1
            h.aether_dropout_fwd(x, y, self.binary_mask, x.numel(), self.rate, self.seed, offset)
        self.output = y
        return self.output

    def backward(self, dvalues):
        dy = to_device(dvalues)
        h = host()
        dx = h.empty_like(dy)
        h.aether_mul(dy, self.binary_mask, dx, dy.numel())
        self.dinputs = dx
        return self.dinputs


# ------------------------------------------------------------------------------------- Batch_Norm
class Batch_Norm(_Saved):
    """Drop-in for ``Batch_Norm`` (CNN_classes_cupy.py:430-526) for 4-D (NHWC) and 2-D inputs.
    ``gamma``/``beta`` (aliased as ``weights``/``biases``) have shape (C,); ``running_mean`` /
    ``running_var`` / ``batch_mean`` / ``batch_var`` are exposed with the reference's keep-dims shape
    ((1,1,1,C) or (1,C)) as views of flat (C,) storage.  ``normalized`` is not stored: the backward
    kernel recomputes x-hat from the saved statistics."""

    def __init__(self, epsilon=1e-5, momentum=0.9, n_features=None):
        self.epsilon = epsilon
        self.momentum = momentum
        self.gamma = None
        self.beta = None
        self.running_mean = None
        self.running_var = None
        self.weight_regularizer_l1 = 0
        self.weight_regularizer_l2 = 0
        self.bias_regularizer_l1 = 0
        self.bias_regularizer_l2 = 0
        self._ws = _Workspace()
        self._ws_for = self._views = None
        self.stats_from = None          # a Conv_Layer whose forward leaves `bn_partials` for this layer's input
        self.fused_alpha = None         # slope of the (Leaky_)ReLU applied inside this layer's kernels (None: not fused)
        self.fused_dropout = None       # a Layer_Dropout_Spatial behind that activation whose mask is applied here too
        self.fused_pool = None          # a max Pooling behind those whose windows are reduced here too
        self.pooled_now = False         # the last forward produced the pooled tensor
        self.lean = False               # do not write fp32 tensors whose only reader takes the bf16 copy (finalize(lean=True))
        self.copy_consumer = None       # the layer that reads the pooled tensor as x (its bf16 copy is written here)
        self.copy_dy_consumer = None    # the Conv_Layer in front (the bf16 copy of its dvalues is written here)
        if n_features is not None:
            self._create(n_features)

    def _restore_transient(self):
        self._ws = _Workspace()
        self._ws_for = self._views = None
        self.stats_from = None
        self.fused_alpha = None
        self.fused_dropout = None
        self.fused_pool = None
        self.pooled_now = False
        self.lean = False
        self.copy_consumer = None
        self.copy_dy_consumer = None
        if getattr(self, "gamma", None) is not None:
            self.running_mean = self._rm
            self.running_var = self._rv
        else:
            self.running_mean = self.running_var = None

    def _create(self, Cc):
        dev = _device()
        self.gamma = torch.ones(Cc, dtype=torch.float32, device=dev)
        self.beta = torch.zeros(Cc, dtype=torch.float32, device=dev)
        self._rm = torch.zeros(Cc, dtype=torch.float32, device=dev)
        self._rv = torch.ones(Cc, dtype=torch.float32, device=dev)
        self.running_mean = self._rm
        self.running_var = self._rv

    @property
    def weights(self):
        return self.gamma

    @weights.setter
    def weights(self, v):
        self.gamma = v

    @property
    def biases(self):
        return self.beta

    @biases.setter
    def biases(self, v):
        self.beta = v

    def forward(self, inputs, training):
        x = to_device(inputs)
        if x.ndim not in (2, 4):
            raise ValueError(f"Expected a 2D or 4D tensor, got {x.ndim} instead.")
        Cc = x.shape[-1]
        if self.gamma is None:
            self._create(Cc)
        rows = x.numel() // Cc
        keep = (1,) * (x.ndim - 1) + (Cc,)
        h = host()
        ws = self._workspace(rows, Cc)
        part = None
        if training:
            self._bm = h.empty(keep)
            self._bv = h.empty(keep)
            part = getattr(self.stats_from, "bn_partials", None) if self.stats_from is not None else None
            if part is not None and part[2] != x.data_ptr():
                part = None
        # Whole block tail in one pass: activation, dropout mask and a max pooling whose windows tile the input are
        # applied while x is read once; the activated tensor is never written (block_fused.cu).
        pool = self.fused_pool
        self.pooled_now = False
        if pool is not None and self.fused_alpha is not None and x.ndim == 4 and Cc % 4 == 0:
            fH, fW = pool.filter_size
            S, H, W = x.shape[0], x.shape[1], x.shape[2]
            if H % fH == 0 and W % fW == 0:
                mask = self.fused_dropout.draw_mask(Cc) if (training and self.fused_dropout is not None) else None
                pshape = (S, H // fH, W // fW, Cc)
                pooled = h.empty(pshape)
                self._pool_arg = h.empty_u8(pshape)
                # the layer behind the pooling reads a bf16 copy of the pooled tensor: written by this same pass
                target = self.copy_consumer.x_copy_target(pshape) if self.copy_consumer is not None else None
                # x at every window's selected cell, for the backward statistics pass (training only)
                self._xsel = h.empty(pshape) if training else None
                h.aether_bn_act_pool_fwd_copy(x, part[0] if part else None, part[1] if part else 0, self.gamma, self.beta,
                                              self._rm, self._rv, self._bm if training else None, self._bv if training else None,
                                              None if (self.lean and target) else pooled, self._pool_arg, S, H, W, Cc, fH, fW,
                                              self.epsilon, self.momentum, self.fused_alpha, mask, 1 if training else 0,
                                              target[0] if target else None, target[1] if target else 0, self._xsel, ws,
                                              self._ws.size)
                if target:
                    if self.lean:
                        _mark_unwritten(pooled)
                    self.copy_consumer.x_copy_written(pooled)
                self._fused_mask = mask
                self.pooled_now = True
                if training:
                    self._expose_statistics(keep)
                self.inputs = x
                self.output = pooled
                return self.output
        y = h.empty_like(x)
        if training:
            if self.fused_alpha is not None:
                # y = act(bn(x)) [* spatial-dropout mask] in the same passes; the layers behind only hand y through
                mask = self.fused_dropout.draw_mask(Cc) if self.fused_dropout is not None else None
                h.aether_bn_act_fwd_train(x, part[0] if part else None, part[1] if part else 0, self.gamma, self.beta, self._rm,
                                          self._rv, self._bm, self._bv, y, rows, Cc, self.epsilon, self.momentum,
                                          self.fused_alpha, mask, ws, self._ws.size)
                self._fused_mask = mask
            elif part is not None:
                # the convolution that produced x already reduced it per channel: merge its partials, read x once
                h.aether_bn_fwd_train_partials(x, part[0], part[1], self.gamma, self.beta, self._rm, self._rv, self._bm, self._bv,
                                               y, rows, Cc, self.epsilon, self.momentum, ws, self._ws.size)
            else:
                h.aether_bn_fwd_train(x, self.gamma, self.beta, self._rm, self._rv, self._bm, self._bv, y, rows, Cc,
                                      self.epsilon, self.momentum, ws, self._ws.size)
            self._expose_statistics(keep)
        elif self.fused_alpha is not None:
            h.aether_bn_act_fwd_eval(x, self.gamma, self.beta, self._rm, self._rv, y, rows, Cc, self.epsilon, self.fused_alpha, ws,
                                     self._ws.size)
        else:
            h.aether_bn_fwd_eval(x, self.gamma, self.beta, self._rm, self._rv, y, rows, Cc, self.epsilon, ws, self._ws.size)
        self.inputs = x
        self.output = y
        return self.output

    def _workspace(self, rows, Cc):
        if self._ws_for != (rows, Cc):
            self._ws_bytes = int(lib().aether_bn_workspace_bytes(rows, Cc))
            self._ws_for = (rows, Cc)
        return self._ws.get(self._ws_bytes)

    def _expose_statistics(self, keep):
        self.batch_mean = self._bm
        self.batch_var = self._bv
        if self._views is None or self._views[0] is not self._rm or self._views[1] is not self._rv or self._views[2] != keep:
            self._views = (self._rm, self._rv, keep, self._rm.view(keep), self._rv.view(keep))
        self.running_mean = self._views[3]       # the reference's stats pick up keep-dims here (:475-476)
        self.running_var = self._views[4]

    def backward(self, dvalues):
        dy = to_device(dvalues)
        x = self.inputs
        Cc = x.shape[-1]
        rows = x.numel() // Cc
        h = host()
        ws = self._workspace(rows, Cc)
        dx = h.empty_like(x)
        if getattr(self, "_grad_views", None) is not None:
            self.dweights, self.dbiases = self._grad_views
        else:
            self.dweights = h.empty((Cc,))
            self.dbiases = h.empty((Cc,))
        if self.pooled_now:                  # dvalues is the gradient w.r.t. the POOLED output of the fused block tail
            S, H, W = x.shape[0], x.shape[1], x.shape[2]
            fH, fW = self.fused_pool.filter_size
            # dx is the dvalues of the convolution in front: its bf16 copy and the column sums for that layer's bias
            # gradient are written by this same pass
            conv = self.copy_dy_consumer
            target = conv.dy_copy_target() if (conv is not None and conv.output is x and 256 % max(Cc // 4, 1) == 0
                                               and Cc // 4 <= 256) else None
            sums = h.aether_bn_act_pool_bwd_copy(x, dy, self._pool_arg, self.gamma, self.beta, self._bm, self._bv,
                                                 None if (self.lean and target) else dx, self.dweights, self.dbiases, S, H, W, Cc,
                                                 fH, fW, self.epsilon, self.fused_alpha, getattr(self, "_fused_mask", None),
                                                 target[0] if target else None, target[1] if target else 0,
                                                 target[2] if target else None, target[3] if target else 0,
                                                 getattr(self, "_xsel", None), ws, self._ws.size)
            if target:
                if self.lean:
                    _mark_unwritten(dx)
                conv.dy_copy_written(dx, sums)
        elif self.fused_alpha is not None:   # dvalues is the gradient w.r.t. the ACTIVATED output
            h.aether_bn_act_bwd(x, self.beta, dy, self.gamma, self._bm, self._bv, dx, self.dweights, self.dbiases, rows, Cc,
                                self.epsilon, self.fused_alpha, getattr(self, "_fused_mask", None), ws, self._ws.size)
        else:
            h.aether_bn_bwd(x, dy, self.gamma, self._bm, self._bv, dx, self.dweights, self.dbiases, rows, Cc, self.epsilon, ws,
                            self._ws.size)
        self.dinputs = dx
        return self.dinputs

    def get_parameters(self):
        return self.gamma, self.beta, self.running_mean, self.running_var

    def set_parameters(self, gamma, beta, running_mean, running_var):
        g = to_device(gamma).reshape(-1)
        if self.gamma is None:
            self._create(g.numel())
        self.gamma.copy_(g)
        self.beta.copy_(to_device(beta).reshape(-1))
        self._rm.copy_(to_device(running_mean).reshape(-1))
        self._rv.copy_(to_device(running_var).reshape(-1))


# ------------------------------------------------------------------------------------- Flatten / Dense
class Flatten(_Saved):
    """Drop-in for ``Flatten`` (CNN_classes_cupy.py:528-539); a view, no kernel."""

    def forward(self, inputs, training):
        x = to_device(inputs)
        self.inputs_shape = x.shape
        self.output = x.reshape(x.shape[0], -1)
        if getattr(x, "_aether_unwritten", False):
            _mark_unwritten(self.output)
        return self.output

    def backward(self, dvalues):
        self.dinputs = to_device(dvalues).reshape(self.inputs_shape)
        return self.dinputs


class Layer_Dense(_TakesCopies, _Saved):
    """Drop-in for ``Layer_Dense`` (CNN_classes_cupy.py:315-362).  The three products run through the
    convolution kernels as a 1x1 convolution on a 1x1 image (x (S,n_in) is NHWC with H=W=1; weights
    (n_in,n_out) are a (1,1,Cin,Cout) filter), so they use the same tensor-core path.  Parameters are
    fp32 (the reference's are fp64 because ``randn`` is); biases keep the (1, n_out) shape."""

    def __init__(self, n_inputs, n_neurons, weight_regularizer_l1=0, bias_regularizer_l1=0,
                 weight_regularizer_l2=0, bias_regularizer_l2=0, math_mode=None):
        w = 0.01 * np.random.randn(n_inputs, n_neurons) * np.sqrt(2.0 / n_inputs)       # :320-321
        self.weights = to_device(w.astype(np.float32))
        self.biases = torch.zeros((1, n_neurons), dtype=torch.float32, device=_device())
        self.weight_regularizer_l1 = weight_regularizer_l1
        self.weight_regularizer_l2 = weight_regularizer_l2
        self.bias_regularizer_l1 = bias_regularizer_l1
        self.bias_regularizer_l2 = bias_regularizer_l2
        self.math_mode = math_mode or DEFAULT_MATH_MODE
        self._ws = _Workspace()
        self._plans = {}
        self._copies = _OperandCopies()
        self._handed = _HandedIn()
        self._used = (None, None)       # plan and weights of the last forward pass

    def _restore_transient(self):
        self._ws = _Workspace()
        self._plans = {}
        self._copies = _OperandCopies()
        self._handed = _HandedIn()
        self._used = (None, None)       # plan and weights of the last forward pass

    def _last_plan(self):
        return self._used[0], self.weights

    def x_copy_target(self, shape):
        """(address, row length) where the bf16 copy of an input of `shape` (any shape that flattens to
        (samples, n_inputs), e.g. the pooled NHWC tensor in front of a Flatten) goes, or None."""
        n_in = self.weights.shape[0]
        total = 1
        for v in shape:
            total *= int(v)
        if len(shape) < 2 or total != int(shape[0]) * n_in:
            return None
        p = self._plan(int(shape[0]))
        lay = p.layout
        # A row of the copy is one SAMPLE here, but the producer writes one PIXEL (shape[-1] channels) per row: the two
        # are the same bytes only when the sample's row is not padded (n_inputs a multiple of 64).
        if lay is None or lay.x_copy_ld != n_in:
            return None
        ws = self._ws.get(p.ws_bytes)
        return ws.data_ptr() + lay.x_copy_offset, int(shape[-1])

    def x_copy_written(self, x):
        self._handed.x = (self._ws.buf.data_ptr(), _array_tag(x))

    def _plan(self, S):
        n_in, n_out = self.weights.shape
        key = (S, n_in, n_out, self.math_mode, host().device())
        p = self._plans.get(key)
        if p is None:
            if len(self._plans) >= 64:
                self._plans.clear()
            p = self._plans[key] = _ConvPlan(AetherConvDesc(S, 1, 1, n_in, n_out, 1, 1, 1, 1, 0, 0, _lib.MATH_MODES[self.math_mode]), 1, 1)
        return p

    def _current(self):
        """The plan of the last forward pass (looked up again when its inputs or weights have been replaced since): looking
        it up costs a microsecond, and a small network's step is bound by what its calls cost the host."""
        p, w = self._used
        if p is None or w is not self.weights or p.x_shape[0] != self.inputs.shape[0]:
            p = self._plan(self.inputs.shape[0])
        return p

    def _operands(self, x, p, training=True):
        """(workspace, which operand copies in it are valid) for a forward pass over `x` by plan `p`."""
        ws = self._ws.get(p.ws_bytes if training else p.fwd_ws_bytes, p)
        flags = 0
        if self._handed.x is not None:
            flags = _lib.CONV_X_COPY_READY if self._handed.x_ready(ws, x) else 0
            self._handed.x = None
        if not flags:
            _require_written(x, "Layer_Dense.forward")
        if self._weights_fixed and p.layout is not None and self._copies.weights_valid(ws, self.weights):
            flags |= _lib.CONV_W_COPY_READY
            if self._branch is not None:
                self._branch.join()
        return ws, flags

    def forward(self, inputs, training):
        x = to_device(inputs)
        w = self.weights
        if x.ndim != 2 or x.shape[1] != w.shape[0]:
            raise ValueError(f"Layer_Dense expects (samples, {w.shape[0]}), got {tuple(x.shape)}")
        p = self._plan(x.shape[0])
        H = host()
        y = H.empty((x.shape[0], w.shape[1]))
        ws, flags = self._operands(x, p, training)
        H.aether_conv2d_fwd_ex(p.raw, x, w, self.biases, y, None, 0, ws, self._ws.size, flags)
        self.inputs = x
        self.output = y
        self._used = (p, w)
        self._copies.record(ws, x, w)
        return y

    def forward_act(self, x, alpha, target, p):
        """`forward` and the (leaky) ReLU behind it in one call (Model): (output, activation's output)."""
        w = self.weights
        ws, flags = self._operands(x, p)
        H = host()
        shape = (p.x_shape[0], p.b_shape[0])
        y, z = H.empty(shape), H.empty(shape)
        H.aether_conv2d_act_fwd(p.raw, x, w, self.biases, y, z, alpha, target[0] if target else None, target[1] if target else 0, ws,
                                self._ws.size, flags)
        self.inputs = x
        self.output = y
        self._used = (p, w)
        self._copies.record(ws, x, w)
        return y, z

    def forward_softmax(self, x, p):
        """`forward` of a classifier head and the SoftMax behind it in one launch (Model): (output, probabilities)."""
        w = self.weights
        ws, _ = self._operands(x, p)
        H = host()
        shape = (p.x_shape[0], p.b_shape[0])
        y, prob = H.empty(shape), H.empty(shape)
        H.aether_head_softmax_fwd(p.raw, x, w, self.biases, y, prob)
        self.inputs = x
        self.output = y
        self._used = (p, w)
        self._copies.record(ws, x, w)
        return y, prob

    def backward_softmax(self, prob, labels, smooth, p):
        """The combined softmax / cross-entropy gradient and this head's `backward`: the gradient with respect to the logits."""
        self._gradients()
        H = host()
        dz, dx = H.empty_like(prob), H.empty_like(self.inputs)
        kinds = [None, None, None]
        kinds[2 if labels.ndim == 2 else 1 if labels.dtype is torch.int64 else 0] = labels
        x, w = self.inputs, self.weights
        ws = self._ws.get(p.ws_bytes)
        if not (self._copies.flags(ws, x, w) & _lib.CONV_X_COPY_READY):
            _require_written(x, "Layer_Dense.backward")
        H.aether_head_cce_bwd_ex(p.raw, prob, *kinds, smooth, x, w, dz, dx, self.dweights, self.dbiases, ws, self._ws.size)
        self._regularize()
        self.dinputs = dx
        return dz

    def _gradients(self):
        if getattr(self, "_grad_views", None) is not None:
            self.dweights, self.dbiases = self._grad_views
        else:
            H = host()
            self.dweights = H.empty_like(self.weights)
            self.dbiases = H.empty_like(self.biases)

    def backward(self, dvalues):
        self._gradients()
        return self._backward(to_device(dvalues), False, self._current())

    def backward_act(self, act_inputs, dvalues, alpha, p):
        """`backward` of the (leaky) ReLU behind this layer and of the layer itself: (the activation's dinputs, dinputs)."""
        self._gradients()
        H = host()
        lay = p.layout
        dy = H.empty_like(act_inputs)
        H.aether_act_bwd_copy(act_inputs, dvalues, dy, p.x_shape[0], p.b_shape[0], alpha, self._ws.get(p.ws_bytes).data_ptr() + lay.dy_copy_offset,
                              lay.dy_copy_ld, self.dbiases)
        return dy, self._backward(dy, True, p)

    def _backward(self, dy, dy_ready, p):
        """``dy_ready``: the operand copy of dy and dbiases are there already."""
        x = self.inputs
        w = self.weights
        H = host()
        dx = H.empty_like(x)
        ws = self._ws.get(p.ws_bytes, p)
        flags = self._copies.flags(ws, x, w)
        if not (flags & _lib.CONV_X_COPY_READY):
            _require_written(x, "Layer_Dense.backward")
        db, rows = self.dbiases, 0
        if dy_ready:
            db, rows, flags = None, 1, flags | _lib.CONV_DY_COPY_READY
        if self._branch is None:
            H.aether_conv2d_bwd_ex(p.raw, x, dy, w, dx, self.dweights, db, ws, self._ws.size, flags, rows)
            self._regularize()
        else:
            self._products(p, x, dy, w, dx, db, ws, flags, rows, self._regularize)
        self.dinputs = dx
        return self.dinputs

    def _regularize(self):
        w = self.weights
        if self.weight_regularizer_l1 > 0 or self.weight_regularizer_l2 > 0:
            host().aether_regularizer_grad(w, self.dweights, w.numel(), self.weight_regularizer_l1, self.weight_regularizer_l2)
        if self.bias_regularizer_l1 > 0 or self.bias_regularizer_l2 > 0:
            host().aether_regularizer_grad(self.biases, self.dbiases, self.biases.numel(), self.bias_regularizer_l1,
                                           self.bias_regularizer_l2)

    def get_parameters(self):
        return self.weights, self.biases

    def set_parameters(self, weights, biases):
        self.weights.copy_(to_device(weights))
        self.biases.copy_(to_device(biases).reshape(1, -1))


# ------------------------------------------------------------------------------------- softmax / loss
def _labels_i32(y_true):
    """Targets as the kernels take them: class indices (int32, shape (rows,)) or, for 2-D input, the rows of target
    probabilities themselves (float32): one-hot or soft, the loss uses them as they are (CNN_classes_cupy.py:625-637)."""
    y = y_true if isinstance(y_true, torch.Tensor) else torch.as_tensor(np.asarray(y_true))
    if y.ndim == 2:
        return to_device(y, torch.float32)
    return to_device(y, torch.int32)


def _labels(y_true):
    """``_labels_i32`` without the conversion of 64-bit class indices that are on the device already: the kernel takes them."""
    if isinstance(y_true, torch.Tensor) and y_true.dtype is torch.int64 and y_true.ndim == 1 and y_true.is_cuda and y_true.is_contiguous():
        return y_true
    return _labels_i32(y_true)


def _softmax_cce(z, labels, want_prob, want_loss, want_dz, want_correct, smooth_fwd, smooth_bwd, input_is_prob=False):
    rows, classes = z.shape
    h = host()
    prob = h.empty((rows, classes)) if want_prob else None
    loss = h.empty((rows,)) if want_loss else None
    dz = h.empty((rows, classes)) if want_dz else None
    correct = h.empty_i32((rows,)) if want_correct else None
    if labels is not None and labels.ndim == 2:
        if tuple(labels.shape) != (rows, classes):
            raise ValueError(f"targets have shape {tuple(labels.shape)}, expected {(rows, classes)}")
        h.aether_softmax_cce_targets(z, labels, prob, loss, dz, correct, rows, classes, smooth_fwd, smooth_bwd, 1 if input_is_prob else 0)
    elif labels is not None and labels.dtype is torch.int64:
        h.aether_softmax_cce_i64(z, labels, prob, loss, dz, correct, rows, classes, smooth_fwd, smooth_bwd, 1 if input_is_prob else 0)
    else:
        h.aether_softmax_cce(z, labels, prob, loss, dz, correct, rows, classes, smooth_fwd, smooth_bwd, 1 if input_is_prob else 0)
    return prob, loss, dz, correct


class SoftMax(_Saved):
    """Drop-in for ``SoftMax`` (CNN_classes_cupy.py:541-563).  ``backward`` is the reference's stand-alone Jacobian
    product (:549-560), as one kernel instead of a Python loop over the samples; networks that end in SoftMax +
    categorical cross-entropy take the combined backward (:666-680) and never call it."""

    def forward(self, inputs, training=True):
        z = to_device(inputs)
        self.inputs = z
        self.output, _, _, _ = _softmax_cce(z, None, True, False, False, False, 0.0, 0.0)
        return self.output

    def backward(self, dvalues):
        dv = to_device(dvalues)
        if tuple(dv.shape) != tuple(self.output.shape):
            raise ValueError(f"dvalues has shape {tuple(dv.shape)}, expected {tuple(self.output.shape)}")
        dx = host().empty_like(dv)
        host().aether_softmax_bwd(self.output, dv, dx, dv.shape[0], dv.shape[1])
        self.dinputs = dx
        return self.dinputs

    def predictions(self, outputs):
        return to_device(outputs).argmax(dim=1)


class Loss(_Saved):
    """Accumulating loss base class, ``Loss`` (CNN_classes_cupy.py:565-609)."""

    def remember_trainable_layers(self, trainable_layers):
        self.trainable_layers = trainable_layers

    def calculate(self, output, y, *, include_regularization=False, training=True):
        sample_losses = self.forward(output, y, training)
        data_loss = sample_losses.mean()
        self.accumulated_sum += sample_losses.sum()
        self.accumulated_count += len(sample_losses)
        if not include_regularization:
            return data_loss
        return data_loss, self.regularization_loss()

    def calculate_accumulated(self, *, include_regularization=False):
        data_loss = self.accumulated_sum / self.accumulated_count
        if not include_regularization:
            return data_loss
        return data_loss, self.regularization_loss()

    def new_pass(self):
        self.accumulated_sum = 0
        self.accumulated_count = 0

    def regularization_loss(self):
        out = None
        for layer in self.trainable_layers:
            for arr, l1, l2 in ((layer.weights, layer.weight_regularizer_l1, layer.weight_regularizer_l2),
                                (layer.biases, layer.bias_regularizer_l1, layer.bias_regularizer_l2)):
                if l1 > 0 or l2 > 0:
                    if out is None:
                        out = torch.zeros(1, dtype=torch.float32, device=_device())
                    host().aether_regularizer_loss(arr, arr.numel(), l1, l2, out)
        return out[0] if out is not None else 0


class Loss_CategoricalCrossEntropy(Loss):
    """Drop-in for ``Loss_CategoricalCrossEntropy`` (CNN_classes_cupy.py:611-652); ``y_pred`` are
    probabilities, ``y_true`` class indices or one-hot rows."""

    def __init__(self, label_smoothing=0.0):
        self.label_smoothing = label_smoothing

    def forward(self, y_pred, y_true, training=True):
        p = to_device(y_pred)
        smooth = self.label_smoothing if training else 0.0
        _, loss, _, _ = _softmax_cce(p, _labels(y_true), False, True, False, False, smooth, 0.0, input_is_prob=True)
        return loss

    def backward(self, dvalues, y_true):
        p = to_device(dvalues)
        _, _, dz, _ = _softmax_cce(p, _labels(y_true), False, False, True, False, 0.0, self.label_smoothing,
                                   input_is_prob=True)
        self.dinputs = dz
        return self.dinputs


class Activation_Softmax_Loss_CategoricalCrossEntropy:
    """Drop-in for the combined class (CNN_classes_cupy.py:654-680); ``backward`` takes the softmax
    OUTPUT and returns (p - y_smooth)/samples."""

    def __init__(self, label_smoothing=0.0):
        self.activation = SoftMax()
        self.loss = Loss_CategoricalCrossEntropy(label_smoothing)
        self.label_smoothing = label_smoothing

    def forward(self, inputs, y_true, training=True):
        self.activation.forward(inputs, training)
        self.output = self.activation.output
        return self.loss.calculate(self.output, y_true, training=training)

    def backward(self, dvalues, y_true, training=True):
        p = to_device(dvalues)
        smooth = self.label_smoothing if training else 0.0
        _, _, dz, _ = _softmax_cce(p, _labels(y_true), False, False, True, False, 0.0, smooth, input_is_prob=True)
        self.dinputs = dz
        return self.dinputs


# ------------------------------------------------------------------------------------- Adam
class Optimizer_Adam(_Saved):
    """Drop-in for ``Optimizer_Adam`` (CNN_classes_cupy.py:685-736).  State lives on the layer under the
    reference's attribute names (``weight_momentums``, ``weight_cache``, ``bias_momentums``,
    ``bias_cache``) and parameters are updated in place.  ``grad_scale`` multiplies every gradient
    first (1/world_size turns an all-reduced sum into the data-parallel average)."""

    def __init__(self, learning_rate=.001, decay=0., epsilon=1e-7, beta_1=0.9, beta_2=.999):
        self.learning_rate = learning_rate
        self.current_learning_rate = learning_rate
        self.decay = decay
        self.iterations = 0
        self.epsilon = epsilon
        self.beta_1 = beta_1
        self.beta_2 = beta_2
        self.grad_scale = 1.0
        self.step_dev = None            # int64 device copy of `iterations` (CUDA-graph train step)

    def _restore_transient(self):
        self.step_dev = None

    def pre_update_parameters(self):
        if self.decay:
            self.current_learning_rate = self.learning_rate * (1. / (1. + self.decay * self.iterations))

    def _step(self, p, g, m, v):
        if self.step_dev is not None:   # iterations, decay and bias corrections evaluated on the device
            host().aether_adam_step_dev(p, g, m, v, p.numel(), self.learning_rate, self.decay, self.beta_1, self.beta_2,
                                        self.epsilon, self.grad_scale, self.step_dev)
            return
        t = self.iterations + 1
        host().aether_adam_step(p, g, m, v, p.numel(), self.current_learning_rate, self.beta_1, self.beta_2, self.epsilon,
                                1 - self.beta_1 ** t, 1 - self.beta_2 ** t, self.grad_scale)

    @staticmethod
    def _ensure_state(layer):
        if not hasattr(layer, "weight_cache"):
            layer.weight_momentums = torch.zeros_like(layer.weights)
            layer.weight_cache = torch.zeros_like(layer.weights)
            layer.bias_momentums = torch.zeros_like(layer.biases)
            layer.bias_cache = torch.zeros_like(layer.biases)

    def update_parameters(self, layer):
        self._ensure_state(layer)
        self._step(layer.weights, layer.dweights, layer.weight_momentums, layer.weight_cache)
        self._step(layer.biases, layer.dbiases, layer.bias_momentums, layer.bias_cache)

    def updates_as_adam(self):
        """Whether ``update_layers`` does what calling ``update_parameters`` for each layer does: not where a subclass or a
        patched method updates in its own way."""
        cls, own = type(self), self.__dict__
        return (cls.update_parameters is Optimizer_Adam.update_parameters and cls._step is Optimizer_Adam._step
                and cls._ensure_state is Optimizer_Adam._ensure_state
                and not ("update_parameters" in own or "_step" in own or "_ensure_state" in own))

    def update_layers(self, layers):
        """``update_parameters`` of every layer in one launch (a layer by itself is two launches of a few microseconds)."""
        if self.step_dev is not None:
            for layer in layers:
                self.update_parameters(layer)
            return
        arrays = []
        for layer in layers:
            self._ensure_state(layer)
            arrays += (layer.weights, layer.dweights, layer.weight_momentums, layer.weight_cache,
                       layer.biases, layer.dbiases, layer.bias_momentums, layer.bias_cache)
        t = self.iterations + 1
        host().aether_adam_steps(arrays, self.current_learning_rate, self.beta_1, self.beta_2, self.epsilon,
                                 1 - self.beta_1 ** t, 1 - self.beta_2 ** t, self.grad_scale)

    def update_flat(self, params, grads, m, v):
        """One launch over a flat parameter buffer (used by the data-parallel trainer)."""
        self._step(params, grads, m, v)

    def post_update_parameters(self):
        self.iterations += 1
