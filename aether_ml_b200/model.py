"""``Model`` orchestration with the public surface of Aether-ML's ``CNN/models/CNN_model_cupy.py``
(add / set / finalize / train / forward / backward / evaluate / predict / get_parameters /
set_parameters / save_parameters / load_parameters), driving the device layers of
:mod:`aether_ml_b200.layers`.  It holds no arithmetic: layers are duck-typed exactly as in the
reference (``forward(inputs, training)`` sets ``.output``, ``backward(dvalues)`` sets ``.dinputs``;
a layer is trainable when it has a ``weights`` attribute, CNN_model_cupy.py:52-53).

Additions that the reference does not have, all optional:
  * ``finalize(flat=True)`` packs every trainable layer's parameters and gradients into two flat
    device buffers (views keep the per-layer attribute names), so one Adam launch and -- under data
    parallelism -- one all-reduce cover the whole network;
  * ``train_step(X, y)`` runs one forward/backward/update without printing or host synchronisation.
"""
import contextlib
import math
import pickle
import weakref

import numpy as np
import torch

from ._lib import host
from .layers import (Activation_Softmax_Loss_CategoricalCrossEntropy, Batch_Norm, Conv_Layer, Flatten, Layer_Dense, Layer_Dropout,
                     Layer_Dropout_Spatial, Leaky_ReLU, Loss_CategoricalCrossEntropy, Optimizer_Adam, Pooling, ReLU, SoftMax, to_device, _Branch, _labels,
                     _labels_i32, _link, _softmax_cce, _Saved, _TakesCopies, _Workspace)


class Layer_Input:
    """Feeds the batch to the first layer (CNN_model_cupy.py:389-391)."""

    def forward(self, inputs, training):
        self.output = inputs


class Accuracy(_Saved):
    """Running accuracy (CNN_model_cupy.py:344-363)."""

    def calculate(self, predictions, y):
        hits = self.compare(predictions, y)
        self.accumulated_sum += hits.sum()
        self.accumulated_count += len(hits)
        return hits.float().mean()

    def calculate_accumulated(self):
        return self.accumulated_sum / self.accumulated_count

    def new_pass(self):
        self.accumulated_sum = 0
        self.accumulated_count = 0


class Accuracy_Categorical(Accuracy):
    """CNN_model_cupy.py:380-387: exact match of class indices (one-hot targets are arg-maxed)."""

    def init(self, y):
        pass

    def compare(self, predictions, y):
        y = y if isinstance(y, torch.Tensor) else torch.as_tensor(np.asarray(y))
        y = y.to(predictions.device)
        if y.ndim == 2:
            y = y.argmax(dim=1)
        return predictions == y


class Accuracy_Regression(Accuracy):
    """CNN_model_cupy.py:367-378: |prediction - y| below std(y)/250."""

    def __init__(self):
        self.precision = None

    def init(self, y, reinit=False):
        if self.precision is None or reinit:
            self.precision = float(np.std(np.asarray(y.cpu() if isinstance(y, torch.Tensor) else y))) / 250

    def compare(self, predictions, y):
        y = to_device(y)
        return (predictions - y).abs() < self.precision


def _batches(n, batch_size):
    if batch_size is None:
        return [slice(None)]
    steps = -(-n // batch_size)
    return [slice(k * batch_size, (k + 1) * batch_size) for k in range(steps)]


def _links(parts):
    """How layers that follow each other are wired: (layer, attribute, the weak reference it holds) going forward and going
    back, one reference object for all that refer to the same layer."""
    return [[(p, name, p.__dict__.get(name)) for p in some] for name, some in (("_link_prev", parts[1:]), ("_link_next", parts[:-1]))]


def _as_wired(links):
    for part, name, ref in links:
        if part.__dict__.get(name) is not ref:
            return False
    return True


class _Chain:
    """A Batch_Norm and the layers right behind it -- (Leaky_)ReLU, optional Layer_Dropout_Spatial, optional max Pooling whose
    stride is its window -- that a model with unfused layers runs in one pass each way (aether_chain_fwd / _bwd): every
    layer keeps the inputs, outputs and gradients it would have produced by itself, written from registers instead of
    one layer after the other.  Decided anew on each pass: anything out of the ordinary (a subclass, a patched method,
    replaced layers, shapes the kernels do not take) runs layer by layer."""

    def __init__(self, parts, conv, consumer):
        self.parts = parts                      # [bn, act[, drop][, pool]]
        self.links = _links(parts)
        self.length = len(parts)
        self.bn, self.act = parts[0], parts[1]
        self.drop = next((l for l in parts if isinstance(l, Layer_Dropout_Spatial)), None)
        self.pool = next((l for l in parts if isinstance(l, Pooling)), None)
        self.conv = conv                        # the Conv_Layer in front: takes the bf16 copy of dx
        self.consumer = consumer                # the layer behind: takes the bf16 copy of the last output
        self.live = None                        # the arrays of the last training pass, while they stand

    @staticmethod
    def find(layers, i):
        """The chain that starts at layers[i], or None."""
        def at(k):
            return layers[k] if k < len(layers) else None
        bn, act = at(i), at(i + 1)
        if type(bn) is not Batch_Norm or type(act) not in (ReLU, Leaky_ReLU):
            return None
        parts, k = [bn, act], i + 2
        if type(at(k)) is Layer_Dropout_Spatial:
            parts.append(at(k))
            k += 1
        pool = at(k)
        if (type(pool) is Pooling and pool.pooling_type == "max" and pool.padding == "valid" and tuple(pool.strides) == tuple(pool.filter_size)
                and pool.filter_size[0] * pool.filter_size[1] <= 255):
            parts.append(pool)
            k += 1
        conv = layers[i - 1] if i > 0 and type(layers[i - 1]) is Conv_Layer else None
        behind = at(k)
        if isinstance(behind, Flatten):
            behind = at(k + 1)
        return _Chain(parts, conv, behind if hasattr(behind, "x_copy_target") else None)

    def _intact(self, layers, i, back):
        if layers[i:i + self.length] != self.parts or not _as_wired(self.links[back]):
            return False
        for part in self.parts:
            d = part.__dict__
            if "forward" in d or "backward" in d:
                return False
        pool = self.pool
        return (self.bn.fused_alpha is None and not self.act.fused_into_prev and (self.drop is None or not self.drop.fused_into_prev)
                and (pool is None or (pool.fused_bn is None and pool.pooling_type == "max" and pool.padding == "valid"
                                      and tuple(pool.strides) == tuple(pool.filter_size))))

    def forward(self, layers, i, inputs, training, keep_all=True):
        """Runs the chain's layers; False when they have to run one by one.  An inference pass with ``keep_all=False`` writes
        the last layer's output only and leaves the attributes of the others alone."""
        self.live = None
        if not self._intact(layers, i, False):
            return False
        x = to_device(inputs)
        bn, act, drop, pool = self.bn, self.act, self.drop, self.pool
        shape = x.shape
        Cc = shape[-1]
        if Cc % 4 or x.ndim not in (2, 4) or (pool is not None and x.ndim != 4) or x.numel() == 0:
            return False
        S, H, W = (shape[0], shape[1], shape[2]) if x.ndim == 4 else (shape[0], 1, 1)
        fH, fW = pool.filter_size if pool is not None else (1, 1)
        alpha = act._alpha
        if H < fH or W < fW or not 0.0 <= alpha < 1.0 or x.numel() >= 1 << 32:
            return False
        if bn.gamma is None:
            bn._create(Cc)
        h = host()
        ws = bn._workspace(S * H * W, Cc)
        keep = (1,) * (x.ndim - 1) + (Cc,)
        part = mask = None
        if training:
            bn._bm, bn._bv = h.empty(keep), h.empty(keep)
            part = bn.stats_from.bn_partials if bn.stats_from is not None else None
            if part is not None and part[2] != x.data_ptr():
                part = None
            if drop is not None:
                mask = drop.draw_mask(Cc)
        bn_out = act_out = drop_out = pooled = arg = None
        if training or keep_all:
            bn_out, last = h.empty(shape), h.empty(shape)
            act_out = last
            if drop is not None:
                last = drop_out = h.empty(shape)
            if pool is not None:
                pshape = (S, H // fH, W // fW, Cc)
                last = pooled = h.empty(pshape)
                arg = h.empty_u8(pshape)
        elif pool is not None:
            last = pooled = h.empty((S, H // fH, W // fW, Cc))
        else:                                   # (spatial dropout does nothing in inference)
            last = act_out = h.empty(shape)
        target = self.consumer.x_copy_target(tuple(last.shape)) if self.consumer is not None else None
        h.aether_chain_fwd(x, part[0] if part else None, part[1] if part else 0, bn.gamma, bn.beta, bn._rm, bn._rv,
                           bn._bm if training else None, bn._bv if training else None, bn_out, act_out, drop_out, pooled, arg, S, H, W,
                           Cc, fH, fW, bn.epsilon, bn.momentum, alpha, mask, 1 if training else 0, target[0] if target else None,
                           target[1] if target else 0, ws, bn._ws.size)
        if training:
            bn._expose_statistics(keep)
        if target:
            self.consumer.x_copy_written(last)
        if bn_out is None:
            self.parts[-1].output = last
            return True
        bn.pooled_now = False
        bn.inputs, bn.output = x, bn_out
        act.inputs, act.output = bn_out, act_out
        if drop is not None:
            drop.inputs, drop.output = act_out, drop_out
        if pool is not None:
            pool.inputs, pool.output, pool._argmax = (act_out if drop is None else drop_out), pooled, arg
        if training:
            self.live = (x, x._version, bn_out, bn_out._version, ws, mask, S, H, W, Cc, fH, fW, alpha)
        return True

    def backward(self, layers, i, dvalues):
        """Runs the chain's backward passes; False when they have to run one by one."""
        live, self.live = self.live, None
        bn, act, drop, pool = self.bn, self.act, self.drop, self.pool
        if live is None or not self._intact(layers, i, True):
            return False
        x, x_version, bn_out, version, ws, mask, S, H, W, Cc, fH, fW, alpha = live
        if (bn.inputs is not x or act.inputs is not bn_out or bn_out._version != version or x._version != x_version or bn._ws.buf is not ws or act._alpha != alpha
                or (drop is not None and drop.channel_mask is not mask)):
            return False
        dy = to_device(dvalues)
        if pool is None and dy.shape != x.shape:
            return False
        h = host()
        shape = x.shape
        pool_dx = h.empty(shape) if pool is not None else None
        drop_dx = h.empty(shape) if drop is not None else None
        act_dx, dx = h.empty(shape), h.empty(shape)
        if getattr(bn, "_grad_views", None) is not None:
            bn.dweights, bn.dbiases = bn._grad_views
        else:
            bn.dweights, bn.dbiases = h.empty((Cc,)), h.empty((Cc,))
        conv = self.conv
        target = None
        if conv is not None and conv.output is x and Cc // 4 <= 256 and 256 % (Cc // 4) == 0:
            target = conv.dy_copy_target()
        rows = h.aether_chain_bwd(x, dy, pool._argmax if pool is not None else None, bn.gamma, bn._bm, bn._bv, pool_dx, drop_dx, act_dx, dx,
                                  bn.dweights, bn.dbiases, S, H, W, Cc, fH, fW, bn.epsilon, alpha, mask, target[0] if target else None,
                                  target[1] if target else 0, target[2] if target else None, target[3] if target else 0, ws, bn._ws.size)
        if pool is not None:
            pool.dinputs = pool_dx
        if drop is not None:
            drop.dinputs = drop_dx
        act.dinputs, bn.dinputs = act_dx, dx
        if target:
            conv.dy_copy_written(dx, rows)
        return True


_OWN = Conv_Layer.__module__     # where this package's layers are


class _ConvChain:
    """A Conv_Layer and the chain behind it that ends in a 2x2 max Pooling, which an inference pass whose layers keep nothing runs in one launch: the
    convolution's epilogue goes on to the pooled output, and the arrays in between are never written.  Conditions as for _Chain."""

    def __init__(self, conv, chain):
        self.conv, self.chain = conv, chain
        self.links = _links([conv, chain.bn])
        self.length = 1 + chain.length

    @staticmethod
    def find(layers, i, chain):
        pool = chain.pool
        if type(layers[i]) is Conv_Layer and pool is not None and tuple(pool.filter_size) == (2, 2):
            return _ConvChain(layers[i], chain)
        return None

    def forward(self, layers, i, inputs, training, keep_all=True):
        conv, chain = self.conv, self.chain
        if training or keep_all or layers[i] is not conv or "forward" in conv.__dict__ or not chain._intact(layers, i + 1, False) or not _as_wired(self.links[0]):
            return False
        bn = chain.bn
        x = to_device(inputs)
        if (x.ndim != 4 or x.shape[3] != conv.filter_weights.shape[2] or bn.gamma is None or chain.pool.filter_size != (2, 2) or tuple(chain.pool.strides) != (2, 2)
                or bn.gamma.numel() != conv.num_filters):
            return False
        alpha = chain.act._alpha
        p = conv._plan(x.shape)
        if p.y_shape is None or not p.pools or not 0.0 <= alpha < 1.0:
            return False
        S, H, W, Cc = p.y_shape
        pooled = host().empty((S, H // 2, W // 2, Cc))
        target = chain.consumer.x_copy_target(tuple(pooled.shape)) if chain.consumer is not None else None
        conv.forward_pooled(x, p, bn, alpha, pooled, target)
        if target:
            chain.consumer.x_copy_written(pooled)
        chain.live = None
        chain.pool.output = pooled
        return True


class _DenseAct:
    """A Layer_Dense and the (Leaky_)ReLU behind it, run in one call each way; every attribute of both layers is as the layers
    leave it.  Same conditions as _Chain, and only where the library has one launch for it."""
    length = 2

    @staticmethod
    def _together(rows, columns):
        """Whether the activation's backward pass goes with its operand copy and column sums (aether_act_bwd_copy: a CTA walks all
        rows of 32 columns, so its time grows with the rows while the passes by themselves spread over the GPU).  Activation
        and layer backward in us, together / apart: 128 columns 256 rows 11.4 / 12.6, 512 14.4 / 14.1, 1024 19.3 / 13.6; 512
        columns 512 rows 16.2 / 18.3, 768 19.2 / 19.5, 1024 22.1 / 20.8; 1024 columns 1024 rows 24.4 / 26.5, 1536 31.8 / 30.5."""
        return 0 < rows <= 384 + min(columns, 1024)

    def __init__(self, dense, act, behind):
        self.parts = [dense, act]
        self.links = _links(self.parts)
        self.dense, self.act = dense, act
        self.consumer = behind if type(behind) is Layer_Dense else None

    @staticmethod
    def find(layers, i):
        if i + 1 < len(layers) and type(layers[i]) is Layer_Dense and type(layers[i + 1]) in (ReLU, Leaky_ReLU):
            return _DenseAct(layers[i], layers[i + 1], layers[i + 2] if i + 2 < len(layers) else None)
        return None

    def _intact(self, layers, i, back):
        if layers[i:i + 2] != self.parts or self.act.fused_into_prev or not _as_wired(self.links[back]):
            return False
        for part in self.parts:
            d = part.__dict__
            if "forward" in d or "backward" in d:
                return False
        return True

    def forward(self, layers, i, inputs, training, keep_all=True):
        if not self._intact(layers, i, False):
            return False
        x = to_device(inputs)
        dense, act = self.dense, self.act
        if x.ndim != 2 or x.shape[1] != dense.weights.shape[0]:
            return False
        p = dense._plan(x.shape[0])
        if p.layout is None:
            return False
        target = self.consumer.x_copy_target((p.x_shape[0], p.b_shape[0])) if self.consumer is not None else None
        act.inputs, act.output = dense.forward_act(x, act._alpha, target, p)
        if target:
            self.consumer.x_copy_written(act.output)
        return True

    def backward(self, layers, i, dvalues):
        dense, act = self.dense, self.act
        y = act.__dict__.get("inputs")
        if y is None or not self._intact(layers, i, True) or dense.__dict__.get("output") is not y or not self._together(*y.shape):
            return False
        dy = to_device(dvalues)
        p = dense._current()
        if p.layout is None or dy.shape != y.shape or y.shape[0] != dense.inputs.shape[0]:
            return False
        act.dinputs, _ = dense.backward_act(y, dy, act._alpha, p)
        return True


class _Head:
    """The Layer_Dense and the SoftMax a classifier ends in: logits and probabilities in one launch and, with the combined
    softmax / cross-entropy loss, the gradient of the logits and of the layer's inputs in one.  Conditions as for _Chain."""
    length = 2

    def __init__(self, dense, softmax):
        self.parts = [dense, softmax]
        self.links = _links(self.parts)
        self.dense, self.softmax = dense, softmax

    @staticmethod
    def find(layers, i):
        return _Head(layers[i], layers[i + 1]) if len(layers) == i + 2 and type(layers[i]) is Layer_Dense and type(layers[i + 1]) is SoftMax else None

    def _intact(self, layers, i, back):
        if layers[i:] != self.parts or not _as_wired(self.links[back]):
            return False
        for part in self.parts:
            d = part.__dict__
            if "forward" in d or "backward" in d:
                return False
        return True

    def forward(self, layers, i, inputs, training, keep_all=True):
        if not self._intact(layers, i, False):
            return False
        x = to_device(inputs)
        dense, softmax = self.dense, self.softmax
        if x.ndim != 2 or x.shape[1] != dense.weights.shape[0] or x.shape[0] == 0:
            return False
        p = dense._plan(x.shape[0])
        if not p.head:
            return False
        softmax.inputs, softmax.output = dense.forward_softmax(x, p)
        return True

    def backward(self, layers, combined, output, y):
        """Both layers' backward passes for the combined loss; False when they have to run one by one."""
        dense, softmax = self.dense, self.softmax
        z = softmax.__dict__.get("inputs")
        if (z is None or type(combined) is not Activation_Softmax_Loss_CategoricalCrossEntropy or "backward" in combined.__dict__
                or softmax.output is not output or dense.__dict__.get("output") is not z or not self._intact(layers, len(layers) - 2, True)
                or z.shape[0] != dense.inputs.shape[0]):
            return False
        p = dense._current()
        if not p.head:
            return False
        labels = _labels(y)
        if labels.shape[0] != z.shape[0] or (labels.ndim == 2 and labels.shape != z.shape):
            return False
        combined.dinputs = softmax.dinputs = dense.backward_softmax(output, labels, combined.label_smoothing, p)
        return True


class Model:
    def __init__(self):
        self.layers = []
        self.softmax_classifier_output = None
        self.loss = None
        self.optimizer = None
        self.accuracy = None
        self.flat_params = None
        self.grad_hook = None      # callable(flat_grads) run between backward and the optimizer (all-reduce)
        self._graph = self._graph_opt = None
        self._graph_memory = None  # arrays that the captured kernels address but that the graph itself does not own
        self._graph_metrics = False
        self._m_last = self._m_sum = None
        self.bucket_reducer = None # dp.BucketReducer: all-reduces the flat gradients bucket by bucket during backward
        self._bucket_of_layer = {}
        self._update_stream = None # side stream on which finished buckets are updated while backward goes on
        self._updated_early = set()
        self._chains = {}          # position of a Batch_Norm or Layer_Dense -> the _Chain or _DenseAct that starts there
        self._chain_ends = {}      # position of a chain's last layer -> where it starts
        self._built, self._wiring = [], []      # the layers as they were wired; of each the attributes and, among them, the layer in front
        self._pass_chains = {}     # _chains and, for inference passes that keep nothing, position of a Conv_Layer -> the _ConvChain that starts there

    def add(self, layer):
        self.layers.append(layer)

    def set(self, *, loss=None, optimizer=None, accuracy=None):
        if loss is not None:
            self.loss = loss
        if optimizer is not None:
            self.optimizer = optimizer
        if accuracy is not None:
            self.accuracy = accuracy

    # ------------------------------------------------------------------ wiring
    # ------------------------------------------------------------------ whole-model files
    def __getstate__(self):
        """What ``save`` writes: the layer list, loss, optimizer and accuracy objects (each without its per-step
        arrays) and the options of the last ``finalize``; flat buffers, graphs and wiring are rebuilt on loading."""
        return {"layers": self.layers, "loss": self.loss, "optimizer": self.optimizer, "accuracy": self.accuracy,
                "finalize_options": getattr(self, "_finalize_options", None)}

    def __setstate__(self, state):
        self.__init__()
        self.layers = state["layers"]
        self.loss, self.optimizer, self.accuracy = state["loss"], state["optimizer"], state["accuracy"]
        if state.get("finalize_options") is not None:
            had_state = [(l, {n: getattr(l, n) for n in ("weight_momentums", "weight_cache", "bias_momentums", "bias_cache")
                              if hasattr(l, n)}) for l in self.layers]
            self.finalize(**state["finalize_options"])
            for l, st in had_state:                      # Adam's moments go back into the (possibly flat) state arrays
                for n, arr in st.items():
                    if getattr(l, n) is not arr:
                        getattr(l, n).copy_(arr.reshape(getattr(l, n).shape))

    def save(self, path):
        """Writes the whole model to one file (``Model.save``, CNN_model_cupy.py:291-309).  As in the reference the
        per-step arrays (inputs, outputs, gradients) and the accumulated loss / accuracy are left out; parameters,
        Adam's state, running statistics and the layer configuration are kept.  Device arrays are stored as NumPy
        arrays; the file is a pickle of this package's classes (it is not interchangeable with the reference's own
        whole-model pickles, which name the reference's modules)."""
        if self.loss is not None:
            self.loss.new_pass()
        if self.accuracy is not None:
            self.accuracy.new_pass()
        with open(path, 'wb') as f:
            pickle.dump(self, f)

    @staticmethod
    def load(path):
        """Reads a file written by ``save`` (``Model.load``, CNN_model_cupy.py:311-317) and returns the model, wired
        with the same ``finalize`` options it had and ready to predict or to go on training."""
        with open(path, 'rb') as f:
            model = pickle.load(f)
        if not isinstance(model, Model):
            raise TypeError("%s does not hold a Model" % path)
        return model

    def finalize(self, flat=False, fuse=False, lean=False):
        """Wires the layers (CNN_model_cupy.py:27-64).  Beyond the reference: `flat` packs parameters and gradients
        into flat buffers, `fuse` merges each block tail into one pass each way, and `lean` (with `fuse`) stops
        writing fp32 tensors that only this library's own next kernel would read and that kernel reads as a bf16
        operand copy anyway: the pooled output of a fused block tail in front of a Conv_Layer / Dense, and the dx of a
        fused tail behind a tensor-core Conv_Layer.  Parameters, gradients and outputs of the model are the same
        numbers as without it; the `.output` of such a Pooling and the `.dinputs` of such a Batch_Norm are then
        placeholders (a layer asked to read one raises)."""
        self._finalize_options = {"flat": bool(flat), "fuse": bool(fuse), "lean": bool(lean)}
        self.input_layer = Layer_Input()
        chain = [self.input_layer] + self.layers + [self.loss]
        for pos, layer in enumerate(self.layers, start=1):
            _link(layer, "prev", chain[pos - 1])
            _link(layer, "next", chain[pos + 1])
        self.output_layer_activation = self.layers[-1]
        if isinstance(self.layers[0], Conv_Layer):
            self.layers[0].first_in_model = True        # backward never asks it for dinputs
        # A Batch_Norm directly behind a Conv_Layer takes its batch statistics from the convolution's epilogue
        # (when the kernel that serves the shape provides them) instead of reducing the activation again.
        for a, b in zip(self.layers[:-1], self.layers[1:]):
            if isinstance(a, Conv_Layer) and isinstance(b, Batch_Norm):
                a.emit_bn_stats = True
                b.stats_from = a
            # fuse=True: a ReLU / Leaky_ReLU directly behind a Batch_Norm is applied by the Batch_Norm's own kernels
            # (one read and one write of the activation less each way).  The Batch_Norm's `output` is then the
            # ACTIVATED tensor and the activation layer hands its input through unchanged.
            if fuse and isinstance(a, Batch_Norm) and isinstance(b, ReLU):
                a.fused_alpha = float(b._alpha)
                b.fused_into_prev = True
                # ... and a Layer_Dropout_Spatial behind that activation: its per-channel mask is folded into the
                # Batch_Norm's per-channel coefficients (act(v) * m = act(m * v) for m >= 0)
                c = getattr(b, "next", None)
                if isinstance(c, Layer_Dropout_Spatial):
                    a.fused_dropout = c
                    c.fused_into_prev = True
                    c = getattr(c, "next", None)
                # ... and a max Pooling with stride == filter behind those: the Batch_Norm then reads the convolution
                # output once and writes the pooled tensor; the activated tensor in between is never materialised
                # (decided per call: the windows must tile the input)
                if (isinstance(c, Pooling) and c.pooling_type == "max" and c.padding == "valid"
                        and tuple(c.strides) == tuple(c.filter_size)):
                    a.fused_pool = c
                    _link(c, "fused_bn", a)
                    # The pooled tensor is the x of the layer behind (through a Flatten, if any) and the dx of this
                    # block tail is the dvalues of the convolution in front: the tail's kernels write the bf16 copies
                    # those layers' tensor-core kernels read, so neither runs a cast pass over the fp32 tensor.
                    nxt = getattr(c, "next", None)
                    if isinstance(nxt, Flatten):
                        nxt = getattr(nxt, "next", None)
                    if hasattr(nxt, "x_copy_target"):
                        a.copy_consumer = nxt
                    a.lean = bool(lean)
                    if isinstance(getattr(a, "prev", None), Conv_Layer):
                        a.copy_dy_consumer = a.prev
        self._chains = {i: c for i in range(len(self.layers))
                        if (c := (None if fuse else _Chain.find(self.layers, i)) or _DenseAct.find(self.layers, i) or _Head.find(self.layers, i)) is not None}
        self._chain_ends = {i + c.length - 1: i for i, c in self._chains.items() if type(c) is not _Head}
        self._built, self._wiring = list(self.layers), [(vars(l), vars(l).get("_link_prev")) for l in self.layers]
        self._pass_chains = self._chains
        if all(type(l).__module__ == _OWN for l in self.layers):
            self._pass_chains = {**self._chains, **{i - 1: c for i, chain in self._chains.items() if i > 0 and type(chain) is _Chain
                                                    and (c := _ConvChain.find(self.layers, i - 1, chain)) is not None}}
        self.trainable_layers = [l for l in self.layers if hasattr(l, "weights")]
        if self.loss is not None:
            self.loss.remember_trainable_layers(self.trainable_layers)
        if isinstance(self.layers[-1], SoftMax) and isinstance(self.loss, Loss_CategoricalCrossEntropy):
            self.softmax_classifier_output = Activation_Softmax_Loss_CategoricalCrossEntropy(self.loss.label_smoothing)
        if flat:
            self._pack_flat()

    def _pack_flat(self):
        """Move all parameters into one flat buffer and pre-allocate one flat gradient buffer plus
        Adam state; the layers keep seeing arrays of their usual shapes (views)."""
        pending = [l for l in self.trainable_layers if l.weights is None]
        if pending:
            raise RuntimeError("finalize(flat=True) needs every trainable layer to own its parameters already "
                               "(give Batch_Norm n_features)")
        sizes = []
        for l in self.trainable_layers:
            sizes += [l.weights.numel(), l.biases.numel()]
        # keep every view 16-byte aligned
        offs, total = [], 0
        for n in sizes:
            offs.append(total)
            total += (n + 3) // 4 * 4
        dev = self.trainable_layers[0].weights.device
        self.flat_params = torch.zeros(total, dtype=torch.float32, device=dev)
        self.flat_grads = torch.zeros(total, dtype=torch.float32, device=dev)
        self.flat_m = torch.zeros(total, dtype=torch.float32, device=dev)
        self.flat_v = torch.zeros(total, dtype=torch.float32, device=dev)
        # element range of each trainable layer (its weights, biases and padding), in forward order: contiguous
        bounds = offs[0::2] + [total]
        self.flat_layer_ranges = [(bounds[i], bounds[i + 1]) for i in range(len(self.trainable_layers))]
        k = 0
        for l in self.trainable_layers:
            views = []
            for name in ("weights", "biases"):
                old = getattr(l, name)
                o, n = offs[k], sizes[k]
                k += 1
                pv = self.flat_params[o:o + n].view(old.shape)
                pv.copy_(old)
                setattr(l, name, pv)
                views.append(self.flat_grads[o:o + n].view(old.shape))
                mom = "weight" if name == "weights" else "bias"
                setattr(l, mom + "_momentums", self.flat_m[o:o + n].view(old.shape))
                setattr(l, mom + "_cache", self.flat_v[o:o + n].view(old.shape))
            l._grad_views = tuple(views)

    def set_bucket_reducer(self, reducer):
        """Installs a gradient reducer (see dp.BucketReducer): bucket i is started as soon as the backward pass has
        written the gradients of its last layer, and waited for right before that bucket's optimizer update."""
        self.bucket_reducer = reducer
        self._bucket_of_layer = {}
        if reducer is not None:
            for i, (_, _, trigger) in enumerate(reducer.buckets):
                self._bucket_of_layer[id(self.trainable_layers[trigger])] = i

    # ------------------------------------------------------------------ passes
    def forward(self, X, training, *, keep=True):
        """``keep=False`` (inference passes whose layers' attributes the next pass replaces): a chain of layers run in one
        pass writes its last output only."""
        self.input_layer.forward(X, training)
        layers, chains, i = self.layers, self._chains, 0
        if not training and not keep and chains:
            chains, keep = self._inference_chains()
        while i < len(layers):
            layer = layers[i]
            link = layer.__dict__.get("_link_prev")       # (layer.prev, the layer in front unless the caller has wired it otherwise)
            inputs = (link() if type(link) is weakref.ref else layer.prev).output
            chain = chains.get(i)
            if chain is not None and chain.forward(layers, i, inputs, training, keep):
                i += chain.length
                continue
            layer.forward(inputs, training)
            i += 1
        return layers[-1].output

    def _inference_chains(self):
        """The chains of an inference pass that need not keep what lies between its layers, and whether it has to after all: where a layer reads another
        one than the model was built with, every output stands.  A layer of the caller's may hold on to any convolution's."""
        if self.layers != self._built:
            return self._chains, True
        chains = self._pass_chains
        for attributes, front in self._wiring:
            if attributes.get("_link_prev") is not front:
                return self._chains, True
            if "forward" in attributes:
                chains = self._chains
        return chains, False

    def backward(self, output, y):
        layers = self.layers
        i = len(layers) - 1
        if self.softmax_classifier_output is not None:
            head = self._chains.get(i - 1)
            if type(head) is _Head and head.backward(layers, self.softmax_classifier_output, output, y):
                i -= 1
                self._gradients_written(layers[i])
            else:
                self.softmax_classifier_output.backward(output, y, training=True)
                layers[-1].dinputs = self.softmax_classifier_output.dinputs
            i -= 1
        else:
            self.loss.backward(output, y)
        first = layers[0]
        while i >= 0:
            layer = layers[i]
            dvalues = layer.next.dinputs
            start = self._chain_ends.get(i)
            if start is not None and self._chains[start].backward(layers, start, dvalues):
                layer = layers[start]           # the chain's only trainable layer is its first
                i = start
            elif layer is first and hasattr(layer, "_desc"):
                layer.backward(dvalues, need_dinputs=False)   # nobody consumes d(loss)/d(images)
            else:
                layer.backward(dvalues)
            i -= 1
            self._gradients_written(layer)

    def _gradients_written(self, layer):
        b = self._bucket_of_layer.get(id(layer)) if self._bucket_of_layer else None
        if b is not None:                       # this layer's gradients complete a bucket: start reducing it
            self.bucket_reducer.start(b)
            self._update_bucket_early(b)

    def _update_bucket_early(self, b):
        """Every bucket but the last is updated as soon as its all-reduce is through, on a side stream, while the
        main stream goes on back-propagating the layers in front: nobody reads those parameters again in this step
        (their layers' backward is over), and the update -- Adam moves 28 bytes per parameter, the dense head is most
        of them -- runs beside tensor-bound convolution kernels instead of after them."""
        r = self.bucket_reducer
        if b == len(r.buckets) - 1 or self.flat_params is None or not hasattr(self.optimizer, "update_flat"):
            return
        if self._update_stream is None:
            self._update_stream = torch.cuda.Stream()
        main = torch.cuda.current_stream()
        side = self._update_stream
        side.wait_stream(main)
        self.optimizer.pre_update_parameters()          # this step's learning rate (idempotent within a step)
        lo, hi, _ = r.buckets[b]
        with torch.cuda.stream(side):
            r.wait(b)
            self.optimizer.update_flat(self.flat_params[lo:hi], self.flat_grads[lo:hi], self.flat_m[lo:hi], self.flat_v[lo:hi])
        self._updated_early.add(b)

    def _apply_optimizer(self, run_hook=True):
        opt = self.optimizer
        if run_hook and self.grad_hook is not None and self.flat_params is not None:
            self.grad_hook(self.flat_grads)
        opt.pre_update_parameters()
        if self.bucket_reducer is not None and self.flat_params is not None and hasattr(opt, "update_flat"):
            # one update per bucket, each behind its own all-reduce only (the first bucket's update overlaps the
            # second bucket's all-reduce)
            if self._updated_early:
                torch.cuda.current_stream().wait_stream(self._update_stream)
            for i, (lo, hi, _) in enumerate(self.bucket_reducer.buckets):
                if i in self._updated_early:
                    continue
                if run_hook:
                    self.bucket_reducer.wait(i)
                opt.update_flat(self.flat_params[lo:hi], self.flat_grads[lo:hi], self.flat_m[lo:hi], self.flat_v[lo:hi])
            self._updated_early = set()
        elif self.flat_params is not None and hasattr(opt, "update_flat"):
            opt.update_flat(self.flat_params, self.flat_grads, self.flat_m, self.flat_v)
        elif isinstance(opt, Optimizer_Adam) and opt.updates_as_adam():
            opt.update_layers(self.trainable_layers)
        else:
            for layer in self.trainable_layers:
                opt.update_parameters(layer)
        opt.post_update_parameters()
        if getattr(self, "_g_step", None) is not None:
            self._g_step.add_(1)            # device copy of the step count (see enable_device_step)

    def train_step(self, X, y):
        """forward + loss gradient + backward + optimizer for one batch; returns the logits' softmax."""
        output = self.forward(X, training=True)
        self.backward(output, y)
        self._apply_optimizer()
        return output

    # ------------------------------------------------------------------ CUDA-graph train step
    def enable_device_step(self):
        """Moves the per-step host state (Adam's iteration count, the dropout call counters) into one int64 device
        counter that every train step increments; the channel masks of spatial dropout are then drawn on the device.
        Required for a captured train step, usable on its own (same numbers eagerly and replayed)."""
        if getattr(self, "_g_step", None) is None:
            dev = self.trainable_layers[0].weights.device
            self._g_step = torch.full((1,), int(self.optimizer.iterations), dtype=torch.int64, device=dev)
            for obj in [self.optimizer] + [l for l in self.layers if hasattr(l, "step_dev")]:
                obj.step_dev = self._g_step
        return self._g_step

    def _graph_body(self):
        out = self.train_step(self._g_X, self._g_y)
        if self._graph_metrics:
            self._step_metrics(out, self._g_y)
        return out

    def _step_metrics(self, output, labels):
        """This step's data loss, accuracy and regularisation loss, kept on the device: `_m_last` holds the three
        values of the latest step, `_m_sum` the running sums of the per-sample losses and of the hits that the
        reference accumulates on the host (CNN_model_cupy.py:104-111, CNN_classes_cupy.py:577-589)."""
        smooth = self.loss.label_smoothing
        _, rows_loss, _, hits = _softmax_cce(output, labels, False, True, False, True, smooth, 0.0, input_is_prob=True)
        self._m_last[0:1].copy_(rows_loss.mean().reshape(1))
        self._m_last[1:2].copy_(hits.float().mean().reshape(1))
        reg = self.loss.regularization_loss()
        if isinstance(reg, torch.Tensor):
            self._m_last[2:3].copy_(reg.reshape(1))
        else:
            self._m_last[2:3].fill_(float(reg))
        self._m_sum[0] += rows_loss.sum()
        self._m_sum[1] += hits.sum()

    def _graph_state(self):
        """Every tensor a train step changes besides activations: parameters, Adam moments, running statistics."""
        ts = [self.flat_params, self.flat_m, self.flat_v, self._g_step, self._m_last, self._m_sum]
        for l in self.layers:
            if isinstance(l, Batch_Norm) and l.gamma is not None:
                ts += [l._rm, l._rv]
        return ts

    def _workspaces(self):
        """(layer, workspace, its buffer, its size) of all layers' workspaces as they are."""
        found = []
        for l in self.layers:
            w = l.__dict__.get("_ws")
            if type(w) is _Workspace:
                found.append((l, w, w.buf, w.size))
                w = l.__dict__.get("_stats_ws")
                if w is not None:
                    found.append((l, w, w.buf, w.size))
        return found

    def _all_ranks_agree(self, ok):
        """True when `ok` holds on every rank (one small eager all-reduce; single process: `ok` itself)."""
        import torch.distributed as dist
        if not (dist.is_initialized() and dist.get_world_size() > 1):
            return ok
        flag = torch.tensor([1.0 if ok else 0.0], device=self.flat_params.device)
        dist.all_reduce(flag, op=dist.ReduceOp.MIN)
        return bool(flag.item() > 0.5)

    def capture_train_step(self, X, y, warmup=2, collectives_in_graph=True, metrics=False):
        """Records ``train_step`` for batches shaped like (X, y) into a CUDA graph; ``train_step_graph`` replays
        it with one launch.  A step of the small reference networks is some forty kernels of a few microseconds
        each, so the eager step is bound by what its calls cost the host, not by the GPU.  Needs ``finalize(flat=True)``.
        Whatever the reference changes on the host per step (Adam's iteration count and decayed learning rate,
        the dropout draws) is read from one int64 device counter that the graph itself increments.  The warm-up
        steps (they size the workspaces) are undone, so capturing does not train.

        Data parallelism: the bucketed all-reduces (dp.BucketReducer) are recorded inside the same graph, forked
        onto NCCL's stream where the backward pass starts them and joined before each bucket's update.  The
        capture runs in thread-local error mode: the process group's watchdog thread polls CUDA events of earlier
        collectives, which a global-mode capture treats as an illegal call and aborts with -- on that rank only.
        A rank whose capture failed must not leave its peers inside a recorded collective, so after the attempt
        every rank reports over one eager all-reduce and, unless all succeeded, all fall back to two graphs with
        the collectives launched eagerly between them.  ``collectives_in_graph=False`` asks for that form.
        ``metrics=True`` also records the step's loss / accuracy bookkeeping (``Model.train`` uses it)."""
        if self.flat_params is None:
            raise RuntimeError("capture_train_step needs finalize(flat=True)")
        self._g_X = to_device(X).clone()
        self._g_y = _labels_i32(y).clone()
        opt = self.optimizer
        dev = self.flat_params.device
        self.enable_device_step()
        self._graph_metrics = bool(metrics)
        if getattr(self, "_m_last", None) is None:
            self._m_last = torch.zeros(3, dtype=torch.float32, device=dev)
            self._m_sum = torch.zeros(2, dtype=torch.float64, device=dev)
        saved = [t.clone() for t in self._graph_state()]
        saved_it = opt.iterations
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(max(int(warmup), 1)):
                self._graph_body()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        for t, sv in zip(self._graph_state(), saved):
            t.copy_(sv)
        reducer = self.bucket_reducer if (self.bucket_reducer is not None and self.bucket_reducer.active) else None
        eager_between = self.grad_hook is not None or (reducer is not None and not collectives_in_graph)
        self._graph = self._graph_opt = None
        # A replay addresses these whatever the layers do meanwhile: a layer that is given a larger batch (evaluation, say)
        # replaces its workspace, whose memory would else go to other arrays that every replay then writes over.
        self._graph_memory = [buf for _, _, buf, _ in self._workspaces()] + self._graph_state() + [self.flat_grads]
        self.capture_note = "one graph"
        if reducer is not None and not eager_between:
            graph, ok, err = torch.cuda.CUDAGraph(), True, ""
            outer = torch.cuda.current_stream()
            try:
                with torch.cuda.graph(graph, capture_error_mode="thread_local"):
                    self._g_out = self._graph_body()
            except Exception as e:                  # noqa: BLE001 -- any failure means "do not replay this graph"
                ok, err = False, repr(e)
                reducer.works = [None] * len(reducer.buckets)
                torch.cuda.set_stream(outer)        # a failed capture may leave its side stream current
            if self._all_ranks_agree(ok):
                self._graph = graph
                self.capture_note = "one graph with %d all-reduce bucket(s) inside" % len(reducer.buckets)
            else:
                eager_between = True
                self.capture_note = "two graphs, collectives eager (in-graph capture failed on a rank%s)" % (": " + err if err else "")
        if self._graph is None:
            # With collectives outside: graph 1 = forward + backward (no bucket is started inside it), then the
            # reduction runs eagerly, then graph 2 = the optimizer.
            self._graph = torch.cuda.CUDAGraph()
            held, self._bucket_of_layer = self._bucket_of_layer, {}
            try:
                with torch.cuda.graph(self._graph, capture_error_mode="thread_local"), self._branched() as branch:
                    self._g_out = self.forward(self._g_X, training=True)
                    self.backward(self._g_out, self._g_y)
                    branch.join()
                    if not eager_between:
                        self._apply_optimizer()
                        if self._graph_metrics:
                            self._step_metrics(self._g_out, self._g_y)
            finally:
                self._bucket_of_layer = held
            if eager_between:
                self._graph_opt = torch.cuda.CUDAGraph()
                with torch.cuda.graph(self._graph_opt, capture_error_mode="thread_local"):
                    self._apply_optimizer(run_hook=False)
                    if self._graph_metrics:
                        self._step_metrics(self._g_out, self._g_y)
                if self.capture_note == "one graph":
                    self.capture_note = "two graphs, collectives eager"
        opt.iterations = saved_it           # capture records work, it does not run it
        return self._graph

    def _as_built(self):
        """Whether the passes run this package's code alone.  Methods of the caller's (a subclass, a patched instance) may use any array that the
        layers in front of them have been asked for, a gradient that they clip, say."""
        own = (type(self).forward is Model.forward and type(self).backward is Model.backward and "forward" not in vars(self) and "backward" not in vars(self))
        return own and all(type(l).__module__ == _OWN and "forward" not in vars(l) and "backward" not in vars(l) for l in self.layers)

    @contextlib.contextmanager
    def _branched(self):
        """Inside it the layers put on a second stream what the layers behind them do not wait for: the operand copies of the weights, made beside
        the first layers, and the parameters' gradients, made beside the layers in front.  Nothing of it where the caller's own methods run in between, on
        the main stream."""
        layers = [l for l in self.layers if isinstance(l, _TakesCopies)] if self._as_built() else []
        branch = _Branch()
        try:
            for l in layers:
                l._branch = branch
            for l in layers:
                l._weights_fixed = l._copy_weights()
            yield branch
        finally:
            for l in layers:
                l._branch, l._weights_fixed = None, False

    def release_graphs(self):
        """Drops the captured graphs (and the batch buffers they read).  A graph that recorded collectives keeps the
        NCCL communicator busy for as long as it exists: destroying the process group while such a graph is alive
        waits for ever, so data-parallel programs call this (or ``dp.shutdown``) before tearing the group down."""
        self._graph = self._graph_opt = None
        self._g_out = None
        self._graph_metrics = False
        if torch.cuda.is_available():
            torch.cuda.synchronize()
        self._graph_memory = None           # (a replay may have been running until here)

    def train_step_graph(self, X, y):
        """One training step by replaying the captured graph on a new batch of the captured shape."""
        if getattr(self, "_graph", None) is None:
            raise RuntimeError("train_step_graph called before capture_train_step")
        self._g_X.copy_(to_device(X), non_blocking=True)
        self._g_y.copy_(_labels(y), non_blocking=True)
        self._graph.replay()
        if self._graph_opt is not None:
            if self.grad_hook is not None:
                self.grad_hook(self.flat_grads)
            elif self.bucket_reducer is not None:
                self.bucket_reducer.reduce_all()
            self._graph_opt.replay()
        opt = self.optimizer
        opt.pre_update_parameters()         # host mirror of what the graph just did on the device
        opt.post_update_parameters()
        return self._g_out

    def _graph_train_possible(self, X, y, chunks):
        """The captured step serves ``train`` when every batch has the same shape and the step is the combined
        softmax + cross-entropy one on flat parameters."""
        if self.flat_params is None or self.softmax_classifier_output is None or not torch.cuda.is_available():
            return False
        if not isinstance(self.accuracy, Accuracy_Categorical) or len(chunks) == 0:
            return False
        sizes = {len(range(*sl.indices(len(X)))) for sl in chunks}
        return len(sizes) == 1

    def train(self, X, y, *, epochs=1, batch_size=None, print_every=1, validation_data=None, use_graph=None):
        """The reference's training loop (CNN_model_cupy.py:67-151), same printed lines.  When every batch has the
        same shape and the model was finalized with ``flat=True`` the step is captured once and replayed
        (``use_graph=None`` decides by itself, True / False force it): loss and accuracy are then computed and
        accumulated on the device inside the replayed step and read back only for the lines that are printed,
        so the loop never waits for the GPU in between."""
        self.accuracy.init(y)
        chunks = _batches(len(X), batch_size)
        graph = self._graph_train_possible(X, y, chunks) if use_graph is None else bool(use_graph)
        if graph and not self._graph_train_possible(X, y, chunks):
            raise RuntimeError("use_graph=True needs finalize(flat=True), softmax + categorical cross-entropy, "
                               "Accuracy_Categorical and batches of one size")
        print("Training")
        if graph:
            first = chunks[0]
            shape = tuple(to_device(X[first]).shape)
            if getattr(self, "_graph", None) is None or not self._graph_metrics or tuple(self._g_X.shape) != shape:
                self.capture_train_step(X[first], y[first], metrics=True)
            per_batch = shape[0]
        for epoch in range(1, epochs + 1):
            print(f' epoch: {epoch}')
            self.loss.new_pass()
            self.accuracy.new_pass()
            if graph:
                self._m_sum.zero_()
            for step, sl in enumerate(chunks):
                batch_X, batch_y = X[sl], y[sl]
                if graph:
                    self.train_step_graph(batch_X, batch_y)
                    data_loss, accuracy, regularization_loss = self._m_last[0], self._m_last[1], self._m_last[2]
                    loss = None
                else:
                    output = self.forward(batch_X, training=True)
                    data_loss, regularization_loss = self.loss.calculate(output, batch_y, include_regularization=True,
                                                                         training=True)
                    loss = data_loss + regularization_loss
                    predictions = self.output_layer_activation.predictions(output)
                    accuracy = self.accuracy.calculate(predictions, batch_y)
                    self.backward(output, batch_y)
                    self._apply_optimizer()
                if not step % print_every or step == len(chunks) - 1:
                    if graph:                   # one read-back of the three device scalars, only for printed steps
                        data_loss, accuracy, regularization_loss = (float(v) for v in self._m_last.tolist())
                        loss = data_loss + regularization_loss
                    print(f'epoch: {epoch}, acc: {float(accuracy):.3f}, loss: {float(loss):.3f} ('
                          f'data_loss: {float(data_loss):.3f}, reg_loss: {float(regularization_loss):.3f}, '
                          f'lr:: {self.optimizer.current_learning_rate}')
            if graph:                           # hand the device-side sums to the reference's accumulators
                self.loss.accumulated_sum = self._m_sum[0].float()
                self.loss.accumulated_count = per_batch * len(chunks)
                self.accuracy.accumulated_sum = self._m_sum[1].float()
                self.accuracy.accumulated_count = per_batch * len(chunks)
        epoch_data_loss, epoch_regularization_loss = self.loss.calculate_accumulated(include_regularization=True)
        epoch_loss = epoch_data_loss + epoch_regularization_loss
        epoch_accuracy = self.accuracy.calculate_accumulated()
        print(f' training, acc: {float(epoch_accuracy):.3f}, loss: {float(epoch_loss):.3f} ('
              f'data_loss: {float(epoch_data_loss):.3f}, reg_loss: {float(epoch_regularization_loss):.3f}, '
              f'lr:: {self.optimizer.current_learning_rate}')
        if validation_data is not None:
            self.evaluate(*validation_data, batch_size=batch_size)

    # Bytes of layer outputs and workspaces that an inference pass takes several batches together up to.  A batch of the
    # reference's networks leaves most of the GPU idle in its deeper layers and takes longer to launch than to run (32x32 network,
    # batch 128: 112 us of host work for 86 us on the GPU), so a pass takes as many whole batches as keep its arrays within
    # what a training batch of 512 of that network needs with its gradients: 1000 images in batches of 128, 900 -> 260 us (in
    # one pass and the last batch; in three of at most a gigabyte 436 us).  Workspaces that training has given the layers
    # are theirs again when the call ends, and where the memory is not there the batches are run one by one.
    INFERENCE_PASS_BYTES = 5 << 28
    _PER_SAMPLE = frozenset((Conv_Layer, Batch_Norm, ReLU, Leaky_ReLU, Layer_Dropout, Layer_Dropout_Spatial, Pooling, Flatten, Layer_Dense, SoftMax))

    def _output_bytes(self, shape):
        """Bytes of all layers' outputs for one sample of ``shape``, and the layers with a workspace that grows with the batch,
        each with the shape of its sample; None when a layer is not one of this package's own, which treat every sample by
        itself in inference, or does not take the shape."""
        total, working, n = 0, [], math.prod(shape)
        for l in self.layers:
            kind = type(l)
            if kind not in self._PER_SAMPLE or "forward" in l.__dict__:
                return None
            if kind is Conv_Layer:
                if len(shape) != 3:
                    return None
                working.append((l, shape))
                _, Ho, Wo = l._extent(shape[0], shape[1])
                if Ho < 1 or Wo < 1:
                    return None
                shape = (Ho, Wo, l.num_filters)
                n = Ho * Wo * l.num_filters
            elif kind is Pooling:
                if len(shape) != 3:
                    return None
                shape = tuple((m - f) // s + 1 for m, f, s in zip(shape, l.filter_size, l.strides)) + (shape[2],)
                n = math.prod(shape)
            elif kind is Flatten:
                shape = (n,)
            elif kind is Layer_Dense:
                working.append((l, ()))
                n = l.weights.shape[1]
                shape = (n,)
            total += 4 * n
        return (total, working) if total > 0 else None

    def _pass_samples(self, X, batch_size, most):
        """Samples of a pass: whole batches, `most` at most, whose arrays stay within INFERENCE_PASS_BYTES (one batch always)."""
        found = self._output_bytes(tuple(X.shape[1:]))
        if found is None:
            return batch_size
        per_sample, working = found
        limit = self.INFERENCE_PASS_BYTES
        n = min(most, max(1, limit // (per_sample * batch_size)) * batch_size)
        while n > batch_size:
            need = n * per_sample + sum(l._plan((n, *shape) if shape else n).fwd_ws_bytes for l, shape in working)
            if need <= limit:
                break
            n = max(1, min(n // batch_size - 1, n * limit // need // batch_size)) * batch_size
        return n

    def _workspaces_to_keep(self, samples, batch_size):
        """What an inference that may join batches goes back to (two batches are never joined)."""
        return self._workspaces() if batch_size is not None and samples > 2 * batch_size else ()

    def _restore_workspaces(self, held, all_of_them=False):
        """The layers' workspaces are again those of ``held``.  A layer that had none keeps its first one, which the next call
        of a program that only infers needs again; ``all_of_them``: it gives that up, too."""
        for l, w, buf, size in held:
            if w.buf is not buf and (buf is not None or all_of_them):
                w.buf, w.size = buf, size
                if isinstance(l, _TakesCopies):
                    l._forget_copies()

    def _own_forward(self):
        """False where a subclass or a patched method runs the passes: it gets the batches and the arguments it knows."""
        return type(self).forward is Model.forward and "forward" not in vars(self)

    def _inference(self, X, batch_size, held=()):
        """Slices and outputs of the forward passes over X: whole batches, several at once where they are small, then the
        last batch by itself, whose inputs and outputs the layers keep.  The weights stay as they are between the passes of
        one call, so from the second on the tensor-core layers use the operand copies of them that the first one made.
        ``held``: the workspaces to go back to where several batches at once find no memory."""
        batches = passes = _batches(len(X), batch_size)
        own = self._own_forward()
        if own and len(batches) > 2 and hasattr(X, "shape"):
            head = (len(batches) - 1) * batch_size
            step = self._pass_samples(X, batch_size, head)
            passes = [slice(k, min(k + step, head)) for k in range(0, head, step)] + batches[-1:]
        fixed = [l for l in self.layers if hasattr(l, "_weights_fixed")]
        k, copied = 0, False
        while k < len(passes):
            sl, done = passes[k], False
            # (set for the pass only: a caller that leaves its loop by an exception does not resume this one, and may train next)
            try:
                if copied:
                    for l in fixed:
                        l._weights_fixed = True
                output = self.forward(X[sl], training=False, **({"keep": k == len(passes) - 1} if own else {}))
                done = True
            except torch.OutOfMemoryError:
                if len(passes) == len(batches):
                    raise
            finally:
                for l in fixed:
                    l._weights_fixed = False
            if not done:                            # one by one then, without what this pass has left in memory
                output = None
                self._restore_workspaces(held, all_of_them=True)
                for l in [self.input_layer] + self.layers:
                    l.inputs = l.output = None
                k, passes, copied = sl.start // batch_size, batches, False
                continue
            yield sl, output
            k, copied = k + 1, True

    def evaluate(self, X_val, y_val, *, batch_size=None):
        self.loss.new_pass()
        self.accuracy.new_pass()
        held = self._workspaces_to_keep(len(X_val), batch_size)
        try:
            for sl, outputs in self._inference(X_val, batch_size, held):
                y_pass = y_val[sl]
                for part in _batches(len(outputs), batch_size):
                    self.loss.calculate(outputs[part], y_pass[part], training=False)
                    self.accuracy.calculate(self.output_layer_activation.predictions(outputs[part]), y_pass[part])
        finally:
            self._restore_workspaces(held)
        validation_loss = self.loss.calculate_accumulated()
        validation_accuracy = self.accuracy.calculate_accumulated()
        print(f'Valdiation, acc: {float(validation_accuracy):.3f}, loss: {float(validation_loss):.3f}')
        return float(validation_accuracy), float(validation_loss)

    def predict(self, X, *, batch_size=None):
        # (SoftMax writes a new array every time; an output layer or a forward pass of the caller's may not)
        new = type(self.layers[-1]) is SoftMax and "forward" not in vars(self.layers[-1]) and self._own_forward()
        held = self._workspaces_to_keep(len(X), batch_size)
        try:
            outs = [output if new else output.clone() for _, output in self._inference(X, batch_size, held)]
        finally:
            self._restore_workspaces(held)
        return torch.vstack(outs)

    # ------------------------------------------------------------------ parameters
    def get_parameters(self):
        return [layer.get_parameters() for layer in self.trainable_layers]

    def set_parameters(self, parameters):
        for parameter_set, layer in zip(parameters, self.trainable_layers):
            layer.set_parameters(*parameter_set)

    def save_parameters(self, path, include_optimizer=False):
        """Same on-disk format as the reference (a pickled list of per-layer tuples,
        CNN_model_cupy.py:277-282), with NumPy arrays so the file loads without a GPU.
        ``include_optimizer=True`` (not in the reference, whose checkpoints drop Adam's state) writes a dict
        {"parameters": that list, "optimizer": iteration count + per-layer moment arrays} instead, so training
        resumes with the same moments and decayed learning rate."""
        host = [tuple(np.asarray(a.detach().cpu()) for a in params) for params in self.get_parameters()]
        payload = host
        if include_optimizer:
            state = []
            for l in self.trainable_layers:
                if hasattr(l, "weight_cache"):
                    state.append(tuple(np.asarray(getattr(l, n).detach().cpu()) for n in
                                       ("weight_momentums", "weight_cache", "bias_momentums", "bias_cache")))
                else:
                    state.append(None)
            payload = {"parameters": host,
                       "optimizer": {"iterations": int(self.optimizer.iterations), "layers": state}}
        with open(path, 'wb') as f:
            pickle.dump(payload, f)

    def load_parameters(self, path):
        """Reads a checkpoint written by ``save_parameters`` here or by the reference (CNN_model_cupy.py:284-289).
        The reference's CuPy model pickles ``cupy`` arrays; they are rebuilt as NumPy arrays (the pickle stores
        them as host arrays wrapped in a ``cupy._core.core.array`` call), so such files load without CuPy.  Only
        array reconstruction is allowed while unpickling; anything else in the file is refused."""
        with open(path, 'rb') as f:
            payload = _CheckpointUnpickler(f).load()
        if isinstance(payload, dict):
            self.set_parameters(payload["parameters"])
            opt_state = payload.get("optimizer")
            if opt_state is not None and self.optimizer is not None:
                self.optimizer.iterations = int(opt_state["iterations"])
                self.optimizer.pre_update_parameters()
                step_dev = getattr(self, "_g_step", None)
                if step_dev is not None:
                    step_dev.fill_(self.optimizer.iterations)
                for l, st in zip(self.trainable_layers, opt_state["layers"]):
                    if st is None:
                        continue
                    for name, arr in zip(("weight_momentums", "weight_cache", "bias_momentums", "bias_cache"), st):
                        cur = getattr(l, name, None)
                        t = to_device(arr)
                        if cur is not None:
                            cur.copy_(t.reshape(cur.shape))     # in place: flat-buffer views stay views
                        else:
                            setattr(l, name, t.clone())
        else:
            self.set_parameters(payload)

    load_paramters = load_parameters      # spelling used by the reference's NumPy model and two of its scripts


class _CheckpointUnpickler(pickle.Unpickler):
    """Unpickler for parameter checkpoints: NumPy's array reconstruction helpers, and ``cupy`` array
    constructors mapped to ``numpy.asarray``; every other global is refused."""

    _NUMPY = {("numpy._core.multiarray", "_reconstruct"), ("numpy.core.multiarray", "_reconstruct"),
              ("numpy._core.multiarray", "scalar"), ("numpy.core.multiarray", "scalar"),
              ("numpy", "ndarray"), ("numpy", "dtype")}

    def find_class(self, module, name):
        if module.split(".")[0] == "cupy" and name in ("array", "asarray", "ndarray"):
            if name == "ndarray":
                raise pickle.UnpicklingError("cupy.ndarray subclass state is not a parameter checkpoint")
            return np.asarray
        if (module, name) in self._NUMPY:
            return super().find_class(module, name)
        raise pickle.UnpicklingError("checkpoint refers to %s.%s, which is not an array constructor" % (module, name))
