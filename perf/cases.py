"""What the performance of this framework is measured on: the work its users have it do, through its public entry points
(INetwork -> Optimize -> IRuntime.LoadNetwork -> LoadedNetwork).

A case names a family of networks, its sizes, and the way the program runs it:

  eager   LoadedNetwork.launch_all on the caller's stream: one C-ABI call per layer, nothing recorded
  graph   LoadedNetwork.CaptureGraph once, then Execute: a resident network whose inputs and outputs stay on the device;
          joined with the caller's stream, which has produced the inputs and goes on to use the outputs
  host    LoadedNetwork.EnqueueWorkload with the caller's own host arrays, as an Arm NN program calls it

Weights belong to the network and are the same for every seed; inputs are made from the seed.
"""
import functools
import math

import numpy as np
import torch

from armnn_b200 import configs, microbench, network
from armnn_b200.network import (ActivationFunction, BinaryOperation, DataType, INetwork, TensorInfo)

_TORCH = {DataType.QAsymmU8: torch.uint8, DataType.QAsymmS8: torch.int8, DataType.QSymmS8: torch.int8,
          DataType.QSymmS16: torch.int16, DataType.Float32: torch.float32, DataType.Signed32: torch.int32}


# ---------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------

def listed():
    return [
        # a single quantised convolution, one image: the smallest call, where launching it is most of its time
        dict(name="conv_56x56x64", family="single_conv", mode="eager"),
        # one row through one large FullyConnected layer: the weights are read for one use each
        dict(name="fc_1x4096x4096", family="fc", m=1, k=4096, n=4096, dtype="s8", mode="eager"),
        # a classifier head over a batch of feature vectors, uint8 with zero points: no extent is a multiple of the tiles
        dict(name="fc_200x1280x1001_u8", family="fc", m=200, k=1280, n=1001, dtype="u8", mode="eager"),
        # the large end of the FullyConnected sweep
        dict(name="fc_4096x4096x4096", family="fc", m=4096, k=4096, n=4096, dtype="s8", mode="eager"),
        # an int8 self-attention layer (projections, BatchMatMul, Softmax, re-layouts, residual Add)
        dict(name="attention_8x512", family="attention", batch=8, seq=512, embed=512, heads=8, mode="graph"),
        # one timestep of a three-layer QLstm encoder
        dict(name="qlstm_128", family="qlstm", batch=128, input=40, units=512, output=256, layers=3, mode="graph"),
        # uint8 image classification, a batch resident on the device
        dict(name="mobilenet_v2_64", family="mobilenet_v2", batch=64, image=224, mode="graph"),
        # the same network, one camera frame at a time in host memory
        dict(name="mobilenet_v2_1_host", family="mobilenet_v2", batch=1, image=224, mode="host"),
        # int8 image classification, a large batch: the most work of all cases
        dict(name="resnet50_256", family="resnet50", batch=256, image=224, mode="graph"),
        # a few images of another size: every layer small, odd extents in the last stages
        dict(name="resnet50_3_i200", family="resnet50", batch=3, image=200, mode="graph"),
        # a Float32 convolutional network (dense, depthwise and pointwise convolutions, Mean, FullyConnected, Softmax)
        dict(name="float_cnn_8", family="float_cnn", batch=8, image=56, c=32, c1=64, c2=128, classes=1001, mode="graph"),
        # the tail of a dense-prediction network: coarse class scores enlarged, added to fine ones, best class per pixel
        dict(name="dense_tail_8", family="dense_tail", batch=8, h=64, w=64, up=4, classes=21, mode="graph"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the listed families, over the sizes that each of them stands for."""
    family = rng.choice(["conv", "fc", "attention", "qlstm", "mobilenet_v2", "resnet50", "float_cnn", "dense_tail"])
    if family == "conv":
        k = rng.choice([1, 3, 3, 5])
        c, oc = (rng.choice([3, 16, 24, 32, 48, 64, 96, 100, 128, 160, 192, 256, 320, 512]) for _ in range(2))
        h, w = _log_int(rng, 7, 112), _log_int(rng, 7, 112)
        most = max(1, min(256, int(1e10 / (h * w * c * oc * k * k)), int(1e8 / (h * w * max(c, oc)))))
        return dict(family="conv", batch=_log_int(rng, 1, most), h=h, w=w, c=c, oc=oc, k=k, stride=rng.choice([1, 1, 2]),
                    relu=rng.random() < 0.7, mode="eager")
    if family == "fc":
        k, n = _log_int(rng, 64, 4096), _log_int(rng, 64, 4096)
        return dict(family="fc", m=_log_int(rng, 1, min(4096, int(1.5e10 / (k * n)))), k=k, n=n, dtype=rng.choice(["s8", "u8"]),
                    mode="eager")
    if family == "attention":
        heads, head = rng.choice([1, 4, 6, 8, 12]), rng.choice([32, 48, 64])
        seq = _log_int(rng, 17, 1024)
        return dict(family="attention", batch=_log_int(rng, 1, max(1, min(32, 8192 // seq))), seq=seq, embed=heads * head,
                    heads=heads, mode="graph")
    if family == "qlstm":
        return dict(family="qlstm", batch=_log_int(rng, 1, 256), input=_log_int(rng, 16, 256), units=_log_int(rng, 64, 640),
                    output=_log_int(rng, 32, 320), layers=rng.choice([1, 2, 3]), mode="graph")
    if family in ("mobilenet_v2", "resnet50"):
        batch = _log_int(rng, 1, 64 if family == "mobilenet_v2" else 256)
        return dict(family=family, batch=batch, image=rng.randrange(64, 225, 4),
                    mode="host" if batch <= 4 and rng.random() < 0.5 else "graph")
    if family == "float_cnn":
        return dict(family="float_cnn", batch=_log_int(rng, 1, 16), image=_log_int(rng, 14, 80), c=rng.choice([3, 16, 24, 32, 40]),
                    c1=rng.choice([32, 50, 64, 96]), c2=rng.choice([64, 100, 128, 192]), classes=_log_int(rng, 10, 1001), mode="graph")
    return dict(family="dense_tail", batch=_log_int(rng, 1, 16), h=_log_int(rng, 16, 96), w=_log_int(rng, 16, 96),
                up=rng.choice([2, 3, 4]), classes=rng.choice([2, 5, 19, 21, 33]), mode="graph")


# ---------------------------------------------------------------------------------------------------------------
# the networks
# ---------------------------------------------------------------------------------------------------------------

def _f32(v):
    return float(np.float32(v))


class _Net:
    """A few shorthands over INetwork."""

    def __init__(self, name):
        self.net = INetwork.Create()
        self.rng = configs._rng(name)

    def input(self, binding, info):
        layer = self.net.AddInputLayer(binding, "input%d" % binding)
        layer.GetOutputSlot(0).SetTensorInfo(info)
        return layer.GetOutputSlot(0)

    def join(self, layer, info, *sources):
        for i, s in enumerate(sources):
            s.Connect(layer.GetInputSlot(i))
        layer.GetOutputSlot(0).SetTensorInfo(info)
        return layer.GetOutputSlot(0)

    def const(self, data, info, name):
        return self.net.AddConstantLayer(data, info, name).GetOutputSlot(0)

    def output(self, slot, binding=0):
        slot.Connect(self.net.AddOutputLayer(binding, "output%d" % binding).GetInputSlot(0))

    def reshape(self, x, shape, name):
        return self.join(self.net.AddReshapeLayer(shape, name), TensorInfo(shape, x.info.dtype, x.info.scale, x.info.offset), x)

    def transpose(self, x, perm, name):
        shape = tuple(x.info.shape[p] for p in perm)
        return self.join(self.net.AddTransposeLayer(perm, name), TensorInfo(shape, x.info.dtype, x.info.scale, x.info.offset), x)


def _fc_u8(m, k, n):
    """uint8 activations and per-tensor uint8 weights with zero points (a MobileNet-style classifier head)."""
    b = _Net("fc_u8_%d_%d_%d" % (m, k, n))
    x = b.input(0, TensorInfo((m, k), DataType.QAsymmU8, 0.02, 3))
    sw = 0.004
    w = b.const(b.rng.integers(0, 256, size=(n, k)).astype(np.uint8), TensorInfo((n, k), DataType.QAsymmU8, sw, 128), "w")
    bias = b.const(b.rng.integers(-1000, 1001, size=n).astype(np.int32), TensorInfo((n,), DataType.Signed32, _f32(np.float32(0.02) * np.float32(sw))), "b")
    std = 0.02 * sw * 146.0 * 73.9 * math.sqrt(k)
    b.output(b.join(b.net.AddFullyConnectedLayer(True, True, "fc"), TensorInfo((m, n), DataType.QAsymmU8, _f32(4.0 * std / 127.0), 128), x, w, bias))
    return b.net, m * k * n


def _attention(batch, seq, embed, heads):
    """x + Wo . softmax(q k^T) v on [batch * seq, embed] int8 rows; per-channel weights, zero points on the activations."""
    b = _Net("attention_%d_%d" % (embed, heads))
    rows, head = batch * seq, embed // heads
    x = b.input(0, TensorInfo((rows, embed), DataType.QAsymmS8, 0.03, 5))

    def project(src, std_in, name, zp):
        ws = b.rng.uniform(0.001, 0.01, size=embed).astype(np.float32)
        w = b.const(b.rng.integers(-127, 128, size=(embed, embed)).astype(np.int8), TensorInfo((embed, embed), DataType.QSymmS8, scales=ws, quant_dim=0), name + "/w")
        bias = b.const(b.rng.integers(-1000, 1001, size=embed).astype(np.int32),
                       TensorInfo((embed,), DataType.Signed32, scales=np.float32(src.info.scale) * ws, quant_dim=0), name + "/b")
        std = std_in * 0.0061 * configs.W_STD_S8 * math.sqrt(embed)
        y = b.join(b.net.AddFullyConnectedLayer(True, True, name), TensorInfo((rows, embed), DataType.QAsymmS8, _f32(4.0 * std / 127.0), zp), src, w, bias)
        return y, std

    def split(t, name):
        return b.transpose(b.reshape(t, (batch, seq, heads, head), name + "/split"), (0, 2, 1, 3), name + "/heads")

    (q, sq), (k, sk), (v, sv) = project(x, 1.2, "q", 2), project(x, 1.2, "k", -3), project(x, 1.2, "v", 1)
    q, k, v = split(q, "q"), split(k, "k"), split(v, "v")
    ss = sq * sk * math.sqrt(head)
    scores = b.join(b.net.AddBatchMatMulLayer(False, True, name="scores"), TensorInfo((batch, heads, seq, seq), DataType.QAsymmS8, _f32(4.0 * ss / 127.0), 0), q, k)
    probs = b.join(b.net.AddSoftmaxLayer(2.0 / ss, -1, "softmax"), TensorInfo((batch, heads, seq, seq), DataType.QAsymmS8, 1.0 / 256.0, -128), scores)
    sc = sv * min(1.0, math.sqrt(50.0 / seq))
    ctx = b.join(b.net.AddBatchMatMulLayer(name="context"), TensorInfo((batch, heads, seq, head), DataType.QAsymmS8, _f32(4.0 * sc / 127.0), 0), probs, v)
    ctx = b.reshape(b.transpose(ctx, (0, 2, 1, 3), "merge"), (rows, embed), "merge/flat")
    o, so = project(ctx, sc, "o", 0)
    b.output(b.join(b.net.AddElementwiseBinaryLayer(BinaryOperation.Add, "residual"), TensorInfo((rows, embed), DataType.QAsymmS8, _f32(4.0 * so / 127.0), 0), x, o))
    return b.net, 4 * rows * embed * embed + 2 * batch * heads * seq * seq * head


def _float_cnn(batch, image, c, c1, c2, classes):
    """conv 3x3 + ReLU, depthwise 3x3 stride 2 + ReLU, conv 1x1 + ReLU, Mean, FullyConnected, Softmax in Float32."""
    b = _Net("float_cnn_%d_%d_%d_%d" % (c, c1, c2, classes))
    F = DataType.Float32

    def f(*shape):
        return TensorInfo(shape, F)

    def weights(shape, fan, name):
        w = b.const((b.rng.standard_normal(shape) * math.sqrt(2.0 / fan)).astype(np.float32), f(*shape), name + "/w")
        n = shape[-1] if shape[0] == 1 else shape[0]
        return w, b.const((b.rng.standard_normal(n) * 0.1).astype(np.float32), f(n), name + "/b")

    def relu(t, name):
        return b.join(b.net.AddActivationLayer(ActivationFunction.ReLu, name=name), f(*t.info.shape), t)

    x = b.input(0, f(batch, image, image, c))
    y = b.join(b.net.AddConvolution2dLayer((1, 1), (1, 1, 1, 1), (1, 1), True, "conv"), f(batch, image, image, c1), x, *weights((c1, 3, 3, c), 9 * c, "conv"))
    y = relu(y, "conv/relu")
    pb, pa = configs.same_pad(image, 3, 2)
    o = (image + 1) // 2
    y = b.join(b.net.AddDepthwiseConvolution2dLayer((2, 2), (pb, pa, pb, pa), (1, 1), True, "dw"), f(batch, o, o, c1), y, *weights((1, 3, 3, c1), 9, "dw"))
    y = relu(y, "dw/relu")
    y = b.join(b.net.AddConvolution2dLayer((1, 1), (0, 0, 0, 0), (1, 1), True, "point"), f(batch, o, o, c2), y, *weights((c2, 1, 1, c1), c1, "point"))
    y = relu(y, "point/relu")
    y = b.join(b.net.AddMeanLayer((1, 2), False, "mean"), f(batch, c2), y)
    y = b.join(b.net.AddFullyConnectedLayer(True, True, "fc"), f(batch, classes), y, *weights((classes, c2), c2, "fc"))
    b.output(b.join(b.net.AddSoftmaxLayer(1.0, -1, "softmax"), f(batch, classes), y))
    macs = batch * (image * image * c1 * 9 * c + o * o * (c1 * 9 + c1 * c2) + c2 * classes)
    return b.net, macs


def _dense_tail(batch, h, w, up, classes):
    """uint8 class scores: Resize (bilinear) of the coarse ones, Add of the fine ones, ArgMax over the classes."""
    b = _Net("dense_tail")
    big = (batch, h * up, w * up, classes)
    coarse = b.input(0, TensorInfo((batch, h, w, classes), DataType.QAsymmU8, 0.05, 120))
    fine = b.input(1, TensorInfo(big, DataType.QAsymmU8, 0.03, 131))
    y = b.join(b.net.AddResizeLayer(h * up, w * up, 0, half_pixel_centers=True, name="resize"), TensorInfo(big, DataType.QAsymmU8, 0.05, 120), coarse)
    y = b.join(b.net.AddElementwiseBinaryLayer(BinaryOperation.Add, "add"), TensorInfo(big, DataType.QAsymmU8, 0.06, 125), y, fine)
    b.output(y, 1)
    b.output(b.join(b.net.AddArgMinMaxLayer(1, -1, "argmax"), TensorInfo(big[:3], DataType.Signed32), y))
    return b.net, batch * h * w * up * up * classes * 4


def _build(case):
    """(INetwork, multiply-accumulates of one pass)"""
    c, family = case, case["family"]
    if family == "single_conv":
        net, info = configs.single_conv()
        return net, info["macs"]
    if family == "conv":
        return microbench.conv_graph(c["batch"], c["h"], c["w"], c["c"], c["oc"], c["k"], c["stride"], c["relu"])
    if family == "fc":
        if c["dtype"] == "u8":
            return _fc_u8(c["m"], c["k"], c["n"])
        net, info = configs.fc_sweep_case(c["m"], c["k"], c["n"])
        return net, info["macs"]
    if family == "attention":
        return _attention(c["batch"], c["seq"], c["embed"], c["heads"])
    if family == "qlstm":
        net, info = configs.qlstm_stack(c["batch"], c["input"], c["units"], c["output"], c["layers"])
        return net, info["macs"]
    if family == "resnet50":
        net, info = configs.resnet50(c["batch"], c["image"])
        return net, info["macs"]
    if family == "mobilenet_v2":
        # class scores, and the feature maps at strides 8 and 16 that a detection head would read
        net, info = configs.mobilenet_v2(c["batch"], c["image"])
        layers = {layer.name: layer for layer in net.layers}
        for i, name in enumerate(("block6/add", "block10/add", "block13/add")):
            layers[name].GetOutputSlot(0).Connect(net.AddOutputLayer(1 + i, name + "/features").GetInputSlot(0))
        return net, info["macs"]
    if family == "float_cnn":
        return _float_cnn(c["batch"], c["image"], c["c"], c["c1"], c["c2"], c["classes"])
    if family == "dense_tail":
        return _dense_tail(c["batch"], c["h"], c["w"], c["up"], c["classes"])
    raise ValueError("unknown family %r" % family)


@functools.lru_cache(maxsize=2)
def _optimized(key):
    """A program parses and optimises a model once, whatever it runs through it afterwards."""
    net, macs = _build(dict(key))
    return network.Optimize(net, ["B200Acc"]), macs


def _network_of(case):
    return _optimized(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "mode"))))


# ---------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------

class _State:
    pass


@functools.lru_cache(maxsize=1)
def _runtime():
    return network.IRuntime.Create(0)


def _values(info, gen, device):
    """Inputs as the networks meet them: image bytes uniform, features and states bell-shaped around their zero point."""
    if info.dtype == DataType.Float32:
        return torch.randn(info.shape, generator=gen, device=device)
    if info.dtype == DataType.QAsymmU8 or (info.dtype == DataType.QAsymmS8 and len(info.shape) == 4):
        lo, hi = (0, 256) if info.dtype == DataType.QAsymmU8 else (-128, 128)
        return torch.randint(lo, hi, info.shape, generator=gen, device=device, dtype=torch.int32).to(_TORCH[info.dtype])
    spread, lo, hi = (2000.0, -32768, 32767) if info.dtype == DataType.QSymmS16 else (40.0, -128, 127)
    t = torch.randn(info.shape, generator=gen, device=device) * spread + info.offset
    return t.round_().clamp_(lo, hi).to(_TORCH[info.dtype])


def prepare(case, seed):
    optimized, _ = _network_of(case)
    s = _State()
    s.mode = case["mode"]
    s.ln = network.LoadedNetwork(_runtime(), optimized)
    device = torch.device("cuda", 0)
    gen = torch.Generator(device=device)
    gen.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    values = {b: _values(slot.info, gen, device) for b, slot in sorted(s.ln.inputs.items())}
    s.outputs = {"out%d" % b: s.ln.output_tensor(b) for b in sorted(s.ln.outputs)}
    if s.mode != "eager":
        s.ln.CaptureGraph()
    if s.mode == "host":
        s.host_in = {b: v.cpu().numpy() for b, v in values.items()}
        s.host_out = {b: np.zeros(slot.info.shape, network._NP_DTYPE[slot.info.dtype]) for b, slot in s.ln.outputs.items()}
    else:
        for b, v in values.items():
            s.ln.input_tensor(b).copy_(v)
    return s


def run(state):
    ln = state.ln
    if state.mode == "eager":
        ln.launch_all(torch.cuda.current_stream().cuda_stream)
        return state.outputs
    if state.mode == "graph":
        stream = torch.cuda.current_stream()
        ln.stream.wait_stream(stream)
        ln.Execute()
        stream.wait_stream(ln.stream)
        return state.outputs
    ln.EnqueueWorkload(state.host_in, state.host_out)
    return {"out%d" % b: v for b, v in sorted(state.host_out.items())}


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far two correct implementations may be apart
# ---------------------------------------------------------------------------------------------------------------

def work(case):
    """Network inputs, weights and network outputs once each; two operations per multiply-accumulate."""
    optimized, macs = _network_of(case)
    nbytes = 0
    for layer in optimized.layers:
        if layer.type in ("Input", "Constant"):
            nbytes += layer.outputs[0].info.GetNumBytes()
        elif layer.type == "Output":
            nbytes += layer.inputs[0].source.info.GetNumBytes()
        elif layer.type == "QLstm":
            nbytes += sum(info.GetNumBytes() for _, info in layer.qlstm_params.values())
    return {"bytes": nbytes, "flops": 2 * macs}


def tolerance(case):
    """Integer contractions, pooling, Add, Resize and ArgMax are exact.  Softmax and the QLstm gates go through exp and
    tanh, whose last bit may move a value across a rounding boundary.  Float32 sums hold about 1e-5."""
    if case["family"] == "float_cnn":
        return {"rel": 1e-5}
    if case["family"] in ("attention", "mobilenet_v2", "resnet50", "qlstm"):
        return {"rel": 0.0, "differ": 0.005}
    return "exact"
