"""MLP surrogate for the parameter search.

An addition of this project (DENSE's SRES search simulates every candidate,
search/sres.cpp:328-345): a small network maps a candidate's
log-parameters to oscillation features -- log period, log amplitude,
inter-cell synchrony of mh1 and an oscillation indicator -- and
pre-screens candidates, so that only the most promising ones are simulated.
Every candidate it accepts is re-simulated by the FP64 engine, which alone
decides acceptance.

Network: in -> 3 x 256 (GELU) -> out, BF16 weights and activations on the
products, FP32 accumulation, FP32 master weights with Adam.  Training,
prediction and ranking run in the whole-network tcgen05 kernels of
csrc/surrogate/chain.cu (``Kernels.gemm`` is the single product of
umma_gemm_persistent.cuh); torch only allocates the buffers and orders the
launches on one stream.
"""

import concurrent.futures as cf
import ctypes as C
import os
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_DIR = os.path.join(HERE, "_lib")
SRC = os.path.join(HERE, "csrc", "surrogate")
LIB = os.path.join(LIB_DIR, "libdense_b200_surrogate.so")

EPI_STORE, EPI_BIAS_GELU, EPI_BIAS = 0, 1, 2
HIDDEN = 256
IN_PAD = 64     # input features padded to the GEMM's K granularity
OUT_PAD = 128   # outputs padded to one UMMA M tile for the weight gradient
MAX_NETS = 64   # networks that one ranking launch takes


def build(force=False):
    include = os.path.join(os.path.dirname(HERE), "include")
    srcs = [os.path.join(SRC, f) for f in os.listdir(SRC)] + [os.path.join(include, f) for f in
                                                              ("dense_b200_surrogate.h", "dense_b200_network.h")]
    if not force and os.path.exists(LIB) and all(os.path.getmtime(s) <= os.path.getmtime(LIB) for s in srcs):
        return LIB
    os.makedirs(os.path.join(LIB_DIR, "obj"), exist_ok=True)
    nvcc = os.environ.get("NVCC", "nvcc")
    base = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-lineinfo",
            "-I", include]
    units = ("mlp", "features", "chain")
    objs = [os.path.join(LIB_DIR, "obj", unit + ".o") for unit in units]

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            raise RuntimeError(r.stderr[-4000:])

    with cf.ThreadPoolExecutor(len(units)) as ex:
        list(ex.map(run, [base + ["-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "-c",
                                  os.path.join(SRC, unit + ".cu"), "-o", obj] for unit, obj in zip(units, objs)]))
    run(base + ["-shared", "-o", LIB] + objs + ["-lcudart"])
    return LIB


_lib = None


def lib():
    global _lib
    if _lib is None:
        L = C.CDLL(build())
        vp, i, f, i64 = C.c_void_p, C.c_int, C.c_float, C.c_int64
        L.dense_mlp_gemm.argtypes = [vp, i, vp, i, vp, i, i, i, i, i, vp, vp, i, vp, vp]
        L.dense_mlp_gemm_ws.argtypes = [vp, i, vp, i, vp, i, i, i, i, i, vp, vp, i, vp, vp, C.c_size_t, vp]
        L.dense_mlp_transpose_bf16.argtypes = [vp, i, i, i, vp, i, vp]
        L.dense_mlp_cast_bf16.argtypes = [vp, i, i, vp, i, vp]
        L.dense_mlp_gelu_backward.argtypes = [vp, vp, i64, vp, vp, vp]
        L.dense_mlp_mse.argtypes = [vp, i, vp, vp, i, i, f, vp, vp, vp, vp]
        L.dense_mlp_colsum.argtypes = [vp, i, i, vp, vp]
        L.dense_mlp_adam.argtypes = [vp, vp, vp, vp, i64, f, f, f, f, i, vp]
        L.dense_mlp_adam_dev.argtypes = [vp, vp, vp, vp, i64, vp, vp]
        L.dense_mlp_mse_dev.argtypes = [vp, i, vp, vp, i, i, vp, vp, vp, vp, vp]
        L.dense_mlp_gather.argtypes = [vp, i, i, vp, vp, i, vp, i, i, vp, i, vp, vp, vp]
        L.dense_features_synchrony.argtypes = [vp, i64, i64, i, vp, i, vp, vp]
        L.dense_features_encode.argtypes = [vp, i, i, vp, vp, i, C.c_double, vp, i, i, vp]
        L.dense_features_ensemble_accumulate.argtypes = [vp, i, i, i, vp, i, vp]
        L.dense_features_score.argtypes = [vp, i, i, i, vp, vp, C.c_double, C.c_double, C.c_double, C.c_double,
                                           C.c_double, vp, vp]
        L.dense_mlp_packed_bytes.restype = i64
        L.dense_mlp_train_bytes.argtypes, L.dense_mlp_train_bytes.restype = [i, i], i64
        L.dense_mlp_pack.argtypes = [vp, vp, i, vp]
        L.dense_mlp_predict.argtypes = [vp, i, i, i, vp, vp, i, vp, vp, vp]
        d = C.c_double
        L.dense_mlp_rank.argtypes = [vp, i, i, vp, vp, i, d, i, vp, vp, i, vp, vp, d, d, d, d, d, vp, vp, vp]
        L.dense_mlp_train_pass.argtypes = [vp, i, i, i, vp, vp, i, vp, i, vp, vp, vp, f, vp, vp, i64, vp, vp]
        L.dense_mlp_train_finish.argtypes = [vp, i64, i, i] + [vp] * 11
        L.dense_mlp_train_epoch.argtypes = [vp, i, i, i, vp, vp, i, vp, i, i, vp, vp, vp, i64] + [vp] * 9
        _lib = L
    return _lib


def _p(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def _pp(ts):
    """A host array of the tensors' device pointers (None: no array)."""
    return None if ts is None else (C.c_void_p * len(ts))(*[t.data_ptr() for t in ts])


class Kernels:
    """Thin launchers over the C ABI for torch CUDA tensors on one stream.

    The GEMM's split-K workspace (FP32 partials) belongs to this object:
    its launches must stay on one stream."""

    WS_BYTES = 32 << 20

    def __init__(self, device=0):
        import torch
        self.torch = torch
        self.L = lib()
        self.dev = torch.device("cuda", device)
        self.stream = torch.cuda.current_stream(self.dev)
        self.err = torch.zeros(1, dtype=torch.int32, device=self.dev)
        self.ws = torch.empty(self.WS_BYTES // 4, dtype=torch.float32, device=self.dev)

    def _s(self):
        return C.c_void_p(self.torch.cuda.current_stream(self.dev).cuda_stream)

    def gemm(self, A, B, D, epilogue=EPI_STORE, bias=None, H=None):
        """D[M][N] = A[M][K] . B[N][K]^T (BF16 in, FP32 out)."""
        M, K = A.shape
        N = B.shape[0]
        rc = self.L.dense_mlp_gemm_ws(_p(A), A.stride(0), _p(B), B.stride(0), _p(D), D.stride(0), M, N, K, epilogue,
                                      _p(bias), _p(H), H.stride(0) if H is not None else 0, _p(self.err),
                                      _p(self.ws), self.WS_BYTES, self._s())
        if rc:
            raise RuntimeError("dense_mlp_gemm rejected M=%d N=%d K=%d (rc %d)" % (M, N, K, rc))

    def transpose(self, src, dst):
        r, c = src.shape
        assert self.L.dense_mlp_transpose_bf16(_p(src), r, c, src.stride(0), _p(dst), dst.stride(0), self._s()) == 0

    def cast(self, src, dst, transpose=False):
        r, c = src.shape
        assert self.L.dense_mlp_cast_bf16(_p(src), r, c, _p(dst), int(transpose), self._s()) == 0

    def gelu_backward(self, dH, Z, dZ, dZb):
        assert self.L.dense_mlp_gelu_backward(_p(dH), _p(Z), dH.numel(), _p(dZ), _p(dZb), self._s()) == 0

    def mse(self, Y, T, mask, dY, dYb, loss):
        rows, nout = T.shape
        inv = 1.0 / max(1.0, float(mask.sum().item()))
        assert self.L.dense_mlp_mse(_p(Y), Y.stride(0), _p(T), _p(mask), rows, nout, inv, _p(dY), _p(dYb),
                                    _p(loss), self._s()) == 0

    def mse_dev(self, Y, T, mask, inv_count, dY, dYb, loss):
        """mse with the 1 / count scale in a one-element device tensor."""
        rows, nout = T.shape
        assert self.L.dense_mlp_mse_dev(_p(Y), Y.stride(0), _p(T), _p(mask), rows, nout, _p(inv_count), _p(dY),
                                        _p(dYb), _p(loss), self._s()) == 0

    def gather(self, X, T, mask, idx, Xb, Tb, Mb):
        """One batch from a device-resident training set: rows idx of X
        (float [n][n_in]) to BF16 Xb [Bp][in_pad] (zero padded), of T and
        mask to Tb and Mb [Bp][n_out]; rows past len(idx) are zeros."""
        n, n_in = X.shape
        Bp, in_pad = Xb.shape
        assert self.L.dense_mlp_gather(_p(X), n, n_in, _p(T), _p(mask), T.shape[1], _p(idx), idx.shape[0], Bp,
                                       _p(Xb), in_pad, _p(Tb), _p(Mb), self._s()) == 0

    def adam_dev(self, w, g, m, v, hyper):
        """adam with {lr, b1, b2, eps, 1 - b1^t, 1 - b2^t} in device memory."""
        assert self.L.dense_mlp_adam_dev(_p(w), _p(g), _p(m), _p(v), w.numel(), _p(hyper), self._s()) == 0

    def synchrony(self, X, counts, out):
        """Mean pairwise Pearson correlation across cells per set: X a
        float64 CUDA tensor [sets][samples][cells] (cells contiguous; any
        set and sample strides), counts int32 [sets] (samples per set),
        out float64 [sets]."""
        B, _, cells = X.shape
        assert X.stride(2) == 1
        assert self.L.dense_features_synchrony(_p(X), X.stride(0), X.stride(1), cells, _p(counts), B, _p(out),
                                               self._s()) == 0

    def encode(self, P, idx, tmpl, log_spread, Xb):
        """Network inputs of candidates P (float64 [n][params]) into BF16
        Xb [Bp][in_pad]: log(P[:, idx] / tmpl) / log_spread, zero padded."""
        n, ldp = P.shape
        Bp, in_pad = Xb.shape
        assert P.stride(1) == 1
        assert self.L.dense_features_encode(_p(P), P.stride(0), n, _p(idx), _p(tmpl), idx.shape[0], float(log_spread),
                                            _p(Xb), in_pad, Bp, self._s()) == 0

    def ensemble_accumulate(self, Y, n, nout, acc, first):
        assert self.L.dense_features_ensemble_accumulate(_p(Y), Y.stride(0), n, nout, _p(acc), int(first),
                                                         self._s()) == 0

    def score(self, acc, nets, mu, sd, weight, period, tol, amp_min, ramp, out):
        """Ranking score from the ensemble sum acc [n][nout] (see
        csrc/surrogate/features.cu); mu and sd numpy float32 [nout]."""
        n, nout = acc.shape
        mu = np.ascontiguousarray(mu, np.float32)
        sd = np.ascontiguousarray(sd, np.float32)
        assert self.L.dense_features_score(_p(acc), n, nout, nets, mu.ctypes.data_as(C.c_void_p),
                                           sd.ctypes.data_as(C.c_void_p), weight, period, tol, amp_min, ramp, _p(out),
                                           self._s()) == 0

    def colsum(self, dZ, db):
        r, c = dZ.shape
        assert self.L.dense_mlp_colsum(_p(dZ), r, c, _p(db), self._s()) == 0

    def adam(self, w, g, m, v, lr, step, b1=0.9, b2=0.999, eps=1e-8):
        assert self.L.dense_mlp_adam(_p(w), _p(g), _p(m), _p(v), w.numel(), lr, b1, b2, eps, step, self._s()) == 0

    def pack(self, W, packed, backward):
        """The BF16 weights of one network in the order the whole-network
        passes read them."""
        assert self.L.dense_mlp_pack(_pp(W), _p(packed), int(backward), self._s()) == 0

    def predict(self, X, packed, bias, out):
        """out [rows][n_out] of the packed network for float32 rows X."""
        n, n_in = X.shape
        assert X.stride(1) == 1 or n_in == 1
        ld = X.stride(0) if n > 1 else n_in  # (the stride of a single row is no leading dimension)
        assert self.L.dense_mlp_predict(_p(X), ld, n, n_in, _p(packed), _pp(bias), out.shape[1], _p(out),
                                        _p(self.err), self._s()) == 0

    def rank(self, P, idx, tmpl, log_spread, packed, biases, n_out, mu, sd, weight, period, tol, amp_min, ramp, out):
        """Ranking scores of candidates P (float64 [n][params]) under the
        ensemble of packed networks: encode, every network and score in one
        launch."""
        assert P.stride(1) == 1
        mu = np.ascontiguousarray(mu, np.float32)
        sd = np.ascontiguousarray(sd, np.float32)
        assert self.L.dense_mlp_rank(_p(P), P.stride(0), P.shape[0], _p(idx), _p(tmpl), idx.shape[0],
                                     float(log_spread), len(packed), _pp(packed), _pp([b for bs in biases for b in bs]),
                                     n_out, mu.ctypes.data_as(C.c_void_p), sd.ctypes.data_as(C.c_void_p), weight,
                                     period, tol, amp_min, ramp, _p(out), _p(self.err), self._s()) == 0

    def train_pass(self, X, T, mask, idx, rows, packed, bias, inv_count, loss, work):
        """One batch forward and back; inv_count a float, or a one-element
        device tensor.  The gradients' parts stay in `work`."""
        n, n_in = X.shape
        dev_inv = inv_count if not isinstance(inv_count, float) else None
        assert self.L.dense_mlp_train_pass(_p(X), n_in, n, n_in, _p(T), _p(mask), T.shape[1], _p(idx), rows,
                                           _p(packed), _pp(bias), _p(dev_inv),
                                           inv_count if dev_inv is None else 0.0, _p(loss), _p(work), work.numel(),
                                           _p(self.err), self._s()) == 0

    def train_finish(self, work, rows, n_out, dW=None, db=None, hyper=None, net=None):
        """Gradients out of `work` into dW and db, and (with `hyper`) one
        Adam step of `net`'s weights, packed for the next pass."""
        state = (net.W, net.b, net.mW, net.vW, net.mb, net.vb) if hyper is not None else (None,) * 6
        assert self.L.dense_mlp_train_finish(_p(work), work.numel(), rows, n_out, _pp(dW), _pp(db), _p(hyper),
                                             *[_pp(t) for t in state], _p(net._packed if net else None),
                                             self._s()) == 0

    def train_epoch(self, X, T, mask, idx, hyper, loss, work, net):
        """hyper.shape[0] steps of `net` on the rows that idx gives each, from
        weights packed for a training pass."""
        steps = hyper.shape[0]
        assert hyper.shape[1] == 8 and idx.numel() % steps == 0
        assert self.L.dense_mlp_train_epoch(_p(X), X.shape[1], X.shape[0], X.shape[1], _p(T), _p(mask), T.shape[1],
                                            _p(idx), idx.numel() // steps, steps, _p(hyper), _p(loss), _p(work),
                                            work.numel(), *[_pp(t) for t in (net.W, net.b, net.mW, net.vW, net.mb,
                                                                             net.vb)],
                                            _p(net._packed), _p(self.err), self._s()) == 0

    def check(self):
        self.torch.cuda.synchronize(self.dev)
        e = int(self.err.item())
        if e:
            raise RuntimeError("tensor-core GEMM reported error bits %d" % e)


class MLP:
    """in -> 3 x 256 GELU -> out on the tensor-core kernels.

    Weights are kept as FP32 masters [out][in] with Adam moments; the passes
    read BF16 copies packed in their own order.  Inputs are padded to IN_PAD
    features and outputs to OUT_PAD rows (the padding weights stay zero:
    their gradients are zero).
    """

    def __init__(self, n_in, n_out, seed=0, device=0, lr=1e-3, group=None):
        """`group`: a torch.distributed process group for data-parallel
        training (every rank the same seed, so the same initial weights; the
        gradients of each step are averaged over the ranks)."""
        import torch
        assert n_in <= IN_PAD and n_out <= OUT_PAD
        self.torch = torch
        self.k = Kernels(device)
        self.dev = self.k.dev
        self.n_in, self.n_out, self.lr = n_in, n_out, lr
        rng = np.random.Generator(np.random.PCG64(seed))
        shapes = [(HIDDEN, IN_PAD), (HIDDEN, HIDDEN), (HIDDEN, HIDDEN), (OUT_PAD, HIDDEN)]
        fan_in = [n_in, HIDDEN, HIDDEN, HIDDEN]
        self.W, self.b = [], []
        for i, (o, n) in enumerate(shapes):
            w = np.zeros((o, n), np.float32)
            rows = o if i < 3 else n_out
            cols = n if i > 0 else n_in
            w[:rows, :cols] = rng.normal(0.0, np.sqrt(2.0 / fan_in[i]), size=(rows, cols))
            self.W.append(torch.tensor(w, device=self.dev))
            self.b.append(torch.zeros(o, device=self.dev))
        self.mW = [torch.zeros_like(w) for w in self.W]
        self.vW = [torch.zeros_like(w) for w in self.W]
        self.mb = [torch.zeros_like(b) for b in self.b]
        self.vb = [torch.zeros_like(b) for b in self.b]
        self.steps = 0
        self._bufs = {}
        self.group = group

    def _buf(self, name, shape, dtype=None):
        t = self._bufs.get(name)
        dtype = dtype or self.torch.float32
        if t is None or tuple(t.shape) != tuple(shape) or t.dtype != dtype:
            t = self.torch.empty(shape, dtype=dtype, device=self.dev)
            self._bufs[name] = t
        return t

    @property
    def _packed(self):
        return self._buf("packed", (int(self.k.L.dense_mlp_packed_bytes()),), self.torch.uint8)

    def _pack(self, backward=False):
        self.k.pack(self.W, self._packed, backward)
        return self._packed

    def forward(self, Xb):
        """Outputs [Bp][OUT_PAD] (float32) of padded BF16 rows Xb [Bp][IN_PAD],
        Bp a multiple of 128, a GEMM a layer: for callers that want the
        layers' own outputs, self.Z (before GELU) and self.H (after; H[0] is
        Xb) besides.  The buffers are this object's and are written again by
        the next call of the same size."""
        bf = self.torch.bfloat16
        Bp = Xb.shape[0]
        self.Z = [self._buf("Z%d" % i, (Bp, HIDDEN)) for i in range(3)]
        self.H = [Xb] + [self._buf("H%d" % i, (Bp, HIDDEN), bf) for i in range(1, 4)]
        Y = self._buf("Y", (Bp, OUT_PAD))
        for i, w in enumerate(self.W):
            Wb = self._buf("Wb%d" % i, w.shape, bf)
            self.k.cast(w, Wb)
            if i < 3:
                self.k.gemm(self.H[i], Wb, self.Z[i], EPI_BIAS_GELU, self.b[i], self.H[i + 1])
            else:
                self.k.gemm(self.H[3], Wb, Y, EPI_BIAS, self.b[3])
        return Y

    def _as_rows(self, X):
        """Whether X is float32 rows [B][n_in] that the kernels read as they
        are (the leading dimension is a C int)."""
        return (X.dtype == self.torch.float32 and X.device == self.dev and X.shape[1] == self.n_in and
                (X.stride(1) == 1 or self.n_in == 1) and
                (X.shape[0] <= 1 or self.n_in <= X.stride(0) < 2 ** 31))

    def _rows(self, X):
        """Float32 CUDA rows [B][n_in] of X, each value rounded as it would
        be to BF16 (once)."""
        torch = self.torch
        X = X.detach()
        if X.dtype != torch.float32:
            X = X.to(torch.bfloat16).to(torch.float32)
        X = X.to(self.dev).expand(X.shape[0], self.n_in)
        return X if self._as_rows(X) else X.contiguous()

    def predict_device(self, X, batch=65536):
        """Outputs [B][n_out] as a CUDA float32 tensor, for inputs already
        on the GPU (a float tensor [B][n_in]); nothing crosses to the host.
        One launch carries every row through the whole network; inputs of
        another type or layout are converted `batch` rows at a time."""
        packed = self._pack()
        out = self.torch.empty((X.shape[0], self.n_out), device=self.dev)
        if self._as_rows(X):
            self.k.predict(X, packed, self.b, out)
        else:
            for s in range(0, X.shape[0], batch):
                self.k.predict(self._rows(X[s:s + batch]), packed, self.b, out[s:s + batch])
        self.k.check()
        return out

    def predict(self, X, batch=65536):
        """Outputs [B][n_out] (float32, on the host)."""
        torch = self.torch
        packed = self._pack()
        out = []
        for s in range(0, X.shape[0], batch):
            x = torch.as_tensor(X[s:s + batch], device=self.dev, dtype=torch.float32)
            y = torch.empty((x.shape[0], self.n_out), device=self.dev)
            self.k.predict(self._rows(x), packed, self.b, y)
            out.append(y.cpu().numpy())
        self.k.check()
        return np.concatenate(out) if out else np.zeros((0, self.n_out), np.float32)

    def _work(self, rows):
        return self._buf("work", (int(self.k.L.dense_mlp_train_bytes(rows, self.n_out)),), self.torch.uint8)

    def _grads(self):
        return ([self._buf("dW%d" % i, w.shape) for i, w in enumerate(self.W)],
                [self._buf("db%d" % i, b.shape) for i, b in enumerate(self.b)])

    def gradients(self, X, T, mask):
        """Loss and gradients (dW, db lists) of one batch."""
        torch = self.torch
        B = X.shape[0]
        f32 = dict(device=self.dev, dtype=torch.float32)
        x = torch.as_tensor(X, **f32).expand(B, self.n_in).contiguous()
        t = torch.as_tensor(np.nan_to_num(T), **f32).expand(B, self.n_out).contiguous()
        m = torch.as_tensor(mask, **f32).expand(B, self.n_out).contiguous()
        count = float(m.sum().item() if torch.is_tensor(mask) else
                      np.broadcast_to(np.asarray(mask, np.float32), (B, self.n_out)).sum(dtype=np.float64))
        loss = torch.zeros(1, device=self.dev)
        dW, db = self._grads()
        work = self._work(B)
        self.k.train_pass(x, t, m, None, B, self._pack(backward=True), self.b, 1.0 / max(1.0, count), loss, work)
        self.k.train_finish(work, B, self.n_out, dW, db)
        self.k.check()
        return float(loss.item()), dW, db

    def _train_buffers(self, batch, steps):
        """Per epoch the host writes the epoch's row indices ("idx", steps x
        batch) and per-step scalars ("hyper", steps x {lr, b1, b2, eps,
        1 - b1^t, 1 - b2^t, 1 / count}) into these device buffers."""
        torch = self.torch
        return {"idx": torch.zeros(steps * batch, dtype=torch.int32, device=self.dev),
                "hyper": torch.zeros((steps, 8), device=self.dev),
                "loss": torch.zeros(1, device=self.dev)}

    def _train_graphs(self, g, data, batch, steps):
        """CUDA graphs of data-parallel training on the device-resident
        training set `data` = (X, T, mask), `steps` steps of `batch` rows per
        epoch, reading the buffers g: per step a gradient graph and an update
        graph, with the gradient all-reduce between them.  The graphs hold
        the addresses of this object's work buffers: they serve one fit call
        only (no other pass may resize a buffer meanwhile)."""
        torch = self.torch
        Xd, Td, Md = data
        work = self._work(batch)
        packed = self._packed
        dW, db = g["dW"], g["db"] = self._grads()

        def grads(j):
            self._pack(backward=True)
            self.k.train_pass(Xd, Td, Md, g["idx"][j * batch:(j + 1) * batch], batch, packed, self.b,
                              g["hyper"][j, 6:7], g["loss"], work)
            self.k.train_finish(work, batch, self.n_out, dW, db)

        def update(j):
            hyper = g["hyper"][j]
            for i in range(4):
                self.k.adam_dev(self.W[i], dW[i], self.mW[i], self.vW[i], hyper)
                self.k.adam_dev(self.b[i], db[i], self.mb[i], self.vb[i], hyper)

        side = torch.cuda.Stream(self.dev)
        side.wait_stream(torch.cuda.current_stream(self.dev))
        with torch.cuda.stream(side):
            grads(0)  # a first launch of each kernel before capture; changes no weight
        torch.cuda.current_stream(self.dev).wait_stream(side)
        torch.cuda.synchronize(self.dev)
        g["grads"], g["update"] = [], []
        for j in range(steps):
            gg, gu = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
            with torch.cuda.graph(gg):
                grads(j)
            with torch.cuda.graph(gu):
                update(j)
            g["grads"].append(gg)
            g["update"].append(gu)

    def _fit_epochs(self, X, T, mask, n, epochs, batch, rng, cosine, data=None, b1=0.9, b2=0.999, eps=1e-8):
        """Generator behind the captured fit: each next() enqueues one epoch
        on the current stream and returns a function that reads that
        epoch's mean loss (call it before the next epoch is enqueued).
        `data`: the training set already on the device (X, T, mask)."""
        torch = self.torch
        steps = n // batch
        if steps == 0:
            for _ in range(epochs):
                yield lambda: 0.0
            return
        if data is None:
            data = device_training_set(X, T, mask, self.dev)
        g = self._train_buffers(batch, steps)
        if self.group is not None:
            self._train_graphs(g, data, batch, steps)
        lr0 = self.lr
        total = epochs * steps
        for ep in range(epochs):
            rows = rng.permutation(X.shape[0])[:n][:steps * batch]
            counts = mask[rows].reshape(steps, batch, -1).sum(axis=(1, 2), dtype=np.float64)
            hyp = np.zeros((steps, 8), np.float64)
            for j in range(steps):
                lr = lr0
                if cosine:
                    t = (ep * steps + j) / max(1, total - 1)
                    lr = lr0 * (0.01 + 0.99 * 0.5 * (1.0 + np.cos(np.pi * t)))
                step = self.steps + j + 1
                hyp[j] = (lr, b1, b2, eps, 1.0 - b1 ** step, 1.0 - b2 ** step, 1.0 / max(1.0, counts[j]), 0.0)
            g["idx"].copy_(torch.as_tensor(rows.astype(np.int32)))
            g["hyper"].copy_(torch.as_tensor(hyp.astype(np.float32)))
            g["loss"].zero_()
            if self.group is None:
                # one call launches the epoch's steps, four kernels each: 10 us
                # a step of the host's time, below the step's on the GPU, so a
                # graph of them gains nothing and its capture cost more than
                # a short fit (57 steps: 14.5 ms with one, 11.2 without; four
                # networks at once over 40 epochs: 203 and 212)
                self._pack(backward=True)
                self.k.train_epoch(*data, g["idx"], g["hyper"], g["loss"], self._work(batch), self)
            else:
                from .distributed import average_
                for j in range(steps):
                    g["grads"][j].replay()
                    average_(g["dW"] + g["db"], self.group)
                    g["update"][j].replay()
            self.steps += steps
            yield lambda: float(g["loss"].item()) / steps
        del g

    def _fit_captured(self, X, T, mask, n, epochs, batch, rng, log, cosine):
        hist = []
        for ep, loss in enumerate(self._fit_epochs(X, T, mask, n, epochs, batch, rng, cosine)):
            hist.append(loss())
            self.k.check()
            if log:
                log("epoch %d loss %.5f" % (ep, hist[-1]))
        return hist

    def step(self, X, T, mask):
        loss, dW, db = self.gradients(X, T, mask)
        if self.group is not None:
            from .distributed import average_
            average_(dW + db, self.group)
        self.steps += 1
        for i in range(4):
            self.k.adam(self.W[i], dW[i], self.mW[i], self.vW[i], self.lr, self.steps)
            self.k.adam(self.b[i], db[i], self.mb[i], self.vb[i], self.lr, self.steps)
        return loss

    def fit(self, X, T, mask, epochs=20, batch=4096, seed=0, log=None, cosine=True, captured=True):
        """Minibatch Adam; with `cosine` the learning rate follows a cosine
        from lr down to lr/100 over the run.  With `captured` (the default)
        the training set is copied to the GPU once and its rows are
        gathered there (one call launches an epoch; with a group every step
        replays two CUDA graphs, gradient and update); otherwise each step
        is launched from the host (`step`), with the same batches and
        schedule."""
        rng = np.random.Generator(np.random.PCG64(seed))
        n = X.shape[0]
        if self.group is not None:
            # every rank takes the same number of steps: the smallest shard's
            import torch.distributed as dist
            t = self.torch.tensor([n], device=self.dev)
            dist.all_reduce(t, op=dist.ReduceOp.MIN, group=self.group)
            n = int(t.item())
        if captured:
            return self._fit_captured(X, T, mask, n, epochs, batch, rng, log, cosine)
        hist = []
        lr0 = self.lr
        per_epoch = max(1, n // batch)
        total = epochs * per_epoch
        for ep in range(epochs):
            order = rng.permutation(X.shape[0])[:n]
            tot = 0.0
            for j, s in enumerate(range(0, n - batch + 1, batch)):
                if cosine:
                    t = (ep * per_epoch + j) / max(1, total - 1)
                    self.lr = lr0 * (0.01 + 0.99 * 0.5 * (1.0 + np.cos(np.pi * t)))
                idx = order[s:s + batch]
                tot += self.step(X[idx], T[idx], mask[idx])
            hist.append(tot / max(1, n // batch))
            if log:
                log("epoch %d loss %.5f" % (ep, hist[-1]))
        self.lr = lr0
        return hist

    def state(self):
        return {"W": [w.cpu().numpy() for w in self.W], "b": [b.cpu().numpy() for b in self.b]}


def device_training_set(X, T, mask, dev):
    """The training set on the device as float32 tensors (NaN targets 0)."""
    import torch
    return (torch.as_tensor(np.ascontiguousarray(X, dtype=np.float32), device=dev),
            torch.as_tensor(np.ascontiguousarray(np.nan_to_num(T), dtype=np.float32), device=dev),
            torch.as_tensor(np.ascontiguousarray(mask, dtype=np.float32), device=dev))


def fit_concurrently(nets, X, T, mask, seeds, epochs=20, batch=4096, log=None, cosine=True):
    """MLP.fit of several networks of one process at once, each on its own
    CUDA stream (a network's epoch is one call, and the tiles of one
    4096-row batch fill only a part of the SMs, so the networks share the
    GPU).  Network k takes the batches of seed seeds[k]: its weights are
    those of nets[k].fit(..., seed=seeds[k]).  Returns the loss histories."""
    import torch
    assert all(net.group is None for net in nets)
    dev = nets[0].dev
    data = device_training_set(X, T, mask, dev)
    n = X.shape[0]
    streams = [torch.cuda.Stream(dev) for _ in nets]
    for st in streams:
        st.wait_stream(torch.cuda.current_stream(dev))
    gens = [net._fit_epochs(X, T, mask, n, epochs, batch, np.random.Generator(np.random.PCG64(sd)), cosine,
                            data=data) for net, sd in zip(nets, seeds)]
    hists = [[] for _ in nets]
    for ep in range(epochs):
        readers = []
        for gen, st in zip(gens, streams):
            with torch.cuda.stream(st):
                readers.append(next(gen))
        for k, (read, st) in enumerate(zip(readers, streams)):
            with torch.cuda.stream(st):
                hists[k].append(read())
        for net in nets:
            net.k.check()
        if log:
            log("epoch %d loss %s" % (ep, " ".join("%.5f" % h[-1] for h in hists)))
    for gen in gens:
        gen.close()
    torch.cuda.current_stream(dev).wait_stream(streams[0])
    for st in streams[1:]:
        torch.cuda.current_stream(dev).wait_stream(st)
    return hists


def bench_gemm(rows=131072, reps=20, device=0):
    """Times the tensor-core GEMM on the MLP's layer shapes (BF16 inputs,
    FP32 outputs): rows x 256 x 64 (first layer), rows x 256 x 256 (hidden
    layers), rows x 128 x 256 (output layer), plain and with the bias+GELU
    epilogue; one dict per shape and epilogue, CUDA-event timed."""
    import torch
    k = Kernels(device)
    dev = "cuda:%d" % device
    out = []
    for (n, kk) in ((256, 64), (256, 256), (128, 256)):
        A = torch.randn(rows, kk, device=dev).to(torch.bfloat16)
        B = torch.randn(n, kk, device=dev).to(torch.bfloat16)
        D = torch.empty(rows, n, device=dev, dtype=torch.float32)
        H = torch.empty(rows, n, device=dev, dtype=torch.bfloat16)
        bias = torch.randn(n, device=dev)
        for epi, name in ((EPI_STORE, "store"), (EPI_BIAS_GELU, "bias_gelu")):
            k.gemm(A, B, D, epi, bias, H)
            torch.cuda.synchronize(device)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s = torch.cuda.current_stream(device)
            e0.record(s)
            for _ in range(reps):
                k.gemm(A, B, D, epi, bias, H)
            e1.record(s)
            torch.cuda.synchronize(device)
            ms = e0.elapsed_time(e1) / reps
            nbytes = rows * kk * 2 + n * kk * 2 + rows * n * 4 + (rows * n * 2 if epi == EPI_BIAS_GELU else 0)
            out.append({"rows": rows, "n": n, "k": kk, "epilogue": name, "us": ms * 1e3,
                        "tflops": 2.0 * rows * n * kk / ms / 1e9, "gbs": nbytes / ms / 1e6})
    k.check()
    return out


def bench_fit(rows=200000, epochs=3, batch=4096, n_in=44, n_out=5, device=0):
    """Wall time per training step of MLP.fit on seeded random data, the
    device-resident form (one call per epoch) and the launched form; each
    after a one-epoch warm-up on a slice."""
    import time
    import torch
    rng = np.random.Generator(np.random.PCG64(0))
    X = rng.uniform(-1, 1, size=(rows, n_in)).astype(np.float32)
    T = rng.normal(size=(rows, n_out)).astype(np.float32)
    M = np.ones((rows, n_out), np.float32)
    out = []
    for captured in (True, False):
        net = MLP(n_in, n_out, seed=0, device=device)
        net.fit(X[:8 * batch], T[:8 * batch], M[:8 * batch], epochs=1, batch=batch, captured=captured)
        torch.cuda.synchronize(device)
        t0 = time.perf_counter()
        net.fit(X, T, M, epochs=epochs, batch=batch, captured=captured)
        torch.cuda.synchronize(device)
        steps = epochs * (rows // batch)
        out.append({"captured": captured, "rows": rows, "batch": batch, "epochs": epochs, "steps": steps,
                    "ms_per_step": 1e3 * (time.perf_counter() - t0) / steps})
    return out


if __name__ == "__main__":
    import argparse
    import json
    ap = argparse.ArgumentParser(description="time the surrogate's tensor-core GEMM, or its training steps")
    ap.add_argument("--rows", type=int, default=131072)
    ap.add_argument("--reps", type=int, default=20)
    ap.add_argument("--fit", action="store_true", help="time MLP.fit steps instead (--rows training rows)")
    ap.add_argument("--epochs", type=int, default=3)
    ap.add_argument("--batch", type=int, default=4096)
    a = ap.parse_args()
    for r in (bench_fit(a.rows, a.epochs, a.batch) if a.fit else bench_gemm(a.rows, a.reps)):
        print(json.dumps(r))
