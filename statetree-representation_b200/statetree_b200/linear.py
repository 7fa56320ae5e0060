"""TreeLinear / TreeSlice / TreeEmbedding: drop-in modules over the sm_100a kernels, with the buffers and call
surface of the reference's statetree/linear.py (TreeLinear 595-1018, TreeSlice 1021-1036, TreeEmbedding 1039-1067,
torch.compile custom ops 1070-1095).

Dispatch is one kernel per regime (no tuner, no multi-kernel ladder): up to GEMV_MAX activation rows run the
memory-order fused decode GEMV, more rows the fused decode + tcgen05 GEMM, and prefill batches (more than PREFILL_MIN rows;
for larger matrices more than FUSED_ROWS or HOST_ROWS, see dense_for) the decode kernel into a BF16 scratch matrix + cuBLAS
(the reference's prefill path).  Workspaces (exchange slots and zeroed
semaphores) are kept per (device, stream) because callers may run layers on side streams concurrently (the reason
given at statetree/linear.py:457-466); they are sized once per shape, so steady-state calls allocate only the output.
"""
import os
import threading
import weakref

import torch
import torch.nn as nn

from . import format as F
from .ops import _raw_stream, built, calls, ext, on_device

# activation rows up to which the GEMV kernel runs (<= 32).  The four projections of a 4096 / 12288 layer in a graph, us with
# the GEMV / the tcgen05 GEMM: 8 rows 57 / 72, 16 rows 68 / 72, 20 rows 125 / 72 (beyond 16 the GEMV holds one CTA per SM)
GEMV_MAX = int(os.environ.get("STATETREE_GEMV_MAX", "16"))
GEMV_AR_MAX = 12                    # rows up to which the GEMV that sums over the ranks itself is used (tensor parallelism)
# more activation rows than this (prefill): the tree is decoded once into a BF16 scratch matrix and cuBLAS multiplies by
# it, the reference's path above 1024 rows (statetree/linear.py:37, 879-886), here from the size at which it overtakes the
# tcgen05 kernel; 0 turns it off
PREFILL_MIN = int(os.environ.get("STATETREE_PREFILL_MIN", "512"))
# ... except that matrices of at least FUSED_WEIGHTS weights stay on the tcgen05 kernel for up to FUSED_ROWS rows, and for up to
# HOST_ROWS rows below DENSE_WEIGHTS weights, where the scratch path, 75 us of Python, events and launches per call, waits for the
# host.  These lines are where the two paths met when a tile was one CTA's (all projections of 36 layers of 4096 / 12288, ms with
# the kernel / the scratch matrix: 960 rows 13.7 / 15.5, 1920 25.6 / 25.9, 2000 28.5 / 25.7).  With CTA pairs the kernel is ahead on
# both sides of them (us per layer, median of 11 passes, the paths in turn):
#   rows               513         960         1536        2000        4096         8192
#   4096 / 12288       201 / 377   313 / 428   488 / 609   657 / 703   1230 / 1395  2517 / 2629
#   2048 / 6144        82 / 342    98 / 342    130 / 343   161 / 343   333 / 365    668 / 682
# The lines have not been moved with it: test_path_of_a_prefill_batch (tests/test_gpu_weights.py) states them, and moving them is a
# change of its own.
FUSED_ROWS, FUSED_WEIGHTS = 1920, 1 << 22
HOST_ROWS, DENSE_WEIGHTS = 2048, 1 << 24
DENSE_MAX = 1 << 28                 # weights: larger matrices (vocabulary-sized tables) never get a dense scratch copy
_STATES = {}
_BUFFERS = ("tree", "esc_rows", "esc_cols", "esc_bits")


class EscapeHeavy(RuntimeError):
    """more weights escape than the caller allows (the layer is better left in BF16)"""


class _DevState:
    """per (device, stream): the fp32 workspace of the small-batch kernels and the semaphore array.  The kernels expect
    every workspace word to hold 0xFFFFFFFF between launches (their exchange-slot sentinel) and every semaphore to be
    zero, and leave them so.  Buffers only ever grow, and a buffer that was handed out is never freed: a CUDA graph
    captured earlier keeps replaying into the old one."""

    def __init__(self, device):
        self.device = device
        self._retired = []
        self._need = {}                                 # workspace bytes per call shape (a pure function of it)
        self.ws = self._new_ws(1 << 20)
        self.scratch = torch.empty(0, dtype=torch.float32, device=device)         # the GEMM's workspace (it asks for none)
        self.cnt = torch.zeros(1 << 16, dtype=torch.int32, device=device)

    def _new_ws(self, words):
        return torch.full((words,), -1, dtype=torch.int32, device=self.device).view(torch.float32)

    def get_ws(self, nbytes):
        if self.ws.numel() * 4 < nbytes:
            self._retired.append(self.ws)
            self.ws = self._new_ws((nbytes + 3) // 4)
        return self.ws

    def gemv_ws(self, M, N, B):
        """workspace for a GEMV of an M x N matrix (M a tuple: a list of matrices) with B rows"""
        need = self._need.get((M, N, B))
        if need is None:
            E = ext()
            with on_device(self.device.index):          # (the size depends on the device's SMs; the caller may be on another one)
                need = E.gemv_list_workspace_bytes(M, N, B) if isinstance(M, tuple) else E.gemv_workspace_bytes(M, N, B)
            if len(self._need) < 4096:
                self._need[(M, N, B)] = need
        return self.get_ws(need)

    def get_scratch(self, nbytes):
        if self.scratch.numel() * 4 < nbytes:
            self._retired.append(self.scratch)
            self.scratch = torch.empty((nbytes + 3) // 4, dtype=torch.float32, device=self.device)
        return self.scratch

    def dense_stage(self):
        if self.__dict__.get("_dense") is None:
            self._dense = _DenseStage(self.device)
        return self._dense

    def get_cnt(self, n):
        if self.cnt.numel() < n:
            self._retired.append(self.cnt)
            self.cnt = torch.zeros(n, dtype=torch.int32, device=self.device)
        return self.cnt


class _Decoded:
    """What a scratch matrix was decoded from: the tensor that holds the tree, as it was then, and the escape tables of that
    time.  By weak reference: ids and addresses are given out again, and a matrix must never pass for that of the layer that took
    the place of another."""

    def __init__(self, layer):
        tree = layer._buffers["tree"]
        self.tree, self.eo = weakref.ref(tree), weakref.ref(layer.tables()[0])
        self.version = None if tree.is_inference() else tree._version

    def __eq__(self, other):
        if not isinstance(other, _Decoded):
            return False
        tree, eo = self.tree(), self.eo()
        return (tree is not None and tree is other.tree() and eo is not None and eo is other.eo()
                and self.version == other.version)

    __hash__ = None


class _DenseStage:
    """Prefill-size batches: decode once, multiply with cuBLAS (statetree/linear.py:286-368 is the reference's form).
    Two BF16 scratch matrices per (device, stream).  While the GEMM reads one, a side stream decodes the layer linked
    as `_next` (by model.prepare, in module order) into the other: the decode is HBM-bound, the GEMM tensor-bound, so
    from the second layer of a pass on the decode hides under the GEMM.  A wrong guess of the next layer costs one
    wasted decode, never a wrong result: a scratch matrix is used only if it holds exactly the asked tree."""

    def __init__(self, device):
        self.device = device
        self.side = torch.cuda.Stream(device)                # (a high-priority stream measured slower: 17.2 against 14.8 ms at 1024 rows)
        self.mat = [None, None]                              # flat BF16 scratch
        self.holds = [None, None]                            # _Decoded: what each holds
        self.decoded = [None, None]                          # event: that decode has finished
        self.read = [None, None]                             # event: the last GEMM that read it has finished
        self.turn = 0
        self.lock = threading.Lock()                         # two threads may share a stream, and so this object

    _ident = _Decoded

    def _matrix(self, slot, layer):
        need = layer.out_features * layer.in_features
        if self.mat[slot] is None or self.mat[slot].numel() < need:
            if self.mat[slot] is not None:
                self.mat[slot].record_stream(self.side)       # a decode on the side stream may still be writing it
            self.mat[slot] = torch.empty(need, dtype=torch.bfloat16, device=self.device)
            self.mat[slot].record_stream(self.side)
            self.holds[slot] = None
        return self.mat[slot][:need].view(layer.out_features, layer.in_features)

    def run(self, layer, x, y):
        with self.lock:                                      # (the decode and the product that reads it go out together)
            self._run(layer, x, y)

    def _run(self, layer, x, y):
        cur = torch.cuda.current_stream(self.device)
        me = self._ident(layer)
        if me in self.holds:
            slot = self.holds.index(me)
            cur.wait_event(self.decoded[slot])
            W = self._matrix(slot, layer)
        else:
            slot = self.turn
            if self.decoded[slot] is not None:
                cur.wait_event(self.decoded[slot])           # a prefetch of some other layer into this slot
            W = self._matrix(slot, layer)
            eo, el, _ = layer.tables()
            ext().dec(layer.tree, eo, el, W)
            self.holds[slot] = me
            self.decoded[slot] = cur.record_event()
        other = 1 - slot
        nxt = layer._next() if layer._next is not None else None
        fork = None
        if (nxt is not None and nxt.dense_for(x.shape[0]) and nxt.tree.device == layer.tree.device
                and self.holds[other] != self._ident(nxt)):
            nxt.tables()                                     # built on the caller's stream, before the fork
            Wn = self._matrix(other, nxt)
            fork = cur.record_event()
        torch.matmul(x, W.t(), out=y)
        self.read[slot] = cur.record_event()
        self.turn = other
        if fork is not None:
            self.side.wait_event(fork)
            if self.read[other] is not None:
                self.side.wait_event(self.read[other])       # the GEMM that last read the other matrix
            with torch.cuda.stream(self.side):
                eo, el, _ = nxt.tables()
                ext().dec(nxt.tree, eo, el, Wn)
                self.decoded[other] = self.side.record_event()
            self.holds[other] = self._ident(nxt)


def _state(device):
    if not isinstance(device, torch.device):
        device = torch.device(device)
    index = device.index
    if index is None:
        index = torch.cuda.current_device()
    key = (index, _raw_stream(index))
    st = _STATES.get(key)
    if st is None:
        st = _STATES[key] = _DevState(torch.device("cuda", index))
    return st


def _rows_2d(x, width):
    """x [..., width] of any float dtype / layout -> BF16 [rows, width], contiguous and 16-byte aligned"""
    flat = x.reshape(-1, width)
    if x.shape[-1] != width and flat.shape[0] != x.shape[:-1].numel():    # (a multiple or a divisor of the width)
        raise RuntimeError(f"statetree_b200: the layer takes inputs of {width} columns, got {tuple(x.shape)}")
    if flat.dtype != torch.bfloat16:
        flat = flat.to(torch.bfloat16)
    if flat.data_ptr() % 16 or not flat.is_contiguous():
        flat = flat.clone(memory_format=torch.contiguous_format)
    return flat


# layers reachable from the custom ops by a string handle (torch.compile passes plain strings, not modules)
_BY_HANDLE = weakref.WeakValueDictionary()


_tracing = getattr(getattr(torch, "compiler", None), "is_compiling", None) or (lambda: False)


class TreeLinear(nn.Module):
    """y = x W^T (+ b) with W [out, in] BF16 stored as a lossless state tree (~12.1 bits/weight).

    Buffers (state dict): tree uint8 [out/16, in/64, 1552], esc_rows / esc_cols int32, esc_bits int16 (exact bits of
    the weights the tree cannot hold), bias (optional, bf16)."""

    def __init__(self, in_features, out_features, bias=False, device=None, n_esc=0):
        super().__init__()
        assert out_features % 16 == 0 and in_features % 64 == 0, "TreeLinear needs out % 16 == 0 and in % 64 == 0"
        self.in_features, self.out_features = in_features, out_features
        dev = torch.device(device) if device is not None else None
        self.register_buffer("tree", torch.empty(out_features // 16, in_features // 64, F.RECORD_BYTES,
                                                 dtype=torch.uint8, device=dev))
        self.register_buffer("esc_rows", torch.empty(n_esc, dtype=torch.int32, device=dev))
        self.register_buffer("esc_cols", torch.empty(n_esc, dtype=torch.int32, device=dev))
        self.register_buffer("esc_bits", torch.empty(n_esc, dtype=torch.int16, device=dev))
        if bias:
            self.register_buffer("bias", torch.empty(out_features, dtype=torch.bfloat16, device=dev))
        else:
            self.bias = None
        self._handle = f"tl{id(self):x}"
        _BY_HANDLE[self._handle] = self
        self._reset_runtime()

    def set_handle(self, name):
        """The string under which the torch.compile custom ops find this layer; a stable name (the module path) keeps a
        compiled graph valid in another process (statetree/linear.py:621-625)."""
        self._handle = str(name)
        _BY_HANDLE[self._handle] = self

    def prepare(self, batch_sizes=(1,)):
        """Side tables and workspaces for these batch sizes now, so that a later call (or a CUDA-graph capture)
        allocates nothing (statetree/linear.py:1014-1018; there is no plan to pick here: one kernel per regime)."""
        if not self.tree.is_cuda:
            raise RuntimeError("TreeLinear.prepare: the layer must be on a GPU")
        E, st = ext(), _state(self.tree.device)
        self.tables()
        M, N = self.out_features, self.in_features
        for B in batch_sizes:
            if B <= min(GEMV_MAX, 32) or M % 128:
                st.get_ws(E.gemv_workspace_bytes(M, N, min(B, 32)))
                st.get_cnt(M // 16)
            else:
                st.get_scratch(E.gemm_workspace_bytes(M, N, B))
                st.get_cnt((M // 128) * ((B + 255) // 256))
        return self

    # ---------------------------------------------------------------- construction / state dict
    @classmethod
    def from_linear(cls, lin, verify=True, max_escape_fraction=None):
        return cls.from_weight(lin.weight, lin.bias, verify=verify, max_escape_fraction=max_escape_fraction)

    @classmethod
    @torch.no_grad()
    def from_weight(cls, W, bias=None, verify=True, max_escape_fraction=None):
        """W [out, in] bf16.  max_escape_fraction: raise EscapeHeavy when more weights escape."""
        W = W.detach()
        if W.dtype != torch.bfloat16:
            raise TypeError(f"TreeLinear.from_weight: expected a bfloat16 weight, got {W.dtype}")
        if max_escape_fraction is not None:
            escapes = F.escape_count(W)
            if escapes > max_escape_fraction * W.numel():
                raise EscapeHeavy(f"{escapes / W.numel():.2%} of the weights escape")
        on_gpu = (W.is_cuda and W.dim() == 2 and W.numel() > 0 and W.shape[0] % 16 == 0 and W.shape[1] % 64 == 0 and built())
        enc, tables = F.encode_with_tables(W) if on_gpu else (F.encode(W), None)
        if verify and on_gpu:
            # (what is stored is checked, not only the tables of this process: a reload builds its tables from the lists)
            bad = ext().check_start(enc["tree"], tables[0], tables[1],
                                    W if W.data_ptr() % 16 == 0 and W.is_contiguous() else W.clone(memory_format=torch.contiguous_format),
                                    (enc["esc_rows"], enc["esc_cols"], enc["esc_bits"], tables[2]))
        out_features, in_features = W.shape             # (the module is made while the check runs)
        layer = cls(in_features, out_features, bias=bias is not None, device="meta", n_esc=int(enc["esc_rows"].numel()))
        layer._buffers.update({name: enc[name] for name in _BUFFERS})
        if bias is not None:
            layer._buffers["bias"] = bias.detach().to(device=W.device, dtype=torch.bfloat16).clone()
        layer._reset_runtime()
        if verify:
            if on_gpu:
                same = int(bad) == 0
            else:
                back = layer.dequantize() if layer.tree.is_cuda else F.decode_reference(*(layer._buffers[n] for n in _BUFFERS))
                same = torch.equal(back.view(torch.int16), W.view(torch.int16))
            if not same:
                raise RuntimeError("TreeLinear: the tree does not decode to the weights it was built from")
        if on_gpu:                                      # (see tables(): complete before any later kernel may start)
            if not verify:                              # (the check has synchronised)
                torch.cuda.current_stream(W.device).synchronize()
            layer._tables = tables
        return layer

    def _load_from_state_dict(self, state_dict, prefix, local_metadata, strict, missing_keys, unexpected_keys,
                              error_msgs):
        # how many weights escape depends on the data: make room for whatever the checkpoint holds
        for name in _BUFFERS[1:]:
            stored = state_dict.get(prefix + name)
            mine = self._buffers[name]
            if stored is not None and stored.shape != mine.shape:
                self._buffers[name] = torch.empty(stored.shape, dtype=stored.dtype, device=mine.device)
        super()._load_from_state_dict(state_dict, prefix, local_metadata, strict, missing_keys, unexpected_keys,
                                      error_msgs)
        self._reset_runtime()

    def _apply(self, fn, *args, **kwargs):
        out = super()._apply(fn, *args, **kwargs)
        self._reset_runtime()
        return out

    def _reset_runtime(self):
        self._tables = None                             # (eo, el, eb) on the tree's device
        self.__dict__["_shared"] = None                 # product shared by the TreeSlice views of this layer
        self.__dict__.setdefault("_next", None)         # weak reference to the layer that runs after this one
        self.__dict__.setdefault("allow_dec", True)     # False: never a dense scratch copy (the reference's flag for
                                                        # vocabulary-sized tables, statetree/linear.py:808-810)

    def __getstate__(self):
        state = self.__dict__.copy()
        state["_next"] = None                           # (a weak reference cannot be pickled; prepare() links again)
        return state

    def dense_ok(self):
        """may this layer be decoded into a BF16 scratch matrix for prefill-size batches"""
        return self.allow_dec and self.tree.is_cuda and self.out_features * self.in_features <= DENSE_MAX

    def dense_for(self, B):
        """do B rows go through the scratch matrix"""
        M, N = self.out_features, self.in_features
        fused = M % 128 == 0 and M * N >= FUSED_WEIGHTS and B <= (HOST_ROWS if M * N < DENSE_WEIGHTS else FUSED_ROWS)
        return 0 < PREFILL_MIN < B and not fused and self.dense_ok()

    def extra_repr(self):
        return (f"in_features={self.in_features}, out_features={self.out_features}, bias={self.bias is not None}, "
                f"escapes={self.esc_rows.numel()}, bits_per_weight={self.bits_per_weight:.3f}")

    @property
    def bits_per_weight(self):
        return F.bits_per_weight(self.out_features, self.in_features, self.esc_rows.numel())

    def storage_bytes(self):
        return sum(self._buffers[n].numel() * self._buffers[n].element_size() for n in _BUFFERS)

    def record_bytes(self):
        return self.tree.numel()

    def tables(self):
        """(eo, el, eb) escape side tables, built on first use (outside any graph capture).  The kernels read them
        before they wait for the preceding kernel of the stream (programmatic dependent launch), so the tables must be
        complete before that kernel starts: the stream is synchronised once after building them."""
        if self._tables is None or self._tables[0].device != self._buffers["tree"].device:
            self._tables = F.escape_tables(self.out_features, self.in_features, self.esc_rows, self.esc_cols,
                                           self.esc_bits)
            if self.tree.is_cuda and not torch.cuda.is_current_stream_capturing():
                torch.cuda.current_stream(self.tree.device).synchronize()
        return self._tables

    def dequantize(self):
        """The exact BF16 weight [out, in] (decoded by the CUDA kernel)."""
        W = torch.empty(self.out_features, self.in_features, dtype=torch.bfloat16, device=self.tree.device)
        eo, el, _ = self.tables()
        ext().dec(self.tree, eo, el, W)
        return W

    @torch.no_grad()
    def rows(self, ids):
        """W[ids] (exact BF16 rows), decoded on the fly: the embedding lookup of a tree-stored table."""
        where = self.tree.device
        index = ids.reshape(-1).to(device=where, dtype=torch.int64).contiguous()
        gathered = torch.empty(index.numel(), self.in_features, dtype=torch.bfloat16, device=where)
        eo, el, _ = self.tables()
        ext().rows(self.tree, eo, el, index, gathered)
        return gathered.view(*ids.shape, self.in_features)

    # ---------------------------------------------------------------- forward
    def _run(self, x, y, yf32=None):
        """x [B, in] bf16 contiguous 16-byte aligned -> y [B, out] (one launch per GEMV_MAX rows or one GEMM)"""
        E = ext()
        B = x.shape[0]
        M, N = self.out_features, self.in_features
        eo, el, eb = self.tables()
        st = _state(x.device)
        if B <= min(GEMV_MAX, 32):
            E.gemv(self._buffers["tree"], eo, eb, el, x, y, st.gemv_ws(M, N, B), st.get_cnt(M // 16), yf32)
        elif self.dense_for(B) and yf32 is None and not torch.cuda.is_current_stream_capturing():
            st.dense_stage().run(self, x, y)                # decode once + cuBLAS, the next layer decoded meanwhile
        elif M % 128 == 0:
            ws = st.get_scratch(E.gemm_workspace_bytes(M, N, B))
            E.gemm(self.tree, eo, el, x, y, ws, st.get_cnt((M // 128) * ((B + 255) // 256)), yf32)
        else:                                           # rows not a multiple of 128: GEMV kernel in row chunks
            step = min(32, max(GEMV_MAX, 16))
            ws = st.get_ws(E.gemv_workspace_bytes(M, N, step))
            for b0 in range(0, B, step):
                E.gemv(self.tree, eo, eb, el, x[b0:b0 + step], y[b0:b0 + step], ws, st.get_cnt(M // 16),
                       None if yf32 is None else yf32[b0:b0 + step])

    def forward(self, x):
        if _tracing() and _OPS_READY:
            return torch.ops.statetree.linear(x, self.tree, self._handle)
        return self._forward(x)

    def _plain(self, x, home):
        """the product in one native call (csrc/py_calls.cpp), for a layer without a bias and BF16 inputs that lie on its device
        contiguous and 16-byte aligned; None for inputs of another width or without rows, for batches that go through the scratch
        matrix and where that module has not been built"""
        M, N, shape = self.out_features, self.in_features, x.shape
        if not shape or shape[-1] != N:
            return None
        B, host = x.numel() // N, calls()
        if B < 1 or host is None:
            return None
        use_gemm = B > GEMV_MAX or B > 32
        if not use_gemm:
            st = _state(home)
            ws, cnt = st.gemv_ws(M, N, B), st.get_cnt(M // 16)
        elif M % 128 == 0 and not self.dense_for(B):
            st = _state(home)
            ws, cnt = st.scratch, st.get_cnt((M // 128) * ((B + 255) // 256))     # (the GEMM asks for no workspace)
        else:
            return None
        eo, el, eb = self._tables or self.tables()                # (tables left on another device: the native call takes none)
        return host[0].linear(host[1], use_gemm, self._buffers["tree"], eo, el, eb, x, ws, cnt)

    def _forward(self, x, yf32=None):
        """any leading shape, any float dtype, any device: the product runs where the tree lives, in BF16, and comes
        back in the caller's dtype on the caller's device"""
        home, asked_dtype, asked_device = self._buffers["tree"].device, x.dtype, x.device
        if home.type != "cuda":
            raise RuntimeError("statetree_b200: the kernels take CUDA tensors only (no CPU path); move the layer to a GPU")
        bias = self.bias
        # (what rules an input out for _plain is looked at before anything is fetched for it)
        if (bias is None and yf32 is None and asked_dtype == torch.bfloat16 and asked_device == home and x.is_contiguous()
                and x.data_ptr() % 16 == 0):
            result = self._plain(x, home)
            if result is not None:
                return result
        lead = x.shape[:-1]
        acts = _rows_2d(x if asked_device == home else x.to(home), self.in_features)
        result = torch.empty(acts.shape[0], self.out_features, dtype=torch.bfloat16, device=home)
        if acts.shape[0] > 0:
            with on_device(home.index):
                self._run(acts, result, yf32)
        if bias is not None:
            result += bias
        if len(lead) != 1:
            result = result.view(*lead, self.out_features)
        if asked_dtype != torch.bfloat16:
            result = result.to(asked_dtype)
        return result if asked_device == home else result.to(asked_device)

    def _fused_part(self, x, start, size, nparts):
        """rows [start, start + size) of the product for a TreeSlice: the first part called with an input computes the
        whole fused output, the others reuse it; after the last part the shared result is dropped"""
        shared = self.__dict__.get("_shared")
        if shared is None or shared[0] is not x:
            shared = self.__dict__["_shared"] = [x, self(x), 0]
        shared[2] += 1
        if shared[2] >= nparts:
            self.__dict__["_shared"] = None
        return shared[1].narrow(-1, start, size)


def interleave_gate_up(gate, up):
    """[2 I, in] weight whose 16-row tiles alternate between the gate and the up projection (tile 2j = gate rows
    16j .. 16j + 15, tile 2j + 1 = the same rows of up): the layout TreeLinear.swiglu expects"""
    I, N = gate.shape
    assert up.shape == gate.shape and I % 16 == 0
    return torch.stack([gate.view(I // 16, 16, N), up.view(I // 16, 16, N)], 1).reshape(2 * I, N).contiguous()


def swiglu(self, x):
    """x [B, in] BF16, B <= 8 -> silu(gate x) * (up x) [B, I] in one launch, for a TreeLinear built from
    interleave_gate_up(gate, up); raises RuntimeError for shapes the fused epilogue does not take"""
    B = x.shape[0]
    eo, el, eb = self.tables()
    E, st = ext(), _state(x.device)
    act = torch.empty(B, self.out_features // 2, dtype=torch.bfloat16, device=x.device)
    ws = st.get_ws(E.gemv_workspace_bytes(self.out_features, self.in_features, B))
    E.gemv_swiglu(self.tree, eo, eb, el, x, act, ws, st.get_cnt(self.out_features // 16))
    return act


TreeLinear.swiglu = swiglu


def forward_list(layers, x):
    """[layer(x) for layer in layers] for TreeLinear layers that read the same input (q / k / v or gate / up of a
    checkpoint that keeps them as separate trees): up to four layers run as ONE launch over the concatenation of their
    tiles (the GEMV up to GEMV_MAX rows, the tcgen05 GEMM beyond, if every layer has a multiple of 128 rows); anything
    else falls back to one call per layer."""
    first = layers[0]
    trees = [l._buffers["tree"] for l in layers]
    home, width, shape = trees[0].device, first.in_features, x.shape
    lead, B = shape[:-1], x.numel() // width
    use_gemm = B > GEMV_MAX or B > 32
    if (home.type != "cuda" or B < 1 or not 2 <= len(layers) <= 4
            or any(l.in_features != width or t.device != home for l, t in zip(layers, trees))
            or (use_gemm and any(l.out_features % 128 for l in layers))):
        return [l(x) for l in layers]
    here, bf16 = x.device == home, x.dtype == torch.bfloat16
    widths, biases = [l.out_features for l in layers], [l.bias for l in layers]
    host = calls() if (here and bf16 and x.is_contiguous() and shape[-1] == width and x.data_ptr() % 16 == 0
                       and all(b is None for b in biases)) else None
    if host is not None:
        st = _state(home)                               # one native call for inputs that need no conversion
        scratch = (st.get_cnt((sum(widths) // 128) * ((B + 255) // 256)) if use_gemm else st.gemv_ws(tuple(widths), width, B))
        res = host[0].linear_list(host[1], use_gemm, trees, [l._tables or l.tables() for l in layers], x, scratch)
        if res is not None:
            return res
    acts = _rows_2d(x if here else x.to(home), width)
    # one allocation, a contiguous [B, width] block per layer
    flat = torch.empty(B * sum(widths), dtype=torch.bfloat16, device=home)
    parts = flat.split([B * w for w in widths])
    tabs = []
    for l, t in zip(layers, trees):
        eo, el, eb = l.tables()
        tabs.append((t, eo, eb, el))
    E = ext()
    with on_device(home.index):
        st = _state(home)
        args = E.gemv_list_args(tabs, parts)
        if use_gemm:
            E.gemm_list(args, acts, st.get_cnt((sum(widths) // 128) * ((B + 255) // 256)))
        else:
            E.gemv_list(args, acts, st.gemv_ws(tuple(widths), width, B))
    res = []
    for bias, y, w in zip(biases, parts, widths):
        y = y.view(*lead, w)
        if bias is not None:
            y += bias
        if not bf16:
            y = y.to(x.dtype)
        res.append(y if here else y.to(x.device))
    return res


class TreeSlice(nn.Module):
    """One of several linear layers that read the same input (q / k / v, gate / up), stored together as one TreeLinear
    on the parent module: rows [start, start + size) of that layer's output.  `fused` is the shared layer; it is not
    registered as a submodule here, its buffers belong to the parent (reference: statetree/linear.py:1021-1036)."""

    def __init__(self, fused, start, size, nparts):
        super().__init__()
        object.__setattr__(self, "fused", fused)
        self.in_features, self.out_features = fused.in_features, size
        self.start, self.nparts = start, nparts

    def forward(self, x):
        return self.fused._fused_part(x, self.start, self.out_features, self.nparts)

    def extra_repr(self):
        return f"in_features={self.in_features}, out_features={self.out_features}, rows from {self.start} of the fused layer"


class TreeEmbedding(nn.Module):
    """Embedding lookup from a tree-stored table: rows are decoded exactly on lookup.  The table is either owned
    (`table`, a registered TreeLinear) or, for tied input / output embeddings, the output layer's TreeLinear
    (`source`, not registered here) (reference: statetree/linear.py:1039-1067)."""

    def __init__(self, num_embeddings, embedding_dim, table=None, source=None):
        super().__init__()
        self.num_embeddings, self.embedding_dim = num_embeddings, embedding_dim
        self.table = table
        object.__setattr__(self, "source", source)

    @classmethod
    def from_embedding(cls, emb, verify=True):
        return cls(emb.num_embeddings, emb.embedding_dim, table=TreeLinear.from_weight(emb.weight, verify=verify))

    def _rows_from(self):
        return self.table if self.table is not None else self.source

    def forward(self, ids):
        src = self._rows_from()
        if _tracing() and _OPS_READY:
            return torch.ops.statetree.rows(ids, src.tree, src._handle)
        return src.rows(ids)

    def extra_repr(self):
        return f"{self.num_embeddings}, {self.embedding_dim}, " + ("own table" if self.table is not None else "tied to the output layer")


# ---------------------------------------------------------------------------------------------- torch.compile
# Under torch.compile the layers appear in the traced graph as two opaque custom ops with shape-only fake kernels, so
# Dynamo neither traces into the ctypes shim nor specialises on it (reference: statetree/linear.py:1070-1095).
_OPS_READY = False


def _register_ops():
    global _OPS_READY
    library = getattr(torch, "library", None)
    if library is None or not hasattr(library, "custom_op"):
        return

    @library.custom_op("statetree::linear", mutates_args=())
    def linear_op(x: torch.Tensor, tree: torch.Tensor, handle: str) -> torch.Tensor:
        return _BY_HANDLE[handle]._forward(x)

    @linear_op.register_fake
    def _(x, tree, handle):
        return x.new_empty(*x.shape[:-1], tree.shape[0] * 16)

    @library.custom_op("statetree::rows", mutates_args=())
    def rows_op(ids: torch.Tensor, tree: torch.Tensor, handle: str) -> torch.Tensor:
        return _BY_HANDLE[handle].rows(ids)

    @rows_op.register_fake
    def _(ids, tree, handle):
        return tree.new_empty(*ids.shape, tree.shape[1] * 64, dtype=torch.bfloat16)

    _OPS_READY = True


try:
    _register_ops()
except Exception:                                       # noqa: BLE001  (a torch without torch.library.custom_op,
    _OPS_READY = False                                  # or the ops already registered by another copy of the package)
