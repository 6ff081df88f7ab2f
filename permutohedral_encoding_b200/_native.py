"""ctypes binding of ``libpermuto_b200.so`` (the C ABI in ``include/permuto_b200.h``) and the
three objects the reference's autograd code talks to.

The reference reaches its kernels through a pybind11 module exposing ``EncodingInput``,
``EncodingFixedParams`` and ``EncodingWrapper`` (reference: src/PyBridge.cxx:13-45).  The same
three names live here with the same constructor arguments and method names, implemented on
top of the C ABI, so the autograd functions read like the reference's
(src/pytorch_modules/funcs.py:8-72).  One deliberate difference: features and their gradients
are ``[N, 2*(L+extra)]`` tensors already in the module's output order instead of
``[L+extra, 2, N]``, which removes the three transposing copies the reference pays per step.

The checks, allocations, launches and the autograd graph of the hot calls live in C++
(csrc/permuto_torch.cpp, ``_permuto_torch``): small batches are dominated by host work.  The classes
here keep the reference's names around it.

There is no CPU implementation and no fallback: if a shared library is missing this module
raises at import time with the command that builds it.
"""
from __future__ import annotations

import ctypes as C
import os
import weakref

import numpy as np
import torch

_PKG_DIR = os.path.dirname(os.path.abspath(__file__))
# PERMUTO_B200_LIB names another build of the same library (`python -m permutohedral_encoding_b200.build --out ...`)
LIB_PATH = os.environ.get("PERMUTO_B200_LIB") or os.path.join(_PKG_DIR, "libpermuto_b200.so")

ABI_VERSION = 2
PERMUTO_OK = 0
PERMUTO_TABLE_F32 = 0
PERMUTO_TABLE_F16 = 1
PERMUTO_ERR_INVALID_ARGUMENT = -1
PERMUTO_ERR_UNSUPPORTED = -2
PERMUTO_ERR_CUDA = -3
PERMUTO_ZERO_OUTPUTS = 1
PERMUTO_NO_AGGREGATE = 2
PERMUTO_KEEP_POSITIONS_GRAD = 4
PERMUTO_CONCAT_POSITIONS_GRAD = 8
ORDER_ALWAYS, ORDER_INFERENCE, ORDER_TRAINING, ORDER_POSITIONS = -1, 0, 1, 2   # when EncodingWrapper.order makes an order
PERMUTO_ACT = {"none": 0, "relu": 1, "gelu": 2}
PERMUTO_ADAM_SKIP_UNTOUCHED = 1
PERMUTO_ADAM_ZERO_GRAD = 2

EXPORTED_SYMBOLS = (
    "permuto_abi_version", "permuto_last_error", "permuto_extra_levels", "permuto_scale_factor",
    "permuto_forward", "permuto_backward", "permuto_double_backward", "permuto_debug_lattice",
    "permuto_probe_random_access", "permuto_adam_step", "permuto_forward_linear", "permuto_forward_mlp",
    "permuto_order_pays", "permuto_order_bytes", "permuto_order_points", "permuto_order_record_bytes",
    "permuto_order_scratch_bytes", "permuto_order_records", "permuto_forward_ordered", "permuto_forward_mlp_ordered",
    "permuto_backward_ordered", "permuto_double_backward_ordered", "permuto_backward_combined",
)


class PermutoConfig(C.Structure):
    _fields_ = [("pos_dim", C.c_int32), ("nr_feat_per_level", C.c_int32), ("nr_levels", C.c_int32),
                ("capacity", C.c_int32), ("concat_points", C.c_int32), ("points_scaling", C.c_float),
                ("levels_per_pass", C.c_int32), ("table_dtype", C.c_int32)]


class PermutoMlpLayer(C.Structure):
    _fields_ = [("weight", C.c_void_p), ("bias", C.c_void_p), ("in_features", C.c_int32), ("out_features", C.c_int32)]


class PermutoInputs(C.Structure):
    _fields_ = [("nr_positions", C.c_int64), ("positions", C.c_void_p), ("pos_stride_n", C.c_int64),
                ("pos_stride_d", C.c_int64), ("lattice_values", C.c_void_p), ("scale_factor", C.c_void_p),
                ("random_shift", C.c_void_p), ("anneal_window", C.c_void_p)]


def _load() -> C.CDLL:
    if not os.path.isfile(LIB_PATH):
        raise ImportError(
            f"{LIB_PATH} is missing: the CUDA extension has not been built. Build it with "
            "`python -m permutohedral_encoding_b200.build` (needs nvcc; no GPU required). "
            "There is no CPU fallback.")
    lib = C.CDLL(LIB_PATH)
    lib.permuto_abi_version.restype = C.c_int
    lib.permuto_last_error.restype = C.c_char_p
    lib.permuto_extra_levels.restype = C.c_int
    lib.permuto_extra_levels.argtypes = [C.c_int32, C.c_int32, C.c_int32]
    lib.permuto_scale_factor.restype = C.c_int
    lib.permuto_scale_factor.argtypes = [C.c_void_p, C.c_int32, C.c_int32, C.c_void_p]
    cfgp, inp = C.POINTER(PermutoConfig), C.POINTER(PermutoInputs)
    lib.permuto_forward.restype = C.c_int
    lib.permuto_forward.argtypes = [cfgp, inp, C.c_void_p, C.c_void_p]
    lib.permuto_backward.restype = C.c_int
    lib.permuto_backward.argtypes = [cfgp, inp, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int32, C.c_int32,
                                     C.c_uint32, C.c_void_p]
    lib.permuto_double_backward.restype = C.c_int
    lib.permuto_double_backward.argtypes = [cfgp, inp, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p,
                                            C.c_uint32, C.c_void_p]
    lib.permuto_debug_lattice.restype = C.c_int
    lib.permuto_debug_lattice.argtypes = [cfgp, inp, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p]
    lib.permuto_probe_random_access.restype = C.c_int
    lib.permuto_probe_random_access.argtypes = [C.c_int32, C.c_void_p, C.c_int64, C.c_int32, C.POINTER(C.c_int64),
                                                C.c_void_p]
    lib.permuto_order_pays.restype = C.c_int
    lib.permuto_order_pays.argtypes = [cfgp, C.c_int64, C.c_int32]
    lib.permuto_order_bytes.restype = C.c_int64
    lib.permuto_order_bytes.argtypes = [C.c_int32, C.c_int64]
    lib.permuto_order_record_bytes.restype = C.c_int64
    lib.permuto_order_record_bytes.argtypes = [C.c_int32, C.c_int64]
    lib.permuto_order_scratch_bytes.restype = C.c_int64
    lib.permuto_order_scratch_bytes.argtypes = [C.c_int32, C.c_int64]
    lib.permuto_order_records.restype = C.c_int
    lib.permuto_order_records.argtypes = [cfgp, inp, C.c_void_p, C.c_void_p, C.c_void_p]
    lib.permuto_order_points.restype = C.c_int
    lib.permuto_order_points.argtypes = [cfgp, inp, C.c_void_p, C.c_int64, C.c_void_p]
    lib.permuto_forward_ordered.restype = C.c_int
    lib.permuto_forward_ordered.argtypes = [cfgp, inp, C.c_void_p, C.c_void_p, C.c_void_p]
    lib.permuto_backward_ordered.restype = C.c_int
    lib.permuto_backward_ordered.argtypes = [cfgp, inp, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int32, C.c_int32,
                                             C.c_uint32, C.c_void_p]
    lib.permuto_double_backward_ordered.restype = C.c_int
    lib.permuto_double_backward_ordered.argtypes = [cfgp, inp, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p,
                                                    C.c_uint32, C.c_void_p]
    lib.permuto_forward_mlp_ordered.restype = C.c_int
    lib.permuto_forward_mlp_ordered.argtypes = [cfgp, inp, C.c_void_p, C.POINTER(PermutoMlpLayer), C.c_int32, C.c_int32,
                                                C.c_void_p, C.c_void_p, C.c_void_p]
    lib.permuto_forward_linear.restype = C.c_int
    lib.permuto_forward_linear.argtypes = [cfgp, inp, C.c_void_p, C.c_void_p, C.c_int32, C.c_void_p, C.c_void_p, C.c_void_p]
    lib.permuto_forward_mlp.restype = C.c_int
    lib.permuto_forward_mlp.argtypes = [cfgp, inp, C.POINTER(PermutoMlpLayer), C.c_int32, C.c_int32, C.c_void_p, C.c_void_p,
                                        C.c_void_p]
    lib.permuto_adam_step.restype = C.c_int
    lib.permuto_adam_step.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int64, C.c_double, C.c_double,
                                      C.c_double, C.c_double, C.c_double, C.c_int64, C.c_uint32, C.c_void_p]
    if lib.permuto_abi_version() != ABI_VERSION:
        raise ImportError(f"{LIB_PATH}: ABI version {lib.permuto_abi_version()} != {ABI_VERSION}; rebuild the extension")
    return lib


lib = _load()


def _load_torch_side():
    path = os.path.join(_PKG_DIR, "_permuto_torch.so")
    if not os.path.isfile(path):
        raise ImportError(f"{path} is missing: the PyTorch side of the CUDA extension has not been built. Build it with "
                          "`python -m permutohedral_encoding_b200.build`. There is no Python fallback.")
    from . import _permuto_torch as ext
    ext.bind_api({name: C.cast(getattr(lib, name), C.c_void_p).value for name in EXPORTED_SYMBOLS})
    return ext


_ext = _load_torch_side()
encode = _ext.encode


def last_error() -> str:
    return (lib.permuto_last_error() or b"").decode("utf-8", "replace")


def check(status: int) -> None:
    """Turn a C-ABI status into the exception the reference would have raised (its CHECK
    macros and std::runtime_error both surface as RuntimeError in Python)."""
    if status != PERMUTO_OK:
        raise RuntimeError(last_error() or f"permuto_b200 error {status}")


def scale_factor(sigmas, pos_dim: int) -> np.ndarray:
    s = np.ascontiguousarray(np.asarray(sigmas, dtype=np.float64))
    out = np.empty((s.shape[0], int(pos_dim)), dtype=np.float32)
    check(lib.permuto_scale_factor(s.ctypes.data, s.shape[0], int(pos_dim), out.ctypes.data))
    return out


def extra_levels(pos_dim: int, concat_points: bool, nr_feat_per_level: int = 2) -> int:
    return int(lib.permuto_extra_levels(int(pos_dim), int(nr_feat_per_level), int(bool(concat_points))))


def _ptr(t):
    # plain integers are accepted for the void* parameters (argtypes are declared)
    return None if t is None else t.data_ptr()


def _stream(device):
    """Handle of the current CUDA stream of ``device`` as an integer."""
    return torch.cuda.current_stream(device).cuda_stream


class EncodingInput:
    """Per-call bundle (reference: include/permutohedral_encoding/Encoding.cuh:14-29)."""

    def __init__(self, lattice_values, positions, anneal_window, require_lattice_values_grad,
                 require_positions_grad, lattice_values_half=None):
        self.m_lattice_values = lattice_values
        # optional fp16 copy of the values that the kernels gather from instead (storage only:
        # arithmetic and gradients stay fp32); no counterpart in the reference
        self.m_lattice_values_half = lattice_values_half
        self.m_positions_raw = positions
        self.m_anneal_window = anneal_window
        self.m_require_lattice_values_grad = bool(require_lattice_values_grad)
        self.m_require_positions_grad = bool(require_positions_grad)
        self.m_order = None   # spatial order of these positions (EncodingWrapper.order), or None
        self.m_all_open = True   # no level is closed by the window (decides about ordering, never about results)


class EncodingFixedParams:
    """Fixed description of an encoding (reference: Encoding.cuh:31-70).  Holds the shift
    tensor by handle, so loading a state dict into the module's parameter is seen by the
    kernels; the scale factor is computed once on the host with the reference's rounding and
    cached per device."""

    def __init__(self, pos_dim, capacity, nr_levels, nr_feat_per_level, sigmas_list, random_shift_per_level,
                 concat_points, points_scaling):
        self.m_pos_dim = int(pos_dim)
        self.m_capacity = int(capacity)
        self.m_nr_levels = int(nr_levels)
        self.m_nr_feat_per_level = int(nr_feat_per_level)
        self.m_sigmas_list = [float(s) for s in np.asarray(sigmas_list, dtype=np.float64).reshape(-1)]
        self.m_random_shift_per_level = random_shift_per_level
        self.m_concat_points = bool(concat_points)
        self.m_points_scaling = float(points_scaling)
        if len(self.m_sigmas_list) != self.m_nr_levels:
            raise RuntimeError(f"scale list has {len(self.m_sigmas_list)} entries for {self.m_nr_levels} levels")
        if not (2 <= self.m_pos_dim <= 7):
            raise RuntimeError("Encoding: pos_dim must be 2,3,4,5,6 or 7")
        self.m_scale_factor_host = torch.from_numpy(scale_factor(self.m_sigmas_list, self.m_pos_dim))
        self.levels_per_pass = 0  # scheduling hint of the kernels (0 = automatic; results never depend on it)

    def config(self, table_half: bool = False) -> PermutoConfig:
        return PermutoConfig(self.m_pos_dim, self.m_nr_feat_per_level, self.m_nr_levels, self.m_capacity,
                             int(self.m_concat_points), self.m_points_scaling, int(self.levels_per_pass),
                             PERMUTO_TABLE_F16 if table_half else PERMUTO_TABLE_F32)


class EncodingWrapper:
    """Type-erased encoding (reference: Encoding.cuh:159-188; launchers src/Encoding.cu:54-334)."""

    def __init__(self, pos_dim, nr_feat_per_level, fixed_params: EncodingFixedParams):
        if int(pos_dim) not in (2, 3, 4, 5, 6, 7):
            raise RuntimeError("Encoding: pos_dim must be 2,3,4,5,6 or 7")
        if int(nr_feat_per_level) not in (2, 4, 8):
            raise RuntimeError("Encoding: nr_feat_per_level must be 2, 4 or 8")
        self.fixed = fixed_params
        self._feat = int(nr_feat_per_level)
        self._width = self._feat * (fixed_params.m_nr_levels + extra_levels(
            fixed_params.m_pos_dim, fixed_params.m_concat_points, self._feat))
        self._native = _ext.Lattice(fixed_params.m_pos_dim, self._feat, fixed_params.m_nr_levels, fixed_params.m_capacity,
                                    fixed_params.m_concat_points, fixed_params.m_points_scaling, self._width,
                                    fixed_params.m_scale_factor_host)
        self._backward_hook = None
        self._double_backward_hook = None

    @staticmethod
    def create(pos_dim, nr_feat_per_level, fixed_params) -> "EncodingWrapper":
        return EncodingWrapper(pos_dim, nr_feat_per_level, fixed_params)

    # -- switches ---------------------------------------------------------------------------------
    @property
    def aggregate_collisions(self) -> bool:
        """Merge colliding scatter-adds before the atomics (default)."""
        return self._native.aggregate

    @aggregate_collisions.setter
    def aggregate_collisions(self, value):
        self._native.aggregate = bool(value)

    @property
    def concat_positions_grad(self) -> bool:
        """The reference gives the positions no gradient through the concatenated raw points (its
        backward skips those columns); True adds that term."""
        return self._native.concat_positions_grad

    @concat_positions_grad.setter
    def concat_positions_grad(self, value):
        self._native.concat_positions_grad = bool(value)

    # -- hooks of distributed.LatticeGradAllReduce ----------------------------------------------------
    @property
    def backward_hook(self):
        return self._backward_hook

    @backward_hook.setter
    def backward_hook(self, fn):
        self._backward_hook = fn
        self._install_hooks()

    @property
    def double_backward_hook(self):
        return self._double_backward_hook

    @double_backward_hook.setter
    def double_backward_hook(self, fn):
        self._double_backward_hook = fn
        self._install_hooks()

    def _install_hooks(self):
        ref = weakref.ref(self)   # the native object must not keep its owner alive

        def backward(values, positions, window, half, order, grad, need_values, need_positions):
            me = ref()
            inp = EncodingInput(values, positions, window, need_values, need_positions, half)
            inp.m_order = order
            return me._backward_hook(me, inp, grad)

        self._native.set_hooks(backward if self._backward_hook is not None else None, self._double_backward_hook)

    # -- calls ------------------------------------------------------------------------------------------
    @staticmethod
    def _table(inp: EncodingInput) -> torch.Tensor:
        """The tensor the kernels gather from: the fp16 copy when one is attached."""
        return inp.m_lattice_values_half if inp.m_lattice_values_half is not None else inp.m_lattice_values

    def _args(self, inp: EncodingInput):
        return (self._native, inp.m_lattice_values, inp.m_positions_raw, inp.m_anneal_window,
                self.fixed.m_random_shift_per_level, inp.m_lattice_values_half)

    def output_width(self) -> int:
        return self._width

    def order(self, inp: EncodingInput, purpose: int = ORDER_ALWAYS):
        """Spatial order of the positions (an opaque device buffer), or None where the batch or the number
        of levels is too small for it to pay for ``purpose``: attached to ``inp.m_order`` it makes the operations below
        visit neighbouring points together.  Results do not depend on it.  It holds a copy of the
        coordinates: an order of another number of points or pos_dim is refused, one made before the
        positions were changed gives the results of the old ones."""
        return _ext.order(*self._args(inp), self.fixed.levels_per_pass, purpose)

    def forward(self, inp: EncodingInput) -> torch.Tensor:
        """features [N, 2*(L+extra)] (reference: Encoding<P,2>::forward + modules.py:87)."""
        return _ext.forward(*self._args(inp), inp.m_order, self.fixed.levels_per_pass)

    def forward_linear(self, inp: EncodingInput, weight: torch.Tensor, bias=None, status=None) -> torch.Tensor:
        """``features @ weight.T + bias`` as ``[N, out_features]`` without materialising the features
        (tensor cores, operands rounded to tf32, fp32 accumulation).  ``weight`` is
        ``[out_features, output_width]`` like ``torch.nn.Linear.weight``; ``status`` is an optional
        int32 CUDA tensor of one element that the kernel sets non-zero if its bounded wait for the
        tensor core ran out.  No gradients.  The reference has no counterpart (its users run the
        module followed by ``torch.nn.Linear``: examples/train_toy_example.py:18-26)."""
        return self.forward_mlp(inp, ((weight, bias),), "none", status)

    def forward_mlp(self, inp: EncodingInput, layers, activation: str = "gelu", status=None) -> torch.Tensor:
        """The encoding followed by a whole small MLP in one kernel: ``layers`` is a sequence of
        ``(weight [out, in], bias [out] | None)`` pairs, ``activation`` ("none", "relu", "gelu")
        is applied after every layer but the last.  Neither the features nor the hidden
        activations reach memory; layers whose width is a multiple of 16 run on the tensor cores
        (tf32 operands, fp32 accumulation), a narrower last layer as fp32 dot products.  Hidden
        widths: multiples of 16 up to 64.  No gradients.  The reference's toy example network
        (examples/train_toy_example.py:18-26) is the model case."""
        if activation not in PERMUTO_ACT:
            raise RuntimeError(f"activation must be one of {sorted(PERMUTO_ACT)}, got {activation!r}")
        return _ext.forward_mlp(*self._args(inp), inp.m_order, self.fixed.levels_per_pass, inp.m_all_open,
                                [w for w, _ in layers], [b for _, b in layers], PERMUTO_ACT[activation], status)

    def backward(self, inp: EncodingInput, grad_features: torch.Tensor, lattice_grad_out=None,
                 level_begin=None, level_end=None, zero=True, positions_grad_out=None):
        """(lattice_values_grad [L,C,2] | None, positions_grad [N,d] | None)
        (reference: Encoding<P,2>::backward).  ``lattice_grad_out`` lets the caller provide the
        buffer; ``level_begin/level_end`` restrict the levels (bucketed all-reduce overlap);
        ``positions_grad_out`` is an existing position gradient to keep accumulating into;
        ``zero=False`` accumulates onto a lattice gradient the caller has cleared itself."""
        return _ext.backward(*self._args(inp), inp.m_order, self.fixed.levels_per_pass, grad_features,
                             inp.m_require_lattice_values_grad, inp.m_require_positions_grad, lattice_grad_out,
                             0 if level_begin is None else int(level_begin), -1 if level_end is None else int(level_end),
                             bool(zero), positions_grad_out)

    def double_backward_from_positions(self, inp: EncodingInput, double_positions_grad: torch.Tensor,
                                       grad_features: torch.Tensor, need_lattice_grad=True,
                                       need_grad_grad_features=True):
        """(lattice_values_grad [L,C,2], grad_grad_features [N,W])
        (reference: Encoding<P,2>::double_backward_from_positions)."""
        return _ext.double_backward(*self._args(inp), inp.m_order, self.fixed.levels_per_pass, double_positions_grad,
                                    grad_features, bool(need_lattice_grad), bool(need_grad_grad_features))

    def debug_lattice(self, inp: EncodingInput, want=("keys", "slots", "bary", "rank")):
        """Lattice keys / hash slots / barycentric weights / ranks per (point, level, vertex)."""
        fp = self.fixed
        pos, dev = inp.m_positions_raw, inp.m_positions_raw.device
        _ext.check_inputs(*self._args(inp))
        n, d, nl = pos.shape[0], fp.m_pos_dim, fp.m_nr_levels
        keys = torch.empty((n, nl, d + 1, d), dtype=torch.int32, device=dev) if "keys" in want else None
        slots = torch.empty((n, nl, d + 1), dtype=torch.int32, device=dev) if "slots" in want else None
        bary = torch.empty((n, nl, d + 1), dtype=torch.float32, device=dev) if "bary" in want else None
        rank = torch.empty((n, nl, d + 1), dtype=torch.int32, device=dev) if "rank" in want else None
        table, scale = self._table(inp), self._native.scale_on(dev)
        cfg = fp.config(table.dtype == torch.float16)
        shift, window = (t.detach().to(device=dev, dtype=torch.float32).contiguous()
                         for t in (fp.m_random_shift_per_level, inp.m_anneal_window))
        ins = PermutoInputs(n, pos.data_ptr(), pos.stride(0), pos.stride(1), table.data_ptr(), scale.data_ptr(),
                            shift.data_ptr(), window.data_ptr())
        with torch.cuda.device(dev):
            check(lib.permuto_debug_lattice(C.byref(cfg), C.byref(ins), _ptr(keys), _ptr(slots), _ptr(bary),
                                            _ptr(rank), _stream(dev)))
        return {"keys": keys, "slots": slots, "bary": bary, "rank": rank}
