"""Host-side mirror of the reference's operator API for the splat hot path, over the C ABI of libb2k.so.

Names, argument meaning and error behaviour follow the reference's C++ interface: Model (src/model.h:14-40),
RenderCtx / RenderParams / CameraGPU (src/gpu/render.h:10-95), ViewGPU / LossParams (src/gpu/loss.h:7-30),
OptimParams (src/gpu/optim.h:6-45) and the free functions render_forward, project_splats, bin_and_sort,
rasterize_forward, rasterize_backward, photometric_loss, accumulate_loss, eval_metrics, optimizer_step. Errors raise
RuntimeError, as the reference's CUDA_CHECK / fail() do (src/gpu/util.cuh:13-15).

torch is used only to own device memory and streams; every computation is a kernel of libb2k.so. There is no CPU
path: importing works without a GPU (so the symbol table can be checked), computing without the library or without a
GPU raises.
"""
import ctypes as C
import os
import struct as _st
from operator import attrgetter, itemgetter

import numpy as np
import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, "libb2k.so")

B2K_OK, B2K_ERR_ARG, B2K_ERR_CAPACITY, B2K_ERR_UNSUPPORTED, B2K_ERR_CUDA, B2K_ERR_OVERFLOW = range(6)
GRAD_LANES = 13


class B2kCamera(C.Structure):
    _fields_ = [("R", C.c_float * 9), ("t", C.c_float * 3), ("pos", C.c_float * 3), ("fx", C.c_float), ("fy", C.c_float),
                ("cx", C.c_float), ("cy", C.c_float), ("W", C.c_int32), ("H", C.c_int32), ("lim_pos_x", C.c_float),
                ("lim_pos_y", C.c_float), ("lim_neg_x", C.c_float), ("lim_neg_y", C.c_float)]


_MODEL_PTRS = ["pos_op", "quat", "lscale", "sh_dc", "sh_hi", "m_pos_op", "v_pos_op", "m_quat", "v_quat", "m_lscale", "v_lscale",
               "m_sh_dc", "m_sh_hi", "v_sh", "refine_norm", "max_screen", "vis_count", "vis_weight", "last_step"]


class B2kModel(C.Structure):
    _fields_ = [("n", C.c_int32), ("cap", C.c_int32), ("degree", C.c_int32)] + [(k, C.c_void_p) for k in _MODEL_PTRS]


class B2kCtx(C.Structure):
    _fields_ = [("W", C.c_int32), ("H", C.c_int32), ("tiles_x", C.c_int32), ("tiles_y", C.c_int32), ("n_tiles", C.c_int32),
                ("tile_bits", C.c_int32), ("n_cap", C.c_int32),
                ("proj0", C.c_void_p), ("proj1", C.c_void_p), ("proj2", C.c_void_p), ("tile_count", C.c_void_p), ("hit_info", C.c_void_p),
                ("depth_keys", C.c_void_p), ("depth_keys_sorted", C.c_void_p), ("order_in", C.c_void_p), ("order", C.c_void_p),
                ("tile_off", C.c_void_p), ("keys", C.c_void_p), ("vals", C.c_void_p), ("keys_sorted", C.c_void_p),
                ("vals_sorted", C.c_void_p), ("isect_cap", C.c_uint64), ("num_isect", C.c_void_p), ("sort_tmp", C.c_void_p),
                ("sort_tmp_bytes", C.c_uint64), ("tile_ranges", C.c_void_p), ("out_rgba", C.c_void_p), ("out_feat", C.c_void_p),
                ("out_depth", C.c_void_p), ("last_idx", C.c_void_p), ("v_splat", C.c_void_p), ("vis_flag", C.c_void_p), ("vis_list", C.c_void_p),
                ("v_out", C.c_void_p), ("loss_accum", C.c_void_p), ("n_chunks", C.c_int32), ("proj3", C.c_void_p), ("chunk_words", C.c_void_p),
                ("bwd_scratch", C.c_void_p), ("bwd_scratch_bytes", C.c_uint64)]


class B2kRenderOpts(C.Structure):
    _fields_ = [("bg", C.c_float * 3), ("sh_degree", C.c_int32), ("bwd_info", C.c_int32), ("pos_override", C.c_void_p),
                ("quat_override", C.c_void_p), ("lscale_override", C.c_void_p), ("feat_mode", C.c_int32), ("feat_buffer", C.c_void_p)]


class B2kLoss(C.Structure):
    _fields_ = [("rgba", C.c_void_p), ("weights", C.c_void_p), ("l1_w", C.c_float), ("ssim_w", C.c_float), ("bg", C.c_float * 3),
                ("composite", C.c_int32), ("mask", C.c_int32), ("alpha_lane", C.c_int32), ("match_alpha_weight", C.c_float),
                ("scale", C.c_float), ("grad_scale", C.c_float)]


class B2kOptim(C.Structure):
    _fields_ = [("active_sh_degree", C.c_int32), ("t", C.c_int32), ("beta1", C.c_float), ("beta2", C.c_float), ("eps", C.c_float),
                ("lr_mean", C.c_float), ("lr_rot", C.c_float), ("lr_scale", C.c_float), ("lr_opac", C.c_float), ("lr_dc", C.c_float),
                ("lr_sh_rest", C.c_float), ("noise_weight", C.c_float), ("noise_clamp", C.c_float), ("seed", C.c_uint32),
                ("step", C.c_uint32), ("sparse", C.c_int32), ("pos_override", C.c_void_p), ("quat_override", C.c_void_p),
                ("lscale_override", C.c_void_p), ("grad_out", C.c_void_p), ("touched_out", C.c_void_p)]


# The records above are filled with one native-layout pack each (assigning field by field cost 2 to 7 us a record, as much as
# the launches of a small step; packing takes about a third). Pads follow the C layout; the assertions hold the two together.
_CAMERA_PACK, _OPTS_PACK = _st.Struct("19f2i4f"), _st.Struct("3f2i4x3Pi4xP")
_MODEL_PACK, _LOSS_PACK = _st.Struct("3i4x%dP" % len(_MODEL_PTRS)), _st.Struct("2P5f3i3f4x")
_OPTIM_PACK = _st.Struct("2i11f2Ii5P")
_CTX_PACK = _st.Struct("7i4x14PQ2PQ10Pi4x3PQ")
for _record, _pack in ((B2kCamera, _CAMERA_PACK), (B2kRenderOpts, _OPTS_PACK), (B2kModel, _MODEL_PACK), (B2kLoss, _LOSS_PACK), (B2kOptim, _OPTIM_PACK),
                       (B2kCtx, _CTX_PACK)):
    assert C.sizeof(_record) == _pack.size, _record


def _packed(record, pack, *values):
    """A record from its fields' values in order, arrays entry by entry."""
    try:
        return record.from_buffer_copy(pack.pack(*values))
    except (OverflowError, _st.error):   # what a pack refuses and an assignment takes: a float beyond the range is infinite, an integer wraps around
        s, values = record(), iter(values)
        for name, kind in record._fields_:
            if issubclass(kind, C.Array):
                getattr(s, name)[:] = [next(values) for _ in range(kind._length_)]
            else:
                setattr(s, name, next(values))
        return s


def _first(a, n):
    """The first n entries of a list or an array."""
    a = a.tolist() if hasattr(a, "tolist") else a
    return a if len(a) == n else [a[i] for i in range(n)]


def _floats(a, n=None):
    return [float(x) for x in (a if n is None else _first(a, n))]


def _addr(t):
    return 0 if t is None else t.data_ptr()


# Every entry point include/b2k.h declares, with its argument types (the symbol-table test walks this list).
_P, _S = C.c_void_p, C.c_void_p
SIGNATURES = {
    "b2k_project": (C.c_int, [_P, _P, _P, _P, _S]),
    "b2k_count_tiles": (C.c_int, [_P, C.c_int32, _S]),
    "b2k_bin_sort": (C.c_int, [_P, C.c_int32, _S]),
    "b2k_read_num_isect": (C.c_int, [_P, _S, _P]),
    "b2k_bin_sort_static": (C.c_int, [_P, C.c_int32, _S]),
    "b2k_bin_sort_profile": (C.c_int, [_P, C.c_int32, _S, _P]),
    "b2k_static_max_splats": (C.c_uint32, []),
    "b2k_raster_fwd": (C.c_int, [_P, _P, _S]),
    "b2k_render_chunked": (C.c_int, [_P, _P, _P, _P, _S]),
    "b2k_sort_tmp_bytes": (C.c_uint64, [C.c_int32, C.c_uint64]),
    "b2k_sort_passes": (C.c_int32, [C.c_int32]),
    "b2k_loss_photometric": (C.c_int, [_P, _P, _S]),
    "b2k_loss_accumulate": (C.c_int, [_P, _S]),
    "b2k_loss_zero": (C.c_int, [_P, C.c_int32, C.c_int32, _S]),
    "b2k_loss_fold": (C.c_int, [_P, _P, _S]),
    "b2k_step_begin": (C.c_int, [_P, _S]),
    "b2k_eval_metrics": (C.c_int, [_P, _P, C.c_int32, _S]),
    "b2k_bwd_scratch_bytes": (C.c_uint64, [C.c_int32, C.c_int32, C.c_int32, C.c_uint64]),
    "b2k_raster_bwd": (C.c_int, [_P, _P, _P, _S]),
    "b2k_raster_bwd_scaled": (C.c_int, [_P, _P, _P, C.c_float, _S]),
    "b2k_optim_fused": (C.c_int, [_P, _P, _P, _P, _S]),
    "b2k_proj_bwd": (C.c_int, [_P, _P, _P, _P, _P, _S]),
    "b2k_adam": (C.c_int, [_P, _P, _P, _S]),
    "b2k_adam_range": (C.c_int, [_P, _P, _P, C.c_int32, C.c_int32, _S]),
    "b2k_sort_pairs_tmp_bytes": (C.c_uint64, []),
    "b2k_sort_pairs_u32": (C.c_int, [_P, _P, _P, _P, C.c_uint32, _P, C.c_uint64, _S]),
    "b2k_refine_flags": (C.c_int, [_P, _P, C.c_float, C.c_float, _P, _P, _P, _S]),
    "b2k_refine_sample_keys": (C.c_int, [_P, _P, _P, C.c_int32, C.c_float, C.c_uint32, _P, _P, _P, _S]),
    "b2k_refine_oversized": (C.c_int, [_P, _P, _P, C.c_float, _P, _S]),
    "b2k_refine_mark": (C.c_int, [_P, C.c_int32, _P, _S]),
    "b2k_refine_split": (C.c_int, [_P, _P, _P, _P, C.c_int32, C.c_int32, C.c_float, _P, _S]),
    "b2k_refine_kill": (C.c_int, [_P, _P, C.c_int32, _S]),
    "b2k_refine_opacity_decay": (C.c_int, [_P, C.c_float, _S]),
    "b2k_refine_bake_floor": (C.c_int, [_P, _S]),
    "b2k_refine_axis_keys": (C.c_int, [_P, C.c_int32, _P, _P, _S]),
    "b2k_key_to_float": (C.c_float, [C.c_uint32]),
    "b2k_evidence_view": (C.c_int, [_P, _P, _P, _P, C.c_int32, C.c_float, _P, _S]),
    "b2k_evidence_fold": (C.c_int, [_P, _P, _P, _P, _S]),
    "b2k_label_vote": (C.c_int, [_P, _P, _P, _P, C.c_int32, _P, _S]),
    "b2k_label_bins": (C.c_int32, []),
    "b2k_dp_unique_id": (C.c_int, [_P]),
    "b2k_dp_init": (C.c_int, [_P, _P, C.c_int32, C.c_int32]),
    "b2k_dp_destroy": (C.c_int, [_P]),
    "b2k_dp_allreduce_grads": (C.c_int, [_P, _P, C.c_uint64, _S]),
    "b2k_dp_allreduce_stat": (C.c_int, [_P, _P, C.c_uint64, C.c_int32, _S]),
    "b2k_dp_barrier": (C.c_int, [_P, _S]),
    "b2k_dp_share": (C.c_int, [_P, _P, _P, _S]),
    "b2k_dp_release_shares": (C.c_int, [_P, _S]),
    "b2k_dp_gather_slices": (C.c_int, [_P, _P, C.c_uint64, C.c_int32, C.c_uint64, C.c_int32, _S]),
    "b2k_dp_slice": (C.c_int, [C.c_int32, C.c_int32, C.c_int32, _P, _P]),
    "b2k_dp_adam_shard": (C.c_int, [_P, _P, _P, _P, _S]),
    "b2k_min_scale": (C.c_int, [_P, _P, _P, C.c_int32, _S]),
    "b2k_select_tmp_words": (C.c_uint64, [C.c_int32]),
    "b2k_select_flagged": (C.c_int, [_P, C.c_int32, _P, _P, _P, _S]),
    "b2k_gather_lanes": (C.c_int, [_P, _P, _P, C.c_int32, C.c_int32, C.c_uint64, C.c_int32, _S]),
    "b2k_model_rows": (C.c_int, [_P, C.c_int32, C.c_int32, _P, _P, _P, _P, _S]),
    "b2k_pack_rgba8": (C.c_int, [_P, _P, C.c_int32, C.c_int32, _S]),
    "b2k_quantize_rgba8": (C.c_int, [_P, _P, C.c_int32, _S]),
    "b2k_error_string": (C.c_char_p, [C.c_int]),
    "b2k_last_cuda_error": (C.c_int, []),
    "b2k_launches_repeated": (C.c_uint64, []),
    "b2k_version": (C.c_char_p, []),
}

_lib = None
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def lib():
    """Loads libb2k.so; raises when it has not been built (there is no fallback path)."""
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise RuntimeError(f"{LIB_PATH} is missing: build it with `python -m b2ctrain_b200.build` (no CPU fallback exists)")
        l = C.CDLL(LIB_PATH)
        for name, (res, args) in SIGNATURES.items():
            f = getattr(l, name)
            f.restype, f.argtypes = res, args
        _lib = l
    return _lib


def _check(status, what):
    if status != B2K_OK:
        l = lib()
        msg = l.b2k_error_string(status).decode()
        if status == B2K_ERR_CUDA:
            msg += f" (cudaError {l.b2k_last_cuda_error()})"
        raise RuntimeError(f"{what}: {msg}")


def _stream(stream):
    if stream is None:
        if _raw_stream is not None and torch.cuda.is_initialized():   # a fifth of the time of building a Stream object; eight of them a step
            return _raw_stream(torch._C._cuda_getDevice())
        return C.c_void_p(torch.cuda.current_stream().cuda_stream)
    if isinstance(stream, torch.cuda.Stream):
        return C.c_void_p(stream.cuda_stream)
    return C.c_void_p(int(stream))


def _ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


_CAMERA_HEAD, _CAMERA_SIZE = itemgetter("fx", "fy", "cx", "cy"), itemgetter("W", "H")
_CAMERA_LIMITS = itemgetter("lim_pos_x", "lim_pos_y", "lim_neg_x", "lim_neg_y")


def camera_from(cam):
    """CameraGPU record from a camera dict of b2ctrain_b200.scenes (CameraGPU::from, src/gpu/render.h:15-24)."""
    size = map(int, _CAMERA_SIZE(cam))
    try:
        return B2kCamera.from_buffer_copy(_CAMERA_PACK.pack(*_first(cam["R"], 9), *_first(cam["t"], 3), *_first(cam["pos"], 3), *_CAMERA_HEAD(cam), *size, *_CAMERA_LIMITS(cam)))
    except (OverflowError, _st.error):
        return _packed(B2kCamera, _CAMERA_PACK, *_floats(cam["R"], 9), *_floats(cam["t"], 3), *_floats(cam["pos"], 3), *_floats(_CAMERA_HEAD(cam)), *map(int, _CAMERA_SIZE(cam)),
                       *_floats(_CAMERA_LIMITS(cam)))


def _capacity_for(n):
    cap = 1024
    while cap < n:
        cap *= 2
    return cap


def _fields(obj, names, get):
    """The named attributes of an object, None where it has none (yet)."""
    try:
        return get(obj)
    except AttributeError:
        return [getattr(obj, k, None) for k in names]


_MODEL_GET = attrgetter(*_MODEL_PTRS)


class Model:
    """Device splat model: parameters, Adam moments and refine statistics (src/model.h:14-40). Capacity doubles from
    1024 (src/model.cu:10-11); SH is planar with stride `cap`."""

    def __init__(self, device="cuda:0"):
        self.device = torch.device(device)
        self.n = self.cap = 0
        self.degree = 3
        self.adam_t = 0
        self.sh_fp16 = False

    def K(self):
        return (self.degree + 1) ** 2

    def upload(self, cloud):
        """cloud: host dict(n, degree, pos_op [n][4], quat [n][4], lscale [n][4], sh [n][K][3]) (Model::upload,
        src/model.cu:46-83; unlike the reference the floor lane lscale[:, 3] is taken from the cloud)."""
        if self.sh_fp16:
            raise RuntimeError("Model.upload: fp16 SH storage is not implemented (unsupported lane)")
        self.n, self.degree = int(cloud["n"]), int(cloud["degree"])
        self.cap = _capacity_for(self.n)
        K, cap, dev = self.K(), self.cap, self.device
        f32 = dict(dtype=torch.float32, device=dev)

        def up4(a):
            t = torch.zeros((cap, 4), **f32)
            t[: self.n] = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(dev)
            return t

        self.pos_op, self.quat, self.lscale = up4(cloud["pos_op"]), up4(cloud["quat"]), up4(cloud["lscale"])
        sh = torch.from_numpy(np.ascontiguousarray(cloud["sh"], dtype=np.float32)).to(dev).reshape(self.n, K * 3)
        planar = torch.zeros((K * 3, cap), **f32)
        planar[:, : self.n] = sh.t()
        self.sh_dc = planar[:3].contiguous()
        self.sh_hi = planar[3:].contiguous() if K > 1 else torch.zeros((0, cap), **f32)
        self.zero_optimizer()
        self.zero_stats()
        return self

    def zero_optimizer(self):
        z = lambda *s: torch.zeros(s, dtype=torch.float32, device=self.device)
        cap, K = self.cap, self.K()
        self.m_pos_op, self.v_pos_op, self.m_quat, self.v_quat, self.m_lscale, self.v_lscale = (z(cap, 4) for _ in range(6))
        self.m_sh_dc, self.m_sh_hi, self.v_sh = z(3, cap), z(3 * (K - 1), cap), z(cap)
        self.last_step = torch.zeros(cap, dtype=torch.int32, device=self.device)
        self.adam_t = 0

    def zero_stats(self):
        z = lambda: torch.zeros(self.cap, dtype=torch.float32, device=self.device)
        self.refine_norm, self.max_screen, self.vis_count, self.vis_weight = z(), z(), z(), z()

    def download(self):
        n, K = self.n, self.K()
        planar = torch.cat([self.sh_dc, self.sh_hi], 0)[:, :n]
        return dict(n=n, degree=self.degree, pos_op=self.pos_op[:n].cpu().numpy(), quat=self.quat[:n].cpu().numpy(),
                    lscale=self.lscale[:n].cpu().numpy(), sh=planar.t().reshape(n, K, 3).contiguous().cpu().numpy())

    def compact(self, keep, extras=(), stream=None):
        """Model::compact (src/model.cu:120-155): keeps the splats whose flag in `keep` (device int32 [n]) is non-zero,
        in their order, across parameters, moments, statistics and the caller's extra per-splat float tensors (each
        [cap], replaced in the returned list). Returns (new n, extras). Synchronises for the count, like the reference."""
        if self.n == 0:
            return 0, list(extras)
        n, cap, dev = self.n, self.cap, self.device
        idx = torch.zeros(n, dtype=torch.int32, device=dev)
        cnt = torch.zeros(1, dtype=torch.int32, device=dev)
        tmp = torch.zeros(int(lib().b2k_select_tmp_words(n)), dtype=torch.int32, device=dev)
        _check(lib().b2k_select_flagged(_ptr(keep), n, _ptr(idx), _ptr(cnt), _ptr(tmp), _stream(stream)), "Model.compact")
        kept = int(cnt.item())
        if kept == n:
            return n, list(extras)

        def gather(t, lanes, elem_bytes):
            if t is None or t.numel() == 0 or lanes == 0:
                return t
            fresh = torch.zeros_like(t)   # an in-place gather would race
            _check(lib().b2k_gather_lanes(_ptr(t), _ptr(fresh), _ptr(idx), kept, lanes, cap, elem_bytes, _stream(stream)), "Model.compact")
            return fresh

        hi_lanes = 3 * (self.K() - 1)
        for k in ("pos_op", "quat", "lscale", "m_pos_op", "v_pos_op", "m_quat", "v_quat", "m_lscale", "v_lscale"):
            setattr(self, k, gather(getattr(self, k), 1, 16))
        for k, lanes in (("sh_dc", 3), ("sh_hi", hi_lanes), ("m_sh_dc", 3), ("m_sh_hi", hi_lanes), ("v_sh", 1), ("refine_norm", 1),
                         ("max_screen", 1), ("vis_count", 1), ("vis_weight", 1), ("last_step", 1)):
            setattr(self, k, gather(getattr(self, k), lanes, 4))
        out = [gather(e, 1, 4) for e in extras]
        self.n = kept
        return kept, out

    def sh_planar_to_host(self, dc, hi):
        n, K = self.n, self.K()
        return torch.cat([dc, hi], 0)[:, :n].t().reshape(n, K, 3).contiguous().cpu().numpy()

    def struct(self):
        return _packed(B2kModel, _MODEL_PACK, self.n, self.cap, self.degree, *map(_addr, _fields(self, _MODEL_PTRS, _MODEL_GET)))


# The pointers of a context in the order of its record (num_isect, which is d_num_isect here, goes between vals_sorted and sort_tmp).
_CTX_PTRS = ("proj0", "proj1", "proj2", "tile_count", "hit_info", "depth_keys", "depth_keys_sorted", "order_in", "order", "tile_off", "keys", "vals",
             "keys_sorted", "vals_sorted", "sort_tmp", "tile_ranges", "out_rgba", "out_feat", "out_depth", "last_idx", "v_splat", "vis_flag", "vis_list",
             "v_out", "loss_accum", "proj3", "chunk_words", "bwd_scratch")
_CTX_GET = attrgetter(*_CTX_PTRS)


class RenderCtx:
    """Per-view scratch (src/gpu/render.h:66-95); member names follow the reference. `setup` sizes everything; the
    intersection buffers start at 2^22 entries (src/gpu/render.cu:20) and double on overflow."""

    def __init__(self, device="cuda:0"):
        self.device = torch.device(device)
        self.W = self.H = self.tiles_x = self.tiles_y = self.n_tiles = self.tile_bits = 0
        self.n_cap = 0
        self.isect_cap = 0
        self.num_isect = 0
        self.want_depth = False
        self.n_chunks = 1          # > 1: render_forward composites the view front to back in this many depth chunks
        self.chunk_words = None

    def setup(self, W, H, n_splats, stream=None, isect_cap=None, n_chunks=None):
        if n_chunks is not None:
            self.n_chunks = max(1, int(n_chunks))
        dev = self.device
        self.W, self.H = int(W), int(H)
        self.tiles_x, self.tiles_y = (self.W + 7) // 8, (self.H + 7) // 8
        self.n_tiles = self.tiles_x * self.tiles_y
        self.tile_bits = 1
        while (1 << self.tile_bits) < self.n_tiles + 1:
            self.tile_bits += 1
        n = max(int(n_splats), 1)
        u32 = lambda *s: torch.zeros(s, dtype=torch.int32, device=dev)
        f32 = lambda *s: torch.zeros(s, dtype=torch.float32, device=dev)
        if n > self.n_cap:
            self.proj0, self.proj1, self.proj2 = f32(n, 4), f32(n, 4), f32(n, 4)
            self.proj3 = f32(n, 2)
            self.tile_count, self.tile_off = u32(n), u32(n)
            self.hit_info = u32(n, 4)
            self.depth_keys, self.depth_keys_sorted, self.order_in, self.order = u32(n), u32(n), u32(n), u32(n)
            self.v_splat, self.vis_flag = f32(n, GRAD_LANES), u32(n)
            self.vis_list = u32(n)
            self.n_cap = n
        P = self.W * self.H
        self.tile_ranges = u32(self.n_chunks * self.n_tiles, 2)
        self.chunk_words = u32(32 + self.n_tiles + (self.tiles_x + 1) * (self.tiles_y + 1)) if self.n_chunks > 1 else None
        self.out_rgba, self.out_feat, self.v_out = f32(P, 4), f32(P, 4), f32(P, 4)
        self.out_depth = f32(P) if self.want_depth else None
        self.last_idx = u32(P)
        self.loss_accum = f32(16)
        self.d_num_isect = u32(4)
        if self.isect_cap == 0 or (isect_cap and isect_cap > self.isect_cap):
            self._alloc_isect(isect_cap or (1 << 22))
        else:
            self._alloc_isect(self.isect_cap)   # the backward scratch depends on the image size and the chunk count
        nbytes = int(lib().b2k_sort_tmp_bytes(self.n_cap, self.isect_cap))
        self.sort_tmp = torch.zeros(nbytes, dtype=torch.uint8, device=dev)
        return self

    def _alloc_isect(self, cap):
        u32 = lambda: torch.zeros(cap, dtype=torch.int32, device=self.device)
        self.keys, self.vals, self.keys_sorted, self.vals_sorted = u32(), u32(), u32(), u32()
        self.isect_cap = int(cap)
        # checkpoints and work list of the segmented backward: sized from the intersection capacity
        self.bwd_scratch = torch.zeros(int(lib().b2k_bwd_scratch_bytes(self.W, self.H, self.n_chunks, self.isect_cap)), dtype=torch.uint8,
                                       device=self.device)

    def struct(self):
        """The context's record, from the tensors as they are now: one may have been given other storage in place."""
        p = [0 if t is None else t.data_ptr() for t in _fields(self, _CTX_PTRS, _CTX_GET)]
        return _packed(B2kCtx, _CTX_PACK, self.W, self.H, self.tiles_x, self.tiles_y, self.n_tiles, self.tile_bits, self.n_cap, *p[:14], self.isect_cap,
                       self.d_num_isect.data_ptr(), p[14], self.sort_tmp.numel(), *p[15:25], self.n_chunks, *p[25:], self.bwd_scratch.numel())


class RenderParams:
    """RenderParams (src/gpu/render.h:29-63). Lanes this library does not implement raise when set. feat: "None",
    "Normals" or "Buffer" (FeatureMode, render.h:27; forward only); feat_buffer: [n][3] device tensor for "Buffer"."""
    _UNSUPPORTED = ("warp", "sh_frame", "app", "col_base", "hollow_z")
    _FEAT = {"None": 0, "Normals": 1, "Buffer": 2}

    def __init__(self, cam, bg=(0.0, 0.0, 0.0), sh_degree=3, bwd_info=True):
        self.cam, self.bg, self.sh_degree, self.bwd_info = cam, tuple(bg), sh_degree, bwd_info
        self.feat = "None"
        self.feat_buffer = None
        self.mip = False
        self.pos_override = self.quat_override = self.lscale_override = None
        for k in self._UNSUPPORTED:
            setattr(self, k, None)

    def struct(self):
        if self.mip or any(getattr(self, k) is not None for k in self._UNSUPPORTED):
            raise RuntimeError("RenderParams: mip / warp / sh_frame / app / hollow lanes are not implemented (unsupported lane)")
        if self.feat not in self._FEAT or (self.feat == "Buffer") != (self.feat_buffer is not None):
            raise RuntimeError("RenderParams: feat is None, Normals or Buffer, and feat_buffer goes with Buffer")
        return _packed(B2kRenderOpts, _OPTS_PACK, *_floats(self.bg, 3), int(self.sh_degree), int(bool(self.bwd_info)), _addr(self.pos_override),
                       _addr(self.quat_override), _addr(self.lscale_override), self._FEAT[self.feat], _addr(self.feat_buffer))

    def camera(self):
        return self.cam if isinstance(self.cam, B2kCamera) else camera_from(self.cam)


class ViewGPU:
    """A training view resident on the GPU (src/gpu/loss.h:7-18): packed RGBA8 target and optional u8 weights."""

    def __init__(self, rgba, weights=None, W=0, H=0):
        self.rgba, self.weights, self.W, self.H = rgba, weights, W, H
        self.normals = None


class LossParams:
    """LossParams (src/gpu/loss.h:20-30)."""

    def __init__(self, **kw):
        self.l1_w, self.ssim_w = 0.8, -0.2
        self.bg = (0.0, 0.0, 0.0)
        self.composite = self.mask = self.alpha_lane = False
        self.match_alpha_weight, self.scale, self.normal_scale, self.grad_scale = 0.1, 1.0, 0.0, 1.0
        for k, v in kw.items():
            if not hasattr(self, k):
                raise TypeError(k)
            setattr(self, k, v)

    def struct(self, view):
        if self.normal_scale != 0.0:
            raise RuntimeError("LossParams: the normal-supervision lane is not implemented (unsupported lane)")
        return _packed(B2kLoss, _LOSS_PACK, _addr(view.rgba), _addr(view.weights), self.l1_w, self.ssim_w, *_floats(self.bg, 3), int(self.composite), int(self.mask),
                       int(self.alpha_lane), self.match_alpha_weight, self.scale, self.grad_scale)


class OptimParams:
    """OptimParams (src/gpu/optim.h:6-45), defaults included."""
    _UNSUPPORTED = ("g_pos_out", "sh_frame", "update_mask", "canon_rot", "spa_z", "stretch_w", "g_app_out")

    def __init__(self, cam, **kw):
        self.cam = cam
        self.mip = False
        self.active_sh_degree = 3
        self.t = 1
        self.beta1, self.beta2, self.eps = 0.9, 0.999, 1e-15
        self.lr_mean = 0.0
        self.lr_rot, self.lr_scale, self.lr_opac, self.lr_dc, self.lr_sh_rest = 2e-3, 5e-3, 0.012, 2e-3, 2e-4
        self.noise_weight = self.noise_clamp = 0.0
        self.seed, self.step = 42, 0
        self.pos_override = self.quat_override = self.lscale_override = None
        self.frozen = False
        self.sparse = False
        self.grad_out = None
        self.touched_out = None   # bitmap of (n + 31) // 32 words: projection_backward marks the splats it adds a row for
        for k in self._UNSUPPORTED:
            setattr(self, k, None)
        for k, v in kw.items():
            if not hasattr(self, k):
                raise TypeError(k)
            setattr(self, k, v)

    def struct(self):
        if self.mip or self.frozen or any(getattr(self, k) is not None for k in self._UNSUPPORTED):
            raise RuntimeError("OptimParams: cage / deformation / sparsification lanes are not implemented (unsupported lane)")
        return _packed(B2kOptim, _OPTIM_PACK, self.active_sh_degree, self.t, self.beta1, self.beta2, self.eps, self.lr_mean, self.lr_rot, self.lr_scale, self.lr_opac,
                       self.lr_dc, self.lr_sh_rest, self.noise_weight, self.noise_clamp, self.seed, self.step, int(bool(self.sparse)), _addr(self.pos_override),
                       _addr(self.quat_override), _addr(self.lscale_override), _addr(self.grad_out), _addr(self.touched_out))

    def camera(self):
        return self.cam if isinstance(self.cam, B2kCamera) else camera_from(self.cam)


# ---- operators (src/gpu/render.h:97-109, src/gpu/loss.h:32-41, src/gpu/optim.h:50) ----

def project_splats(ctx, m, p, stream=None):
    ms, cs, os_, cam = m.struct(), ctx.struct(), p.struct(), p.camera()
    _check(lib().b2k_project(C.byref(ms), C.byref(cam), C.byref(os_), C.byref(cs), _stream(stream)), "project_splats")


def count_tiles(ctx, m, stream=None):
    """Tile counts, hit masks and depth keys from the records already in ctx.proj0 / ctx.proj1."""
    cs = ctx.struct()
    _check(lib().b2k_count_tiles(C.byref(cs), m.n, _stream(stream)), "count_tiles")


def bin_and_sort(ctx, m, stream=None, sync=True):
    """With sync=True behaves like the reference (binning.cu:125-133): reads the intersection total back, and when it
    exceeds the buffers grows them by doubling and redoes the binning. sync=False leaves the total on the device."""
    _bin_and_sort(ctx, m, ctx.struct(), _stream(stream), sync)


def _bin_and_sort(ctx, m, cs, stream, sync):
    """bin_and_sort over the context's record; returns the record, which is another one when the buffers grew."""
    _check(lib().b2k_bin_sort(C.byref(cs), m.n, stream), "bin_and_sort")
    if not sync:
        return cs
    total = C.c_uint32(0)
    st = lib().b2k_read_num_isect(C.byref(cs), stream, C.byref(total))
    if st == B2K_ERR_OVERFLOW:
        cap = ctx.isect_cap
        while cap < total.value:
            cap *= 2
        ctx._alloc_isect(cap)
        cs = ctx.struct()
        _check(lib().b2k_bin_sort(C.byref(cs), m.n, stream), "bin_and_sort")
        st = lib().b2k_read_num_isect(C.byref(cs), stream, C.byref(total))
    _check(st, "bin_and_sort")
    ctx.num_isect = int(total.value)
    return cs


def bin_and_sort_profile(ctx, m, stream=None):
    """bin_and_sort timed phase by phase with CUDA events inside the library; returns the ten durations in ms (see
    b2k_bin_sort_profile in include/b2k.h). Synchronises."""
    cs = ctx.struct()
    ms = (C.c_float * 10)()
    _check(lib().b2k_bin_sort_profile(C.byref(cs), m.n, _stream(stream), ms), "bin_and_sort_profile")
    return list(ms)


def rasterize_forward(ctx, p, stream=None):
    cs, os_ = ctx.struct(), p.struct()
    _check(lib().b2k_raster_fwd(C.byref(cs), C.byref(os_), _stream(stream)), "rasterize_forward")


def render_forward(ctx, m, p, stream=None, sync=True):
    """render_forward (src/gpu/render.h:97). A context set up with n_chunks > 1 renders front to back in depth chunks
    (b2k_render_chunked: same image and gradients, intersections behind saturated pixels never sorted)."""
    if ctx.n_chunks > 1:
        return render_chunked(ctx, m, p, stream, sync=sync)
    cs, ms, os_, cam, st = ctx.struct(), m.struct(), p.struct(), p.camera(), _stream(stream)
    _check(lib().b2k_project(C.byref(ms), C.byref(cam), C.byref(os_), C.byref(cs), st), "project_splats")
    cs = _bin_and_sort(ctx, m, cs, st, sync)
    _check(lib().b2k_raster_fwd(C.byref(cs), C.byref(os_), st), "rasterize_forward")


def forward_fits(ctx, stream=None):
    """Waits for a render_forward(sync=False) and says whether its intersections fitted the context's buffers."""
    cs, total = ctx.struct(), C.c_uint32(0)
    st = lib().b2k_read_num_isect(C.byref(cs), _stream(stream), C.byref(total))
    ctx.num_isect = int(total.value)
    if st != B2K_ERR_OVERFLOW:
        _check(st, "forward_fits")
    return st != B2K_ERR_OVERFLOW


def render_chunked(ctx, m, p, stream=None, sync=True):
    """b2k_render_chunked; with sync the slot count is read back and the view redone with larger buffers on overflow."""
    while True:
        cs, ms, os_, cam = ctx.struct(), m.struct(), p.struct(), p.camera()
        _check(lib().b2k_render_chunked(C.byref(ms), C.byref(cam), C.byref(os_), C.byref(cs), _stream(stream)), "render_chunked")
        if not sync:
            return None
        total = C.c_uint32(0)
        st = lib().b2k_read_num_isect(C.byref(cs), _stream(stream), C.byref(total))
        ctx.num_isect = int(total.value)
        if st == B2K_ERR_OVERFLOW:
            cap = ctx.isect_cap
            while cap < ctx.num_isect + 32 * ctx.n_chunks:
                cap *= 2
            ctx._alloc_isect(cap)
            continue
        _check(st, "render_chunked")
        return ctx.num_isect


# Records of the calls that read a few fields only, with those fields: a whole one takes about 4 us of the host's time, and
# the launches of a small step leave it little more than a step's GPU time (64x64 step: host 106 us with whole records, 93 so).
def _loss_record(ctx):
    s = B2kCtx()
    s.loss_accum, s.num_isect = _addr(ctx.loss_accum), _addr(ctx.d_num_isect)
    return s


def _image_record(ctx):
    s = B2kCtx()
    s.W, s.H, s.out_rgba, s.v_out, s.loss_accum = ctx.W, ctx.H, _addr(ctx.out_rgba), _addr(ctx.v_out), _addr(ctx.loss_accum)
    return s


def photometric_loss(ctx, view, lp, stream=None):
    cs, ls = _image_record(ctx), lp.struct(view)
    _check(lib().b2k_loss_photometric(C.byref(cs), C.byref(ls), _stream(stream)), "photometric_loss")


def accumulate_loss(ctx, stream=None):
    cs = _loss_record(ctx)
    _check(lib().b2k_loss_accumulate(C.byref(cs), _stream(stream)), "accumulate_loss")


def zero_loss(ctx, first=0, count=16, stream=None):
    """loss_accum[first : first + count] = 0 on the stream."""
    cs = _loss_record(ctx)
    _check(lib().b2k_loss_zero(C.byref(cs), int(first), int(count), _stream(stream)), "zero_loss")


def step_begin(ctx, stream=None):
    """Clears the context's loss accumulator and its running intersection maximum (start of a training step)."""
    cs = _loss_record(ctx)
    _check(lib().b2k_step_begin(C.byref(cs), _stream(stream)), "step_begin")


def fold_loss(dst_ctx, src_ctx, stream=None):
    """Adds the running loss sum and view count of src_ctx into dst_ctx's."""
    a, b = _loss_record(dst_ctx), _loss_record(src_ctx)
    _check(lib().b2k_loss_fold(C.byref(a), C.byref(b), _stream(stream)), "fold_loss")


def eval_metrics(ctx, view, mask_weighted=False, stream=None):
    cs = _image_record(ctx)
    _check(lib().b2k_eval_metrics(C.byref(cs), _ptr(view.rgba), int(mask_weighted), _stream(stream)), "eval_metrics")


def _weight_record(m):
    s = B2kModel()
    s.n, s.cap, s.degree, s.vis_weight = m.n, m.cap, m.degree, _addr(getattr(m, "vis_weight", None))
    return s


def rasterize_backward(ctx, m, p, stream=None):
    cs, ms, os_ = ctx.struct(), _weight_record(m), p.struct()
    _check(lib().b2k_raster_bwd(C.byref(cs), C.byref(ms), C.byref(os_), _stream(stream)), "rasterize_backward")


def rasterize_backward_tc(ctx, m, p, grad_scale, stream=None):
    """rasterize_backward_tc (src/gpu/render.h:107-109): v_out carries grad_scale, the per-splat lanes leave divided by it."""
    cs, ms, os_ = ctx.struct(), _weight_record(m), p.struct()
    _check(lib().b2k_raster_bwd_scaled(C.byref(cs), C.byref(ms), C.byref(os_), C.c_float(grad_scale), _stream(stream)), "rasterize_backward_tc")


def _lanes_record(ctx):
    s = B2kCtx()
    s.n_cap, s.isect_cap, s.num_isect = ctx.n_cap, ctx.isect_cap, _addr(ctx.d_num_isect)
    s.v_splat, s.vis_flag, s.tile_count, s.vis_list = _addr(ctx.v_splat), _addr(ctx.vis_flag), _addr(ctx.tile_count), _addr(getattr(ctx, "vis_list", None))
    return s


def optimizer_step(ctx, m, op, stream=None):
    cs, ms, os_, cam = _lanes_record(ctx), m.struct(), op.struct(), op.camera()
    _check(lib().b2k_optim_fused(C.byref(cs), C.byref(ms), C.byref(cam), C.byref(os_), _stream(stream)), "optimizer_step")


# ---- data-parallel split of optimizer_step ----

def projection_backward(ctx, m, op, grad, stream=None):
    cs, ms, os_, cam = _lanes_record(ctx), m.struct(), op.struct(), op.camera()
    _check(lib().b2k_proj_bwd(C.byref(cs), C.byref(ms), C.byref(cam), C.byref(os_), _ptr(grad), _stream(stream)), "projection_backward")


def adam_step(m, op, grad, stream=None, first=0, count=None):
    """The update half of the data-parallel split from the accumulator grad[n][11+3K]; first/count restrict it to a
    slice of splats (first a multiple of 4)."""
    ms, os_ = m.struct(), op.struct()
    if first == 0 and count is None:
        _check(lib().b2k_adam(C.byref(ms), C.byref(os_), _ptr(grad), _stream(stream)), "adam_step")
    else:
        count = m.n - first if count is None else count
        _check(lib().b2k_adam_range(C.byref(ms), C.byref(os_), _ptr(grad), int(first), int(count), _stream(stream)), "adam_step")


def update_min_scale(m, cam_pos, cam_focal, stream=None):
    """RefineState::update_min_scale (src/gpu/refine.cu:166-170): cam_pos [c][3], cam_focal [c] device tensors."""
    ms = m.struct()
    _check(lib().b2k_min_scale(C.byref(ms), _ptr(cam_pos), _ptr(cam_focal), int(cam_focal.numel()), _stream(stream)), "update_min_scale")


def pack_rgba8(rgba, out, alpha_override=-1, stream=None):
    _check(lib().b2k_pack_rgba8(_ptr(rgba), _ptr(out), int(out.numel()), int(alpha_override), _stream(stream)), "pack_rgba8")
