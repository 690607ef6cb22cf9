"""Bindings of the raw-GGUF-block kernels: linear layers, router top-k, route grouping and
the routed-expert pass. Weights are uint8 tensors holding the file's blocks unchanged."""
from __future__ import annotations

from ctypes import c_float, c_int, c_void_p

import torch

from . import _check, _ptr, _sm_count, _stream
from . import lib as _lib

# device type ids (reference: src/loader/gguf/quant_types.py, plus q8_0 and bf16)
DEVICE_TYPE = {"iq2_xxs": 0, "q2_k": 1, "iq1_m": 2, "q4_k": 3, "q5_k": 4, "iq2_xs": 5, "iq3_xxs": 6, "iq4_xs": 7, "mxfp4": 11,
               "q6_k": 8, "q8_0": 9, "bf16": 10}
SCORE_FUNCS = {"softmax": 0, "sigmoid": 1, "sqrtsoftplus": 2}


def row_bytes(type_name: str, K: int) -> int:
    return K // 256 * _lib.kernels().pk_gguf_block_bytes(DEVICE_TYPE[type_name])


def gguf_linear(x: torch.Tensor, w_raw: torch.Tensor, type_name: str, N: int, *, gamma: torch.Tensor | None = None,
                eps: float = 1e-6, epi: int = 0, status: torch.Tensor | None = None) -> torch.Tensor:
    """y = rmsnorm?(x) @ dequant(W)^T for any number of rows.

    `status` (int32 [1], here and in the expert functions): the first bounded wait that ran out is recorded there. A product of
    `UMMA_TYPES` whose wait ran out gives NaN, and so does one that finds the word set; its owner reads the word once per step
    (`StepWord`) and clears it.

    Up to `UMMA_MAX_ROWS - 1` rows (of more than 2^24 weights `UMMA_MAX_ROWS_LARGE - 1`) of the types in `UMMA_TYPES` are decoded inside a
    tensor-core kernel, once per 64 rows.
    Of the other types, up to `TENSOR_CORE_MIN_ROWS - 1` rows decode the blocks in registers (groups of up to 8 rows per
    launch). Above, the weight is decoded once into a bf16 scratch and the product runs on the tcgen05 GEMM (the
    reference switches to its prefill kernels for rows > 1, src/components/gguf/quantized_ops.py:9-76)."""
    M, K = x.shape
    ncols = N // 2 if epi == 1 else N
    most = UMMA_MAX_ROWS if N * K <= 1 << 24 else UMMA_MAX_ROWS_LARGE
    if 0 < M < most and K * 4 <= 200 * 1024 and _umma_takes(w_raw, type_name, N, K) and not _registers_faster(type_name, M, N * K):
        return _umma_linear(_aligned(x), w_raw, type_name, N, _aligned(gamma), eps, epi, status)
    if M >= TENSOR_CORE_MIN_ROWS and K % 64 == 0 and (epi != 1 or (N // 2) % 128 == 0):
        from . import gemm_bf16, rmsnorm, EPI_BF16, EPI_SWIGLU, EPI_F32
        w = _dequant_scratch(w_raw, type_name, N, K)
        xin = x.contiguous() if gamma is None else rmsnorm(x.contiguous(), gamma, mode=2, eps=eps)
        return gemm_bf16(xin, w, epi={0: EPI_BF16, 1: EPI_SWIGLU, 2: EPI_F32}[epi], status=status)
    y = torch.empty(M, ncols, device=x.device, dtype=torch.float32 if epi == 2 else torch.bfloat16)
    step = max(1, min(8, (184 * 1024) // (K * 4)))
    step = 8 if step >= 8 else 4 if step >= 4 else 2 if step >= 2 else 1
    for m0 in range(0, M, step):
        m = min(step, M - m0)
        st = _lib.kernels().pk_gguf_linear(_ptr(w_raw), c_int(DEVICE_TYPE[type_name]), c_int(N), c_int(K), c_int(m),
                                           _ptr(x[m0:]), _ptr(gamma), c_float(eps), c_int(epi), _ptr(y[m0:]), c_int(ncols),
                                           c_int(_sm_count()), _stream())
        _check(st, "pk_gguf_linear")
    return y


# Block types whose integer part fits fp16: decoded inside the tensor-core kernel (`csrc/kernels/quant_umma.cu`)
UMMA_TYPES = frozenset({"iq2_xxs", "q4_k", "q5_k"})
# Against decoding per eight rows or (from 32 rows) to a bf16 scratch, 4096 x 4096 / 8192 x 3072 / 24576 x 6144, us: IQ2_XXS, 256 rows
# 28 / 36 / 187 against 47 / 58 / 244, 384 rows 45 / 54 / 242 against 47 / 60 / 288, 512 rows 48 / 72 / 310 against 50 / 66 / 285; Q4_K, 384 rows
# 44 / 57 / 226 against 51 / 65 / 308; Q5_K, 256 rows 30 / 45 / 220 against 54 / 73 / 297, 384 rows 58 / 70 / 280 against 54 / 81 / 339, 512 rows
# 63 / 90 / 365 against 61 / 78 / 337. Up to 2^24 weights the line stays at 256 rows, from when the kernel was slower: with 257 to 384 rows it takes 0.32 to 0.93 of
# the scratch's time at 4096 x 4096, 8192 x 2048, 2048 x 8192 and 1024 x 16384.
UMMA_MAX_ROWS, UMMA_MAX_ROWS_LARGE = 257, 385
UMMA_SPLIT_ROUTES = 64
UMMA_MAX_GROUPS = 512


def _umma_takes(w_raw: torch.Tensor, type_name: str, rows: int, K: int, groups: int = 1) -> bool:
    """Whether the kernel takes `groups` groups of `rows` rows, which may be the beginning of a longer buffer."""
    if type_name not in UMMA_TYPES or w_raw.data_ptr() % 16 != 0 or K % 256 != 0:
        return False
    n = rows * row_bytes(type_name, K)
    return n % 4 == 0 and n < 1 << 32 and w_raw.numel() >= n * groups       # whole words: IQ2 blocks are copied by four bytes


def _registers_faster(type_name: str, rows: int, weights: int) -> bool:
    """Few rows of a small weight decode faster in registers: one launch there, two and a pipeline to fill here (12 us at least), against
    a multiply-add per weight and row. Weights from memory, us: one row of 2048 x 2048 / 4096 x 4096 / 8192 x 3072, IQ2_XXS 6.5 against
    13.3, 14.2 / 15.9, 20.4 / 16.9; Q4_K 7.9 / 11.9, 17.4 / 15.0, 23.5 / 16.3; Q5_K 8.8 / 12.8, 21.2 / 16.6, 27.4 / 17.9. Four rows of
    2048 x 2048: 12.3 / 13.6, 13.2 / 12.1, 14.1 / 12.5; eight 19.9 / 13.5, 20.1 / 12.3, 21.1 / 12.9. Lines at half these
    sizes would be up to 3 us faster (one row of 8192 x 3072 in IQ2_XXS); they stay, since the two forms add in other orders, and a row's bits
    would change with the line."""
    if rows > 8:
        return False
    width = 1 << (rows - 1).bit_length()        # the kernels have one, two, four or eight rows
    return width * weights <= (1 << 25 if type_name == "iq2_xxs" and rows <= 2 else 1 << 24)


class StepWord:
    """A step's token and the error word of its products in one device buffer, so that one copy reads both."""

    def __init__(self, device):
        self.buf = torch.zeros(2, dtype=torch.int64, device=device)
        self.status = self.buf.view(torch.int32)[2:3]

    def pick(self, logits: torch.Tensor) -> None:
        """The greedy token of `logits` [vocab] goes into the buffer."""
        torch.argmax(logits, dim=0, out=self.buf[0])

    def read(self) -> tuple[int, int]:
        """(token, error word); the word is cleared when it was set."""
        token, failed = self.buf.tolist()
        if failed:
            self.status.zero_()
        return token, failed


def _aligned(t: torch.Tensor | None) -> torch.Tensor | None:
    """`t` itself, or a copy that begins on 16 bytes and has its rows one after the other."""
    if t is None:
        return None
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


class _Staged:
    """Token rows for the tensor-core kernel and the work space of one product, in one allocation."""

    def __init__(self, x: torch.Tensor, type_name: str, rows: int, terms: int, *, index=None, gamma=None, eps: float = 0.0, counters: int = 0,
                 ws_floats: int = 0):
        K = x.shape[1]
        pitch = _lib.kernels().pk_quant_stage_pitch(c_int(DEVICE_TYPE[type_name]), c_int(K))
        counters += 1       # the last one: the product's error word where the caller has none
        sizes = (rows * terms * pitch * 2, rows * 4, counters * 4, ws_floats * 4)
        offs, at = [], 0
        for n in sizes:
            offs.append(at)
            at += -(-n // 256) * 256
        self.buf = torch.empty(at, device=x.device, dtype=torch.uint8)
        self.rows, self.terms = rows, terms
        p = self.buf.data_ptr()
        self.data, self.scale, self.counters, self.ws = (c_void_p(p + o) for o in offs)
        self.status = c_void_p(p + offs[2] + 4 * counters - 4)
        _check(_lib.kernels().pk_quant_stage_rows(_ptr(x), c_int(int(x.dtype == torch.float32)), c_int(K), c_int(K), _ptr(index), c_int(rows),
                                                 _ptr(gamma), c_float(eps), c_int(0), c_void_p(0), c_void_p(0), c_void_p(0),
                                                 c_int(DEVICE_TYPE[type_name]), c_int(terms), self.data, self.scale, self.counters, c_int(counters),
                                                 _stream()), "pk_quant_stage_rows")


def _umma(st: _Staged, w_raw: torch.Tensor, type_name: str, N: int, K: int, seg, groups: int, epi: int, out: torch.Tensor, limit: float, columns: int,
          parts: int, splits: int, status: torch.Tensor | None) -> None:
    _check(_lib.kernels().pk_quant_rows(_ptr(w_raw), c_int(DEVICE_TYPE[type_name]), c_int(N), c_int(K), _ptr(seg), c_int(groups), c_int(st.rows), st.data,
                                       st.scale, c_int(st.terms), c_int(epi), _ptr(out), c_int(out.stride(0)), c_void_p(0), c_float(limit), c_int(columns),
                                       c_int(parts), c_int(splits), st.ws, st.counters, st.status if status is None else _ptr(status), c_void_p(0), c_int(0),
                                       c_int(_sm_count()), _stream()), "pk_quant_rows")


def _umma_cost(tiles: int, K: int, parts: int, slots: int, columns: int) -> float:
    """What `tiles` tiles with K in `parts` take on `slots` CTAs, in blocks of 256 weights: rounds of CTAs, each with its blocks and, with
    parts, the exchange of a part: its 128 x `columns` sums and the counter, then all parts by the last CTA. 128-row tiles, us by parts:
    IQ2_XXS, 192 tiles of K = 3072 22.5 / 26.6 / 29.4 (1 / 2 / 3), 24 tiles 20.5 / 18.4 / 16.4 / 16.4 (1 / 2 / 4 / 6); Q5_K, 24 tiles of K =
    6144, 16 columns 32.7 / 23.4 / 19.2 / 17.2 / 22.6 (1 / 2 / 4 / 6 / 8), 64 columns 36.9 / 27.6 / 24.6 / 25.4 / 36.8; 64 tiles of K = 3072
    22.5 / 18.5 / 22.5 (1 / 2 / 3); Q4_K, 256 tiles 28.7 / 38.9 / 43.0."""
    return -(-tiles * parts // slots) * (K / 256 / parts + (3 + parts * columns / 32 if parts > 1 and columns else 0))


def _umma_splits(tiles: int, K: int, slots: int, columns: int = 0) -> int:
    """Parts of K for `tiles` tiles of `columns` columns on `slots` CTAs (columns 0: as if the exchange cost nothing, which no product asks for), two
    256-weight blocks in a part at least."""
    return min(range(1, max(1, min(K // 512, 4 * slots // tiles)) + 1), key=lambda s: _umma_cost(tiles, K, s, slots, columns))


def _umma_slots(type_name: str, columns: int) -> int:
    return _sm_count()      # resident CTAs of the kernel: one an SM for every type and tile


def _umma_linear(x: torch.Tensor, w_raw: torch.Tensor, type_name: str, N: int, gamma, eps: float, epi: int,
                 status: torch.Tensor | None) -> torch.Tensor:
    M, K = x.shape
    columns = 16 if M <= 16 else 32 if M <= 32 else 64
    tiles = (-(-(N // 2) // 64) if epi == 1 else -(-N // 128)) * -(-M // columns)
    splits = _umma_splits(tiles, K, _umma_slots(type_name, columns), columns)
    st = _Staged(x, type_name, M, 1, gamma=gamma, eps=eps, counters=tiles if splits > 1 else 0, ws_floats=tiles * splits * columns * 128 if splits > 1 else 0)
    y = torch.empty(M, N // 2 if epi == 1 else N, device=x.device, dtype=torch.float32 if epi == 2 else torch.bfloat16)
    _umma(st, w_raw, type_name, N, K, None, 1, epi, y, 0.0, columns, splits, splits, status)
    return y


def _umma_experts(x: torch.Tensor, w13_raw: torch.Tensor, w2_raw: torch.Tensor, type13: str, type2: str, inter: int, routes: "Routes", limit: float,
                  E: int, expert_offset: int, local: int, terms: int, status: torch.Tensor | None) -> torch.Tensor:
    """fp32 [R, H]: every route's expert output, without its weight. `terms`: fp16 terms that a hidden value is multiplied as."""
    seg, tok, _ = routes
    H, R, dev = x.shape[1], tok.numel(), x.device
    seg = seg[expert_offset:]

    def columns(t: int) -> int:      # of an expert's tile: what most experts with routes need
        n = t * R / E      # a rank's experts see their share of the routes: the same tiles however the experts are split
        return 16 if n <= 10 else 32 if n <= 24 else 64

    def product(x, w_raw, type_name, N, K, t, epi, out, limit, index):
        c, row_tiles = columns(t), -(-(N // 2) // 64) if epi == 3 else -(-N // 128)
        most = max(1, min(R, local)) * row_tiles        # tiles, if every route is an expert of its own
        parts = splits = 1
        slots = _umma_slots(type_name, c)
        if c == 16:
            # K is cut as for one token's routes whatever the step holds and however the experts are split over ranks: a token's sum does
            # not depend on the tokens beside it. CTAs of their own take the parts where that fills the SMs better.
            parts = _umma_splits(routes.topk * row_tiles, K, slots, c)
            if R <= UMMA_SPLIT_ROUTES and most * parts <= 4 * slots and _umma_cost(most, K, parts, slots, c) < _umma_cost(most, K, 1, slots, c):
                splits = parts
        elif R <= UMMA_SPLIT_ROUTES:       # beyond, the tiles fill the SMs
            parts = splits = _umma_splits(most, K, slots, c)
        tiles = (min(R, local) + R * t // c) * row_tiles if splits > 1 else 0
        st = _Staged(x, type_name, R, t, index=index, counters=tiles, ws_floats=tiles * splits * c * 128)
        _umma(st, w_raw, type_name, N, K, seg, local, epi, out, limit, c, parts, splits, status)

    h = torch.empty(R, inter, device=dev, dtype=torch.float32)
    y = torch.empty(R, H, device=dev, dtype=torch.float32)
    product(_aligned(x), w13_raw, type13, 2 * inter, H, 1, 3, h, limit, tok)
    product(h, w2_raw, type2, H, inter, terms, 2, y, 0.0, None)
    return y


def _umma_experts_take(w13_raw: torch.Tensor, w2_raw: torch.Tensor, type13: str, type2: str, H: int, inter: int, local: int) -> bool:
    return (_umma_takes(w13_raw, type13, 2 * inter, H, local) and _umma_takes(w2_raw, type2, H, inter, local) and max(H, inter) * 4 <= 200 * 1024
            and local <= UMMA_MAX_GROUPS)


def _reduce_routes(y: torch.Tensor, routes: "Routes", shape, expert_offset: int, local: int, out: torch.Tensor) -> torch.Tensor:
    """out[t] += sum over the token's local routes, in route order, of weight * y[route]."""
    seg, tok, rw = routes
    T, H = shape
    pos = torch.empty(tok.numel(), device=y.device, dtype=torch.int32)
    _check(_lib.kernels().pk_moe_reduce_routes(_ptr(y), _ptr(rw), _ptr(routes.src), _ptr(seg), c_int(T), c_int(routes.topk), c_int(H),
                                               c_int(expert_offset), c_int(local), _ptr(pos), _ptr(out), _stream()), "pk_moe_reduce_routes")
    return out


TENSOR_CORE_MIN_ROWS = 32
_scratch: dict = {}


def _dequant_scratch(w_raw: torch.Tensor, type_name: str, N: int, K: int) -> torch.Tensor:
    """bf16 [N, K] copy of a quantised weight in a per-device buffer that the next call reuses (stream ordered)."""
    key = (w_raw.device.index, torch.cuda.current_stream().cuda_stream)
    buf = _scratch.get(key)
    if buf is None or buf.numel() < N * K:
        buf = torch.empty(N * K, device=w_raw.device, dtype=torch.bfloat16)
        _scratch[key] = buf
    out = buf[: N * K].view(N, K)
    rb = row_bytes(type_name, K)
    st = _lib.kernels().pk_gguf_dequant_rows(_ptr(w_raw), c_int(DEVICE_TYPE[type_name]), c_void_p(0), c_int(N), c_int(K), c_int(0),
                                             c_int(w_raw.numel() // rb), _ptr(out), _stream())
    _check(st, "pk_gguf_dequant_rows")
    return out


def router_topk(x: torch.Tensor, router_w: torch.Tensor, topk: int, *, bias: torch.Tensor | None = None,
                score_func: str = "sigmoid", norm_topk: bool = True, route_scale: float = 1.0) -> tuple[torch.Tensor, torch.Tensor]:
    T, H = x.shape
    E = router_w.shape[0]
    ids = torch.empty(T, topk, device=x.device, dtype=torch.int32)
    w = torch.empty(T, topk, device=x.device, dtype=torch.float32)
    st = _lib.kernels().pk_router_topk(_ptr(x), _ptr(router_w), _ptr(bias), c_int(T), c_int(H), c_int(E), c_int(topk),
                                       c_int(SCORE_FUNCS[score_func]), c_int(int(norm_topk)), c_float(route_scale), _ptr(ids),
                                       _ptr(w), _stream())
    _check(st, "pk_router_topk")
    return ids, w


class Routes(tuple):
    """(seg_start [E+1], route_token [R], route_weight [R]) plus `.src` [R]: original route index t * topk + k of each
    sorted route, and `.topk`."""
    src: torch.Tensor
    topk: int


def group_routes(ids: torch.Tensor, weights: torch.Tensor, E: int) -> Routes:
    """Sort routes by expert (stable in route index)."""
    T, topk = ids.shape
    seg = torch.empty(E + 1, device=ids.device, dtype=torch.int32)
    tok = torch.empty(T * topk, device=ids.device, dtype=torch.int32)
    rw = torch.empty(T * topk, device=ids.device, dtype=torch.float32)
    src = torch.empty(T * topk, device=ids.device, dtype=torch.int32)
    st = _lib.kernels().pk_group_routes(_ptr(ids), _ptr(weights), c_int(T), c_int(topk), c_int(E), _ptr(seg), _ptr(tok),
                                        _ptr(rw), _ptr(src), _stream())
    _check(st, "pk_group_routes")
    r = Routes((seg, tok, rw))
    r.src, r.topk = src, topk
    return r


def gguf_moe_forward(x: torch.Tensor, w13_raw: torch.Tensor, w2_raw: torch.Tensor, type13: str, type2: str, E: int, inter: int,
                     seg: torch.Tensor, tok: torch.Tensor, rw: torch.Tensor, *, limit: float = 0.0, expert_offset: int = 0,
                     local_experts: int | None = None, out: torch.Tensor | None = None, routes: "Routes | None" = None,
                     status: torch.Tensor | None = None) -> torch.Tensor:
    """Routed experts of this rank accumulated into fp32 `out` [T, H] (zeroed when not given). With `routes` (the object
    `group_routes` returned) the per-token sum runs in a fixed order and the result is bitwise reproducible; without it
    the routes are added with atomics."""
    T, H = x.shape
    R = tok.numel()
    local = E if local_experts is None else local_experts
    if out is None:
        out = torch.zeros(T, H, device=x.device, dtype=torch.float32)
    if routes is not None and _umma_experts_take(w13_raw, w2_raw, type13, type2, H, inter, local):
        # hidden values in two fp16 terms: as good as the fp32 values of the kernels that decode in registers
        y = _umma_experts(x, w13_raw, w2_raw, type13, type2, inter, routes, limit, E, expert_offset, local, 2, status)
        return _reduce_routes(y, routes, x.shape, expert_offset, local, out)
    hbuf = torch.empty(R, inter, device=x.device, dtype=torch.float32)
    if routes is not None:
        ybuf = torch.empty(R, H, device=x.device, dtype=torch.float32)
        pos = torch.empty(R, device=x.device, dtype=torch.int32)
        st = _lib.kernels().pk_gguf_moe_forward_det(
            _ptr(w13_raw), _ptr(w2_raw), c_int(DEVICE_TYPE[type13]), c_int(DEVICE_TYPE[type2]), c_int(E), c_int(H), c_int(inter),
            _ptr(x), _ptr(seg), _ptr(tok), _ptr(rw), _ptr(routes.src), _ptr(hbuf), _ptr(ybuf), _ptr(pos), _ptr(out), c_int(T),
            c_int(routes.topk), c_float(limit), c_int(expert_offset), c_int(local), c_int(_sm_count()), _stream())
        _check(st, "pk_gguf_moe_forward_det")
        return out
    st = _lib.kernels().pk_gguf_moe_forward(
        _ptr(w13_raw), _ptr(w2_raw), c_int(DEVICE_TYPE[type13]), c_int(DEVICE_TYPE[type2]), c_int(E), c_int(H), c_int(inter),
        _ptr(x), _ptr(seg), _ptr(tok), _ptr(rw), _ptr(hbuf), _ptr(out), c_float(limit), c_int(expert_offset), c_int(local),
        c_int(_sm_count()), _stream())
    _check(st, "pk_gguf_moe_forward")
    return out


_GROUPED_SCRATCH: dict = {}


def gguf_moe_forward_grouped(x: torch.Tensor, w13_raw: torch.Tensor, w2_raw: torch.Tensor, type13: str, type2: str, E: int, inter: int,
                             routes: "Routes", *, expert_offset: int = 0, local_experts: int | None = None,
                             out: torch.Tensor | None = None, peer=None, status: torch.Tensor | None = None) -> torch.Tensor:
    """Routed experts of this rank on the tensor cores, for steps with many routes (prefill). Types in `UMMA_TYPES` are decoded
    inside the product up to `UMMA_MAX_ROUTES_PER_EXPERT`; otherwise the rank's experts are decoded to bf16 once per call
    into a scratch that is reused across layers, token rows are gathered in expert order, and two
    grouped tcgen05 GEMMs (gate|up with the SwiGLU epilogue, then down) run one persistent launch each over every
    (expert, row tile, column block) that has rows; the tile list comes from the route segments on the device. The
    per-token sum runs in route order (bitwise reproducible). Same result as `gguf_moe_forward` up to bf16 rounding of the
    hidden activations. With `peer` (a `PeerAllReduce` of the expert-parallel group) whose arena holds T * H floats the result
    is already summed over the ranks (`routes.combined` is set): the combine runs as peer stores out of the reduce."""
    from . import EPI_F32, EPI_SWIGLU
    seg, tok, rw = routes
    T, H = x.shape
    R = tok.numel()
    local = E if local_experts is None else local_experts
    dev = x.device
    if out is None:
        out = torch.zeros(T, H, device=dev, dtype=torch.float32)
    K = _lib.kernels()
    if R <= UMMA_MAX_ROUTES_PER_EXPERT * E and _umma_experts_take(w13_raw, w2_raw, type13, type2, H, inter, local):
        ybuf = _umma_experts(x, w13_raw, w2_raw, type13, type2, inter, routes, 0.0, E, expert_offset, local, 1, status)
    else:
        key = (dev.index, local, H, inter)
        sc = _GROUPED_SCRATCH.get(key)
        if sc is None:
            sc = (torch.empty(local * 2 * inter, H, device=dev, dtype=torch.bfloat16), torch.empty(local * H, inter, device=dev, dtype=torch.bfloat16))
            _GROUPED_SCRATCH.clear()          # one shape at a time: the scratch is as large as the layer's experts in bf16
            _GROUPED_SCRATCH[key] = sc
        w13, w2 = sc
        _check(K.pk_gguf_dequant_rows(_ptr(w13_raw), c_int(DEVICE_TYPE[type13]), c_void_p(0), c_int(local * 2 * inter), c_int(H), c_int(0),
                                      c_int(local * 2 * inter), _ptr(w13), _stream()), "pk_gguf_dequant_rows(w13)")
        _check(K.pk_gguf_dequant_rows(_ptr(w2_raw), c_int(DEVICE_TYPE[type2]), c_void_p(0), c_int(local * H), c_int(inter), c_int(0), c_int(local * H),
                                      _ptr(w2), _stream()), "pk_gguf_dequant_rows(w2)")
        xg = x.index_select(0, tok.long())                                   # [R, H] rows in expert order
        hbuf = torch.empty(R, inter, device=dev, dtype=torch.bfloat16)
        ybuf = torch.empty(R, H, device=dev, dtype=torch.float32)
        if status is None:
            status = torch.zeros(1, device=dev, dtype=torch.int32)
        segl = seg[expert_offset:]
        _check(K.pk_gemm_bf16_grouped(_ptr(xg), c_int(H), _ptr(w13), _ptr(segl), c_int(local), c_int(R), c_int(2 * inter), c_int(H), c_int(EPI_SWIGLU),
                                      _ptr(hbuf), c_int(inter), _ptr(status), c_int(_sm_count()), _stream()), "pk_gemm_bf16_grouped(w13)")
        _check(K.pk_gemm_bf16_grouped(_ptr(hbuf), c_int(inter), _ptr(w2), _ptr(segl), c_int(local), c_int(R), c_int(H), c_int(inter), c_int(EPI_F32),
                                      _ptr(ybuf), c_int(H), _ptr(status), c_int(_sm_count()), _stream()), "pk_gemm_bf16_grouped(w2)")
    routes.combined = False
    if peer is not None and T * H <= peer.capacity:
        pos = torch.empty(R, device=dev, dtype=torch.int32)
        # several ranks: the per-token reduce is the producer of the combine kernel, which stores this rank's sums into every
        # rank's arena, signals, waits (bounded) and adds the ranks' slots: `out` is the sum over all ranks' experts
        _check(K.pk_invert_routes(_ptr(routes.src), c_int(R), _ptr(pos), _stream()), "pk_invert_routes")
        peer.moe_combine(ybuf, rw, pos, seg, expert_offset, local, T, routes.topk, out)
        routes.combined = True
        return out
    return _reduce_routes(ybuf, routes, x.shape, expert_offset, local, out)


UMMA_MAX_ROUTES_PER_EXPERT = 384      # far above this a decode per 64 routes costs more than one decode to a bf16 scratch. Time inside the product over that
#                                        with the scratch, routes spread at random, IQ2_XXS / Q4_K / Q5_K, at 192, 256, 320, 384 routes: 1536 x 3072 .63 / .61 / .64,
#                                        .76 / .73 / .76, .86 / .84 / .87, .94 / .91 / .96, even at 448; 1024 x 2048 .78 / .76 / .76, .93 / .89 / .91, 1.03 / .99 / 1.03,
#                                        1.15 / 1.12 / 1.15; 768 x 2048 .81 / .78 / .79, .95 / .91 / .95, 1.07 / 1.04 / 1.06, 1.14 / 1.13 / 1.17. The smaller matrices,
#                                        whose tiles have few blocks of K to set against filling and folding, lose from 300 routes on; hidden values keep 11 bits
#                                        here and 8 with the scratch, so the line is the same for all
GROUPED_MIN_ROUTES_PER_EXPERT = 4     # below this the decode of every local expert costs more than the route kernels' per-route decode


def moe_forward(x: torch.Tensor, w13_raw: torch.Tensor, w2_raw: torch.Tensor, type13: str, type2: str, E: int, inter: int, routes: "Routes", *,
                limit: float = 0.0, expert_offset: int = 0, local_experts: int | None = None, peer=None,
                status: torch.Tensor | None = None) -> torch.Tensor:
    """Routed experts of this rank, fp32 [T, H]: the grouped form for steps with many routes per expert (prefill),
    otherwise (decode, clamped SwiGLU) the form that keeps hidden values in fp32."""
    seg, tok, rw = routes
    local = E if local_experts is None else local_experts
    H = x.shape[1]
    if (limit == 0.0 and tok.numel() >= GROUPED_MIN_ROUTES_PER_EXPERT * local and inter % 128 == 0 and H % 128 == 0 and local <= 512):
        return gguf_moe_forward_grouped(x, w13_raw, w2_raw, type13, type2, E, inter, routes, expert_offset=expert_offset, local_experts=local,
                                        peer=peer, status=status)
    routes.combined = False
    return gguf_moe_forward(x, w13_raw, w2_raw, type13, type2, E, inter, seg, tok, rw, limit=limit, expert_offset=expert_offset,
                            local_experts=local, routes=routes, status=status)


def gguf_dequant_rows(w_raw: torch.Tensor, type_name: str, K: int, rows: torch.Tensor | None = None, *, nrows: int | None = None,
                      row_offset: int = 0) -> torch.Tensor:
    """Decode rows of a quantised table to bf16 (quantised embedding gather, or a whole
    weight when `rows` is None)."""
    rb = row_bytes(type_name, K)
    table_rows = w_raw.numel() // rb
    n = rows.numel() if rows is not None else (nrows if nrows is not None else table_rows)
    out = torch.empty(n, K, device=w_raw.device, dtype=torch.bfloat16)
    st = _lib.kernels().pk_gguf_dequant_rows(_ptr(w_raw), c_int(DEVICE_TYPE[type_name]), _ptr(rows), c_int(n), c_int(K),
                                             c_int(row_offset), c_int(table_rows), _ptr(out), _stream())
    _check(st, "pk_gguf_dequant_rows")
    return out
