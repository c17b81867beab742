"""Mixers that keep a state of fixed size per request instead of keys and values: a selective
state-space mixer and a gated delta rule (kernels: csrc/recurrent.cu).

Both ask the cache manager for one 32-bit state row per request (zeroed at admission): the
recurrence's matrices, then the last ``taps - 1`` inputs of the short causal convolution.  A step
brings any mix of prompt portions and single tokens; the kernels find each request's tokens and
state row through the step's device arrays, so the parts run inside replayed CUDA graphs.
Projections are matrix products in the activation type; what enters a recurrence (step sizes,
decays, gates of the recurrence, unit norms, the state) is 32-bit.
"""
from __future__ import annotations

import torch

from ..config.specs import ParamSpec
from ..csrc import ops
from .base import Mixer, StateRequest, make_position, once_per_step, register_mixer
from .linear import linear, pad_rows
from .position import as_rotary_args


def _check_state_rows(rows: int, what: str) -> None:
    if not 0 < rows <= ops.LIMITS["recurrent_max_state_rows"]:
        raise ValueError(f"{what} {rows} is not supported (1 to {ops.LIMITS['recurrent_max_state_rows']}: a state "
                         "column's rows live in the registers of one warp's lanes)")


def takes_chunks(mixer, step, heads: int, rows: int, columns: int, prepare: float, device, *, chunk: int = 64, block=(22.0, 4.0),
                 launches: float = 8.0, token: float = 0.58, walk=None) -> bool:
    """Whether a step's recurrence runs in chunks: by what either form is estimated to take (us), if the longest entry has
    ``chunk_min_tokens`` tokens (by that number alone where ``chunks_by_estimate`` is off).  ``walk``: token by token, of the longest
    entry's tokens, the entries and all tokens; by default ``token`` per token of the longest, or 5.9e-5 per token and state column of 128 rows
    where the device is full.  In chunks: ``launches``, then ``block`` = (an entry's first chunk, each further one) for each block of 32
    columns, side by side over the device, and ``prepare`` per head and token of the chunks, full or not: single tokens beside a
    portion cost a block and a chunk each, which is why the entries' own lengths count.  Measured on one B200, a layer (state space
    of 64 heads, 64 x 128; delta per channel and per head, 16 heads of 128 x 128), us token by token / in chunks: one entry of 48 tokens
    51/57, 62/57, 57/55, of 128 86/66, 109/64, 100/62, of 2,048 975/349, 1,537/371, 1,416/336; four of 96 135/150, 110/116,
    100/113, of 192 238/195, 180/164, 177/152; sixty-four of 64 1,099/1,318, 686/908, 693/895; one of 300 beside 7 single tokens
    190/219, 237/174, 228/166, beside 31 188/588, 244/367, 234/403, of 1,024 beside 31 594/752, 791/546, 753/577."""
    longest = step.max_q_len
    if mixer.chunk_min_tokens is None or longest < mixer.chunk_min_tokens:
        return False
    if not getattr(mixer, "chunks_by_estimate", True):
        return True
    entries, tokens, sms = step.num_seqs, step.num_tokens, ops.sm_count(device)
    lens = getattr(step, "q_lens", None) or [longest] + [(tokens - longest) // max(1, entries - 1)] * (entries - 1)
    pieces = sum(-(-n // chunk) for n in lens)
    if walk is not None:
        one_by_one = walk(longest, entries, tokens)
    else:
        one_by_one = 4 + 0.06 * entries + max(token * longest, 4.5e-7 * 148 / sms * tokens * heads * columns * rows)
    first, further = block
    share = heads * -(-columns // 32) / sms                        # of a full device that an entry's blocks are
    chunks = max(first + further * (-(-longest // chunk) - 1), (first * entries + further * (pieces - entries)) * share)
    return launches + chunks + prepare * chunk * pieces * heads < one_by_one


class StateSpaceMixer(Mixer):
    """``[z | x | B | C | dt] = in_proj(h)``; x, B, C through a causal convolution (bias) and silu;
    ``dt = softplus(dt + dt_bias)``; per head ``S <- exp(-exp(A_log) dt) S + dt B x^T``,
    ``y = S^T C + D x``; ``y * silu(z)`` RMS-normed in ``norm_groups`` parts, times a weight; out
    projection."""
    graph_safe = True
    # The longest entry of a step from which the recurrence may run in chunks of 64 one after another; None: in no chunks at all.  Below, the launch that
    # they take more costs a small step, which waits for the host, what the kernels save (a layer's call at 64 tokens: 86 us without, 96
    # with).  Chunks side by side (`in_tiles`) go by estimates alone.
    chunk_min_tokens = 96
    # the engine option that sets it and switches the estimate off that chunks take less time than tokens one by one: either form of chunks is then taken
    # from that many tokens on, the one that is estimated to take less time
    chunk_tuning_key = "recurrence_chunk_min_tokens"

    def __init__(self, spec, dtype):
        super().__init__(spec, dtype)
        s = spec
        if min(s.num_heads, s.head_dim, s.groups, s.conv_taps, s.norm_groups, s.hidden_size) <= 0:
            raise ValueError("the sizes of a state-space mixer must be positive")
        if s.num_heads % s.groups:
            raise ValueError("num_heads must be a multiple of groups")
        if (s.num_heads * s.head_dim) % s.norm_groups:
            raise ValueError("norm_groups must divide num_heads * head_dim")
        if s.num_heads > ops.LIMITS["grid_dim_yz"] or s.norm_groups > ops.LIMITS["grid_dim_yz"]:
            raise ValueError("heads and norm groups are grid dimensions of the kernels (at most 65,535)")
        _check_state_rows(s.state_size, "state_size")
        self.inner = s.num_heads * s.head_dim
        self.conv_channels = self.inner + 2 * s.groups * s.state_size
        self.conv_off = s.num_heads * s.head_dim * s.state_size

    def parameters(self):
        s = self.spec
        return {"in_proj": ParamSpec((2 * self.inner + 2 * s.groups * s.state_size + s.num_heads, s.hidden_size)),
                "conv_w": ParamSpec((self.conv_channels, s.conv_taps), "float32"),
                "conv_b": ParamSpec((self.conv_channels,), "float32", "bias"),
                "dt_bias": ParamSpec((s.num_heads,), "float32", "bias"),
                "a_log": ParamSpec((s.num_heads,), "float32", "bias"),
                "d_skip": ParamSpec((s.num_heads,), "float32", "norm"),
                "norm_w": ParamSpec((self.inner,), "float32", "norm"),
                "o": ParamSpec((s.hidden_size, self.inner))}

    def state_request(self):
        return StateRequest((self.conv_off + (self.spec.conv_taps - 1) * self.conv_channels,), torch.float32)

    def token_by_token(self, longest: int, entries: int, tokens: int, sms: int) -> float:
        """Estimated us of the shorter of csrc/recurrent.cu's two forms, lane groups and tiles."""
        s = self.spec
        size = s.num_heads * s.head_dim * s.state_size / 524288 * 148 / sms
        return min(3 + 0.65 * size * entries + max(max(0.8, 0.45 * size) * longest, 0.24 * size * tokens),
                   6 + 1.45 * size * entries + max(max(0.44, 0.33 * size) * longest, 0.23 * size * tokens))

    def in_chunks(self, step, device) -> bool:
        if self.chunk_min_tokens is None or step.max_q_len < self.chunk_min_tokens:
            return False
        s, sms = self.spec, ops.sm_count(device)
        return once_per_step(step, ("state_space.in_chunks", s.num_heads, s.state_size, s.head_dim), lambda: (
            takes_chunks(self, step, s.num_heads, s.state_size, s.head_dim, 2.1e-4, device, block=(19.5, 7.0), launches=17.0,
                         walk=lambda longest, entries, tokens: self.token_by_token(longest, entries, tokens, sms))
            and ops.chunk_walk_supported(s.state_size, s.head_dim)))

    def in_tiles(self, step, device) -> int:
        """Heads that a block takes (true) of a step that csrc/ssm_tiles.cu takes (bfloat16, states of 128 rows, heads of 64 columns) and that goes there; else 0.
        By estimates of it, of the form token by token and of chunks of 64 one after another (where those would be next), which read C and B once per head and take
        4 us a chunk where their blocks leave half of the device idle, else 7.  Measured, device us of a layer, the other forms (s, w) / here: 64 heads in 8
        groups, one entry of 90 tokens s 66/48, of 128 w 52/49, of 257 66/60, of 512 84/67, of 4,096 437/317, four of 96 s 117/80, of 130 w 153/88, sixteen of 40 s 185/139, sixty-four of 96
        s 1,529/616, 300 beside 15 single tokens w 188/139, 1,024 beside 63 s 611/465; 32 heads in 8, 128 tokens w 42/46, 200 49/47, 512 64/54,
        in one group 128 w 65/45; 16 heads in 8, two entries of 130 w 43/47, 1,024 tokens w 90/58; 8 heads in 8, 200 w 45/45, 257 w 46/46, 1,024 w 90/56.
        The chunks' states take 32 KB per head and chunk: no more than 256 MB, or than the other chunks' workspace."""
        least = self.chunk_min_tokens
        if least is None or step.max_q_len < min(least, 17):
            return 0

        def ask():
            s, sms = self.spec, ops.sm_count(device)
            longest, entries, tokens = step.max_q_len, step.num_seqs, step.num_tokens
            if (tokens // 128 + entries) * s.num_heads * 8193 > max(1 << 26, tokens * s.num_heads * 67):
                return 0
            lens = getattr(step, "q_lens", None) or [longest] + [(tokens - longest) // max(1, entries - 1)] * (entries - 1)
            chunks, rep = sum(-(-n // 128) for n in lens), s.num_heads // s.groups
            us, per = ops.ssm_tiles_plan(chunks, s.num_heads, s.groups, sms)
            if getattr(self, "chunks_by_estimate", True):
                most = min(8, rep)
                shared_out = 35 + chunks * s.groups * -(-rep // most) * (10 + 13 * most) / sms
                if s.num_heads * longest <= 2048 or shared_out >= self.token_by_token(longest, entries, tokens, sms):
                    return 0
                if not self.in_chunks(step, device):
                    return per
            elif longest < least:
                return 0
            share = s.num_heads * -(-s.head_dim // 32) / sms
            first, further = (19.5, 7.0) if share > 0.5 else (17.0, 4.2)
            pieces = sum(-(-n // 64) for n in lens)
            walk = max(first + further * (-(-longest // 64) - 1), (first * entries + further * (pieces - entries)) * share)
            return per if 26 + us < 17 + walk + 2.1e-4 * 64 * pieces * s.num_heads + 0.8 * rep else 0
        return once_per_step(step, ("state_space.in_tiles", self.spec.num_heads, self.spec.groups, self.spec.state_size, self.spec.head_dim), ask)

    def forward(self, x, step, slot):
        s = self.spec
        tokens = x.shape[0]
        proj = linear(x, self.in_proj)
        xbc = torch.empty(tokens, self.conv_channels, dtype=torch.float32, device=x.device)
        ops.causal_conv(proj, self.inner, self.conv_w, self.conv_b, slot.state, self.conv_off, step, xbc)
        y = torch.empty(tokens, self.inner, dtype=torch.float32, device=x.device)
        args = (xbc, proj, self.inner + self.conv_channels, self.dt_bias, self.a_log, self.d_skip, slot.state, step, y)
        sizes = dict(heads=s.num_heads, head_dim=s.head_dim, state_size=s.state_size, groups=s.groups)
        per = self.in_tiles(step, x.device)
        if per and ops.ssm_tiles_supported(s.state_size, s.head_dim, proj, slot.state):
            ops.ssm_tiles(*args, **sizes, heads_per_block=per)
        else:
            (ops.ssm_walk if self.in_chunks(step, x.device) else ops.ssm_scan)(*args, **sizes)
        gated = torch.empty(tokens, self.inner, dtype=x.dtype, device=x.device)
        ops.gated_group_norm(y, proj, 0, self.norm_w, gated, parts=s.norm_groups, eps=s.norm_eps)
        return linear(gated, self.o)


class GatedDeltaMixer(Mixer):
    """``[q | k | v | b | a | g] = in_proj(h)``; q, k, v through causal convolutions and silu; q and
    k unit vectors per head (q times ``head_dim ** -0.5``); ``beta = sigmoid(b)``; decay per head and key
    channel ``exp(-exp(A_log) softplus(a2(a) + dt_bias))``; per head ``S <- diag(decay) S``,
    ``u = beta (v - S^T k)``, ``S <- S + k u^T``, ``o = S^T q``; each head's ``o`` over its root
    mean square, times a weight shared by the heads, times ``sigmoid(g2(g))``; out projection.
    With ``decay_per="head"`` the decay is one number per head, ``exp(-exp(A_log) softplus(a + dt_bias))``
    with ``a`` a column of the input projection, and the gate ``gate_activation(g)`` with ``g`` columns of
    the input projection (no low ranks)."""
    graph_safe = True
    # The longest entry of a step from which the recurrence may run in chunks; None: never.  Below, token by token is as fast (an entry
    # of 32 tokens: 27 against 29 us).
    chunk_min_tokens = 48
    chunk_tuning_key = "recurrence_chunk_min_tokens"     # the engine option that sets it (and switches the estimate off)

    def __init__(self, spec, dtype):
        super().__init__(spec, dtype)
        s = spec
        if s.decay_per not in ("channel", "head") or s.gate_activation not in ("sigmoid", "silu"):
            raise ValueError("decay_per is 'channel' or 'head', gate_activation 'sigmoid' or 'silu'")
        self.per_head = s.decay_per == "head"
        self.sizes = dict(heads=s.num_heads, kv_heads=s.num_kv_heads, head_dim=s.head_dim, v_head_dim=s.v_head_dim)
        self.inputs = dict(unit_eps=s.unit_eps, q_scale=s.head_dim ** -0.5, per_head=self.per_head)
        ranks = () if self.per_head else (s.decay_rank, s.gate_rank)
        if min(s.num_heads, s.num_kv_heads, s.head_dim, s.v_head_dim, s.conv_taps, s.hidden_size, *ranks) <= 0:
            raise ValueError("the sizes of a gated-delta mixer must be positive")
        if s.num_heads % s.num_kv_heads:
            raise ValueError("num_heads must be a multiple of num_kv_heads")
        if s.num_heads > ops.LIMITS["grid_dim_yz"]:
            raise ValueError("heads are a grid dimension of the kernels (at most 65,535)")
        _check_state_rows(s.head_dim, "head_dim")
        self.qk = s.num_kv_heads * s.head_dim
        self.vv = s.num_heads * s.v_head_dim
        self.conv_channels = 2 * self.qk + self.vv
        self.conv_off = s.num_heads * s.v_head_dim * s.head_dim
        self.b_off = self.conv_channels
        self.a_off = self.b_off + s.num_heads
        # one decay per head: the decay's and the gate's columns come straight from the input projection
        self.a_cols = s.num_heads if self.per_head else s.decay_rank
        self.g_off = self.a_off + self.a_cols
        self.g_cols = self.vv if self.per_head else s.gate_rank

    def parameters(self):
        s = self.spec
        out = {"in_proj": ParamSpec((self.g_off + self.g_cols, s.hidden_size)),
               "conv_w": ParamSpec((self.conv_channels, s.conv_taps), "float32"),
               "dt_bias": ParamSpec((s.num_heads * (1 if self.per_head else s.head_dim),), "float32", "bias"),
               "a_log": ParamSpec((s.num_heads,), "float32", "bias"),
               "norm_w": ParamSpec((s.v_head_dim,), "float32", "norm"),
               "o": ParamSpec((s.hidden_size, self.vv))}
        if not self.per_head:
            out["a2"] = ParamSpec((s.num_heads * s.head_dim, s.decay_rank))
            out["g2"] = ParamSpec((self.vv, s.gate_rank))
        return out

    def state_request(self):
        return StateRequest((self.conv_off + (self.spec.conv_taps - 1) * self.conv_channels,), torch.float32)

    def in_chunks(self, step, device) -> bool:
        if self.chunk_min_tokens is None or step.max_q_len < self.chunk_min_tokens:
            return False
        s = self.spec
        costs = (dict(prepare=1.9e-3) if self.per_head else dict(prepare=2.8e-3, chunk=32, block=(15.0, 3.0), launches=15.0, token=0.63))
        return once_per_step(step, ("delta.in_chunks", self.per_head, s.num_heads, s.head_dim, s.v_head_dim), lambda: (
            takes_chunks(self, step, s.num_heads, s.head_dim, s.v_head_dim, device=device, **costs)))

    def forward(self, x, step, slot):
        s = self.spec
        tokens, dev = x.shape[0], x.device
        proj = linear(x, self.in_proj)
        qkv = torch.empty(tokens, self.conv_channels, dtype=torch.float32, device=dev)
        ops.causal_conv(proj, 0, self.conv_w, None, slot.state, self.conv_off, step, qkv)
        a, gate = proj[:, self.a_off:self.a_off + self.a_cols], proj[:, self.g_off:self.g_off + self.g_cols]
        if not self.per_head:       # through the low ranks
            a, gate = linear(a, self.a2), linear(gate, self.g2)
        # Steps with prompt portions run the recurrence in chunks, prepared side by side and walked (csrc/chunk_walk.cuh); others
        # (single tokens, short pieces, head sizes the chunks do not take) prepare q, k, decays and beta, then walk the tokens.
        sizes, inputs = self.sizes, self.inputs
        o = torch.empty(tokens, self.vv, dtype=torch.float32, device=dev)
        long = self.in_chunks(step, dev)
        # (decays per channel are read four at a time: a bias bound as a view off 16 bytes goes token by token)
        if (long and ops.chunk_walk_supported(s.head_dim, s.v_head_dim)
                and (self.per_head or (self.dt_bias.data_ptr() | a.data_ptr()) % 16 == 0)):
            ops.delta_walk(qkv, a, proj, self.b_off, self.dt_bias, self.a_log, slot.state, step, o, **sizes, **inputs)
        else:
            # One decay per head: chunks of 64 tokens in one kernel, while its (entry, head, 32 columns) blocks do not fill the
            # device (it does about twice the multiply-adds of the walk token by token).
            chunked = (long and self.per_head and s.head_dim <= ops.LIMITS["delta_chunk_max_head_dim"]
                       and step.num_seqs * s.num_heads * (-(-s.v_head_dim // 32)) <= ops.sm_count(dev))
            log_dec = torch.empty(tokens, s.num_heads, dtype=torch.float32, device=dev) if chunked else None
            dec = torch.empty(tokens, s.num_heads * s.head_dim, dtype=torch.float32, device=dev)
            beta = torch.empty(tokens, s.num_heads, dtype=torch.float32, device=dev)
            ops.delta_prep(qkv, a, proj, self.b_off, self.dt_bias, self.a_log, dec, beta, **sizes, **inputs, log_dec=log_dec)
            if chunked:
                ops.delta_chunk(qkv, log_dec, beta, slot.state, step, o, **sizes)
            else:
                ops.delta_scan(qkv, dec, beta, slot.state, step, o, **sizes)
        out = torch.empty(tokens, self.vv, dtype=x.dtype, device=dev)
        ops.delta_out(o, gate, self.norm_w, out, heads=s.num_heads, v_head_dim=s.v_head_dim, eps=s.norm_eps,
                      silu=s.gate_activation == "silu")
        return linear(out, self.o)


class RetentionMixer(Mixer):
    """``[q | k | v | g] = in_proj(h)``; q and k rotated by position, k times a factor; per
    head ``S <- decay S + k v^T``, ``o = S^T q`` with a fixed decay; each head's ``o`` over its root
    mean square, times ``silu(g)``; out projection (kernels: csrc/retention.cu).  The state is one
    32-bit ``[heads, head_dim, v_head_dim]`` row per request.  Options (``config.specs.RetentionSpec``): q, k and v through
    a silu first; one norm with a weight over the concatenated heads and a sigmoid gate."""
    # the parameter that projects the mixer's input (a mixer of mixers may stack it with its neighbours' and
    # hand `forward` the product's columns as `proj`)
    input_projection = "in_proj"
    graph_safe = True
    chunk_min_tokens = 16        # the longest entry of a step from which the chunked kernel runs; None: never
    chunk_tuning_key = "retention_chunk_min_tokens"

    def __init__(self, spec, dtype):
        super().__init__(spec, dtype)
        s = spec
        if min(s.num_heads, s.head_dim, s.v_head_dim, s.hidden_size) <= 0:
            raise ValueError("the sizes of a retention mixer must be positive")
        if len(s.decays) != s.num_heads:
            raise ValueError(f"a retention mixer needs one decay per head ({s.num_heads}), got {len(s.decays)}")
        if s.head_dim > ops.LIMITS["retention_max_head_dim"]:
            raise ValueError(f"head_dim {s.head_dim} is not supported (at most {ops.LIMITS['retention_max_head_dim']}: "
                             "a state column's rows live in the registers of eight warps)")
        if s.num_heads > ops.LIMITS["grid_dim_yz"]:
            raise ValueError("heads are a grid dimension of the kernels (at most 65,535)")
        if s.activation not in (None, "silu") or s.output_norm not in ("per_head", "joint"):
            raise ValueError("a retention mixer's activation is None or 'silu', its output_norm 'per_head' or 'joint'")
        self.k_scale = float(s.k_scale) if s.k_scale is not None else s.head_dim ** -0.5
        self.position = make_position(s.position, dtype) if s.position is not None else None
        if self.position is not None:
            if s.position.pairing != "split_half":
                raise ValueError("the retention kernels rotate split halves only")
            if s.position.rotary_dim > s.head_dim:
                raise ValueError(f"the position encoding rotates {s.position.rotary_dim} dims, a head has {s.head_dim}")
        self.qk = s.num_heads * s.head_dim
        self.vv = s.num_heads * s.v_head_dim
        self._decay = None

    def parameters(self):
        s = self.spec
        out = {"in_proj": ParamSpec((2 * self.qk + 2 * self.vv, s.hidden_size)),
               "o": ParamSpec((s.hidden_size, self.vv))}
        if s.output_norm == "joint":
            out["norm_w"] = ParamSpec((self.vv,), "act", "norm")
        return out

    def bind(self, tensors):
        super().bind(tensors)
        self.in_proj = pad_rows(self.in_proj)

    def state_request(self):
        s = self.spec
        return StateRequest((s.num_heads * s.head_dim * s.v_head_dim,), torch.float32)

    def in_walk(self, step, device) -> bool:
        """Whether a step in chunks has them prepared side by side and walked, or goes through the kernel that does a chunk at a time.
        The walk's blocks take an SM each and 2.5 us more for an entry's first chunk, but 6 less for each further one, or 0.25 a token of
        the longest entry, which the other kernel takes in segments.  Measured, a layer, us chunk at a time / walk, 16 and 32 heads of
        128 x 128: one portion of 90 tokens beside 63 single ones 434/491 and 857/983, of 300 515/526 and 968/1,034, of 1,024 838/648
        and 1,380/1,239, of 90 beside 15 151/127 and 286/301; 64 entries of 96 tokens 1,045/914 and 2,368/2,099; four
        entries of 17 to 64 tokens, 32 heads, 118 to 135 against 124 to 143 with the host's launches.  Where all blocks run at once
        the walk is ahead from the first chunk on (one such entry 92 and 76)."""
        s = self.spec

        def ask():
            share = s.num_heads * -(-s.v_head_dim // 32) / ops.sm_count(device)        # of a full device that an entry's blocks are
            if step.num_seqs * share <= 1:
                return True
            lens = getattr(step, "q_lens", None) or [step.max_q_len] * step.num_seqs
            further = sum(-(-n // 64) for n in lens) - len(lens)
            return step.max_q_len > 64 and 2.5 * step.num_seqs * share < max(0.25 * step.max_q_len, 6 * further * share)
        return once_per_step(step, ("retention.in_walk", s.num_heads, s.v_head_dim), ask)

    def in_tiles(self, step, tokens: int, rotary_dim: int, device) -> bool:
        """Whether a step in chunks that csrc/retention_tiles.cu takes (bfloat16, heads of 128 x 128) goes there.  Not where all of the walk's
        blocks run at once and its longest chain is three chunks: each of the two kernels takes some 15 us for a chunk, the walk and its preparation
        7 to 14 and 4 more a chunk; unless it is the host that takes the time (one launch instead of three), which it is until the projections' weights
        take the device as long as 100 MB do.  Measured, device us of a layer without its projections, the other forms / here: 4, 8, 16 and 32 heads, one
        portion of 17 tokens 25/45, 25/41, 27/43, 33/45, of 128 30/41, 31/41, 33/43, 41/45, of 200 35/39, 37/41, 39/43, 48/48, of
        257 39/42, 41/40, 44/45, 56/51, of 1,024 72/41, 76/46, 84/50, 123/80; 17 tokens beside 15 single ones 43/46, 71/45, 117/78, 213/125, 90 beside 63
        86/76, 226/122, 425/221, 823/400; two entries of 40 27/41, 27/41, 33/43, 52/45, sixty-four of 96 156/98, 296/171, 574/301, 1,115/569.  Whole layers over
        17 tokens, 16 heads of 2,048 (42 MB): on the device 31/45, calls one behind the other 73/60, a call waited for 83/93; 24 of 3,072 (94 MB) 47/60, 71/69,
        86/99; 24 of 4,096 (126 MB) 56/70, 71/78, 87/99; 32 of 4,096 (168 MB) 61/73, 72/79, 89/98, over 128 tokens 70/77, 78/84, 99/104, over 250 84/84, 92/90, 112/109.
        And as long as its workspace, 64 KB per head and entry or 128 tokens, is no larger than that of the other forms or 256 MB."""
        s = self.spec
        if step.max_q_len <= 192 and step.num_seqs * s.num_heads * -(-s.v_head_dim // 32) <= ops.sm_count(device):
            weights = 2 * s.hidden_size * (2 * self.qk + 3 * self.vv)
            if weights > 100e6 or torch.cuda.is_initialized() and torch.cuda.is_current_stream_capturing():
                return False
        return once_per_step(step, ("retention.in_tiles", s.num_heads, rotary_dim), lambda: (
            ops.retention_tiles_plan(step, tokens, s.num_heads, rotary_dim, device)[2] <= max(1 << 26, tokens * s.num_heads * 322)))

    def forward(self, x, step, slot, proj=None):
        s = self.spec
        tokens, dev = x.shape[0], x.device
        if self._decay is None or self._decay.device != dev:
            self._decay = torch.tensor([float(g) for g in s.decays], dtype=torch.float32, device=dev)
        inv_freq, rotary_dim = None, 0
        if self.position is not None:
            rope = as_rotary_args(self.position.kernel_args(dev))
            if rope.scale != 1.0:
                raise ValueError("the retention kernels take no factor on cos and sin")
            inv_freq, rotary_dim = rope.inv_freq, rope.rotary_dim
        if proj is None:
            proj = linear(x, self.in_proj)
        silu = s.activation == "silu"
        # a step with a prompt portion takes the recurrence in chunks of 64 tokens (closed form per chunk);
        # steps of single tokens and of short pieces walk it token by token
        chunked = self.chunk_min_tokens is not None and step.max_q_len >= self.chunk_min_tokens
        if (chunked and not silu and self.in_tiles(step, tokens, rotary_dim, dev)
                and ops.retention_tiles_supported(s.head_dim, s.v_head_dim, rotary_dim, proj, slot.state, self.qk, self.vv)):
            out = torch.empty(tokens, self.vv, dtype=x.dtype, device=dev)
            normed = s.output_norm == "per_head"
            o = None if normed else torch.empty(tokens, self.vv, dtype=torch.float32, device=dev)
            ops.retention_tiles(proj, 0, self.qk, 2 * self.qk, 2 * self.qk + self.vv, self.k_scale,
                                (inv_freq, rotary_dim, step.positions) if rotary_dim else None, self._decay, slot.state, step, heads=s.num_heads,
                                head_dim=s.head_dim, v_head_dim=s.v_head_dim, eps=s.norm_eps, **({"out": out} if normed else {"o": o}))
            if not normed:
                ops.retention_out_joint(o, proj, 2 * self.qk + self.vv, self.norm_w, out, eps=s.norm_eps)
            return linear(out, self.o)
        o = torch.empty(tokens, self.vv, dtype=torch.float32, device=dev)
        args = (proj, 2 * self.qk, self._decay, slot.state, step, o)
        sizes = dict(heads=s.num_heads, head_dim=s.head_dim, v_head_dim=s.v_head_dim, silu=silu)
        if not chunked and rotary_dim == 0:      # q and k straight from the projection, as they are staged
            ops.retention_scan(None, None, *args, **sizes, qk=(0, self.qk, self.k_scale))
        elif (chunked and self.in_walk(step, dev) and ops.retention_walk_supported(s.head_dim, s.v_head_dim, rotary_dim, proj, self.qk)
              and (inv_freq is None or inv_freq.data_ptr() % 16 == 0)):
            ops.retention_chunk(None, None, *args, **sizes, qk=(0, self.qk, self.k_scale),
                                rotation=(inv_freq, rotary_dim, step.positions) if rotary_dim else None)
        else:
            q32 = torch.empty(tokens, self.qk, dtype=torch.float32, device=dev)
            k32 = torch.empty(tokens, self.qk, dtype=torch.float32, device=dev)
            ops.retention_prep(proj, 0, self.qk, inv_freq, step.positions, q32, k32, heads=s.num_heads, head_dim=s.head_dim,
                               rotary_dim=rotary_dim, k_scale=self.k_scale, silu=silu)
            (ops.retention_chunk if chunked else ops.retention_scan)(q32, k32, *args, **sizes)
        gated = torch.empty(tokens, self.vv, dtype=x.dtype, device=dev)
        if s.output_norm == "joint":
            ops.retention_out_joint(o, proj, 2 * self.qk + self.vv, self.norm_w, gated, eps=s.norm_eps)
            return linear(gated, self.o)
        ops.retention_out(o, proj, 2 * self.qk + self.vv, gated, heads=s.num_heads, v_head_dim=s.v_head_dim, eps=s.norm_eps)
        return linear(gated, self.o)


class MatrixMemoryMixer(Mixer):
    """``[q | k | v | g | i | f] = in_proj(h)``; per head a matrix memory with exponential gates held stable
    by a running maximum (``config.specs.MatrixMemorySpec``; kernels: csrc/matrix_memory.cu).  The state is
    one 32-bit row per request: ``[heads, head_dim, v_head_dim + 1]`` (the normaliser is the last column),
    then the maximum per head."""
    graph_safe = True
    chunk_min_tokens = 16        # the longest entry of a step from which the chunked kernel runs; None: never
    chunk_tuning_key = "retention_chunk_min_tokens"

    def __init__(self, spec, dtype):
        super().__init__(spec, dtype)
        s = spec
        if min(s.num_heads, s.head_dim, s.v_head_dim, s.hidden_size) <= 0 or not s.gate_cap > 0:
            raise ValueError("the sizes and the gate cap of a matrix memory must be positive")
        if s.head_dim > ops.LIMITS["memory_max_head_dim"]:
            raise ValueError(f"head_dim {s.head_dim} is not supported (at most {ops.LIMITS['memory_max_head_dim']}: "
                             "a state column's rows live in the registers of eight warps)")
        if s.num_heads > ops.LIMITS["grid_dim_yz"]:
            raise ValueError("heads are a grid dimension of the kernels (at most 65,535)")
        self.qk = s.num_heads * s.head_dim
        self.vv = s.num_heads * s.v_head_dim
        self.g_off = 2 * self.qk + self.vv
        self.i_off = self.g_off + self.vv
        self.f_off = self.i_off + s.num_heads
        self.m_off = s.num_heads * s.head_dim * (s.v_head_dim + 1)

    def parameters(self):
        s = self.spec
        return {"in_proj": ParamSpec((self.f_off + s.num_heads, s.hidden_size)),
                "gate_bias": ParamSpec((2 * s.num_heads,), "float32", "bias"),       # input gates, then forget gates
                "norm_w": ParamSpec((self.vv,), "float32", "norm"),
                "o": ParamSpec((s.hidden_size, self.vv))}

    def state_request(self):
        return StateRequest((self.m_off + self.spec.num_heads,), torch.float32)

    # the parameter that projects the mixer's input (a mixer of mixers may stack it with its neighbours' and
    # hand `forward` the product's columns as `proj`)
    input_projection = "in_proj"

    def forward(self, x, step, slot, proj=None):
        s = self.spec
        tokens, dev = x.shape[0], x.device
        if proj is None:
            proj = linear(x, self.in_proj)
        gates = torch.empty(tokens, s.num_heads, 3, dtype=torch.float32, device=dev)
        ops.memory_gates(proj, self.i_off, self.f_off, self.gate_bias, s.gate_cap, slot.state, self.m_off, step, gates,
                         heads=s.num_heads)
        o = torch.empty(tokens, s.num_heads, s.v_head_dim + 1, dtype=torch.float32, device=dev)
        # a step with a prompt portion takes the recurrence in chunks of 64 tokens (closed form per chunk);
        # steps of single tokens and of short pieces walk it token by token
        chunked = self.chunk_min_tokens is not None and step.max_q_len >= self.chunk_min_tokens
        (ops.memory_chunk if chunked else ops.memory_scan)(
            proj, 0, self.qk, 2 * self.qk, gates, s.head_dim ** -0.5, slot.state, step, o, heads=s.num_heads,
            head_dim=s.head_dim, v_head_dim=s.v_head_dim)
        gated = torch.empty(tokens, self.vv, dtype=x.dtype, device=dev)
        ops.memory_out(o, gates, proj, self.g_off, self.norm_w, gated, heads=s.num_heads, v_head_dim=s.v_head_dim,
                       eps=s.norm_eps, den_eps=s.den_eps)
        return linear(gated, self.o)


class MinGRUMixer(Mixer):
    """``[z | x | g] = in_proj(h)``; a gated running average per channel (``config.specs.MinGRUSpec``; kernels:
    csrc/min_gru.cu).  The state is one 32-bit row of ``width`` numbers per request."""
    graph_safe = True
    chunk_min_tokens = 8         # the longest entry of a step from which the chunked kernel runs; None: never
    chunk_tuning_key = "retention_chunk_min_tokens"

    def __init__(self, spec, dtype):
        super().__init__(spec, dtype)
        if min(spec.width, spec.hidden_size) <= 0:
            raise ValueError("the sizes of a minGRU mixer must be positive")
        if -(-spec.width // 64) > ops.LIMITS["grid_dim_yz"]:
            raise ValueError(f"width {spec.width} is not supported (groups of 64 channels are a grid dimension of the kernels)")

    max_step_entries = ops.LIMITS["grid_dim_yz"]

    def parameters(self):
        s = self.spec
        return {"in_proj": ParamSpec((3 * s.width, s.hidden_size)),
                "gate_bias": ParamSpec((2 * s.width,), "float32", "bias"),      # of z, then of x
                "o": ParamSpec((s.hidden_size, s.width))}

    def state_request(self):
        return StateRequest((self.spec.width,), torch.float32)

    def forward(self, x, step, slot):
        proj = linear(x, self.in_proj)
        y = torch.empty(x.shape[0], self.spec.width, dtype=x.dtype, device=x.device)
        # a step with a prompt portion deals a request's tokens out to many warps; steps of single tokens and of
        # short pieces walk them
        chunked = self.chunk_min_tokens is not None and step.max_q_len >= self.chunk_min_tokens
        (ops.min_gru_chunk if chunked else ops.min_gru_scan)(proj, self.gate_bias, slot.state, step, y)
        return linear(y, self.o)


register_mixer("mingru", MinGRUMixer)
register_mixer("matrix_memory", MatrixMemoryMixer)
register_mixer("retention", RetentionMixer)
register_mixer("mamba2", StateSpaceMixer)
register_mixer("channel_delta", GatedDeltaMixer)
