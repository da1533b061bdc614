"""What a program that keeps its recurrent states packed has this framework do, as cases that can be timed and compared.

A decode case is a burst of ``tokens`` decode tokens through ``layers`` layers on ``batch`` slots, launched the way the
case says: as a CUDA graph captured once (how a serving engine decodes; the steps neither allocate nor synchronise) or
call by call (a Hugging Face model on the lockstep container, or an engine's step outside its graphs).  Eight tokens
are one fold period of the default buffer length, so a pass folds every slot exactly once: in ``phase`` 'same' all
slots on the same token (a batch that was prefilled together), in 'mixed' each on a token of its own (continuous
batching).  The prefill case is what surrounds a chunk of prompt: the slots' states are read as fp32, and states of
the same shape are written back packed.

Head counts, head dims, formats and distributions are those of the repository's benchmark, tests and documents; a
tensor-parallel rank holds an integer share of the heads.
"""
import math

import torch

import statequant_b200 as sq
from statequant_b200.kernels import GGAPacked, KDASlotLayout, Mamba2SlotLayout, PackedGDNState, SlotLayout
from statequant_b200.kernels.conv import causal_conv1d_update, split_qkv
from statequant_b200.kernels.gga import StepPlan

M = 8                                       # buffer length of every case (the default everywhere)
WIDTHS = (4, 6, 4, 4, 6, 4)                 # GGA: bits per layer, repeating
FORMATS = {'pace4': (4, 'k', 64), 'int4v': (4, 'v', 32), 'int8k': (8, 'k', 32), 'int8v': (8, 'v', 32)}
DEV = 'cuda'


def _case(name, op, fmt, heads, dims, batch, layers, tokens=M, phase='mixed', graph=True, slots=0):
    return {'name': name, 'op': op, 'fmt': fmt, 'hv': heads[0], 'hk': heads[1], 'dk': dims[0], 'dv': dims[1],
            'batch': batch, 'layers': layers, 'tokens': tokens, 'phase': phase, 'graph': graph, 'slots': slots or batch + 1}


def listed():
    return [
        # one user at the keyboard: a whole 24-layer stack, nothing but latency and launches
        _case('gdn_pace4_b1', 'gdn', 'pace4', (32, 16), (128, 128), 1, 24, phase='same'),
        # a packed Hugging Face model, four sequences in lockstep, fp32 activations, no graph
        _case('gdn_lockstep_b4', 'lockstep', 'pace4', (32, 16), (128, 128), 4, 3, phase='same', graph=False),
        # one rank of four, an odd batch of a lightly loaded server
        _case('gdn_int8k_tp4_b37', 'gdn', 'int8k', (8, 4), (128, 128), 37, 24),
        # the benchmark's batch, all sequences started together
        _case('gdn_int8k_b256', 'gdn', 'int8k', (32, 16), (128, 128), 256, 4, phase='same'),
        # a step with prompts in it runs outside the engine's graphs: convolution, split, step, layer by layer
        _case('gdn_int4v_conv_b192', 'conv_gdn', 'int4v', (32, 16), (128, 128), 192, 4, tokens=2, graph=False),
        # a full node's slot table, half of it running
        _case('gdn_pace4_b4096', 'gdn', 'pace4', (32, 16), (128, 128), 4096, 1, slots=8192),
        # head dims that are not powers of two
        _case('gdn_96x192_pace4_b64', 'gdn', 'pace4', (30, 30), (96, 192), 64, 4),
        # the unquantised control state
        _case('gdn_bf16_b96', 'gdn', 'bf16', (32, 16), (128, 128), 96, 2),
        _case('mamba2_int8k_b256', 'mamba2', 'int8k', (128, 8), (128, 64), 256, 2),
        _case('kda_pace4_b200', 'kda', 'pace4', (32, 32), (128, 128), 200, 4, phase='same'),
        # mixed widths with the pure-write window: every token re-fits the whole state
        _case('gga_window_b64', 'gga', 'gga', (32, 16), (128, 128), 64, 6, tokens=4),
        # chunked prefill: a dozen prompts' states out and back, in the four layers of one pipeline stage's share
        _case('prefill_int8k_b12', 'prefill', 'int8k', (32, 16), (128, 128), 12, 4, tokens=1, graph=False, slots=257),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(['gdn', 'gdn', 'gdn', 'gdn96', 'lockstep', 'conv_gdn', 'mamba2', 'kda', 'gga', 'prefill'])
    share = rng.choice([1, 1, 2, 4])                     # tensor-parallel ranks
    heads, dims, graph, tokens, slots = (32 // share, 16 // share), (128, 128), True, M, 0
    phase = rng.choice(['same', 'mixed', 'mixed'])
    fmt = rng.choice(['pace4', 'int8k', 'int4v', 'int8v', 'bf16'])
    if op == 'gdn':
        batch = log_int(1, 4096)
        if rng.random() < 0.25:
            slots = batch * rng.choice([2, 3]) + 1
    elif op == 'gdn96':
        op, heads, dims, batch = 'gdn', rng.choice([(30, 30), (15, 15), (10, 10)]), (96, 192), log_int(1, 512)
        fmt = rng.choice(['pace4', 'int8k', 'int4v'])
    elif op == 'lockstep':
        batch, phase, graph, heads = log_int(1, 32), 'same', False, (32, 16)
    elif op == 'conv_gdn':
        batch, graph, tokens = log_int(1, 512), False, rng.choice([1, 2])
    elif op == 'mamba2':
        hv, hk = rng.choice([(128, 8), (112, 8), (64, 4), (56, 4), (16, 1)])
        heads, dims, batch, fmt = (hv, hk), (128, 64), log_int(1, 512), rng.choice(['int8k', 'pace4', 'bf16'])
    elif op == 'kda':
        heads, batch, fmt = (32 // share, 32 // share), log_int(1, 1024), rng.choice(['pace4', 'int8k'])
    elif op == 'gga':
        fmt, batch, tokens = 'gga', log_int(1, 512), rng.choice([2, 4])
    else:
        batch, graph, tokens, fmt = log_int(1, 256), False, 1, rng.choice(['pace4', 'int8k', 'int4v', 'bf16'])
        slots = 257
    c = _case('', op, fmt, heads, dims, batch, 1, tokens, phase, graph, slots)
    top = max(work(x)['bytes'] for x in listed())
    c['layers'] = max(1, min(rng.choice([1, 2, 4, 24]), int(top / work(c)['bytes']), 24 if batch <= 64 else 4))
    if op == 'prefill' or op == 'lockstep':
        c['layers'] = min(c['layers'], 4)
    while work(c)['bytes'] > top:
        c['batch'] = c['batch'] * 3 // 4
        c['slots'] = max(257 if op == 'prefill' else 0, c['batch'] + 1)
    del c['name']
    return c


# ---- layouts --------------------------------------------------------------------------------------------------------
def _layout(c):
    fmt = c['fmt'] if c['fmt'] in ('bf16', 'fp32') else sq.Quantizer(*FORMATS[c['fmt']])
    if c['op'] == 'mamba2':
        return Mamba2SlotLayout(fmt, c['hv'], c['hk'], c['dk'], c['dv'], m=M, buffer_bits=8)
    if c['op'] == 'kda':
        return KDASlotLayout(fmt, c['hv'], c['dk'], c['dv'], m=M, buffer_bits=8)
    return SlotLayout(fmt, c['hv'], c['hk'], c['dk'], c['dv'], m=M, buffer_bits=8)


def _gga_state_bytes(c, layer):
    w = WIDTHS[layer % len(WIDTHS)]
    return c['hv'] * (c['dk'] * c['dv'] * w // 8 + 2 * (c['dk'] + c['dv']))


def _io_bytes(c):
    """Activations of one token and layer, inputs and output (bf16; the decays and betas of KDA and the lockstep
    container fp32, that container's vectors too)."""
    hv, hk, dk, dv = c['hv'], c['hk'], c['dk'], c['dv']
    if c['op'] == 'lockstep':
        return 4 * (2 * hk * dk + 2 * hv) + 6 * hv * dv
    if c['op'] == 'kda':
        return 2 * (2 * hv * dk + 2 * hv * dv) + 4 * (hv * dk + hv)
    if c['op'] == 'mamba2':
        return 2 * (2 * hk * dk + 2 * hv * dv + hv)
    io = 2 * (2 * hk * dk + 2 * hv * dv + 2 * hv)
    if c['op'] == 'conv_gdn':                            # the row and three taps of state in, both out again
        io += 2 * (2 * hk * dk + hv * dv) * (1 + 1 + 3 + 3) - 2 * (2 * hk * dk + hv * dv)
    return io


def work(c):
    """Bytes: the stored state read every token and rewritten once a fold period, the live half of the buffer, the
    appended entry, counters, activations and output.  Operations: the two read-outs and the state's update."""
    hv, hk, dk, dv = c['hv'], c['hk'], c['dk'], c['dv']
    n = c['batch'] * c['layers'] * c['tokens']
    cells = hv * dk * dv
    if c['op'] == 'gga':
        state = sum(_gga_state_bytes(c, layer) for layer in range(c['layers'])) / c['layers']
        window = hv * (M * (dk + dv) + 2 * M * 4)
        return {'bytes': n * (2 * state + window + hv * (dk + dv + 4 * M + 4) + _io_bytes(c)), 'flops': n * 8.0 * cells}
    b = _layout(c).breakdown()
    stored = b['S'] + b.get('SC', 0)
    if c['op'] == 'prefill':                             # read and write: packed one way each, fp32 one way each
        return {'bytes': n * 2.0 * (stored + 4 * cells), 'flops': n * 4.0 * cells}
    buf = b['KB'] + b['UB'] + b.get('KBS', 0) + b.get('UBS', 0) + b['GB']
    per = stored * (1 + 1 / M) + buf * (M - 1) / (2 * M) + buf / M + 2 * (b['GCUR'] + b['NPTR']) + _io_bytes(c)
    reads = 1 if c['op'] == 'mamba2' else 2
    return {'bytes': n * float(per), 'flops': n * 2.0 * cells * (reads + 1)}


# ---- inputs ---------------------------------------------------------------------------------------------------------
class _State:
    pass


def _unit(x):
    return x / x.norm(dim=-1, keepdim=True)


def _activations(c, r, layers, tokens):
    """[layers][tokens] tuples of one token's inputs."""
    hv, hk, dk, dv, B = c['hv'], c['hk'], c['dk'], c['dv'], c['batch']
    n = lambda *s: torch.randn(*s, generator=r, device=DEV)                              # noqa: E731

    def one():
        if c['op'] == 'mamba2':
            return n(B, hv, dv).bfloat16(), n(B, hv).bfloat16(), n(B, hk, dk).bfloat16(), n(B, hk, dk).bfloat16()
        if c['op'] == 'kda':
            g = torch.nn.functional.logsigmoid(n(B, hv, dk) + 3.0)
            return (_unit(n(B, hv, dk)).bfloat16(), _unit(n(B, hv, dk)).bfloat16(), n(B, hv, dv).bfloat16(), g,
                    torch.sigmoid(n(B, hv)))
        if c['op'] == 'lockstep':
            return (_unit(n(B * hk, dk)), _unit(n(B * hk, dk)), n(B * hv, dv),
                    torch.nn.functional.logsigmoid(n(B * hv) + 2.0), torch.sigmoid(n(B * hv)))
        if c['op'] == 'conv_gdn':
            return n(B, 2 * hk * dk + hv * dv).bfloat16(), (n(B, hv) - 2.0).bfloat16(), n(B, hv).bfloat16()
        return (_unit(n(B, hk, dk)).bfloat16(), _unit(n(B, hk, dk)).bfloat16(), n(B, hv, dv).bfloat16(),
                (n(B, hv) - 2.0).bfloat16(), n(B, hv).bfloat16())

    return [[one() for _ in range(tokens)] for _ in range(layers)]


def _start_states(c, r, lo, hi, scale=0.5):
    """Value-major fp32 states of rows lo..hi."""
    return torch.randn(hi - lo, c['hv'], c['dv'], c['dk'], generator=r, device=DEV) * scale


def prepare(c, seed):
    r = torch.Generator(device=DEV).manual_seed(seed)
    hv, hk, dk, dv, B, L, T = c['hv'], c['hk'], c['dk'], c['dv'], c['batch'], c['layers'], c['tokens']
    s = _State()
    s.case = c
    if c['op'] == 'lockstep':
        fmt = c['fmt'] if c['fmt'] == 'bf16' else sq.Quantizer(*FORMATS[c['fmt']])
        s.layers = [PackedGDNState(_start_states(c, r, 0, B).transpose(-1, -2), fmt, m=M, hv=hv, hk=hk) for _ in range(L)]
        s.x = _activations(c, r, L, T)
        return s

    s.perm = torch.randperm(c['slots'] - 1, generator=r, device=DEV)[:B]
    s.idx = (s.perm + 1).to(torch.int32)                 # slot 0 is the null block
    if c['op'] == 'gga':
        plan = {layer: (torch.full((hv,), WIDTHS[layer % len(WIDTHS)]), (torch.rand(hv, dk, generator=r, device=DEV) + 0.5).cpu())
                for layer in range(L)}
        s.lay = GGAPacked(StepPlan(plan, 32, name='cases'), hv, hk, dk, dv, pw=True, m=M)
    else:
        s.lay = _layout(c)
    s.blob = torch.zeros(L, c['slots'], s.lay.nbytes, dtype=torch.uint8, device=DEV)
    s.views = [s.lay.views(s.blob[layer]) for layer in range(L)]
    for layer in range(L):
        more = {'layer': layer} if c['op'] == 'gga' else {}
        for lo in range(0, B, 512):
            hi = min(B, lo + 512)
            s.lay.write(s.views[layer], s.idx[lo:hi], _start_states(c, r, lo, hi), **more)
    if c['op'] == 'prefill':
        s.states = [_start_states(c, r, 0, B) for _ in range(L)]                         # what the prompt's kernel hands back
    else:
        s.x = _activations(c, r, L, T)
    n = lambda *z: torch.randn(*z, generator=r, device=DEV)                              # noqa: E731
    s.A_log, s.dt_bias = n(hv) * 0.3, n(hv) * 0.3
    if c['op'] == 'mamba2':
        s.A = -torch.exp(torch.rand(hv, generator=r, device=DEV) * math.log(16.0))
        s.D = n(hv)
        s.dt_bias = torch.rand(hv, generator=r, device=DEV) * 2.0 - 4.0
    s.out = torch.zeros(L, T, B, hv, dv, dtype=torch.bfloat16, device=DEV)
    if c['op'] == 'conv_gdn':
        dim = 2 * hk * dk + hv * dv
        s.conv = (n(L, c['slots'], 3, dim) * 0.5).bfloat16()                             # [line, token, channel]
        s.taps, s.bias = (n(dim, 4) * 0.5).bfloat16(), (n(dim) * 0.1).bfloat16()
        s.row = torch.empty(B, dim, dtype=torch.bfloat16, device=DEV)

    # realistic codes, scales and buffers: a full fold period, then each slot's own share of the next one
    phase = torch.randint(0, M, (B,), generator=r, device=DEV)
    if c['phase'] == 'same':
        phase.zero_()
    warm = _activations(c, r, 1, M)[0]
    scratch = torch.empty(B, hv, dv, dtype=torch.bfloat16, device=DEV)
    for layer in range(L):
        for x in warm:
            _token(s, layer, s.idx, x, scratch)
        for t, x in enumerate(warm[:-1] if c['phase'] == 'mixed' else []):
            _token(s, layer, torch.where(t < phase, s.idx, torch.zeros_like(s.idx)), x, scratch)
    s.graph = None
    if c['graph']:
        keep = s.blob.clone()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _burst(s)                                    # once outside the capture, as an engine warms up
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            _burst(s)
        s.blob.copy_(keep)
    return s


# ---- passes ---------------------------------------------------------------------------------------------------------
def _token(s, layer, idx, x, out):
    """One layer's decode token."""
    c, lay, views = s.case, s.lay, s.views[layer]
    if c['op'] == 'mamba2':
        lay.step(views, idx, *x, out, s.A, D=s.D, dt_bias=s.dt_bias)
    elif c['op'] == 'kda':
        lay.step(views, idx, *x, out)
    elif c['op'] == 'conv_gdn':
        row, a, b = x
        s.row.copy_(row)                                 # stands for the projection that writes the mixed row
        y = causal_conv1d_update(s.row, s.conv[layer].transpose(1, 2), s.taps, s.bias, 'silu', conv_state_indices=idx)
        q, k, v = split_qkv(y, c['hk'], c['dk'], c['hv'], c['dv'])
        lay.step(views, idx, q, k, v, out, c['dk'] ** -0.5, gate=(a, b, s.A_log, s.dt_bias))
    else:
        q, k, v, a, b = x
        more = {'layer': layer} if c['op'] == 'gga' else {}
        lay.step(views, idx, q, k, v, out, c['dk'] ** -0.5, gate=(a, b, s.A_log, s.dt_bias), **more)


def _burst(s):
    for t in range(s.case['tokens']):
        for layer in range(s.case['layers']):
            _token(s, layer, s.idx, s.x[layer][t], s.out[layer, t])


def _fields(s):
    """The stacked layers' state, field by field."""
    if s.case['op'] == 'gga':
        return {'blob': s.blob}
    L, n = s.blob.shape[:2]
    return {name: s.blob[:, :, off:off + nb].view(dt).view(L, n, -1) for name, (off, dt, _, nb) in s.lay.fields.items()}


def run(s):
    c = s.case
    if c['op'] == 'lockstep':
        scale = c['dk'] ** -0.5
        for t in range(c['tokens']):
            for layer, st in enumerate(s.layers):
                st.step(*s.x[layer][t], scale)
        return [dict(out=st.O, codes=st.codes, scales=st.scales, KB=st.KB, UB=st.UB, KBS=st.KBS, UBS=st.UBS, GB=st.GB,
                     GCUR=st.GCUR, NPTR=st.NPTR) for st in s.layers]
    if c['op'] == 'prefill':
        got = []
        for layer in range(c['layers']):
            got.append(s.lay.read(s.views[layer], s.idx))
            s.lay.write(s.views[layer], s.idx, s.states[layer])
        f = _fields(s)
        return {'read': got, **{k: f[k] for k in ('S', 'SC', 'NPTR', 'GCUR') if k in f}}
    if s.graph is not None:
        s.graph.replay()
    else:
        _burst(s)
    got = {'out': s.out, **_fields(s)}
    if c['op'] == 'conv_gdn':
        got['conv'] = s.conv
    return got


def tolerance(c):
    """About four times what the framework's own kernels (tensor-core, staged, generic; register tile, shared tile) differ
    by on the same inputs after three passes.  Their fp32 sums run in another order, which moves a code or a buffered
    value that lies next to a rounding boundary by one step: up to 1.4e-4 of the whole values (an int8 state), 6e-4 of
    the outputs' norm and 0.22 of an output's size (one step of an int4 code); for the GGA state, whose every token
    re-fits all codes, 5.9e-3, 3.1e-3 and 0.36."""
    if c['op'] == 'gga':
        return {'rel': 1.2e-2, 'max': 0.95, 'differ': 1e-2}
    return {'rel': 2.5e-3, 'max': 0.9, 'differ': 6e-4}
