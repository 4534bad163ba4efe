"""What a user of this framework has it do, as cases that can be timed and checked.

A case is a dict of plain values. ``prepare(case, seed)`` makes what a
program has in hand before the call (recordings, templates, a handle),
``run(state)`` is one pass through the public entry points, ``work(case)`` the
bytes and operations the path cannot do without, and ``exact(case, seed)`` the
same outputs from plain torch in 64 bits where they are defined by the inputs
alone.

Kinds of cases:

* ``batch``: one batch of int16 rows sorted into spike records
  (``Sorter.sort_batch``, or ``sort_batch_async`` from device or pinned rows,
  with the batch's drift correction set before it);
* ``stream``: a block of samples pushed to each probe of a ``ProbeServer`` and
  its records polled (the serving loop's latency path);
* ``match``: ``Sorter.match`` on a filtered batch (Kilosort's ``run_matching``:
  spikes, amplitudes and the residual);
* ``filter``: ``Sorter.filter`` (CAR, highpass, whitening, drift);
* ``scores``: ``Sorter.scores`` (template score field of a filtered batch);
* ``recon``: the differentiable reconstruction, forward and backward, as in
  template refinement.

Recordings follow the generator of ``livespikesorter_b200.synth`` (biphasic
units with Gaussian footprints, Poisson trains, white and 1/f noise, int16 at
0.195 uV/bit), written for the GPU so that making them is quick.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from livespikesorter_b200 import adjoint
from livespikesorter_b200 import setup_tensors as st
from livespikesorter_b200 import synth
from livespikesorter_b200.serve import ProbeServer
from livespikesorter_b200.sorter import Sorter

FS = 30000
UV_PER_BIT = 0.195
TH = 8.0
NT0MIN = 20
N_NEAREST = 10
DRIFT_UM = 4.0      # footprint shift of a drifting recording, corrected by its drift matrix


# ------------------------------------------------------------------- the cases
def _batch(name, C, T, NT, *, precision='fp32', io='host', drift=False, post=False, first=False, dup=0.0, K=6, nt=61):
    c = dict(kind='batch', C=C, T=T, NT=NT, precision=precision, io=io, drift=drift, post=post, first=first, dup=dup,
             K=K, nt=nt)
    return dict(c, name=name) if name else c


def _stream(name, C, Ts, blocks):
    c = dict(kind='stream', C=C, Ts=','.join(map(str, Ts)), blocks=','.join(map(str, blocks)))
    return dict(c, name=name) if name else c


def listed():
    return [
        # a 64-channel probe with 32 units, a 2-s batch handed over from host memory, records back on the host
        _batch('batch 64ch 32t', 64, 32, 60000),
        # a Neuropixels-like probe, 400 templates, drift corrected per batch, rows already on the GPU
        _batch('batch 384ch 400t drift', 384, 400, 60000, io='device', drift=True),
        # 800 templates with near-duplicates, BF16 scores with FP32 re-check, rows uploaded from pinned memory
        _batch('batch 384ch 800t bf16', 384, 800, 60000, precision='bf16', io='pinned', drift=True, dup=0.1),
        # the first batch of a recording (replicated lead, zero tail), synchronous, with positions, clusters,
        # duplicate removal and time order
        _batch('batch 384ch 800t first post', 384, 800, 60000, post=True, first=True),
        # the shortest blocks of the serving loop: 10 ms of one probe with 800 templates
        _stream('stream 800t 300', 384, (800,), (300,)),
        # the serving rig: four probes, 100 ms down to 10 ms blocks
        _stream('stream four probes', 384, (200, 400, 600, 800), (3000, 1500, 600, 300)),
        # run_matching on a filtered batch of odd length, with the residual
        dict(kind='match', name='match 96ch 150t', C=96, T=150, N=30011, K=6, nt=61),
        # preprocessing alone: the whitened, drift-corrected batch
        dict(kind='filter', name='filter 384ch', C=384, NT=60000, drift=True, nt=61),
        # the score field alone
        dict(kind='scores', name='scores 384ch 400t', C=384, T=400, N=60122, K=6, nt=61, precision='fp32'),
        # template refinement: one batch's reconstruction and its gradients
        dict(kind='recon', name='recon 384ch 400t', C=384, T=400, N=60000, K=6, nt=61, spikes=9000, dtype='float32'),
        # the small double-precision copy that gradients are checked on
        dict(kind='recon', name='recon 8ch 4t float64', C=8, T=4, N=3000, K=6, nt=61, spikes=30, dtype='float64'),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['batch', 'batch', 'batch', 'stream', 'match', 'filter', 'scores', 'recon'])
    C = _log_int(rng, 32, 384)
    T = _log_int(rng, 16, 800)
    K = rng.choice([4, 5, 6, 6, 6, 8])
    nt = rng.choice([41, 61, 61, 61, 81])
    if kind == 'batch':
        post = rng.random() < 0.25
        # post-processing carries state from batch to batch, which the first batch resets
        return _batch(None, C, T, _log_int(rng, 3000, 60000), precision=rng.choice(['fp32', 'bf16']),
                      io='host' if post else rng.choice(['host', 'device', 'pinned']), drift=rng.random() < 0.5,
                      post=post, first=post or rng.random() < 0.2, K=K, nt=nt)
    if kind == 'stream':
        return _stream(None, C, (T,), (_log_int(rng, 300, 3000),))
    if kind == 'match':
        return dict(kind='match', C=C, T=T, N=_log_int(rng, 3000, 60000), K=K, nt=nt)
    if kind == 'filter':
        return dict(kind='filter', C=C, NT=_log_int(rng, 3000, 60000), drift=rng.random() < 0.5, nt=nt)
    if kind == 'scores':
        return dict(kind='scores', C=C, T=T, N=_log_int(rng, 3000, 60000), K=K, nt=nt,
                    precision=rng.choice(['fp32', 'bf16']))
    N = _log_int(rng, 3000, 60000)
    return dict(kind='recon', C=C, T=T, N=N, K=K, nt=nt, spikes=max(8, int(N * T / 2700 * rng.uniform(0.5, 1.0))),
                dtype=rng.choice(['float32', 'float32', 'float64']))


# ------------------------------------------------------------- synthetic inputs
def _gen(seed):
    return torch.Generator(device='cuda').manual_seed(int(seed))


def _probe(C):
    return synth.probe_two_column(C) if C <= 64 else synth.probe_staggered(C)


@functools.lru_cache(maxsize=None)
def _hp():
    return st.get_highpass_filter(FS, 300)


@functools.lru_cache(maxsize=None)
def _geometry(C):
    """(probe, iCC [nC, C], iKxx): per-probe tables."""
    p = _probe(C)
    ds = (p.xc - p.xc[:, None]) ** 2 + (p.yc - p.yc[:, None]) ** 2
    return p, torch.from_numpy(np.argsort(ds, 0)[:N_NEAREST].copy()), st.inv_kernel(p.xc, p.yc, 20.0)


def _drift_matrix(C, shift):
    p, _, iK = _geometry(C)
    return st.get_drift_matrix(p.xc, p.yc, shift, iK).float()


def _highpass64(X):
    """fft_highpass of X [C, n] in 64 bits: the impulse response padded or cropped to n."""
    hp, n = _hp().double(), X.shape[1]
    ft = hp.shape[0]
    if ft < n:
        pad = (n - ft) // 2
        hp = torch.cat((torch.zeros(pad, dtype=hp.dtype), hp, torch.zeros(n - pad - ft, dtype=hp.dtype)))
    elif ft > n:
        crop = (ft - n) // 2
        hp = hp[crop:crop + n]
    fw = torch.fft.fft(hp.to(X.device))
    return torch.fft.fftshift(torch.real(torch.fft.ifft(torch.fft.fft(X.double()) * torch.conj(fw))), dim=-1)


def _noise(g, n, C):
    """Background in uV [n, C]: 10 uV RMS, white with a 1/f component."""
    white = torch.randn(n, C, generator=g, device='cuda') * 9.0
    f = torch.fft.rfftfreq(n, device='cuda')
    f[0] = f[1]
    spec = torch.complex(*(torch.randn(len(f), C, generator=g, device='cuda') for _ in range(2))) / f.sqrt()[:, None]
    pink = torch.fft.irfft(spec, n, dim=0)
    return white + pink * (4.4 / pink.std())


def _whitening(C, seed):
    """Local ZCA (32 nearest channels) of the filtered noise covariance."""
    p, _, _ = _geometry(C)
    X = (_noise(_gen(seed), 16384, C) / UV_PER_BIT).round().T.double()
    X = X - X.mean(1, keepdim=True)
    X = X - X.median(0)[0]
    X = _highpass64(X)[:, 61:-61]
    CC = X @ X.T / X.shape[1]
    ds = (p.xc - p.xc[:, None]) ** 2 + (p.yc - p.yc[:, None]) ** 2
    ix = torch.from_numpy(np.argsort(ds, 1, kind='stable')[:, :min(32, C)].copy()).cuda()
    D, E = torch.linalg.eigh(CC[ix[:, :, None], ix[:, None, :]])
    W = (E / (D + 1e-6).sqrt()[:, None, :]) @ E.transpose(1, 2)
    out = torch.zeros(C, C, dtype=torch.float64, device='cuda')
    out.scatter_(1, ix, W[:, 0, :])
    return out


def _units(C, T, nt, g, dup=0.0):
    """Unit parameters: waveforms [T, nt], centres, rates."""
    p, _, _ = _geometry(C)
    u = torch.rand(4, T, generator=g, device='cuda', dtype=torch.float64)
    cx = p.xc.min() + u[0] * (p.xc.max() - p.xc.min())
    cy = p.yc.min() + u[1] * (p.yc.max() - p.yc.min())
    m = torch.arange(nt, device='cuda', dtype=torch.float64)
    sig, lobe = 0.3e-3 * FS / 2.355, NT0MIN + 0.5e-3 * FS
    w = -torch.exp(-(m - NT0MIN) ** 2 / (2 * sig ** 2)) + torch.exp(-(m - lobe) ** 2 / (2 * (2 * sig) ** 2)) / 3.0
    w = w + 0.05 * torch.randn(T, nt, generator=g, device='cuda', dtype=torch.float64)
    n_dup = int(round(dup * T / 2))
    if n_dup:
        # near-duplicate pairs: footprint centres 10 um apart, nearly the same waveform
        a, b = slice(0, 2 * n_dup, 2), slice(1, 2 * n_dup, 2)
        ang = 2 * math.pi * u[3, :n_dup]
        cx[b], cy[b] = cx[a] + 10.0 * ang.cos(), cy[a] + 10.0 * ang.sin()
        w[b] = w[a] + 0.05 * torch.randn(n_dup, nt, generator=g, device='cuda', dtype=torch.float64)
    w = w / w[:, NT0MIN:NT0MIN + 1].abs()
    return dict(waves=w, cx=cx, cy=cy, rates=2.0 + 18.0 * u[2])


def _footprints(C, units, shift=0.0):
    p, _, _ = _geometry(C)
    xc, yc = (torch.from_numpy(np.asarray(v, np.float64)).cuda() for v in (p.xc, p.yc))
    d2 = (xc - units['cx'][:, None]) ** 2 + (yc - units['cy'][:, None] - shift) ** 2
    return torch.exp(-d2 / (2 * 30.0 ** 2))


def _templates(C, T, K, nt, units, Wrot):
    """(U [T, K, C], wPCA [K, nt]) float32: whitened footprints on the SVD basis of the filtered waveforms."""
    pad = torch.zeros(T, 4096, device='cuda', dtype=torch.float64)
    at = 2048 - nt // 2
    pad[:, at:at + nt] = units['waves']
    wf = _highpass64(pad)[:, at:at + nt]
    # basis vectors ordered and signed so that they do not depend on the solver's choices
    ev, V = torch.linalg.eigh(wf.T @ wf)
    W = V.T.flip(0)[:K]
    top = W.gather(1, W.abs().argmax(1, keepdim=True))
    W = W * -torch.sign(top)
    U = (wf @ W.T)[:, :, None] * (_footprints(C, units) @ Wrot.T)[:, None, :] * (80.0 / UV_PER_BIT)
    return U.float().contiguous(), W.float().contiguous()


def _ctc(U, W):
    """Template cross-correlations [T, T, 2nt+1] (prepare_matching), summed in 64 bits."""
    T, K, C = U.shape
    nt = W.shape[1]
    W64 = W.double()
    Wp = torch.nn.functional.pad(W64, (nt, nt)).unfold(1, nt, 1)          # [K, 2nt+1, nt]
    WtW = torch.einsum('kla,ma->kml', Wp, W64).flip(2)
    U64 = U.double().reshape(T * K, C)
    out = torch.empty(T, T, 2 * nt + 1, device=U.device)
    for i in range(0, T, 100):                                             # 100 templates at a time
        n = min(100, T - i)
        UtU = (U64[i * K:(i + n) * K] @ U64.T).reshape(n, K, T, K).permute(0, 2, 1, 3).reshape(n * T, K * K)
        out[i:i + n] = (UtU @ WtW.reshape(K * K, -1)).float().reshape(n, T, -1)
    return out


def _spikes(units, T, L, g):
    """Poisson trains with a 1.5 ms refractory period: (time, unit, amplitude in uV), sorted by unit and time."""
    n = torch.poisson(units['rates'] * (L / FS), generator=g).long()
    unit = torch.repeat_interleave(torch.arange(T, device='cuda'), n)
    t = (torch.rand(len(unit), generator=g, device='cuda', dtype=torch.float64) * L).long()
    o = torch.argsort(unit * (L + 1) + t, stable=True)
    unit, t = unit[o], t[o]
    keep = torch.ones_like(unit, dtype=torch.bool)
    keep[1:] = (unit[1:] != unit[:-1]) | (t[1:] - t[:-1] >= 45)
    amp = 80.0 * torch.exp(0.3 * torch.randn(len(unit), generator=g, device='cuda', dtype=torch.float64))
    return t[keep], unit[keep], amp[keep]


def _render(C, T, L, nt, units, g, shift=0.0):
    """int16 rows [L, C] of a recording with footprints shifted by ``shift`` um."""
    t, unit, amp = _spikes(units, T, L, g)
    S = torch.zeros((L + 2 * nt) * T, device='cuda')
    rows = (t - NT0MIN + nt)[:, None] + torch.arange(nt, device='cuda')
    # trains are refractory, so at most two waveforms of a unit meet in a sample: the sums have one value
    S.index_add_(0, (rows * T + unit[:, None]).reshape(-1), (amp[:, None] * units['waves'][unit]).float().reshape(-1))
    x = S.reshape(L + 2 * nt, T)[nt:nt + L] @ _footprints(C, units, shift).float() + _noise(g, L, C)
    return (x / UV_PER_BIT).round().clamp(-32768, 32767).to(torch.int16)


def _setup(C, T, K, nt, seed, dup=0.0):
    """Sorter arguments of one probe (host tensors), its units and what they were made from."""
    g = _gen(seed)
    units = _units(C, T, nt, g, dup)
    Wrot = _whitening(C, seed + 1)
    U, W = _templates(C, T, K, nt, units, Wrot)
    p, iCC, _ = _geometry(C)
    iU = (U ** 2).sum(1).argmax(-1).cpu()
    Uh = U.cpu()
    kw = dict(U=Uh, wPCA=W.cpu(), ctc=_ctc(U, W).cpu(), Wrot=Wrot.float().cpu(), hp_filter=_hp(), iCC=iCC, iU=iU,
              Ucc=Uh[torch.arange(T), :, iCC[:, iU]].contiguous(), nt0min=NT0MIN, Th=TH)
    return kw, units


def _filtered(C, T, N, U, W, spikes, g):
    """A filtered, whitened batch X [C, N]: unit noise plus spikes of the templates; and its spikes (x, y, amp), in
    distinct columns and with whole windows."""
    nt = W.shape[1]
    h = nt // 2
    x = (torch.randperm(N - 2 * h, generator=g, device='cuda')[:spikes] + h).sort()[0]
    y = torch.randint(0, T, (spikes,), generator=g, device='cuda')
    a = torch.exp(0.3 * torch.randn(spikes, generator=g, device='cuda', dtype=torch.float64))
    X = torch.randn(C, N, generator=g, device='cuda')
    X += _reconstruct64(U.double(), W.double(), x, y, a, N).float()
    return X.contiguous(), x, y, a


def _reconstruct64(U, W, x, y, a, N):
    """R[c, s] = sum_i a_i sum_k U[y_i, k, c] W[k, s - x_i + nt/2], columns outside [0, N) dropped."""
    T, K, C = U.shape
    nt = W.shape[1]
    # trains A[t, s] and one correlation per (component, lag): deterministic, differentiable in U, W and a
    A = torch.zeros(T, N + 2 * nt, device=U.device, dtype=U.dtype).index_put((y, x + nt), a)
    R = torch.zeros(C, N, device=U.device, dtype=U.dtype)
    for k in range(K):
        V = U[:, k, :].T @ A                                               # [C, N + 2nt]
        Z = torch.nn.functional.unfold(V[:, None, None, nt - nt // 2:nt + N + nt // 2], (1, nt))
        R = R + torch.einsum('cms,m->cs', Z, W[k].flip(0))
    return R


# ---------------------------------------------------------------------- prepare
def _store(cap, K, device, post=False):
    """Where a program collects the spikes it gets."""
    kw = dict(device=device)
    d = dict(time=torch.zeros(cap, dtype=torch.int64, **kw), template=torch.zeros(cap, dtype=torch.int32, **kw),
             amplitude=torch.zeros(cap, **kw), pc=torch.zeros(cap, N_NEAREST, K, **kw))
    if post:
        d.update(x=torch.zeros(cap, **kw), y=torch.zeros(cap, **kw), cluster=torch.zeros(cap, dtype=torch.int32, **kw))
    return d


def _collect(store, rec):
    """The batch's records into the store; they come first, whatever was there before follows."""
    n = len(rec['time'])
    for k, v in store.items():
        v[:n].copy_(torch.as_tensor(rec[k]))
    return dict(store, count=n)


def prepare(case, seed):
    return globals()['_prepare_' + case['kind']](case, seed)


def _prepare_batch(c, seed):
    C, T, NT, nt = c['C'], c['T'], c['NT'], c['nt']
    kw, units = _setup(C, T, c['K'], nt, seed, c['dup'])
    s = Sorter(**kw, NT=NT, precision=c['precision'])
    shift = DRIFT_UM if c['drift'] else 0.0
    n_rows = NT + nt if c['first'] else NT + 2 * nt
    rows = _render(C, T, n_rows, nt, units, _gen(seed + 2), shift)
    state = dict(kind='batch', sorter=s, M=_drift_matrix(C, -shift) if c['drift'] else None, ibatch=0 if c['first'] else 1,
                 io=c['io'])
    cap = 4096 + int(NT * T / 1800)
    if c['io'] == 'host':
        state['rows'] = rows.cpu().numpy()
        state['store'] = _store(cap, c['K'], 'cpu', c['post'])
    else:
        state['rows'] = rows if c['io'] == 'device' else rows.cpu().pin_memory()
        # a ring entry that the program keeps: device records, or pinned ones that the batch writes across the bus
        rec = s.records(capacity=cap, pinned=c['io'] == 'pinned')
        for v in rec.values():
            v.zero_()
        state['records'] = rec
    if c['post']:
        p, _, _ = _geometry(C)
        s.set_postprocess(xc=p.xc, yc=p.yc, dt=7)
    return state


def _prepare_stream(c, seed):
    Ts, blocks = ([int(v) for v in c[k].split(',')] for k in ('Ts', 'blocks'))
    srv = ProbeServer(memory_budget=40 << 30, max_probes=4)
    probes = []
    for i, (T, block) in enumerate(zip(Ts, blocks)):
        kw, units = _setup(c['C'], T, 6, 61, seed + 31 * i)
        n = 8
        rows = _render(c['C'], T, n * block, 61, units, _gen(seed + 31 * i + 2)).cpu().numpy()
        pid = srv.admit(depth=4, capacity=8192, NT=block, **kw)
        probes.append(dict(pid=pid, rows=rows, block=block, n=n, k=0, store=_store(8192, 6, 'cpu')))
    return dict(kind='stream', server=srv, probes=probes)


def _prepare_match(c, seed):
    kw, _ = _setup(c['C'], c['T'], c['K'], c['nt'], seed)
    s = Sorter(**kw, NT=c['N'] - 2 * c['nt'])
    X, _, _, _ = _filtered(c['C'], c['T'], c['N'], kw['U'].cuda(), kw['wPCA'].cuda(),
                           max(4, int(c['N'] * c['T'] / 2700)), _gen(seed + 2))
    cap = 4096 + c['N'] * c['T'] // 1800
    return dict(kind='match', sorter=s, X=X, st=torch.zeros(cap, 2, dtype=torch.int64, device='cuda'),
                amps=torch.zeros(cap, 1, device='cuda'))


def _prepare_filter(c, seed):
    C, nt, T = c['C'], c['nt'], 16
    kw, units = _setup(C, T, 6, nt, seed)
    s = Sorter(**kw, NT=c['NT'], drift=_drift_matrix(C, -DRIFT_UM) if c['drift'] else None)
    rows = _render(C, T, c['NT'] + 2 * nt, nt, units, _gen(seed + 2), DRIFT_UM if c['drift'] else 0.0)
    return dict(kind='filter', sorter=s, rows=rows, Wrot=kw['Wrot'])


def _prepare_scores(c, seed):
    kw, _ = _setup(c['C'], c['T'], c['K'], c['nt'], seed)
    s = Sorter(**kw, NT=c['N'] - 2 * c['nt'], precision=c['precision'])
    X, _, _, _ = _filtered(c['C'], c['T'], c['N'], kw['U'].cuda(), kw['wPCA'].cuda(),
                           max(4, int(c['N'] * c['T'] / 2700)), _gen(seed + 2))
    return dict(kind='scores', sorter=s, X=X, U=kw['U'], W=kw['wPCA'])


def _recon_inputs(c, seed):
    dt = getattr(torch, c['dtype'])
    g = _gen(seed)
    units = _units(c['C'], c['T'], c['nt'], g)
    U, W = _templates(c['C'], c['T'], c['K'], c['nt'], units, _whitening(c['C'], seed + 1))
    # the data come from templates with other footprints, so that there is a residual to descend on
    U1 = (_footprints(c['C'], units, 10.0) / _footprints(c['C'], units).clamp_min(1e-12)).clamp(0.5, 2.0)
    X, x, y, a = _filtered(c['C'], c['T'], c['N'], U * U1[:, None, :].float(), W, c['spikes'], _gen(seed + 2))
    return dict(X=X.to(dt), U=U.to(dt), W=W.to(dt), x=x.to(torch.int32), y=y.to(torch.int32), amp=a.to(dt))


def _prepare_recon(c, seed):
    d = _recon_inputs(c, seed)
    for k in ('U', 'W', 'amp'):
        d[k].requires_grad_(True)
    return dict(d, kind='recon')


# -------------------------------------------------------------------------- run
def run(state):
    return globals()['_run_' + state['kind']](state)


def _run_batch(s):
    h = s['sorter']
    if s['M'] is not None:
        h.set_drift(s['M'])
    if s['io'] == 'host':
        return _collect(s['store'], h.sort_batch(s['rows'], s['ibatch'], 1000))
    return h.sort_batch_async(s['rows'], s['ibatch'], 1000, out=s['records'])


def _run_stream(s):
    srv, out = s['server'], {}
    for p in s['probes']:
        k = p['k'] % p['n']
        p['k'] += 1
        srv.push(p['pid'], p['rows'][k * p['block']:(k + 1) * p['block']])
    for i, p in enumerate(s['probes']):
        batch, rec = srv.poll(p['pid'], wait=True)
        out['probe%d' % i] = _collect(p['store'], rec)
    return out


def _run_match(s):
    st_, amps, xres = s['sorter'].match(s['X'])
    n = len(st_)
    s['st'][:n].copy_(st_)
    s['amps'][:n].copy_(amps)
    return dict(st=s['st'], amps=s['amps'], xres=xres, count=n)


def _run_filter(s):
    return s['sorter'].filter(s['rows'], 1, 1000)


def _run_scores(s):
    return s['sorter'].scores(s['X'])


def _run_recon(s):
    R = adjoint.reconstruct(s['U'], s['W'], s['x'], s['y'], s['amp'], s['X'].shape[1])
    loss = 0.5 * (s['X'] - R).square().sum()
    dU, dW, damp = torch.autograd.grad(loss, (s['U'], s['W'], s['amp']))
    return dict(R=R.detach(), loss=loss.detach(), dU=dU, dW=dW, damp=damp)


# ------------------------------------------------------------------------- work
def _sort_work(C, T, N, K, nt, spikes):
    """Rows in, templates and their cross-correlations read once, records out; the projection, the scores and the
    subtraction of every spike's cross-correlations."""
    L2 = 2 * nt + 1
    return dict(bytes=2 * C * N + 4 * T * K * C + 4 * T * T * L2 + spikes * (16 + 4 * N_NEAREST * K),
                flops=2 * N * (C * K * nt + T * K * C) + 2 * spikes * T * L2)


def work(case):
    c, kind = case, case['kind']
    if kind == 'batch':
        N = c['NT'] + 2 * c['nt']
        return _sort_work(c['C'], c['T'], N, c['K'], c['nt'], int(11.0 * c['T'] * N / FS))
    if kind == 'stream':
        tot = dict(bytes=0, flops=0)
        for T, b in zip(*([int(v) for v in c[k].split(',')] for k in ('Ts', 'blocks'))):
            w = _sort_work(c['C'], T, b + 122, 6, 61, int(11.0 * T * b / FS))
            # a short block meets a fraction of the templates' cross-correlations
            w['bytes'] = 2 * c['C'] * b + 4 * T * 6 * c['C'] + int(11.0 * T * b / FS) * (256 + 4 * T * 123)
            tot = {k: tot[k] + w[k] for k in tot}
        return tot
    C, nt = c['C'], c['nt']
    if kind == 'filter':
        N = c['NT'] + 2 * nt
        return dict(bytes=2 * C * N + 4 * C * N + 8 * C * C, flops=2 * C * C * N + 10 * C * N * math.log2(N))
    T, N, K = c['T'], c['N'], c['K']
    if kind == 'match':
        w = _sort_work(C, T, N, K, nt, int(N * T / 2700))
        return dict(bytes=w['bytes'] - 2 * C * N + 8 * C * N, flops=w['flops'])
    if kind == 'scores':
        return dict(bytes=4 * C * N + 4 * T * K * C + 4 * T * N, flops=2 * N * (C * K * nt + T * K * C))
    e, n = (8 if c['dtype'] == 'float64' else 4), c['spikes']
    # X and R in, R and the gradients out; the waveforms are separable: K components per (spike, channel, lag), both ways
    return dict(bytes=e * (3 * C * N + 2 * T * K * C + 2 * n), flops=2 * n * C * nt * K * 3 + 3 * C * N)


# ------------------------------------------------------------------------ exact
def exact(case, seed):
    """The outputs in 64 bits; None for kinds whose outputs follow greedy decisions (spike sequences and what hangs on
    them), which another rounding of the scores may take differently."""
    kind = case['kind']
    if kind == 'filter':
        s = _prepare_filter(case, seed)
        X = s['rows'].T.double()
        X = X - X.mean(1, keepdim=True)
        X = X - X.sort(0)[0][(X.shape[0] - 1) // 2]
        M = s['Wrot'].double().cuda()
        if case['drift']:
            M = _drift_matrix(case['C'], -DRIFT_UM).double().cuda() @ M
        return M @ _highpass64(X)
    if kind == 'scores':
        s = _prepare_scores(case, seed)
        X, U, W = s['X'].double(), s['U'].double().cuda(), s['W'].double().cuda()
        h, N = W.shape[1] // 2, X.shape[1]
        Xp = torch.nn.functional.pad(X, (h, h))
        B = torch.zeros(U.shape[0], N, device='cuda', dtype=torch.float64)
        for k in range(U.shape[1]):
            P = sum(W[k, m] * Xp[:, m:m + N] for m in range(W.shape[1]))
            B += U[:, k, :] @ P
        return B
    if kind == 'recon':
        d = _recon_inputs(case, seed)
        U, W, a = (d[k].detach().double().requires_grad_(True) for k in ('U', 'W', 'amp'))
        x, y, X = d['x'].long(), d['y'].long(), d['X'].double()
        T, K, C = U.shape
        nt, N = W.shape[1], X.shape[1]
        with torch.no_grad():
            R = _reconstruct64(U, W, x, y, a, N)
            G = torch.nn.functional.pad(R - X, (nt // 2, nt // 2))          # dL/dR
            dU, dW, damp = torch.zeros_like(U), torch.zeros_like(W), torch.zeros_like(a)
            lag = torch.arange(nt, device='cuda')
            for i in range(0, len(x), 256):
                xi, yi, ai = x[i:i + 256], y[i:i + 256], a[i:i + 256]
                g = G[:, xi[:, None] + lag]                                  # [C, n, nt]
                P = torch.einsum('cnm,km->nkc', g, W)
                dU.index_add_(0, yi, ai[:, None, None] * P)
                damp[i:i + 256] = (U[yi] * P).sum((1, 2))
                dW += torch.einsum('nkc,cnm->km', ai[:, None, None] * U[yi], g)
        return dict(R=R, loss=0.5 * (X - R).square().sum(), dU=dU, dW=dW, damp=damp)
    return None
