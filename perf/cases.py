"""What users of tremor_b200 have it do, as timed cases: template searches over a resident
record (kNN, threshold, batches of many lengths, serving), the one-shot search of a program
that loads a record and leaves, and the window statistics. Sizes are those of bench.py's
workloads, some with a shorter record, and of the tests.

Records: the generator of tremor_b200/synth.py (AR(2) noise times a slow envelope with
injected chirp events), evaluated on the GPU because records are made many times, with a
few gaps of missing samples as real records have them."""
import math

import numpy as np
import torch

import tremor_b200 as tb
from tremor_b200 import synth

KERNELS = {'auto': tb.KERNEL_AUTO, 'bf16': tb.KERNEL_SPLIT_BF16, 'fp32': tb.KERNEL_FP32}


def listed():
    return [
        # the planner's worker seam: one short template against a rank's small partition;
        # latency, launches and synchronisations
        dict(name='seam_knn', kind='seam', n=1 << 16, m=256, templates=1, mode='knn', k=5, merge=128, gaps=2),
        # the command line's life: load a record, search it once, leave (first pass of all)
        dict(name='one_shot', kind='oneshot', n=(1 << 22) + 12345, m=500, templates=8, mode='threshold', corr=0.75,
             merge=250, gaps=4),
        # the plain kNN workload, host templates in, answers out
        dict(name='plain_knn', kind='call', n=1 << 22, m=1024, templates=16, mode='knn', k=10, merge=512, gaps=0),
        # the plain FP32 kernel, the drop-in form; ragged sizes
        dict(name='plain_fp32', kind='call', n=2000003, m=777, templates=70, mode='threshold', corr=0.8, merge=0,
             gaps=3, kernel='fp32'),
        # the threshold workload, templates prepared once
        dict(name='threshold', kind='batch', n=1 << 25, m=2048, templates=256, mode='threshold', corr=0.8, merge=0,
             gaps=0),
        # the precision workload with the contraction that it names, shorter record
        dict(name='precision_bf16', kind='batch', n=1 << 25, m=4096, templates=128, mode='knn', k=100, merge=0,
             gaps=0, kernel='bf16'),
        # the same as a user has it without choosing a kernel; the largest case
        dict(name='precision_auto', kind='batch', n=1 << 27, m=4096, templates=128, mode='knn', k=100, merge=0,
             gaps=0),
        # the batching workload (its small form): many lengths, kNN and threshold mixed
        dict(name='batching', kind='mixed_batch', n=1 << 25, m_lo=256, m_hi=8192, templates=512, gaps=4),
        # serving (small form): a burst of requests of any length through the server
        dict(name='serving', kind='serve', n=1 << 26, m_lo=128, m_hi=16384, templates=48, gaps=4),
        # few templates of the longest lengths, templates handed over per call
        dict(name='long_templates', kind='call', n=1 << 25, m=16384, templates=8, mode='knn', k=10, merge=8192,
             gaps=0),
        # few templates of 8192
        dict(name='fft_templates', kind='batch', n=1 << 25, m=8192, templates=8, mode='knn', k=10, merge=4096,
             gaps=0),
        # the statistics that the reference keeps per window
        dict(name='window_stats', kind='stats', n=(1 << 20) + 999, m=1000, gaps=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['seam', 'oneshot', 'call', 'call', 'batch', 'batch', 'mixed_batch', 'serve', 'stats'])
    if kind == 'stats':
        m = _log_int(rng, 64, 4096)
        return dict(kind=kind, n=_log_int(rng, 1 << 16, 1 << 21) + m, m=m, gaps=rng.randrange(5))
    if kind in ('mixed_batch', 'serve'):
        lo = _log_int(rng, 100, 1000)
        return dict(kind=kind, n=_log_int(rng, 1 << 19, 1 << 25), m_lo=lo, m_hi=_log_int(rng, 2 * lo, 16384),
                    templates=_log_int(rng, 4, 200 if kind == 'mixed_batch' else 64), gaps=rng.randrange(5))
    m = _log_int(rng, 100, 16384)
    case = dict(kind=kind, m=m, mode=rng.choice(['knn', 'threshold']), gaps=rng.randrange(5))
    if kind == 'seam':
        case.update(n=_log_int(rng, 1 << 16, 1 << 23) + m, templates=1)
    elif kind == 'oneshot':
        case.update(n=_log_int(rng, 1 << 18, 1 << 23) + m, templates=_log_int(rng, 1, 16))
    else:
        kernel = rng.choice(['auto', 'auto', 'auto', 'bf16', 'fp32'])
        top = 1 << (21 if kernel == 'fp32' else 25)
        case.update(n=_log_int(rng, 1 << 18, top) + m, templates=_log_int(rng, 1, 128), kernel=kernel)
    if case['mode'] == 'knn':
        case.update(k=rng.choice([1, 10, 100]), merge=rng.choice([0, m // 2]))
    else:
        # short templates match noise too; the thresholds of use rise as the length falls
        case.update(corr=rng.uniform(0.6, 0.9) if m >= 500 else rng.uniform(0.8, 0.95), merge=rng.choice([0, m // 2]))
    return case


def _templates(case, rng):
    """Chirps of the workload: one length, or lengths log-uniform between two."""
    if 'm' in case:
        return list(synth.chirp_templates(case['templates'], case['m'], rng)) if case['kind'] != 'stats' else []
    lengths = np.exp(rng.uniform(np.log(case['m_lo']), np.log(case['m_hi']), size=case['templates']))
    return [synth.chirp_templates(1, int(m), rng, center_freq=True)[0] for m in np.round(lengths)]


def _record(case, templates, seed, rng):
    n = case['n']
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    g = torch.Generator(device=dev).manual_seed(seed)
    x = torch.randn(n, generator=g, device=dev, dtype=torch.float32)
    # 1 / (1 - 1.6 z + 0.7 z^2) as a product of 1 + 2 Re(p^s) z^s + |p|^2s z^2s, s = 1, 2, 4, ...
    p, s = complex(0.8, math.sqrt(0.06)), 1
    while s <= 64:
        y = x.clone()
        y[s:] += (2.0 * p.real) * x[:-s]
        y[2 * s:] += (abs(p) ** 2) * x[:-2 * s]
        x, p, s = y, p * p, 2 * s
    grid = n // 4096 + 2
    w = np.empty(grid)
    v = 0.0
    for i, step in enumerate(rng.normal(scale=0.05, size=grid)):
        w[i] = v
        v = 0.99 * v + step
    w = torch.from_numpy(w - np.median(w)).to(dev, torch.float32)
    for a in range(0, n, 1 << 24):
        i = torch.arange(a, min(n, a + (1 << 24)), device=dev)
        f = (i & 4095).to(torch.float32) / 4096.0
        x[a:a + (1 << 24)] *= torch.exp(w[i >> 12] * (1.0 - f) + w[(i >> 12) + 1] * f)
    x = x.cpu().numpy()
    for e in range(min(300, max(2, n >> 16))):
        if not templates:
            break
        t = templates[e % len(templates)]
        if len(t) < n:
            synth.inject_events(x, t[None, :], 1, rng) if n < (1 << 20) else _inject(x, t, rng)
    for _ in range(case['gaps']):
        at, length = int(rng.integers(0, n)), int(rng.integers(1, max(2, min(20000, n // 64))))
        x[at:at + length] = tb.MISSING_VALUE
    return x


def _inject(x, t, rng):
    """synth.inject_events for one event, without its pass over the record."""
    off = int(rng.integers(0, len(x) - len(t)))
    local = float(np.std(x[off:off + len(t)]))
    rms = float(np.sqrt(np.mean(t.astype(np.float64) ** 2))) + 1e-30
    x[off:off + len(t)] += (rng.uniform(0.5, 3.0) * local / rms * t).astype(np.float32)


def _requests(case, templates, rng):
    if 'm' not in case:  # as the batching and serving workloads draw them
        return [tb.Request(t, tb.MODE_KNN, k=int(rng.choice([1, 10, 100])), merge_offset=len(t) // 2) if i % 2 == 0
                else tb.Request(t, tb.MODE_THRESHOLD, correlation=float(rng.uniform(0.6, 0.9)))
                for i, t in enumerate(templates)]
    if case['mode'] == 'knn':
        return [tb.Request(t, tb.MODE_KNN, k=case['k'], merge_offset=case['merge']) for t in templates]
    return [tb.Request(t, tb.MODE_THRESHOLD, correlation=case['corr'], merge_offset=case['merge']) for t in templates]


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    templates = _templates(case, rng)
    x = _record(case, templates, seed, rng)
    return x, templates, _requests(case, templates, rng) if case['kind'] != 'stats' else []


def _room(case):
    """Answers that the program's arrays have room for. The number of threshold answers
    depends on the record; the rest of the arrays stays 0."""
    if case.get('mode') == 'knn':
        return case['k'] * case['templates']
    return 1 << 22 if 'm' not in case else 1 << 20


def prepare(case, seed):
    x, templates, requests = _inputs(case, seed)
    state = dict(case=case, x=x, requests=requests)
    room = _room(case)
    state['pos'], state['dist'] = np.zeros(room, np.int64), np.zeros(room, np.float32)
    if case['kind'] in ('seam', 'oneshot', 'call'):
        state['queries'] = np.stack(templates)
    if case['kind'] != 'oneshot':  # the record is resident
        state['ctx'] = ctx = tb.Context(x)
        ctx.set_kernel(KERNELS[case.get('kernel', 'auto')])
        if case['kind'] in ('batch', 'mixed_batch'):
            state['batch'] = ctx.batch(requests)
        elif case['kind'] == 'serve':
            state['server'] = ctx.serve()
    return state


def _joined(state, answers):
    """Answers of all requests one after another in the program's own arrays (positions,
    distances), and how many each request has."""
    counts = np.array([len(a[0]) for a in answers], np.int64)
    if counts.sum() > len(state['pos']):
        state['pos'], state['dist'] = np.zeros(counts.sum(), np.int64), np.zeros(counts.sum(), np.float32)
    np.concatenate([a[0].view(np.int64) for a in answers], out=state['pos'][:counts.sum()])
    np.concatenate([a[1] for a in answers], out=state['dist'][:counts.sum()])
    return state['pos'], state['dist'], counts


def _search(ctx, state):
    case, queries = state['case'], state['queries']
    if case['mode'] == 'knn':
        pos, dist = ctx.search_knn(queries, case['k'], case['merge'])
        return pos.view(np.int64), dist
    return _joined(state, ctx.search_threshold(queries, case['corr'], case['merge']))


def run(state):
    case, kind = state['case'], state['case']['kind']
    if kind == 'seam':
        if case['mode'] == 'knn':
            pos, dist = state['ctx'].scan_knn(state['queries'][0], case['k'], case['merge'])
        else:
            return _joined(state, [state['ctx'].scan_threshold(state['queries'][0], case['corr'], case['merge'])])
        return pos.view(np.int64), dist
    if kind == 'oneshot':
        with tb.Context(state['x']) as ctx:
            return _search(ctx, state)
    if kind == 'call':
        return _search(state['ctx'], state)
    if kind in ('batch', 'mixed_batch'):
        return _joined(state, state['batch'].run())
    if kind == 'stats':
        return state['ctx'].window_stats(case['m'])
    server, done = state['server'], {}
    tickets = [server.submit(r) for r in state['requests']]
    while len(done) < len(tickets):
        for c in server.poll():
            if c.status != 0:
                raise RuntimeError(f'a served request failed ({c.status})')
            done[c.ticket] = c.answers
    return _joined(state, [done[t] for t in tickets])


def _lengths(case):
    """The template lengths, or for lengths drawn from a range their mean quantiles."""
    if 'm' in case:
        return [case['m']] * case['templates']
    q = (np.arange(case['templates']) + 0.5) / case['templates']
    return [int(case['m_lo'] * (case['m_hi'] / case['m_lo']) ** f) for f in q]


def work(case):
    """Bytes: the record and the templates read once, the answers written once (threshold
    answers, whose number depends on the data, are left out). Flops per (template, window)
    pair: the cheaper of the direct dot product and overlap-save transforms of 4 m points, and
    about 8 for the distance and the selection."""
    n = case['n']
    if case['kind'] == 'stats':
        windows = n - case['m'] + 1
        return dict(bytes=4.0 * n + 8.0 * windows, flops=10.0 * windows)
    lengths = _lengths(case)
    flops = 0.0
    for m in lengths:
        flops += (min(2.0 * m, 4.0 / 3.0 * (2.5 * math.log2(4 * m) + 3.0)) + 8.0) * (n - m + 1)
    return dict(bytes=4.0 * n + 4.0 * sum(lengths) + 12.0 * case.get('k', 0) * len(lengths), flops=flops)


# ---- the same answers in 64 bits, by plain torch ---------------------------------------

def _exact_windows(clean, t, pos):
    """FP64 squared z-normalised distances of template t to the windows at pos."""
    m = len(t)
    q = (t - t.mean()) / t.std(correction=0)
    out = torch.empty(len(pos), dtype=torch.float64, device=clean.device)
    step = max(1, (1 << 27) // m)
    i = torch.arange(m, device=clean.device)
    for a in range(0, len(pos), step):
        w = clean[pos[a:a + step, None] + i]
        w = w - w.mean(1, keepdim=True)
        w = w / (w * w).mean(1, keepdim=True).sqrt()
        out[a:a + step] = ((w - q) ** 2).sum(1)
    return out


def _exact_profile(clean, searched, sums, t):
    """FP64 distance of t to every window (inf where the window is not searched)."""
    n, m = len(clean), len(t)
    W = n - m + 1
    q = (t - t.mean()) / t.std(correction=0)
    L = min(1 << 20, 1 << (4 * m + 4096).bit_length())
    S = L - m + 1
    rows = -(-W // S)
    Y = torch.fft.rfft(torch.nn.functional.pad(q, (0, L - m))).conj()
    dot = torch.empty(rows * S, dtype=torch.float64, device=clean.device)
    per = max(1, (1 << 25) // L)
    padded = torch.nn.functional.pad(clean, (0, rows * S + L - n))
    for a in range(0, rows, per):
        b = min(rows, a + per)
        piece = padded[a * S:(b - 1) * S + L].unfold(0, L, S)
        dot[a * S:b * S] = torch.fft.irfft(torch.fft.rfft(piece) * Y, n=L)[:, :S].reshape(-1)
    s1, s2 = sums[0][m:] - sums[0][:W], sums[1][m:] - sums[1][:W]
    var = s2 / m - (s1 / m) ** 2
    d = 2.0 * (m - dot[:W] / var.clamp_min(1e-300).sqrt())
    return torch.where(searched[:W] & (var > 1e-12), d, math.inf)


def exact(case, seed):
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    x, templates, requests = _inputs(case, seed)
    raw = torch.from_numpy(x).to(dev)
    missing = raw == float(tb.MISSING_VALUE)
    clean = torch.where(missing, 0.0, raw.double())
    if case['kind'] == 'stats':
        m = case['m']
        W = len(x) - m + 1
        mean, std = (torch.empty(W, dtype=torch.float64, device=dev) for _ in range(2))
        for a in range(0, W, 1 << 16):
            w = clean[a:min(W, a + (1 << 16)) + m - 1].unfold(0, m, 1)
            mean[a:a + (1 << 16)] = w.mean(1)
            std[a:a + (1 << 16)] = w.std(1, correction=0)
        keep = ~missing[:W]
        return (mean * keep).cpu().numpy(), (std * keep).cpu().numpy()
    # sums of the record about its mean: what they lose to cancellation is far below FP32
    zero = torch.zeros(1, dtype=torch.float64, device=dev)
    sums = [torch.cat([zero, torch.cumsum(v, 0)]) for v in (clean, clean * clean)]
    dists = []
    for r in requests:
        t = torch.from_numpy(r.template).to(dev).double()
        d = _exact_profile(clean, ~missing, sums, t)
        if r.mode == tb.MODE_KNN:
            pos = []
            for _ in range(r.k):
                j = int(torch.argmin(d))
                if not math.isfinite(float(d[j])):
                    return None  # fewer answers than asked for: padding, no computed numbers
                pos.append(j)
                d[max(0, j - max(1, r.merge_offset) + 1):j + max(1, r.merge_offset)] = math.inf
            got = _exact_windows(clean, t, torch.tensor(pos, device=dev)).sort().values
        else:
            limit = 2.0 * len(t) * (1.0 - r.correlation)
            pos = torch.nonzero(d <= limit).flatten()
            if len(pos) * len(t) > 1 << 34 or bool(((d - limit).abs() < 2e-6 * limit).any()):
                return None  # hundreds of thousands of matches, or one that FP32 cannot decide
            if r.merge_offset > 0:
                kept, last = [], -1 << 60
                for p in pos.tolist():
                    if p >= last + r.merge_offset + 1:
                        kept.append(p)
                        last = p
                pos = torch.tensor(kept, dtype=torch.int64, device=dev)
            got = _exact_windows(clean, t, pos)
        dists.append(got.cpu().numpy())
    if case['kind'] == 'seam' and case['mode'] == 'knn':
        return None, dists[0]
    if case['kind'] in ('call', 'oneshot') and case['mode'] == 'knn':
        return None, np.stack(dists)
    found = np.concatenate(dists)
    return None, np.pad(found, (0, max(0, _room(case) - len(found)))), None
