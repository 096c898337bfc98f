"""The algebra of the two- and four-step passes of the recorded step graphs, restated in numpy (float64) on
random data, which step of a call goes in which pass, and the autotuner's option-set numbering.

Face pairs (step.cu: group_conv + group_fix): a centre's convolution at time t is
    sum_j sum_k ( -s_jk N_j[t-k] + d_jk D_j[t-k] ),  k = 0..15, with D_j[t] (unknown) left out.
At time t+1 every term is known before step t except d_j1 D_j[t]; the pass computes the rest from
the time-t windows shifted by one tap (tap -1 = N[t+1]) and adds sum_j d_j1 D_j[t] afterwards.

A four-step pass computes times t .. t+3 so: step t+j leaves out d_j1 D[t+j-1] .. d_jj D[t], which are added
when those D are known (taps 1..j with the D of the pass's steps).

Grid-cache records (step.cu: near_terms2, near_terms4 + near_terms_complete): BEM-near terms pair record tap m
with history tap m, FDTD-near terms with history tap m-1; at time t+1 the only unknown product is
the one with D[t+1] (record tap 0, resp. 1), added from one factor per record afterwards; at time t+j of a
four-step pass those with D[t+j] .. D[t+1] (record taps 0..j-1, resp. 1..j), from three factors.
"""
import numpy as np

from pppm_b200 import Solver

TAPS = 16


def _history(rng, n, t):
    """N[tau], D[tau] for tau = t-31 .. t+1 (dict-like arrays indexed by tau - (t - 31))."""
    return rng.standard_normal((n, 33)), rng.standard_normal((n, 33))


def _at(h, t, tau):
    return h[..., tau - (t - 31)]


def test_face_pair_two_step_identity():
    rng = np.random.default_rng(3)
    npair, t = 40, 100
    s = rng.standard_normal((npair, TAPS))
    d = rng.standard_normal((npair, TAPS))
    N, D = _history(rng, npair, t)

    def conv(time):  # one pass, D[time] left out (it is the step's unknown)
        acc = 0.0
        for k in range(TAPS):
            dk = 0.0 if k == 0 else _at(D, t, time - k)
            acc += np.sum(-s[:, k] * _at(N, t, time - k) + d[:, k] * dk)
        return acc

    # the two-step pass: time-t windows (taps t .. t-15), shifted by one for time t+1
    hn = np.stack([_at(N, t, t - k) for k in range(TAPS)], 1)
    hd = np.stack([_at(D, t, t - k) for k in range(TAPS)], 1)
    hd[:, 0] = 0.0  # D[t] unknown at conv time
    c0 = np.sum(-s * hn + d * hd)
    sn = np.concatenate([_at(N, t, t + 1)[:, None], hn[:, :-1]], 1)  # tap 0 of t+1 is N[t+1]
    sd = np.concatenate([np.zeros((npair, 2)), hd[:, 1:-1]], 1)  # D[t+1] and D[t] left out
    partial = np.sum(-s * sn + d * sd)
    fix = np.sum(d[:, 1] * _at(D, t, t))  # D[t] known after finish(t)
    assert abs(c0 - conv(t)) < 1e-12 * max(1.0, abs(c0))
    assert abs(partial + fix - conv(t + 1)) < 1e-12 * max(1.0, abs(partial))


def test_near_terms_two_step_identity():
    rng = np.random.default_rng(4)
    t = 50
    w_s = rng.standard_normal((54, TAPS))
    w_d = rng.standard_normal((54, TAPS))
    N, D = _history(rng, 1, t)
    N, D = N[0], D[0]

    def term(r, time):  # one pass: BEM-near (r >= 27) taps m; FDTD-near (r < 27) record tap m, history m-1
        acc = 0.0
        for m in range(TAPS):
            k = m if r >= 27 else m - 1
            if k < 0:
                continue
            acc += -w_s[r, m] * _at(N, t, time - k) + w_d[r, m] * _at(D, t, time - k)
        return acc

    # partial terms of time t+1 from the time-t window, D[t+1] left out, then completed
    for r in range(54):
        partial = 0.0
        for m in range(TAPS):
            k = m if r >= 27 else m - 1
            if k < 0:
                continue
            tau = t + 1 - k
            dval = 0.0 if tau == t + 1 else _at(D, t, tau)
            partial += -w_s[r, m] * _at(N, t, tau) + w_d[r, m] * dval
        factor = w_d[r, 0] if r >= 27 else w_d[r, 1]
        full = partial + factor * _at(D, t, t + 1)
        assert abs(full - term(r, t + 1)) < 1e-12 * max(1.0, abs(full))


def test_face_pair_four_step_identity():
    rng = np.random.default_rng(5)
    npair, t = 40, 100
    s, d = rng.standard_normal((npair, TAPS)), rng.standard_normal((npair, TAPS))
    N, D = rng.standard_normal((npair, 36)), rng.standard_normal((npair, 36))  # times t-31 .. t+4

    def conv(time):
        return sum(np.sum(-s[:, k] * _at(N, t, time - k)) + (np.sum(d[:, k] * _at(D, t, time - k)) if k else 0)
                   for k in range(TAPS))

    # quad lane q's window of time t: taps 4q..4q+3; before tap 0 lie (N[t+1], unknown), (N[t+2], unknown), ...
    win = [(_at(N, t, t - k), _at(D, t, t - k) if k else np.zeros(npair)) for k in range(TAPS)]
    fut = [(_at(N, t, t + 1 + k), np.zeros(npair)) for k in range(3)]
    for j in range(4):
        total = 0.0
        for q in range(4):
            for i in range(4):
                tap = 4 * q + i - j  # of time t
                n, dv = win[tap] if tap >= 0 else fut[-tap - 1]
                total += np.sum(-s[:, 4 * q + i] * n + d[:, 4 * q + i] * dv)
        for m in range(1, j + 1):  # group_fix: taps 1..j, D[t+j-m] of the pass's steps
            total += np.sum(d[:, m] * _at(D, t, t + j - m))
        assert abs(total - conv(t + j)) < 1e-12 * max(1.0, abs(total))


def test_near_terms_four_step_identity():
    rng = np.random.default_rng(6)
    t = 50
    w_s, w_d = rng.standard_normal((54, TAPS)), rng.standard_normal((54, TAPS))
    N, D = rng.standard_normal(36), rng.standard_normal(36)

    def term(r, time):
        return sum(-w_s[r, m] * _at(N, t, time - k) + w_d[r, m] * _at(D, t, time - k)
                   for m, k in ((m, m if r >= 27 else m - 1) for m in range(TAPS)) if k >= 0)

    win = [(_at(N, t, t - k), _at(D, t, t - k)) for k in range(TAPS)]  # D[t] known
    fut = [(_at(N, t, t + 1 + k), 0.0) for k in range(3)]
    for r in range(54):
        shift = 0 if r >= 27 else 1
        # gc_factors: the factor of D[t+j-m] in the term of time t+j, by age m of the value
        factor = [w_d[r, m + shift] for m in range(3)]
        for j in range(4):
            total = 0.0
            for m in range(TAPS):
                if m < shift:
                    continue  # the FDTD-near record's tap 0 has no partner
                tap = m - shift - j
                n, dv = win[tap] if tap >= 0 else fut[-tap - 1]
                total += -w_s[r, m] * n + w_d[r, m] * dv
            for m in range(j):
                total += factor[m] * _at(D, t, t + j - m)
            assert abs(total - term(r, t + j)) < 1e-12 * max(1.0, abs(total))


def _pass_at(j, n):
    """step.cu: pass_at with several steps per pass: (size, position)"""
    first = j & ~3
    if first + 4 < n:
        return 4, j - first
    if j & 1 or j + 1 < n:
        return 2, j & 1
    return 1, 0


def test_passes_cover_every_call():
    """Fours while a step follows them, then pairs, then one; the last step of a call never heads a pass;
    chunks of whole passes have the passes of the whole call."""
    for n in range(1, 80):
        at = 0
        while at < n:
            size, pos = _pass_at(at, n)
            assert pos == 0 and at + size <= n
            assert [_pass_at(at + i, n) for i in range(size)] == [(size, i) for i in range(size)]
            assert size < 4 or at + 4 < n
            at += size
        for chunk in (4, 8, 32):
            chunks = (n - 1) // chunk if n > chunk else 0
            rest = n - chunks * chunk
            for j in range(n):
                c, k = divmod(j, chunk)
                want = _pass_at(k, 1 << 40) if c < chunks else _pass_at(j - chunks * chunk, rest)
                assert _pass_at(j, n) == want


def test_autotune_config_numbering():
    # config j of phase 2: conv_pairs = j / 6, threads = {64, 128, 256}[(j / 2) % 3], terms = j % 2
    for j, (pairs, threads, terms) in enumerate(Solver.TUNE_CONFIGS):
        assert (pairs, threads, terms) == (j // 6, (64, 128, 256)[(j // 2) % 3], j % 2)
    for i, (pairs, threads) in enumerate(Solver.TUNE_CANDIDATES):
        assert (pairs, threads) == (i // 3, (64, 128, 256)[i % 3])
