"""The spectral column pass (mk_prop_cols_rows, mk_prop.cu) replayed on the CPU
with the kernel's index arithmetic: radix-8 passes on padded lines, their
twiddle table, the digit-reversed frequencies H is applied at, the rows outside
the field, and the lines' layout in shared memory.

Tolerance: a radix-8 FFT in float32 loses below 6e-8 sqrt(log2 N) of the largest
value a transform; the replay is in FP64 with FP32 twiddles, so 1e-6."""
import numpy as np
import pytest

SMEM, SMEM_MAX, NT = 74 << 10, 227 << 10, 512


def pad8(i):
    return i + (i >> 3)


def ld_of(nz2, W):
    ld = nz2 + nz2 // 8
    while ld % 16 != (16 // W) % 16:
        ld += 1
    return ld


def width(ny2, nz2):
    W = 16
    while W > 4 and 8 * W * ld_of(nz2, W) > SMEM:
        W //= 2
    while W > 1 and 8 * W * ld_of(nz2, W) > SMEM_MAX:
        W //= 2
    return max(1, min(W, ny2))


def twiddles(nz2):
    """mk_prop_tables_kernel's table, entry by entry."""
    tw = np.full(nz2, np.nan + 0j)
    for i in range(nz2):
        M, e = nz2, i
        while M >= 8 and e >= 7 * (M // 8):
            e -= 7 * (M // 8)
            M //= 8
        if M >= 8:
            k, t = e // (M // 8) + 1, (e % (M // 8)) * (e // (M // 8) + 1) * (nz2 // M)
            assert t < nz2 and 1 <= k <= 7
            tw[i] = np.exp(-2j * np.pi * t / nz2).astype(np.complex64)
    return tw


def dft(v, inv):
    R = len(v)
    j = np.arange(R)
    return np.exp((2j if inv else -2j) * np.pi * np.outer(j, j) / R) @ v


def column(x, H, logn, z0, nz, mode, cval):
    """One column of the kernel: x holds the field's nz rows; returns them after
    the transform, H and the inverse transform (unnormalised)."""
    N, last = 1 << logn, (logn % 3) or 3
    P, RL = (logn - last) // 3, 1 << last
    line = np.full(ld_of(N, 1), np.nan + 0j)
    tw = twiddles(N)

    def load(r):
        s = r - z0
        if mode == 1 and not 0 <= s < nz:
            return cval
        return x[min(max(s, 0), nz - 1)]

    at = 0
    for p in range(P):
        logm = logn - 3 * (p + 1)
        m, out, hit = 1 << logm, {}, np.zeros(N, int)
        for q in range(N >> 3):
            i = q & (m - 1)
            base = ((q >> logm) << (logm + 3)) + i
            idx = [base + (r << logm) for r in range(8)]
            hit[idx] += 1
            v = dft(np.array([load(j) if p == 0 else line[pad8(j)] for j in idx]), False)
            for k in range(8):
                out[pad8(idx[k])] = v[k] * (tw[at + (k - 1) * m + i] if k else 1.0)
        assert (hit == 1).all()
        for a, v in out.items():
            line[a] = v
        at += 7 * m
    seen = np.zeros(N, int)
    for q in range(N >> 3):
        assert all(pad8(8 * q + j) == 9 * q + j for j in range(8))
        v = line[9 * q:9 * q + 8].copy()
        for g in range(8 // RL):
            w = dft(v[g * RL:(g + 1) * RL], False)
            pos = 8 * q + g * RL
            f = sum(((pos >> (logn - 3 * (p + 1))) & 7) << (3 * p) for p in range(P))
            fs = [f + (k << (3 * P)) for k in range(RL)]
            seen[fs] += 1
            v[g * RL:(g + 1) * RL] = dft(w * H[fs], True)
        line[9 * q:9 * q + 8] = v
    assert (seen == 1).all()                 # every frequency once
    res = np.zeros(nz, complex)
    for p in range(P - 1, -1, -1):
        logm = logn - 3 * (p + 1)
        m = 1 << logm
        at -= 7 * m
        for q in range(N >> 3):
            i = q & (m - 1)
            base = ((q >> logm) << (logm + 3)) + i
            idx = [base + (r << logm) for r in range(8)]
            v = dft(np.array([line[pad8(idx[k])] * (np.conj(tw[at + (k - 1) * m + i]) if k else 1.0)
                              for k in range(8)]), True)
            for r in range(8):
                if p > 0:
                    line[pad8(idx[r])] = v[r]
                elif 0 <= idx[r] - z0 < nz:
                    res[idx[r] - z0] = v[r]
    assert at == 0
    return res


@pytest.mark.parametrize("logn", range(4, 12))
@pytest.mark.parametrize("mode", [0, 1])
def test_column_pass_matches_numpy(logn, mode):
    N = 1 << logn
    rng = np.random.default_rng(logn)
    nz = max(1, N // 3)
    z0 = (N - nz) // 2
    x = rng.standard_normal(nz) + 1j * rng.standard_normal(nz)
    H = np.exp(1j * rng.uniform(-3, 3, N))
    cval = 0.3 - 0.7j
    full = np.full(N, cval)
    full[z0:z0 + nz] = x
    if mode == 0:
        full[:z0], full[z0 + nz:] = x[0], x[-1]
    ref = np.fft.ifft(np.fft.fft(full) * H)[z0:z0 + nz] * N
    got = column(x, H, logn, z0, nz, mode, cval)
    assert np.abs(got - ref).max() <= 1e-6 * np.abs(ref).max()


@pytest.mark.parametrize("logn", range(4, 14))
def test_lines_fit_and_table_is_whole(logn):
    N = 1 << logn
    for ny2 in (1, 2, 16, 1024, 8192):
        W = width(ny2, N)
        ld = ld_of(N, W)
        assert ny2 % W == 0 and 8 * W * ld <= SMEM_MAX
        assert pad8(N - 1) < ld                 # a line's points stay in the line
    last = (logn % 3) or 3
    used = sum(7 * (1 << (logn - 3 * (p + 1))) for p in range((logn - last) // 3))
    assert used <= N and not np.isnan(twiddles(N)[:used]).any()


@pytest.mark.parametrize("logn", range(7, 14))
def test_half_warps_meet_different_banks(logn):
    """16 neighbouring threads' 8-byte accesses (W lines x 16 / W items) in a
    pass: different 8-byte banks at every stride a block of the kernel's width
    has."""
    N = 1 << logn
    W = width(8192, N)
    ld, last = ld_of(N, W), (logn % 3) or 3
    t = np.arange(min(W * (N >> 3), 4096))
    c, q = t % W, t // W
    for p in range((logn - last) // 3):
        logm = logn - 3 * (p + 1)
        i = q & ((1 << logm) - 1)
        base = ((q >> logm) << (logm + 3)) + i
        for r in range(8):
            bank = (c * ld + pad8(base + (r << logm))) % 16
            per = np.array([len(set(b)) for b in bank.reshape(-1, 16)])
            assert per.min() == 16, (p, r, per.min())
    for j in range(8):                          # the pass around H: 8 consecutive points a thread
        bank = (c * ld + 9 * q + j) % 16
        per = np.array([len(set(b)) for b in bank.reshape(-1, 16)])
        assert per.min() == 16, (j, per.min())
