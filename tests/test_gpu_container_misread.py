"""Containers whose sort-position table the reference's thread-count rule reads
for fewer chunks than were written (SZp/include/szp_detect_threads.h:153-190):
the chunks that it finds walk one by one, but do not follow one another.  The
positions are those of these chunks, each decoded on its own; the rule and the
walks are restated here."""
import struct

import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu


def _span(s, p, n, tags):
    """End of the block of n elements at s[p], None when it does not walk."""
    if p + 4 > len(s):
        return None
    p += 4
    if n > 1:
        if p >= len(s) or s[p] > 32:
            return None
        bc = s[p]
        p += 1
        if bc:
            p += (n + 6) // 8 + (bc // 8) * (n - 1) + ((bc % 8) * (n - 1) + 7) // 8
    p += (2 * n + 7) // 8 if tags else 0
    return p if p <= len(s) else None


def _chunks(s, n, B, T, tags):
    """[(first element, elements, start, end)] of the T chunks of a table, None when one does not walk."""
    nb = -(-n // B)
    per = -(-nb // T)
    out = []
    for t in range(T):
        b0, b1 = t * per, min((t + 1) * per, nb)
        if b0 >= nb:
            break
        start = p = 8 * T + struct.unpack_from("<Q", s, 8 * t)[0]
        if p >= len(s):
            return None
        for b in range(b0, b1):
            p = _span(s, p, min(B, n - b * B), tags)
            if p is None:
                return None
        out.append((b0 * B, min(b1 * B, n) - b0 * B, start, p))
    return out


def _rule(s, n, B, tags, first):
    """Chunks of the first thread count whose table and chunks are valid within the bound."""
    bound = 8 * n + 1024 if tags else 4 * n + 4
    lim = s[:min(len(s), bound)]
    for T in range(first, min(128, len(s) // 8) + 1):
        tab = struct.unpack_from("<%dQ" % T, s, 0)
        if any(tab[k] > bound or tab[k] < tab[k - 1] for k in range(1, T)) or tab[0]:
            break
        c = _chunks(lim, n, B, T, tags)
        if c:
            return T, c
    return 1, _chunks(s, n, B, 1, tags)


def _table(payload, n, B, T, tags):
    """The stream of a writer of T threads."""
    offs, p = [], 0
    nb = -(-n // B)
    for b in range(nb):
        offs.append(p)
        p = _span(payload, p, min(B, n - b * B), tags)
    assert p == len(payload)
    per = -(-nb // T)
    return b"".join(struct.pack("<Q", offs[t * per] if t * per < nb else p) for t in range(T)) + payload


def _ints(s, p, n, B):
    """The n values of the blocks from s[p] on."""
    out = np.zeros(n, np.int64)
    for i in range(0, n, B):
        m = min(B, n - i)
        q = [struct.unpack_from("<i", s, p)[0]]
        bc = s[p + 4] if m > 1 else 0
        if bc:
            at = p + 5
            signs = np.unpackbits(np.frombuffer(s, np.uint8, (m + 6) // 8, at))
            at += (m + 6) // 8
            full, rem = bc // 8, bc % 8
            low = np.unpackbits(np.frombuffer(s, np.uint8, (rem * (m - 1) + 7) // 8, at + full * (m - 1)))
            for j in range(m - 1):
                v = int.from_bytes(s[at + j * full:at + (j + 1) * full], "little") << rem
                v |= int("".join(map(str, low[j * rem:(j + 1) * rem])) or "0", 2)
                q.append(q[-1] + (-v if signs[j] else v))
        else:
            q += q * (m - 1)
        out[i:i + m] = q
        p = _span(s, p, m, False)
    return out.astype(np.uint32).view(np.int32)


CASES = [((300, 301), "steps", 64, 33), ((80, 90), "steps", 16, 40),
         ((37, 53), "noise", 64, 40), ((37, 53), "noise", 16, 128), ((70, 90), "noise", 64, 128),
         ((9, 9, 9), "noise", 16, 7), ((20, 30, 40), "steps", 64, 33), ((12, 20), "noise", 16, 3)]


@pytest.mark.parametrize("dims,kind,B,T", CASES)
def test_positions_of_the_chunks_found(ora, dims, kind, B, T):
    import torch
    import toposzp_b200
    eb = 1e-2
    if kind == "steps":
        d = np.floor(np.random.default_rng(3).standard_normal(dims) * 3).astype(np.float32)
    else:
        d = synth.small_field(dims, seed=11, kind="noise")
    n = d.size
    cp = ora.sort_cp(ora.find_cp(d, eb), d)
    single = ora.encode_topo(d, eb, B, ora.mark_types(cp, dims))
    sp = np.asarray(ora.extract_sp(cp), np.int32)
    E = len(sp)
    assert n % B != 1 and E % B != 1          # no one-element block, which the two layouts write differently
    topo = _table(single[8:], n, B, T, True)
    sort = _table(ora.encode_ints(sp, B)[8:], E, B, T, False)
    blob = topo + struct.pack("<Q", E) + sort + struct.pack("<QQ", len(topo), 8 + len(sort))
    # the topology is found as one walk; the sort positions are not
    _, ct = _rule(topo, n, B, True, 1)
    assert all(a[3] == b[2] for a, b in zip(ct, ct[1:]))
    Ts, cs = _rule(sort, E, B, False, 2)
    assert any(a[3] != b[2] for a, b in zip(cs, cs[1:])) and Ts != T
    assert (_ints(ora.encode_ints(sp, B), 8, E, B) == sp).all()
    got_sp = np.zeros(E, np.int32)
    for e0, m, start, end in cs:
        got_sp[e0:e0 + m] = _ints(sort, start, m, B)
    raw, fn, _ = ora.decode_topo(single, n, eb, B)
    want, _ = ora.post(raw.reshape(dims), raw.reshape(dims), fn.reshape(dims), got_sp, eb)
    ctx = toposzp_b200.Context()
    cont = torch.from_numpy(np.frombuffer(blob, np.uint8).copy()).cuda()
    for _ in range(2):
        got = ctx.decompress_container(cont, dims, eb, B, postprocess=1).cpu().numpy()
        assert (got.view(np.int32) == want.reshape(-1).view(np.int32)).all()
    ctx.close()
