"""Integer model of where a bucket-kernel item reads and writes, every shape.

k_fb_accum (csrc/zg_bucket.cuh) finds an item's sort output, table points and
output from its number alone. This restates that arithmetic (`item`) and the
host's plan of a blob's sets (`sets`, zg_encoder.cu), and checks for every
context shape and every number of wide classes in use, over one and two blobs:
the addresses stay inside their buffers and inside 31 and 32 bits, an item's
points lie inside its table line, no two items share an output, and the items
of a (coset, line) cover every (point, bucket) once.
"""
import pytest

WINDOWS, BUCKETS, UNIT_LOG = 24, 1024, 6


def wd_windows(ulog):
    return 254 // (ulog + 1) + 1


def wide_classes(lr):
    """plan_wide_classes of a device with room for every class (1024 columns)"""
    out, nxt = [], 0
    for u in range(16, 10, -1):
        ulog = min(u, 15)
        nq = 0
        while nxt + nq < lr and min(16, lr + 9 - (nxt + nq)) == u:
            nq += 1
        hi = min(16, lr + 10) == u
        if nq or hi:
            out.append(dict(ulog=ulog, mlog=u - ulog, W=wd_windows(ulog), l0=nxt, nl=nq + hi, hi=hi))
            nxt += nq
    return out


def sets(lr, lc, wd):
    """the sets of one blob's MSM: kind, items, table lines"""
    N, L = 1 << (lr + lc), lr + 2
    nxt = sum(k["nl"] - k["hi"] for k in wd)
    high = any(k["hi"] for k in wd)
    out = []
    if lc >= UNIT_LOG:
        chunks = [(lc, nxt, lr + 1 - nxt + (not high))]
    else:
        top, chunks = min(UNIT_LOG, lc + 6), []
        for l in range(lr + 1):
            u = min(top, lr + lc - 1 - l) if l < lr else lc
            if chunks and chunks[-1][0] == u:
                chunks[-1] = (u, chunks[-1][1], chunks[-1][2] + 1)
            else:
                chunks.append((u, l, 1))
        chunks.append((min(top, lr + lc), L - 1, 1))
    assert len(chunks) <= 8
    for u, l0, nl in chunks:
        out.append(dict(wide=False, lc=u, lr=lr + lc - u, lines=nl, l0=l0, Ltot=L, W=WINDOWS, items=3 * (N >> u) * nl))
    for k in wd:
        out.append(dict(wide=True, lc=lc, lr=lr - k["mlog"], lines=k["nl"], l0=0, Ltot=k["nl"], W=k["W"],
                        ulog=k["ulog"], mlog=k["mlog"], items=3 * (1 << (lr - k["mlog"])) * k["nl"]))
    return out


def item(a, u, N):
    """k_fb_accum's item_of: offset index, entry index (of each sort unit), table
    point, points per item"""
    nch = 1 << a["lr"]
    l, g = u % a["lines"], u // a["lines"]
    coset, b = g // nch, g % nch
    tab = (coset * a["Ltot"] + a["l0"] + l) * a["W"] * N
    if not a["wide"]:
        return dict(coset=coset, line=l, offs=[g * (BUCKETS + 1)], ents=[g * (WINDOWS << a["lc"])],
                    tab=tab + (b << a["lc"]), points=1 << a["lc"], first=b << a["lc"], block=0)
    bl, ul, ml = a["ulog"] - 10, a["ulog"], a["mlog"]
    unit, blk = b >> bl, b & ((1 << bl) - 1)
    cu = coset * ((nch >> bl) << ml) + (unit << ml)
    return dict(coset=coset, line=l, offs=[(cu + i) * ((1 << ul) + 1) + blk * BUCKETS for i in range(1 << ml)],
                ents=[(cu + i) * (a["W"] << ul) for i in range(1 << ml)], tab=tab + (unit << (ul + ml)),
                points=1 << (ul + ml), first=unit << (ul + ml), block=blk)


@pytest.mark.parametrize("lc", range(3, 11))
@pytest.mark.parametrize("lr", range(1, 12))
def test_items_stay_inside_their_buffers(lr, lc):
    N, R, L = 1 << (lr + lc), 1 << lr, lr + 2
    allw = wide_classes(lr) if lc == 10 else []
    for on in range(len(allw) + 1):
        blob = sets(lr, lc, allw[:on])
        total = sum(a["items"] for a in blob)
        assert total <= 3 * R * L  # blob_items_max, the output's size
        lines = set()
        for k, a in enumerate(blob):
            if a["wide"]:
                n_offs = 3 * (N >> a["ulog"]) * ((1 << a["ulog"]) + 1)
                n_ents = 3 * (N >> a["ulog"]) * (a["W"] << a["ulog"])
            else:
                n_offs = 3 * (N >> a["lc"]) * (BUCKETS + 1)
                n_ents = 3 * N * WINDOWS
                lines |= {a["l0"] + i for i in range(a["lines"])}
            assert n_ents < 1 << 32
            assert 3 * a["Ltot"] * a["W"] * N < 1 << 31
            # every item at small shapes, the ends of every (coset, line) at large ones
            step = max(1, a["items"] // 4096)
            seen = {}
            for u in sorted(set(range(0, a["items"], step)) | set(range(a["items"] - 3 * a["lines"], a["items"]))):
                it = item(a, u, N)
                assert it["coset"] < 3
                for o in it["offs"]:
                    assert 0 <= o and o + BUCKETS < n_offs
                for e in it["ents"]:
                    assert 0 <= e and e + ((a["W"] << a["ulog"]) if a["wide"] else (WINDOWS << a["lc"])) <= n_ents
                line0 = (it["coset"] * a["Ltot"] + a["l0"] + it["line"]) * a["W"] * N
                assert line0 <= it["tab"] and it["first"] + it["points"] <= N
                assert it["tab"] + (a["W"] - 1) * N + it["points"] <= line0 + a["W"] * N
                seen.setdefault((it["coset"], it["line"]), []).append((it["first"], it["block"]))
            if step == 1:
                for pairs in seen.values():
                    points = item(a, 0, N)["points"]
                    blocks = 1 << (a["ulog"] - 10) if a["wide"] else 1
                    assert sorted(pairs) == [(f, b) for f in range(0, N, points) for b in range(blocks)]
                assert len(seen) == 3 * a["lines"]
        assert lines == set(range(L)) - {i for w in allw[:on] for i in range(w["l0"], w["l0"] + w["nl"] - w["hi"])} - (
            {L - 1} if any(w["hi"] for w in allw[:on]) else set())
