"""The barriers between the score, softmax and value stages of csrc/attn_prefill_tc.cu, walked over every interleaving on the CPU.

Which barrier and which parity each wait, arrival and commit names is read from the kernel's source, so that the walk is over the
protocol as written: the thread that issues the products, the tensor core (products end in the order of their issue) and row
warps, every one of which may find at any page that its rows' maximum grows or does not, and that the next scores are there
before or after it has stored its weights.
"""
import re
import subprocess
from pathlib import Path

import pytest

SRC = (Path(__file__).resolve().parent.parent / "vllm_rs_b200" / "csrc" / "attn_prefill_tc.cu").read_text()
KERNEL = SRC[SRC.index("attn_prefill_tc_kernel(const"):SRC.index("static int prefill_attn_mode")]
ISSUER = KERNEL[KERNEL.index("} else if (warp == 1) {"):KERNEL.index("// ---- epilogue")]
ISSUER, ROWS = ISSUER[:ISSUER.index("float m_ref")], ISSUER[ISSUER.index("float m_ref"):]


def _one(pattern, text):
    """The bar and parity expressions of the one place that matches; an expression in C becomes a function of the page j."""
    found = set(re.findall(pattern, text))
    assert len(found) == 1, (pattern, found)
    got = found.pop()
    return [_expr(e) for e in ((got,) if isinstance(got, str) else got)]


def _expr(text):
    m = re.fullmatch(r"&?(\w+)\[(.*)\]", text)
    if m:
        code = compile(m.group(2), text, "eval")
        return lambda j: (m.group(1), eval(code, {"j": j, "s": j & 1}))
    if re.fullmatch(r"[a-z_]+", text):
        return lambda j: (text, 0)
    code = compile(text, text, "eval")
    return lambda j: eval(code, {"j": j, "s": j & 1})


def _needed(name):
    counts = set(re.findall(rf"mbar_init\(&?{name}(?:\[\w\])?, (\d+)\)", KERNEL))
    assert len(counts) == 1, (name, counts)
    return int(counts.pop())


def protocol():
    p = {}
    p["s_free_wait"] = _one(r"if \(j > 0\) mbar_wait_bounded\((s_free), (.+)\);", ISSUER)
    p["s_commit"] = _one(r"tc_commit\((&?s_full[^)]*)\);", ISSUER)
    p["p_wait"] = _one(r"mbar_wait_bounded\((&?p_full[^,]*), (.+)\);", ISSUER)
    p["pv_commit"] = _one(r"tc_commit\((&?pv_done[^)]*)\);", ISSUER)
    p["s_wait"] = _one(r"mbar_wait_bounded\((s_full), (\(j \+ 1\) & 1)\);", ROWS)
    assert f"mbar_probe_addr(smem_u32(s_full), (j + 1) & 1)" in ROWS
    assert "mbar_wait_bounded(s_full, 0);" in ROWS
    p["s_arrive"] = _one(r"mbar_arrive\((s_free)\);", ROWS)
    p["place_wait"] = _one(r"if \(j > 1\) mbar_wait_bounded\((&?pv_done[^,]*), (.+)\);", ROWS)
    grow = ROWS[ROWS.index("if (j > 0 && __any_sync"):]
    p["o_wait"] = _one(r"mbar_wait_bounded\((&?pv_done[^,]*), (.+)\);", grow[:grow.index("tc_fence_after")])
    p["p_arrive"] = _one(r"mbar_arrive\((&?p_full[^)]*)\);", ROWS)
    last = KERNEL[KERNEL.index("// ---- epilogue"):]
    assert "mbar_wait_bounded(&pv_done[(npages - 1) & 1], ((npages - 1) >> 1) & 1);" in last
    # one warp's share of the arrivals; four warps in the kernel
    p["needed"] = {n: _needed(n) // (4 if n in ("s_free", "p_full") else 1) for n in ("s_full", "s_free", "p_full", "pv_done")}
    assert _needed("s_free") == _needed("p_full") == 4 and _needed("s_full") == _needed("pv_done") == 1
    return p


def walk(p, pages, warps):
    """First fault of any interleaving, with its steps; None where there is none.  A state: bars {(name, i): (phases, arrivals)},
    the issuer's place, the products in flight, per warp its place and what it has stored, products ended."""
    need = {n: c * (warps if n in ("s_free", "p_full") else 1) for n, c in p["needed"].items()}
    issue = [("qk", 0)]
    for j in range(pages):
        if j + 1 < pages:
            issue += [("sfree", j + 1), ("qk", j + 1)]
        issue += [("pwait", j), ("pv", j)]
    # of a warp: (next step, page, does its maximum grow); steps: take -> store -> (take of the next page in between) -> ..
    start = ((), 0, (), tuple((("take", 0),) for _ in range(warps)), (), ())

    def bar(bars, key):
        return dict(bars).get(key, (0, 0))

    def passes(bars, wait, j):
        return (bar(bars, wait[0](j))[0] & 1) != wait[1](j)

    def arrive(bars, at, j):
        key = at[0](j)
        d = dict(bars)
        n, a = d.get(key, (0, 0))
        a += 1
        d[key] = (n + 1, 0) if a == need[key[0]] else (n, a)
        return tuple(sorted(d.items()))

    seen, todo = {start}, [(start, ())]
    while todo:
        (bars, at, flying, todo_w, stored, ended), path = todo.pop()
        nxt, fault = [], None

        def go(step, **kw):
            s = dict(bars=bars, at=at, flying=flying, w=todo_w, stored=stored, ended=ended)
            s.update(kw)
            nxt.append(((s["bars"], s["at"], s["flying"], s["w"], s["stored"], s["ended"]), step))

        if at < len(issue):
            what, j = issue[at]
            if what == "sfree":
                if passes(bars, p["s_free_wait"], j):
                    go(f"s_free {j - 1}", at=at + 1)
            elif what == "pwait":
                if passes(bars, p["p_wait"], j):
                    go(f"p_full {j}", at=at + 1)
            else:
                if what == "pv" and any((w, j) not in stored for w in range(warps)):
                    fault = f"P V {j} before every warp has stored its weights"
                if what == "qk" and any(t[0] in (("take", j - 1), ("early", j - 1)) for t in todo_w if t):
                    fault = f"scores {j} over scores that a warp has not read"
                go(f"issue {what} {j}", at=at + 1, flying=flying + ((what, j),))
        if flying:
            what, j = flying[0]
            go(f"end {what} {j}", flying=flying[1:], ended=ended + ((what, j),),
               bars=arrive(bars, p["s_commit"] if what == "qk" else p["pv_commit"], j))
        begun = set(ended) | set(flying)
        for w, steps in enumerate(todo_w):
            if not steps:
                continue
            (what, j), rest = steps[0], steps[1:]

            def put(*new):
                return todo_w[:w] + (tuple(new) + rest,) + todo_w[w + 1:]

            if what == "take":                                    # a page's scores into registers
                if passes(bars, p["s_wait"], j - 1):              # (the wait for page j + 1 stands in page j)
                    if ("qk", j) not in ended:
                        fault = f"warp {w} reads scores {j} that are not there"
                    b = arrive(bars, p["s_arrive"], j)
                    if j + 1 < pages:                             # the next scores come before or after the store
                        go(f"warp {w} takes {j}", bars=b, w=put(("store", j), ("take", j + 1)))
                        go(f"warp {w} takes {j}, will ask for {j + 1} early", bars=b, w=put(("ask", j + 1)))
                    else:
                        go(f"warp {w} takes {j}", bars=b, w=put(("store", j)))
            elif what == "ask":                                   # only where the probe says that the scores are there
                if passes(bars, p["s_wait"], j - 1):
                    if ("qk", j) not in ended:
                        fault = f"warp {w} asks for scores {j} that are not there"
                    go(f"warp {w} asks for {j}", w=put(("store", j - 1), ("early", j)))
                go(f"warp {w} finds no scores {j}", w=put(("store", j - 1), ("take", j)))
            elif what == "early":                                 # asked for before the store: read now
                b = arrive(bars, p["s_arrive"], j)
                if j + 1 < pages:
                    go(f"warp {w} has {j}", bars=b, w=put(("store", j), ("take", j + 1)))
                    go(f"warp {w} has {j}, will ask for {j + 1} early", bars=b, w=put(("ask", j + 1)))
                else:
                    go(f"warp {w} has {j}", bars=b, w=put(("store", j)))
            else:
                ready = j < 2 or passes(bars, p["place_wait"], j)
                for grow in (False, True) if j > 0 else (False,):
                    if ready and (not grow or passes(bars, p["o_wait"], j)):
                        if j > 1 and ("pv", j - 2) not in ended:
                            fault = f"warp {w} stores {j} over weights that P V {j - 2} reads"
                        if grow and (("pv", j - 1) not in ended or ("pv", j) in begun):
                            fault = f"warp {w} rescales at {j} under a product"
                        go(f"warp {w} stores {j}" + (", rescaled" if grow else ""), bars=arrive(bars, p["p_arrive"], j), w=put(),
                           stored=tuple(sorted(set(stored) | {(w, j)})))
        if fault:
            return fault, path
        if not nxt and (at < len(issue) or any(todo_w)):
            return "nobody can go on", path
        for state, step in nxt:
            if state not in seen:
                seen.add(state)
                todo.append((state, path + (step,)))
    return None


@pytest.mark.parametrize("pages,warps", [(1, 2), (2, 2), (5, 2), (3, 3)])
def test_every_interleaving_is_in_order(pages, warps):
    assert walk(protocol(), pages, warps) is None


def test_the_walk_finds_one_barrier_for_all_pages():
    """With two places for the weights and one barrier for their arrival a warp can arrive twice before another one does."""
    p = protocol()
    p["p_wait"], p["p_arrive"] = [lambda j: ("p_full", 0), lambda j: j & 1], [lambda j: ("p_full", 0)]
    fault, _ = walk(p, 3, 2)
    assert "before every warp" in fault or "nobody" in fault


def test_no_register_of_a_page_is_spilled(tmp_path):
    """A page's scores are on their way from tensor memory into registers while the page before is stored: none of these may go
    through memory in between."""
    from vllm_rs_b200 import build
    src = build.CSRC / "attn_prefill_tc.cu"
    r = subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-Xptxas", "-v", "-cubin", "-o", str(tmp_path / "k.cubin"), str(src)],
                       capture_output=True, text=True, check=True)
    frames = re.findall(r"(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", r.stdout + r.stderr)
    assert frames == [("0", "0", "0")] * 4, frames
