"""The order that dependent launches rest on, read from the kernels' source.

A kernel may read ahead of its wait what was written before its predecessor started.  That holds only where every kernel lets its
dependents start after its own wait, and where every kernel that is launched to overlap its predecessor waits at all."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "qwen3.8-flash-next-2x-p100_b200" / "csrc"
WAIT, START = re.compile(r"\bpdl_wait\(\)|\bpdl_begin\(\)"), re.compile(r"\bpdl_launch_dependents\(\)")
NAME = re.compile(r"__global__[^;{}]*?\b(k_\w+)\(|void (nm_body|gdn_body)\(")   # (these two are the bodies of several kernels)


def _functions():
    for path in sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh"))):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in NAME.finditer(text):
            at, depth = m.end(), 1
            while depth:                     # (to the end of the parameters)
                depth += {"(": 1, ")": -1}.get(text[at], 0)
                at += 1
            if text[at:].lstrip().startswith("{"):
                yield path.name, m.group(1) or m.group(2), text[at:text.index("\n}\n", at)]


def test_a_kernel_lets_its_dependents_start_after_its_own_wait():
    seen = 0
    for file, name, body in _functions():
        if not START.search(body):
            continue
        seen += 1
        wait = WAIT.search(body)
        assert wait and wait.start() < START.search(body).start(), f"{file}: {name}"
    assert seen >= 20


def test_a_kernel_launched_to_overlap_its_predecessor_waits_for_it():
    bodies = {name: body for _, name, body in _functions()}
    text = "".join(re.sub(r"//[^\n]*", "", p.read_text()) for p in CSRC.glob("*.cu"))
    names = set(re.findall(r"launch_(?:after\(|dep\((?:true|early), )(k_\w+)", text)) | set(re.findall(r"auto kernel = [^;]*?(k_\w+)", text))
    names |= set(re.findall(r"(?:launch_after\(|launch_dep\((?:true|early), )[^,;]*\? (k_\w+)", text))
    assert len(names) >= 30
    for name in sorted(names):
        assert name in bodies, name
        body = bodies[name]
        assert WAIT.search(body) or any(WAIT.search(bodies[b]) for b in ("nm_body", "gdn_body") if re.search(rf"\b{b}<", body)), name
