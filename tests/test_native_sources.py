"""Properties of the CUDA sources that neither a compiler nor a run on a GPU would show to be lost."""
import re
from pathlib import Path

from open_transformers_b200 import build_native

CUDA = build_native.CSRC / "cuda"


def _source(path: Path) -> str:
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


def test_entry_points_called_across_files_are_declared_once():
    """A prototype written out beside its call would go on linking, with shifted arguments, when the definition changes."""
    defined, declared, called = {}, {}, {}
    for path in sorted(CUDA.glob("*.cu*")):
        text = _source(path)
        for m in re.finditer(r"\b(otb_\w+)\s*\(", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[end], 0)
                end += 1
            before, after = text[:m.start()].rstrip(), text[end:].lstrip()
            if re.search(r"(?:^|[;{}\"])\s*(?:int|long|void)$", before):
                (defined if after.startswith("{") else declared).setdefault(m[1], set()).add(path.name)
            else:
                called.setdefault(m[1], set()).add(path.name)
    across = {name for name, users in called.items() if name in defined and users - defined[name] and not any(f.endswith(".cuh") for f in defined[name])}
    assert across >= {"otb_gemm_bf16", "otb_attn_fwd"}
    for name in across:
        assert len(declared.get(name, ())) == 1, (name, declared.get(name))
        header = next(iter(declared[name]))
        for user in defined[name] | called[name]:
            assert header == user or '#include "%s"' % header in (CUDA / user).read_text(), (name, user, header)
