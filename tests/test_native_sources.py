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


def _kernels(text: str):
    """(name, parameters, body) of every __global__ function."""
    for m in re.finditer(r"__global__[^{;]*?\b(\w+_kernel)\s*\(", text):
        def close(i, pair):
            depth = 1
            while depth:
                depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
                i += 1
            return i
        end = close(m.end(), "()")
        start = text.index("{", end) + 1
        yield m[1], text[m.end():end], text[start:close(start, "{}")]


WRITTEN_ONLY = {"y", "O", "Cv", "rstd_out", "dx", "dgamma_partial", "out", "din", "h", "dgu", "ce_out", "lse_out", "status"}


def test_kernels_that_wait_promise_nothing_of_what_they_read():
    """A kernel that is launched while its predecessor still writes must not call its inputs unchanging: the compiler might take
    a load past the wait. It has to wait in the first place, and the early kernel of a pair at its end."""
    waiting, early, launched = set(), set(), set()
    for path in sorted(CUDA.glob("*.cu")):
        text = _source(path)
        for name, params, body in _kernels(text):
            if re.match(r"\s*(?:after|wait_for)_predecessor\(\);", body) or "after_predecessor();" in body or "!PAIR) wait_for_predecessor();" in body:
                waiting.add(name)
                assert "__ldg" not in re.sub(r"if constexpr \(TP == 1\).*?\n    }\n  }\n", "", body, flags=re.S), name
                for const, p in re.findall(r"(const\s+)?[\w:]+\s*\*\s*__restrict__\s+(\w+)", params):
                    assert not const and p in WRITTEN_ONLY, (name, p)
            elif "wait_for_predecessor()" in body:
                early.add(name)
        aliases = dict(re.findall(r"auto (\w+) = [^;]*?\b(\w+_kernel)\b", text))
        aliases["KERN"] = "rmsnorm_fwd_kernel"  # (a macro's argument)
        launched |= {aliases.get(n, n) for n in re.findall(r"\botb_launch_(?:early\(|if_early\(\s*\w+,)\s*(\w+)", text)}
    assert early == {"attn_bwd_q2_kernel"}
    assert launched | {"rmsnorm_fwd_wide_kernel"} == waiting | early, launched ^ (waiting | early)


def test_warps_give_up_together():
    """What whole warps do after a bounded wait (tensor-memory accesses, votes, shuffles) needs all of their lanes: lanes that left alone
    would keep the others waiting without a limit. Outside code that one lane runs, a wait has one answer for the warp, or its answer is
    left alone or only added to ``ok``, and nothing is decided before the warp has voted on that or on the abort word."""
    waits = {}
    for path in sorted(CUDA.glob("*.cu")):
        text = _source(path)
        for name, _, body in _kernels(text):
            blocks = [(False, False)]  # of each open block: whether a single lane runs it, whether it is a loop that goes on while ``ok``
            voted = True
            for m in re.finditer(r"[{}]|\bmbar_wait(?:_cluster|_warp)?\(|\bok\b", body):
                before, after = body[:m.start()], body[m.start():m.start() + 200]
                if m[0] == "{":
                    one_lane = re.search(r"if \((?:half == 0 && )?(?:elect_one\(\)|lane == 0)\) $", before)
                    head = before[before.rfind("\n"):]
                    blocks.append((bool(one_lane) or blocks[-1][0], bool(re.search(r"\b(?:for|while) \(.*\bok\b", head))))
                elif m[0] == "}":
                    one_lane, loop = blocks.pop()
                    assert voted or not loop, (path.name, name)
                elif not blocks[-1][0]:
                    if m[0] == "mbar_wait_warp(":
                        waits.setdefault(name, set()).add("one answer")
                    elif m[0] != "ok":
                        adds, alone = re.search(r"\n\s*ok = ok &&[^;]*$", before), re.search(r"[;}{]\s*$", before) and re.match(r"mbar_wait\([^;]*\);", after)
                        assert adds or alone, (path.name, name, after)
                        waits.setdefault(name, set()).add("a vote on the answers" if adds else "a vote on the abort word")
                        voted = False
                    elif re.match(r"ok = __all_sync\(0xffffffffu, (?:ok|\*abort_flag == 0)\);", after):
                        assert voted or ("abort_flag" in after[:40]) == ("a vote on the abort word" in waits[name]), (path.name, name)
                        voted = True
                    else:
                        adds = re.match(r"ok = ok && mbar_wait\(", after) or re.search(r"ok = $", before) and after.startswith("ok && mbar_wait(") \
                            or before.endswith("__all_sync(0xffffffffu, ")
                        assert voted or adds, (path.name, name, after)
            assert voted, (path.name, name)
    assert waits == {"gemm_tc05_kernel": {"one answer"}, "attn_bwd_kv3_kernel": {"one answer"}, "attn_bwd_q2_kernel": {"a vote on the abort word"},
                     "attn_fwd_i8pv_kernel": {"a vote on the answers"}, "attn_fwd2_kernel": {"a vote on the answers"}}
