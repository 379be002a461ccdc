"""Recorded ncu commands leave the GPU's clocks alone: without ``--clock-control none`` ncu locks them while it runs."""
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
WRITTEN = sorted(p for d in ("profiles", "docs", "scripts", "benchmarks") for p in (ROOT / d).rglob("*") if p.suffix in (".md", ".py", ".sh")) + [ROOT / "README.md"]


def test_every_ncu_command_keeps_the_clocks():
    found = 0
    for path in WRITTEN:
        for line in path.read_text().splitlines():
            for command in re.findall(r"\bncu\s+-[^`]*", line):
                if re.match(r"ncu\s+(-i|--import)\b", command):  # reads a report, runs nothing
                    continue
                found += 1
                assert "--clock-control none" in command, "%s: %s" % (path.relative_to(ROOT), line.strip())
    assert found
