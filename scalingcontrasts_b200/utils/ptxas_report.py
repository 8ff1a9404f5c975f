"""Writes the table of what the compiler made of every kernel: registers, spills, stack and static shared memory per
kernel, as reported by ``ptxas -v`` while the CUDA sources are compiled for sm_100a (nothing is disassembled).

    python -m scalingcontrasts_b200.utils.ptxas_report profiles/ptxas.md

Dynamic shared memory is chosen at launch and does not appear in ptxas' output; the tile kernels' figures are quoted
from their launchers in the notes under the table.
"""
from __future__ import annotations

import os
import re
import shutil
import subprocess
import sys
from typing import Dict, List

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
CSRC = os.path.join(ROOT, "scalingcontrasts_b200", "csrc")
SOURCES = ("collectives.cu", "loss_small.cu", "loss_fwd.cu", "loss_bwd.cu", "no_alloc.cu", "tower.cu", "optim.cu")
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
         "-Xptxas", "-v", "-c", "-o", os.devnull]


def _demangle(names: List[str]) -> Dict[str, str]:
    tool = shutil.which("c++filt")
    if tool is None or not names:
        return {name: name for name in names}
    result = subprocess.run([tool], input="\n".join(names), capture_output=True, text=True)
    plain = result.stdout.strip().splitlines()
    return dict(zip(names, plain)) if len(plain) == len(names) else {name: name for name in names}


def _short(name: str) -> str:
    name = re.sub(r"sc::\(anonymous namespace\)::", "", name)
    name = re.sub(r"\((?:[^()]|\([^()]*\))*\)$", "", name)  # drop the parameter list
    name = name.replace("(sc::payload_type)0", "f32").replace("(sc::payload_type)1", "bf16")
    return re.sub(r"^void ", "", name)


def collect() -> List[Dict[str, object]]:
    rows: List[Dict[str, object]] = []
    for source in SOURCES:
        command = ["nvcc", *FLAGS, "-I", CSRC, os.path.join(CSRC, source)]
        result = subprocess.run(command, capture_output=True, text=True, cwd=CSRC)
        if result.returncode != 0:
            raise RuntimeError(f"nvcc failed on {source}:\n{result.stderr[-4000:]}")
        current = None
        for line in result.stderr.splitlines():
            entry = re.search(r"Compiling entry function '([^']+)' for 'sm_100a'", line)
            if entry:
                current = {"source": source, "mangled": entry.group(1), "registers": None, "spill_stores": 0, "spill_loads": 0,
                           "stack": 0, "shared": 0}
                rows.append(current)
                continue
            if current is None:
                continue
            frame = re.search(r"(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", line)
            if frame and current["registers"] is None:  # the entry's own line comes before those of the functions it calls
                current["stack"], current["spill_stores"], current["spill_loads"] = (int(v) for v in frame.groups())
            used = re.search(r"Used (\d+) registers", line)
            if used:
                current["registers"] = int(used.group(1))
                shared = re.search(r"(\d+) bytes smem", line)
                current["shared"] = int(shared.group(1)) if shared else 0
    names = _demangle([str(row["mangled"]) for row in rows])
    for row in rows:
        row["name"] = _short(names[str(row["mangled"])])
    return rows


def render(rows: List[Dict[str, object]]) -> str:
    lines = ["# What ptxas made of every kernel (sm_100a)", "",
             "Generated by `python -m scalingcontrasts_b200.utils.ptxas_report profiles/ptxas.md` from `nvcc -Xptxas -v` with the",
             "build's flags (`-O3 -std=c++17 -lineinfo -gencode arch=compute_100a,code=sm_100a --expt-relaxed-constexpr`).",
             "Registers per thread, spill traffic and stack in bytes per thread, static shared memory in bytes per block.", "",
             "| source | kernel | registers | spill stores | spill loads | stack | static smem |", "|---|---|---|---|---|---|---|"]
    for row in sorted(rows, key=lambda r: (str(r["source"]), str(r["name"]))):
        lines.append(f"| `{row['source']}` | `{row['name']}` | {row['registers']} | {row['spill_stores']} | {row['spill_loads']} | "
                     f"{row['stack']} | {row['shared']} |")
    lines += ["",
              "Dynamic shared memory (set by the launchers), K the number of prefixes: `forward_kernel<K, form>` (forms: 0 one CTA per tile,",
              "1 pairs of CTAs, 2 pairs without anything of the diagonal, 3 fused) as many stages as fit, up to eight (24 KB each, in a pair",
              "16 KB), beside 16 KB of store patches per band (four bands in rotation from K = 7 on), norms and row factors; fused two 32 KB stages of the",
              "gradient GEMM and six to two scoring stages (227,968 bytes, three stages, at K = 5); `backward_kernel` 214,128 bytes (a 208 KB",
              "ring of three to six stages, a stage being the CTA's row blocks of the cube plus its tile's candidates), or half the ring",
              "where two CTAs share a multiprocessor. Threads per block: 640 (forward; 96 registers at launch, 104 in the epilogue's",
              "warpgroups and 64 in the helpers' after the hand-over), 192 (backward), 512 (bandwidth collectives), up to 1024 (one-round",
              "all-reduce, norms).", ""]
    return "\n".join(lines)


def main() -> int:
    target = sys.argv[1] if len(sys.argv) > 1 else os.path.join(ROOT, "profiles", "ptxas.md")
    text = render(collect())
    with open(target, "w") as handle:
        handle.write(text)
    print(f"wrote {target}")
    return 0


if __name__ == "__main__":
    sys.exit(main())
