"""Registers / spills / shared memory of every kernel, from `nvcc -Xptxas -v` (runs without a GPU):

    python tools/ptxas_table.py > profiles/ptxas_resources.md

Same flags as gllm_b200/build.py. A spill or a register count near the launch bound is the first thing to check
before spending GPU time on a kernel change."""
import os
import re
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
from gllm_b200 import build as B  # noqa: E402


def main():
    rows = []
    for src in B._sources():
        cmd = [B.nvcc_path(), *B.NVCC_FLAGS, "-I", B.CSRC, "-Xptxas", "-v", "-c", src, "-o", "/tmp/_ptxas_table.o"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        text = subprocess.run(["cu++filt"], input=r.stderr, capture_output=True, text=True).stdout
        cur = None
        for line in text.splitlines():
            m = re.search(r"Compiling entry function '(.*)' for 'sm_100a'", line)
            if m:
                cur = {"name": m.group(1), "file": os.path.relpath(src, B.CSRC)}
                continue
            if cur is None:
                continue
            m = re.search(r"(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", line)
            if m:
                cur["stack"], cur["sst"], cur["sld"] = map(int, m.groups())
            m = re.search(r"Used (\d+) registers(?:, used (\d+) barriers)?(?:, (\d+) bytes smem)?", line)
            if m:
                cur["regs"] = int(m.group(1))
                cur["bars"] = int(m.group(2) or 0)
                cur["smem"] = int(m.group(3) or 0)
                rows.append(cur)
                cur = None
    print("# ptxas resource usage per kernel (`nvcc -Xptxas -v`, sm_100a, flags of gllm_b200/build.py)\n")
    print("Generated by `tools/ptxas_table.py`. `smem` is static shared memory only (the TMA / tcgen05 kernels take "
          "their pipeline stages as dynamic shared memory, up to 220 KB); spills are bytes of local-memory traffic "
          "inserted by the register allocator.\n")
    print("| kernel | source | registers | static smem (B) | stack (B) | spill stores / loads (B) |")
    print("|---|---|---|---|---|---|")
    for r in rows:
        short = re.sub(r"^(void )?b200::", "", r["name"])
        short = re.sub(r"\((?:[^()]|\([^()]*\))*\)$", "", short).replace("(int)", "").replace("(bool)", "")
        print(f"| `{short}` | `{r['file']}` | {r.get('regs', '?')} | {r.get('smem', 0)} | {r.get('stack', 0)} | "
              f"{r.get('sst', 0)} / {r.get('sld', 0)} |")
    spills = [r for r in rows if r.get("sst", 0) or r.get("sld", 0)]
    print(f"\n{len(rows)} kernels, {len(spills)} with register spills"
          + (": " + ", ".join(re.sub(r'^(void )?b200::', '', r['name']).split('(')[0] for r in spills) if spills else "."))


if __name__ == "__main__":
    main()
