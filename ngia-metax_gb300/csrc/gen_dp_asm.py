"""Generates dp_asm.cuh: the per-residue update of a register tile of the
banded bit-parallel LCS as one inline-PTX block per tile width (and planes).

For every slot m of the tile (one 32-bit word of representative rows):
    x  = row & match word
    t  = row + x + carry                    add on the carry flag (add.cc/addc.cc)
    row = t | (row ^ x)                      one LOP3
so the carry of the multi-word addition rides the hardware carry flag from
slot to slot without leaving the flag.  The next column carry is popped from
the top bit of `cw` and the final carry is pushed into `ncw`, one instruction
each.

dp_tile builds the match word from P plane registers (one LOP3 per plane);
dp_tile_eqf takes it from the representative's match table (e[m]: one AND)
and pops and pushes the column carry by multiply-adds with a run-time 1
(mad.lo.cc / madc: cw*1 + cw), which issue on the FMA pipe.  (Every 2nd or
3rd slot's add as a multiply-add with carry was swept on GB300, 1M DNA
s=0.85: 0.97x and 0.98x.)

Run `python gen_dp_asm.py` after editing; the output is committed.
"""
from pathlib import Path

PLANES = (2, 5)
WIDTHS = tuple(range(1, 17))


def block(sig: str, outs: list, ins: list, lines: list) -> str:
    body = "\n".join(f'      "{ln}\\n\\t"' for ln in ["{"] + lines + ["}"])
    return f"{sig} {{\n  asm(\n{body}\n      : " + ", ".join(outs) + "\n      : " + ", ".join(ins) + ");\n}\n\n"


def one(P: int, TW: int) -> str:
    # operand numbering: row[0..TW-1], cw, ncw, then the planes and the column's masks
    outs = [f'"+r"(row[{m}])' for m in range(TW)] + ['"+r"(cw)', '"+r"(ncw)']
    ins = [f'"r"(pl[{p}][{m}])' for p in range(P) for m in range(TW)] + [f'"r"(mk[{p}])' for p in range(P)]
    cw, ncw, pl, mk = TW, TW + 1, TW + 2, TW + 2 + P * TW
    lines = [".reg .u32 a, x, t;", f"add.cc.u32 %{cw}, %{cw}, %{cw};"]
    for m in range(TW):
        src = f"%{m}"
        for p in range(P):
            dst = "x" if p == P - 1 else "a"
            lines.append(f"lop3.b32 {dst}, {src}, %{pl + p * TW + m}, %{mk + p}, 0x90;")
            src = "a"
        lines += [f"addc.cc.u32 t, %{m}, x;", f"lop3.b32 %{m}, t, %{m}, x, 0xF6;"]
    lines.append(f"addc.u32 %{ncw}, %{ncw}, %{ncw};")
    return block(f"template <>\n__device__ __forceinline__ void dp_tile<{P}, {TW}>(uint32_t (&row)[{TW}], "
                 f"const uint32_t (&pl)[{P}][{TW}], const uint32_t (&mk)[{P}], uint32_t &cw, uint32_t &ncw)",
                 outs, ins, lines)


def one_eqf(TW: int) -> str:
    outs = [f'"+r"(row[{m}])' for m in range(TW)] + ['"+r"(cw)', '"+r"(ncw)']
    ins = [f'"r"(e[{m}])' for m in range(TW)] + ['"r"(one)']
    cw, ncw, e, k = TW, TW + 1, TW + 2, 2 * TW + 2
    lines = [".reg .u32 x, t;", f"mad.lo.cc.u32 %{cw}, %{cw}, %{k}, %{cw};"]
    for m in range(TW):
        lines += [f"and.b32 x, %{m}, %{e + m};", f"addc.cc.u32 t, %{m}, x;", f"lop3.b32 %{m}, t, %{m}, x, 0xF6;"]
    lines.append(f"madc.lo.u32 %{ncw}, %{ncw}, %{k}, %{ncw};")
    return block(f"template <>\n__device__ __forceinline__ void dp_tile_eqf<{TW}>(uint32_t (&row)[{TW}], "
                 f"const uint32_t (&e)[{TW}], uint32_t &cw, uint32_t &ncw, uint32_t one)", outs, ins, lines)


def one_wave(W: int) -> str:
    """The update with a mask per row word (act[m]) on the match word: a row
    whose mask is 0 stays as it is."""
    outs = [f'"+r"(row[{m}])' for m in range(W)] + ['"+r"(cw)', '"+r"(ncw)']
    ins = [f'"r"(e[{m}])' for m in range(W)] + [f'"r"(act[{m}])' for m in range(W)]
    cw, ncw, e, act = W, W + 1, W + 2, 2 * W + 2
    lines = [".reg .u32 x, t;", f"add.cc.u32 %{cw}, %{cw}, %{cw};"]
    for m in range(W):
        lines += [f"lop3.b32 x, %{m}, %{e + m}, %{act + m}, 0x80;", f"addc.cc.u32 t, %{m}, x;",
                  f"lop3.b32 %{m}, t, %{m}, x, 0xF6;"]
    lines.append(f"addc.u32 %{ncw}, %{ncw}, %{ncw};")
    return block(f"template <>\n__device__ __forceinline__ void dp_wave<{W}>(uint32_t (&row)[{W}], "
                 f"const uint32_t (&e)[{W}], const uint32_t (&act)[{W}], uint32_t &cw, uint32_t &ncw)",
                 outs, ins, lines)


def main() -> None:
    parts = ["// dp_asm.cuh — generated by gen_dp_asm.py; do not edit by hand.\n"
             "// One residue (column) update of a TW-slot register tile of the banded\n"
             "// bit-parallel LCS; see gen_dp_asm.py for the algebra.\n"
             "#pragma once\n#include <stdint.h>\n\nnamespace ngia {\n\n"
             "template <int P, int TW>\n"
             "__device__ __forceinline__ void dp_tile(uint32_t (&row)[TW], const uint32_t (&pl)[P][TW],\n"
             "                                        const uint32_t (&mk)[P], uint32_t &cw, uint32_t &ncw);\n\n"
             "template <int TW>\n"
             "__device__ __forceinline__ void dp_tile_eqf(uint32_t (&row)[TW], const uint32_t (&e)[TW], uint32_t &cw,\n"
             "                                            uint32_t &ncw, uint32_t one);\n\n"
             "template <int W>\n"
             "__device__ __forceinline__ void dp_wave(uint32_t (&row)[W], const uint32_t (&e)[W], const uint32_t (&act)[W],\n"
             "                                        uint32_t &cw, uint32_t &ncw);\n\n"]
    parts += [one(P, TW) for P in PLANES for TW in WIDTHS]
    parts += [one_eqf(TW) for TW in WIDTHS]
    parts += [one_wave(W) for W in (1, 2, 4, 8, 16)]
    parts.append("}  // namespace ngia\n")
    (Path(__file__).resolve().parent / "dp_asm.cuh").write_text("".join(parts))


if __name__ == "__main__":
    main()
