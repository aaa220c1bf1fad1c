"""functs_b200_rprogram (include/functs_b200.h) for ctypes, and a program of interleaved regions in it."""
import ctypes
from ctypes import Structure, c_float, c_int32, c_uint16, c_uint32, c_void_p

END, LOAD, CONST, MUL_IMM = 0, 1, 2, 62


class Load(Structure):
    _fields_ = [("tensor", c_int32), ("dtype", c_int32), ("base", c_int32), ("coef", c_int32 * 4)]


class Region(Structure):
    _fields_ = [("rank", c_int32), ("count", c_int32), ("shape", c_int32 * 4), ("div_magic", c_uint32 * 4), ("div_shift", c_uint32 * 4),
                ("out_base", c_int32), ("out_coef", c_int32 * 4), ("first_instr", c_int32), ("first_load", c_int32), ("num_loads", c_int32)]


class Instr(Structure):
    _fields_ = [("op", c_uint16), ("arg", c_uint16), ("imm", c_float)]


class Program(Structure):
    _fields_ = [("num_regions", c_int32), ("interleave", c_int32), ("out_dtype", c_int32), ("numel", c_int32), ("num_instr", c_int32),
                ("num_loads", c_int32), ("in_ptr", c_void_p * 16), ("out_ptr", c_void_p), ("region", Region * 16), ("instr", Instr * 384),
                ("load", Load * 96)]


def interleaved(width: int, rows: int, bases, x_ptr: int, out_ptr: int) -> Program:
    """out[i, r] = 2 * x[i, bases[r]] for r < len(bases), r for the columns behind them; x and out are [rows, width]."""
    p = Program()
    p.num_regions = p.interleave = width
    p.numel = rows * width
    p.in_ptr[0], p.out_ptr = x_ptr, out_ptr
    for r in range(width):
        g = p.region[r]
        g.rank, g.count, g.out_base, g.first_instr, g.first_load = 1, rows, r, p.num_instr, p.num_loads
        g.shape[:], g.out_coef[0] = [rows, 1, 1, 1], width
        if r < len(bases):
            load = p.load[p.num_loads]
            load.base, load.coef[0] = bases[r], width
            code = [(LOAD, p.num_loads, 0.0), (MUL_IMM, 0, 2.0)]
            g.num_loads = 1
            p.num_loads += 1
        else:
            code = [(CONST, 0, float(r))]
        for op, arg, imm in code + [(END, 0, 0.0)]:
            p.instr[p.num_instr] = Instr(op, arg, imm)
            p.num_instr += 1
    return p


def address(p: Program) -> int:
    return ctypes.addressof(p)
