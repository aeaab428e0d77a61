"""TEST INFRASTRUCTURE: executes the instruction list that the compiler produces on numpy arrays, one per memory location.

Memory is what the GPU's would be: views share their array's bytes, an instruction that writes into another location's
memory overwrites it, a variable keeps its array from call to call. So an instruction that runs on the wrong side of an
update sees the wrong value here too. What is a race on the GPU is an error here: an operand that the blocks of one
launch read while other blocks of it overwrite it.
"""
from types import SimpleNamespace

import numpy as np

from cgt_b200 import compilation, core
from oracle import cpu_backend
from oracle import oracle as O

_UNARY = {code: name for (name, code) in core.UNARY_OPCODE.items()}
_BINARY = {code: name for (name, code) in core.BINARY_OPCODE.items()}


def _same_memory(a, b):
    return a.__array_interface__["data"] == b.__array_interface__["data"] and a.size == b.size


def _no_race(op, reads, write):
    for r in reads:
        assert not np.shares_memory(r, write), "%r reads the memory that it overwrites" % (op,)


def _chain(op, args, shape):
    """Results of a FusedElwise's program, `args` in the order of its inputs."""
    regs = []
    for (k, (x, kind)) in enumerate(zip(args, op.in_kinds)):
        if kind in (2, 3):
            x = np.full(shape, np.asarray(x).reshape(-1)[0], "f4")
        elif kind == 7:
            (first, pitch) = op.views[k]
            x = np.asarray(x).reshape(shape[0], pitch)[:, first:first + shape[1]]
        elif kind == 4:
            x = np.broadcast_to(np.asarray(x), shape)
        else:
            x = np.asarray(x).reshape(shape)
        regs.append(np.ascontiguousarray(x, "f4"))
    for (arity, code, a, b) in op.program:
        r = O.unary(_UNARY[code], regs[a], "f4") if arity == 1 else O.binary(_BINARY[code], regs[a], regs[b], "f4")
        regs.append(np.asarray(r, "f4").reshape(shape))
    return [regs[r] for r in op.out_regs]


class HostRun(object):
    """f = HostRun(inputs, outputs, updates): call it like the compiled function; ``value(variable)`` reads a variable."""

    def __init__(self, inputs, outputs, updates=()):
        self.variables = {}
        for node in core.topsorted(list(outputs) + [n for (_v, n) in updates] + [v for (v, _n) in updates]):
            if node.is_data():
                self.variables[node.op] = np.array(node.op.get_value(), order="C", copy=True)
        (self.eg, outs, memloc) = compilation.execution_graph(list(inputs), list(outputs), list(updates), [])
        self.out_locs = [memloc[o].index for o in outs]
        self._oracle = cpu_backend.OracleFunction([], [])
        self._oracle.values = self.variables

    def value(self, variable):
        return self.variables[variable.op].copy()

    def ops(self):
        return [i.op for i in self.eg.instrs if getattr(i, "op", None) is not None]

    def __call__(self, *args):
        mem = {}
        for ins in self.eg.instrs:
            w = ins.write_loc.index
            if isinstance(ins, compilation.LoadArgument):
                mem[w] = np.ascontiguousarray(args[ins.ind])
                continue
            reads = [mem[r.index] for r in ins.read_locs]
            if isinstance(ins, compilation.Alloc):
                mem[w] = np.full([int(s) for s in reads], np.nan if ins.dtype[0] == "f" else 77, ins.dtype)
            elif isinstance(ins, compilation.BuildTup):
                mem[w] = tuple(reads)
            elif isinstance(ins, compilation.ReturnByVal):
                mem[w] = self._view(ins, reads)
            else:
                self._into(ins, reads, mem[w])
        return [np.array(mem[o], copy=True) for o in self.out_locs]

    def _view(self, ins, reads):
        op = ins.op
        if isinstance(op, core.InMemoryData):
            return self.variables[op]
        if isinstance(op, core.LeadingSlice):
            return reads[0][int(reads[1]):int(reads[2])]
        return self._oracle._eval(SimpleNamespace(op=op, dtype=None), reads)

    def _into(self, ins, reads, write):
        op = ins.op
        if isinstance(op, core.FusedElwise):
            writes = write if isinstance(write, tuple) else (write,)
            for r in reads:
                for out in writes:
                    assert _same_memory(r, out) or not np.shares_memory(r, out) or out.size == 1, "%r overlaps its result" % (op,)
            results = _chain(op, reads, writes[0].shape)
        elif isinstance(op, core.MultiFusedElwise):
            n_in = len(op.fused.in_kinds)
            writes = (write,) + tuple(reads[op.k * n_in:])
            per = [reads[t * n_in:(t + 1) * n_in] for t in range(op.k)]
            for (t, args) in enumerate(per):
                for (u, out) in enumerate(writes):
                    if u != t:
                        _no_race(op, args, out)
            results = [_chain(op.fused, args, out.shape)[0] for (args, out) in zip(per, writes)]
        elif isinstance(op, core.Mul22Chain):
            writes = write if isinstance(write, tuple) else (write,)
            for out in writes:
                _no_race(op, reads[:2], out)
            args = list(reads[2:])
            args.insert(op.product, O.mul22(reads[0], reads[1], op.tA, op.tB))
            results = _chain(op.chain, args, op.shape)
        elif isinstance(op, core.SumSquares):
            (writes, results) = (write, [np.square(r).sum(dtype="f4") for r in reads])
        else:
            if not isinstance(op, (core.ElwiseUnary, core.ElwiseBinary)) and op.writes_to_input < 0:
                _no_race(op, [r for r in reads if isinstance(r, np.ndarray)], write)
            (writes, results) = ((write,), [self._oracle._eval(SimpleNamespace(op=op, dtype=write.dtype.str[1:]), reads)])
        results = [np.array(r, copy=True) for r in results]
        for (out, r) in zip(writes, results):
            out[...] = r.reshape(out.shape)
