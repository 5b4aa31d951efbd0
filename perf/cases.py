"""The work a user of this library has it do, as measurable cases.

Every case is a negacyclic product c = a*b mod (X^N + 1, q), or several, through a public entry
point of the Python mirror over the C ABI. A case holds the ring size `n`, the bit width `bits`
of q (L = ceil(bits / 32) limbs per coefficient) and the `form`:

  device   Plan.run_device: device arrays in and out, enqueued on the current stream
  static   Plan.run_device_static: the same without allocation, work space in the library
  batch    Batch.run_device: `count` uneven products in one graph launch
  pinned   Plan.run: page-locked host arrays in and out
  host     fherma_run: pageable host arrays, a fresh result array per call
  serve    Server: `count` requests submitted at once and waited for

Moduli are random and odd with exactly `bits` bits; operands are uniform below q's top word times
2^(32 (L-1)), and so below q.
"""
import importlib
import math

import numpy as np
import torch

fpc = importlib.import_module("fherma-polynomial-cuda_b200")


def listed():
    return [
        # A toy ring with a one-word-pair modulus: what an interactive user or a unit test calls;
        # launches and latency are all there is.
        {"name": "device n256 64b", "form": "device", "n": 256, "bits": 64},
        # A small RLWE-sized ring with an odd number of limbs and a width that is no multiple of 32.
        {"name": "device n2048 397b", "form": "device", "n": 2048, "bits": 397},
        # The smallest configuration of the benchmark set: N=4096, 64 limbs.
        {"name": "device n4096 2048b", "form": "device", "n": 4096, "bits": 2048},
        # The entry point for processes that may not allocate, near its size limit.
        {"name": "static n8192 4096b", "form": "static", "n": 8192, "bits": 4096},
        # The reference's two ranked points, operands already on the device.
        {"name": "device n32768 868b", "form": "device", "n": 32768, "bits": 868},
        {"name": "device n65536 1747b", "form": "device", "n": 65536, "bits": 1747},
        # Wide rows of a ragged length (301 limbs, a partial top word), between the two groups.
        {"name": "device n16384 9601b", "form": "device", "n": 16384, "bits": 9601},
        # The benchmark set's second and third configurations: 868 and 1747 limbs.
        {"name": "device n32768 27776b", "form": "device", "n": 32768, "bits": 27776},
        {"name": "device n65536 55904b", "form": "device", "n": 65536, "bits": 55904},
        # A batch of uneven small and medium products, as a scheduler of ciphertext work issues them.
        {"name": "batch 24 uneven", "form": "batch", "n": 8192, "bits": 4704, "count": 24},
        # The reference's smaller ranked point exactly as its harness calls it: pageable arrays in,
        # a fresh array out.
        {"name": "host n32768 868b", "form": "host", "n": 32768, "bits": 868},
        # The larger one from page-locked arrays.
        {"name": "pinned n65536 1747b", "form": "pinned", "n": 65536, "bits": 1747},
    ]


def draw(rng):
    """One more case: ring sizes 2^6..2^16 and widths 32..55904 bits, spread over their logarithms."""
    form = rng.choices(["device", "batch", "host", "pinned", "serve"], [14, 2, 1, 1, 1])[0]
    n = 1 << rng.randint(6, 16)
    bits = max(33, int(round(math.exp(rng.uniform(math.log(33), math.log(55904))))))
    if form in ("batch", "serve"):  # many products: each of moderate size
        return {"form": form, "n": min(n, 1 << 13), "bits": min(bits, 6000), "count": rng.randint(3, 24)}
    if form in ("host", "pinned"):  # host rows of up to 256 limbs, N up to 2^16
        return {"form": form, "n": n, "bits": min(bits, 8192)}
    return {"form": form, "n": n, "bits": bits}


def _products(case):
    """(n, bits) of every product of the case. Batches and request mixes are uneven: ring sizes from
    n/4 to 2n and widths from an eighth of `bits` to all of it, in a fixed order."""
    count = case.get("count", 1)
    if count == 1:
        return [(case["n"], case["bits"])]
    out = []
    for i in range(count):
        n = max(64, case["n"] * (1, 2, 4, 8)[(5 * i + 2) % 4] // 4)
        bits = case["bits"]
        if case["form"] == "batch":  # every product has a modulus of its own
            bits = max(33, bits * (1 + (3 * i) % 8) // 8 - 7 * (i % 5))
        out.append((n, bits))
    return out


def _modulus(bits, seed):
    """Random odd q with exactly `bits` bits, as limbs."""
    limbs = (bits + 31) // 32
    q = np.random.Generator(np.random.PCG64([seed, bits])).integers(0, 1 << 32, limbs, dtype=np.uint64).astype(np.uint32)
    top = bits - 32 * (limbs - 1)
    q[-1] = (int(q[-1]) & ((1 << top) - 1)) | (1 << (top - 1))
    q[0] |= 1
    return q


def _operand(n, q, generator):
    """[n][L] random words on the device (as int32), every coefficient below q."""
    a = torch.randint(-(1 << 31), 1 << 31, (n, len(q)), dtype=torch.int32, device="cuda", generator=generator)
    if len(q) > 1:
        top = torch.randint(0, int(q[-1]), (n,), dtype=torch.int64, device="cuda", generator=generator)
    else:
        top = torch.randint(0, int(q[0]), (n,), dtype=torch.int64, device="cuda", generator=generator)
    a[:, -1] = top.to(torch.int32)  # keeps the low 32 bits
    return a


def _operands(case, seed):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for i, (n, bits) in enumerate(_products(case)):
        q = _modulus(bits, seed if case["form"] == "serve" else seed + i)
        out.append((n, bits, q, _operand(n, q, generator), _operand(n, q, generator)))
    return out


class _Owner:
    """Releases a library handle with the last thing that refers to it: the state, and any view of
    the handle's own buffers."""

    def __init__(self, handle):
        self.handle = handle

    def __del__(self):
        try:
            self.handle.close()
        except Exception:
            pass


def _host(t):
    return t.cpu().numpy().view(np.uint32)


def prepare(case, seed):
    form, ops = case["form"], _operands(case, seed)
    state = {"form": form}
    n, bits, q, a, b = ops[0]
    limbs = len(q)
    if form in ("device", "static"):
        state["handle"] = fpc.Plan(n, bits, limbs, q, external_work=form == "static")
        state["a"], state["b"], state["c"] = a, b, torch.empty_like(a)
    elif form == "batch":
        batch = fpc.Batch([(n, bits, len(q), q) for n, bits, q, _, _ in ops])
        state["handle"], state["owner"], state["c"] = batch, _Owner(batch), []
        for i, (n, bits, q, a, b) in enumerate(ops):
            views = [torch.as_tensor(_Array(state["owner"], p, n, len(q)), device="cuda") for p in batch.io(i)]
            views[0].copy_(a)
            views[1].copy_(b)
            state["c"].append(views[2])
    elif form == "pinned":
        state["handle"] = fpc.Plan(n, bits, limbs, q)
        pinned = [torch.empty((n, limbs), dtype=torch.int32, pin_memory=True) for _ in range(3)]
        pinned[0].copy_(a)
        pinned[1].copy_(b)
        state["a"], state["b"], state["c"] = (t.numpy().view(np.uint32) for t in pinned)
        state["pinned"] = pinned
    elif form == "host":
        state["handle"] = fpc.fherma_init(fpc.Point(n, bits, limbs, q))
        state["inputs"] = fpc.Inputs(_host(a), _host(b))
    else:
        server = fpc.Server()
        state["handle"] = server
        state["session"] = server.open_session(bits, limbs, q, sorted({n for n, *_ in ops}))
        state["requests"] = []
        for n, bits, q, a, b in ops:
            bufs = [torch.empty((n, len(q)), dtype=torch.int32, pin_memory=True) for _ in range(3)]
            bufs[0].copy_(a)
            bufs[1].copy_(b)
            state["requests"].append((bufs, *(t.numpy().view(np.uint32) for t in bufs)))
    if "owner" not in state:
        state["owner"] = _Owner(state["handle"])
    return state


class _Array:
    """A device buffer of a library handle, for torch.as_tensor, which keeps this object and so the
    handle for as long as the tensor lives."""

    def __init__(self, owner, ptr, n, limbs):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n, limbs), "typestr": "<i4", "data": (ptr, False), "version": 3}


def run(state):
    form, handle = state["form"], state["handle"]
    if form in ("device", "static"):
        call = handle.run_device if form == "device" else handle.run_device_static
        call(state["a"].data_ptr(), state["b"].data_ptr(), state["c"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return state["c"]
    if form == "batch":
        handle.run_device(torch.cuda.current_stream().cuda_stream)
        return state["c"]
    if form == "pinned":
        return handle.run(state["a"], state["b"], state["c"])
    if form == "host":
        return fpc.fherma_run(handle, state["inputs"]).c
    tickets = [handle.submit(state["session"], a, b, c) for _, a, b, c in state["requests"]]
    return [handle.wait(t)[0] for t in tickets]


def work(case):
    """Bytes: both operands read once, the result written once. Operations: the byte products of the
    two base conversions (limbs to residues of 31-bit primes, and back), which grow with N L^2; the
    transforms between them grow with N L log N and are not counted."""
    moved = ops = 0
    for n, bits in _products(case):
        limbs = (bits + 31) // 32
        primes = -(-(2 * bits + n.bit_length() + 1) // 31)
        moved += 12 * n * limbs
        ops += 2 * (2 * n) * (4 * limbs) * (4 * primes) + 2 * n * (4 * primes) * (4 * (limbs + 2))
    return {"bytes": moved, "flops": ops}


def _exact_product(n, q, a, b):
    """The product by one multiplication of big integers (Kronecker substitution)."""
    limbs = len(q)
    modulus = int.from_bytes(q.tobytes(), "little")
    slot = (2 * modulus.bit_length() + n.bit_length() + 7) // 8

    def packed(x):
        wide = np.zeros((n, slot), np.uint8)
        wide[:, : 4 * limbs] = _host(x).view(np.uint8).reshape(n, 4 * limbs)
        return int.from_bytes(wide.tobytes(), "little")

    raw = (packed(a) * packed(b)).to_bytes(2 * n * slot, "little")
    at = [int.from_bytes(raw[i * slot:(i + 1) * slot], "little") for i in range(2 * n)]
    out = b"".join(((at[i] - at[i + n]) % modulus).to_bytes(4 * limbs, "little") for i in range(n))
    return torch.from_numpy(np.frombuffer(out, np.int32).reshape(n, limbs).copy())


def exact(case, seed):
    """Every word of the result is a whole number; it is computed here for the sizes that Python's
    own big-integer multiplication reaches in a few seconds."""
    if case.get("count", 1) > 1 or case["n"] * case["bits"] > 1 << 21:
        return None
    n, _, q, a, b = _operands(case, seed)[0]
    c = _exact_product(n, q, a, b)
    return c if case["form"] in ("device", "static") else c.numpy().view(np.uint32)
