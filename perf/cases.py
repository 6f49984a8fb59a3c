"""The work a program using this framework has it do, as cases that can be timed: batches of requests answered from
host buffers and from device memory, the serving loop, and the offline set-up of a database, over databases of
64 MiB to 16 GiB and batches of 1 to 1024 requests.

Every answer runs at the scheme's parameters (ring dimension 2048, 4 gadget digits, Q = 2^32 - 12287), the only set
`service.params` builds; the record size is any multiple of 2,048 bytes and the record count a power of two.
"""
import ctypes
import importlib.util
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package directory `altopir-public_b200` as the module `altopir_b200`."""
    if "altopir_b200" not in sys.modules:
        path = os.path.join(ROOT, "altopir-public_b200")
        spec = importlib.util.spec_from_file_location("altopir_b200", os.path.join(path, "__init__.py"),
                                                      submodule_search_locations=[path])
        module = importlib.util.module_from_spec(spec)
        sys.modules["altopir_b200"] = module
        spec.loader.exec_module(module)
    return sys.modules["altopir_b200"]


_package()
from altopir_b200 import engine, lib, offline, server, service  # noqa: E402

LEAD = 7           # a device frame starts 7 bytes into its slot, which puts its key words on a 16-byte boundary
STREAM_BATCHES = 4  # batches a streaming pass keeps in flight on two lanes
SLAB = 2048        # records a refresh loads before it sets the database up again

# entry: how the program calls the framework
#   host     alto_answer: frames and responses in pinned host memory, the whole call (uploads, answer, downloads)
#   device   alto_answer_device with graph replay: frames already in HBM, the caller waits for the batch
#   noalloc  alto_answer_device_noalloc: the same without any device allocation
#   stream   alto_enqueue_device: four batches on two lanes with graph replay, then one wait
#   serve    the serving loop: `b` clients submit, then collect their answers; their packing keys are resident
#   refresh  a database update: 2,048 new records loaded, the offline set-up on the device, one answer from it


def listed():
    return [
        # the plain small configuration, one query: the smallest call, where launches and latency count
        {"name": "host 64 MiB b1", "entry": "host", "rows": 2048, "record": 32768, "b": 1},
        # one lone request over 1 GiB, end to end and from HBM (the one-query-per-launch path)
        {"name": "host 1 GiB b1", "entry": "host", "rows": 32768, "record": 32768, "b": 1},
        {"name": "device 1 GiB b1", "entry": "device", "rows": 32768, "record": 32768, "b": 1},
        # the headline batch: 128 clients over 1 GiB, end to end and as a stream of batches from HBM
        {"name": "host 1 GiB b128", "entry": "host", "rows": 32768, "record": 32768, "b": 128},
        {"name": "stream 1 GiB b128", "entry": "stream", "rows": 32768, "record": 32768, "b": 128},
        # an odd batch over a record size that is no power of two (7 response parts of 2,048 bytes)
        {"name": "device 896 MiB b37", "entry": "device", "rows": 65536, "record": 14336, "b": 37},
        # the uneven batches of an 8 GiB server: a small one, one above a power of two, the largest
        {"name": "device 8 GiB b33", "entry": "device", "rows": 262144, "record": 32768, "b": 33},
        {"name": "host 8 GiB b200", "entry": "host", "rows": 262144, "record": 32768, "b": 200},
        {"name": "device 8 GiB b1024", "entry": "device", "rows": 262144, "record": 32768, "b": 1024},
        # a serving loop over 16 GiB with clients that come back with new queries
        {"name": "serve 16 GiB b48", "entry": "serve", "rows": 524288, "record": 32768, "b": 48},
        # a database put into service, or updated: once per database
        {"name": "refresh 1 GiB", "entry": "refresh", "rows": 32768, "record": 32768, "b": 1},
        {"name": "refresh 8 GiB", "entry": "refresh", "rows": 262144, "record": 32768, "b": 1},
    ]


def draw(rng):
    entry = rng.choice(["host", "host", "device", "device", "stream", "noalloc", "serve", "refresh"])
    while True:
        rows = 1 << rng.randint(11, 18)
        record = 2048 * int(2 ** rng.uniform(0, 4.001))   # 2 KB .. 32 KB, log-uniform, odd multiples among them
        b = int(2 ** rng.uniform(0, 10.001))              # 1 .. 1024, log-uniform
        frame = 9 + 4 * (2 * 8192 + rows)
        if entry == "host" and b * frame > 230 << 20:     # the pinned frames of the largest listed host batch
            continue
        if entry == "stream" and b * STREAM_BATCHES > 1024:
            continue
        if entry == "serve" and (b > 256 or b * frame > 128 << 20):
            continue
        if entry == "noalloc" and _noalloc_bytes(rows, record, b) > 16 << 20:
            continue
        return {"entry": entry, "rows": rows, "record": record, "b": 1 if entry == "refresh" else b}


def _noalloc_bytes(rows, record, b):
    """Scratch of a batch on the allocation-free path (the formula of include/altopir_gpu.h, terms rounded up)."""
    up = lambda x: -(-x // 256) * 256  # noqa: E731
    bp = -(-b // 4) * 4
    r = rows if rows <= 32768 else -(-rows // 32768) * 32768
    return up(4 * b) + up(4 * bp * r) + up(4 * bp * 8192) + 2 * up(4 * b * record)


def work(case):
    p = service.params(case["rows"], case["record"])
    b, rows, cols, count = case["b"], p.rows, p.record_bytes, p.count
    frame, resp = service.request_len(p), service.response_len(p)
    batches = STREAM_BATCHES if case["entry"] == "stream" else 1
    # an answer: the database and the packing matrix (4 bytes a value) once, frames in, responses out; the scan and
    # pack products on byte limbs (8-bit records x 32-bit query words, 32-bit x 32-bit)
    scan_bytes, pack_bytes = rows * cols, 4 * cols * count
    scan_ops, pack_ops = 2 * cols * rows * 4 * b, 2 * 4 * cols * count * 4 * b
    if case["entry"] == "serve":  # returning clients: their pack results are resident
        pack_bytes, pack_ops = 4 * cols * b, 0
    need = {"bytes": float(batches * (scan_bytes + pack_bytes + b * (frame + resp))),
            "flops": float(batches * (scan_ops + pack_ops))}
    if case["entry"] == "refresh":
        # plus the new records in and out, the database read, the walk's key-switch words and the packing matrix
        # written; transforms: one of n words per 2,048 records of a column, n per output and 2 (1 + tg) a walk step
        n = p.n
        ntts = cols * rows // n + cols + p.instances * (n // 2 - 1) * 2 * (1 + p.tg)
        need["bytes"] += 2.0 * min(SLAB, rows) * cols + rows * cols + 3.0 * 4 * cols * count
        need["flops"] += 3.0 * ntts * (n // 2) * 11
    return need


class _State:
    """An engine over a database (synthetic records, the first of them replaced by the seed's) with the scheme's
    offline state, and the seed's frames where the entry takes them."""

    def __init__(self, case, seed):
        self.case = dict(case)
        engine.init()
        torch.cuda.init()
        self.p = p = service.params(case["rows"], case["record"])
        rng = np.random.default_rng(seed)
        self.e = offline.blank_engine(p)
        self.public = offline.public_inputs(p)
        slab = rng.integers(0, 256, size=(min(256, p.rows), p.record_bytes), dtype=np.uint8)
        self.e.load_records(slab, int(rng.integers(0, p.rows - len(slab) + 1)))
        self.e.offline(*self.public)
        self.resp = self.e.response_len()
        self.frame = self.e.request_len()
        getattr(self, "_" + case["entry"])(case["b"], int(seed))

    def close(self):
        if getattr(self, "srv", None) is not None:
            self.srv.close()
            self.srv = None
        self.e.close()

    def __del__(self):
        self.close()

    # ------------------------------------------------------------------ inputs
    def _device_frames(self, b, seed, first=0):
        stride = -(-(LEAD + self.frame) // 256) * 256
        slots = torch.empty(b * stride, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        service.synthetic_requests_device(self.p, b, seed, slots.data_ptr(), stride, LEAD, first)
        return slots, stride

    def _host_frames(self, b, seed, first=0):
        slots, stride = self._device_frames(b, seed, first)
        frames = torch.empty((b, self.frame), dtype=torch.uint8, pin_memory=True)
        frames.copy_(slots.view(b, stride)[:, LEAD:LEAD + self.frame])
        torch.cuda.synchronize()
        return frames

    def _host(self, b, seed):
        self.frames = self._host_frames(b, seed)
        self.out = torch.zeros((b, self.resp), dtype=torch.uint8, pin_memory=True)
        self.status = np.full(b, -1, dtype=np.int32)
        self.req_p = (ctypes.c_void_p * b)(*[self.frames[i].data_ptr() for i in range(b)])
        self.len_p = (ctypes.c_size_t * b)(*[self.frame] * b)
        self.out_p = (ctypes.c_void_p * b)(*[self.out[i].data_ptr() for i in range(b)])

    def _device(self, b, seed):
        self.slots, self.stride = self._device_frames(b, seed)
        self.out = torch.zeros((b, self.resp), dtype=torch.uint8, device="cuda")
        self.status = np.full(b, -1, dtype=np.int32)
        torch.cuda.synchronize()
        self.e.set_graphs(True)

    def _noalloc(self, b, seed):
        self._device(b, seed)
        self.d_status = torch.full((b,), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()

    def _stream(self, b, seed):
        self.sets = [self._device_frames(b, seed, k * b) for k in range(STREAM_BATCHES)]
        self.out = torch.zeros((STREAM_BATCHES, b, self.resp), dtype=torch.uint8, device="cuda")
        self.d_status = torch.full((STREAM_BATCHES, b), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        self.e.set_graphs(True)
        self.e.set_lanes(2)

    def _serve(self, b, seed):
        self.frames = self._host_frames(b, seed).numpy()
        self.srv = server.Server(self.e, max_batch=256, queue_cap=512, key_bytes=256 * 4 * self.p.record_bytes)
        self.serve()  # the clients' first requests: their keys are resident from here on

    def _refresh(self, b, seed):
        self._device(b, seed)
        rng = np.random.default_rng(seed + 1)
        count = min(SLAB, self.p.rows)
        self.records = rng.integers(0, 256, size=(count, self.p.record_bytes), dtype=np.uint8)
        self.first = int(rng.integers(0, self.p.rows - count + 1))

    # ------------------------------------------------------------------ passes
    def host(self):
        r = self.e.answer_raw(self.req_p, self.len_p, self.case["b"], self.out_p, self.status)
        _check(r, self.case["b"])
        return {"responses": self.out, "status": self.status}

    def device(self):
        r = self.e.answer_device(self.slots.data_ptr(), self.stride, self.case["b"], self.out.data_ptr(), self.resp,
                                 self.status)
        _check(r, self.case["b"])
        return {"responses": self.out, "status": self.status}

    def noalloc(self):
        r = lib().alto_answer_device_noalloc(self.e.ptr, self.slots.data_ptr(), self.stride, self.case["b"],
                                             self.out.data_ptr(), self.resp, self.d_status.data_ptr())
        _check(r, 0)
        return {"responses": self.out, "status": self.d_status}

    def stream(self):
        b = self.case["b"]
        for k, (slots, stride) in enumerate(self.sets):
            self.e.enqueue_device(slots.data_ptr(), stride, b, self.out[k].data_ptr(), self.resp,
                                  self.d_status[k].data_ptr())
        self.e.sync()
        return {"responses": self.out, "status": self.d_status}

    def serve(self):
        tickets = [self.srv.submit(f) for f in self.frames]
        answers = [self.srv.wait(t) for t in tickets]
        return {"responses": np.stack([a[1] for a in answers]),
                "status": np.array([a[0] for a in answers], dtype=np.int32)}

    def refresh(self):
        self.e.load_records(self.records, self.first)
        self.e.offline(*self.public)
        return self.device()


def _check(r, want):
    if r != want:
        raise RuntimeError(f"engine returned {r}, {want} expected: {lib().alto_last_error().decode()}")


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    return getattr(state, state.case["entry"])()
