"""Reading and writing safetensors files as plain {name: (dtype, shape, bytes)}, for tests that put checkpoints together."""
import json
import struct


def read_safetensors(path):
    with open(path, "rb") as f:
        header = json.loads(f.read(struct.unpack("<Q", f.read(8))[0]))
        data = f.read()
    return {k: (v["dtype"], v["shape"], data[v["data_offsets"][0]:v["data_offsets"][1]]) for k, v in header.items() if k != "__metadata__"}


def write_safetensors(path, tensors):
    header, at = {}, 0
    for k, (dtype, shape, raw) in tensors.items():
        header[k] = {"dtype": dtype, "shape": shape, "data_offsets": [at, at + len(raw)]}
        at += len(raw)
    text = json.dumps(header, separators=(",", ":")).encode()
    text += b" " * (-len(text) % 8)
    with open(path, "wb") as f:
        f.write(struct.pack("<Q", len(text)) + text)
        for _, _, raw in tensors.values():
            f.write(raw)
    return path
