"""The work a user of this library has it do, as cases that can be timed and compared.

`listed()` names twelve fixed cases, `draw()` gives further ones of the same ranges, `prepare()` makes what a
program holds before the call (a loaded texture set, resident latents and networks, queries, images), `run()`
is one pass through the public entry points of `rtxntc-library_b200/binding.py`, `work()` states the bytes and
operations that pass cannot do without.

The kinds of case:
  decode     one decode launch of a resident set: the whole mip chain (or mip 0 alone) as fp16 texels on the device
  load       a container taken in, decompressed, and every mip read back to pinned host memory
  pixels     decompress with the converting epilogue: the client's pixels straight into a device buffer
  sample     inference on sample, (u, v, lod) queries against resident data
  lookup     the same at the texture-set level, where the call waits for its answers
  transcode  decompress, then every texture of the set as BCn blocks, mip by mip, by the set's own texture headers
  search     the offline BC7 encoder: full search over one image
  finalize   the end of a compression run: latents packed, the network quantised to both blobs
"""
from __future__ import annotations

import numpy as np
import torch

import __graft_entry__ as entry

entry.load_package()
from rtxntc_library_b200 import binding, geometry, synthetic  # noqa: E402

FLOPS_PER_TEXEL = 2 * sum(i * o for i, o in zip(geometry.MLP_LAYER_INPUTS, geometry.MLP_LAYER_OUTPUTS))
PIXEL_FORMATS = {"unorm8": (binding.CHANNEL_FORMAT_UNORM8, torch.uint8), "unorm16": (binding.CHANNEL_FORMAT_UNORM16, torch.int16),
                 "float16": (binding.CHANNEL_FORMAT_FLOAT16, torch.float16), "float32": (binding.CHANNEL_FORMAT_FLOAT32, torch.float32)}
BLOCK_BYTES = {"BC1": 8, "BC4": 8, "BC5": 16, "BC7": 16}


def listed():
    return [
        # a material's smallest set, ragged in both directions: launch and host cost are all there is
        dict(name="decode_96x40", kind="decode", width=96, height=40, channels=8, mips=0, scale=3, features=12,
             weights="fp8", numerics="reference", layout="interleaved"),
        # one streamed-in mip of a simple material
        dict(name="decode_1024_mip0", kind="decode", width=1024, height=1024, channels=4, mips=1, scale=2, features=8,
             weights="int8", numerics="reference", layout="interleaved"),
        # the PBR set of the benchmark: 12 channels, full chain, FP8 weights
        dict(name="decode_4096", kind="decode", width=4096, height=4096, channels=12, mips=0, scale=4, features=12,
             weights="fp8", numerics="reference", layout="interleaved"),
        # the largest set: 16 channels of high-quality latents
        dict(name="decode_8192", kind="decode", width=8192, height=8192, channels=16, mips=0, scale=4, features=16,
             weights="int8", numerics="reference", layout="interleaved"),
        # a screen-sized, non-power-of-two set with the other accumulation and the other layout
        dict(name="decode_1920x1080_exact", kind="decode", width=1920, height=1080, channels=10, mips=0, scale=4, features=8,
             weights="int8", numerics="exact", layout="planar"),
        # one set of a batch, from its file's bytes to texels in host memory
        dict(name="load_2048", kind="load", width=2048, height=2048, channels=8, mips=0, scale=4, features=8,
             weights="int8", format="float16"),
        # the PBR set as 8-bit pixels, its colour channels encoded to sRGB, for a renderer on the same GPU
        dict(name="pixels_4096", kind="pixels", width=4096, height=4096, channels=12, mips=0, scale=4, features=12,
             weights="fp8", format="unorm8", first=0, count=12, components=12, srgb=3, dither=False),
        # incoherent queries against the PBR set
        dict(name="sample_16m", kind="sample", width=4096, height=4096, channels=12, mips=0, scale=4, features=12,
             weights="fp8", queries=1 << 24),
        # a handful of queries, as a picking or streaming-feedback pass asks them
        dict(name="lookup_3000", kind="lookup", width=2048, height=2048, channels=8, mips=0, scale=4, features=8,
             weights="int8", queries=3000),
        # "decompress on load, then BCn": albedo by stored BC7 modes, normals, two masks and a colour, full chain
        dict(name="transcode_2048", kind="transcode", width=2048, height=2048, channels=12, mips=0, scale=4, features=12, weights="fp8"),
        # the offline pass that chooses the BC7 modes of an albedo map
        dict(name="search_1024", kind="search", width=1024, height=1024, channels=12, first=0, count=3),
        # the end of compressing a 4096 x 4096 set
        dict(name="finalize_4096", kind="finalize", width=4096, height=4096, channels=12, mips=0, scale=4, features=12),
    ]


def draw(rng):
    def side(low, high):
        value = int(round(2.0 ** rng.uniform(np.log2(low), np.log2(high))))
        return 1 << int(round(np.log2(value))) if rng.random() < 0.3 else value  # powers of two are common in earnest

    kind = rng.choice(["decode", "decode", "decode", "load", "pixels", "sample", "lookup", "transcode", "search", "finalize"])
    case = dict(kind=kind, width=side(40, 2048 if kind in ("load", "transcode", "search") else 4096))
    # textures are square or near it; the sides are drawn apart so that ragged ones come up in either direction
    case["height"] = max(24, int(case["width"] * rng.choice([1.0, 1.0, 0.5, 0.7321]))) if rng.random() < 0.7 else side(40, 2048)
    case["channels"] = rng.choice([4, 6, 8, 10, 12, 16])
    if kind == "search":
        case["first"] = rng.choice([0, 1])
        case["count"] = rng.choice([3, 3, 1])
        return case
    case.update(mips=rng.choice([0, 0, 0, 1]), scale=rng.choice([2, 3, 4, 4, 5, 6]), features=rng.choice([4, 8, 12, 16]))
    if kind == "finalize":
        return case
    case["weights"] = rng.choice(["int8", "fp8"])
    if kind == "decode":
        case["numerics"] = rng.choice(["reference", "reference", "reference", "exact"])
        case["layout"] = rng.choice(["interleaved", "interleaved", "planar"])
    elif kind == "load":
        case["format"] = rng.choice(["float16", "unorm8"])
    elif kind == "pixels":
        first = rng.choice([0, 0, 2])
        count = rng.randint(1, min(4, case["channels"] - first)) if rng.random() < 0.5 else case["channels"] - first
        case.update(format=rng.choice(["unorm8", "unorm8", "unorm16", "float16", "float32"]), first=first, count=count,
                    components=4 if count == 3 else count, srgb=rng.choice([0, min(3, count)]), dither=rng.random() < 0.3)
    elif kind in ("sample", "lookup"):
        case["queries"] = int(2.0 ** (rng.uniform(14, 24) if kind == "sample" else rng.uniform(6, 17)))
    elif kind == "transcode":
        case["channels"] = rng.choice([8, 10, 12])
    return case


# ---- what a program has in hand before the call -------------------------------------------------------------


def _geometry(case):
    mips = case["mips"] or geometry.full_mip_count(case["width"], case["height"])
    return geometry.make_geometry(case["width"], case["height"], case["channels"], min(mips, geometry.MAX_MIPS), case["scale"],
                                  case["features"])


def _smooth(generator, planes, height, width, coarseness, noise):
    """[planes][height][width] in [0, 1]: values that vary over `coarseness` pixels, with a little noise on top, as
    latents and texels of real textures do."""
    coarse = torch.rand((1, planes, height // coarseness + 2, width // coarseness + 2), device="cuda", generator=generator)
    image = torch.nn.functional.interpolate(coarse, size=(height, width), mode="bilinear", align_corners=False)[0]
    return (image + noise * (torch.rand(image.shape, device="cuda", generator=generator) - 0.5)).clamp_(0, 1)


def _latents(geo, generator):
    words = []
    for width, height in zip(geo.latent_width, geo.latent_height):
        layers = []
        for _ in range(geo.num_layers):
            codes = (_smooth(generator, 4, height, width, 8, 0.2) * 15).round_().to(torch.int32)
            layers.append(codes[0] | codes[1] << 4 | codes[2] << 8 | codes[3] << 12)
        words.append(torch.stack(layers).cpu().numpy().astype(np.uint16))
    return words


def _into_unit_range(blob, scale_offset, bias_offset):
    """The blob with its output layer scaled and moved so that texels lie around 0.5 +- 0.2, as texture data does."""
    data = bytearray(blob)
    scale = np.frombuffer(blob, "<f4", 16, scale_offset) * np.float32(0.2)
    bias = np.frombuffer(blob, "<i4", 16, bias_offset) + np.rint(0.44 / scale).astype(np.int32)
    data[scale_offset:scale_offset + 64] = scale.astype("<f4").tobytes()
    data[bias_offset:bias_offset + 64] = bias.astype("<i4").tobytes()
    return bytes(data)


def _texture_set(case, seed, textures=None):
    geo = _geometry(case)
    generator = torch.Generator(device="cuda").manual_seed(seed)
    # the networks depend on the seed alone
    network = synthetic.make_texture_set(synthetic.TextureSetSpec(16, 16, 4, 1, 1, 4, seed=seed, network="unit"))
    hidden = sum(geometry.MLP_LAYER_OUTPUTS[:3])
    weights = sum(i * o for i, o in zip(geometry.MLP_LAYER_INPUTS, geometry.MLP_LAYER_OUTPUTS))
    int8 = _into_unit_range(network.int8_blob, weights + 4 * hidden, weights + 4 * (hidden + 16) + 4 * hidden)
    fp8 = _into_unit_range(network.fp8_blob, weights + 2 * hidden, weights + 2 * hidden + 64)
    return synthetic.SyntheticSet(network.spec, geo, _latents(geo, generator), int8, fp8, textures=textures)


def _textures(channels):
    """Texture headers of a material of 8 to 12 channels."""
    headers = [{"name": "Albedo", "firstChannel": 0, "numChannels": 3, "rgbColorSpace": "sRGB", "bcFormat": "BC7"},
               {"name": "Normal", "firstChannel": 3, "numChannels": 2, "bcFormat": "BC5"},
               {"name": "Roughness", "firstChannel": 5, "numChannels": 1, "bcFormat": "BC4"},
               {"name": "Metalness", "firstChannel": 6, "numChannels": 1, "bcFormat": "BC4"}]
    if channels >= 10:
        headers.append({"name": "Emissive", "firstChannel": 7, "numChannels": 3, "bcFormat": "BC1"})
    return headers[:4 if channels < 12 else 5]


class _Loaded:
    """A texture set loaded from its container on a context of its own, both closed with the object."""

    def __init__(self, container):
        self.context = binding.Context(torch.cuda.current_device())
        self.set = self.context.create_texture_set(container)

    def __del__(self):
        self.set.close()
        self.context.close()


def _queries(case, seed):
    mips = _geometry(case).mips
    generator = torch.Generator(device="cuda").manual_seed(seed + 1)
    return torch.rand((case["queries"], 3), device="cuda", generator=generator) * torch.tensor([1.0, 1.0, mips - 1.0], device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "search":
        generator = torch.Generator(device="cuda").manual_seed(seed)
        image = _smooth(generator, case["channels"], case["height"], case["width"], 16, 0.1)
        state["texels"] = image.permute(1, 2, 0).to(torch.float16).contiguous()
        return state
    if kind == "finalize":
        # what training leaves: per neural mip the fp16 latents in [0, 1], and the fp16 network
        geo = _geometry(case)
        generator = torch.Generator(device="cuda").manual_seed(seed)
        state["latents"] = []
        for width, height in zip(geo.latent_width, geo.latent_height):
            count = width * height
            features = _smooth(generator, 4 * geo.num_layers, height, width, 8, 0.2).to(torch.float16)
            # layer by layer: features 0 and 1 of every texel, then features 2 and 3
            pairs = features.reshape(geo.num_layers, 2, 2, count).permute(0, 1, 3, 2).contiguous()
            state["latents"].append((pairs.reshape(-1), width, height, geo.num_layers, 2 * count))
        state["weights"] = (torch.randn(binding.NETWORK_WEIGHT_COUNT, device="cuda", generator=generator) * 0.2).to(torch.float16)
        state["biases"] = (torch.randn(binding.NETWORK_COLUMN_COUNT, device="cuda", generator=generator) * 0.3).to(torch.float16)
        return state

    geo = _geometry(case)
    state["int8"] = case["weights"] == "int8"
    if kind in ("decode", "sample"):
        layout = binding.LAYOUT_PLANAR_PAIRS if case.get("layout") == "planar" else binding.LAYOUT_INTERLEAVED
        numerics = binding.NUMERICS_EXACT if case.get("numerics") == "exact" else binding.NUMERICS_REFERENCE
        state["resident"] = binding.ResidentTextureSet.from_synthetic(
            _texture_set(case, seed), device="cuda:%d" % torch.cuda.current_device(), layout=layout, numerics=numerics,
            allocate_output=kind == "decode")
        if kind == "sample":
            state["queries"] = _queries(case, seed)
            state["resident"].interleave_latents()
        return state
    data = _texture_set(case, seed, _textures(case["channels"]) if kind == "transcode" else None)
    loaded = state["loaded"] = _Loaded(data.container)
    if kind == "load":
        state["container"] = data.container
        state["host"] = torch.empty(geo.total_texels * geo.channels, dtype=PIXEL_FORMATS[case["format"]][1]).pin_memory()
    elif kind == "pixels":
        channel_format, dtype = PIXEL_FORMATS[case["format"]]
        spaces = [binding.COLOR_SPACE_SRGB] * case["srgb"] + [binding.COLOR_SPACE_LINEAR] * (case["count"] - case["srgb"])
        state["conversion"] = binding.make_conversion(channel_format, case["count"], case["first"], case["components"],
                                                      dst_color_spaces=spaces, use_dithering=case["dither"])
        state["pixels"] = torch.empty(geo.total_texels * case["components"], dtype=dtype, device="cuda")
    elif kind == "lookup":
        state["queries"] = _queries(case, seed)
    elif kind == "transcode":
        # the set carries the BC7 modes that an offline search chose
        loaded.set.decompress(state["int8"])
        for mip in range(geo.mips):
            blocks = loaded.set.block_compress(mip, binding.BLOCK_FORMAT_BC7, 0, 3)
            loaded.set.make_and_store_bc7_mode_buffer(0, mip, blocks.cpu().numpy())
    return state


# ---- one pass ---------------------------------------------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "decode":
        state["resident"].decode(state["int8"])
        return state["resident"].out
    if kind == "load":
        texture_set = state["loaded"].set
        texture_set.load_from_memory(state["container"])
        texture_set.decompress(state["int8"])
        host, channels = state["host"], texture_set.desc.channels
        address = host.data_ptr()
        for mip in range(texture_set.desc.mips):
            width, height = texture_set.mip_size(mip)
            texture_set.read_channels_into(mip, address, channel_format=PIXEL_FORMATS[case["format"]][0])
            address += width * height * channels * host.element_size()
        return host
    if kind == "pixels":
        state["loaded"].set.decompress_converted(state["conversion"], state["int8"], device_address=state["pixels"].data_ptr())
        return state["pixels"]
    if kind == "sample":
        return state["resident"].sample(state["queries"], state["int8"], interleaved=True)
    if kind == "lookup":
        return state["loaded"].set.sample(state["queries"], state["int8"])
    if kind == "transcode":
        texture_set = state["loaded"].set
        texture_set.decompress(state["int8"])
        return [texture_set.block_compress_texture(texture, mip)
                for texture in range(len(_textures(case["channels"]))) for mip in range(texture_set.desc.mips)]
    if kind == "search":
        return binding.block_compress(state["texels"], binding.BLOCK_FORMAT_BC7, case["first"], num_channels=case["count"])
    packed = [binding.pack_latents(*arguments) for arguments in state["latents"]]
    blobs = [binding.quantize_network(state["weights"], state["biases"], mode) for mode in (binding.WEIGHTS_INT8, binding.WEIGHTS_FP8)]
    return packed + blobs


# ---- what a pass cannot do without ------------------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "search":
        blocks = ((case["width"] + 3) // 4) * ((case["height"] + 3) // 4)
        return {"bytes": case["width"] * case["height"] * case["count"] * 2 + blocks * 16, "flops": 0}
    geo = _geometry(case)
    if kind == "finalize":
        blobs = geometry.INT8_BLOB_BYTES + geometry.FP8_BLOB_BYTES + 2 * (binding.NETWORK_WEIGHT_COUNT + binding.NETWORK_COLUMN_COUNT)
        return {"bytes": geo.total_latent_pixels * geo.num_layers * (8 + 2) + blobs, "flops": 0}
    data = geo.encoded_latent_bytes + (geometry.INT8_BLOB_BYTES if case["weights"] == "int8" else geometry.FP8_BLOB_BYTES)
    if kind in ("sample", "lookup"):
        # a query reads at most eight latent pixels, however large the set is
        touched = min(geo.encoded_latent_bytes, case["queries"] * 8 * geo.num_layers * 2)
        return {"bytes": touched + case["queries"] * (12 + 2 * geo.channels), "flops": case["queries"] * FLOPS_PER_TEXEL}
    flops = geo.total_texels * FLOPS_PER_TEXEL
    if kind == "transcode":
        blocks = sum(((mip.width + 3) // 4) * ((mip.height + 3) // 4) for mip in geo.color_mips)
        return {"bytes": data + blocks * sum(BLOCK_BYTES[t["bcFormat"]] for t in _textures(case["channels"])), "flops": flops}
    values = geo.total_texels * (case["components"] if kind == "pixels" else geo.channels)
    size = torch.empty(0, dtype=PIXEL_FORMATS[case.get("format", "float16")][1]).element_size()
    return {"bytes": data + values * size, "flops": flops}


def tolerance(case):
    # Texels, answers, pixels, blocks and blobs are a fixed function of the file: every rounding of the arithmetic is
    # part of the format's contract, so another correct implementation gives the same bits.
    return "exact"
