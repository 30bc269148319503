// Convolution and InnerProduct: parameter handling on the host, tensor-core /
// depthwise / direct kernels on the device, fused tails folded into
// per-channel scale and shift arrays.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "../filler.h"
#include "../syncedmem.h"
#include "layers.h"

namespace caffe {

// ---------------------------------------------------------------- helpers

void DeviceArray::Assign(const std::vector<float>& host) {
  if (!blob_ || blob_->count() != static_cast<int>(host.size())) {
    blob_.reset(new Blob(vector<int>(1, static_cast<int>(host.size()))));
  }
  std::memcpy(blob_->mutable_cpu_data(), host.data(), host.size() * sizeof(float));
}

float* DeviceScratch::Reserve(size_t floats) {
  CHECK_LE(floats, static_cast<size_t>(0x7fffffff));
  if (!blob_ || static_cast<size_t>(blob_->count()) < floats) {
    blob_.reset(new Blob(vector<int>(1, static_cast<int>(floats ? floats : 1))));
  }
  return blob_->mutable_gpu_data();
}

const float* HostInput::Take(const Blob& blob) {
  const shared_ptr<SyncedMemory>& data = blob.data();
  const void* host = data ? data->host_only() : nullptr;
  if (!host) return nullptr;
  const bool again = memory_ == data.get() && version_ == data->host_version();
  memory_ = data.get();
  version_ = data->host_version();
  return again ? nullptr : static_cast<const float*>(host);
}

unsigned long long TailVersion(const FusedTail& tail) {
  unsigned long long v = 0;
  for (Layer* l : tail.affine) v += l->ParamVersion();
  if (tail.activation) v += tail.activation->ParamVersion();
  return v;
}

void FoldTail(const FusedTail& tail, int channels, const float* bias, std::vector<float>* scale,
              std::vector<float>* shift, bool* has_scale, bool* has_shift) {
  std::vector<double> s(channels, 1.0), b(channels, 0.0);
  *has_scale = false;
  *has_shift = false;
  if (bias) {
    for (int c = 0; c < channels; ++c) b[c] = bias[c];
    *has_shift = true;
  }
  for (Layer* l : tail.affine) {
    std::vector<double> ls, lb;
    CHECK(l->AsChannelAffine(channels, &ls, &lb)) << l->type() << " layer cannot be folded";
    for (int c = 0; c < channels; ++c) {
      s[c] *= ls[c];
      b[c] = b[c] * ls[c] + lb[c];
    }
    *has_scale = true;
    *has_shift = true;
  }
  if (tail.self_coeff != 1.f) {
    for (int c = 0; c < channels; ++c) {
      s[c] *= tail.self_coeff;
      b[c] *= tail.self_coeff;
    }
    *has_scale = true;
  }
  scale->assign(s.begin(), s.end());
  shift->assign(b.begin(), b.end());
}

void FillTailEpilogue(const FusedTail& tail, const DeviceArray& scale, const DeviceArray& shift,
                      ResidualCopy residual_copy, int channels, mcb200_epilogue* ep) {
  *ep = mcb200_epilogue();
  ep->scale = scale.get();
  ep->shift = shift.get();
  ep->residual_coeff = 1.f;
  if (tail.residual) {
    ep->residual = residual_copy == kResidualNhwcHalf
                       ? static_cast<const float*>(tail.residual->gpu_data_nhwc_bf16())   // 16-bit cells
                       : (residual_copy == kResidualNhwc ? tail.residual->gpu_data_nhwc() : tail.residual->gpu_data());
    ep->residual_ld = channels;
    ep->residual_coeff = tail.residual_coeff;
  }
  if (tail.activation) {
    ActivationSpec spec;
    CHECK(tail.activation->AsActivation(&spec));
    ep->act = spec.kind;
    ep->slope = spec.slope;
    if (spec.kind == 2) {
      ep->prelu = spec.slopes->gpu_data();
      ep->prelu_shared = spec.shared ? 1 : 0;
    }
  }
}

// ---------------------------------------------------------------- Convolution

// Kernel, stride, pad and dilation of a 2-D convolution from either the _h/_w
// fields or the repeated fields (src/layers/base_conv_layer.cpp:22-88, same rules
// and messages).
void ParseConvolutionGeometry(const ConvolutionParameter& p, mcb200_conv_shape* shape) {
  mcb200_conv_shape& s = *shape;
  auto pick = [&](bool has_h, bool has_w, int vh, int vw, int rep_size, const char* what, int dflt, int* oh, int* ow,
                  auto rep) {
    if (has_h || has_w) {
      CHECK_EQ(0, rep_size) << "Either " << what << " or " << what << "_h/w should be specified; not both.";
      *oh = vh;
      *ow = vw;
    } else {
      CHECK(rep_size == 0 || rep_size == 1 || rep_size == 2)
          << what << " must be specified once, or once per spatial dimension (" << what << " specified " << rep_size
          << " times; 2 spatial dims).";
      *oh = rep_size == 0 ? dflt : static_cast<int>(rep(0));
      *ow = rep_size == 0 ? dflt : static_cast<int>(rep(rep_size == 1 ? 0 : 1));
    }
  };
  CHECK(p.has_kernel_h() || p.has_kernel_w() || p.kernel_size_size() > 0) << "kernel_size must be specified";
  pick(p.has_kernel_h(), p.has_kernel_w(), p.kernel_h(), p.kernel_w(), p.kernel_size_size(), "kernel_size", 0, &s.kh,
       &s.kw, [&](int i) { return p.kernel_size(i); });
  CHECK_GT(s.kh, 0) << "Filter dimensions must be nonzero.";
  CHECK_GT(s.kw, 0) << "Filter dimensions must be nonzero.";
  pick(p.has_stride_h(), p.has_stride_w(), p.stride_h(), p.stride_w(), p.stride_size(), "stride", 1, &s.stride_h,
       &s.stride_w, [&](int i) { return p.stride(i); });
  CHECK_GT(s.stride_h, 0) << "Stride dimensions must be nonzero.";
  CHECK_GT(s.stride_w, 0) << "Stride dimensions must be nonzero.";
  pick(p.has_pad_h(), p.has_pad_w(), p.pad_h(), p.pad_w(), p.pad_size(), "pad", 0, &s.pad_h, &s.pad_w,
       [&](int i) { return p.pad(i); });
  pick(false, false, 0, 0, p.dilation_size(), "dilation", 1, &s.dil_h, &s.dil_w, [&](int i) { return p.dilation(i); });
  CHECK_GT(s.dil_h, 0);
  CHECK_GT(s.dil_w, 0);

}

void ConvolutionLayer::LayerSetUp(const vector<Blob*>& bottom, const vector<Blob*>& top) {
  const ConvolutionParameter& p = layer_param_.convolution_param();
  const int channel_axis = bottom[0]->CanonicalAxisIndex(p.axis());
  const int spatial_axes = bottom[0]->num_axes() - channel_axis - 1;
  CHECK(channel_axis == 1 && spatial_axes == 2)
      << "this engine implements 2-D convolution over (N, C, H, W) blobs; got axis " << channel_axis << " with "
      << spatial_axes << " spatial axes";
  mcb200_conv_shape& s = shape_;
  ParseConvolutionGeometry(p, &s);

  s.c = bottom[0]->shape(1);
  s.cout = static_cast<int>(p.num_output());
  CHECK_GT(s.cout, 0);
  s.group = static_cast<int>(p.group());
  CHECK_GT(s.group, 0);
  CHECK_EQ(s.c % s.group, 0);
  CHECK_EQ(s.cout % s.group, 0) << "Number of output should be multiples of group.";
  bias_term_ = p.bias_term();

  const vector<int> weight_shape = {s.cout, s.c / s.group, s.kh, s.kw};
  const vector<int> bias_shape(bias_term_ ? 1 : 0, s.cout);
  if (!blobs_.empty()) {
    CHECK_EQ(static_cast<size_t>(1 + (bias_term_ ? 1 : 0)), blobs_.size()) << "Incorrect number of weight blobs.";
    if (weight_shape != blobs_[0]->shape()) {
      Blob expected(weight_shape);
      LOG(FATAL) << "Incorrect weight shape: expected shape " << expected.shape_string() << "; instead, shape was "
                 << blobs_[0]->shape_string();
    }
    if (bias_term_ && bias_shape != blobs_[1]->shape()) {
      Blob expected(bias_shape);
      LOG(FATAL) << "Incorrect bias shape: expected shape " << expected.shape_string() << "; instead, shape was "
                 << blobs_[1]->shape_string();
    }
  } else {
    blobs_.resize(bias_term_ ? 2 : 1);
    blobs_[0].reset(new Blob(weight_shape));
    FillBlob(p.weight_filler(), blobs_[0].get());
    if (bias_term_) {
      blobs_[1].reset(new Blob(bias_shape));
      FillBlob(p.bias_filler(), blobs_[1].get());
    }
  }
  // Depthwise layers (one channel per group) are pure data movement and have a kernel of their
  // own; every other layer, grouped or not, is a contraction and runs on the tensor cores (a
  // grouped layer as block-diagonal weight tiles, src/layers/base_conv_layer.cpp:265-270).
  if (s.group > 1 && s.group == s.c && s.cout == s.c && s.c % 4 == 0) {
    path_ = kDepthwise;
  } else {
    path_ = kTensorCore;
  }
  const char* force_direct = getenv("MCB200_CONV_DIRECT");   // "1": the plain kernel, for comparisons in tests
  if (force_direct && force_direct[0] == '1' && path_ == kTensorCore) path_ = kDirect;
  // Limits of the im2col tensor map (8-bit signed corners, 8-bit tap offsets).
  if (path_ == kTensorCore && (s.pad_h > 127 || s.pad_w > 127 || (s.kh - 1) * s.dil_h > 255 ||
                               (s.kw - 1) * s.dil_w > 255)) {
    path_ = kDirect;
  }
}

void ConvolutionLayer::Reshape(const vector<Blob*>& bottom, const vector<Blob*>& top) {
  CHECK_EQ(4, bottom[0]->num_axes()) << "Convolution input must be (N, C, H, W)";
  for (size_t i = 1; i < bottom.size(); ++i) {
    CHECK(bottom[0]->shape() == bottom[i]->shape()) << "All inputs must have the same shape.";
  }
  CHECK_EQ(bottom[0]->shape(1), shape_.c) << "Input size incompatible with convolution kernel.";
  shape_.n = bottom[0]->shape(0);
  shape_.h = bottom[0]->shape(2);
  shape_.w = bottom[0]->shape(3);
  CHECK_EQ(mcb200_conv_out_shape(&shape_), 0) << "convolution window larger than the padded input";
  // Few input channels (an image in front of the first layer): one filter row per k-iteration.
  const bool rows = path_ == kTensorCore && !rows_rejected_ && mcb200_conv_rows_supported(&shape_) != 0;
  if (rows != use_rows_) {
    use_rows_ = rows;
    weight_version_ = 0;   // the packed weight image differs between the two modes
  }
  for (size_t i = 0; i < top.size(); ++i) top[i]->Reshape(shape_.n, shape_.cout, shape_.ho, shape_.wo);
}

// With the pooling in its store the march pays earlier than without: it saves the pooling's launch.  In fp32 from a row a
// slab on (march with pooling and general kernel with pooling kernel, 56 x 56, replayed from a graph: one image 9.5 and 7.7 us,
// five 10.2 and 9.6, six, 348 rows for 296 slabs, 10.3 and 12.8, eight 10.5 and 13.3); with bfloat16 operands always (one
// image 6.8 and 7.6, eight 7.2 and 10.3).
bool ConvolutionLayer::AcceptsFusedPool(const FusedTail& tail, bool half_net) const {
  const char* off = getenv("MCB200_MARCH");
  const double pixels = static_cast<double>(shape_.n) * shape_.h * shape_.w;   // far from the plan's limits
  if (!half_net && mcb200_conv_march_rows_per_slab(&shape_) < 1) return false;
  return path_ == kTensorCore && !use_rows_ && !march_rejected_ && !tail.residual && !(off && off[0] == '0') && pixels < 1e8 &&
         shape_.c % 8 == 0 && mcb200_conv_march_supported(&shape_, 0) != 0;
}

bool ConvolutionLayer::MarchesAlone() const {
  if (tail_.pooled) return true;              // decided when the net was planned
  const char* off = getenv("MCB200_MARCH");   // "0": the general kernel, for comparisons in tests
  return path_ == kTensorCore && !use_rows_ && !march_rejected_ && !tail_.residual && !(off && off[0] == '0') &&
         mcb200_conv_march_pays(&shape_, half_operands_ ? 1 : 0) != 0;
}

bool ConvolutionLayer::AcceptsSibling(const Layer* layer) const {
  const ConvolutionLayer* other = dynamic_cast<const ConvolutionLayer*>(layer);
  if (!other || other == this) return false;
  auto plain = [](const ConvolutionLayer& l) {
    ActivationSpec act;
    if (l.tail_.activation && (!l.tail_.activation->AsActivation(&act) || act.kind != 1 || act.slope != 0.f)) return false;
    // (A pooling in the store is the march's: the launch of two writes the unpooled rows.)
    return l.path_ == kTensorCore && !l.use_rows_ && l.shape_.group == 1 && !l.tail_.residual && !l.tail_.pooled;
  };
  const mcb200_conv_shape &a = shape_, &b = other->shape_;
  // A layer that marches on its own (whatever the plan before this one merged) gives that up in a launch of two, which pays
  // where runs are short: beside a layer that does not march up to four rows a slab, beside one that does up to thirteen.
  // In one launch and alone, fp32 and bfloat16: 64 -> 128 beside 64 -> 64 at 56 x 56, 16 images (three rows) 30.0 and 32.1 us,
  // 29.5 and 31.0, 24 images (four) 42.0 and 41.7, 32.4 and 31.9, 48 images 78 and 72, 56 and 47; 64 -> 64 twice, 64 images
  // (twelve rows) 57.7 and 61.6, 37.0 and 36.8, 72 images (fourteen) 61.8 and 64.8, 51.6 and 44.4, 112 images 108 and 100, 69 and 63.
  const int marching = (MarchesAlone() ? 1 : 0) + (other->MarchesAlone() ? 1 : 0);
  if (marching > 0 && mcb200_conv_march_rows_per_slab(&shape_) >= (marching == 2 ? 13 : 4)) return false;
  // Short sums whose results fill HBM take as long as their stores, which are quickest from tiles of 256 columns.  A layer whose
  // columns divide by 256 keeps its launch there if the two together do not.  In one launch and in two, 1 x 1 at 56 x 56, fp32
  // and bfloat16: 64 -> 256 and 64 at 8 images (8 million cells) 14.3 and 17.5 us, 12.0 and 14.0, at 16 images 25.4 and
  // 23.5, 20.8 and 21.4, at 64 images 80 and 69, 71 and 58; 128 -> 512 and 128 (640 columns still run in tiles of 128)
  // at 32 million cells 45.2 and 48.3, 31.9 and 33.0, at 64 million 77.9 and 75.8, 58.9 and 57.5.  Others gain: 96 -> 384 and 96 at
  // 64 images 90 and 122, 83 and 92; 256 -> 512 and 128 at stride 2, longer sums, 52 and 62, 34 and 37.
  const int both = shape_.cout + other->shape_.cout;
  const double cells = static_cast<double>(shape_.n) * shape_.ho * shape_.wo * both;
  const bool splits_wide = (shape_.cout % 256 == 0 || other->shape_.cout % 256 == 0) && both % 256 != 0;
  if (shape_.c * shape_.kh * shape_.kw < 256 && splits_wide && cells > (both % 128 == 0 ? 60e6 : 16e6)) return false;
  return plain(*this) && plain(*other) && a.n == b.n && a.h == b.h && a.w == b.w && a.c == b.c && a.kh == b.kh && a.kw == b.kw &&
         a.stride_h == b.stride_h && a.stride_w == b.stride_w && a.pad_h == b.pad_h && a.pad_w == b.pad_w && a.dil_h == b.dil_h &&
         a.dil_w == b.dil_w && (half_operands_ && HalfOperandsCapable()) == (other->half_operands_ && other->HalfOperandsCapable()) &&
         (half_top_ && HalfTopCapable()) == (other->half_top_ && other->HalfTopCapable());
}

void ConvolutionLayer::SetSibling(Layer* other) {
  ConvolutionLayer* partner = static_cast<ConvolutionLayer*>(other);
  if (partner == partner_) return;
  partner_ = sibling_ = partner;
  weight_version_ = tail_version_ = 0;   // packed weights and per-column arrays hold both layers
}

// `shape`'s rows of the packed tensor-core weight image.
void ConvolutionLayer::PackRows(const mcb200_conv_shape& shape, const float* weights, float* packed) {
  Context& ctx = Context::Get();
  if (half_operands_) {
    KERNEL_CHECK(mcb200_conv_pack_weights_bf16(&shape, weights, reinterpret_cast<uint16_t*>(packed), ctx.stream_ptr()));
  } else {
    KERNEL_CHECK(mcb200_conv_pack_weights(&shape, weights, packed, ctx.stream_ptr()));
  }
}

void ConvolutionLayer::FoldRows(std::vector<float>* scale, std::vector<float>* shift, bool* has_scale, bool* has_shift) {
  FoldTail(tail_, shape_.cout, bias_term_ ? blobs_[1]->cpu_data() : nullptr, scale, shift, has_scale, has_shift);
}

void ConvolutionLayer::RefreshParameters() {
  Context& ctx = Context::Get();
  if (packed_march_ != Marches()) {
    packed_march_ = !packed_march_;
    weight_version_ = 0;
  }
  // (versions only grow: so does their sum)
  const unsigned long long wv = blobs_[0]->host_version() + (sibling_ ? sibling_->blobs_[0]->host_version() : 0);
  if (wv != weight_version_) {
    if (path_ == kTensorCore && use_rows_) {
      float* packed = packed_weights_.Reserve(mcb200_conv_rows_packed_weight_count(&shape_));
      KERNEL_CHECK(mcb200_conv_rows_pack_weights(&shape_, blobs_[0]->gpu_data(), packed, ctx.stream_ptr()));
    } else if (packed_march_) {
      const int half = half_operands_ ? 1 : 0;
      float* packed = packed_weights_.Reserve(mcb200_conv_march_packed_weight_bytes(&shape_, half) / sizeof(float));
      KERNEL_CHECK(mcb200_conv_march_pack_weights(&shape_, half, blobs_[0]->gpu_data(), packed, ctx.stream_ptr()));
    } else if (path_ == kTensorCore) {
      mcb200_conv_shape all = shape_;
      all.cout = columns();
      const size_t count = half_operands_ ? (mcb200_conv_packed_weight_count_bf16(&all) + 1) / 2
                                          : mcb200_conv_packed_weight_count(&all);
      float* packed = packed_weights_.Reserve(count);
      if (sibling_) {
        // Rows: this layer's, zeros up to the sibling's first column, the sibling's.  (A row is whole 128-byte cells.)
        const size_t row = count / all.cout;
        CUDA_CHECK(cudaMemsetAsync(packed + shape_.cout * row, 0, (second_begin() - shape_.cout) * row * sizeof(float), ctx.stream()));
        PackRows(sibling_->shape_, sibling_->blobs_[0]->gpu_data(), packed + second_begin() * row);
      }
      PackRows(shape_, blobs_[0]->gpu_data(), packed);
    } else if (path_ == kDepthwise) {
      float* packed = packed_weights_.Reserve(static_cast<size_t>(shape_.c) * shape_.kh * shape_.kw);
      KERNEL_CHECK(mcb200_dw_pack_weights(&shape_, blobs_[0]->gpu_data(), packed, ctx.stream_ptr()));
    }
    weight_version_ = wv;
    constants_settled_ = false;
    for (auto& slot : plans_) {
      if (slot) slot->valid = false;
    }
  }
  unsigned long long tv = 1 + TailVersion(tail_) + (bias_term_ ? blobs_[1]->host_version() : 0);
  if (sibling_) tv += TailVersion(sibling_->tail_) + (sibling_->bias_term_ ? sibling_->blobs_[1]->host_version() : 0);
  if (tv != tail_version_) {
    constants_settled_ = false;
    std::vector<float> scale, shift;
    bool has_scale = false, has_shift = false;
    FoldRows(&scale, &shift, &has_scale, &has_shift);
    if (sibling_) {
      std::vector<float> scale2, shift2;
      bool has_scale2 = false, has_shift2 = false;
      sibling_->FoldRows(&scale2, &shift2, &has_scale2, &has_shift2);
      scale.resize(second_begin(), 1.f);
      shift.resize(second_begin(), 0.f);
      scale.insert(scale.end(), scale2.begin(), scale2.end());
      shift.insert(shift.end(), shift2.begin(), shift2.end());
      has_scale = has_scale || has_scale2;
      has_shift = has_shift || has_shift2;
    }
    if (has_scale) scale_.Assign(scale); else scale_.Clear();
    if (has_shift) shift_.Assign(shift); else shift_.Clear();
    tail_version_ = tv;
  }
}

double ConvolutionLayer::PartSeconds(const vector<Blob*>& bottom, const vector<Blob*>& top, bool first_of_net) const {
  const mcb200_conv_shape& s = shape_;
  if (bottom.size() != 1 || path_ == kDirect || s.cout % 8 != 0) return 0;
  // Of the net's input only a layer that reads (N, C, H, W) rows itself may take a part.
  if (first_of_net ? !use_rows_ || s.c % 4 == 0 : s.c % 8 != 0) return 0;
  const double in_cell = half_operands_ && HalfOperandsCapable() ? 2.0 : 4.0;
  const double out_cell = half_top_ && HalfTopCapable() ? 2.0 : 4.0;
  double bytes = in_cell * bottom[0]->count() + out_cell * top[0]->count();
  if (tail_.residual) bytes += in_cell * top[0]->count();
  double outputs = static_cast<double>(s.n) * s.cout * s.ho * s.wo;
  if (partner_) {
    if (partner_->shape_.cout % 8 != 0) return 0;
    outputs += top[1]->count();
    bytes += out_cell * top[1]->count();
  }
  const double flops = 2.0 * outputs * (s.c / s.group) * s.kh * s.kw;
  const double rate = path_ == kDepthwise ? 20e12 : in_cell == 2.0 ? 1.1e15 : 0.6e15;
  return std::max(bytes / kPartBytesPerSecond, flops / rate);
}

void ConvolutionLayer::Forward_gpu(const vector<Blob*>& bottom, const vector<Blob*>& top) {
  if (partner_) {
    RunTwo(bottom[0], top, 0, shape_.n, 0);
    return;
  }
  RefreshParameters();
  for (size_t i = 0; i < bottom.size(); ++i) RunImages(bottom[i], top[i], i, 0, shape_.n, i);
  constants_settled_ = true;
}

void ConvolutionLayer::ForwardImages_gpu(const vector<Blob*>& bottom, const vector<Blob*>& top, int first, int count,
                                         int part) {
  if (partner_) {
    RunTwo(bottom[0], top, first, count, part);
    return;
  }
  if (first == 0) RefreshParameters();
  RunImages(bottom[0], top[0], 0, first, count, part);
  if (first + count == shape_.n) constants_settled_ = true;
}

// This layer and the net's partner: in one launch, or, once the plan of two has been refused, one behind the other.
void ConvolutionLayer::RunTwo(Blob* bottom, const vector<Blob*>& top, int first, int count, size_t slot) {
  RefreshParameters();
  RunImages(bottom, top[0], 0, first, count, slot, top[1]);
  const bool through = first + count == shape_.n;
  if (through) constants_settled_ = true;
  if (sibling_) return;
  partner_->RefreshParameters();
  partner_->RunImages(bottom, top[1], 0, first, count, slot);
  if (through) partner_->constants_settled_ = true;
}

void ConvolutionLayer::RunImages(Blob* bottom, Blob* top, size_t i, int first, int count, size_t slot_index, Blob* second_top) {
  Context& ctx = Context::Get();
  const bool half_out = half_top_ && HalfTopCapable();
  const bool half = half_operands_ && HalfOperandsCapable();
  if (count == 0 && path_ == kTensorCore) {   // a batch of no images: the tops are there and hold nothing
    CHECK(!half && !half_out) << "cannot build the tensor-core plan for layer " << layer_param_.name() << " (no images)";
    top->mutable_gpu_data_nhwc();
    if (second_top) second_top->mutable_gpu_data_nhwc();
    return;
  }
  mcb200_conv_shape s = shape_;
  s.n = count;
  s.cout = columns();
  const size_t in_at = static_cast<size_t>(first) * s.c * s.h * s.w;
  const size_t out_at = first == 0 ? 0 : static_cast<size_t>(first) * (top->count() / shape_.n);
  const float* in = nullptr;
  if (half) {
    s.c_stride = s.c;
    in = reinterpret_cast<const float*>(static_cast<const uint16_t*>(bottom->gpu_data_nhwc_bf16()) + in_at);
  } else if (path_ == kTensorCore && use_rows_) {
    int hp = 0, wp = 0;
    CHECK_EQ(mcb200_conv_rows_padded_dims(&s, &hp, &wp), 0);
    s.c_stride = 4;
    const size_t image = static_cast<size_t>(hp) * wp * 4;
    float* padded = padded_input_.Reserve(shape_.n * image) + first * image;
    KERNEL_CHECK(mcb200_conv_rows_pad_input(&s, bottom->gpu_data() + in_at, padded, ctx.stream_ptr()));
    in = padded;
  } else if (shape_.c % 4 == 0) {
    s.c_stride = s.c;
    in = bottom->gpu_data_nhwc() + in_at;
  } else {
    // Pad the channels to a multiple of four (16-byte pixels) in a private
    // channels-last copy, e.g. the three colour planes of the first layer.
    s.c_stride = (s.c + 3) / 4 * 4;
    const size_t image = static_cast<size_t>(s.h) * s.w * s.c_stride;
    float* padded = padded_input_.Reserve(shape_.n * image) + first * image;
    if (bottom->device_is_nhwc()) {
      // The pad lanes meet zero weights but still have to be finite.
      CUDA_CHECK(cudaMemsetAsync(padded, 0, static_cast<size_t>(s.n) * s.h * s.w * s.c_stride * sizeof(float),
                                 ctx.stream()));
      KERNEL_CHECK(mcb200_copy_2d(bottom->gpu_data_nhwc() + in_at, s.c, padded, s.c_stride,
                                  static_cast<long long>(s.n) * s.h * s.w, s.c, ctx.stream_ptr()));
    } else {
      KERNEL_CHECK(mcb200_nchw_to_nhwc(bottom->gpu_data() + in_at, padded, s.n, s.c, s.h, s.w, s.c_stride,
                                       ctx.stream_ptr()));
    }
    in = padded;
  }
  mcb200_epilogue ep;
  FillTailEpilogue(i == 0 ? tail_ : FusedTail(), scale_, shift_, half ? kResidualNhwcHalf : kResidualNhwc,
                   shape_.cout, &ep);
  if (ep.residual) {
    ep.residual = half ? reinterpret_cast<const float*>(reinterpret_cast<const uint16_t*>(ep.residual) + out_at)
                       : ep.residual + out_at;
  }
  float* out = half_out ? reinterpret_cast<float*>(static_cast<uint16_t*>(top->mutable_gpu_data_nhwc_bf16()) + out_at)
                        : top->mutable_gpu_data_nhwc() + out_at;
  if (path_ == kTensorCore) {
    if (plans_.size() <= slot_index) plans_.resize(slot_index + 1);
    if (!plans_[slot_index]) plans_[slot_index].reset(new PlanSlot);
    PlanSlot& slot = *plans_[slot_index];
    const float* w = packed_weights_.Reserve(0);
    if (!slot.valid || slot.in != in || slot.weights != w || slot.pooled != tail_.pooled ||
        std::memcmp(&slot.shape, &s, sizeof(s)) != 0) {
      slot.valid = false;   // (a plan that is refused leaves nothing behind)
      int rc = packed_march_ ? mcb200_conv_march_plan(&s, half ? 1 : 0, in, w, tail_.pooled ? 1 : 0, &slot.march)
               : half ? mcb200_conv_tc_plan_bf16(&s, reinterpret_cast<const uint16_t*>(in),
                                               reinterpret_cast<const uint16_t*>(w), &slot.plan)
               : use_rows_ ? mcb200_conv_rows_plan(&s, in, w, &slot.plan)
                           : mcb200_conv_tc_plan(&s, in, w, &slot.plan);
      if (rc != 0 && use_rows_) {
        // The driver refused the row-mode tensor map: use the general path from now on.
        LOG(WARNING) << "layer " << layer_param_.name() << ": row-mode plan rejected (" << rc
                     << "), using the im2col path";
        rows_rejected_ = true;
        use_rows_ = false;
        weight_version_ = 0;
        RefreshParameters();
        RunImages(bottom, top, i, first, count, slot_index);
        return;
      }
      if (rc != 0 && packed_march_ && !tail_.pooled) {
        march_rejected_ = true;   // the general kernel from now on
        RefreshParameters();
        RunImages(bottom, top, i, first, count, slot_index);
        return;
      }
      CHECK(rc == 0 || !tail_.pooled) << "cannot build the plan for layer " << layer_param_.name();
      if (rc != 0 && sibling_) {
        // A geometry the tensor maps cannot express for both (and mostly for neither): two layers of their own from now on.
        sibling_ = nullptr;
        weight_version_ = tail_version_ = 0;
        RefreshParameters();
        RunImages(bottom, top, i, first, count, slot_index);
        return;
      }
      if (rc != 0 && !half && !half_out) {
        // A shape the tensor maps cannot express (for instance a stride above 8, which the
        // im2col map refuses as traversal stride): the plain kernel runs it from now on.
        LOG(WARNING) << "layer " << layer_param_.name() << ": tensor-core plan rejected (" << rc
                     << "), using the direct kernel";
        path_ = kDirect;
        RunImages(bottom, top, i, first, count, slot_index);
        return;
      }
      CHECK_EQ(rc, 0) << "cannot build the tensor-core plan for layer " << layer_param_.name();
      slot.in = in;
      slot.weights = w;
      slot.shape = s;
      slot.pooled = tail_.pooled;
      slot.valid = true;
    }
    const int flags = constants_settled_ ? MCB200_CONV_CONSTANTS_SETTLED : 0;
    if (packed_march_) {
      KERNEL_CHECK(mcb200_conv_march_launch(&slot.march, out, half_out ? 1 : 0, s.cout, &ep, flags, ctx.status_word(), ctx.stream_ptr()));
    } else if (sibling_) {
      CHECK_EQ(second_top->count(), shape_.n * sibling_->shape_.cout * s.ho * s.wo) << "top of layer " << sibling_->layer_param_.name();
      mcb200_conv_second second;
      second.begin = second_begin();
      second.first_cout = shape_.cout;
      second.out_ld = sibling_->shape_.cout;
      second.act = sibling_->tail_.activation ? 1 : 0;
      const size_t second_at = static_cast<size_t>(first) * second.out_ld * s.ho * s.wo;
      second.out = half_out ? static_cast<void*>(static_cast<uint16_t*>(second_top->mutable_gpu_data_nhwc_bf16()) + second_at)
                            : static_cast<void*>(second_top->mutable_gpu_data_nhwc() + second_at);
      KERNEL_CHECK(mcb200_conv_tc_launch_two(&slot.plan, out, half_out ? 1 : 0, shape_.cout, &ep, &second, flags, ctx.status_word(),
                                             ctx.stream_ptr()));
    } else {
      KERNEL_CHECK(mcb200_conv_tc_launch_flags(&slot.plan, out, half_out ? 1 : 0, s.cout, &ep, flags, ctx.status_word(),
                                               ctx.stream_ptr()));
    }
  } else if (path_ == kDepthwise && (half || half_out)) {
    KERNEL_CHECK(mcb200_conv_depthwise_bf16(&s, in, half ? 1 : 0, packed_weights_.Reserve(0), out, half_out ? 1 : 0,
                                            &ep, ctx.stream_ptr()));
  } else if (path_ == kDepthwise) {
    const char* dw_tma = getenv("MCB200_DW_TMA");   // "0": the register-window kernel, for comparisons
    // Outputs of 8 x 8 pixels and more: the TMA-staged kernel's 8 x 16 tiles; on smaller maps
    // (the 7 x 7 end of MobileNet) most of a tile is outside the image and the register-window
    // kernel is quicker (11 / 14 us against 15 / 18 us at batch 64).  The rule looks at the
    // layer's geometry only, never at the batch.
    const bool roomy = s.ho >= 8 && s.wo >= 8;
    if (!ep.residual && roomy && mcb200_conv_depthwise_tma_supported(&s) && !(dw_tma && dw_tma[0] == '0')) {
      KERNEL_CHECK(mcb200_conv_depthwise_tma(&s, in, packed_weights_.Reserve(0), out, &ep, ctx.status_word(),
                                             ctx.stream_ptr()));
    } else {
      KERNEL_CHECK(mcb200_conv_depthwise(&s, in, packed_weights_.Reserve(0), out, &ep, ctx.stream_ptr()));
    }
  } else {
    KERNEL_CHECK(mcb200_conv_direct(&s, in, blobs_[0]->gpu_data(), out, s.cout, &ep, ctx.stream_ptr()));
  }
}

static shared_ptr<Layer> CreateConvolution(const LayerParameter& param) {
  return shared_ptr<Layer>(new ConvolutionLayer(param));
}
REGISTER_LAYER_CREATOR(Convolution, CreateConvolution);
// The reference registers its depthwise kernel under its own type name as
// well (src/layers/conv_dw_layer.cpp:158); here the one class picks the path.
REGISTER_LAYER_CREATOR(ConvolutionDepthwise, CreateConvolution);

// ---------------------------------------------------------------- InnerProduct

void InnerProductLayer::LayerSetUp(const vector<Blob*>& bottom, const vector<Blob*>& top) {
  const InnerProductParameter& p = layer_param_.inner_product_param();
  N_ = static_cast<int>(p.num_output());
  bias_term_ = p.bias_term();
  transpose_ = p.transpose();
  const int axis = bottom[0]->CanonicalAxisIndex(p.axis());
  K_ = bottom[0]->count(axis);
  if (blobs_.empty()) {
    blobs_.resize(bias_term_ ? 2 : 1);
    blobs_[0].reset(new Blob(transpose_ ? vector<int>{K_, N_} : vector<int>{N_, K_}));
    FillBlob(p.weight_filler(), blobs_[0].get());
    if (bias_term_) {
      blobs_[1].reset(new Blob(vector<int>(1, N_)));
      FillBlob(p.bias_filler(), blobs_[1].get());
    }
  }
}

void InnerProductLayer::Reshape(const vector<Blob*>& bottom, const vector<Blob*>& top) {
  const int axis = bottom[0]->CanonicalAxisIndex(layer_param_.inner_product_param().axis());
  CHECK_EQ(K_, bottom[0]->count(axis)) << "Input size incompatible with inner product parameters.";
  M_ = bottom[0]->count(0, axis);
  vector<int> top_shape = bottom[0]->shape();
  top_shape.resize(axis + 1);
  top_shape[axis] = N_;
  top[0]->Reshape(top_shape);
}

void InnerProductLayer::Forward_gpu(const vector<Blob*>& bottom, const vector<Blob*>& top) {
  Context& ctx = Context::Get();
  mcb200_conv_shape s = mcb200_conv_shape();
  s.n = M_;
  s.h = s.w = 1;
  s.c = s.c_stride = K_;
  s.cout = N_;
  s.kh = s.kw = s.stride_h = s.stride_w = s.dil_h = s.dil_w = s.group = 1;
  s.ho = s.wo = 1;
  const bool tensor_core = (K_ % 4 == 0);

  // Weights as [N, K] rows (transpose: stored [K, N], re-laid on the host).
  const unsigned long long wv = blobs_[0]->host_version();
  const float* w_rows = nullptr;
  if (transpose_) {
    if (wv != weight_version_) {
      std::vector<float> rows(static_cast<size_t>(N_) * K_);
      const float* src = blobs_[0]->cpu_data();
      for (int k = 0; k < K_; ++k)
        for (int n = 0; n < N_; ++n) rows[static_cast<size_t>(n) * K_ + k] = src[static_cast<size_t>(k) * N_ + n];
      float* staged = staged_weights_.Reserve(rows.size());
      CUDA_CHECK(cudaMemcpyAsync(staged, rows.data(), rows.size() * sizeof(float), cudaMemcpyHostToDevice,
                                 ctx.stream()));
      ctx.Sync();  // `rows` is pageable and dies with this scope
    }
    w_rows = staged_weights_.Reserve(0);
  } else {
    w_rows = blobs_[0]->gpu_data();
  }
  if (wv != weight_version_) {
    if (tensor_core) {
      float* packed = packed_weights_.Reserve(mcb200_conv_packed_weight_count(&s));
      KERNEL_CHECK(mcb200_conv_pack_weights(&s, w_rows, packed, ctx.stream_ptr()));
    }
    weight_version_ = wv;
    plan_in_ = nullptr;
    constants_settled_ = false;
  }
  const unsigned long long tv = 1 + TailVersion(tail_) + (bias_term_ ? blobs_[1]->host_version() : 0);
  if (tv != tail_version_) {
    constants_settled_ = false;
    std::vector<float> scale, shift;
    bool has_scale = false, has_shift = false;
    FoldTail(tail_, N_, bias_term_ ? blobs_[1]->cpu_data() : nullptr, &scale, &shift, &has_scale, &has_shift);
    if (has_scale) scale_.Assign(scale); else scale_.Clear();
    if (has_shift) shift_.Assign(shift); else shift_.Clear();
    tail_version_ = tv;
  }
  // Rows of the (N, C, H, W)-ordered input are the K-vectors.
  const float* in = bottom[0]->gpu_data();
  mcb200_epilogue ep;
  FillTailEpilogue(tail_, scale_, shift_, kResidualNchw, N_, &ep);
  float* out = top[0]->mutable_gpu_data();
  if (tensor_core) {
    if (!plan_) {
      plan_storage_.reset(new char[sizeof(mcb200_conv_plan) + 64]);
      uintptr_t a = (reinterpret_cast<uintptr_t>(plan_storage_.get()) + 63) & ~static_cast<uintptr_t>(63);
      plan_ = reinterpret_cast<mcb200_conv_plan*>(a);
    }
    const float* w = packed_weights_.Reserve(0);
    if (plan_in_ != in || plan_w_ != w || plan_m_ != M_) {
      CHECK_EQ(mcb200_conv_tc_plan(&s, in, w, plan_), 0) << "cannot build the tensor-core plan for layer "
                                                         << layer_param_.name();
      plan_in_ = in;
      plan_w_ = w;
      plan_m_ = M_;
    }
    KERNEL_CHECK(mcb200_conv_tc_launch_flags(plan_, out, 0, N_, &ep, constants_settled_ ? MCB200_CONV_CONSTANTS_SETTLED : 0,
                                             ctx.status_word(), ctx.stream_ptr()));
    constants_settled_ = true;
  } else {
    KERNEL_CHECK(mcb200_conv_direct(&s, in, w_rows, out, N_, &ep, ctx.stream_ptr()));
  }
}

REGISTER_LAYER_CLASS(InnerProduct);

}  // namespace caffe
