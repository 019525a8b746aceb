// Operation classes of the CNN forward hot path on top of the C ABI.  Each class keeps the
// reference's parameter keys, weight-file reading order and tensor semantics (fp32 NCHW tensors
// between ops for operation<float>; int8 only inside the convolution), and runs its arithmetic
// through libexcalibur_b200's kernels on the legacy default stream, like the reference's GPU path.
#include "ops.hpp"

#include <cmath>
#include <limits>
#include <random>

namespace glasssix {
namespace excalibur {

void exb_check(int rc, const char* what) {
    if (rc != EXB_OK) LOG(FATAL) << what << " failed (" << rc << "): " << exb_last_error_string();
}

device_scratch::~device_scratch() {
    if (ptr_) cudaFree(ptr_);
}
void* device_scratch::get(size_t bytes, int device) {
    if (bytes > cap_) {
        if (ptr_) cudaFree(ptr_);
        ptr_ = nullptr;
        CUDA_CHECK(cudaSetDevice(device));
        CUDA_CHECK(cudaMalloc(&ptr_, bytes));
        cap_ = bytes;
    }
    return ptr_;
}

namespace {
int round_up(int a, int b) { return (a + b - 1) / b * b; }

template <typename T>
std::shared_ptr<memory::tensor<T>> make_tensor(const std::vector<int>& shape, int device, memory::orderType order,
                                               memory::pool_allocator<T>* alloc = nullptr) {
    return std::shared_ptr<memory::tensor<T>>(new memory::tensor<T>(shape, device, order, alloc));
}

void read_or_die(void* dst, size_t bytes, FILE* fp, const char* what) {
    if (bytes && fread(dst, 1, bytes, fp) != bytes) LOG(FATAL) << "weight file ended while reading " << what;
}
}  // namespace

// ---------------------------------------------------------------------------------------------
// general conv: parameter parsing
// ---------------------------------------------------------------------------------------------
template <typename Dtype>
operation_general_conv<Dtype>::operation_general_conv(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        const int v = std::atoi(kv.second.c_str());
        switch (kv.first) {
        case 0: output_channel_ = v; break;
        case 1: kernel_size_w_ = kernel_size_h_ = v; break;
        case 2: dilation_w_ = dilation_h_ = v; break;
        case 3: stride_w_ = stride_h_ = v; break;
        case 4: pad_left_ = pad_right_ = pad_top_ = pad_bottom_ = v; break;
        case 5: bias_term_ = v != 0; break;
        case 6: weight_data_size_ = v; break;
        case 7: group_ = v; break;
        case 8:
            int8_scale_term_ = v != 0;
            this->params_.set_int8_quantization(int8_scale_term_);
            break;
        case 9: activation_type_ = v; break;
        case 10: NOT_IMPLEMENTED; break;
        case 11: kernel_size_h_ = v; break;
        case 12: dilation_h_ = v; break;
        case 13: stride_h_ = v; break;
        case 14: pad_top_ = v; break;
        case 15: pad_right_ = v; break;
        case 16: pad_bottom_ = v; break;
        case 17: impl_type_ = v; break;
        case 18: case 19: case 20: case 21: break;  // output padding / dims: deconvolution only
        case -23330: break;
        default: LOG(FATAL) << "Un-supported Convolution Attribution " << kv.first;
        }
    }
    CHECK_GT(output_channel_, 0);
    CHECK_GT(group_, 0);
    CHECK_EQ(output_channel_ % group_, 0);
    CHECK(kernel_size_h_ > 0 && kernel_size_w_ > 0) << "convolution kernel size missing";
    const int per_group = (output_channel_ / group_) * kernel_size_h_ * kernel_size_w_;
    if (weight_data_size_ > 0) {
        CHECK_EQ(weight_data_size_ % (per_group * group_), 0) << "weight_data_size does not match the kernel shape";
        input_channel_ = weight_data_size_ / (per_group * group_) * group_;
    }
}
INSTANCE_CLASS(operation_general_conv);

// ---------------------------------------------------------------------------------------------
// dense convolution
// ---------------------------------------------------------------------------------------------
template <typename Dtype>
operation_convolution<Dtype>::operation_convolution(const operation_param& param)
    : operation_general_conv<Dtype>(param) {}

template <typename Dtype>
operation_convolution<Dtype>::~operation_convolution() {
    for (auto& e : packed_) exb_conv_weights_destroy(e.w);
}

// .racy record: int32 tag; tag 0: fp32 OIHW weights (+ bias); tag 871224: int8 weights padded to
// a multiple of 4 bytes (+ fp32 bias), per-output-channel weight scales, one activation scale.
template <typename Dtype>
int operation_convolution<Dtype>::init_weights(FILE* fp) {
    int tag = 0;
    read_or_die(&tag, sizeof(int), fp, "the quantize tag");
    const int dev = this->params_.device_;
    int mem = 0;
    if (tag == 0) {
        this->weights_f32_.push_back(make_tensor<float>({this->weight_data_size_}, dev, memory::NCHW));
        read_or_die(this->weights_f32_[0]->mutable_cpu_data(), sizeof(float) * this->weight_data_size_, fp, "weights");
        mem += this->weight_data_size_ * sizeof(float);
        if (this->bias_term_) {
            this->weights_f32_.push_back(make_tensor<float>({this->output_channel_}, dev, memory::NCHW));
            read_or_die(this->weights_f32_[1]->mutable_cpu_data(), sizeof(float) * this->output_channel_, fp, "bias");
            mem += this->output_channel_ * sizeof(float);
        }
    } else if (tag == 871224) {
        const size_t aligned = ((size_t)this->weight_data_size_ + 3) & ~(size_t)3;
        this->weights_i8_.push_back(make_tensor<signed char>({(int)aligned}, dev, memory::NCHW));
        read_or_die(this->weights_i8_[0]->mutable_cpu_data(), aligned, fp, "int8 weights");
        mem += (int)aligned;
        if (this->bias_term_) {
            this->weights_f32_.push_back(make_tensor<float>({1}, dev, memory::NCHW));   // slot 0 unused, as in the reference
            this->weights_f32_.push_back(make_tensor<float>({this->output_channel_}, dev, memory::NCHW));
            read_or_die(this->weights_f32_[1]->mutable_cpu_data(), sizeof(float) * this->output_channel_, fp, "bias");
            mem += this->output_channel_ * sizeof(float);
        }
        this->weights_scaletable_i8_ = make_tensor<float>({this->output_channel_}, dev, memory::NCHW);
        read_or_die(this->weights_scaletable_i8_->mutable_cpu_data(), sizeof(float) * this->output_channel_, fp, "weight scales");
        this->featmap_scaletable_i8_ = make_tensor<float>({1}, dev, memory::NCHW);
        read_or_die(this->featmap_scaletable_i8_->mutable_cpu_data(), sizeof(float), fp, "activation scale");
        mem += (this->output_channel_ + 1) * sizeof(float);
        this->params_.set_int8_quantization(true);
    } else {
        NOT_IMPLEMENTED << " (weight record tag " << tag << ")";
    }
    return mem;
}

// Seeded dummy weights: N(0, 0.3) fp32, U[-128,127] int8, from a default-seeded engine.
template <typename Dtype>
int operation_convolution<Dtype>::init_weights() {
    std::default_random_engine e;
    std::normal_distribution<float> n(0, 0.3);
    std::uniform_int_distribution<int> u(-128, 127);
    const int dev = this->params_.device_;
    int mem = 0;
    if (!this->params_.int8_quantization_) {
        this->weights_f32_.push_back(make_tensor<float>({this->weight_data_size_}, dev, memory::NCHW));
        float* w = this->weights_f32_[0]->mutable_cpu_data();
        for (int i = 0; i < this->weight_data_size_; ++i) w[i] = n(e);
        mem += this->weight_data_size_ * sizeof(float);
        if (this->bias_term_) {
            this->weights_f32_.push_back(make_tensor<float>({this->output_channel_}, dev, memory::NCHW));
            float* b = this->weights_f32_[1]->mutable_cpu_data();
            for (int i = 0; i < this->output_channel_; ++i) b[i] = n(e);
            mem += this->output_channel_ * sizeof(float);
        }
    } else {
        const size_t aligned = ((size_t)this->weight_data_size_ + 3) & ~(size_t)3;
        this->weights_i8_.push_back(make_tensor<signed char>({(int)aligned}, dev, memory::NCHW));
        signed char* w = this->weights_i8_[0]->mutable_cpu_data();
        for (size_t i = 0; i < aligned; ++i) w[i] = (signed char)u(e);
        mem += (int)aligned;
        if (this->bias_term_) {
            this->weights_f32_.push_back(make_tensor<float>({1}, dev, memory::NCHW));
            this->weights_f32_.push_back(make_tensor<float>({this->output_channel_}, dev, memory::NCHW));
            float* b = this->weights_f32_[1]->mutable_cpu_data();
            for (int i = 0; i < this->output_channel_; ++i) b[i] = n(e);
            mem += this->output_channel_ * sizeof(float);
        }
        this->weights_scaletable_i8_ = make_tensor<float>({this->output_channel_}, dev, memory::NCHW);
        float* s = this->weights_scaletable_i8_->mutable_cpu_data();
        for (int i = 0; i < this->output_channel_; ++i) s[i] = n(e);
        this->featmap_scaletable_i8_ = make_tensor<float>({1}, dev, memory::NCHW);
        this->featmap_scaletable_i8_->mutable_cpu_data()[0] = n(e);
        mem += (this->output_channel_ + 1) * sizeof(float);
    }
    return mem;
}

template <typename Dtype>
float operation_convolution<Dtype>::act_scale() const {
    CHECK(this->featmap_scaletable_i8_ != nullptr) << "convolution has no activation scale";
    if (this->featmap_scaletable_i8_->count() != 1)
        NOT_IMPLEMENTED << " (per-channel activation scales)";
    return this->featmap_scaletable_i8_->cpu_data()[0];
}

template <typename Dtype>
int operation_convolution<Dtype>::exb_activation() const {
    switch (this->activation_type_) {
    case 0: return EXB_ACT_NONE;
    case 1: return EXB_ACT_RELU;
    case 3: return EXB_ACT_RELU6_QUIRK;
    case 4: return EXB_ACT_SIGMOID;
    case 5: return EXB_ACT_MISH;
    default: NOT_IMPLEMENTED << " (convolution activation type " << this->activation_type_ << ")";
    }
    return EXB_ACT_NONE;
}

template <typename Dtype>
exb_conv_desc operation_convolution<Dtype>::base_desc(int N, int H, int W) const {
    exb_conv_desc d;
    std::memset(&d, 0, sizeof(d));
    d.N = N; d.H = H; d.W = W;
    d.Cin = this->input_channel_; d.Cout = this->output_channel_;
    d.kh = this->kernel_size_h_; d.kw = this->kernel_size_w_;
    d.stride_h = this->stride_h_; d.stride_w = this->stride_w_;
    d.pad_t = this->pad_top_; d.pad_b = this->pad_bottom_; d.pad_l = this->pad_left_; d.pad_r = this->pad_right_;
    d.dilation = 1;   // the reference's forward ignores keys 2/12 as well
    d.group = this->group_;
    d.in_dtype = is_int8() ? EXB_I8 : EXB_F16;
    d.out_dtype = EXB_F16; d.out2_dtype = -1; d.res_dtype = -1;
    d.act = EXB_ACT_NONE; d.out_scale = 1.f; d.out2_scale = 1.f; d.impl = 0;
    return d;
}

template <typename Dtype>
exb_conv_weights* operation_convolution<Dtype>::packed(exb_ctx* ctx, const exb_conv_desc& d, const float* post_mul,
                                                       const float* post_add, const void* tag) {
    const int cin_stride = d.cin_stride ? d.cin_stride : d.Cin;
    const int cout_stride = d.cout_stride ? d.cout_stride : d.Cout;
    for (auto& e : packed_)
        if (e.in_dtype == d.in_dtype && e.cin_stride == cin_stride && e.cout_stride == cout_stride &&
            e.w_pitch == d.x_w_pitch && e.w_pad == d.x_w_pad && e.tag == tag)
            return e.w;
    exb_conv_weights* w = nullptr;
    const int Cout = this->output_channel_;
    const float* bias = this->bias_term_ ? this->weights_f32_[1]->cpu_data() : nullptr;
    std::vector<float> fbias, fw, fscale;
    if (post_mul) {     // (conv + bias) * mul + add
        fbias.resize(Cout);
        for (int c = 0; c < Cout; ++c) fbias[c] = (bias ? bias[c] : 0.f) * post_mul[c] + (post_add ? post_add[c] : 0.f);
        bias = fbias.data();
    }
    if (d.in_dtype == EXB_I8) {
        CHECK(is_int8()) << "int8 convolution requested but the weights are fp32";
        const float* ws = this->weights_scaletable_i8_->cpu_data();
        int n_ws = this->weights_scaletable_i8_->count();
        if (post_mul) {
            // the dequantise multiplier is 1 / (ws * fs): dividing ws by mul multiplies the result by mul
            fscale.resize(Cout);
            for (int c = 0; c < Cout; ++c) {
                const float w0 = ws[n_ws == 1 ? 0 : c];
                fscale[c] = post_mul[c] != 0.f ? w0 / post_mul[c] : std::numeric_limits<float>::infinity();
            }
            ws = fscale.data();
            n_ws = Cout;
        }
        exb_check(exb_conv_weights_pack_i8(ctx, &d, this->weights_i8_[0]->cpu_data(), bias, ws, n_ws, act_scale(), &w),
                  "exb_conv_weights_pack_i8");
    } else {
        CHECK(!is_int8()) << "fp16 convolution requested but the weights are int8";
        const float* wsrc = this->weights_f32_[0]->cpu_data();
        if (post_mul) {
            const size_t per = (size_t)this->weights_f32_[0]->count() / Cout;
            fw.resize((size_t)Cout * per);
            for (int c = 0; c < Cout; ++c)
                for (size_t k = 0; k < per; ++k) fw[c * per + k] = wsrc[c * per + k] * post_mul[c];
            wsrc = fw.data();
        }
        exb_check(exb_conv_weights_pack_f16(ctx, &d, wsrc, bias, &w), "exb_conv_weights_pack_f16");
    }
    packed_.push_back({d.in_dtype, cin_stride, cout_stride, d.x_w_pitch, d.x_w_pad, w, tag});
    return w;
}

// Stand-alone op semantics of the reference: fp32 NCHW tensor in, fp32 NCHW tensor out.  int8:
// quantise the input with the conv's activation scale (half away from zero), int8 x int8 -> int32
// on the tensor cores, y = acc * 1/(ws*fs) + bias, activation - the reference's forward_cpu_i8
// (src/Excalibur/operation_convolution.cpp:332-409).  fp32: fp16 operands, fp32 accumulation.
template <typename Dtype>
void operation_convolution<Dtype>::forward_nchw_f32(exb_ctx* h, const f32_list& bottoms, f32_list& tops, bool int8) {
    CHECK_EQ(bottoms.size(), (size_t)1);
    CHECK_EQ(tops.size(), (size_t)1);
    CHECK(h != nullptr) << "null context";
    if (bottoms[0]->order() == memory::NHWC) bottoms[0]->convert_order();
    const int N = bottoms[0]->num(), C = bottoms[0]->channels(), H = bottoms[0]->height(), W = bottoms[0]->width();
    CHECK_EQ(C, this->input_channel_) << "input channels do not match the weights";
    const int dev = this->params_.device_;
    exb_conv_desc d = base_desc(N, H, W);
    d.in_dtype = int8 ? EXB_I8 : EXB_F16;
    d.cin_stride = this->group_ == 1 ? round_up(C, int8 ? 32 : 16) : C;
    d.out_dtype = EXB_F32;
    // Activation scales are taken from this path: one kernel, and so one order of the fp32 sums, whatever the batch - int8
    // scales then do not depend on how many calibration images a forward holds.
    if (!int8) d.impl = 2;
    d.act = exb_activation();
    int OH = 0, OW = 0;
    exb_check(exb_conv_out_dims(&d, &OH, &OW), "exb_conv_out_dims");
    tops[0] = make_tensor<float>({N, this->output_channel_, OH, OW}, dev, memory::NCHW, bottoms[0]->allocator());
    if (N == 0) return;
    const size_t es = int8 ? 1 : 2;
    void* xin = scratch_in_.get((size_t)N * H * W * d.cin_stride * es, dev);
    void* yout = scratch_out_.get((size_t)N * OH * OW * this->output_channel_ * sizeof(float), dev);
    exb_check(exb_nchw_f32_to_nhwc(h, bottoms[0]->gpu_data(), xin, d.in_dtype, N, C, H, W, d.cin_stride,
                                   int8 ? act_scale() : 1.f, 0, nullptr),
              "exb_nchw_f32_to_nhwc");
    exb_check(exb_conv2d_fwd(h, &d, xin, packed(h, d), nullptr, yout, nullptr, nullptr), "exb_conv2d_fwd");
    exb_check(exb_nhwc_to_nchw_f32(h, yout, EXB_F32, tops[0]->mutable_gpu_data(), N, this->output_channel_, OH, OW,
                                   this->output_channel_, 1.f, nullptr),
              "exb_nhwc_to_nchw_f32");
}

template <typename Dtype>
void operation_convolution<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    forward_nchw_f32(h, bottoms, tops, false);
}
template <typename Dtype>
void operation_convolution<Dtype>::forward_gpu_i8(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    forward_nchw_f32(h, bottoms, tops, true);
}

// fp16 tensors: NHWC, channels already padded by the caller to a multiple of 16 when the tensor
// cores are wanted; no layout conversion at all.
template <typename Dtype>
void operation_convolution<Dtype>::forward_gpu_f16(exb_ctx*& h, const f16_list& bottoms, f16_list& tops) {
    CHECK_EQ(bottoms.size(), (size_t)1);
    CHECK_EQ(tops.size(), (size_t)1);
    if (bottoms[0]->order() != memory::NHWC) NOT_IMPLEMENTED << " (fp16 tensors must be NHWC)";
    const int N = bottoms[0]->num(), C = bottoms[0]->channels(), H = bottoms[0]->height(), W = bottoms[0]->width();
    CHECK_EQ(C, this->input_channel_);
    exb_conv_desc d = base_desc(N, H, W);
    d.in_dtype = EXB_F16;
    d.out_dtype = EXB_F16;
    d.act = exb_activation();
    int OH = 0, OW = 0;
    exb_check(exb_conv_out_dims(&d, &OH, &OW), "exb_conv_out_dims");
    tops[0] = make_tensor<unsigned short>({N, OH, OW, this->output_channel_}, this->params_.device_, memory::NHWC,
                                          bottoms[0]->allocator());
    if (N == 0) return;
    exb_check(exb_conv2d_fwd(h, &d, bottoms[0]->gpu_data(), packed(h, d), nullptr, tops[0]->mutable_gpu_data(),
                             nullptr, nullptr),
              "exb_conv2d_fwd");
}
INSTANCE_CLASS(operation_convolution);
REGISTE(operation_convolution);

// ---------------------------------------------------------------------------------------------
// depthwise convolution
// ---------------------------------------------------------------------------------------------
template <typename Dtype>
operation_convolutiondepthwise<Dtype>::operation_convolutiondepthwise(const operation_param& param)
    : operation_convolution<Dtype>(param) {}

template <typename Dtype>
operation_convolutiondepthwise<Dtype>::~operation_convolutiondepthwise() {
    if (dw_w_) exb_dw_weights_destroy(dw_w_);
}

template <typename Dtype>
const float* operation_convolutiondepthwise<Dtype>::dw_weights_f32() {
    if (!this->is_int8()) return this->weights_f32_[0]->cpu_data();
    if (dequantized_.empty()) {
        // w = q * (scale <= 1e-6 ? 0 : 1/scale), per output channel
        const int per = this->weight_data_size_ / this->output_channel_;
        dequantized_.resize((size_t)this->weight_data_size_);
        const signed char* q = this->weights_i8_[0]->cpu_data();
        const float* s = this->weights_scaletable_i8_->cpu_data();
        for (int c = 0; c < this->output_channel_; ++c) {
            const float inv = s[c] <= 1e-6 ? 0.f : 1.f / s[c];
            for (int i = 0; i < per; ++i) dequantized_[(size_t)c * per + i] = q[(size_t)c * per + i] * inv;
        }
    }
    return dequantized_.data();
}

template <typename Dtype>
exb_dwconv_desc operation_convolutiondepthwise<Dtype>::dw_desc(int N, int H, int W, int c_stride) const {
    exb_dwconv_desc d;
    std::memset(&d, 0, sizeof(d));
    d.N = N; d.H = H; d.W = W; d.C = this->output_channel_; d.c_stride = c_stride;
    d.kh = this->kernel_size_h_; d.kw = this->kernel_size_w_;
    d.stride_h = this->stride_h_; d.stride_w = this->stride_w_;
    d.pad_t = this->pad_top_; d.pad_b = this->pad_bottom_; d.pad_l = this->pad_left_; d.pad_r = this->pad_right_;
    d.in_dtype = EXB_F16; d.out_dtype = EXB_F16; d.act = this->exb_activation();
    d.in_scale = 1.f; d.out_scale = 1.f;
    return d;
}

template <typename Dtype>
exb_dw_weights* operation_convolutiondepthwise<Dtype>::dw_packed(exb_ctx* ctx, const exb_dwconv_desc& d, const float* post_mul,
                                                                 const float* post_add, const void* tag) {
    const int cs = d.c_stride ? d.c_stride : d.C;
    if (dw_w_ && dw_cs_ == cs && dw_tag_ == tag) return dw_w_;
    if (dw_w_) exb_dw_weights_destroy(dw_w_);
    dw_w_ = nullptr;
    const float* bias = this->bias_term_ ? this->weights_f32_[1]->cpu_data() : nullptr;
    const float* wsrc = dw_weights_f32();
    std::vector<float> fw, fbias;
    if (post_mul) {
        const int C = d.C;
        const size_t per = (size_t)d.kh * d.kw;
        fw.resize((size_t)C * per);
        fbias.resize(C);
        for (int c = 0; c < C; ++c) {
            for (size_t k = 0; k < per; ++k) fw[c * per + k] = wsrc[c * per + k] * post_mul[c];
            fbias[c] = (bias ? bias[c] : 0.f) * post_mul[c] + (post_add ? post_add[c] : 0.f);
        }
        wsrc = fw.data();
        bias = fbias.data();
    }
    exb_check(exb_dw_weights_pack(ctx, &d, wsrc, bias, &dw_w_), "exb_dw_weights_pack");
    dw_cs_ = cs;
    dw_tag_ = tag;
    return dw_w_;
}

template <typename Dtype>
void operation_convolutiondepthwise<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), (size_t)1);
    CHECK_EQ(tops.size(), (size_t)1);
    CHECK_EQ(this->output_channel_, this->group_);
    if (bottoms[0]->order() == memory::NHWC) bottoms[0]->convert_order();
    const int N = bottoms[0]->num(), C = bottoms[0]->channels(), H = bottoms[0]->height(), W = bottoms[0]->width();
    CHECK_EQ(C, this->output_channel_);
    const int dev = this->params_.device_;
    const int cs = round_up(C, 8);
    exb_dwconv_desc d = dw_desc(N, H, W, cs);
    const int OH = (H + d.pad_t + d.pad_b - d.kh) / d.stride_h + 1, OW = (W + d.pad_l + d.pad_r - d.kw) / d.stride_w + 1;
    tops[0] = make_tensor<float>({N, C, OH, OW}, dev, memory::NCHW, bottoms[0]->allocator());
    if (N == 0) return;
    void* xin = this->scratch_in_.get((size_t)N * H * W * cs * 2, dev);
    void* yout = this->scratch_out_.get((size_t)N * OH * OW * cs * 2, dev);
    exb_check(exb_nchw_f32_to_nhwc(h, bottoms[0]->gpu_data(), xin, EXB_F16, N, C, H, W, cs, 1.f, 0, nullptr),
              "exb_nchw_f32_to_nhwc");
    exb_check(exb_dwconv2d_fwd(h, &d, xin, dw_packed(h, d), yout, nullptr), "exb_dwconv2d_fwd");
    exb_check(exb_nhwc_to_nchw_f32(h, yout, EXB_F16, tops[0]->mutable_gpu_data(), N, C, OH, OW, cs, 1.f, nullptr),
              "exb_nhwc_to_nchw_f32");
}
// int8 depthwise = dequantised weights, float activations (the reference does the same).
template <typename Dtype>
void operation_convolutiondepthwise<Dtype>::forward_gpu_i8(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    forward_gpu_f32(h, bottoms, tops);
}
template <typename Dtype>
void operation_convolutiondepthwise<Dtype>::forward_gpu_f16(exb_ctx*& h, const f16_list& bottoms, f16_list& tops) {
    CHECK_EQ(bottoms.size(), (size_t)1);
    CHECK_EQ(tops.size(), (size_t)1);
    if (bottoms[0]->order() != memory::NHWC) NOT_IMPLEMENTED << " (fp16 tensors must be NHWC)";
    const int N = bottoms[0]->num(), C = bottoms[0]->channels(), H = bottoms[0]->height(), W = bottoms[0]->width();
    exb_dwconv_desc d = dw_desc(N, H, W, C);
    const int OH = (H + d.pad_t + d.pad_b - d.kh) / d.stride_h + 1, OW = (W + d.pad_l + d.pad_r - d.kw) / d.stride_w + 1;
    tops[0] = make_tensor<unsigned short>({N, OH, OW, C}, this->params_.device_, memory::NHWC, bottoms[0]->allocator());
    if (N == 0) return;
    exb_check(exb_dwconv2d_fwd(h, &d, bottoms[0]->gpu_data(), dw_packed(h, d), tops[0]->mutable_gpu_data(), nullptr),
              "exb_dwconv2d_fwd");
}
INSTANCE_CLASS(operation_convolutiondepthwise);
REGISTE(operation_convolutiondepthwise);

// ---------------------------------------------------------------------------------------------
// pooling
// ---------------------------------------------------------------------------------------------
template <typename Dtype>
operation_pooling<Dtype>::operation_pooling(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        const int v = std::atoi(kv.second.c_str());
        switch (kv.first) {
        case 0: type_ = v; break;
        case 1: kernel_size_w_ = kernel_size_h_ = v; break;
        case 2: stride_w_ = stride_h_ = v; break;
        case 3: pad_left_ = pad_right_ = pad_top_ = pad_bottom_ = v; break;
        case 4: global_pooling_ = v != 0; break;
        case 5: pad_mode_ = v; break;
        case 6: avgpool_count_include_pad_ = v; break;
        case 11: kernel_size_h_ = v; break;
        case 12: stride_h_ = v; break;
        case 13: pad_top_ = v; break;
        case 14: pad_right_ = v; break;
        case 15: pad_bottom_ = v; break;
        case -23330: break;
        default: LOG(FATAL) << "Un-supported Pooling Attribution " << kv.first;
        }
    }
}

template <typename Dtype>
exb_pool_desc operation_pooling<Dtype>::desc(int N, int H, int W, int C, int c_stride, int dtype) const {
    exb_pool_desc d;
    std::memset(&d, 0, sizeof(d));
    if (type_ != MAX && type_ != AVE) LOG(FATAL) << "Unknown pooling method.";
    if (pad_mode_ != 0 && pad_mode_ != 1) NOT_IMPLEMENTED;
    d.N = N; d.H = H; d.W = W; d.C = C; d.c_stride = c_stride; d.type = type_;
    d.kh = kernel_size_h_; d.kw = kernel_size_w_; d.stride_h = stride_h_; d.stride_w = stride_w_;
    d.pad_t = pad_top_; d.pad_b = pad_bottom_; d.pad_l = pad_left_; d.pad_r = pad_right_;
    d.global_pool = global_pooling_; d.pad_mode = pad_mode_; d.count_include_pad = avgpool_count_include_pad_;
    d.dtype = dtype; d.out2_dtype = -1; d.out2_scale = 1.f;
    return d;
}

template <typename Dtype>
void operation_pooling<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), tops.size());
    for (size_t i = 0; i < bottoms.size(); ++i) {
        const auto& b = bottoms[i];
        const int N = b->num(), C = b->channels(), H = b->height(), W = b->width();
        const int dev = b->device();
        if (b->order() == memory::NHWC && C % 4 == 0) {   // native layout, no conversion
            exb_pool_desc d = desc(N, H, W, C, C, EXB_F32);
            int PH, PW;
            exb_check(exb_pool_out_dims(&d, &PH, &PW), "exb_pool_out_dims");
            tops[i] = make_tensor<float>({N, PH, PW, C}, dev, memory::NHWC, b->allocator());
            if (N) exb_check(exb_pool2d_fwd(h, &d, b->gpu_data(), tops[i]->mutable_gpu_data(), nullptr, nullptr), "exb_pool2d_fwd");
            continue;
        }
        if (b->order() == memory::NHWC) b->convert_order();
        const int cs = round_up(C, 4);
        exb_pool_desc d = desc(N, H, W, C, cs, EXB_F32);
        int PH, PW;
        exb_check(exb_pool_out_dims(&d, &PH, &PW), "exb_pool_out_dims");
        tops[i] = make_tensor<float>({N, C, PH, PW}, dev, memory::NCHW, b->allocator());
        if (N == 0) continue;
        void* xin = scratch_in_.get((size_t)N * H * W * cs * 4, dev);
        void* yout = scratch_out_.get((size_t)N * PH * PW * cs * 4, dev);
        exb_check(exb_nchw_f32_to_nhwc(h, b->gpu_data(), xin, EXB_F32, N, C, H, W, cs, 1.f, 0, nullptr), "exb_nchw_f32_to_nhwc");
        exb_check(exb_pool2d_fwd(h, &d, xin, yout, nullptr, nullptr), "exb_pool2d_fwd");
        exb_check(exb_nhwc_to_nchw_f32(h, yout, EXB_F32, tops[i]->mutable_gpu_data(), N, C, PH, PW, cs, 1.f, nullptr),
                  "exb_nhwc_to_nchw_f32");
    }
}

template <typename Dtype>
void operation_pooling<Dtype>::forward_gpu_f16(exb_ctx*& h, const f16_list& bottoms, f16_list& tops) {
    CHECK_EQ(bottoms.size(), tops.size());
    for (size_t i = 0; i < bottoms.size(); ++i) {
        const auto& b = bottoms[i];
        if (b->order() != memory::NHWC) NOT_IMPLEMENTED << " (fp16 tensors must be NHWC)";
        const int N = b->num(), C = b->channels(), H = b->height(), W = b->width();
        exb_pool_desc d = desc(N, H, W, C, C, EXB_F16);
        int PH, PW;
        exb_check(exb_pool_out_dims(&d, &PH, &PW), "exb_pool_out_dims");
        tops[i] = make_tensor<unsigned short>({N, PH, PW, C}, b->device(), memory::NHWC, b->allocator());
        if (N) exb_check(exb_pool2d_fwd(h, &d, b->gpu_data(), tops[i]->mutable_gpu_data(), nullptr, nullptr), "exb_pool2d_fwd");
    }
}
INSTANCE_CLASS(operation_pooling);
REGISTE(operation_pooling);

// ---------------------------------------------------------------------------------------------
// eltwise / binaryop / relu / clip / sigmoid (layout-agnostic element-wise passes)
// ---------------------------------------------------------------------------------------------
template <typename Dtype>
operation_eltwise<Dtype>::operation_eltwise(const operation_param& param) : operation<Dtype>(param) {
    coeffs_ = std::vector<float>(param.input_count_, 1.0f);
    for (const auto& kv : param_list(param.specific_params_).kv) {
        if (kv.first == 0) {
            type_ = std::atoi(kv.second.c_str());
        } else if (kv.first == -23301) {
            // "<n>,c1,c2,...": the reference reads entries 1..n-1 (so n-1 coefficients; the
            // rest keep their default 1.0) - src/Excalibur/operation_eltwise.cpp:22-30.
            auto parts = split_string(kv.second, ",");
            CHECK_EQ(type_, (int)SUM);
            const int n = parts.empty() ? 0 : std::atoi(parts[0].c_str());
            for (int j = 1; j < n && j < (int)parts.size() && j - 1 < (int)coeffs_.size(); ++j)
                coeffs_[j - 1] = (float)std::atof(parts[j].c_str());
        } else if (kv.first != -23330) {
            LOG(FATAL) << "Un-supported Eltwise Attribution " << kv.first;
        }
    }
}

template <typename T, typename L>
static void eltwise_run(exb_ctx* h, int type, const std::vector<float>& coeffs, const L& bottoms, L& tops, int dtype) {
    CHECK_GE(bottoms.size(), (size_t)2);
    for (size_t i = 1; i < bottoms.size(); ++i) CHECK(bottoms[i]->data_shape() == bottoms[0]->data_shape());
    CHECK_EQ(tops.size(), (size_t)1);
    if (type < 0 || type > 2) LOG(FATAL) << "Unknown elementwise operation.";
    tops[0] = make_tensor<T>(bottoms[0]->data_shape(), bottoms[0]->device(), bottoms[0]->order(), bottoms[0]->allocator());
    std::vector<const void*> xs;
    for (auto& b : bottoms) xs.push_back(b->gpu_data());
    std::vector<float> cf(bottoms.size(), 1.f);
    for (size_t i = 0; i < cf.size() && i < coeffs.size(); ++i) cf[i] = coeffs[i];
    exb_check(exb_eltwise_fwd(h, type, (int)xs.size(), xs.data(), cf.data(), tops[0]->mutable_gpu_data(),
                              tops[0]->count(), dtype, nullptr),
              "exb_eltwise_fwd");
}
template <typename Dtype>
void operation_eltwise<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    eltwise_run<float>(h, type_, coeffs_, bottoms, tops, EXB_F32);
}
template <typename Dtype>
void operation_eltwise<Dtype>::forward_gpu_f16(exb_ctx*& h, const f16_list& bottoms, f16_list& tops) {
    eltwise_run<unsigned short>(h, type_, coeffs_, bottoms, tops, EXB_F16);
}
INSTANCE_CLASS(operation_eltwise);
REGISTE(operation_eltwise);

template <typename Dtype>
operation_binaryop<Dtype>::operation_binaryop(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        switch (kv.first) {
        case 0: op_type_ = std::atoi(kv.second.c_str()); break;
        case 1: with_scalar_ = std::atoi(kv.second.c_str()); break;
        case 2: coef_ = (float)std::atof(kv.second.c_str()); break;
        default: LOG(FATAL) << "Un-supported BinaryOp Attribution " << kv.first;
        }
    }
}
template <typename T, typename L>
static void binaryop_run(exb_ctx* h, int op, int with_scalar, float coef, const L& bottoms, L& tops, int dtype) {
    CHECK_GE(bottoms.size(), (size_t)1);
    CHECK_EQ(tops.size(), (size_t)1);
    if (op < 0 || op > 3) NOT_IMPLEMENTED << " (binary op type " << op << ")";
    tops[0] = make_tensor<T>(bottoms[0]->data_shape(), bottoms[0]->device(), bottoms[0]->order(), bottoms[0]->allocator());
    if (with_scalar) {
        exb_check(exb_binaryop_scalar_fwd(h, op, bottoms[0]->gpu_data(), coef, tops[0]->mutable_gpu_data(),
                                          tops[0]->count(), dtype, nullptr),
                  "exb_binaryop_scalar_fwd");
        return;
    }
    CHECK_GE(bottoms.size(), (size_t)2);
    if (bottoms[0]->data_shape() != bottoms[1]->data_shape()) {
        // (N,C,H,W) with (N or 1,C,1,1) in either order: the per-channel gate of a squeeze-and-excitation block
        const bool first_big = bottoms[0]->count() >= bottoms[1]->count();
        const auto& big = bottoms[first_big ? 0 : 1];
        const auto& small = bottoms[first_big ? 1 : 0];
        const bool gate = big->order() == memory::NCHW && small->channels() == big->channels() && small->height() == 1 &&
                          small->width() == 1 && (small->num() == big->num() || small->num() == 1);
        if (!gate) NOT_IMPLEMENTED << " (broadcasting binary op other than (N,C,H,W) with (N,C,1,1))";
        tops[0] = make_tensor<T>(big->data_shape(), big->device(), big->order(), big->allocator());
        exb_check(exb_binaryop_channel_bcast_fwd(h, op, big->gpu_data(), small->gpu_data(), first_big ? 0 : 1, tops[0]->mutable_gpu_data(),
                                                 big->num(), small->num(), big->channels(), 0,
                                                 (int64_t)big->height() * big->width(), dtype, 0, nullptr),
                  "exb_binaryop_channel_bcast_fwd");
        return;
    }
    exb_check(exb_binaryop_fwd(h, op, bottoms[0]->gpu_data(), bottoms[1]->gpu_data(), tops[0]->mutable_gpu_data(),
                               tops[0]->count(), dtype, nullptr),
              "exb_binaryop_fwd");
}
template <typename Dtype>
void operation_binaryop<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    binaryop_run<float>(h, op_type_, with_scalar_, coef_, bottoms, tops, EXB_F32);
}
template <typename Dtype>
void operation_binaryop<Dtype>::forward_gpu_f16(exb_ctx*& h, const f16_list& bottoms, f16_list& tops) {
    binaryop_run<unsigned short>(h, op_type_, with_scalar_, coef_, bottoms, tops, EXB_F16);
}
INSTANCE_CLASS(operation_binaryop);
REGISTE(operation_binaryop);

template <typename Dtype>
operation_relu<Dtype>::operation_relu(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        if (kv.first == 0) slope_ = (float)std::atof(kv.second.c_str());
        else if (kv.first != -23330) LOG(FATAL) << "Un-supported ReLU Attribution " << kv.first;
    }
    this->params_.inplace_ = true;   // flagged in place, yet a new top is allocated (as the reference does)
}
template <typename T, typename L>
static void act_run(exb_ctx* h, int act, const L& bottoms, L& tops, int dtype) {
    CHECK_EQ(bottoms.size(), tops.size());
    for (size_t i = 0; i < bottoms.size(); ++i) {
        tops[i] = make_tensor<T>(bottoms[i]->data_shape(), bottoms[i]->device(), bottoms[i]->order(), bottoms[i]->allocator());
        int rc = act == EXB_ACT_RELU
                     ? exb_relu_fwd(h, bottoms[i]->gpu_data(), tops[i]->mutable_gpu_data(), tops[i]->count(), dtype, nullptr)
                     : exb_activation_fwd(h, act, bottoms[i]->gpu_data(), tops[i]->mutable_gpu_data(), tops[i]->count(), dtype, nullptr);
        exb_check(rc, "activation kernel");
    }
}
template <typename Dtype>
void operation_relu<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    act_run<float>(h, EXB_ACT_RELU, bottoms, tops, EXB_F32);
}
template <typename Dtype>
void operation_relu<Dtype>::forward_gpu_f16(exb_ctx*& h, const f16_list& bottoms, f16_list& tops) {
    act_run<unsigned short>(h, EXB_ACT_RELU, bottoms, tops, EXB_F16);
}
INSTANCE_CLASS(operation_relu);
REGISTE(operation_relu);

template <typename Dtype>
operation_relu6<Dtype>::operation_relu6(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv)
        if (kv.first != 0 && kv.first != 1 && kv.first != -23330) LOG(FATAL) << "Un-supported ReLU6 Attribution " << kv.first;
    this->params_.inplace_ = true;
}
template <typename Dtype>
void operation_relu6<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    act_run<float>(h, EXB_ACT_RELU6_QUIRK, bottoms, tops, EXB_F32);
}
template <typename Dtype>
void operation_relu6<Dtype>::forward_gpu_f16(exb_ctx*& h, const f16_list& bottoms, f16_list& tops) {
    act_run<unsigned short>(h, EXB_ACT_RELU6_QUIRK, bottoms, tops, EXB_F16);
}
INSTANCE_CLASS(operation_relu6);
REGISTE(operation_relu6);

INSTANCE_CLASS(operation_split);
REGISTE(operation_split);

template <typename Dtype>
operation_clip<Dtype>::operation_clip(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        if (kv.first == 0) min_ = std::stof(kv.second);
        else if (kv.first == 1) max_ = std::stof(kv.second);
        else if (kv.first != -23330) LOG(FATAL) << "Un-supported Clip Attribution " << kv.first;
    }
}
template <typename Dtype>
void operation_clip<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    if (!is_relu6()) NOT_IMPLEMENTED << " (Clip is implemented for the ReLU6 range 0..6 only)";
    act_run<float>(h, EXB_ACT_RELU6, bottoms, tops, EXB_F32);
}
INSTANCE_CLASS(operation_clip);
REGISTE(operation_clip);

template <typename Dtype>
void operation_sigmoid<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    act_run<float>(h, EXB_ACT_SIGMOID, bottoms, tops, EXB_F32);
}
INSTANCE_CLASS(operation_sigmoid);
REGISTE(operation_sigmoid);

// ---------------------------------------------------------------------------------------------
// inner product
// ---------------------------------------------------------------------------------------------
template <typename Dtype>
operation_innerproduct<Dtype>::operation_innerproduct(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        const int v = std::atoi(kv.second.c_str());
        switch (kv.first) {
        case 0: num_output_ = v; break;
        case 1: bias_term_ = v != 0; break;
        case 2: weight_data_size_ = v; break;
        case 8:
            int8_scale_term_ = v != 0;
            this->params_.set_int8_quantization(int8_scale_term_);
            break;
        case 9: activation_type_ = v; break;
        case 10: case -23330: break;
        default: LOG(FATAL) << "Un-supported InnerProduct Attribution " << kv.first;
        }
    }
    CHECK_GT(num_output_, 0);
}
template <typename Dtype>
operation_innerproduct<Dtype>::~operation_innerproduct() {
    if (w_) exb_conv_weights_destroy(w_);
}
template <typename Dtype>
int operation_innerproduct<Dtype>::init_weights(FILE* fp) {
    int tag = 0;
    read_or_die(&tag, sizeof(int), fp, "the quantize tag");
    if (tag != 0) NOT_IMPLEMENTED << " (int8 InnerProduct: the reference has only an ARM implementation)";
    const int dev = this->params_.device_;
    this->weights_f32_.push_back(make_tensor<float>({weight_data_size_}, dev, memory::NCHW));
    read_or_die(this->weights_f32_[0]->mutable_cpu_data(), sizeof(float) * weight_data_size_, fp, "weights");
    int mem = weight_data_size_ * sizeof(float);
    if (bias_term_) {
        this->weights_f32_.push_back(make_tensor<float>({num_output_}, dev, memory::NCHW));
        read_or_die(this->weights_f32_[1]->mutable_cpu_data(), sizeof(float) * num_output_, fp, "bias");
        mem += num_output_ * sizeof(float);
    }
    return mem;
}
template <typename Dtype>
int operation_innerproduct<Dtype>::init_weights() {
    std::default_random_engine e;
    std::normal_distribution<float> n(0, 0.3);
    const int dev = this->params_.device_;
    this->weights_f32_.push_back(make_tensor<float>({weight_data_size_}, dev, memory::NCHW));
    float* w = this->weights_f32_[0]->mutable_cpu_data();
    for (int i = 0; i < weight_data_size_; ++i) w[i] = n(e);
    if (bias_term_) {
        this->weights_f32_.push_back(make_tensor<float>({num_output_}, dev, memory::NCHW));
        float* b = this->weights_f32_[1]->mutable_cpu_data();
        for (int i = 0; i < num_output_; ++i) b[i] = n(e);
    }
    return (weight_data_size_ + (bias_term_ ? num_output_ : 0)) * (int)sizeof(float);
}
template <typename Dtype>
exb_conv_desc operation_innerproduct<Dtype>::fc_desc(int N, int cin_stride) const {
    exb_conv_desc d;
    std::memset(&d, 0, sizeof(d));
    d.N = N; d.H = 1; d.W = 1; d.Cin = in_features(); d.Cout = num_output_; d.cin_stride = cin_stride;
    d.kh = d.kw = 1; d.stride_h = d.stride_w = 1; d.dilation = 1; d.group = 1;
    d.in_dtype = EXB_F16; d.out_dtype = EXB_F32; d.out2_dtype = -1; d.res_dtype = -1;
    d.act = activation_type_ == 1 ? EXB_ACT_RELU : (activation_type_ == 4 ? EXB_ACT_SIGMOID : EXB_ACT_NONE);
    d.out_scale = d.out2_scale = 1.f;
    return d;
}
template <typename Dtype>
exb_conv_weights* operation_innerproduct<Dtype>::packed(exb_ctx* ctx, const exb_conv_desc& d) {
    if (w_ && w_cin_stride_ == d.cin_stride && w_cout_stride_ == d.cout_stride) return w_;
    if (w_) exb_conv_weights_destroy(w_);
    w_ = nullptr;
    const float* bias = bias_term_ ? this->weights_f32_[1]->cpu_data() : nullptr;
    exb_check(exb_conv_weights_pack_f16(ctx, &d, this->weights_f32_[0]->cpu_data(), bias, &w_), "exb_conv_weights_pack_f16");
    w_cin_stride_ = d.cin_stride;
    w_cout_stride_ = d.cout_stride;
    return w_;
}
// bottoms[0]: {N, C, H, W} fp32 NCHW, flattened to N x (C*H*W) like the reference.
template <typename Dtype>
void operation_innerproduct<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), (size_t)1);
    CHECK_EQ(tops.size(), (size_t)1);
    if (bottoms[0]->order() == memory::NHWC) bottoms[0]->convert_order();
    const int N = bottoms[0]->num(), K = bottoms[0]->count(1, 4);
    CHECK_EQ(K, in_features()) << "flattened input size does not match the weights";
    const int dev = this->params_.device_;
    const int ks = round_up(K, 16);
    exb_conv_desc d = fc_desc(N, ks);
    tops[0] = make_tensor<float>({N, num_output_, 1, 1}, dev, memory::NCHW, bottoms[0]->allocator());
    if (N == 0) return;
    void* xin = scratch_in_.get((size_t)N * ks * 2, dev);
    // {N, K, 1, 1} NCHW -> NHWC fp16 with padded channels
    exb_check(exb_nchw_f32_to_nhwc(h, bottoms[0]->gpu_data(), xin, EXB_F16, N, K, 1, 1, ks, 1.f, 0, nullptr),
              "exb_nchw_f32_to_nhwc");
    exb_check(exb_conv2d_fwd(h, &d, xin, packed(h, d), nullptr, tops[0]->mutable_gpu_data(), nullptr, nullptr),
              "exb_conv2d_fwd");
}
INSTANCE_CLASS(operation_innerproduct);
REGISTE(operation_innerproduct);

// ---------------------------------------------------------------------------------------------
// graph glue: concat, nearest resize, batch norm
// ---------------------------------------------------------------------------------------------
template <typename Dtype>
operation_concat<Dtype>::operation_concat(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        if (kv.first == 0) axis_ = (int)std::atof(kv.second.c_str());
        else if (kv.first != -23330) LOG(FATAL) << "Un-supported Concat Attribution " << kv.first;
    }
}
template <typename Dtype>
void operation_concat<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_GE(bottoms.size(), 2u);
    CHECK_EQ(tops.size(), 1u);
    if (!is_channel_concat()) NOT_IMPLEMENTED << " (Concat is implemented along the channel axis, key 0=-1)";
    CHECK(bottoms[0]->order() == memory::NCHW) << "Concat expects NCHW tensors";
    const int N = bottoms[0]->num(), H = bottoms[0]->height(), W = bottoms[0]->width();
    int C = 0;
    std::vector<const void*> xs;
    std::vector<int64_t> widths;
    for (const auto& b : bottoms) {
        CHECK_EQ(b->num(), N);
        CHECK_EQ(b->height(), H);
        CHECK_EQ(b->width(), W);
        C += b->channels();
        xs.push_back(b->gpu_data());
        widths.push_back((int64_t)b->channels() * H * W);
    }
    tops[0] = make_tensor<float>({N, C, H, W}, bottoms[0]->device(), memory::NCHW, bottoms[0]->allocator());
    if (tops[0]->count() == 0) return;
    exb_check(exb_concat_fwd(h, (int)xs.size(), xs.data(), widths.data(), widths.data(), tops[0]->mutable_gpu_data(),
                             (int64_t)C * H * W, N, EXB_F32, nullptr), "exb_concat_fwd");
}
INSTANCE_CLASS(operation_concat);
REGISTE(operation_concat);

template <typename Dtype>
operation_interp<Dtype>::operation_interp(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        switch (kv.first) {
        case 0: resize_type_ = std::atoi(kv.second.c_str()); break;
        case 1: width_scale_ = std::stof(kv.second); break;
        case 2: height_scale_ = std::stof(kv.second); break;
        case 3: output_width_ = std::atoi(kv.second.c_str()); break;
        case 4: output_height_ = std::atoi(kv.second.c_str()); break;
        case 6: align_corner_ = std::atoi(kv.second.c_str()); break;
        default: LOG(FATAL) << "Un-supported Interp Attribution " << kv.first;
        }
    }
}
template <typename Dtype>
void operation_interp<Dtype>::out_dims(int H, int W, int* OH, int* OW) const {
    if (output_width_ == 0 || output_height_ == 0) {
        *OH = static_cast<int>(H * height_scale_);
        *OW = static_cast<int>(W * width_scale_);
    } else {
        *OH = output_height_;
        *OW = output_width_;
    }
}
template <typename Dtype>
void operation_interp<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(tops.size(), 1u);
    if (bottoms.size() != 1) NOT_IMPLEMENTED << " (Interp with a size tensor as second input)";
    if (resize_type_ != 1 || align_corner_ != 0) NOT_IMPLEMENTED << " (Interp is implemented for nearest mode, keys 0=1 6=0)";
    CHECK(bottoms[0]->order() == memory::NCHW) << "Interp expects an NCHW tensor";
    const int N = bottoms[0]->num(), C = bottoms[0]->channels(), H = bottoms[0]->height(), W = bottoms[0]->width();
    int OH = 0, OW = 0;
    out_dims(H, W, &OH, &OW);
    CHECK_GT(OH, 0);
    CHECK_GT(OW, 0);
    tops[0] = make_tensor<float>({N, C, OH, OW}, bottoms[0]->device(), memory::NCHW, bottoms[0]->allocator());
    if (tops[0]->count() == 0) return;
    exb_check(exb_interp_nearest_fwd(h, bottoms[0]->gpu_data(), tops[0]->mutable_gpu_data(), N, H, W, C, 0, OH, OW, EXB_F32,
                                     0, nullptr), "exb_interp_nearest_fwd");
}
INSTANCE_CLASS(operation_interp);
REGISTE(operation_interp);

template <typename Dtype>
operation_batchnorm<Dtype>::operation_batchnorm(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        if (kv.first == 0) channels_ = std::atoi(kv.second.c_str());
        else if (kv.first == 1) eps_ = (float)std::atof(kv.second.c_str());
        else LOG(FATAL) << "Un-supported Batchnorm Attribution " << kv.first;
    }
    this->params_.inplace_ = true;
}
template <typename Dtype>
void operation_batchnorm<Dtype>::derive() {
    const int dev = this->params_.device_;
    const float* slope = this->weights_f32_[0]->cpu_data();
    const float* mean = this->weights_f32_[1]->cpu_data();
    const float* var = this->weights_f32_[2]->cpu_data();
    const float* bias = this->weights_f32_[3]->cpu_data();
    a_ = make_tensor<float>({channels_}, dev, memory::NCHW);
    b_ = make_tensor<float>({channels_}, dev, memory::NCHW);
    float* a = a_->mutable_cpu_data();
    float* b = b_->mutable_cpu_data();
    for (int i = 0; i < channels_; ++i) {
        const float sqrt_var = static_cast<float>(std::sqrt(var[i] + eps_));
        a[i] = bias[i] - slope[i] * mean[i] / sqrt_var;
        b[i] = slope[i] / sqrt_var;
    }
}
template <typename Dtype>
int operation_batchnorm<Dtype>::init_weights(FILE* fp) {
    const int dev = this->params_.device_;
    static const char* const what[4] = {"slope", "mean", "var", "bias"};
    for (int k = 0; k < 4; ++k) {
        this->weights_f32_.push_back(make_tensor<float>({channels_}, dev, memory::NCHW));
        read_or_die(this->weights_f32_[k]->mutable_cpu_data(), sizeof(float) * channels_, fp, what[k]);
    }
    derive();
    return channels_ * (int)sizeof(float) * 4;
}
template <typename Dtype>
int operation_batchnorm<Dtype>::init_weights() {
    std::default_random_engine e;
    std::normal_distribution<float> n(0, 0.3);
    const int dev = this->params_.device_;
    for (int k = 0; k < 4; ++k) {
        this->weights_f32_.push_back(make_tensor<float>({channels_}, dev, memory::NCHW));
        float* w = this->weights_f32_[k]->mutable_cpu_data();
        for (int i = 0; i < channels_; ++i) w[i] = n(e);
    }
    derive();
    return channels_ * (int)sizeof(float) * 4;
}
template <typename Dtype>
void operation_batchnorm<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), 1u);
    CHECK_EQ(tops.size(), 1u);
    CHECK(bottoms[0]->order() == memory::NCHW) << "BatchNorm expects an NCHW tensor";
    CHECK_EQ(bottoms[0]->channels(), channels_);
    tops[0] = make_tensor<float>(bottoms[0]->data_shape(), bottoms[0]->device(), memory::NCHW, bottoms[0]->allocator());
    if (tops[0]->count() == 0) return;
    exb_check(exb_channel_affine_fwd(h, bottoms[0]->gpu_data(), tops[0]->mutable_gpu_data(), b_->gpu_data(), a_->gpu_data(),
                                     bottoms[0]->num(), channels_, 0, (int64_t)bottoms[0]->height() * bottoms[0]->width(),
                                     EXB_F32, 0, EXB_ACT_NONE, nullptr), "exb_channel_affine_fwd");
}
INSTANCE_CLASS(operation_batchnorm);
REGISTE(operation_batchnorm);

// ---------------------------------------------------------------------------------------------
// HardSwish, Input normalisation, YoloV5Focus
// ---------------------------------------------------------------------------------------------
template <typename Dtype>
operation_hardswish<Dtype>::operation_hardswish(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        if (kv.first == 0) alpha_ = std::stof(kv.second);
        else if (kv.first == 1) beta_ = std::stof(kv.second);
        else LOG(FATAL) << "Un-supported HardSwish Attribution " << kv.first;
    }
}
template <typename Dtype>
void operation_hardswish<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), 1u);
    CHECK_EQ(tops.size(), 1u);
    tops[0] = make_tensor<float>(bottoms[0]->data_shape(), bottoms[0]->device(), bottoms[0]->order(), bottoms[0]->allocator());
    exb_check(exb_hardswish_fwd(h, bottoms[0]->gpu_data(), tops[0]->mutable_gpu_data(), tops[0]->count(), EXB_F32, alpha_,
                                beta_, nullptr), "exb_hardswish_fwd");
}
INSTANCE_CLASS(operation_hardswish);
REGISTE(operation_hardswish);

template <typename Dtype>
operation_input<Dtype>::operation_input(const operation_param& param) : operation<Dtype>(param) {
    auto list_of = [](const std::string& v) {
        std::vector<float> out;
        size_t pos = 0;
        while (pos <= v.size()) {
            const size_t next = v.find(',', pos);
            const std::string tok = v.substr(pos, next == std::string::npos ? std::string::npos : next - pos);
            if (!tok.empty()) out.push_back((float)std::atof(tok.c_str()));
            if (next == std::string::npos) break;
            pos = next + 1;
        }
        return out;
    };
    for (const auto& kv : param_list(param.specific_params_).kv) {
        switch (kv.first) {
        case 0: w_ = std::atoi(kv.second.c_str()); break;
        case 1: h_ = std::atoi(kv.second.c_str()); break;
        case 2: c_ = std::atoi(kv.second.c_str()); break;
        case 3: means_ = list_of(kv.second); break;
        case 4:
            vars_ = list_of(kv.second);
            if (c_ != 1 && (int)vars_.size() != c_) {   // one value stands for every channel
                if (!vars_.empty()) vars_.resize(1);
                for (int i = 1; i < c_; ++i) vars_.push_back(vars_[0]);
            }
            break;
        case -23330: break;
        default: LOG(FATAL) << "Un-supported Input Attribution " << kv.first;
        }
    }
}
template <typename Dtype>
void operation_input<Dtype>::coefficients(int channels, const float** mul, const float** add) {
    if (channels != 1 && channels != 3) LOG(FATAL) << "Un-supprted channel num: " << channels;
    CHECK_EQ((size_t)channels, means_.size());
    CHECK_GE(vars_.size(), (size_t)channels);
    if (!mul_ || mul_->count() != channels) {
        const int dev = this->params_.device_;
        mul_ = make_tensor<float>({channels}, dev, memory::NCHW);
        add_ = make_tensor<float>({channels}, dev, memory::NCHW);
        for (int c = 0; c < channels; ++c) {
            mul_->mutable_cpu_data()[c] = vars_[c];
            add_->mutable_cpu_data()[c] = -means_[c] * vars_[c];
        }
    }
    *mul = mul_->gpu_data();
    *add = add_->gpu_data();
}
template <typename Dtype>
void operation_input<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), tops.size());
    for (size_t i = 0; i < bottoms.size(); ++i) {
        CHECK(bottoms[i]->order() == memory::NCHW) << "Input expects an NCHW tensor";
        const float* mul = nullptr;
        const float* add = nullptr;
        coefficients(bottoms[i]->channels(), &mul, &add);
        tops[i] = make_tensor<float>(bottoms[i]->data_shape(), bottoms[i]->device(), memory::NCHW, bottoms[i]->allocator());
        if (tops[i]->count() == 0) continue;
        exb_check(exb_channel_affine_fwd(h, bottoms[i]->gpu_data(), tops[i]->mutable_gpu_data(), mul, add, bottoms[i]->num(),
                                         bottoms[i]->channels(), 0, (int64_t)bottoms[i]->height() * bottoms[i]->width(),
                                         EXB_F32, 0, EXB_ACT_NONE, nullptr), "exb_channel_affine_fwd");
    }
}
INSTANCE_CLASS(operation_input);
REGISTE(operation_input);

template <typename Dtype>
void operation_yolov5focus<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), 1u);
    CHECK_EQ(tops.size(), 1u);
    CHECK(bottoms[0]->order() == memory::NCHW) << "YoloV5Focus expects an NCHW tensor";
    const int N = bottoms[0]->num(), C = bottoms[0]->channels(), H = bottoms[0]->height(), W = bottoms[0]->width();
    tops[0] = make_tensor<float>({N, 4 * C, H / 2, W / 2}, bottoms[0]->device(), memory::NCHW, bottoms[0]->allocator());
    if (tops[0]->count() == 0) return;
    exb_check(exb_focus_fwd(h, bottoms[0]->gpu_data(), tops[0]->mutable_gpu_data(), N, C, H, W, 0, 0, EXB_F32, 0, nullptr),
              "exb_focus_fwd");
}
INSTANCE_CLASS(operation_yolov5focus);
REGISTE(operation_yolov5focus);

// ---------------------------------------------------------------------------------------------
// PReLU, LeakyRelu
// ---------------------------------------------------------------------------------------------
template <typename Dtype>
operation_prelu<Dtype>::operation_prelu(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        if (kv.first == 0) {
            num_slope_ = std::atoi(kv.second.c_str());
            CHECK_GE(num_slope_, 1);
        } else if (kv.first != -23330) {
            LOG(FATAL) << "Un-supported PReLU Attribution " << kv.first;
        }
    }
    this->params_.inplace_ = true;
}
template <typename Dtype>
int operation_prelu<Dtype>::init_weights(FILE* fp) {
    this->weights_f32_.push_back(make_tensor<float>({num_slope_}, this->params_.device_, memory::NCHW));
    read_or_die(this->weights_f32_[0]->mutable_cpu_data(), sizeof(float) * num_slope_, fp, "PReLU slopes");
    return num_slope_ * (int)sizeof(float);
}
template <typename Dtype>
int operation_prelu<Dtype>::init_weights() {
    std::default_random_engine e;
    std::normal_distribution<float> n(0, 0.3);
    this->weights_f32_.push_back(make_tensor<float>({num_slope_}, this->params_.device_, memory::NCHW));
    for (int i = 0; i < num_slope_; ++i) this->weights_f32_[0]->mutable_cpu_data()[i] = std::fabs(n(e));
    return num_slope_ * (int)sizeof(float);
}
template <typename Dtype>
void operation_prelu<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), tops.size());
    for (size_t i = 0; i < bottoms.size(); ++i) {
        CHECK(bottoms[i]->order() == memory::NCHW) << "PReLU expects an NCHW tensor";
        if (num_slope_ != 1) CHECK_EQ(bottoms[i]->channels(), num_slope_);
        tops[i] = make_tensor<float>(bottoms[i]->data_shape(), bottoms[i]->device(), memory::NCHW, bottoms[i]->allocator());
        if (tops[i]->count() == 0) continue;
        exb_check(exb_prelu_fwd(h, bottoms[i]->gpu_data(), tops[i]->mutable_gpu_data(), slopes_gpu(), num_slope_,
                                bottoms[i]->num(), bottoms[i]->channels(), 0,
                                (int64_t)bottoms[i]->height() * bottoms[i]->width(), EXB_F32, 0, nullptr), "exb_prelu_fwd");
    }
}
INSTANCE_CLASS(operation_prelu);
REGISTE(operation_prelu);

template <typename Dtype>
operation_leakyrelu<Dtype>::operation_leakyrelu(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        if (kv.first == 0) alpha_ = std::stof(kv.second);
        else LOG(FATAL) << "Un-supported Leakyrelu Attribution " << kv.first;
    }
}
template <typename Dtype>
const float* operation_leakyrelu<Dtype>::slope_gpu() {
    if (!slope_) {
        slope_ = make_tensor<float>({1}, this->params_.device_, memory::NCHW);
        slope_->mutable_cpu_data()[0] = alpha_;
    }
    return slope_->gpu_data();
}
template <typename Dtype>
void operation_leakyrelu<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), 1u);
    CHECK_EQ(tops.size(), 1u);
    tops[0] = make_tensor<float>(bottoms[0]->data_shape(), bottoms[0]->device(), bottoms[0]->order(), bottoms[0]->allocator());
    if (tops[0]->count() == 0) return;
    // one shared slope: the layout does not matter, the tensor is a flat array of count() values
    exb_check(exb_prelu_fwd(h, bottoms[0]->gpu_data(), tops[0]->mutable_gpu_data(), slope_gpu(), 1, 1, 1, 0,
                            (int64_t)tops[0]->count(), EXB_F32, 0, nullptr), "exb_prelu_fwd");
}
INSTANCE_CLASS(operation_leakyrelu);
REGISTE(operation_leakyrelu);

// ---------------------------------------------------------------------------------------------
// Deconvolution
// ---------------------------------------------------------------------------------------------
template <typename Dtype>
operation_deconvolution<Dtype>::operation_deconvolution(const operation_param& param)
    : operation_general_conv<Dtype>(param) {}
template <typename Dtype>
operation_deconvolution<Dtype>::~operation_deconvolution() {
    for (auto& e : packed_) exb_conv_weights_destroy(e.w);
}
template <typename Dtype>
int operation_deconvolution<Dtype>::init_weights(FILE* fp) {
    int tag = 0;
    read_or_die(&tag, sizeof(int), fp, "the quantize tag");
    if (tag != 0) NOT_IMPLEMENTED << " (quantised deconvolution weights, tag " << tag << ")";
    const int dev = this->params_.device_;
    this->weights_f32_.push_back(make_tensor<float>({this->weight_data_size_}, dev, memory::NCHW));
    read_or_die(this->weights_f32_[0]->mutable_cpu_data(), sizeof(float) * this->weight_data_size_, fp, "weights");
    int mem = this->weight_data_size_ * (int)sizeof(float);
    if (this->bias_term_) {
        this->weights_f32_.push_back(make_tensor<float>({this->output_channel_}, dev, memory::NCHW));
        read_or_die(this->weights_f32_[1]->mutable_cpu_data(), sizeof(float) * this->output_channel_, fp, "bias");
        mem += this->output_channel_ * (int)sizeof(float);
    }
    return mem;
}
template <typename Dtype>
int operation_deconvolution<Dtype>::init_weights() {
    if (this->params_.int8_quantization_) NOT_IMPLEMENTED << " (int8 deconvolution)";
    std::default_random_engine e;
    std::normal_distribution<float> n(0, 0.3);
    const int dev = this->params_.device_;
    this->weights_f32_.push_back(make_tensor<float>({this->weight_data_size_}, dev, memory::NCHW));
    float* w = this->weights_f32_[0]->mutable_cpu_data();
    for (int i = 0; i < this->weight_data_size_; ++i) w[i] = n(e);
    int mem = this->weight_data_size_ * (int)sizeof(float);
    if (this->bias_term_) {
        this->weights_f32_.push_back(make_tensor<float>({this->output_channel_}, dev, memory::NCHW));
        float* b = this->weights_f32_[1]->mutable_cpu_data();
        for (int i = 0; i < this->output_channel_; ++i) b[i] = n(e);
        mem += this->output_channel_ * (int)sizeof(float);
    }
    return mem;
}
template <typename Dtype>
bool operation_deconvolution<Dtype>::supported() const {
    return this->group_ == 1 && this->kernel_size_h_ == this->stride_h_ && this->kernel_size_w_ == this->stride_w_ &&
           this->pad_left_ == 0 && this->pad_right_ == 0 && this->pad_top_ == 0 && this->pad_bottom_ == 0 &&
           this->dilation_h_ == 1 && this->dilation_w_ == 1 && this->activation_type_ == 0;
}
template <typename Dtype>
exb_conv_desc operation_deconvolution<Dtype>::inner_desc(int N, int H, int W, int cin_stride) const {
    exb_conv_desc d;
    std::memset(&d, 0, sizeof(d));
    d.N = N; d.H = H; d.W = W;
    d.Cin = this->input_channel_;
    d.Cout = this->output_channel_ * this->kernel_size_h_ * this->kernel_size_w_;
    d.kh = d.kw = 1; d.stride_h = d.stride_w = 1; d.dilation = 1; d.group = 1;
    d.in_dtype = EXB_F16; d.cin_stride = cin_stride;
    d.out_dtype = EXB_F16; d.out2_dtype = -1; d.res_dtype = -1;
    d.act = EXB_ACT_NONE; d.out_scale = 1.f; d.out2_scale = 1.f; d.impl = 0;
    return d;
}
template <typename Dtype>
exb_conv_weights* operation_deconvolution<Dtype>::packed(exb_ctx* ctx, const exb_conv_desc& d, const float* post_mul,
                                                         const float* post_add, const void* tag) {
    if (!supported())
        NOT_IMPLEMENTED << " (Deconvolution is implemented for kernel == stride, no padding, no dilation, one group)";
    const int cin_stride = d.cin_stride ? d.cin_stride : d.Cin;
    const int cout_stride = d.cout_stride ? d.cout_stride : d.Cout;
    for (auto& e : packed_)
        if (e.cin_stride == cin_stride && e.cout_stride == cout_stride && e.tag == tag) return e.w;
    const int Cin = this->input_channel_, Cout = this->output_channel_;
    const int taps = this->kernel_size_h_ * this->kernel_size_w_;
    const float* src = this->weights_f32_[0]->cpu_data();     // [Cin][Cout][taps]
    const float* bias = this->bias_term_ ? this->weights_f32_[1]->cpu_data() : nullptr;
    std::vector<float> w((size_t)taps * Cout * Cin), b((size_t)taps * Cout);
    for (int t = 0; t < taps; ++t)
        for (int co = 0; co < Cout; ++co) {
            const float m = post_mul ? post_mul[co] : 1.f;
            const size_t o = (size_t)t * Cout + co;
            for (int ci = 0; ci < Cin; ++ci) w[o * Cin + ci] = src[((size_t)ci * Cout + co) * taps + t] * m;
            b[o] = (bias ? bias[co] : 0.f) * m + (post_add ? post_add[co] : 0.f);
        }
    exb_conv_weights* out = nullptr;
    exb_check(exb_conv_weights_pack_f16(ctx, &d, w.data(), b.data(), &out), "exb_conv_weights_pack_f16");
    packed_.push_back({cin_stride, cout_stride, out, tag});
    return out;
}
// Stand-alone semantics: fp32 NCHW in and out; fp16 operands, fp32 accumulation.
template <typename Dtype>
void operation_deconvolution<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), (size_t)1);
    CHECK_EQ(tops.size(), (size_t)1);
    if (bottoms[0]->order() == memory::NHWC) bottoms[0]->convert_order();
    const int N = bottoms[0]->num(), C = bottoms[0]->channels(), H = bottoms[0]->height(), W = bottoms[0]->width();
    CHECK_EQ(C, this->input_channel_) << "input channels do not match the weights";
    const int dev = this->params_.device_;
    const int rh = this->kernel_size_h_, rw = this->kernel_size_w_, Cout = this->output_channel_;
    exb_conv_desc d = inner_desc(N, H, W, round_up(C, 16));
    d.out_dtype = EXB_F32;
    tops[0] = make_tensor<float>({N, Cout, H * rh, W * rw}, dev, memory::NCHW, bottoms[0]->allocator());
    if (tops[0]->count() == 0) return;
    void* xin = scratch_in_.get((size_t)N * H * W * d.cin_stride * 2, dev);
    void* mid = scratch_mid_.get((size_t)N * H * W * d.Cout * sizeof(float), dev);
    void* yout = scratch_out_.get((size_t)tops[0]->count() * sizeof(float), dev);
    exb_check(exb_nchw_f32_to_nhwc(h, bottoms[0]->gpu_data(), xin, EXB_F16, N, C, H, W, d.cin_stride, 1.f, 0, nullptr),
              "exb_nchw_f32_to_nhwc");
    exb_check(exb_conv2d_fwd(h, &d, xin, packed(h, d), nullptr, mid, nullptr, nullptr), "exb_conv2d_fwd");
    exb_check(exb_depth_to_space_fwd(h, mid, yout, N, H, W, rh, rw, Cout, 0, 0, EXB_F32, nullptr), "exb_depth_to_space_fwd");
    exb_check(exb_nhwc_to_nchw_f32(h, yout, EXB_F32, tops[0]->mutable_gpu_data(), N, Cout, H * rh, W * rw, Cout, 1.f, nullptr),
              "exb_nhwc_to_nchw_f32");
}
INSTANCE_CLASS(operation_deconvolution);
REGISTE(operation_deconvolution);

// ---------------------------------------------------------------------------------------------
// Reshape, Transpose
// ---------------------------------------------------------------------------------------------
template <typename Dtype>
operation_reshape<Dtype>::operation_reshape(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        const int v = std::atoi(kv.second.c_str());
        switch (kv.first) {
        case 0: w_ = v; break;
        case 1: h_ = v; break;
        case 2: c_ = v; break;
        case 3: permute_ = v; break;
        case -23330: break;
        default: LOG(FATAL) << "Un-supported Reshape Attribution " << kv.first;
        }
    }
    this->params_.inplace_ = true;
}
template <typename Dtype>
std::vector<int> operation_reshape<Dtype>::out_shape(const std::vector<int>& in) const {
    CHECK_EQ(in.size(), (size_t)4);
    std::vector<int> s = in;
    const int64_t count = (int64_t)in[0] * in[1] * in[2] * in[3];
    if (c_ > 0) s[1] = c_;
    if (h_ > 0) s[2] = h_;
    if (w_ > 0) s[3] = w_;
    auto deduce = [&](int axis) {
        int64_t rest = 1;
        for (int a = 0; a < 4; ++a) if (a != axis) rest *= s[a];
        CHECK(rest > 0 && count % rest == 0) << "Reshape: " << count << " values do not divide into the requested shape";
        s[axis] = (int)(count / rest);
    };
    if (c_ < 0) deduce(1);
    if (h_ < 0) deduce(2);
    if (w_ < 0) deduce(3);
    CHECK_EQ((int64_t)s[0] * s[1] * s[2] * s[3], count) << "Reshape changes the number of values";
    return s;
}
template <typename Dtype>
void operation_reshape<Dtype>::forward_gpu_f32(exb_ctx*&, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), 1u);
    CHECK_EQ(tops.size(), 1u);
    CHECK(bottoms[0]->order() == memory::NCHW) << "Reshape expects an NCHW tensor";
    bottoms[0]->reshape(out_shape(bottoms[0]->data_shape()));
    tops[0] = bottoms[0];
}
INSTANCE_CLASS(operation_reshape);
REGISTE(operation_reshape);

template <typename Dtype>
operation_transpose<Dtype>::operation_transpose(const operation_param& param) : operation<Dtype>(param), perms_{0, 1, 2} {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        if (kv.first != 0) LOG(FATAL) << "Un-supported Transpose Attribution " << kv.first;
        perms_.clear();
        size_t pos = 0;
        const std::string& v = kv.second;
        while (pos <= v.size()) {
            const size_t next = v.find(',', pos);
            const std::string tok = v.substr(pos, next == std::string::npos ? std::string::npos : next - pos);
            if (!tok.empty()) perms_.push_back(std::atoi(tok.c_str()));
            if (next == std::string::npos) break;
            pos = next + 1;
        }
    }
}
template <typename Dtype>
void operation_transpose<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), 1u);
    CHECK_EQ(tops.size(), 1u);
    CHECK(bottoms[0]->order() == memory::NCHW) << "Transpose expects an NCHW tensor";
    if (is_identity()) {
        tops[0] = bottoms[0];
        return;
    }
    if (!is_swap_hw()) NOT_IMPLEMENTED << " (Transpose is implemented for the permutations 0,1,2 and 1,0,2)";
    const int N = bottoms[0]->num(), C = bottoms[0]->channels(), H = bottoms[0]->height(), W = bottoms[0]->width();
    tops[0] = make_tensor<float>({N, C, W, H}, bottoms[0]->device(), memory::NCHW, bottoms[0]->allocator());
    if (tops[0]->count() == 0) return;
    exb_check(exb_transpose_hw_f32(h, bottoms[0]->gpu_data(), tops[0]->mutable_gpu_data(), (int64_t)N * C, H, W, nullptr),
              "exb_transpose_hw_f32");
}
INSTANCE_CLASS(operation_transpose);
REGISTE(operation_transpose);

// ---------------------------------------------------------------------------------------------
// HardSigmoid, Softmax, Flatten
// ---------------------------------------------------------------------------------------------
template <typename Dtype>
operation_hardsigmoid<Dtype>::operation_hardsigmoid(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        if (kv.first == 0) alpha_ = std::stof(kv.second);
        else if (kv.first == 1) beta_ = std::stof(kv.second);
        else LOG(FATAL) << "Un-supported Hardsigmoid Attribution " << kv.first;
    }
}
template <typename Dtype>
void operation_hardsigmoid<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), 1u);
    CHECK_EQ(tops.size(), 1u);
    tops[0] = make_tensor<float>(bottoms[0]->data_shape(), bottoms[0]->device(), bottoms[0]->order(), bottoms[0]->allocator());
    exb_check(exb_hardsigmoid_fwd(h, bottoms[0]->gpu_data(), tops[0]->mutable_gpu_data(), tops[0]->count(), EXB_F32, alpha_,
                                  beta_, nullptr), "exb_hardsigmoid_fwd");
}
INSTANCE_CLASS(operation_hardsigmoid);
REGISTE(operation_hardsigmoid);

template <typename Dtype>
operation_softmax<Dtype>::operation_softmax(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        if (kv.first == 0) axis_ = std::atoi(kv.second.c_str());
        else if (kv.first != 1 && kv.first != -23330) LOG(FATAL) << "Un-supported Softmax Attribution " << kv.first;
    }
}
template <typename Dtype>
void operation_softmax<Dtype>::forward_gpu_f32(exb_ctx*& h, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), tops.size());
    for (size_t i = 0; i < bottoms.size(); ++i) {
        CHECK(bottoms[i]->order() == memory::NCHW) << "Softmax expects an NCHW tensor";
        tops[i] = make_tensor<float>(bottoms[i]->data_shape(), bottoms[i]->device(), memory::NCHW, bottoms[i]->allocator());
        if (tops[i]->count() == 0) continue;
        exb_check(exb_softmax_channels_f32(h, bottoms[i]->gpu_data(), tops[i]->mutable_gpu_data(), bottoms[i]->num(),
                                           bottoms[i]->channels(), (int64_t)bottoms[i]->height() * bottoms[i]->width(), 0,
                                           nullptr), "exb_softmax_channels_f32");
    }
}
INSTANCE_CLASS(operation_softmax);
REGISTE(operation_softmax);

template <typename Dtype>
operation_flatten<Dtype>::operation_flatten(const operation_param& param) : operation<Dtype>(param) {
    for (const auto& kv : param_list(param.specific_params_).kv) {
        if (kv.first == 0) axis_ = std::atoi(kv.second.c_str());
        else LOG(FATAL) << "Un-supported flatten Attribution " << kv.first;
    }
}
template <typename Dtype>
std::vector<int> operation_flatten<Dtype>::out_shape(const std::vector<int>& in) const {
    CHECK_EQ(in.size(), (size_t)4);
    const int c = in[1], h = in[2], w = in[3];
    switch (axis_) {
    case 0: return {in[0], 1, c * h * w, 1};
    case 1: return {in[0], 1, c * h, w};
    case 2: return {in[0], 1, c, h * w};
    case 3: return {in[0], 1, 1, c * h * w};
    default: NOT_IMPLEMENTED << " (Flatten axis " << axis_ << ")";
    }
    return in;
}
template <typename Dtype>
void operation_flatten<Dtype>::forward_gpu_f32(exb_ctx*&, const f32_list& bottoms, f32_list& tops) {
    CHECK_EQ(bottoms.size(), 1u);
    CHECK_EQ(tops.size(), 1u);
    CHECK(bottoms[0]->order() == memory::NCHW) << "Flatten expects an NCHW tensor";
    tops[0] = make_tensor<float>(out_shape(bottoms[0]->data_shape()), bottoms[0]->device(), memory::NCHW, bottoms[0]->allocator());
    if (tops[0]->count() == 0) return;
    CUDA_CHECK(cudaMemcpy(tops[0]->mutable_gpu_data(), bottoms[0]->gpu_data(), sizeof(float) * tops[0]->count(),
                          cudaMemcpyDeviceToDevice));
}
INSTANCE_CLASS(operation_flatten);
REGISTE(operation_flatten);

}  // namespace excalibur
}  // namespace glasssix
