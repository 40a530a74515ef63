// gw_math_tables.h -- generated by gen_math_tables.py; do not edit.
#pragma once
namespace gw {
namespace math64 {
constexpr unsigned long long kLog2e63 = 0xb8aa3b295c17f0bcull;  // 1/ln2, 63 fractional bits
constexpr unsigned long long kLn2 = 0xb17217f7d1cf79acull;      // ln2, 64 fractional bits
// 2048 times that, as two words
constexpr unsigned long long kLn2BiasHi = 0x58bull, kLn2BiasLo = 0x90bfbe8e7bcd6000ull;
constexpr unsigned long long kExp1 = 0xb17217f7d1cf79acull;  // ln2^1/1!, 64 fractional bits
constexpr unsigned long long kExp2 = 0x3d7f7bff058b1d51ull;  // ln2^2/2!, 64 fractional bits
constexpr unsigned long long kExp3 = 0xe35846b82505fc6ull;  // ln2^3/3!, 64 fractional bits
constexpr unsigned int kExp4 = 0x276556eu;  // ln2^4/4!, 32 fractional bits
constexpr unsigned int kExp5 = 0x576200u;  // ln2^5/5!, 32 fractional bits
constexpr long long kLog1 = 4611686018427387904ll;  // (-1)^0/1, 62 fractional bits
constexpr long long kLog2 = -2305843009213693952ll;  // (-1)^1/2, 62 fractional bits
constexpr long long kLog3 = 1537228672809129301ll;  // (-1)^2/3, 62 fractional bits
constexpr int kLog4 = -268435456;  // (-1)^3/4, 30 fractional bits
constexpr int kLog5 = 214748365;  // (-1)^4/5, 30 fractional bits
constexpr int kLog6 = -178956971;  // (-1)^5/6, 30 fractional bits
constexpr int kLog7 = 153391689;  // (-1)^6/7, 30 fractional bits
// 2^(j/256), 63 fractional bits
#define GW_EXP2_TABLE \
    { \
        0x8000000000000000ull, 0x8058d7d2d5e5f6b1ull, 0x80b1ed4fd999ab6cull, 0x810b40a1d81406d4ull, \
        0x8164d1f3bc030773ull, 0x81bea1708dde6056ull, 0x8218af4373fc25ecull, 0x8272fb97b2a5894cull, \
        0x82cd8698ac2ba1d7ull, 0x83285071e0fc4547ull, 0x8383594eefb6ee37ull, 0x83dea15b9541b132ull, \
        0x843a28c3acde4046ull, 0x8495efb3303efd30ull, 0x84f1f656379c1a29ull, 0x854e3cd8f9c8c95dull, \
        0x85aac367cc487b15ull, 0x86078a2f23642a9full, 0x8664915b923fba04ull, 0x86c1d919caef5c88ull, \
        0x871f61969e8d1010ull, 0x877d2afefd4e256cull, 0x87db357ff698d792ull, 0x88398146b919f1d4ull, \
        0x88980e8092da8527ull, 0x88f6dd5af155ac6bull, 0x8955ee03618e5fddull, 0x89b540a7902557a4ull, \
        0x8a14d575496efd9aull, 0x8a74ac9a79896e47ull, 0x8ad4c6452c728924ull, 0x8b3522a38e1e1032ull, \
        0x8b95c1e3ea8bd6e7ull, 0x8bf6a434adde0085ull, 0x8c57c9c4646f4ddeull, 0x8cb932c1bae97a95ull, \
        0x8d1adf5b7e5ba9e6ull, 0x8d7ccfc09c50e2f8ull, 0x8ddf042022e69cd6ull, 0x8e417ca940e35a01ull, \
        0x8ea4398b45cd53c0ull, 0x8f073af5a2013520ull, 0x8f6a8117e6c8e5c4ull, 0x8fce0c21c6726481ull, \
        0x9031dc431466b1dcull, 0x9095f1abc540ca6bull, 0x90fa4c8beee4b12bull, 0x915eed13c89689d3ull, \
        0x91c3d373ab11c336ull, 0x9228ffdc10a051adull, 0x928e727d9531f9acull, 0x92f42b88f673aa7cull, \
        0x935a2b2f13e6e92cull, 0x93c071a0eef94bc1ull, 0x9426ff0fab1c04b6ull, 0x948dd3ac8ddb7ed3ull, \
        0x94f4efa8fef70961ull, 0x955c5336887894d5ull, 0x95c3fe86d6cc7fefull, 0x962bf1cbb8d97560ull, \
        0x96942d3720185a00ull, 0x96fcb0fb20ac4ba3ull, 0x97657d49f17ab08eull, 0x97ce9255ec4357abull, \
        0x9837f0518db8a96full, 0x98a1976f7597e996ull, 0x990b87e266c189aaull, 0x9975c1dd47518c77ull, \
        0x99e0459320b7fa65ull, 0x9a4b13371fd166caull, 0x9ab62afc94ff864aull, 0x9b218d16f441d63dull, \
        0x9b8d39b9d54e5539ull, 0x9bf93118f3aa4cc1ull, 0x9c6573682ec32c2dull, 0x9cd200db8a0774cbull, \
        0x9d3ed9a72cffb751ull, 0x9dabfdff6367a2aaull, 0x9e196e189d472420ull, 0x9e872a276f0b98ffull, \
        0x9ef5326091a111aeull, 0x9f6386f8e28ba651ull, 0x9fd228256400dd06ull, 0xa041161b3d0121beull, \
        0xa0b0510fb9714fc2ull, 0xa11fd9384a344cf7ull, 0xa18faeca8544b6e4ull, 0xa1ffd1fc25cea188ull, \
        0xa27043030c496819ull, 0xa2e102153e918f9eull, 0xa3520f68e802bb93ull, 0xa3c36b345991b47cull, \
        0xa43515ae09e6809eull, 0xa4a70f0c95768ec5ull, 0xa5195786be9ef339ull, 0xa58bef536dbeb6eeull, \
        0xa5fed6a9b15138eaull, 0xa6720dc0be08a20cull, 0xa6e594cfeee86b1eull, 0xa7596c0ec55ff55bull, \
        0xa7cd93b4e965356aull, 0xa8420bfa298f70d1ull, 0xa8b6d5167b320e09ull, 0xa92bef41fa77771bull, \
        0xa9a15ab4ea7c0ef8ull, 0xaa1717a7b5693979ull, 0xaa8d2652ec907629ull, 0xab0386ef48868de1ull, \
        0xab7a39b5a93ed337ull, 0xabf13edf162675e9ull, 0xac6896a4be3fe929ull, 0xace0413ff83e5d04ull, \
        0xad583eea42a14ac6ull, 0xadd08fdd43d01491ull, 0xae493452ca35b80eull, 0xaec22c84cc5c9465ull, \
        0xaf3b78ad690a4375ull, 0xafb51906e75b8661ull, 0xb02f0dcbb6e04584ull, 0xb0a957366fb7a3c9ull, \
        0xb123f581d2ac2590ull, 0xb19ee8e8c94feb09ull, 0xb21a31a66618fe3bull, 0xb295cff5e47db4a4ull, \
        0xb311c412a9112489ull, 0xb38e0e38419fae18ull, 0xb40aaea2654b9841ull, 0xb487a58cf4a9c180ull, \
        0xb504f333f9de6484ull, 0xb58297d3a8b9f0d2ull, 0xb60093a85ed5f76cull, 0xb67ee6eea3b22b8full, \
        0xb6fd91e328d17791ull, 0xb77c94c2c9d725e9ull, 0xb7fbefca8ca41e7cull, 0xb87ba337a1743834ull, \
        0xb8fbaf4762fb9ee9ull, 0xb97c143756844dbfull, 0xb9fcd2452c0b9debull, 0xba7de9aebe5fea09ull, \
        0xbaff5ab2133e45fbull, 0xbb81258d5b704b6full, 0xbc034a7ef2e9fb0dull, 0xbc85c9c560e7b269ull, \
        0xbd08a39f580c36bfull, 0xbd8bd84bb67ed483ull, 0xbe0f6809860993e2ull, 0xbe935317fc378238ull, \
        0xbf1799b67a731083ull, 0xbf9c3c248e2486f8ull, 0xc0213aa1f0d08db0ull, 0xc0a6956e8836ca8dull, \
        0xc12c4cca66709456ull, 0xc1b260f5ca0fbb33ull, 0xc238d2311e3d6673ull, 0xc2bfa0bcfad907c9ull, \
        0xc346ccda24976407ull, 0xc3ce56c98d21b15dull, 0xc4563ecc5334cb33ull, 0xc4de8523c2c07baaull, \
        0xc5672a115506daddull, 0xc5f02dd6b0bbc3d9ull, 0xc67990b5aa245f79ull, 0xc70352f04336c51eull, \
        0xc78d74c8abb9b15dull, 0xc817f681416452b2ull, 0xc8a2d85c8ffe2c45ull, 0xc92e1a9d517f0eccull, \
        0xc9b9bd866e2f27a3ull, 0xca45c15afcc72624ull, 0xcad2265e4290774eull, 0xcb5eecd3b38597c9ull, \
        0xcbec14fef2727c5dull, 0xcc799f23d11510e5ull, 0xcd078b86503dcdd2ull, 0xcd95da6a9ff06445ull, \
        0xce248c151f8480e4ull, 0xceb3a0ca5dc6a55dull, 0xcf4318cf191918c1ull, 0xcfd2f4683f94eeb5ull, \
        0xd06333daef2b2595ull, 0xd0f3d76c75c5db8dull, 0xd184df6251699ac6ull, 0xd2164c023056bcabull, \
        0xd2a81d91f12ae45aull, 0xd33a5457a3029054ull, 0xd3ccf099859ac379ull, 0xd45ff29e0972c561ull, \
        0xd4f35aabcfedfa1full, 0xd5872909ab75d18aull, 0xd61b5dfe9f9bce07ull, 0xd6aff9d1e13ba2feull, \
        0xd744fccad69d6af4ull, 0xd7da67311797f56aull, 0xd870394c6db32c84ull, 0xd9067364d44a929cull, \
        0xd99d15c278afd7b6ull, 0xda3420adba4d8704ull, 0xdacb946f2ac9cc72ull, 0xdb63714f8e295255ull, \
        0xdbfbb797daf23755ull, 0xdc9467913a4f1c92ull, 0xdd2d818508324c20ull, 0xddc705bcd378f7f0ull, \
        0xde60f4825e0e9124ull, 0xdefb4e1f9d1037f2ull, 0xdf9612deb8f04420ull, 0xe031430a0d99e627ull, \
        0xe0ccdeec2a94e111ull, 0xe168e6cfd3295d23ull, 0xe2055afffe83d369ull, 0xe2a23bc7d7d91226ull, \
        0xe33f8972be8a5a51ull, 0xe3dd444c46499619ull, 0xe47b6ca0373da88dull, 0xe51a02ba8e26d681ull, \
        0xe5b906e77c8348a8ull, 0xe658797368b3a717ull, 0xe6f85aaaee1fce22ull, 0xe798aadadd5b9cbfull, \
        0xe8396a503c4bdc68ull, 0xe8da9958464b42abull, 0xe97c38406c4f8c57ull, 0xea1e4756550eb27bull, \
        0xeac0c6e7dd24392full, 0xeb63b74317369840ull, 0xec0718b64c1cbddcull, 0xecaaeb8ffb03ab41ull, \
        0xed4f301ed9942b84ull, 0xedf3e6b1d418a491ull, 0xee990f980da3025bull, 0xef3eab20e032bc6bull, \
        0xefe4b99bdcdaf5cbull, 0xf08b3b58cbe8b76aull, 0xf13230a7ad094509ull, 0xf1d999d8b7708cc1ull, \
        0xf281773c59ffb13aull, 0xf329c9233b6bae9cull, 0xf3d28fde3a641a5bull, 0xf47bcbbe6db9fddfull, \
        0xf5257d152486cc2cull, 0xf5cfa433e6537290ull, 0xf67a416c733f846eull, 0xf7255510c4288239ull, \
        0xf7d0df730ad13bb9ull, 0xf87ce0e5b2094d9cull, 0xf92959bb5dd4ba74ull, 0xf9d64a46eb939f35ull, \
        0xfa83b2db722a033aull, 0xfb3193cc4227c3f4ull, 0xfbdfed6ce5f09c49ull, 0xfc8ec01121e447bbull, \
        0xfd3e0c0cf486c175ull, 0xfdedd1b496a89f35ull, 0xfe9e115c7b8f884cull, 0xff4ecb59511ec8a5ull, \
    }
// {c_j, -log(c_j / 2^16) with 64 fractional bits}
#define GW_LOG_TABLE \
    { \
        {65281ull, 0xff7f551588de02ull}, {64777ull, 0x2fb6debf18dcec2ull}, \
        {64281ull, 0x4f32c10f02dd34dull}, {63792ull, 0x6e7a009f8646364ull}, \
        {63310ull, 0x8d8aec49a6ec158ull}, {62836ull, 0xac531d7e47a6a46ull}, \
        {62369ull, 0xcae148768667548ull}, {61909ull, 0xe933ac58b121f92ull}, \
        {61455ull, 0x1075993598e4f130ull}, {61008ull, 0x1254062f0a9416feull}, \
        {60568ull, 0x142e64bec266e772ull}, {60133ull, 0x1606c5a94e854a48ull}, \
        {59705ull, 0x17dae56d93235379ull}, {59283ull, 0x19abc1463fb43747ull}, \
        {58867ull, 0x1b79412bcd862a0bull}, {58457ull, 0x1d434cd6730bde4full}, \
        {58053ull, 0x1f09cbc0254f2124ull}, {57654ull, 0x20cdc825a774d78bull}, \
        {57260ull, 0x228f2f08d10d590eull}, {56872ull, 0x244cc63215d596e9ull}, \
        {56489ull, 0x26079d31c99025f7ull}, {56111ull, 0x27bfa061daf8d3afull}, \
        {55738ull, 0x2974bbe7408dcd1eull}, {55370ull, 0x2b26dbb3463311b5ull}, \
        {55007ull, 0x2cd5eb84f22b2472ull}, {54649ull, 0x2e81d6ea81dbc97aull}, \
        {54295ull, 0x302bbe428df456d5ull}, {53946ull, 0x31d25bbd110c8156ull}, \
        {53601ull, 0x3376d35d10af8c3bull}, {53261ull, 0x3517daf9105eb186ull}, \
        {52925ull, 0x36b69a3d1f93c8dcull}, {52593ull, 0x385301ab1ce201dfull}, \
        {52265ull, 0x39ed019c40144a15ull}, {51942ull, 0x3b8347415cbafa1full}, \
        {51622ull, 0x3d1846a55d36c149ull}, {51306ull, 0x3eaaaeacc54880a2ull}, \
        {50995ull, 0x40392616dafce571ull}, {50686ull, 0x41c7777f6156459full}, \
        {50382ull, 0x4351b75e6b0f2c83ull}, {50081ull, 0x44da6d0a5b73442full}, \
        {49784ull, 0x46603cb750adbd9eull}, {49490ull, 0x47e46879387dd045ull}, \
        {49200ull, 0x496590437e58e7c1ull}, {48913ull, 0x4ae4f9eae8cd1368ull}, \
        {48630ull, 0x4c614125741807aeull}, {48349ull, 0x4ddd0a8b1851f320ull}, \
        {48072ull, 0x4f55969716fc4194ull}, {47798ull, 0x50cc32a82ed25732ull}, \
        {47528ull, 0x523f720137472b12ull}, {47260ull, 0x53b208c98dd1a3baull}, \
        {46995ull, 0x55228c0eb74a0b3full}, {46733ull, 0x5690efc3dc8c081dull}, \
        {46474ull, 0x57fd27c2b2a15488ull}, {46218ull, 0x596727cc1ca9ccd5ull}, \
        {45965ull, 0x5acee388d6797625ull}, {45714ull, 0x5c35bd8a202af406ull}, \
        {45467ull, 0x5d98cd48fdcbb4c9ull}, {45222ull, 0x5efae6290860eea4ull}, \
        {44979ull, 0x605c01768802d770ull}, {44739ull, 0x61baa168dc5b03fdull}, \
        {44502ull, 0x6316b92165a429d8ull}, {44267ull, 0x6471b6ad17a9762full}, \
        {44035ull, 0x65ca160468edd914ull}, {43805ull, 0x6721490b8346057full}, \
        {43577ull, 0x6877489360bed762ull}, {43352ull, 0x69ca8a59af87a85aull}, \
        {43129ull, 0x6b1c860965281068ull}, {42908ull, 0x6c6d343b3cf98f70ull}, \
        {42690ull, 0x6dbb0474f7ef76f4ull}, {42474ull, 0x6f07742c37162906ull}, \
        {42260ull, 0x70527bc457c89ab3ull}, {42048ull, 0x719c139005bfe0f5ull}, \
        {41838ull, 0x72e433d173cd44a5ull}, {41631ull, 0x742941b9d40e0e43ull}, \
        {41425ull, 0x756e596b9b469301ull}, {41222ull, 0x76b04af8d697432eull}, \
        {41020ull, 0x77f23a641dded53full}, {40820ull, 0x79328aa1ece436ffull}, \
        {40623ull, 0x7a6f96966efc52a9ull}, {40427ull, 0x7bac8e1903b450d8ull}, \
        {40233ull, 0x7ce7cdf20a61f00dull}, {40041ull, 0x7e214ddbfd2788f3ull}, \
        {39851ull, 0x7f590583de3e4651ull}, {39662ull, 0x80909389767e73a4ull}, \
        {39476ull, 0x81c4a37e80e1d6deull}, {39291ull, 0x82f87ce935755ffbull}, \
        {39108ull, 0x842a704274706af0ull}, {38926ull, 0x855c23f6884894c8ull}, \
        {38746ull, 0x868be4661b47e680ull}, {38568ull, 0x87b9a8e4fe6bf740ull}, \
        {38392ull, 0x88e568bc4d87be8dull}, {38217ull, 0x8a10d229263aa70eull}, \
        {38044ull, 0x8b3a295da2384e51ull}, {37872ull, 0x8c63207fbaf82dc3ull}, \
        {37702ull, 0x8d89f7ac2836dcb4ull}, {37533ull, 0x8eb064f33de4980bull}, \
        {37366ull, 0x8fd4a45c537c5805ull}, {37200ull, 0x90f86fe32e775f14ull}, \
        {37036ull, 0x9219ff7a52519b1bull}, {36873ull, 0x933b1109a1877e69ull}, \
        {36712ull, 0x9459d86fe75bfd5aull}, {36552ull, 0x957817815f255709ull}, \
        {36393ull, 0x9695cb097a816dc5ull}, {36236ull, 0x97b120ca89f230b5ull}, \
        {36080ull, 0x98cbe07d407350f0ull}, {35926ull, 0x99e433d1f80e6b8bull}, \
        {35772ull, 0x9afdbb6ec63d1090ull}, {35620ull, 0x9c14cbf30ed41c49ull}, \
        {35470ull, 0x9d295bf40731c82bull}, {35320ull, 0x9e3f180014b06184ull}, \
        {35172ull, 0x9f52489b9342f600ull}, {35026ull, 0xa062e44475890483ull}, \
        {34880ull, 0xa174a36f0405f810ull}, {34735ull, 0xa285a589f4cd024aull}, \
        {34592ull, 0xa39401f9af556e0dull}, {34450ull, 0xa4a1961d20623d50ull}, \
        {34309ull, 0xa5ae5e4ad0e8242bull}, {34169ull, 0xa6ba56d23d9cc5efull}, \
        {34031ull, 0xa7c38efa89fbc2a7ull}, {33893ull, 0xa8cddb06119ed15full}, \
        {33757ull, 0xa9d55b2dcd306552ull}, {33622ull, 0xaadbf8a5d3a05444ull}, \
        {33487ull, 0xabe3a49a1df94142ull}, {33354ull, 0xace873300596024eull}, \
        {33222ull, 0xadec53874ed59eefull}, {33091ull, 0xaeef41b8b0f99e3cull}, \
        {32961ull, 0xaff139d6950d45f3ull}, {32832ull, 0xb0f237ed2b233612ull}, \
    }
}  // namespace math64
}  // namespace gw
